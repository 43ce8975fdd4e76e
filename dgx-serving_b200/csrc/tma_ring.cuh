// The order in which a CTA fills, awaits and uses the slots of a shared-memory ring, and how it leaves when a wait runs out.
// No CUDA construct in it: the same text is driven on the CPU with counters in place of copies and barriers.
#pragma once
#ifdef __CUDACC__
#define W4A8_RING_FN __device__ __forceinline__
#else
#define W4A8_RING_FN inline
#endif

namespace w4a8 {

// n K-tiles through STAGES slots, STAGES - 1 of them in flight; what each thread of the CTA does.
//   copy(i, ok)  the thread that starts bulk copies starts those of K-tile i into slot i % STAGES, if ok; nothing for i >= n
//   landed(i)    waits for them, bounded
//   sync(i)      the CTA's barrier: K-tile i has landed for everybody, everybody is done with K-tile i - 1
//   use(i)       reads slot i % STAGES
//   settle()     gives copies in flight the time to end
// False when a wait of this thread ran out; it then waits no more and what it uses is void.  The thread that starts the copies goes
// by its own waits, which cover every slot it refills: after one that ran out it starts no copy, because the slot's barrier may not
// have completed its phase and one more arrival would corrupt it, and it settles before the CTA can leave, because shared memory
// that a copy still writes to would be the next CTA's.  Neither a vote of the CTA on the outcome nor anything but a branch inside
// the loop: 48 rows x 3840 x 15360 in three ranges 36.0 us so, 36.7 with the settling inside.
template <int STAGES, class Copy, class Landed, class Sync, class Use, class Settle>
W4A8_RING_FN bool run_ring(int n, Copy &&copy, Landed &&landed, Sync &&sync, Use &&use, Settle &&settle) {
    bool ok = true;
#pragma unroll
    for (int s = 0; s < STAGES - 1; s++) copy(s, true);
    for (int i = 0; i < n; i++) {
        if (ok && !landed(i)) ok = false;
        sync(i);
        copy(i + STAGES - 1, ok);                     // into the slot K-tile i - 1 used
        use(i);
    }
    if (!ok) settle();
    return ok;
}

}  // namespace w4a8
