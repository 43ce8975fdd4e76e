"""Several matrices against two to sixteen shared rows in one launch: every matrix has the bits of its own call and the oracle's MMQ
order; row counts that end inside a 16-row tile, one tile or many per CTA, both step lengths, with and without the relay.  Where outputs
share memory the matrices keep their order instead."""
import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("S,K,OUTS", [(2, 512, (1, 17)), (8, 2048, (300, 200)), (8, 2304, (1000, 8, 31, 500)), (3, 256, (5000, 3001)),
                                      (16, 1536, (2000, 2000)), (9, 768, (40, 7)), (16, 2816, (3000, 2500, 100)), (8, 1280, (20000, 9000)),
                                      (16, 512, (300, 17)), (9, 512, (300, 17)), (16, 2048, (5000, 3001)), (9, 2048, (5000, 3001)),
                                      (12, 1536, (2000, 3000)), (12, 3840, (4000, 900))])    # each is relayed alone, together they are not
def test_one_launch(w4a8, oracle, cuda, S, K, OUTS, scale_dtype):
    import torch
    X = oracle.make_activations(S, K, seed=S + K, outliers=True)
    xq, xs, _ = oracle.quantize_x_q8(X)
    mats = [oracle.make_weights(n, K, seed=n + i, scale_dtype=scale_dtype) for i, n in enumerate(OUTS)]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xq_d, xs_d, Wq_d, sw_d = dev(xq), dev(xs), [dev(w) for w, _ in mats], [dev(s) for _, s in mats]
    Ys = [torch.full((S + 1, n), float("nan"), dtype=torch.float32, device=cuda) for n in OUTS]     # last row: canary

    def call(stream):
        w4a8.gemv_multi(xq_d, xs_d, Wq_d, sw_d, Ys, OUTS, K, S, scale_dtype, stream)

    call(None)
    w4a8.device_status()
    names = launched_kernels(call)
    tiles = sum((n + 15) // 16 for n in OUTS)
    few = S <= 8 or (tiles <= 2 * 148 and (K >= 1536 or K // 256 % 2 == 1))            # up to eight rows it is the same kernel
    steps = "Li8ELi3E" if K // 256 % 2 == 1 or (S > 8 and few) else "Li16ELi2E"
    want = "gemv_w4a8_mma_kernelILi%dE%s%sLb0ELb1ELb%dE" % (1 if S <= 8 else 2, steps, ("f", "6__half")[scale_dtype], few)
    assert len(names) == 1, names
    assert want in names[0] or torch.cuda.get_device_properties(0).multi_processor_count != 148, (want, names)
    for y, n, (Wq, sw), wd, sd in zip(Ys, OUTS, mats, Wq_d, sw_d):
        Y1 = torch.empty((S, n), dtype=torch.float32, device=cuda)
        w4a8.launch_gemv_w4a8_sb(xq_d, xs_d, wd, sd, Y1, K, n, S, scale_dtype)
        y = y.cpu().numpy()
        assert np.all(np.isnan(y[S]))
        assert np.array_equal(y[:S].view(np.uint32), Y1.cpu().numpy().view(np.uint32))
        if n * K <= 6000000:
            assert np.array_equal(y[:S].view(np.uint32), oracle.gemm_mmq_w4a8(xq, xs, Wq, sw).view(np.uint32))


@pytest.mark.parametrize("S,K,OUTS", [(8, 512, (300, 300)), (12, 2048, (300, 200)), (1, 2048, (500, 500)), (1, 4096, (300, 200))])
def test_outputs_that_share_memory_keep_their_order(w4a8, oracle, cuda, S, K, OUTS):
    """The second matrix's output lies over the first one's: what both calls write is the second's, as with two calls."""
    import torch
    xq, xs, _ = oracle.quantize_x_q8(oracle.make_activations(S, K, seed=K, outliers=True))
    mats = [oracle.make_weights(n, K, seed=n + i) for i, n in enumerate(OUTS)]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xq_d, xs_d, Wq_d, sw_d = dev(xq), dev(xs), [dev(w) for w, _ in mats], [dev(s) for _, s in mats]
    shift = 40
    got, want = (torch.full((S * max(OUTS) + shift,), float("nan"), device=cuda) for _ in range(2))
    call = lambda stream: w4a8.gemv_multi(xq_d, xs_d, Wq_d, sw_d, [got, got[shift:]], OUTS, K, S, 0, stream)
    for i, n in enumerate(OUTS):
        w4a8.launch_gemv_w4a8_sb(xq_d, xs_d, Wq_d[i], sw_d[i], want[shift * i:], K, n, S)
    call(None)
    w4a8.device_status()
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want.cpu().numpy().view(np.uint32))
    assert len(launched_kernels(call)) == 2
