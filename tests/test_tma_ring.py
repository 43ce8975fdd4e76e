"""csrc/tma_ring.cuh on the CPU: the order in which the register-resident GEMM fills, awaits and uses its ring.  Counters stand in
for copies and barriers, and one wait after the other is made to run out: no copy may be started after that, every copy in flight has
to be given its time before the CTA leaves, and a slot is refilled only when its last use is over."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "dgx-serving_b200", "csrc")

DRIVER = r"""
#include "tma_ring.cuh"
#include <cstdio>
#include <vector>
static int bad = 0;
#define CHECK(c) do { if (!(c)) { printf("STAGES %d n %d fail_at %d: %s\n", STAGES, n, fail_at, #c); bad = 1; } } while (0)

template <int STAGES> void drive(int n, int fail_at) {
    int started = 0, used = 0, waited = 0, synced = 0, settled = 0;
    bool gave_up = false;
    std::vector<int> slot(STAGES, -1);
    auto copy = [&](int i, bool ok) {
        CHECK(ok == !gave_up && settled == 0);
        if (i >= n || !ok) return;
        CHECK(i == started);
        CHECK(i < STAGES || (used == i - STAGES + 1 && synced == used + 1));        // everybody has used the K-tile that was in the slot
        CHECK(i < STAGES || waited > i - STAGES);                                   // and its copies have landed
        slot[i % STAGES] = i;
        started++;
    };
    auto landed = [&](int i) {
        CHECK(!gave_up && i == waited && i < started && slot[i % STAGES] == i);
        waited++;
        gave_up = i == fail_at;
        return !gave_up;
    };
    auto sync = [&](int i) { CHECK(i == synced && i == used); synced++; };
    auto use = [&](int i) { CHECK(i == used && synced == i + 1); used++; };
    auto settle = [&]() { settled++; };
    const bool ok = w4a8::run_ring<STAGES>(n, copy, landed, sync, use, settle);
    CHECK(ok == !gave_up && used == n && synced == n && settled == (gave_up ? 1 : 0));
    CHECK(started == (gave_up && fail_at + STAGES - 1 < n ? fail_at + STAGES - 1 : n));
}
int main() {
    for (int n = 0; n < 14; n++)
        for (int f = -1; f < n; f++) { drive<2>(n, f); drive<3>(n, f); drive<4>(n, f); drive<5>(n, f); }
    return bad;
}
"""


def test_a_wait_that_runs_out_leaves_no_copy_behind(tmp_path):
    src, exe = tmp_path / "ring.cpp", tmp_path / "ring"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def test_kernel_waits_for_its_operands_in_that_order_only():
    """The kernel's one wait is the one that run_ring calls, and one thread starts all bulk copies, if it may."""
    text = open(os.path.join(CSRC, "gemm_w4a8_mma.cuh")).read()
    assert text.count("run_ring<STAGES>(nkt, copy, landed, sync, use, settle)") == 1 and text.count("ptx::mbar_wait(") == 1
    assert "ptx::mbar_wait(" in text[text.index("auto landed = "):text.index("auto sync = ")]
    assert "clock64() - t0 < (1ll << 21)" in text[text.index("auto settle = "):text.index("run_ring<STAGES>")]
    copy = text[text.index("auto copy = "):text.index("cp_async_commit();\n    };")]
    guarded = copy[copy.index("== ISSUER && ok) {"):copy.index("// scales:")]
    assert text.count("ptx::tma_load_2d(") == guarded.count("ptx::tma_load_2d(") and "ptx::mbar_arrive_expect_tx(" not in text.replace(guarded, "")
