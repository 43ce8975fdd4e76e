"""csrc/gemv_mma_plan.cuh on the CPU, over all row counts and row lengths: a launch's static and dynamic shared memory together are what
a CTA may have, and the relay's mailboxes never cost a call its plan."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dgx-serving_b200", "csrc")

DRIVER = r"""
#include "gemv_mma_plan.cuh"
#include <cstdio>
#include <initializer_list>
using namespace w4a8::gemv_mma;
int main() {
    int bad = 0;
    const long outs[] = {1, 24, 4735, 4736, 4737, 17408, 151936};
    for (int S = 1; S <= 16; S++)
        for (int nb = 1; nb <= 4096; nb++)
            for (long out : outs)
                for (int gs : {16, 8})
                    for (int st : {0, 2, 3, 4, 6, 8}) {
                        bool fits = false;                              // some ring beside the rows, mailboxes aside
                        for (int g : {16, 8})
                            for (int s : {2, 3, 4, 6, 8}) {
                                const bool exists = g == 16 ? s <= 4 : (s == 3 || s >= 6);
                                if (exists && g <= gs && nb % g == 0 && s <= (st ? st : g == 16 ? 2 : 3) && smem_bytes(S > 8 ? 2 : 1, S, nb, g, s) <= SMEM_LIMIT) fits = true;
                            }
                        Plan p = {};
                        const bool ok = plan_rows(nb, out, S, 148, gs, st, &p);
                        bool good = ok == fits;
                        if (ok) {
                            const bool boxes = p.MH == 1 || p.relay;
                            good = good && p.MH == (S > 8 ? 2 : 1) && nb % p.GS == 0;
                            good = good && launch_smem(p.MH, S, nb, p.GS, p.STAGES) + static_bytes(p.MH, boxes) <= SMEM_CTA;
                            good = good && (!p.relay || (p.MH == 2 && p.GS == 8 && p.STAGES == 3 && (out + 7) / 8 <= 4 * 148));
                        }
                        if (!good && bad++ < 10) printf("S %d nb %d OUT %ld gs %d st %d: %d %d, MH %d GS %d STAGES %d relay %d\n", S, nb, out, gs, st, ok, fits, p.MH, p.GS, p.STAGES, p.relay);
                    }
    // more than eight rows: one CTA per SM, whose 228 KB hold 1 KB more than it asks for
    for (int nb = 8; nb <= 512; nb += 8) {
        Plan p = {};
        if (plan_rows(nb, 9000, 12, 148, 16, 0, &p) && 2 * (launch_smem(p.MH, 12, nb, p.GS, p.STAGES) + 1024) <= 228 * 1024) { printf("nb %d\n", nb); bad++; }
    }
    // rows beside which the mailboxes of 9 to 16 rows do not fit
    const int full[][2] = {{16, 9216}, {11, 12800}, {10, 13824}, {9, 15104}};
    for (auto &f : full) {
        Plan p = {};
        if (!plan_rows(f[1] / 32, 24, f[0], 148, 16, 0, &p) || p.relay || p.GS != 8) { printf("%d x %d\n", f[0], f[1]); bad++; }
    }
    return bad != 0;
}
"""


def test_shared_memory_of_every_plan(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", CSRC, str(src), "-o", str(exe)], check=True, capture_output=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
