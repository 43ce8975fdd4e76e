"""Decode products of 9 to 16 rows around the sizes at which several warps take turns at a tile (at most two 16-row tiles per CTA on 148
SMs; rows of 48 groups or more, or of an odd multiple of eight), and past the last row of the matrix: the kernel that the plan names, and
bit for bit the oracle's MMQ order."""
import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("S,N,K", [(9, 1, 1536), (16, 17, 1536), (12, 300, 1280), (16, 2368, 2048), (10, 2500, 2304), (13, 4729, 1536),
                                   (16, 4736, 1536), (9, 4737, 1536), (16, 1000, 3840), (11, 2371, 5376), (16, 40, 8192),
                                   (12, 2254, 256), (9, 405, 768), (13, 1065, 1280), (10, 5000, 768), (14, 700, 512), (16, 3000, 1024)])
def test_9_to_16_rows(w4a8, oracle, cuda, S, N, K, scale_dtype):
    import torch
    X = oracle.make_activations(S, K, seed=S + N, outliers=True)
    Wq, sw = oracle.make_weights(N, K, seed=K, scale_dtype=scale_dtype)
    xq, xs, _ = oracle.quantize_x_q8(X)
    d = [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in (xq, xs, Wq, sw)]
    Y = torch.full((S + 1, N), 7.0, dtype=torch.float32, device=cuda)            # the last row is a canary

    def call(stream):
        w4a8.launch_gemv_w4a8_sb(d[0], d[1], d[2], d[3], Y, K, N, S, scale_dtype, stream)

    call(None)
    w4a8.device_status()
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        relayed = N <= 16 * 2 * 148 and (K >= 1536 or K // 256 % 2 == 1)
        steps = "Li8ELi3E" if relayed or K // 256 % 2 == 1 else "Li16ELi2E"
        # rows / 8, groups per step, stages, scales, peers, several matrices, relay
        assert ["gemv_w4a8_mma_kernelILi2E%s%sLb0ELb0ELb%dE" % (steps, ("f", "6__half")[scale_dtype], relayed) in n for n in launched_kernels(call)] == [True]
    y = Y.cpu().numpy()
    assert np.array_equal(y[:S].view(np.uint32), oracle.gemm_mmq_w4a8(xq, xs, Wq, sw).view(np.uint32))
    assert np.all(y[S] == 7.0)
