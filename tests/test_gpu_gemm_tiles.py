"""Every tile of the register-resident GEMM (csrc/gemm_w4a8_mma.cuh) at the edges of its rows, columns and K, bit for bit
against the oracle's MMQ order: 16- to 64-row tiles, 48- and 64-row tiles repeated, 128 x 128 tiles, rows, columns and K-tiles
that end ragged, odd N (unpaired stores), rows of scales that are not a multiple of four, split K with an empty last range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 8, 32), (16, 129, 96), (17, 40, 160), (32, 300, 512), (33, 128, 1120), (48, 257, 256), (49, 131, 544), (64, 384, 2080),
          (65, 200, 128), (96, 520, 288), (100, 130, 640), (130, 1000, 128), (2048, 2048, 160), (2047, 2046, 128), (129, 17408, 64)]


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("M,N,K", SHAPES)
def test_gemm_tiles(w4a8, oracle, cuda, M, N, K, scale_dtype):
    import torch
    X = oracle.make_activations(M, K, seed=M + N, outliers=True)
    Wq, sw = oracle.make_weights(N, K, seed=K + N, scale_dtype=scale_dtype)
    xq, xs, _ = oracle.quantize_x_q8(X)
    d = [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in (xq, xs, Wq, sw)]
    Y = torch.full((M + 1, N), 7.0, dtype=torch.float32, device=cuda)            # the last row is a canary
    w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype)
    w4a8.device_status()
    y = Y.cpu().numpy()
    assert np.array_equal(y[:M].view(np.uint32), oracle.gemm_mmq_w4a8(xq, xs, Wq, sw).view(np.uint32))
    assert np.all(y[M] == 7.0)


@pytest.mark.parametrize("M,N,K,splitk", [(48, 130, 1120, 3), (20, 300, 160, 4), (70, 256, 480, 2), (64, 1, 2048, 8)])
def test_gemm_tiles_split_k(w4a8, oracle, cuda, M, N, K, splitk):
    import torch
    X = oracle.make_activations(M, K, seed=3)
    Wq, sw = oracle.make_weights(N, K, seed=4)
    xq, xs, _ = oracle.quantize_x_q8(X)
    d = [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in (xq, xs, Wq, sw)]
    Y = torch.empty((M, N), dtype=torch.float32, device=cuda)
    ws = torch.full((w4a8.gemm_splitk_workspace_bytes(M, N, K, splitk),), 255, dtype=torch.uint8, device=cuda)   # NaNs: all of it is written
    w4a8.launch_gemm_bm16_splitk(d[0], d[1], d[2], d[3], Y, M, N, K, 0, splitk, ws)
    torch.cuda.synchronize()
    assert np.array_equal(Y.cpu().numpy().view(np.uint32), oracle.gemm_splitk_w4a8(xq, xs, Wq, sw, splitk).view(np.uint32))
