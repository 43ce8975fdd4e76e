"""Every tile of the register-resident GEMM (csrc/gemm_w4a8_mma.cuh) at the edges of its rows, columns and K, bit for bit
against the oracle's MMQ order: 16- to 64-row tiles, 48- and 64-row tiles repeated, 128 x 128 tiles, rows, columns and K-tiles
that end ragged, odd N (unpaired stores), rows of scales that are not a multiple of four through more K-tiles than the ring
has stages, split K with ranges that are not, and with an empty last range; the few tiles with such scales that stay on the
tcgen05 kernel too.  Each case names the kernel and tile the dispatch has to choose for it on 148 SMs, so that no later rule
can leave one of them untested."""
import re

import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu

# (M, N, K, rows of the tile, 0: tcgen05).  K / 32 is a multiple of four in the first list: scales copied 16 (8) bytes at a time.
LINED_UP = [(1, 8, 128, 16), (16, 129, 256, 16), (17, 130, 640, 32), (32, 300, 512, 32), (33, 128, 1152, 48), (48, 257, 256, 48),
            (49, 131, 640, 64), (64, 384, 2048, 64), (65, 200, 128, 48), (100, 130, 640, 48), (193, 4095, 256, 64), (150, 17401, 384, 64), (130, 1000, 128, 48),
            (193, 7700, 128, 0), (2047, 2046, 128, 128), (2048, 2047, 640, 128)]
# ... and not here: element by element, wherever more than two CTAs per SM cover those loads
ELEMENTWISE = [(1, 8, 32, 16), (16, 129, 96, 16), (9, 40, 1120, 16), (17, 37889, 288, 32), (33, 37889, 544, 48), (49, 37890, 544, 64),
               (64, 38000, 672, 64), (129, 17408, 64, 48), (145, 23809, 288, 64), (2048, 2048, 160, 128), (2040, 2047, 544, 128),
               (17, 40, 160, 0), (33, 128, 1120, 0), (49, 131, 544, 0), (64, 384, 2080, 0), (96, 520, 288, 0)]
# (M, N, K, splits, rows of the tile)
SPLIT_K = [(64, 1, 2048, 8, 64), (24, 258, 1024, 3, 32), (48, 12801, 960, 3, 48), (20, 9600, 288, 4, 32), (64, 5000, 1120, 8, 64), (3, 130, 1120, 3, 16),
           (100, 8000, 480, 3, 64), (48, 130, 1120, 3, 0), (20, 300, 160, 4, 0), (70, 256, 480, 2, 0)]


def tile_rows(names):
    """Rows of the one GEMM launch's tile, 0 for the tcgen05 kernel."""
    gemm = [n for n in names if "gemm_w4a8" in n]
    assert len(gemm) == 1, names
    m = re.search(r"gemm_w4a8_mma_kernelI.*?3CfgILi(\d+)ELi\d+ELi(\d+)E", gemm[0])
    if m is None:
        assert "gemm_w4a8_tc_kernel" in gemm[0], gemm
        return 0
    return 16 * int(m.group(1)) * int(m.group(2))


def operands(oracle, cuda, M, N, K, scale_dtype, seed):
    import torch
    X = oracle.make_activations(M, K, seed=seed, outliers=True)
    Wq, sw = oracle.make_weights(N, K, seed=seed + 1, scale_dtype=scale_dtype)
    xq, xs, _ = oracle.quantize_x_q8(X)
    return (xq, xs, Wq, sw), [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in (xq, xs, Wq, sw)]


@pytest.fixture
def sms148(cuda):
    import torch
    if torch.cuda.get_device_properties(cuda).multi_processor_count != 148:
        pytest.skip("the tile each shape takes is worked out for 148 SMs")


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("M,N,K,rows", LINED_UP + ELEMENTWISE)
def test_gemm_tiles(w4a8, oracle, cuda, sms148, M, N, K, rows, scale_dtype):
    import torch
    host, d = operands(oracle, cuda, M, N, K, scale_dtype, M + N + K)
    Y = torch.full((M + 1, N), 7.0, dtype=torch.float32, device=cuda)            # the last row is a canary

    def call(stream):
        w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, stream)

    call(None)
    w4a8.device_status()
    assert tile_rows(launched_kernels(call)) == rows
    y = Y.cpu().numpy()
    assert np.array_equal(y[:M].view(np.uint32), oracle.gemm_mmq_w4a8(*host).view(np.uint32))
    assert np.all(y[M] == 7.0)


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("M,N,K,splitk,rows", SPLIT_K)
def test_gemm_tiles_split_k(w4a8, oracle, cuda, sms148, M, N, K, splitk, rows, scale_dtype):
    import torch
    host, d = operands(oracle, cuda, M, N, K, scale_dtype, 3)
    Y = torch.empty((M, N), dtype=torch.float32, device=cuda)
    ws = torch.full((w4a8.gemm_splitk_workspace_bytes(M, N, K, splitk),), 255, dtype=torch.uint8, device=cuda)   # NaNs: all of it is written

    def call(stream):
        w4a8.launch_gemm_bm16_splitk(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, splitk, ws, stream)

    call(None)
    torch.cuda.synchronize()
    assert tile_rows(launched_kernels(call)) == rows
    assert np.array_equal(Y.cpu().numpy().view(np.uint32), oracle.gemm_splitk_w4a8(*host, splitk).view(np.uint32))


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("M,N,K,rows", [(16, 130, 256, 16), (17, 130, 640, 32), (48, 130, 256, 48), (64, 130, 512, 64), (49, 131, 544, 0),
                                        (193, 7700, 128, 0), (2048, 2047, 128, 128)])
def test_tiny_activation_scales(w4a8, oracle, cuda, sms148, M, N, K, rows, kernel, scale_dtype):
    """Activation scales down to a few multiples of the smallest subnormal: a factor folded into them would lose bits, and the
    tile that M and N select would show in the result."""
    import torch
    (xq, xs, Wq, sw), _ = operands(oracle, cuda, M, N, K, 0, 17)
    rng = np.random.default_rng(18)
    xs = np.ldexp(rng.uniform(1, 4, xs.shape), rng.integers(-146, -115, (M, 1))).astype(np.float32)
    sw = (sw * 1000).astype(np.float16 if scale_dtype else np.float32)
    d = [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in (xq, xs, Wq, sw)]
    Y = torch.empty((M, N), dtype=torch.float32, device=cuda)
    w4a8.config("gemm_kernel", kernel)
    try:
        def call(stream):
            w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, stream)
        call(None)
        w4a8.device_status()
        assert kernel == 0 or tile_rows(launched_kernels(call)) == rows
    finally:
        w4a8.config("gemm_kernel", 1)
    assert np.array_equal(Y.cpu().numpy().view(np.uint32), oracle.gemm_mmq_w4a8(xq, xs, Wq, sw).view(np.uint32))
