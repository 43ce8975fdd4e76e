"""Every tile of the register-resident GEMM (csrc/gemm_w4a8_mma.cuh) at the edges of its rows, columns and K, bit for bit
against the oracle's MMQ order: 16- to 96-row tiles alone and repeated, rows, columns and K-tiles that end ragged, odd N
(unpaired stores), the three ways of copying scales (K / 32 and the ranges of a split K multiples of four, even, odd)
through more K-tiles than the ring has stages, and split K with an empty last range.  Each case names the tile that the
dispatch has to choose for it on 148 SMs, so that no later rule can leave one of them untested; the names follow the rule."""
import re

import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu

# The kernels: rows of the tile / stages of its ring, "e" where scales do not line up (VEC = false).  A pair where fp32 and fp16
# scales differ.
# (M, N, K, kernel); K / 32 is a multiple of four
LINED_UP = [(1, 8, 128, "16/4"), (16, 129, 256, "16/4"), (17, 130, 640, "16/4"), (32, 300, 512, "16/4"),
            (65, 200, 128, "16/4"), (100, 130, 640, "16/4"), (33, 9601, 1152, "48/4"), (48, 15001, 256, "48/4"),
            (130, 1000, 128, "16/4"), (64, 15001, 640, "64/4"), (193, 4095, 256, "32/4"), (150, 17401, 384, "80/4"),
            (64, 20001, 512, "32/4"), (2047, 2046, 128, "48/4"), (2048, 2047, 640, "48/4"), (193, 7700, 128, "32/4"),
            (193, 12723, 128, ("32/4", "64/3")), (147, 14287, 128, "80/4"), (262, 11397, 128, "96/4"),
            (97, 15171, 128, "64/4")]
# ... even, or odd
OTHERS = [(1, 8, 32, "16/4e"), (16, 129, 96, "16/4e"), (9, 40, 1120, "16/4e"), (17, 40, 160, "16/4e"),
          (32, 300, 1120, "16/4e"), (64, 384, 2080, "16/4e"), (33, 140, 1600, "16/4e"), (33, 37889, 544, "48/4e"),
          (48, 12001, 704, ("48/4e", "16/4e")), (129, 17408, 64, "48/4e"), (200, 3001, 320, "48/4e"),
          (333, 5001, 352, "32/4e"), (49, 37890, 544, ("32/4e", "64/3e")), (64, 9601, 704, ("64/4e", "32/4e")),
          (145, 23809, 288, "64/4e"), (64, 15001, 736, "64/4e"), (2040, 2047, 544, "48/4e"),
          (250, 6000, 544, "32/4e"), (104, 14336, 1600, "64/4e"), (201, 12621, 96, ("32/4e", "64/3e")),
          (164, 14495, 96, ("96/4e", "64/3e")), (99, 14311, 96, "64/4e"), (149, 14307, 96, "80/4e"),
          (259, 11493, 96, "96/4e"), (171, 3105, 224, "48/4e"), (149, 14307, 64, "80/4e"),
          (201, 12621, 64, ("32/4e", "64/3e")), (259, 11493, 64, "96/4e")]
# (M, N, K, splits, kernel)
SPLIT_K = [(64, 1, 2048, 8, "16/4"), (24, 258, 1024, 3, "16/4"), (48, 3840, 1536, 3, "16/4"),
           (64, 4000, 1024, 3, ("16/4", "32/4")), (48, 12801, 960, 3, "48/4e"), (20, 9600, 288, 4, "32/4e"),
           (64, 5000, 1120, 8, ("32/4e", "64/3e")), (3, 130, 1120, 3, "16/4e"),
           (100, 8000, 480, 3, ("32/4e", "64/3e")), (48, 130, 1120, 3, "16/4e"), (20, 300, 160, 4, "16/4e"),
           (70, 256, 480, 2, "16/4e"), (300, 7000, 1024, 2, ("80/4", "64/3")), (96, 1500, 992, 2, "16/4e"),
           (98, 7049, 512, 2, "64/4"), (195, 6307, 512, 2, ("32/4", "64/3")), (33, 6421, 512, 2, "48/4")]


def tile_name(names):
    """Which kernel the one GEMM launch among the names is."""
    gemm = [n for n in names if "gemm_w4a8" in n]
    assert len(gemm) == 1, names
    m = re.search(r"gemm_w4a8_mma_kernelI.*?3CfgILi(\d+)ELi\d+ELi(\d+)ELi\d+ELi(\d+)ELi\d+EE.*?Lb0ELb([01])E", gemm[0])
    assert m, gemm
    return "%d/%s%s" % (16 * int(m.group(1)) * int(m.group(2)), m.group(3), "" if m.group(4) == "1" else "e")


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
@pytest.mark.parametrize("M,N,K,kernel", LINED_UP + OTHERS)
def test_gemm_tiles(w4a8, oracle, cuda, sms148, M, N, K, kernel, scale_dtype):
    import torch
    host, d = operands(oracle, cuda, M, N, K, scale_dtype, M + N + K)
    Y = torch.full((M + 1, N), 7.0, dtype=torch.float32, device=cuda)            # the last row is a canary

    def call(stream):
        w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, stream)

    call(None)
    w4a8.device_status()
    assert tile_name(launched_kernels(call)) == (kernel if isinstance(kernel, str) else kernel[scale_dtype])
    y = Y.cpu().numpy()
    assert np.array_equal(y[:M].view(np.uint32), oracle.gemm_mmq_w4a8(*host).view(np.uint32))
    assert np.all(y[M] == 7.0)


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("M,N,K,splitk,kernel", SPLIT_K)
def test_gemm_tiles_split_k(w4a8, oracle, cuda, sms148, M, N, K, splitk, kernel, scale_dtype):
    import torch
    host, d = operands(oracle, cuda, M, N, K, scale_dtype, 3)
    Y = torch.empty((M, N), dtype=torch.float32, device=cuda)
    ws = torch.full((w4a8.gemm_splitk_workspace_bytes(M, N, K, splitk),), 255, dtype=torch.uint8, device=cuda)   # NaNs: all of it is written

    def call(stream):
        w4a8.launch_gemm_bm16_splitk(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, splitk, ws, stream)

    call(None)
    torch.cuda.synchronize()
    assert tile_name(launched_kernels(call)) == (kernel if isinstance(kernel, str) else kernel[scale_dtype])
    assert np.array_equal(Y.cpu().numpy().view(np.uint32), oracle.gemm_splitk_w4a8(*host, splitk).view(np.uint32))


@pytest.mark.parametrize("shift_xs,shift_sw", [(1, 0), (0, 1), (0, 2)])
@pytest.mark.parametrize("scale_dtype", [0, 1])
def test_unaligned_scales(w4a8, oracle, cuda, sms148, scale_dtype, shift_xs, shift_sw):
    """Scales whose rows would line up, at addresses that do not: fp16 ones at odd multiples of two bytes among them."""
    import torch
    M, N, K = 32, 300, 768
    host, d = operands(oracle, cuda, M, N, K, scale_dtype, 5)
    for i, shift in ((1, shift_xs), (3, shift_sw)):
        flat = torch.zeros(d[i].numel() + 8, dtype=d[i].dtype, device=cuda)
        flat[shift:shift + d[i].numel()] = d[i].reshape(-1)
        d[i] = flat[shift:]
    Y = torch.empty((M, N), dtype=torch.float32, device=cuda)

    def call(stream):
        w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, stream)

    call(None)
    w4a8.device_status()
    assert tile_name(launched_kernels(call)) == "16/4e"
    assert np.array_equal(Y.cpu().numpy().view(np.uint32), oracle.gemm_mmq_w4a8(*host).view(np.uint32))


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("policy", [0, 1])
@pytest.mark.parametrize("M,N,K,kernel", [(16, 130, 256, "16/4"), (17, 130, 640, "16/4"), (48, 15001, 256, "48/4"),
                                          (64, 15001, 256, ("16/4", "32/4")), (150, 17401, 128, "80/4"),
                                          (49, 131, 544, "16/4e"), (64, 9601, 224, "16/4e"),
                                          (193, 7700, 128, "32/4"), (2048, 2047, 128, "48/4"),
                                          (193, 12723, 128, ("32/4", "64/3")), (97, 15171, 128, "64/4"),
                                          (262, 11397, 128, "96/4"), (149, 14307, 96, "80/4e")])
def test_tiny_activation_scales(w4a8, oracle, cuda, sms148, M, N, K, kernel, policy, scale_dtype):
    """Activation scales down to a few multiples of the smallest subnormal: a factor folded into them would lose bits, and the
    tile that M and N select would show in the result."""
    import torch
    (xq, xs, Wq, sw), _ = operands(oracle, cuda, M, N, K, 0, 17)
    rng = np.random.default_rng(18)
    xs = np.ldexp(rng.uniform(1, 4, xs.shape), rng.integers(-146, -115, (M, 1))).astype(np.float32)
    sw = (sw * 1000).astype(np.float16 if scale_dtype else np.float32)
    d = [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in (xq, xs, Wq, sw)]
    Y = torch.empty((M, N), dtype=torch.float32, device=cuda)
    w4a8.config("gemm_kernel", policy)
    try:
        def call(stream):
            w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, stream)
        call(None)
        w4a8.device_status()
        assert policy == 0 or tile_name(launched_kernels(call)) == (kernel if isinstance(kernel, str) else kernel[scale_dtype])
    finally:
        w4a8.config("gemm_kernel", 1)
    assert np.array_equal(Y.cpu().numpy().view(np.uint32), oracle.gemm_mmq_w4a8(xq, xs, Wq, sw).view(np.uint32))
