"""Tiles of the register-resident GEMM (csrc/gemm_w4a8_mma.cuh) through many turns of the ring: ragged rows, columns and last
K-tiles, the three ways of copying scales, one range of K and several, the last of them shorter.  Bit for bit against the tcgen05
kernel with fp16 operands, which shares no code with them, and the smallest against the oracle.  Each case names the tile the
dispatch has to choose on 148 SMs."""
import numpy as np
import pytest

from test_gpu_gemm_tiles import operands, sms148, tile_name  # noqa: F401 (sms148 is a fixture)
from conftest import launched_kernels

pytestmark = pytest.mark.gpu

# (M, N, K, tile for fp32 scales, for fp16 scales)
CASES = [(1, 3, 2176, "16/4", "16/4"), (31, 129, 2176, "16/4", "16/4"), (33, 9489, 2176, "48/4", "48/4"),
         (49, 9528, 2176, "64/4", "64/3"), (129, 7620, 2176, "80/4", "80/4"), (241, 9508, 2176, "96/4", "96/4"),
         (6, 1, 2112, "16/4e", "16/4e"), (42, 130, 2112, "16/4e", "16/4e"), (33, 9551, 2112, "48/4e", "16/4e"),
         (65, 9496, 2112, "32/4e", "32/4e"), (161, 6282, 2112, "32/4e", "32/4e"), (49, 9473, 2112, "64/4e", "64/3e"),
         (2, 9, 2144, "16/4e", "16/4e"), (55, 131, 2144, "16/4e", "16/4e"), (33, 9474, 2144, "48/4e", "48/4e"),
         (129, 7554, 2144, "80/4e", "80/4e"), (241, 9505, 2144, "96/4e", "96/4e"),
         (162, 9478, 2144, "64/4e", "64/4e"), (97, 14273, 2176, "64/4", "64/4"), (65, 9913, 2176, "80/4", "80/4"),
         (162, 103, 2176, "32/4", "32/4"), (50, 9487, 2176, "64/4", "64/3"), (33, 12589, 2112, "48/4e", "48/4e"),
         (98, 14285, 2112, "64/4e", "64/4e"), (65, 12627, 2112, "80/4e", "80/4e"),
         (163, 14401, 2112, "96/4e", "96/4e"), (49, 9475, 2112, "64/4e", "64/3e"),
         (33, 9755, 2144, "48/4e", "48/4e"), (65, 12573, 2144, "80/4e", "80/4e"),
         (162, 14321, 2144, "96/4e", "96/4e"), (250, 12555, 2144, "64/4e", "64/3e")]
# (M, N, K, splits, tile for fp32, for fp16 scales): ranges of 72, 72 and 68 groups, of 70, 70 and 66, of 66, 66 and 63
SPLIT_K = [(6, 101, 6784, 3, "16/4", "16/4"), (172, 101, 6784, 3, "32/4", "32/4"),
           (34, 3303, 6784, 3, "48/4", "48/4"), (97, 4767, 6784, 3, "64/4", "64/4"),
           (67, 3077, 6784, 3, "80/4", "80/4"), (243, 3085, 6784, 3, "96/4", "96/4"),
           (49, 3077, 6784, 3, "64/4", "64/3"), (10, 129, 6592, 3, "16/4e", "16/4e"),
           (169, 107, 6592, 3, "32/4e", "32/4e"), (33, 4225, 6592, 3, "48/4e", "48/4e"),
           (97, 4803, 6592, 3, "64/4e", "64/4e"), (65, 4149, 6592, 3, "80/4e", "80/4e"),
           (241, 3155, 6592, 3, "96/4e", "96/4e"), (50, 3095, 6592, 3, "64/4e", "64/3e"),
           (5, 119, 6240, 3, "16/4e", "16/4e"), (162, 119, 6240, 3, "32/4e", "32/4e"),
           (34, 3145, 6240, 3, "48/4e", "48/4e"), (49, 3073, 6240, 3, "64/4e", "64/4e"),
           (65, 4167, 6240, 3, "80/4e", "80/4e"), (241, 3147, 6240, 3, "96/4e", "96/4e"),
           (242, 4097, 6240, 3, "64/4e", "64/3e")]


def fp16_operands(w4a8, call):
    import torch
    w4a8.config("gemm_kernel", 0)
    try:
        call(None)
        torch.cuda.synchronize()
    finally:
        w4a8.config("gemm_kernel", 1)


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("M,N,K,splitk,fp32,fp16", SPLIT_K)
def test_gemm_long_ranges_of_a_split_k(w4a8, oracle, cuda, sms148, M, N, K, splitk, fp32, fp16, scale_dtype):  # noqa: F811
    import torch
    host, d = operands(oracle, cuda, M, N, K, scale_dtype, M + N + K)
    Y, R = torch.empty((M, N), dtype=torch.float32, device=cuda), torch.empty((M, N), dtype=torch.float32, device=cuda)
    ws = torch.full((w4a8.gemm_splitk_workspace_bytes(M, N, K, splitk),), 255, dtype=torch.uint8, device=cuda)   # NaNs: all of it is written
    partial = torch.empty_like(ws)

    def call(stream, Y=Y, ws=ws):
        w4a8.launch_gemm_bm16_splitk(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, splitk, ws, stream)

    call(None)
    w4a8.device_status()
    assert tile_name(launched_kernels(call)) == (fp16 if scale_dtype else fp32)
    fp16_operands(w4a8, lambda stream: call(stream, R, partial))
    assert torch.equal(ws, partial) and torch.equal(Y.view(torch.int32), R.view(torch.int32))      # each range's sums, and theirs
    if M * N < 7000:
        assert np.array_equal(Y.cpu().numpy().view(np.uint32), oracle.gemm_splitk_w4a8(*host, splitk).view(np.uint32))


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("M,N,K,fp32,fp16", CASES)
def test_gemm_long_k(w4a8, oracle, cuda, sms148, M, N, K, fp32, fp16, scale_dtype):  # noqa: F811
    import torch
    host, d = operands(oracle, cuda, M, N, K, scale_dtype, M + N + K)
    Y = torch.full((M + 1, N), 7.0, dtype=torch.float32, device=cuda)            # the last row is a canary
    R = torch.empty((M, N), dtype=torch.float32, device=cuda)

    def call(stream):
        w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, stream)

    call(None)
    w4a8.device_status()
    assert tile_name(launched_kernels(call)) == (fp16 if scale_dtype else fp32)
    fp16_operands(w4a8, lambda stream: w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], R, M, N, K, scale_dtype, stream))
    assert torch.equal(Y[:M].view(torch.int32), R.view(torch.int32)) and bool((Y[M] == 7.0).all())
    if M * N < 5000:
        assert np.array_equal(R.cpu().numpy().view(np.uint32), oracle.gemm_mmq_w4a8(*host).view(np.uint32))
