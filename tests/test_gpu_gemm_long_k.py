"""Tiles of the register-resident GEMM that ranges of more than 50 groups take (csrc/gemm_w4a8_mma.cuh, LONG_K), the operands
copied by TMA through many turns of the ring: ragged rows, columns and last K-tiles, the three ways of copying scales.  Bit for bit
against the tcgen05 kernel with fp16 operands, which shares no code with them, and the smallest against the oracle.  Each case names
the tile the dispatch has to choose on 148 SMs."""
import numpy as np
import pytest

from test_gpu_gemm_tiles import operands, sms148, tile_name  # noqa: F401 (sms148 is a fixture)
from conftest import launched_kernels

pytestmark = pytest.mark.gpu

# (M, N, K, tile for fp32 scales, for fp16 scales)
CASES = [(1, 3, 2176, "16/4", "16/4"), (31, 129, 2176, "32/4", "32/4"), (33, 9489, 2176, "48/4", "48/4"), (49, 9528, 2176, "64/4", "64/4"),
         (129, 7620, 2176, "80/4", "80/4"), (241, 9508, 2176, "96/4", "96/4"),
         (6, 1, 2112, "16/4e", "16/4e"), (42, 130, 2112, "32/4e", "32/4e"),
         (33, 9551, 2112, "64/4e", "48/4e"), (65, 9496, 2112, "80/4e", "80/4e"),
         (161, 6282, 2112, "96/4e", "96/4e"), (49, 9473, 2112, "64/4e", "64/4e"),
         (2, 9, 2144, "16/4e", "16/4e"), (55, 131, 2144, "32/4e", "32/4e"),
         (33, 9474, 2144, "64/4e", "48/4e"), (129, 7554, 2144, "80/4e", "80/4e"),
         (241, 9505, 2144, "96/4e", "96/4e"), (162, 9478, 2144, "64/4e", "64/4e")]


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
    w4a8.config("gemm_kernel", 0)
    try:
        w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], R, M, N, K, scale_dtype)
        torch.cuda.synchronize()
    finally:
        w4a8.config("gemm_kernel", 1)
    assert torch.equal(Y[:M].view(torch.int32), R.view(torch.int32)) and bool((Y[M] == 7.0).all())
    if M * N < 5000:
        assert np.array_equal(R.cpu().numpy().view(np.uint32), oracle.gemm_mmq_w4a8(*host).view(np.uint32))
