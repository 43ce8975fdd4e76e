"""Tiles with two CTAs per SM in more than one wave, where the second CTA of an SM starts later than the first: bit for bit against the
kernel with fp16 operands, which shares no code with them.  Each case names the tile the dispatch has to choose on 148 SMs."""
import pytest

from conftest import launched_kernels
from test_gpu_gemm_long_k import fp16_operands
from test_gpu_gemm_tiles import operands, sms148, tile_name  # noqa: F401 (sms148 is a fixture)

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,scale_dtype,kernel", [
    (305, 13609, 128, 0, "64/4"), (305, 13609, 128, 1, "64/4"), (301, 15070, 96, 0, "64/4e"), (301, 15070, 96, 1, "64/4e"),
    (316, 17318, 256, 0, "80/4"), (316, 17318, 256, 1, "80/4"), (348, 14845, 96, 0, "80/4e"), (393, 14099, 96, 1, "80/4e"),
    (365, 18197, 256, 0, "96/4"), (330, 16737, 96, 0, "96/4e")])
def test_more_than_one_wave(w4a8, oracle, cuda, sms148, M, N, K, scale_dtype, kernel):  # noqa: F811
    import torch
    _, d = operands(oracle, cuda, M, N, K, scale_dtype, M + N + K)
    Y = torch.full((M + 1, N), 7.0, dtype=torch.float32, device=cuda)            # the last row is a canary
    R = torch.empty((M, N), dtype=torch.float32, device=cuda)

    def call(stream):
        w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], Y, M, N, K, scale_dtype, stream)

    call(None)
    w4a8.device_status()
    assert tile_name(launched_kernels(call)) == kernel
    fp16_operands(w4a8, lambda stream: w4a8.launch_gemm_mmq_w4a8(d[0], d[1], d[2], d[3], R, M, N, K, scale_dtype, stream))
    assert torch.equal(Y[:M].view(torch.int32), R.view(torch.int32)) and bool((Y[M] == 7.0).all())
