"""A call that CUDA refuses reports its error once: the next call, which nothing is wrong with, succeeds."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", ["quantize", "rmsnorm", "glu", "gemv", "gemm"])
def test_refused_launch_leaves_no_error_behind(w4a8, cuda, name):
    """The launch is refused on a stream whose capture another call has invalidated; nothing reaches the GPU."""
    import torch
    from cuda.bindings import driver as D
    K, N = 256, 64
    S = 32 if name == "gemm" else 2
    x = torch.ones((S, K), device=cuda)
    w = torch.ones(K, device=cuda)
    xq = torch.zeros((S, K), dtype=torch.int8, device=cuda)
    xs = torch.zeros((S, K // 32), device=cuda)
    xsum = torch.zeros((S, K // 32), dtype=torch.int32, device=cuda)
    wq = torch.zeros((N, K // 2), dtype=torch.uint8, device=cuda)
    sw = torch.zeros((N, K // 32), device=cuda)
    y = torch.zeros((S, N), device=cuda)

    def call(stream):
        if name == "quantize":
            w4a8.launch_quantize_x_q8(x, xq, xs, xsum, K, S, stream)
        elif name == "rmsnorm":
            w4a8.launch_rmsnorm_quantize_x_q8(x, w, 1e-6, 0, None, xq, xs, xsum, K, S, stream)
        elif name == "glu":
            w4a8.launch_glu_quantize_x_q8(x, x, 0, None, xq, xs, xsum, K, S, stream)
        elif name == "gemv":
            w4a8.launch_gemv_w4a8_sb(xq, xs, wq, sw, y, K, N, S, 0, stream)
        else:
            w4a8.launch_gemm_mmq_w4a8(xq, xs, wq, sw, y, S, N, K, 0, stream)

    call(None)
    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    assert D.cuStreamBeginCapture(s.cuda_stream, D.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL)[0] == D.CUresult.CUDA_SUCCESS
    assert D.cuStreamSynchronize(s.cuda_stream)[0] != D.CUresult.CUDA_SUCCESS          # not allowed in a capture: invalidates it
    with pytest.raises(w4a8.W4A8Error):
        call(s.cuda_stream)
    assert D.cuStreamEndCapture(s.cuda_stream)[0] == D.CUresult.CUDA_ERROR_STREAM_CAPTURE_INVALIDATED
    call(None)
    torch.cuda.synchronize()
