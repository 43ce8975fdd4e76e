"""linear of one row in one launch (the GEMV quantizes the row itself): Y, xq, xs and xsum must equal quantize_x followed by the
GEMV of the same row, bit for bit, whichever kernel either of them takes."""
import numpy as np
import pytest
import torch

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


def _case(K, N, sd, seed=0):
    g = torch.Generator(device="cuda").manual_seed(1000 * K + N + sd + seed)
    x = torch.randn((1, K), generator=g, device="cuda") * 3.0
    x[0, 32:64] = 0.0                                                     # a block of zeros
    wq = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, generator=g, device="cuda")
    sw = torch.rand((N, K // 32), generator=g, device="cuda") * 0.01
    return x, wq, (sw.half() if sd else sw)


def _out(K, N):
    return (torch.full((1, K), 77, dtype=torch.int8, device="cuda"), torch.full((1, K // 32), -1.0, device="cuda"),
            torch.full((1, K // 32), -1, dtype=torch.int32, device="cuda"), torch.full((1, N), float("nan"), device="cuda"))


def _bits(t):
    return t.view(torch.int32) if t.dtype == torch.float32 else t


def _check(w4a8, x, wq, sw, sd, x_call=None):
    K, N = wq.shape[1] * 2, wq.shape[0]
    xq, xs, xsum, y = _out(K, N)
    w4a8.launch_quantize_x_q8(x, xq, xs, xsum, K, 1)
    w4a8.linear(None, xq, xs, xsum, wq, sw, y, 1, N, K, sd, 1)           # the two launches
    got = _out(K, N)
    w4a8.linear(x if x_call is None else x_call, got[0], got[1], got[2], wq, sw, got[3], 1, N, K, sd)
    torch.cuda.synchronize()
    w4a8.device_status()
    for a, b in zip((xq, xs, xsum, y), got):
        assert torch.equal(_bits(a), _bits(b))


# rows of 33 .. 544 groups (one to six batches of loads, ragged last lane), fewer rows than SMs, a row count that the CTAs do not
# share evenly, matrices on either side of the line between the two kernels, fp16 scales with and without the tensor path
@pytest.mark.parametrize("K,N,sd", [
    (1056, 1, 0), (1056, 147, 1), (1280, 300, 1), (2048, 2048, 0), (2048, 4500, 1), (2080, 149, 0), (3840, 4096, 0), (5088, 5000, 0),
    (5120, 4096, 0), (5120, 7001, 0), (5120, 1024, 1), (5120, 7001, 1), (5632, 9000, 0), (7680, 1500, 0), (7680, 1500, 1), (8192, 999, 1),
    (15360, 3840, 0), (17408, 513, 0), (17440, 65, 1)])
def test_linear_row_equals_two_launches(w4a8, cuda, K, N, sd):
    _check(w4a8, *_case(K, N, sd), sd)


# Long rows, and fp16 scales where the plain kernel's 32 to 48 warps per SM take fewer rounds than the 24 of the one that quantizes:
# either side of each line; rows of the matrix per SM
@pytest.mark.parametrize("K,per_sm,sd,launches", [
    (19456, 1, 0, 1), (19488, 1, 0, 2), (30720, 1, 0, 2), (19456, 25, 0, 1), (15328, 2, 1, 1), (15392, 2, 1, 2), (17440, 1, 1, 2), (9184, 24, 1, 1),
    (9184, 25, 1, 2), (9184, 33, 1, 1), (9184, 49, 1, 2), (3040, 25, 1, 1), (4000, 25, 1, 2), (2016, 75, 1, 1), (2016, 150, 1, 2)])
def test_linear_row_takes_one_launch_where_that_is_faster(w4a8, cuda, K, per_sm, sd, launches):
    N = per_sm * torch.cuda.get_device_properties(cuda).multi_processor_count
    x, wq, sw = _case(K, N, sd)
    _check(w4a8, x, wq, sw, sd)
    out = _out(K, N)
    assert len(launched_kernels(lambda st: w4a8.linear(x, out[0], out[1], out[2], wq, sw, out[3], 1, N, K, sd, 0, st))) == launches


@pytest.mark.parametrize("policy", [1, 2, 3, 5])
def test_linear_row_under_every_gemv_policy(w4a8, cuda, policy):
    w4a8.config("gemv_kernel", policy)
    try:
        for K, N, sd in ((5120, 700, 0), (5120, 700, 1), (2048, 148, 1)):
            _check(w4a8, *_case(K, N, sd), sd)
    finally:
        w4a8.config("gemv_kernel", 0)


def test_linear_row_unaligned_overlapping_and_host_x(w4a8, cuda):
    x, wq, sw = _case(5120, 700, 0)
    buf = torch.empty(5121, device="cuda")
    buf[1:] = x[0]
    _check(w4a8, x, wq, sw, 0, x_call=buf[1:].view(1, 5120))              # 4-byte aligned only: the general way
    x2, wq2, sw2 = _case(2048, 2048, 0)
    q, inplace = _out(2048, 2048), x2.clone()
    want = _out(2048, 2048)
    w4a8.linear(x2, want[0], want[1], want[2], wq2, sw2, want[3], 1, 2048, 2048)
    w4a8.linear(inplace, q[0], q[1], q[2], wq2, sw2, inplace, 1, 2048, 2048)                # the outputs replace the row
    torch.cuda.synchronize()
    assert torch.equal(_bits(inplace), _bits(want[3])) and torch.equal(q[0], want[0])
    Yh, Xh = torch.empty((1, 700)).pin_memory(), x.cpu().pin_memory()
    xq, xs, xsum, y = _out(5120, 700)
    w4a8.linear_host(Xh, Yh, torch.empty_like(x), xq, xs, xsum, y, wq, sw, 1, 700, 5120)
    want = _out(5120, 700)
    w4a8.linear(x, want[0], want[1], want[2], wq, sw, want[3], 1, 700, 5120)
    torch.cuda.synchronize()
    assert np.array_equal(Yh.numpy().view(np.uint32), want[3].cpu().numpy().view(np.uint32))


def test_linear_row_in_a_graph_and_after_its_own_output(w4a8, cuda):
    """A chain in which every row is the output of the launch before it, captured and replayed."""
    K = 2048
    mats = [_case(K, K, 0, seed=i)[1:] for i in range(3)]
    x0 = _case(K, K, 0)[0]
    bufs = [torch.empty((1, K), device="cuda") for _ in range(3)]
    q = _out(K, K)

    def chain():
        src = x0
        for (wq, sw), y in zip(mats, bufs):
            w4a8.linear(src, q[0], q[1], q[2], wq, sw, y, 1, K, K)
            src = y
    want, src = [], x0
    for wq, sw in mats:
        y = torch.empty((1, K), device="cuda")
        w4a8.launch_quantize_x_q8(src, q[0], q[1], q[2], K, 1)
        torch.cuda.synchronize()
        w4a8.linear(None, q[0], q[1], q[2], wq, sw, y, 1, K, K, 0, 1)
        torch.cuda.synchronize()
        want.append(y)
        src = y
    chain()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        chain()
    for _ in range(20):
        g.replay()
    torch.cuda.synchronize()
    for a, b in zip(want, bufs):
        assert torch.equal(_bits(a), _bits(b))
