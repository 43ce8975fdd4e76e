"""linear of one row in one launch (the GEMV quantizes the row itself): Y, xq, xs and xsum must equal quantize_x followed by the
GEMV of the same row, bit for bit, whichever kernel either of them takes."""
import re

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


def _route(call):
    """How a call goes: "dp4a" or "bulk" where that kernel quantizes the row itself, "two" for quantizer and product."""
    names = launched_kernels(call)
    if len(names) == 2 and "quantize_x_q8" in names[0] and "gemv_w4a8" in names[1]:
        return "two"
    assert len(names) == 1, names
    if re.search(r"gemv_w4a8_dp4a_kernelILi1ELi\dE(f|6__half)Lb0ELi24E", names[0]):
        return "dp4a"
    m = re.search(r"gemv_w4a8_bulk_kernelILi(\d)E(f|6__half)Lb0ELb1E", names[0])
    assert m, names
    return "bulk" + m.group(1)


def _check(w4a8, x, wq, sw, sd, x_call=None):
    """Compares the call with the two launches and returns its route."""
    K, N = wq.shape[1] * 2, wq.shape[0]
    xq, xs, xsum, y = _out(K, N)
    w4a8.launch_quantize_x_q8(x, xq, xs, xsum, K, 1)
    w4a8.linear(None, xq, xs, xsum, wq, sw, y, 1, N, K, sd, 1)           # the two launches
    got = _out(K, N)

    def call(stream):
        w4a8.linear(x if x_call is None else x_call, got[0], got[1], got[2], wq, sw, got[3], 1, N, K, sd, 0, stream)

    call(None)
    torch.cuda.synchronize()
    w4a8.device_status()
    for a, b in zip((xq, xs, xsum, y), got):
        assert torch.equal(_bits(a), _bits(b))
    return _route(call)


# rows of 33 .. 544 groups (one to six batches of loads, ragged last lane), fewer rows than SMs, a row count that the CTAs do not
# share evenly; both sides of the lines between the two kernels for each number of groups per lane; fp16 scales with and without the
# tensor path; the largest ring and row that share an SM's memory
@pytest.mark.parametrize("K,N,sd,route", [
    (1024, 300, 0, "two"), (1056, 1, 0, "dp4a"), (1056, 147, 1, "dp4a"), (1280, 300, 1, "two"), (2048, 2048, 0, "dp4a"), (2080, 149, 0, "dp4a"),
    (3840, 4096, 0, "dp4a"), (3840, 45000, 0, "bulk4"), (5088, 5000, 0, "dp4a"), (5120, 4096, 0, "dp4a"), (5120, 7001, 0, "bulk5"),
    (5632, 9000, 0, "dp4a"), (5632, 9600, 0, "bulk6"), (7680, 1500, 0, "dp4a"), (15360, 3840, 0, "dp4a"), (17408, 513, 0, "dp4a"),
    (2048, 4500, 1, "dp4a"), (2048, 4600, 1, "bulk2"), (2304, 4200, 1, "bulk3"), (4096, 2400, 1, "bulk4"), (5120, 1024, 1, "dp4a"),
    (5120, 7001, 1, "bulk5"), (6144, 1600, 1, "bulk6"), (7168, 1400, 1, "bulk7"), (7680, 1500, 1, "bulk8"), (8192, 999, 1, "dp4a"),
    (8192, 1200, 1, "bulk8"), (17440, 65, 1, "two")])
def test_linear_row_equals_two_launches(w4a8, cuda, K, N, sd, route):
    assert _check(w4a8, *_case(K, N, sd), sd) == route


# Long rows, and fp16 scales where the plain kernel's 32 to 48 warps per SM take fewer rounds than the 24 of the one that quantizes:
# either side of each line; rows of the matrix per SM
@pytest.mark.parametrize("K,per_sm,sd,route", [
    (19456, 1, 0, "dp4a"), (19488, 1, 0, "two"), (30720, 1, 0, "two"), (19456, 25, 0, "dp4a"), (15328, 2, 1, "dp4a"), (15392, 2, 1, "two"),
    (17440, 1, 1, "two"), (9184, 24, 1, "dp4a"), (9184, 25, 1, "two"), (9184, 33, 1, "dp4a"), (9184, 49, 1, "two"), (3040, 25, 1, "dp4a"),
    (4000, 25, 1, "two"), (2016, 75, 1, "dp4a"), (2016, 150, 1, "two")])
def test_linear_row_takes_one_launch_where_that_is_faster(w4a8, cuda, K, per_sm, sd, route):
    N = per_sm * torch.cuda.get_device_properties(cuda).multi_processor_count
    assert _check(w4a8, *_case(K, N, sd), sd) == route


@pytest.mark.parametrize("policy", [1, 2, 3, 5])
def test_linear_row_under_every_gemv_policy(w4a8, cuda, policy):
    w4a8.config("gemv_kernel", policy)
    try:
        for K, N, sd, ng in ((5120, 700, 0, 5), (5120, 700, 1, 5), (2048, 148, 1, 2)):
            route = {1: "dp4a", 3: "bulk%d" % ng}.get(policy, "two")
            assert _check(w4a8, *_case(K, N, sd), sd) == route
    finally:
        w4a8.config("gemv_kernel", 0)


def test_linear_row_unaligned_overlapping_and_host_x(w4a8, cuda):
    x, wq, sw = _case(5120, 700, 0)
    buf = torch.empty(5121, device="cuda")
    buf[1:] = x[0]
    assert _check(w4a8, x, wq, sw, 0, x_call=buf[1:].view(1, 5120)) == "two"        # 4-byte aligned only
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


@pytest.mark.parametrize("pair", [("x", "y"), ("x", "xq"), ("x", "xs"), ("x", "xsum"), ("y", "xq"), ("y", "xs"), ("y", "xsum")])
def test_linear_row_keeps_two_launches_where_buffers_overlap(w4a8, cuda, pair):
    """The call is captured, not run: what overlapping buffers hold afterwards is the caller's business, how they are used is not."""
    K, N = 5120, 700
    _, wq, sw = _case(K, N, 0)
    size = {"x": K * 4, "xq": K, "xs": K // 8, "xsum": K // 8, "y": N * 4}
    for shared, route in ((16, "two"), (0, "dp4a")):                       # the last 16 bytes of the first are the second's; side by side
        arena = torch.zeros(1 << 17, dtype=torch.uint8, device="cuda")
        at, pos = {}, 1 << 15
        at[pair[0]], at[pair[1]] = 0, size[pair[0]] - shared
        for n in size:
            if n not in at:
                at[n], pos = pos, pos + (1 << 15)
        p = {n: arena.data_ptr() + o for n, o in at.items()}
        assert _route(lambda st: w4a8.linear(p["x"], p["xq"], p["xs"], p["xsum"], wq, sw, p["y"], 1, N, K, 0, 0, st)) == route


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
