"""Decode products of 9 to 16 rows whose activations leave no shared memory beside the rings: bit for bit the oracle's MMQ order, one
launch for all rows, alone, several matrices at once and into peers' arenas."""
import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("S,K", [(16, 9216), (11, 12800), (10, 13824), (9, 15104)])
def test_rows_that_fill_shared_memory(w4a8, oracle, cuda, S, K, scale_dtype):
    import torch
    X = oracle.make_activations(S, K, seed=S + K, outliers=True)
    xq, xs, _ = oracle.quantize_x_q8(X)
    OUTS = (24, 17)
    mats = [oracle.make_weights(n, K, seed=n + S, scale_dtype=scale_dtype) for n in OUTS]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xq_d, xs_d, Wq_d, sw_d = dev(xq), dev(xs), [dev(w) for w, _ in mats], [dev(s) for _, s in mats]
    want = [oracle.gemm_mmq_w4a8(xq, xs, w, s).view(np.uint32) for w, s in mats]
    for i, n in enumerate(OUTS):
        Y = torch.full((S, n), float("nan"), device=cuda)
        call = lambda stream: w4a8.launch_gemv_w4a8_sb(xq_d, xs_d, Wq_d[i], sw_d[i], Y, K, n, S, scale_dtype, stream)
        call(None)
        w4a8.device_status()
        assert len(launched_kernels(call)) == 1
        assert np.array_equal(Y.cpu().numpy().view(np.uint32), want[i])
    Ys = [torch.full((S, n), float("nan"), device=cuda) for n in OUTS]
    w4a8.gemv_multi(xq_d, xs_d, Wq_d, sw_d, Ys, OUTS, K, S, scale_dtype)
    w4a8.device_status()
    for y, r in zip(Ys, want):
        assert np.array_equal(y.cpu().numpy().view(np.uint32), r)
    arena = w4a8.Arena(S * OUTS[0] * 4, 0, 1)
    try:
        arena.connect_pointers([arena.base])
        arena.gemv_allgather(xq_d, xs_d, Wq_d[0], sw_d[0], 0, K, OUTS[0], 0, OUTS[0], S, scale_dtype, 1)
        arena.wait(1, timeout_us=200000)
        w4a8.device_status()
        assert np.array_equal(arena.tensor(0, (S, OUTS[0])).cpu().numpy().view(np.uint32), want[0])
    finally:
        arena.close()
