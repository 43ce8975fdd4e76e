"""Several matrices against two to sixteen shared rows in one launch: every matrix has the bits of its own call and the oracle's MMQ
order; row counts that end inside a 16-row tile, one tile or many per CTA, both step lengths, with and without the relay."""
import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale_dtype", [0, 1])
@pytest.mark.parametrize("S,K,OUTS", [(2, 512, (1, 17)), (8, 2048, (300, 200)), (8, 2304, (1000, 8, 31, 500)), (3, 256, (5000, 3001)),
                                      (16, 1536, (2000, 2000)), (9, 768, (40, 7)), (16, 2816, (3000, 2500, 100)), (8, 1280, (20000, 9000))])
def test_one_launch(w4a8, oracle, cuda, S, K, OUTS, scale_dtype):
    import torch
    X = oracle.make_activations(S, K, seed=S + K, outliers=True)
    xq, xs, _ = oracle.quantize_x_q8(X)
    mats = [oracle.make_weights(n, K, seed=n + i, scale_dtype=scale_dtype) for i, n in enumerate(OUTS)]
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    xq_d, xs_d, Wq_d, sw_d = dev(xq), dev(xs), [dev(w) for w, _ in mats], [dev(s) for _, s in mats]
    Ys = [torch.full((S + 1, n), float("nan"), dtype=torch.float32, device=cuda) for n in OUTS]     # last row: canary

    def call(stream):
        w4a8.gemv_multi(xq_d, xs_d, Wq_d, sw_d, Ys, OUTS, K, S, scale_dtype, stream)

    call(None)
    w4a8.device_status()
    names = launched_kernels(call)
    assert len(names) == 1 and "gemv_w4a8_mma_kernel" in names[0], names
    for y, n, (Wq, sw), wd, sd in zip(Ys, OUTS, mats, Wq_d, sw_d):
        Y1 = torch.empty((S, n), dtype=torch.float32, device=cuda)
        w4a8.launch_gemv_w4a8_sb(xq_d, xs_d, wd, sd, Y1, K, n, S, scale_dtype)
        y = y.cpu().numpy()
        assert np.all(np.isnan(y[S]))
        assert np.array_equal(y[:S].view(np.uint32), Y1.cpu().numpy().view(np.uint32))
        if n * K <= 6000000:
            assert np.array_equal(y[:S].view(np.uint32), oracle.gemm_mmq_w4a8(xq, xs, Wq, sw).view(np.uint32))
