"""Decode products of two rows with fp16 scales and three slots a lane (65 to 96 groups, or a multiple of three slots), either side of
the numbers of weight rows at which the form of the unpacking, and with it the CTAs per SM, changes: the kernel by name, and bit for
bit the documented order."""
import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,K,N,longer", [(2, 2080, 17, 0), (2, 2080, 3 * 148 * 8, 0), (2, 2080, 3 * 148 * 8 + 1, 1), (2, 2912, 4 * 148 * 8, 1),
                                          (2, 2080, 4 * 148 * 8 + 1, 0), (2, 2080, 7200, 1), (2, 5152, 3600, 1), (6, 2080, 3600, 1)])
def test_two_rows(w4a8, oracle, cuda, S, K, N, longer):
    import torch
    X = oracle.make_activations(S, K, seed=N, outliers=True)
    Wq, sw = oracle.make_weights(N, K, seed=K, scale_dtype=1)
    xq, xs, _ = oracle.quantize_x_q8(X)
    d = [torch.from_numpy(np.ascontiguousarray(a)).to(cuda) for a in (xq, xs, Wq, sw)]
    Y = torch.full((S + 1, N), 7.0, dtype=torch.float32, device=cuda)            # the last row is a canary

    def call(stream):
        w4a8.launch_gemv_w4a8_sb(d[0], d[1], d[2], d[3], Y, K, N, S, 1, stream)

    call(None)
    w4a8.device_status()
    y = Y.cpu().numpy()
    assert np.array_equal(y[:S].view(np.uint32), oracle.gemv_b200_order(xq, xs, Wq, sw).view(np.uint32))
    assert np.all(y[S] == 7.0)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert "gemv_w4a8_dp4a_kernelILi2ELi3E6__halfLb0ELi8ELb%dE" % longer in launched_kernels(call)[-1]
