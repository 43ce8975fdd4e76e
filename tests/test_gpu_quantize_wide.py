"""The quantizer with eight elements a thread (X aligned to 32 bytes) against the oracle at sizes that do not fill a warp or a CTA, and
against the kernel for X aligned to 16 bytes with what is not finite, subnormal or on a tie: the same bits."""
import numpy as np
import pytest

from conftest import launched_kernels

pytestmark = pytest.mark.gpu


def _run(w4a8, cuda, X, shift):
    import torch
    S, K = X.shape
    flat = torch.zeros(X.size + 8, dtype=torch.float32, device=cuda)
    flat[shift:shift + X.size] = torch.from_numpy(X.reshape(-1)).to(cuda)
    xq = torch.full((S + 1, K), 77, dtype=torch.int8, device=cuda)
    xs = torch.full((S + 1, K // 32), 7.0, dtype=torch.float32, device=cuda)
    xsum = torch.full((S + 1, K // 32), 7, dtype=torch.int32, device=cuda)

    def call(stream):
        w4a8.launch_quantize_x_q8(flat[shift:], xq, xs, xsum, K, S, stream)

    call(None)
    torch.cuda.synchronize()
    assert [("wide_kernel" in n, "vec_kernel" in n) for n in launched_kernels(call)] == [(shift == 0, shift != 0)]
    assert bool((xq[S] == 77).all()) and bool((xs[S] == 7.0).all()) and bool((xsum[S] == 7).all())
    return xq[:S].cpu().numpy(), xs[:S].cpu().numpy().view(np.uint32), xsum[:S].cpu().numpy()


@pytest.mark.parametrize("S,K", [(1, 32), (1, 96), (3, 160), (1, 2048), (7, 2080), (33, 1056), (129, 5120), (1200, 4128)])
def test_sizes(w4a8, oracle, cuda, S, K):
    X = oracle.make_activations(S, K, seed=S + K, outliers=True)
    X[0, :32] = 0.0
    for got in (_run(w4a8, cuda, X, 0), _run(w4a8, cuda, X, 4)):
        for g, want in zip(got, oracle.quantize_x_q8(X)):
            assert np.array_equal(g, want.view(g.dtype))


def test_values_that_are_not_ordinary(w4a8, oracle, cuda):
    rng = np.random.default_rng(5)
    X = rng.standard_normal((64, 640)).astype(np.float32)
    X[1:8] = np.rint(X[1:8] * 40) * 0.5                                   # ties
    X[1:8, ::32] = 127.0
    X[9:16] *= np.float32(1e-38)                                          # subnormal scales
    X[17:24] *= np.float32(1e33)
    X[25, ::5], X[26, ::7], X[27, 3::11] = np.nan, np.inf, -np.inf
    X[28, :64], X[29, ::2] = np.nan, np.float32(-0.0)
    for a, b in zip(_run(w4a8, cuda, X, 0), _run(w4a8, cuda, X, 4)):
        assert np.array_equal(a, b)
