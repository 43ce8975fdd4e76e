"""The quantizer's reciprocal path against its division path, bit for bit.

Pointers that are not 16-byte aligned take quantize_x_q8_scalar_kernel, which divides every element; aligned ones take the
vector kernel, which divides only where x / d lies too near a half-integer for the reciprocal to decide.  Both are defined
as q = rintf(x / d), d = amax / 127, so every bit has to agree.  Inputs: quotients on and one ulp beside every half-integer,
scales from subnormal to near overflow, zero blocks, infinities and NaN."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _blocks(kind, rng):
    n = 4096
    x = rng.normal(0, 1, (n, 32)).astype(np.float32)
    if kind == "ties":
        amax = np.exp2(rng.uniform(-20, 20, (n, 1))).astype(np.float32)
        d = amax / np.float32(127)
        x = ((rng.integers(-127, 127, (n, 32)) + np.float32(0.5)) * d).astype(np.float32)
        x = np.where(rng.random((n, 32)) < 0.5, x, np.nextafter(x, np.float32(np.inf) * np.sign(rng.normal(size=(n, 32))).astype(np.float32)))
        x[:, 0] = amax[:, 0]
    elif kind == "range":
        x *= np.exp2(rng.uniform(-149, 126, (n, 1))).astype(np.float32)
        x[::7] = 0.0
        x[3::97, 5] = np.float32(np.finfo(np.float32).max)
    elif kind == "special":
        x[::3, 1] = np.inf
        x[1::3, 2] = np.nan
        x[2::9] = np.nan
        x[5::9, 4] = -np.inf
    return np.ascontiguousarray(x.astype(np.float32))


@pytest.mark.parametrize("kind", ["normal", "ties", "range", "special"])
def test_reciprocal_path_equals_division_path(w4a8, cuda, kind):
    import torch
    rng = np.random.default_rng(11)
    x = _blocks(kind, rng)
    S, K = x.shape[0] // 8, 256
    res = []
    for pad in (0, 1):                                    # 1: everything four bytes off, the division kernel
        xb = torch.zeros(S * K + 4, dtype=torch.float32, device=cuda)
        X = xb[pad:pad + S * K]
        X.copy_(torch.from_numpy(x.reshape(-1)))
        xq = torch.empty(S * K, dtype=torch.int8, device=cuda)
        xs = torch.empty(S * K // 32, dtype=torch.float32, device=cuda)
        xsum = torch.empty(S * K // 32, dtype=torch.int32, device=cuda)
        w4a8.launch_quantize_x_q8(X, xq, xs, xsum, K, S)
        torch.cuda.synchronize()
        res.append((xq.cpu().numpy(), xs.cpu().numpy().view(np.uint32), xsum.cpu().numpy(), np.isnan(xs.cpu().numpy())))
    (q0, s0, m0, n0), (q1, s1, m1, n1) = res
    assert np.array_equal(n0, n1)
    assert np.array_equal(s0[~n0], s1[~n0])
    assert np.array_equal(q0, q1) and np.array_equal(m0, m1)


def test_subnormal_blocks(w4a8, oracle, cuda):
    """Blocks whose scale d = amax / 127 is a few multiples of the smallest subnormal: d is rounded so coarsely that x / d reaches
    190, and both ends have to be clamped to 127 in magnitude as the definition says."""
    import torch
    rng = np.random.default_rng(12)
    step = np.ldexp(1.0, -149)
    amax = rng.integers(64, 2000, (512, 1))                                   # in steps; below 64 d is zero
    amax[:4, 0] = 64, 127, 190, 191
    x = np.rint(rng.uniform(-1, 1, (512, 32)) * amax)
    x[:, 0], x[:, 1] = amax[:, 0], -amax[:, 0]
    x = (x * step).astype(np.float32).reshape(16, 1024)
    xq_o, xs_o, xsum_o = oracle.quantize_x_q8(x)
    assert xq_o.min() == -127
    for pad in (0, 1):
        xb = torch.zeros(x.size + 4, dtype=torch.float32, device=cuda)
        X = xb[pad:pad + x.size]
        X.copy_(torch.from_numpy(x.reshape(-1)))
        xq = torch.empty(x.size, dtype=torch.int8, device=cuda)
        xs = torch.empty(x.size // 32, dtype=torch.float32, device=cuda)
        xsum = torch.empty(x.size // 32, dtype=torch.int32, device=cuda)
        w4a8.launch_quantize_x_q8(X, xq, xs, xsum, 1024, 16)
        torch.cuda.synchronize()
        assert np.array_equal(xq.cpu().numpy(), xq_o.reshape(-1)), pad
        assert np.array_equal(xs.cpu().numpy().view(np.uint32), xs_o.reshape(-1).view(np.uint32))
        assert np.array_equal(xsum.cpu().numpy(), xsum_o.reshape(-1))
