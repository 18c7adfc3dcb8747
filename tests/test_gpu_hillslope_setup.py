"""The linear hillslope solve's set-up: its residual and norms are FP64.

A surface times a power of two takes the same solve (every rounding scales with
it) as long as no number leaves its range. At 2^46 the squares of the residual
are above FP32's range and everything else is within it; the largest residual
is bit for bit what the expression gives in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solve(z, D, dt):
    import lsdtt_gb300 as G
    out, rep = G.hillslope_linear_implicit(z, np.ones(z.shape, np.uint8), 1.0, "nnon", D, dt)
    return out.cpu().numpy(), rep


@pytest.mark.parametrize("nr,nc", [(70, 91), (33, 260)])
@pytest.mark.parametrize("k", [20, 46, -40])
def test_scaled_surface(nr, nc, k):
    z = (np.random.default_rng(nr).random((nr, nc)) * 20.0).astype(np.float32)
    want, r0 = _solve(z, 1e4, 1e-3)
    got, r1 = _solve(np.ldexp(z, k).astype(np.float32), 1e4, 1e-3)
    assert r0.iterations == r1.iterations > 0
    assert r1.initial_residual_inf == np.ldexp(r0.initial_residual_inf, k)
    assert np.array_equal(np.ldexp(want, k), got)


@pytest.mark.parametrize("seed", range(6))
def test_largest_residual(seed):
    rng = np.random.default_rng(seed)
    z = rng.random((40, 50)).astype(np.float32)
    r, c = rng.integers(2, 38), rng.integers(2, 48)
    z[r, c] = 1000.0 + 10.0 * rng.random()
    D = np.float32(rng.uniform(0.01, 0.5))
    _, rep = _solve(z, float(D), 10.0)
    zd = z.astype(np.float64)
    flux = 0.0
    for a, b in ((-1, 0), (0, 1), (1, 0), (0, -1)):
        flux += zd[r + a, c + b] - zd[r, c]
    assert rep.initial_residual_inf == abs(-np.float64(D) * flux)
