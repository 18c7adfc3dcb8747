"""The hillslope solvers on grids whose strips are 16 rows tall, where they end
ragged: a last strip of one and of nine rows, columns that fill 1 of the last
strip's 30, wrapped axes, holes and channel cells. Bar as for the 8-row
strips: 5e-6 of the relief (the solve's relative residual of 1e-8 and FP32
vectors times a condition number of at most 41 give 3e-6 of the largest
increment, and the result is rounded to FP32)."""
import numpy as np
import pytest

from oracle import hillslope as H

pytestmark = pytest.mark.gpu


def _surface(nr, nc, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:nr, 0:nc]
    return (20.0 * np.sin(x / 17.0) * np.cos(y / 23.0) + rng.random((nr, nc))).astype(np.float32)


def _rows(nr, nc):
    """Rows of a strip: 16 where that leaves at least 4 blocks of 8 strips for each of 152 SMs."""
    strips = -(-nc // 30) * -(-nr // 16)
    return 16 if -(-strips // 8) >= 4 * 152 else 8


@pytest.mark.parametrize("nr,nc,bc", [(3001, 811, "popo"), (2050, 2051, "opop"), (1609, 1471, "nnon")])
def test_linear_step(nr, nc, bc):
    import lsdtt_gb300 as G
    assert _rows(nr, nc) == 16
    z = _surface(nr, nc, nr * 7 + nc)
    m = np.ones((nr, nc), np.uint8)
    chan = np.zeros((nr, nc), np.uint8)
    m[nr // 3:nr // 3 + 5, nc // 4:nc // 4 + 9] = 0
    m[-1, 100:130] = 0
    chan[nr // 2, nc // 2:] = 1
    got, rep = G.hillslope_linear_implicit(z, m, 10.0, bc, 0.05, 10000.0, is_channel=chan)
    want, _, _ = H.linear_step(z, m, 10.0, bc, 0.05, 10000.0, is_channel=chan, solver="pcg", rel_tol=1e-12)
    err = float(np.abs(got.cpu().numpy().astype(np.float64) - want).max())
    print(f"{nr}x{nc} {bc}: {rep.iterations} iterations, max difference {err:.2e}")
    assert err <= 5e-6 * 21.0
    assert rep.relative_residual <= 1e-8


@pytest.mark.parametrize("nr,nc,bc,up,across", [(93, 811, "popo", 33, 1), (811, 93, "opnp", 1, 33),
                                                (61, 97, "pppp", 27, 17)])
def test_roering_step(nr, nc, bc, up, across):
    """A surface that repeats along its wrapped axes, whose step is one period's (which the oracle's sparse
    factorisation can afford)."""
    import lsdtt_gb300 as G
    assert _rows(nr * up, nc * across) == 16
    z = 0.2 * _surface(nr, nc, nr + nc)
    m = np.ones((nr, nc), np.uint8)
    m[nr // 3:nr // 3 + 5, nc // 4:nc // 4 + 9] = 0
    got, rep = G.hillslope_implicit(np.tile(z, (up, across)), np.tile(m, (up, across)), 10.0, bc, 0.01, 1.2, 2000.0)
    want, ok, _, _ = H.newton_step(z, z, m, 10.0, bc, 0.01, 1.2, 1.0 / 2000.0)
    err = float(np.abs(got.cpu().numpy().astype(np.float64) - np.tile(want, (up, across))).max())
    print(f"{nr * up}x{nc * across} {bc}: {rep.iterations} iterations, max difference {err:.2e}")
    assert ok and err <= 5e-6 * 4.2
