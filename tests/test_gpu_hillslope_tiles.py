"""The tiled linear and Roering solvers at their tiles' edges: one row or
column, a tile and one cell more, rows that end inside a tile, both tile
heights, wrapped axes, holes and channel cells; element counts that are not a
multiple of four.

Bar: the solves stop at a relative residual of 1e-8 with FP32 vectors, so an
increment is right to about (1e-8 + 2^-24) times the operator's condition
number (at most 1 + 8 D dt / dx^2 = 41 here): 3e-6 of the largest increment;
the result is then rounded to FP32. 1e-5 of the surface's largest magnitude is
the repository's bar for a step and is held here with the tighter of the two
stated below (5e-6 of the relief)."""
import numpy as np
import pytest

from oracle import hillslope as H

pytestmark = pytest.mark.gpu


def _surface(nr, nc, seed):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:nr, 0:nc]
    return (20.0 * np.sin(x / 17.0) * np.cos(y / 23.0) + rng.random((nr, nc))).astype(np.float32)


@pytest.mark.parametrize("nr,nc,bc,holes", [(1, 1, "nnnn", 0), (1, 300, "nono", 0), (300, 1, "onon", 0),
                                            (8, 128, "nnon", 0), (9, 129, "oooo", 0), (33, 131, "nnnn", 1),
                                            (65, 257, "popo", 0), (64, 250, "opop", 1), (3, 3, "oooo", 0),
                                            (2435, 513, "nnon", 1)])
def test_linear_step(nr, nc, bc, holes):
    import lsdtt_gb300 as G
    z = _surface(nr, nc, nr * 7 + nc)
    m = np.ones((nr, nc), np.uint8)
    chan = np.zeros((nr, nc), np.uint8)
    if holes:
        m[nr // 3:nr // 3 + 5, nc // 4:nc // 4 + 9] = 0
        chan[nr // 2, nc // 2:] = 1
    got, rep = G.hillslope_linear_implicit(z, m, 10.0, bc, 0.05, 10000.0, is_channel=chan)
    want, _, _ = H.linear_step(z, m, 10.0, bc, 0.05, 10000.0, is_channel=chan, solver="pcg", rel_tol=1e-12)
    err = float(np.abs(got.cpu().numpy().astype(np.float64) - want).max())
    print(f"{nr}x{nc} {bc}: {rep.iterations} iterations, max difference {err:.2e}")
    assert err <= 5e-6 * 21.0
    assert rep.relative_residual <= 1e-8


@pytest.mark.parametrize("nr,nc,bc", [(9, 129, "oooo"), (40, 131, "nnon"), (61, 257, "popo")])
def test_roering_step(nr, nc, bc):
    import lsdtt_gb300 as G
    z = 0.2 * _surface(nr, nc, nr + nc)
    m = np.ones((nr, nc), np.uint8)
    got, rep = G.hillslope_implicit(z, m, 10.0, bc, 0.01, 1.2, 2000.0)
    want, ok, _, _ = H.newton_step(z, z, m, 10.0, bc, 0.01, 1.2, 1.0 / 2000.0)
    err = float(np.abs(got.cpu().numpy().astype(np.float64) - want).max())
    print(f"{nr}x{nc} {bc}: {rep.iterations} iterations, max difference {err:.2e}")
    assert ok and err <= 5e-6 * 4.2
