"""The tile relaxation at its edges: ragged last tiles, wrapped axes whose last
tile is ragged, one tile wide, one or two cells across, a tile's width and one
more; holes, NaN cells, regions without an outlet; long meandering spill paths
that cross tiles many times. Bar: bits against the oracle's fill at slope 0,
and at 1e-3 against its flood with (row, col) heap ties (where the relaxation
only chooses the windows)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rough(nr, nc, seed):
    return (np.random.default_rng(seed).random((nr, nc)) * 50.0).astype(np.float32)


def _maze(nr, nc, seed):
    """Walls with one gap each: the spill path winds through every corridor."""
    rng = np.random.default_rng(seed)
    z = rng.random((nr, nc)).astype(np.float32)
    for k, r in enumerate(range(2, nr - 2, 4)):
        z[r, 1:-1] = 100.0 + k
        z[r, (2 if k % 2 else nc - 3)] = 0.5
    z[0, :] = z[-1, :] = 200.0
    z[:, 0] = z[:, -1] = 200.0
    z[0, 1] = 0.0
    return z


CASES = [(1, 1, "oooo"), (2, 70, "popo"), (70, 2, "opop"), (1, 97, "popo"), (32, 32, "oooo"), (33, 31, "popo"),
         (31, 33, "opop"), (64, 65, "popo"), (65, 64, "opop"), (97, 130, "nnon"), (100, 100, "popo"), (129, 200, "opop")]


@pytest.mark.parametrize("nr,nc,bc", CASES)
@pytest.mark.parametrize("eps", [0.0, 1e-3])
def test_ragged_and_wrapped(port, nr, nc, bc, eps):
    import lsdtt_gb300 as G
    z = _rough(nr, nc, nr * 1000 + nc)
    m = np.ones((nr, nc), np.uint8)
    if nr > 40 and nc > 40:
        m[10:20, 12:30] = 0
    fn = port.fill_pits if eps == 0.0 else port.fill_pits_index_ties
    want = fn(z, m, 10.0, bc, eps)
    got = G.fill_pits(z, m, 10.0, bc, eps).cpu().numpy()
    assert int((got.view(np.uint32) != want.view(np.uint32)).sum()) == 0


@pytest.mark.parametrize("nr,nc", [(99, 67), (200, 300)])
@pytest.mark.parametrize("eps", [0.0, 1e-3])
def test_maze(port, nr, nc, eps):
    import lsdtt_gb300 as G
    z = _maze(nr, nc, nr)
    m = np.ones((nr, nc), np.uint8)
    fn = port.fill_pits if eps == 0.0 else port.fill_pits_index_ties
    want = fn(z, m, 10.0, "oooo", eps)
    got = G.fill_pits(z, m, 10.0, "oooo", eps).cpu().numpy()
    assert int((got.view(np.uint32) != want.view(np.uint32)).sum()) == 0
