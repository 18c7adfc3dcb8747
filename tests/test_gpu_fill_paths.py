"""Fills whose spill path crosses the relaxation's tiles many more times than
the grid has rows and columns: one-cell corridors that wind from end to end of
the grid. Bar: bits against the oracle's fill at slope 0, and with a slope
against its flood with (row, col) heap ties."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _serpentine(nr, nc, pitch, seed):
    """A wall every `pitch` rows, its one gap at alternate ends."""
    z = np.random.default_rng(seed).random((nr, nc)).astype(np.float32)
    for k, r in enumerate(range(2, nr - 2, pitch)):
        z[r, 1:-1] = 100.0 + k
        z[r, (1 if k % 2 else nc - 2)] = 0.5
    z[0, :] = z[-1, :] = 1000.0
    z[:, 0] = z[:, -1] = 1000.0
    z[0, 1] = 0.0
    return z


# (the last slope stays below the walls all along the path, the one before
# spills over them)
@pytest.mark.parametrize("n,pitch,eps", [(640, 2, 0.0), (1100, 4, 0.0), (640, 2, 1e-3), (640, 2, 1e-6)])
def test_serpentine(port, n, pitch, eps):
    import lsdtt_gb300 as G
    z = _serpentine(n, n, pitch, n + pitch)
    m = np.ones((n, n), np.uint8)
    fn = port.fill_pits if eps == 0.0 else port.fill_pits_index_ties
    want = fn(z, m, 10.0, "oooo", eps)
    got = G.fill_pits(z, m, 10.0, "oooo", eps).cpu().numpy()
    assert int((got.view(np.uint32) != want.view(np.uint32)).sum()) == 0
