"""The block replay's three forms of a FIFO sweep (short, narrow, wide) where
they can go wrong: generations around and past each form's room, equal
elevations (heap ties by cell index, also across a wrapped edge), axes one to
three cells across, steps of the minimum slope from below a float's spacing to
large. Against the oracle's priority flood with (row, col) heap ties, bit for
bit."""
import numpy as np
import pytest

from tests import surfaces

pytestmark = pytest.mark.gpu


def _bowl(n, depth, noise, seed):
    """A closed depression across the whole grid: its lake's generations are
    rings as wide as the grid's sides."""
    y, x = np.mgrid[0:n, 0:n]
    r = np.hypot(y - n / 2, x - n / 2) / (n / 2)
    z = np.minimum(r, 1.0) ** 2 * depth + np.random.default_rng(seed).random((n, n)) * noise
    return z.astype(np.float32)


def _steps(nr, nc, levels, seed):
    """Whole-number elevations: equal neighbours everywhere."""
    return np.random.default_rng(seed).integers(0, levels, (nr, nc)).astype(np.float32)


CASES = [
    ("bowl_90", lambda: _bowl(90, 20.0, 0.3, 1), "oooo", 10.0, 1e-4),
    ("bowl_300", lambda: _bowl(300, 40.0, 0.3, 2), "oooo", 10.0, 1e-4),
    ("bowl_800_smooth", lambda: _bowl(800, 60.0, 0.0, 3), "nnon", 10.0, 1e-3),
    ("bowl_700_rough", lambda: _bowl(700, 60.0, 30.0, 4), "oooo", 10.0, 1e-4),
    ("ties_200x180", lambda: _steps(200, 180, 5, 5), "oooo", 10.0, 1e-4),
    ("ties_popo", lambda: _steps(64, 97, 4, 6), "popo", 10.0, 1e-3),
    ("ties_opop", lambda: _steps(97, 64, 4, 7), "opop", 10.0, 1e-3),
    ("wrap_3_rows", lambda: _steps(3, 400, 6, 8), "popo", 10.0, 1e-3),
    ("wrap_2_columns", lambda: _steps(300, 2, 6, 9), "opop", 10.0, 1e-3),
    ("wrap_1_column", lambda: _steps(300, 1, 6, 10), "opop", 10.0, 1e-3),
    ("slope_below_spacing", lambda: _bowl(160, 2000.0, 500.0, 11), "oooo", 0.01, 1e-9),
    ("slope_large", lambda: surfaces.fractal_pits(256, seed=12), "oooo", 10.0, 0.5),
]


@pytest.mark.parametrize("name,make,bc,cell,eps", CASES, ids=[c[0] for c in CASES])
def test_sweep_forms_bitwise(port, name, make, bc, cell, eps):
    import lsdtt_gb300 as G
    z = make()
    m = np.ones(z.shape, np.uint8)
    want = port.fill_pits_index_ties(z, m, cell, bc, eps)
    got = G.fill_pits(z, m, cell, bc, eps).cpu().numpy()
    differ = int((got.view(np.uint32) != want.view(np.uint32)).sum())
    print(f"{name}: {int((want != z).sum())} raised cells, {differ} differ")
    assert differ == 0


def test_wide_sweeps_repeat(port):
    """Noise at a slope whose sweeps outgrow the shared-memory forms: every call ends, with the same bits."""
    import lsdtt_gb300 as G
    z = (np.random.default_rng(5).random((160, 147)) + 0.03 * np.arange(159, -1, -1)[:, None]).astype(np.float32)
    m = np.ones(z.shape, np.uint8)
    want = port.fill_pits_index_ties(z, m, 30.0, "oooo", 1e-2).view(np.uint32)
    for _ in range(150):
        got = G.fill_pits(z, m, 30.0, "oooo", 1e-2).cpu().numpy().view(np.uint32)
        assert int((got != want).sum()) == 0
