"""The fill where values compare equal but differ in their bits, or take no part:
zeros of both signs, NaN cells, regions that no seed reaches.

A cell at or below the value it is reached from takes that value, sign of zero
included: with every seed at one zero, all that lies at or below zero ends up
as that zero. Bar: bits against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _zeros(nr, nc, seed, sign):
    z = np.random.default_rng(seed).choice(np.array([0.0, -0.0, -1.0, -2.5, 3.0], np.float32), (nr, nc),
                                           p=[0.3, 0.3, 0.15, 0.15, 0.1]).astype(np.float32)
    s = np.float32(np.copysign(0.0, sign))
    z[0, :] = z[-1, :] = s
    z[:, 0] = z[:, -1] = s
    return z


@pytest.mark.parametrize("nr,nc,bc", [(20, 20, "oooo"), (33, 65, "oooo"), (100, 97, "oooo"), (64, 130, "popo"),
                                      (131, 64, "opop")])
@pytest.mark.parametrize("sign", [1.0, -1.0])
@pytest.mark.parametrize("eps", [0.0, 1e-3])
def test_zeros_of_both_signs(port, nr, nc, bc, sign, eps):
    import lsdtt_gb300 as G
    z = _zeros(nr, nc, nr + nc, sign)
    m = np.ones((nr, nc), np.uint8)
    fn = port.fill_pits if eps == 0.0 else port.fill_pits_index_ties
    want = fn(z, m, 10.0, bc, eps)
    got = G.fill_pits(z, m, 10.0, bc, eps).cpu().numpy()
    assert int((got.view(np.uint32) != want.view(np.uint32)).sum()) == 0


def test_mixed_zeros_repeat():
    """Seeds at zeros of both signs: which of them a cell takes is settled by the order of the tiles, the same in every
    call and in the fill with fixed scratch."""
    from tests.test_zz_no_alloc import _abi, _run
    G, L = _abi()
    rng = np.random.default_rng(3)
    z = rng.choice(np.array([0.0, -0.0, -1.0, 3.0], np.float32), (400, 333)).astype(np.float32)
    m = np.ones(z.shape, np.uint8)
    status, want = _run(G, L, L.lsdtt_gpu_fill_pits_noalloc, z, m, 10.0, "oooo", 0.0)
    assert status == 0
    want = want.view(np.uint32)
    for _ in range(10):
        got = G.fill_pits(z, m, 10.0, "oooo", 0.0).cpu().numpy().view(np.uint32)
        assert int((got != want).sum()) == 0


def _fixed_point(z, fixed, per_ns, per_ew):
    """F = max(z, lowest neighbour) from +inf, fixed cells at z; NaN cells are no neighbours."""
    F = np.where(fixed, z, np.float32(np.inf))
    while True:
        P = np.pad(np.where(np.isnan(F), np.float32(np.inf), F), 1, constant_values=np.float32(np.inf))
        if per_ns:
            P[0], P[-1] = P[-2], P[1]
        if per_ew:
            P[:, 0], P[:, -1] = P[:, -2], P[:, 1]
        nr, nc = z.shape
        low = np.min([P[1 + a:1 + a + nr, 1 + b:1 + b + nc] for a in (-1, 0, 1) for b in (-1, 0, 1) if a or b], axis=0)
        N = np.where(fixed, F, np.minimum(F, np.maximum(z, low)))
        if np.array_equal(N, F, equal_nan=True):
            return F
        F = N


@pytest.mark.parametrize("nr,nc,bc", [(40, 37, "oooo"), (70, 100, "oooo"), (65, 64, "popo"), (33, 97, "opop")])
def test_nan_cells_and_regions_without_an_outlet(nr, nc, bc):
    """NaN cells stay NaN and nothing spills through them: a region that they
    close off has no outlet and no finite level."""
    import lsdtt_gb300 as G
    rng = np.random.default_rng(nr * nc)
    z = (rng.random((nr, nc)) * 50.0 + 1.0).astype(np.float32)
    z[rng.random((nr, nc)) < 0.02] = np.nan
    r, c = nr // 3, nc // 3
    z[r, c:c + 8] = z[r + 7, c:c + 8] = np.nan
    z[r:r + 8, c] = z[r:r + 8, c + 7] = np.nan
    z[r + 3, c + 3] = 5.0
    per_ns, per_ew = bc[0] == "p", bc[1] == "p"
    y, x = np.mgrid[0:nr, 0:nc]
    seed = (not per_ns) & ((y == 0) | (y == nr - 1)) | (not per_ew) & ((x == 0) | (x == nc - 1))
    want = _fixed_point(z, seed | np.isnan(z), per_ns, per_ew)
    got = G.fill_pits(z, np.ones((nr, nc), np.uint8), 10.0, bc, 0.0).cpu().numpy()
    assert np.isinf(want[r + 3, c + 3]) and np.array_equal(got, want, equal_nan=True)
