"""The routing passes at their edges: a sort tile (4096 pairs) less one, whole
and plus one, a scan tile likewise, cells of a warp's first lane masked, one
cell or one row or column, wrapped axes (two cells across too); weighted
accumulation through wide levels, a long tail of narrow ones and a chain with a
cell a level. Bar: bits, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _surface(nr, nc, kind, seed):
    rng = np.random.default_rng(seed)
    z = rng.random((nr, nc)).astype(np.float32)
    if kind == "tilt":  # long slopes: many narrow levels
        z = (z * 0.01 + np.arange(nr)[:, None] * 1.0 + np.arange(nc)[None, :] * 0.3).astype(np.float32)
    elif kind == "ramp":  # a chain: every level one row of cells
        z = np.broadcast_to(np.arange(nr * 1.0)[:, None], (nr, nc)).astype(np.float32).copy()
    return z


CASES = [(1, 1, "oooo", "noise"), (1, 700, "oooo", "tilt"), (3000, 1, "oooo", "ramp"), (2, 2048, "opop", "noise"),
         (2048, 2, "popo", "noise"), (63, 65, "nnon", "noise"), (64, 64, "oooo", "noise"), (17, 241, "popo", "tilt"),
         (128, 96, "oooo", "mask"), (257, 160, "opop", "mask"), (301, 307, "nnon", "noise"), (600, 70, "oooo", "tilt"),
         (1500, 3, "popo", "ramp"), (420, 400, "popo", "tilt"),
         # the largest tour whose rulers one block ranks, and one row of cells more
         (191, 256, "nnon", "noise"), (192, 256, "oooo", "tilt"), (700, 701, "nnon", "tilt"),
         # the largest range-max table that one block builds, and a cell-row more
         (512, 256, "oooo", "noise"), (513, 256, "nnon", "noise"),
         # histograms of the sort scanned by one block (128 tiles), and past it
         (512, 1024, "oooo", "noise"), (513, 1024, "oooo", "noise")]


@pytest.mark.parametrize("nr,nc,bc,kind", CASES)
def test_routes(port, nr, nc, bc, kind):
    import lsdtt_gb300 as G
    z = _surface(nr, nc, kind, nr * 7 + nc)
    m = np.ones((nr, nc), np.uint8)
    if kind == "mask":  # the first lane of every warp's cells, and a hole
        m[:, ::32] = 0
        m[nr // 3:nr // 2, 5:nc // 2] = 0
    w = np.random.default_rng(3).random(nr * nc) * 1e3
    want = port.flowinfo(z, m, 10.0, bc, allow_pits_as_outlets=True, weights=w)
    fi = G.FlowInfo(z, m, 10.0, bc, allow_pits_as_outlets=True)
    for name, got in (("receiver", fi.receiver()), ("donors", fi.donor_count()), ("outlets", fi.outlets()),
                      ("topo", fi.topological_order()), ("s_vector", fi.s_vector()),
                      ("sv_start", fi.s_vector_start())):
        assert np.array_equal(got.cpu().numpy(), want[name]), name
    acc = fi.accumulate(w).cpu().numpy()
    assert np.array_equal(acc.view(np.uint64), np.asarray(want["accum"]).ravel().view(np.uint64))
    fi.close()
