"""Stream power where its level sweep changes form: chains of one-cell levels
longer than a block's offset window, levels at and past the one-block limit,
both together, wrapped edges, holes, an erodibility raster, an incision
threshold, in place; n = 1 (the reciprocal-corrected quotient) over weak to
near-total incision. Bar: the oracle's bits."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _ramp(nr, nc, seed, axis, rough):
    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:nr, 0:nc]
    return ((x if axis else y) * 1.0 + rng.random((nr, nc)) * rough + 5.0).astype(np.float32)


CASES = [("chain_1x3000", 1, 3000, 1, 0.3, "nnno", 0), ("chain_3x2500", 3, 2500, 1, 0.3, "nnno", 0),
         ("wide_3000x40", 3000, 40, 1, 0.0, "nnno", 0), ("limit_1024x64", 1024, 64, 1, 0.0, "nnno", 0),
         ("over_1025x64", 1025, 64, 1, 0.0, "nnno", 0), ("mixed_700x900", 700, 900, 0, 3.0, "onon", 0),
         ("wrap_300x200", 300, 200, 0, 2.0, "opop", 0), ("holes_150x170", 150, 170, 0, 4.0, "oooo", 1)]


@pytest.mark.parametrize("n_exp", [1.0, 1.5, 2.0, 1.3])
@pytest.mark.parametrize("name,nr,nc,axis,rough,bc,holes", CASES, ids=[c[0] for c in CASES])
def test_levels_bitwise(port, name, nr, nc, axis, rough, bc, holes, n_exp):
    import torch
    import lsdtt_gb300 as G
    z = _ramp(nr, nc, nr + nc, axis, rough)
    m = np.ones((nr, nc), np.uint8)
    if holes:
        m[40:60, 30:90] = 0
    fi = G.FlowInfo(z, m, 30.0, bc, allow_pits_as_outlets=True)
    kf = (10.0 ** np.random.default_rng(3).uniform(-7, -1, (nr, nc))).astype(np.float32)
    for K, field, threshold in ((1e-6, None, 0.0), (1e-2, None, 0.0), (10.0, None, 0.0), (1e-4, kf, 0.0),
                                (1e-3, None, 5000.0)):
        want = port.stream_power(z, m, 30.0, bc, K, 0.45, n_exp, 1000.0, threshold, True, 1e-5, field)
        got = G.stream_power_d8(fi, z, K, 0.45, n_exp, 1000.0, threshold, True, 1e-5, field).cpu().numpy()
        differ = int((got.view(np.uint32) != want.view(np.uint32)).sum())
        assert differ == 0, (name, n_exp, K, differ)
    # in place
    zt = torch.from_numpy(z).cuda()
    G._check(G.lib().lsdtt_gpu_stream_power_d8(
        fi._h, ctypes.c_void_p(zt.data_ptr()), ctypes.c_void_p(0), ctypes.c_float(1e-3), ctypes.c_float(0.45),
        ctypes.c_float(n_exp), ctypes.c_float(1000.0), ctypes.c_float(5000.0), ctypes.c_int32(1), ctypes.c_float(1e-5),
        ctypes.c_void_p(zt.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    assert np.array_equal(zt.cpu().numpy().view(np.uint32), want.view(np.uint32))
