"""The U-Net's gradient kernels at the sizes where their tiles, splits and
copies can go wrong: a single position on the coarsest level, fewer positions
than splits, ragged last tiles, rows that tiles straddle.

Bar: the gradient is an FP32 sum of at most 2^16 products (error at most
2^16 * 2^-24 = 4e-3 of the sum of magnitudes, in practice its square root's
2^8 * 2^-24 = 2e-5) behind a BF16 forward pass whose roundings can flip
against the oracle's: 1e-3 relative L2 a tensor, the bar of the gradient
test in test_gpu_unet.py."""
import numpy as np
import pytest

from oracle import unet
from tests.test_gpu_unet import _params, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,cap", [((8, 8), (8, 8)), ((8, 136), (64, 256)), ((24, 40), (24, 40)),
                                       ((136, 72), (136, 72)), ((200, 328), (256, 328))])
def test_gradients_match_oracle_at_tile_edges(shape, cap):
    import lsdtt_gb300 as G
    P = _params()
    rng = np.random.default_rng(shape[0] * 1000 + shape[1])
    r = rng.normal(0, 1, shape).astype(np.float32)
    e = rng.normal(0, 1, shape).astype(np.float32)
    net = G.UNet(*cap)
    net.set_params(G.unet_flatten(P))
    loss, g = net.loss_grad(r, e)
    L, want, _ = unet.loss_and_grads(P, r, e)
    assert abs(loss - L) <= 1e-2 * abs(L)
    got = G.unet_unflatten(g)
    errors = {n + k: _rel(got[n + k], want[n + k]) for n, _, _ in G.UNET_LAYERS for k in (".w", ".b")}
    print(shape, {k: f"{v:.1e}" for k, v in errors.items()})
    assert max(errors.values()) < 1e-3, errors
    assert np.array_equal(g, net.loss_grad(r, e)[1])  # the same bits on every run
