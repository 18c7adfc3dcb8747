"""The FP32 sums of the U-Net's gradient, by themselves: a network of whole
weights on a residual of +-1 in 8 x 8 blocks, whose activations BF16 holds
exactly, so that nothing but the backward pass rounds. Against the same
gradient in 64 bits.

Bar: 2^-24 of each tensor's root mean square, one FP32 rounding's largest
error. A sum's result is rounded once (2^-24 / sqrt(12) to 2^-25 on average);
the additions before it are the runs within a thread, whose errors are random
and those of a small part of the sum each, and trees of them with the errors
carried along."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _params(rng, layers):
    """Centre taps only: each output takes two or three inputs with +-1, each input is used."""
    parts = []
    for _, ci, co in layers:
        w = np.zeros((co, 9, ci), np.float32)
        for o in range(co):
            w[o, 4, [o % ci, (7 * o + 3) % ci]] = rng.choice([-1.0, 1.0], 2)
        for i in range(ci):
            w[i % co, 4, i] = rng.choice([-1.0, 1.0])
        parts.append(w.ravel())
    return np.concatenate(parts + [rng.integers(0, 2, co).astype(np.float32) for _, _, co in layers])


def _gradient(layers, params, r, e):
    import torch
    import torch.nn.functional as F
    p = torch.from_numpy(params).cuda().double().requires_grad_(True)
    at, bat, k = 0, sum(9 * ci * co for _, ci, co in layers), []
    for _, ci, co in layers:
        w = p[at:at + 9 * ci * co].view(co, 3, 3, ci).permute(0, 3, 1, 2)
        k.append((w, p[bat:bat + co]))
        at, bat = at + 9 * ci * co, bat + co

    def conv(x, l):
        y = F.conv2d(x, *k[l], padding=1)
        assert torch.equal(y, y.bfloat16().double())  # held exactly
        return y

    def up(x):
        return x.repeat_interleave(2, -1).repeat_interleave(2, -2)

    x = torch.from_numpy(r).cuda().double()[None, None]
    e0 = F.relu(conv(x, 0))
    e1 = F.relu(conv(F.avg_pool2d(e0, 2), 1))
    e2 = F.relu(conv(F.avg_pool2d(e1, 2), 2))
    e3 = F.relu(conv(F.avg_pool2d(e2, 2), 3))
    d2 = F.relu(conv(up(e3), 4)) + e2
    d1 = F.relu(conv(up(d2), 5)) + e1
    d0 = F.relu(conv(up(d1), 6)) + e0
    y = conv(d0, 7)[0, 0]
    t = torch.from_numpy(e).cuda().double()
    (((y - t) ** 2).sum() / (t * t).sum()).backward()
    return p.grad.cpu().numpy()


@pytest.mark.parametrize("shape", [(64, 64), (72, 96), (200, 160), (512, 512), (1024, 1024)])
def test_gradient_sums(shape):
    import lsdtt_gb300 as G
    layers = G.UNET_LAYERS
    rng = np.random.default_rng(shape[0] + shape[1])
    P = _params(rng, layers)
    r = np.kron(rng.choice([-1.0, 1.0], (shape[0] // 8, shape[1] // 8)), np.ones((8, 8))).astype(np.float32)
    e = (3.0 * rng.standard_normal(shape)).astype(np.float32)
    net = G.UNet(*shape)
    net.set_params(P)
    got = net.loss_grad(r, e)[1].astype(np.float64)
    want = _gradient(layers, P, r, e)
    at, errors = 0, {}
    for name, n in [(n, 9 * ci * co) for n, ci, co in layers] + [("biases", sum(co for _, _, co in layers))]:
        d, w = got[at:at + n] - want[at:at + n], want[at:at + n]
        errors[name] = float(np.sqrt((d * d).mean() / (w * w).mean()))
        at += n
    print(shape, {k: f"{v:.1e}" for k, v in errors.items()})
    assert max(errors.values()) < 2.0 ** -24, errors
