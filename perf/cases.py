"""The work that a user of lsdtt_gb300 has it do, as timed cases.

Each case is one call (or one timestep) through the package's public Python
surface on inputs that are made from a seed alone: the epsilon fill, the D8
engine, stream power, the two implicit hillslope steps, the landscape
timestep, the batched ensemble and the learned preconditioner's network, from
the smallest grids, where a call is launches and latency, to the largest that
a pass of a second or two allows. Sizes and parameters come from the
repository's benchmark configurations and tests, with odd and ragged sides
beside the round ones.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import lsdtt_gb300 as G

# Multiply-adds of the U-Net's eight 3x3 convolutions per full-resolution
# pixel: 9 Cin Cout, over the level's area.
UNET_MACS = (9 * 16 + 9 * 16 * 32 / 4 + 9 * 32 * 64 / 16 + 9 * 64 * 64 / 64 + 9 * 64 * 64 / 16 + 9 * 64 * 32 / 4 +
             9 * 32 * 16 + 9 * 16)


def listed():
    return [
        # a field plot or a test tile: the call is launches and latency
        dict(name="fill_tile", kind="fill", surface="noise", rows=97, cols=131, bc="nnon", slope=1e-4, holes=0),
        # a DEM tile filled before routing: fractal relief with closed pits
        dict(name="fill_dem", kind="fill", surface="fractal", rows=1500, cols=1403, bc="oooo", slope=1e-4, holes=0),
        # spill levels only (no imposed gradient), a large grid that wraps east-west
        dict(name="fill_spill", kind="fill", surface="fractal", rows=4099, cols=4000, bc="opop", slope=0.0, holes=0),
        # routing a small catchment and summing a rainfall raster down it
        dict(name="route_catchment", kind="route", rows=129, cols=203, bc="nnon", weights=True),
        # routing a large DEM: receivers, topological order, s-vector, counts, drainage area
        dict(name="route_dem", kind="route", rows=4096, cols=4003, bc="oooo", weights=False),
        # one implicit incision step over an existing flow graph
        dict(name="stream_power", kind="incise", rows=2048, cols=2048, bc="nnon", n=1.5),
        # linear hillslope diffusion over a long step (D dt / dx^2 = 10)
        dict(name="diffuse_linear", kind="diffuse", rows=2048, cols=2051, bc="nnon", number=10.0),
        # the critical-slope law on a steep surface, same diffusion number
        dict(name="diffuse_roering", kind="roering", rows=1024, cols=1000, bc="oooo", number=10.0, steep=0.8),
        # one step of a single landscape-evolution run, some way into it
        dict(name="timestep", kind="timestep", rows=512, cols=512, bc="nnon", n=1.0),
        # one step of a 256-run parameter sweep, grids of uneven sides
        dict(name="ensemble", kind="ensemble", members=256, low=128, high=1024, shapes=4),
        # one application of the learned preconditioner
        dict(name="unet_apply", kind="unet_apply", rows=2048, cols=2048),
        # one gradient of its training, on the training surfaces' size
        dict(name="unet_train", kind="unet_train", rows=512, cols=512),
    ]


def draw(rng: random.Random):
    def side(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    def sides(low, high, of=1):
        a = side(low, high)
        b = min(high, max(low, int(a * math.exp(rng.uniform(-0.5, 0.5)))))
        return max(of, a // of * of), max(of, b // of * of)

    kind = rng.choice(["fill", "fill", "spill", "route", "route", "incise", "diffuse", "roering", "timestep",
                       "ensemble", "unet_apply", "unet_train"])
    if kind == "fill":
        r, c = sides(64, 1400)
        surface = rng.choice(["noise", "fractal"])
        return dict(kind="fill", surface=surface, rows=r, cols=c,
                    bc=rng.choice(["nnon", "oooo", "popo", "opop"] if surface == "fractal" else ["nnon", "oooo"]),
                    slope=rng.choice([1e-4, 1e-4, 1e-3, 1e-2]), holes=rng.choice([0, 0, 3]))
    if kind == "spill":
        r, c = sides(64, 4096)
        return dict(kind="fill", surface="fractal", rows=r, cols=c, bc=rng.choice(["oooo", "popo", "opop"]), slope=0.0,
                    holes=rng.choice([0, 0, 3]))
    if kind == "route":
        r, c = sides(64, 4096)
        return dict(kind="route", rows=r, cols=c, bc=rng.choice(["nnon", "oooo", "opop"]),
                    weights=rng.random() < 0.3 and r * c < 1 << 20)
    if kind == "incise":
        r, c = sides(64, 2048)
        return dict(kind="incise", rows=r, cols=c, bc=rng.choice(["nnon", "oooo"]), n=rng.choice([1.0, 1.5, 2.0]))
    if kind == "diffuse":
        r, c = sides(64, 2048)
        return dict(kind="diffuse", rows=r, cols=c, bc=rng.choice(["nnon", "oooo"]),
                    number=round(math.exp(rng.uniform(math.log(0.05), math.log(20.0))), 3))
    if kind == "roering":
        r, c = sides(64, 1000)
        return dict(kind="roering", rows=r, cols=c, bc=rng.choice(["nnon", "oooo"]),
                    number=round(math.exp(rng.uniform(math.log(0.1), math.log(10.0))), 3),
                    steep=round(rng.uniform(0.3, 0.8), 2))
    if kind == "timestep":
        r, c = sides(64, 700)
        return dict(kind="timestep", rows=r, cols=c, bc="nnon", n=rng.choice([1.0, 1.5, 2.0]))
    if kind == "ensemble":
        return dict(kind="ensemble", members=side(2, 200), low=64, high=side(128, 512), shapes=rng.randrange(1000))
    r, c = sides(64, 2048 if kind == "unet_apply" else 512, 8)
    return dict(kind=kind, rows=r, cols=c)


# ---- inputs -----------------------------------------------------------------
def _gen(seed, salt=0):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + salt)


def _uniform(shape, g):
    return torch.rand(shape, generator=g, device="cuda", dtype=torch.float64)


def _fractal(rows, cols, g, beta):
    """Spectral synthesis, power spectrum ~ k^-beta, scaled to 0..1."""
    ky = torch.fft.fftfreq(rows, device="cuda", dtype=torch.float64)[:, None]
    kx = torch.fft.rfftfreq(cols, device="cuda", dtype=torch.float64)[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = 1.0
    amp = k ** (-beta / 2.0)
    amp[0, 0] = 0.0
    phase = 2.0 * math.pi * _uniform(amp.shape, g)
    z = torch.fft.irfft2(torch.polar(amp, phase), s=(rows, cols))
    return (z - z.min()) / (z.max() - z.min())


def _pitted(rows, cols, g):
    """A k^-2 fractal of 1000 m relief on 10 m cells (in proportion on a
    smaller grid) with paraboloid pits, 100,000 of them on 8192 x 8192."""
    z = _fractal(rows, cols, g, 2.0) * (1000.0 * max(rows, cols) / 8192.0)
    n = max(4, round(1e5 * rows * cols / 8192.0 ** 2))
    cy = (_uniform((n,), g) * rows).long().clamp_(max=rows - 1)
    cx = (_uniform((n,), g) * cols).long().clamp_(max=cols - 1)
    radius = 1.0 + 3.0 * _uniform((n,), g)
    depth = 5.0 * _uniform((n,), g)
    cut = torch.zeros(rows * cols, device="cuda", dtype=torch.float64)
    for dy in range(-4, 5):
        for dx in range(-4, 5):
            w = (1.0 - (dy * dy + dx * dx) / (radius * radius)).clamp_(min=0.0) * depth
            y, x = cy + dy, cx + dx
            inside = (y >= 0) & (y < rows) & (x >= 0) & (x < cols)
            # a maximum does not depend on the order of the pits
            cut.scatter_reduce_(0, (y * cols + x)[inside], w[inside], "amax")
    return (z - cut.view(rows, cols)).float()


def _noise_tilt(rows, cols, bc, g):
    """Uniform noise 0-1 m and a 0.001 tilt to the open edges (30 m cells)."""
    y = torch.arange(rows, device="cuda", dtype=torch.float64)[:, None]
    x = torch.arange(cols, device="cuda", dtype=torch.float64)[None, :]
    away = torch.full((rows, cols), float(rows + cols), device="cuda", dtype=torch.float64)
    for edge, d in zip(bc, (y + 0 * x, cols - 1 - x + 0 * y, rows - 1 - y + 0 * x, x + 0 * y)):
        if edge == "o":
            away = torch.minimum(away, d)
    return (_uniform((rows, cols), g) + 0.03 * away).float()


def _valley(rows, cols, g):
    """A smooth fractal on a regional slope to the south: long rivers, and the
    few pits that the landscape timestep takes as outlets."""
    y = torch.arange(rows, device="cuda", dtype=torch.float64)[:, None]
    return (_fractal(rows, cols, g, 3.2) * (0.6 * rows) + 0.9 * (rows - 1 - y)).float()


def _hills(rows, cols, cell, steepest, g):
    """A k^-3 fractal whose steepest slope is `steepest`."""
    z = _fractal(rows, cols, g, 3.0)
    gx, gy = torch.diff(z, dim=1) / cell, torch.diff(z, dim=0) / cell
    cx, cy = (z[1:-1, 2:] - z[1:-1, :-2]) / (2 * cell), (z[2:, 1:-1] - z[:-2, 1:-1]) / (2 * cell)
    top = max(float(gx.abs().max()), float(gy.abs().max()), float(torch.sqrt(cx * cx + cy * cy).max()))
    return (z * (steepest / top)).float()


def _mask(rows, cols, holes, g):
    m = torch.ones((rows, cols), device="cuda", dtype=torch.uint8)
    at = _uniform((max(1, holes), 2), g).cpu().numpy()
    for k in range(holes):  # lakes of nodata inside the grid
        r, c = int(at[k, 0] * rows * 0.8), int(at[k, 1] * cols * 0.8)
        m[r + 2:r + 2 + max(1, rows // 12), c + 2:c + 2 + max(1, cols // 9)] = 0
    return m


def _unet_params(seed):
    """He-style weights, as a network early in its training has them."""
    g = torch.Generator().manual_seed(7 + int(seed))
    parts = []
    for name, ci, co in G.UNET_LAYERS:
        std = math.sqrt(2.0 / (9 * ci)) if name != "out" else 0.1 * math.sqrt(1.0 / (9 * ci))
        parts.append(torch.randn(co * 9 * ci, generator=g) * std)
    for _, _, co in G.UNET_LAYERS:
        parts.append(0.02 * torch.randn(co, generator=g))
    return torch.cat(parts).numpy()


def _residual_pair(rows, cols, g):
    """A residual of a diffusion solve (rough, stronger in places) and the
    smooth correction that goes with it, metres."""
    r = torch.randn((rows, cols), generator=g, device="cuda") * (0.02 + 0.2 * _fractal(rows, cols, g, 3.0).float())
    e = r[None, None]
    for _ in range(3):
        e = torch.nn.functional.avg_pool2d(e, 5, 1, 2, count_include_pad=False)
    return r.contiguous(), (4.0 * e[0, 0]).contiguous()


def _ensemble_shapes(case):
    r = random.Random(case["shapes"])
    return [(r.randint(case["low"], case["high"]), r.randint(case["low"], case["high"])) for _ in range(case["members"])]


# Parameters that the cases share: the benchmark configurations' values.
HILL = dict(D=0.01, cell=5.0, Sc=1.0)
LEM = dict(timestep=1000.0, erodibility=1e-5, m_exponent=0.5, uplift_rate=1e-3, hillslope_diffusivity=0.01,
           fill_min_slope=1e-4)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "ensemble":
        rng = np.random.default_rng(int(seed))
        specs = []
        for nr, nc in _ensemble_shapes(case):
            z = rng.random((nr, nc), dtype=np.float32)
            z += (0.03 * np.arange(nr - 1, -1, -1, dtype=np.float32))[:, None]
            specs.append(dict(z=z, cell_size=30.0, boundary_conditions="nnon", timestep=1000.0,
                              erodibility=float(10.0 ** rng.uniform(-6.0, -4.0)),
                              m_exponent=float(rng.uniform(0.35, 0.6)), n_exponent=float(rng.choice([1.0, 1.5, 2.0])),
                              hillslope_diffusivity=float(10.0 ** rng.uniform(-3.0, -1.0)),
                              uplift_rate=float(10.0 ** rng.uniform(-4.0, -2.0)), fill_min_slope=1e-4))
        return dict(case=case, ensemble=G.Ensemble(specs))
    rows, cols = case["rows"], case["cols"]
    g = _gen(seed)
    if kind == "fill":
        z = _pitted(rows, cols, g) if case["surface"] == "fractal" else _noise_tilt(rows, cols, case["bc"], g)
        return dict(case=case, z=z, mask=_mask(rows, cols, case["holes"], g),
                    cell=10.0 if case["surface"] == "fractal" else 30.0)
    if kind == "route":
        z, mask = _valley(rows, cols, g), _mask(rows, cols, 0, g)
        rain = 0.5 + _uniform((rows, cols), g) if case["weights"] else None
        flow = G.FlowInfo(z, mask, 10.0, case["bc"], allow_pits_as_outlets=True)
        return dict(case=case, z=z, mask=mask, rain=rain, flow=flow)
    if kind == "incise":
        z, mask = _valley(rows, cols, g), _mask(rows, cols, 0, g)
        return dict(case=case, z=z, flow=G.FlowInfo(z, mask, 30.0, case["bc"], allow_pits_as_outlets=True))
    if kind in ("diffuse", "roering"):
        return dict(case=case, mask=_mask(rows, cols, 0, g),
                    z=_hills(rows, cols, HILL["cell"], case.get("steep", 1.0) * HILL["Sc"], g),
                    dt=case["number"] * HILL["cell"] ** 2 / HILL["D"])
    if kind == "timestep":
        # a filled surface with fresh small pits: what a step meets after the
        # first (the fill's result does not depend on how it is computed)
        mask = _mask(rows, cols, 0, g)
        z = G.fill_pits(_noise_tilt(rows, cols, case["bc"], g), mask, 30.0, case["bc"], 1e-4)
        cut = (_uniform((rows, cols), g) < 0.05) * (0.01 * _uniform((rows, cols), g))
        z = z - cut.float()
        model = G.LandscapeModel(z, mask, 30.0, case["bc"], n_exponent=case["n"], **LEM)
        return dict(case=case, z=z, model=model)
    r, e = _residual_pair(rows, cols, g)
    net = G.UNet(rows, cols)
    net.set_params(_unet_params(seed))
    return dict(case=case, r=r, e=e, net=net)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "fill":
        return G.fill_pits(state["z"], state["mask"], state["cell"], case["bc"], case["slope"])
    if kind == "route":
        f = state["flow"].build(state["z"], state["mask"])
        out = dict(receiver=f.receiver(), order=f.topological_order(), stack=f.s_vector(), start=f.s_vector_start(),
                   count=f.s_vector_size(), donors=f.donor_count(), area=f.accumulate(state["rain"]))
        for t in out.values():
            t.engine = f  # the rasters are the engine's own: it lives as long as they do
        return out
    if kind == "incise":
        return G.stream_power_d8(state["flow"], state["z"], 2e-5, 0.45, case["n"], 500.0)
    if kind == "diffuse":
        return G.hillslope_linear_implicit(state["z"], state["mask"], HILL["cell"], case["bc"], HILL["D"],
                                           state["dt"])[0]
    if kind == "roering":
        return G.hillslope_implicit(state["z"], state["mask"], HILL["cell"], case["bc"], HILL["D"], HILL["Sc"],
                                    state["dt"])[0]
    if kind == "timestep":
        # every pass is the same step: the run's surface is put back first
        state["model"].z.copy_(state["z"])
        state["model"].step()
        return state["model"].z
    if kind == "ensemble":
        # the sweep goes on from pass to pass, and every run's surface is read
        ens = state["ensemble"]
        ens.step()
        return torch.cat([ens.get(k).view(-1) for k in range(ens.n_members)])
    if kind == "unet_apply":
        return state["net"].apply(state["r"])
    loss, grad = state["net"].loss_grad(state["r"], state["e"])
    return dict(loss=loss, grad=grad)


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        n = sum(r * c for r, c in _ensemble_shapes(case))
        return {"bytes": 8 * n, "flops": 0}  # surfaces in and out
    n = case["rows"] * case["cols"]
    if kind == "fill":
        return {"bytes": 9 * n, "flops": 0}  # elevation, mask in; surface out
    if kind == "route":
        # elevation, mask (and weights) in; five 8-byte rasters, donors, area out
        return {"bytes": (4 + 1 + (8 if case["weights"] else 0) + 4 * 8 + 8 + 1 + 8) * n, "flops": 0}
    if kind == "incise":
        return {"bytes": (4 + 8 + 1 + 8 + 4) * n, "flops": 0}  # elevation, receiver, direction, count in; surface out
    if kind in ("diffuse", "roering", "timestep"):
        return {"bytes": 9 * n, "flops": 0}
    if kind == "unet_apply":
        return {"bytes": 8 * n, "flops": 2 * UNET_MACS * n}
    return {"bytes": 8 * n, "flops": 6 * UNET_MACS * n}


# ---- the same in 64 bits ----------------------------------------------------
def _shift(z, dy, dx, fill):
    """z at (row + dy, col + dx), `fill` outside."""
    p = torch.nn.functional.pad(z[None, None], (1, 1, 1, 1), value=fill)[0, 0]
    return p[1 + dy:1 + dy + z.shape[0], 1 + dx:1 + dx + z.shape[1]]


def _edges(rows, cols, bc):
    """Cells held fixed: those on an open edge."""
    held = torch.zeros((rows, cols), device="cuda", dtype=torch.bool)
    for edge, s in zip(bc, ((0, slice(None)), (slice(None), -1), (-1, slice(None)), (slice(None), 0))):
        if edge == "o":
            held[s] = True
    return held


def _cg(apply, diag, b, tol):
    x = torch.zeros_like(b)
    r = b.clone()
    q = r / diag
    p = q.clone()
    rq = (r * q).sum()
    stop = tol * float(b.norm())
    for k in range(20000):
        a = apply(p)
        alpha = rq / (p * a).sum()
        x += alpha * p
        r -= alpha * a
        if k % 16 == 15 and float(r.norm()) <= stop:
            break
        q = r / diag
        new = (r * q).sum()
        p = q + (new / rq) * p
        rq = new
    return x


def _exact_diffusion(case, z32, dt, nonlinear):
    rows, cols = case["rows"], case["cols"]
    h, D, Sc = HILL["cell"], HILL["D"], HILL["Sc"]
    held = _edges(rows, cols, case["bc"])
    free = (~held).double()
    zn = z32.double()
    DA, inv_dt = float(np.float32(D)) / (h * h), 1.0 / float(np.float32(dt))

    def nb(a, dy, dx):  # the neighbour, or the cell itself off the grid
        p = torch.nn.functional.pad(a[None, None], (1, 1, 1, 1), mode="replicate")[0, 0]
        return p[1 + dy:1 + dy + rows, 1 + dx:1 + dx + cols]

    faces = ((-1, 0), (0, 1), (1, 0), (0, -1))
    z = zn.clone()
    for _ in range(60 if nonlinear else 3):
        alphas = []
        if nonlinear:
            sx, sy = (nb(z, 0, 1) - nb(z, 0, -1)) / (2 * h), (nb(z, 1, 0) - nb(z, -1, 0)) / (2 * h)
        F = inv_dt * (z - zn)
        for k, (dy, dx) in enumerate(faces):
            sn = (nb(z, dy, dx) - z) / h
            if nonlinear:
                s = sx if k % 2 == 0 else sy
                st = 0.5 * (s + nb(s, dy, dx))
                al = 1.0 / (1.0 - torch.clamp((sn * sn + st * st) / (Sc * Sc), max=0.9999))
            else:
                al = torch.ones_like(z)
            alphas.append(al)
            F = F - DA * al * sn * h
        F = F * free
        if float(F.abs().max()) <= 1e-14:
            break

        inside = [_shift(torch.ones_like(z), dy, dx, 0.0) for dy, dx in faces]
        diag = inv_dt + DA * sum(a * i for a, i in zip(alphas, inside))

        def apply(v):
            out = inv_dt * v
            for (dy, dx), a in zip(faces, alphas):
                out = out + DA * a * (v - nb(v, dy, dx))
            return out * free

        z = z + _cg(apply, diag, -F, 1e-12 if nonlinear else 1e-14)
    return z


def _exact_incision(case, z32):
    """D8 receivers, drainage areas and the implicit step, level by level."""
    rows, cols, n = case["rows"], case["cols"], case["n"]
    N = rows * cols
    z = z32.double()
    cell = 30.0
    steps = ((-1, 0), (-1, 1), (0, 1), (1, 1), (1, 0), (1, -1), (0, -1), (-1, -1))
    best = torch.zeros_like(z)
    recv = torch.full((rows, cols), -1, device="cuda", dtype=torch.long)
    dist = torch.full_like(z, cell)
    flat = torch.arange(N, device="cuda").view(rows, cols)
    for d, (dy, dx) in enumerate(steps):
        length = cell * (math.sqrt(2.0) if d % 2 else 1.0)
        s = (z - _shift(z, dy, dx, math.inf)) / length
        better = s > best
        best = torch.where(better, s, best)
        recv = torch.where(better, flat + dy * cols + dx, recv)
        dist = torch.where(better, torch.full_like(dist, length), dist)
    recv, dist, old = recv.view(-1), dist.view(-1), z.reshape(-1)
    up = torch.where(recv >= 0, recv, flat.view(-1))
    depth = (recv >= 0).long()
    while True:  # distance to the outlet by doubling
        further = depth + depth[up]
        if torch.equal(further, depth):
            break
        depth, up = further, up[up]
    order = torch.argsort(depth)
    bounds = torch.searchsorted(depth[order], torch.arange(int(depth.max()) + 2, device="cuda")).tolist()
    levels = [order[a:b] for a, b in zip(bounds[:-1], bounds[1:])]
    area = torch.full((N,), cell * cell, device="cuda", dtype=torch.float64)
    for at in reversed(levels[1:]):
        area.index_add_(0, recv[at], area[at])
    kdt = float(np.float32(2e-5)) * (area / cell) ** float(np.float32(0.45)) * 500.0
    new = old.clone()
    for at in levels[1:]:
        zo, zr, k, dx = old[at], new[recv[at]], kdt[at], dist[at]
        x = zo.clone()
        for _ in range(1 if n == 1.0 else 12):
            s = torch.clamp((x - zr) / dx, min=0.0)
            x = x - (x - zo + k * s ** n) / (1.0 + k * n / dx * s ** (n - 1.0))
        new[at] = torch.where(zr >= zo, zo, x)
    return new.view(rows, cols)


def _exact_unet(params, r, e):
    """The network as it is defined (weights and activations rounded to
    bf16 between layers), every sum in 64 bits; e: the loss and gradients."""
    def bf(x):  # rounds, and lets gradients through as they are
        return x + (x.detach().bfloat16().double() - x.detach())

    p = torch.from_numpy(params).cuda().double().requires_grad_(e is not None)
    ws, at = [], 0
    for _, ci, co in G.UNET_LAYERS:
        ws.append(bf(p[at:at + co * 9 * ci].view(co, 3, 3, ci).permute(0, 3, 1, 2)))
        at += co * 9 * ci
    bs = []
    for _, _, co in G.UNET_LAYERS:
        bs.append(p[at:at + co])
        at += co

    def conv(x, k):
        return torch.nn.functional.conv2d(x, ws[k], bs[k], padding=1)

    def pool(x):
        return bf(torch.nn.functional.avg_pool2d(x, 2))

    def up(x):
        return x.repeat_interleave(2, -1).repeat_interleave(2, -2)

    rd = r.double()
    rms = torch.sqrt((rd * rd).mean()).float()
    x0 = bf((r / rms).double())[None, None]
    e0 = bf(torch.relu(conv(x0, 0)))
    e1 = bf(torch.relu(conv(pool(e0), 1)))
    e2 = bf(torch.relu(conv(pool(e1), 2)))
    e3 = bf(torch.relu(conv(pool(e2), 3)))
    d2 = bf(torch.relu(conv(up(e3), 4)) + e2)
    d1 = bf(torch.relu(conv(up(d2), 5)) + e1)
    d0 = bf(torch.relu(conv(up(d1), 6)) + e0)
    y = conv(d0, 7)[0, 0] * rms.double()
    if e is None:
        return y.detach()
    ed = e.double()
    loss = ((y - ed) ** 2).sum() / (ed * ed).sum()
    loss.backward()
    return dict(loss=float(loss), grad=p.grad)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("diffuse", "roering", "incise", "unet_apply", "unet_train"):
        g = _gen(seed)
        rows, cols = case["rows"], case["cols"]
        if kind == "incise":
            return _exact_incision(case, _valley(rows, cols, g))
        if kind in ("unet_apply", "unet_train"):
            r, e = _residual_pair(rows, cols, g)
            return _exact_unet(_unet_params(seed), r, e if kind == "unet_train" else None)
        _mask(rows, cols, 0, g)
        z = _hills(rows, cols, HILL["cell"], case.get("steep", 1.0) * HILL["Sc"], g)
        return _exact_diffusion(case, z, case["number"] * HILL["cell"] ** 2 / HILL["D"], kind == "roering")
    # A fill is a sequence of 32-bit roundings in its own order, and so are the
    # steps that start with one; a routing pass returns whole numbers, and its
    # area is a count or a sum in the receivers' order.
    return None
