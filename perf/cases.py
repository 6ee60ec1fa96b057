"""The work that the framework's performance is measured on.

Each case is what a user's program does with grids, ensembles or networks that it has set up: a run of the solver
from given initial conditions to its outputs (the time loop between two output events, with the state going in and
the state and the maximum fields coming out in pinned host arrays), a batched run of source scenarios, and the
surrogate's inference and gradients.  Outputs are whole.  exact() restates each of them in 64-bit torch.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("cliffs-src_gb300")
cg = pkg.cliffs_gpu

GRAV = 9.800000190734863  # (double)9.8f, the solver's gravity
SQR2 = 1.4142135381698608
EARTH = 6371009.0
DRY = -1.0e32  # the output fields' value where no water was
F64 = torch.float64


def listed():
    return [
        # the smallest grid: a wave tank or a beach transect, one sweep a step, where launches and latency count
        dict(name="channel 2000", kind="channel", n=2000, along="x", steps=400),
        # a harbour or a quick-look basin: a two-dimensional grid that fits in a fraction of the chip
        dict(name="basin 256x256", kind="basin", nx=256, ny=256, metric="plane", friction=True, steps=200),
        # a regional grid of odd, ragged sizes and unequal spacing in x and y
        dict(name="basin 1003x777", kind="basin", nx=1003, ny=777, metric="plane", friction=True, steps=120),
        # the 2048 x 2048 shelf, the framework's headline grid: 100 m, runup on, friction on
        dict(name="shelf 2048x2048", kind="basin", nx=2048, ny=2048, metric="plane", friction=True, steps=100),
        # an ocean basin at 1/12 degree on the sphere, out of the second-level cache
        dict(name="sphere 4320x2160", kind="basin", nx=4320, ny=2160, metric="sphere", friction=False, steps=60),
        # a spherical grid refined towards its coast: variable spacing along both axes
        dict(name="stretched 1201x903", kind="basin", nx=1201, ny=903, metric="stretched", friction=True, steps=100),
        # a nested child: forced at its four edges by its parent's records, runup on its coast
        dict(name="forced child 600x600", kind="forced", nx=600, ny=600, records=12, steps=150),
        # a source study: scenarios on grids of uneven size, stepped together, gauges and maxima read
        dict(name="ensemble of 24", kind="ensemble", scenarios=24, side=768, steps=64),
        # the surrogate asked for a hazard study's scenarios: the gauge network, and the map network
        dict(name="predict gauges 4096", kind="predict", batch=4096, width=512, depth=3, map=False),
        dict(name="predict maps 256", kind="predict", batch=256, width=512, depth=3, map=True),
        # the surrogate in training: forward and backward of a batch, every gradient read
        dict(name="gradients maps 512", kind="gradients", batch=512, width=512, depth=3, map=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channel", "basin", "basin", "basin", "forced", "ensemble", "predict", "gradients"])
    if kind == "channel":
        return dict(kind=kind, n=_log(rng, 300, 6000), along=rng.choice(["x", "y"]), steps=rng.randint(100, 400))
    if kind == "basin":
        nx, ny = _log(rng, 190, 3600), _log(rng, 150, 2400)
        steps = max(20, min(200, int(4.0e8 / (nx * ny))))
        return dict(kind=kind, nx=nx, ny=ny, metric=rng.choice(["plane", "plane", "sphere", "stretched"]),
                    friction=rng.random() < 0.7, steps=steps - rng.randint(0, 9))
    if kind == "forced":
        return dict(kind=kind, nx=_log(rng, 250, 1000), ny=_log(rng, 250, 1000), records=rng.randint(5, 20),
                    steps=rng.randint(60, 150))
    if kind == "ensemble":
        return dict(kind=kind, scenarios=rng.randint(4, 24), side=rng.randint(300, 800), steps=rng.randint(33, 70))
    maps = rng.random() < 0.5
    batch = 16 * _log(rng, 4, 32) if kind == "gradients" else _log(rng, 50, 300 if maps else 4096)
    return dict(kind=kind, batch=batch, width=rng.choice([128, 256, 512]), depth=rng.choice([2, 3]), map=maps)


# ---- inputs --------------------------------------------------------------------------------------------------

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) + 12345)
    return g


def _f32(a):
    return a.to(torch.float32).to(F64)


def _rough(g, ny, nx):
    """A random field with a k^-2 power spectrum and unit deviation: sea-floor roughness."""
    ky = torch.fft.fftfreq(ny, dtype=F64, device="cuda")[:, None]
    kx = torch.fft.rfftfreq(nx, dtype=F64, device="cuda")[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = math.inf
    ph = torch.randn((ny, nx // 2 + 1, 2), dtype=F64, device="cuda", generator=g)
    f = torch.fft.irfft2(torch.view_as_complex(ph) / k, s=(ny, nx))
    return f / (f.std() + 1e-30)


def _profile(nx, land):
    """Depth across a basin with its coast on the high-x side: a 4000 m abyss, a break to a 200 m shelf, a slope
    over the shelf to the shore and `land` columns of beach that rises to a few metres, then steeply."""
    s = (nx - 1 - land) - torch.arange(nx, dtype=F64, device="cuda")  # columns seaward of the shore
    shelf = 0.22 * nx
    slope = torch.where(s < 24, 0.4 * s, 9.6 + (s - 24).clamp(min=0) * (190.4 / max(0.8 * shelf - 24, 1.0)))
    d = torch.minimum(slope, torch.full_like(s, 200.0))
    deep = 200.0 + 1900.0 * (1.0 + torch.tanh((s - shelf - 0.04 * nx) / (0.015 * nx)))
    d = torch.where(s > shelf, deep, d)
    return torch.where(s < -12, -4.8 + 2.0 * (s + 12), d)


def _uplift(g, x, y, shore):
    """A source on the shelf: an elliptical hump with a trough beside it, 1-2 m high, that reaches the shore."""
    r = torch.rand(5, dtype=F64, device="cuda", generator=g).tolist()
    lx, ly = float(x[-1] - x[0]), float(y[-1] - y[0])
    cx, cy = float(x[int(shore * (0.80 + 0.1 * r[0]))]), float(y[0]) + (0.3 + 0.4 * r[1]) * ly
    ax, ay, th = 0.16 * lx, 0.25 * ly, 0.3 * (r[2] - 0.5)
    X, Y = (x - cx)[None, :], (y - cy)[:, None]
    a, b = (X * math.cos(th) + Y * math.sin(th)) / ax, (-X * math.sin(th) + Y * math.cos(th)) / ay
    return (1.0 + r[3]) * (torch.exp(-(a * a + b * b)) - 0.4 * r[4] * torch.exp(-(a * a + (b - 2.0) ** 2)))


def _basin(g, nx, ny, metric, friction, dx=100.0, ground=0.01):
    """Depth, initial water depth, spacings and constants of a basin with a beach along its high-x side."""
    land = max(16, nx // 40)
    d = _profile(nx, land)[None, :].repeat(ny, 1)
    d = _f32(d + 0.04 * d.abs() * _rough(g, ny, nx))
    n = torch.arange(max(nx, ny), dtype=F64, device="cuda")
    if metric == "plane":
        x, y = n[:nx] * dx, n[:ny] * (0.8 * dx if nx != ny else dx)
        hx, hy, rs, zeta = (x[1:] - x[:-1]), (y[1:] - y[:-1]), None, None
        small = min(dx, float(hy.min()))
    else:
        if metric == "sphere":
            lon, lat = n[:nx] / 12.0, -72.0 + n[:ny] * (144.0 / max(ny - 1, 1))
        else:  # refined smoothly, by up to two fifths, towards the coast and the middle latitudes
            lon = torch.cumsum(torch.cat([n[:1], (1.0 - 0.4 * n[1:nx] / nx) / 12.0]), 0)
            w = 1.0 - 0.4 * torch.sin(math.pi * n[1:ny] / ny)
            lat = -60.0 + torch.cumsum(torch.cat([n[:1], w * (105.0 / float(w.sum()))]), 0)
        beta = math.pi * EARTH / 180.0
        hx, hy = beta * (lon[1:] - lon[:-1]), beta * (lat[1:] - lat[:-1])
        rs, zeta = torch.cos(torch.deg2rad(lat)), (0.125 / EARTH) * torch.tan(torch.deg2rad(lat))
        small = min(float(hx.min() * rs.min()), float(hy.min()))
        x, y = lon, lat
    eta = _uplift(g, x, y, nx - 1 - land) if metric == "plane" else _uplift(g, n[:nx], n[:ny], nx - 1 - land)
    h0 = torch.where(d > 0, d + eta, d)
    dt = 0.8 * small / math.sqrt(GRAV * float(d.max() + 3.0))
    return dict(d=d, h0=h0, hx=hx, hy=hy, rs=rs, zeta=zeta, ground=ground, crough=0.000625 if friction else 0.0, dt=dt)


def _channel(g, n, along):
    """A wave tank: 1 m of water, a 1:20 beach to 0.5 m above it, a solitary hump before the slope."""
    r = torch.rand(2, dtype=F64, device="cuda", generator=g).tolist()
    dx = 100.0 / n
    x = torch.arange(n, dtype=F64, device="cuda") * dx
    toe = 60.0
    d = _f32(torch.where(x < toe, torch.ones_like(x), 1.0 - (x - toe) / 20.0).clamp(min=-0.5))
    amp = 0.02 + 0.04 * r[0]
    eta = amp / torch.cosh(math.sqrt(0.75 * amp) * (x - (toe + 6.0 + 6.0 * r[1]))) ** 2
    h0 = torch.where(d > 0, d + eta, d)
    h = torch.full((n - 1,), dx, dtype=F64, device="cuda")
    shape = (1, n) if along == "x" else (n, 1)
    return dict(d=d.reshape(shape), h0=h0.reshape(shape), hx=h if along == "x" else None,
                hy=h if along == "y" else None, rs=None, zeta=None, ground=0.003, crough=0.0,
                dt=0.8 * dx / math.sqrt(GRAV * 1.06))


def _records(g, b, nrec, steps):
    """Edge records of a parent grid over the run: a wave train with u and v in step with the elevation."""
    ny, nx = b["d"].shape
    t = torch.arange(nrec, dtype=F64, device="cuda") * (steps * b["dt"] * 1.1 / (nrec - 1))
    out = [t]
    for length in (ny, ny, nx, nx):
        ph, s = float(torch.rand(1, device="cuda", generator=g)), torch.linspace(0, 1, length, dtype=F64, device="cuda")
        eta = 0.3 * torch.sin(2 * math.pi * (t[:, None] / (40 * b["dt"]) + ph + 0.2 * s[None, :]))
        out.append(torch.stack([0.05 * eta, 0.02 * eta, eta], 1))
    return out


def _sides(case):
    """The grids of an ensemble: a quarter of the scenarios each at 256 and at a half, three quarters and the whole
    of the largest side, in turn."""
    return [(256, case["side"] // 2, case["side"] * 3 // 4, case["side"])[k % 4] for k in range(case["scenarios"])]


def _net(case, seed):
    """Weights, biases, inputs and targets of a network, scaled as training leaves them."""
    rng = np.random.default_rng(seed)
    side, ch = (128, (32, 16, 8, 1)) if case["map"] else (0, (32, 16, 8, 1))
    n_out, lat = 64, (side // 8) ** 2 * ch[0]
    dims = [9] + [case["width"]] * case["depth"] + [n_out + lat]
    shapes = [(dims[i + 1], dims[i]) for i in range(len(dims) - 1)]
    if side:
        shapes += [(ch[i + 1], 9 * ch[i]) for i in range(3)]
    w = [(rng.standard_normal(s) * math.sqrt(1.6 / s[1])).astype(np.float32) for s in shapes]
    b = [rng.normal(0, 0.05, s[0]).astype(np.float32) for s in shapes]
    x = rng.uniform(-1, 1, (case["batch"], 9)).astype(np.float32)
    t = rng.standard_normal((case["batch"], n_out + side * side)).astype(np.float32)
    t[:, n_out:] = np.maximum(t[:, n_out:] + 1.0, 0.0)  # a map holds depths: none below zero
    return dict(w=w, b=b, x=x, t=t, n_out=n_out, side=side, ch=ch)


def _inputs(case, seed):
    g = _gen(seed)
    if case["kind"] == "channel":
        return _channel(g, case["n"], case["along"])
    if case["kind"] == "basin":
        return _basin(g, case["nx"], case["ny"], case["metric"], case["friction"])
    if case["kind"] == "forced":
        b = _basin(g, case["nx"], case["ny"], "plane", True, dx=50.0, ground=0.05)
        return dict(b, feed=_records(g, b, case["records"], case["steps"]))
    if case["kind"] == "ensemble":
        return [_basin(g, s, s, "plane", True) for s in _sides(case)]
    return _net(case, seed)


# ---- the passes ----------------------------------------------------------------------------------------------

def _pinned(t, dtype=np.float64):
    a = cg.pinned(tuple(t.shape), dtype)
    torch.from_numpy(a).copy_(t)
    return a


def _grid(b):
    host = lambda t: None if t is None else t.cpu().numpy()  # noqa: E731
    h0 = _pinned(b["h0"])
    g = pkg.GpuGrid(host(b["d"]), dx=host(b["hx"]), row_scale=host(b["rs"]), dy=host(b["hy"]), zeta=host(b["zeta"]),
                    ground=b["ground"], crough=b["crough"], dt=b["dt"])
    g.set_initial(h0)
    return g, h0


def prepare(case, seed):
    b = _inputs(case, seed)
    if case["kind"] in ("channel", "basin", "forced"):
        g, h0 = _grid(b)
        shape = tuple(b["d"].shape)
        s = dict(kind=case["kind"], grid=g, h0=h0, steps=case["steps"],
                 state=[cg.pinned(shape) for _ in range(3)], most=[cg.pinned(shape, np.float32) for _ in range(2)])
        if "feed" in b:
            s["feed"] = [r.cpu().numpy() for r in b["feed"]]
        return s
    if case["kind"] == "ensemble":
        made = [_grid(m) for m in b]
        batch = pkg.Batch([g for g, _ in made])
        batch.set_plan(cg.GRAPH, graph_steps=32)
        return dict(kind=case["kind"], grids=[g for g, _ in made], h0=[h for _, h in made], batch=batch,
                    steps=case["steps"], most=[[cg.pinned(h.shape, np.float32) for _ in range(2)] for _, h in made])
    S = importlib.import_module("cliffs-src_gb300.surrogate")
    net = S.MLP(9, case["width"], case["depth"], b["n_out"], seed=seed, map_side=b["side"], map_ch=b["ch"][:3])
    for k, (w, c) in enumerate(zip(b["w"], b["b"])):
        net.set(k, 0, w)
        net.set(k, 1, c)
    return dict(kind=case["kind"], net=net, x=b["x"], t=b["t"])


def run(state):
    kind = state["kind"]
    if kind == "predict":
        return state["net"].predict(state["x"])
    if kind == "gradients":
        loss, gw, gb = state["net"].gradients(state["x"], state["t"])
        return dict(loss=np.float32(loss), weights=gw, biases=gb)
    if kind == "ensemble":
        for g, h0 in zip(state["grids"], state["h0"]):
            g.set_initial(h0)
        state["batch"].step(state["steps"])
        return [g.maxwave(out=m) for g, m in zip(state["grids"], state["most"])]
    g = state["grid"]
    g.set_initial(state["h0"])
    if "feed" in state:
        t, w, e, s, n = state["feed"]
        g.t.value = 0.0
        g.set_feed(t, w, e, s, n, irec=1, freeze=False)
    g.step(state["steps"])
    return dict(state=g.download_state(out=state["state"]), most=g.maxwave(out=state["most"]))


def work(case):
    """A step reads the depth and the state and writes the state, and reads and writes the two maximum fields:
    44 bytes a cell, and about 120 operations a cell and sweep.  A run moves its state over the host link once each
    way besides."""
    k = case["kind"]
    if k == "channel":
        return dict(bytes=case["n"] * (44.0 * case["steps"] + 40), flops=120.0 * case["n"] * case["steps"])
    if k in ("basin", "forced"):
        cells = case["nx"] * case["ny"]
        return dict(bytes=cells * (44.0 * case["steps"] + 40), flops=240.0 * cells * case["steps"])
    if k == "ensemble":
        cells = sum(s * s for s in _sides(case))
        return dict(bytes=cells * (44.0 * case["steps"] + 16), flops=240.0 * cells * case["steps"])
    n, w, m = case["batch"], case["width"], 128 * 128 if case["map"] else 0
    last = 64 + (16 * 16 * 32 if case["map"] else 0)
    par = 9 * w + (case["depth"] - 1) * w * w + w * last
    conv = (m // 16) * 9 * 32 * 16 + (m // 4) * 9 * 16 * 8 + m * 9 * 8
    ops, io = 2.0 * n * (par + conv), 4.0 * n * (9 + 64 + m) + 2.0 * par
    return dict(bytes=io if k == "predict" else 2 * io, flops=ops if k == "predict" else 3 * ops)


# ---- the same in 64 bits ---------------------------------------------------------------------------------------

def _shift(a, k, fill):
    """a at position i + k along the last axis, `fill` past its ends."""
    out = torch.full_like(a, fill)
    if k > 0:
        out[:, :-k] = a[:, k:]
    else:
        out[:, -k:] = a[:, :k]
    return out


def _sweep(H, u, v, d, h, zeta, scale, b, edges):
    """One dimensional sweep of the VTCS-2 scheme (cliffs.f:17-346) along the last axis of every row: H total depth,
    u normal and v tangential velocity; h spacings, zeta a metric term a position, scale a factor on h a row; edges
    the forced (u, v, eta) at either end of each row."""
    n, g, ground, dt = H.shape[1], GRAV, b["ground"], b["dt"]
    z = torch.zeros((), dtype=F64, device=H.device)
    land = H <= ground
    eta = H - d
    # flooding of a land cell from a wet neighbour (cliffs.f:74-111)
    Rf = land & ~_shift(land, -1, True) & (_shift(u, -1, 0.0) >= 0) & (_shift(eta, -1, 0.0) + d > ground)
    Lf = land & ~Rf & ~_shift(land, 1, True) & (_shift(u, 1, 0.0) <= 0) & (_shift(eta, 1, 0.0) + d > ground)
    fl, water = Rf | Lf, (~land).any(1, keepdim=True)
    wet = ~land | fl
    celmin = math.sqrt(g * ground)
    U = torch.where(Rf, _shift(u, -1, 0.0), torch.where(Lf, _shift(u, 1, 0.0), u))
    V = torch.where(Rf, _shift(v, -1, 0.0), torch.where(Lf, _shift(v, 1, 0.0), v))
    C = torch.where(fl, torch.full_like(H, celmin), torch.sqrt(g * H.clamp(min=ground)))
    Hf = torch.where(fl, torch.full_like(H, ground), H)
    E = torch.where(fl, ground - d, eta)
    # neighbours, or the mirror image of the cell where there is none (cliffs.f:137-152)
    wl, wr = _shift(wet, -1, False), _shift(wet, 1, False)
    at = lambda a, k, w, own: torch.where(w, _shift(a, k, 0.0), own)  # noqa: E731
    ua, ub = at(U, -1, wl, -U), at(U, 1, wr, -U)
    va, vb = at(V, -1, wl, V), at(V, 1, wr, V)
    ca, cb = at(C, -1, wl, C), at(C, 1, wr, C)
    ea, eb = at(E, -1, wl, E), at(E, 1, wr, E)
    da, db = at(d, -1, wl, d), at(d, 1, wr, d)
    al = torch.ones((H.shape[0], 1), dtype=F64, device=H.device) if scale is None else scale[:, None]
    hp = torch.ones(n, dtype=F64, device=H.device)
    hm = hp.clone()
    hm[1:], hp[:-1] = h, h
    hm[0], hp[-1] = h[0], h[-1]
    hm, hp = hm[None, :] * al, hp[None, :] * al
    zt = z if zeta is None else zeta[None, :]

    def flux(ul, cl, el, ur, cr, er):
        s, k = g * (er - el), (ul + ur) * (cr - cl)
        return s + k + 0.5 * (ul + ur + cl + cr) * (ur - ul), s - k + 0.5 * (ul + ur - cl - cr) * (ur - ul)

    FPl, FQl = flux(ua, ca, ea, U, C, E)
    FPr, FQr = flux(U, C, E, ub, cb, eb)
    Hs = Hf.clamp(min=ground)
    fr = g * b["crough"] * U * torch.sqrt(U * U + V * V) / (Hs * torch.sqrt(Hs))
    sph = 8.0 * C * U * zt
    P, Q, dtx = U + C, U - C, dt / (hm + hp)
    mP, pP, mQ, pQ = FPl / hm, FPr / hp, FQl / hm, FQr / hp
    SP, SQ = 0.5 * (mP + pP), 0.5 * (mQ + pQ)
    deep = (d > ground) & (da > ground) & (db > ground)  # transcritical points (cliffs.f:228-245)
    sd = 2.0 * g * (torch.sqrt((d * db).clamp(min=0)) - torch.sqrt((d * da).clamp(min=0)))
    SP = torch.where(deep & (ua + ca < 0) & (ub + cb > 0), (P * (2.0 * (cb - ca) + ub - ua) - sd) / (hm + hp), SP)
    SQ = torch.where(deep & (ua - ca < 0) & (ub - cb > 0), (Q * (-2.0 * (cb - ca) + ub - ua) - sd) / (hm + hp), SQ)
    dP = -dt * (SP + P * dtx * (mP - pP) + fr - sph)
    dQ = -dt * (SQ + Q * dtx * (mQ - pQ) + fr + sph)
    Qv = (vb - V) / hp - (V - va) / hm
    nv = V - U * dtx * ((vb - va) - Qv * (U * dt + hp - hm))
    nc, nu = C + 0.25 * (dP - dQ), U + 0.5 * (dP + dQ)
    # the angle limiter of a newly flooded cell at the shore (cliffs.f:264-285), against its wet neighbour
    k = torch.arange(n, device=H.device)[None, :]
    inner = (k >= 1) & (k <= n - 2)
    ic, iu = torch.where(inner, nc, C), torch.where(inner, nu, U)
    for side, cond in ((1, Lf & ~wl), (-1, Rf & ~wr)):
        oc, ou = _shift(ic, side, 0.0), _shift(iu, side, 0.0)
        lim = torch.where(cond & (SQR2 * nc > oc), oc / SQR2, nc)
        nu = torch.where(cond, torch.maximum(nu, ou) if side == 1 else torch.minimum(nu, ou), nu)
        nc = lim
    nH = nc * nc.abs() / g
    # ends of the rows: open or forced (cliffs.f:287-329), else as flooded
    for e, o, sgn in ((0, 1, 1.0), (n - 1, n - 2, -1.0)):
        fu, fv, fe = edges[0 if e == 0 else 1] if edges is not None else (z, z, z)
        c0, u0, v0, e0, d0 = C[:, e], U[:, e], V[:, e], E[:, e], d[:, e]
        ih = 1.0 / hp[:, 0] if e == 0 else 1.0 / hm[:, -1]
        if e == 0:
            FP, FQ = flux(u0, c0, e0, U[:, o], C[:, o], E[:, o])
        else:
            FP, FQ = flux(U[:, o], C[:, o], E[:, o], u0, c0, e0)
        s0 = 8.0 * c0 * u0 * (z if zeta is None else zeta[e])
        cbn = torch.sqrt(g * (d0 + fe).clamp(min=ground))
        jump = 2.0 * g * (fe - e0) / (cbn + c0)
        eP, eQ = ((fu - u0) + jump, -dt * (FQ * ih + s0)) if e == 0 else (-dt * (FP * ih - s0), (fu - u0) - jump)
        on = wet[:, e] & wet[:, o] & (fe + d0 > ground)
        slope = (V[:, o] - v0) * sgn
        out = u0 < 0 if e == 0 else u0 > 0
        c1 = c0 + 0.25 * (eP - eQ)
        nH[:, e] = torch.where(on, c1 * c1.abs() / g, Hf[:, e])
        nu[:, e] = torch.where(on, u0 + 0.5 * (eP + eQ), u0)
        nv[:, e] = torch.where(on, torch.where(out, v0 - dt * slope * u0 * ih, fv + z * v0), v0)
    # new land in a row with water; a row without water is left alone (cliffs.f:113-122)
    dry = ~wet & water
    keep = ~wet & ~water
    nH = torch.where(dry, z, torch.where(keep, H, nH))
    nu = torch.where(dry, z, torch.where(keep, u, nu))
    nv = torch.where(dry, z, torch.where(keep, v, nv))
    return nH, nu, nv


def _solve(b, steps):
    """The time loop (cliffs_main.f:303-355): state and the maximum fields after `steps` steps."""
    d = b["d"]
    ny, nx = d.shape
    H = torch.where(b["h0"] <= b["ground"], torch.zeros_like(d), b["h0"])
    u, v = torch.zeros_like(d), torch.zeros_like(d)
    top, fast, t = -d, torch.zeros_like(d), 0.0
    feed = b.get("feed")
    times = feed[0].tolist() if feed else None
    irec = 1
    T = lambda a: a.t().contiguous()  # noqa: E731
    dT = T(d)
    js, cs = slice(1, ny - 1) if ny > 2 else slice(0, 1), slice(1, nx - 1) if nx > 2 else slice(0, 1)
    for _ in range(steps):
        ex = ey = None
        t += b["dt"]
        if feed:
            while t >= times[irec - 1]:
                irec += 1
            w = (times[irec - 1] - t) / (times[irec - 1] - times[irec - 2])
            W, E, S, N = (r[irec - 2] * w + r[irec - 1] * (1.0 - w) for r in feed[1:])
            ex = [[e[k][js] for k in (0, 1, 2)] for e in (W, E)]
            ey = [[e[k][cs] for k in (1, 0, 2)] for e in (S, N)]
        if nx > 2:
            rows = (H[js], u[js], v[js])
            new = _sweep(*rows, d[js], b["hx"], None, None if b["rs"] is None else b["rs"][js], b, ex)
            H, u, v = H.clone(), u.clone(), v.clone()
            H[js], u[js], v[js] = new
        if ny > 2:
            Ht, ut, vt = T(H), T(u), T(v)
            Ht[cs], vt[cs], ut[cs] = _sweep(Ht[cs], vt[cs], ut[cs], dT[cs], b["hy"], b["zeta"], None, b, ey)
            H, u, v = T(Ht), T(ut), T(vt)
        top = torch.maximum(top, H - d)
        fast = torch.maximum(fast, u * u + v * v)
    cel = torch.sign(H) * torch.sqrt(GRAV * H.abs())
    ever = d + top > b["ground"]
    dry = torch.full_like(d, DRY)
    return dict(state=(cel, u, v), most=(torch.where(ever, top, dry), torch.where(ever, torch.sqrt(fast), dry)))


def _up2(a):
    return a.repeat_interleave(2, 1).repeat_interleave(2, 2)


def _forward(m, w, c, x):
    """The network in 64 bits: dense layers with ReLUs, then the decoder's upsamplings and 3 x 3 convolutions."""
    depth = len(w) - (3 if m["side"] else 0)
    for k in range(depth):
        x = x @ w[k].T + c[k]
        if k < depth - 1:
            x = torch.relu(x)
    if not m["side"]:
        return x
    s = m["side"] // 8
    a = torch.relu(x[:, m["n_out"]:]).reshape(len(x), s, s, m["ch"][0])
    for k in range(3):
        a = torch.nn.functional.pad(_up2(a), (0, 0, 1, 1, 1, 1))
        n = a.shape[1] - 2
        ker = w[depth + k].reshape(-1, 9, m["ch"][k])
        a = sum(a[:, i:i + n, j:j + n] @ ker[:, 3 * i + j].T for i in range(3) for j in range(3)) + c[depth + k]
        if k < 2:
            a = torch.relu(a)
    return torch.cat([x[:, :m["n_out"]], a.reshape(len(x), -1)], 1)


def exact(case, seed):
    m = _inputs(case, seed)
    if case["kind"] in ("channel", "basin", "forced"):
        return _solve(m, case["steps"])
    if case["kind"] == "ensemble":
        return [_solve(b, case["steps"])["most"] for b in m]
    grads = case["kind"] == "gradients"
    on = lambda a: torch.from_numpy(a).to("cuda", F64)  # noqa: E731
    w, c = [on(a).requires_grad_(grads) for a in m["w"]], [on(a).requires_grad_(grads) for a in m["b"]]
    x, t = on(m["x"]), on(m["t"])
    if not grads:
        with torch.no_grad():
            return torch.cat([_forward(m, w, c, p) for p in x.split(64)])
    no, loss = m["n_out"], 0.0
    for p, q in zip(x.split(64), t.split(64)):  # the mean over the batch, and over each head's outputs
        e = (_forward(m, w, c, p) - q) ** 2
        part = e[:, :no].sum() / (len(x) * no) + (e[:, no:].sum() / (len(x) * m["side"] ** 2) if m["side"] else 0.0)
        part.backward()
        loss += float(part)
    return dict(loss=loss, weights=[a.grad for a in w], biases=[a.grad for a in c])
