"""Whole steps in one kernel (step_kernel, the default tiled kernels of a
two-dimensional grid) against a launch per sweep (CLIFFS_SWEEP_DIRECT):
bit-identical states, max-wave fields and status.

Grids around the kernel's tiles, as small as 3 cells across and large enough
for each of its three tiles (64 columns x 30 rows on large grids, 32 x 14 and
32 x 10 on smaller ones), in plane, spherical and stretched coordinates; on each a rough sea
floor with islands and ponds, so that every kind of cell (plain, shoreline,
flooded, drying, land at rest, line ends) lies in tiles' middles, edges and
corners; odd and even step counts (a call's last odd step runs a sweep at a
time); forced edges; and two contexts stepped in turn.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
pkg = importlib.import_module("cliffs-src_gb300")
cg = pkg.cliffs_gpu


def _case(nx, ny, metric, seed):
    """Depths of -0.18 to 0.3 m and a surface of +-0.05 m: a third of the grid is land."""
    rng = np.random.default_rng(seed)
    d = (0.3 * rng.uniform(-0.6, 1.0, (ny, nx))).astype(np.float32).astype(np.float64)
    k = max(2, nx // 3)
    d[:, :k] += np.float32(1.5)  # a deep west, plain cells for the most part
    h = np.maximum(d + 0.1 * rng.uniform(-0.5, 0.5, (ny, nx)), 0.0)
    dx, dy = np.full(nx - 1, 10.0), np.full(ny - 1, 10.0)
    rs = zeta = None
    if metric == "sphere":
        lat = np.radians(np.linspace(10.0, 60.0, ny))
        rs, zeta = np.cos(lat), 1e-4 * np.tan(lat)
        dx = dx * 2.0
    elif metric == "stretched":
        dx, dy = rng.uniform(8.0, 12.0, nx - 1), rng.uniform(8.0, 12.0, ny - 1)
        rs = rng.uniform(0.9, 1.1, ny)
    return dict(d=d.astype(np.float32).astype(np.float64), h=h, dx=dx, dy=dy, rs=rs, zeta=zeta)


def _grid(c, kind):
    g = pkg.GpuGrid(c["d"], dx=c["dx"], row_scale=c["rs"], dy=c["dy"], zeta=c["zeta"], ground=0.01, crough=0.000625,
                    dt=0.15)
    g.set_initial(c["h"])
    g.set_sweep_kernel(kind)
    return g


def _same(a, b):
    for x, y in zip((*a.download_state(), *a.maxwave()), (*b.download_state(), *b.maxwave())):
        assert np.array_equal(x, y)
    assert a.status() == b.status() and a.courant() == b.courant()
    assert np.isfinite(a.download_state()[0]).all()


@pytest.mark.parametrize("nx,ny,metric", [
    (3, 3, "plane"), (4, 95, "plane"), (130, 3, "plane"), (63, 29, "plane"), (64, 30, "plane"), (65, 31, "plane"),
    (66, 62, "sphere"), (127, 33, "stretched"), (129, 61, "sphere"), (200, 91, "stretched"), (257, 130, "plane"),
    (31, 11, "plane"), (33, 21, "sphere"), (97, 41, "stretched"),
    (1290, 311, "plane"), (1279, 323, "sphere"), (1665, 309, "stretched"),  # 32 x 14 tiles
    (1601, 751, "plane"), (1663, 749, "sphere"), (1665, 781, "stretched")])  # 64 x 30 tiles
def test_whole_steps_match_sweeps(nx, ny, metric):
    c = _case(nx, ny, metric, nx * 1000 + ny)
    a, b = _grid(c, cg.TILED), _grid(c, cg.DIRECT)
    for steps in (41, 2, 3, 17):
        a.step(steps)
        b.step(steps)
    _same(a, b)


def test_forced_whole_steps_match_sweeps():
    c = _case(190, 97, "plane", 7)
    grids = [_grid(c, k) for k in (cg.TILED, cg.DIRECT)]
    t = np.arange(8) * 1.5
    rec = [0.05 * np.sin(t[:, None, None] + np.arange(3)[None, :, None] + 0.01 * np.arange(n)[None, None, :])
           for n in (97, 97, 190, 190)]
    for g in grids:
        g.set_feed(t, *rec, irec=1, freeze=False)
        g.step(90)  # past the last record
    _same(*grids)


def test_contexts_in_turn():
    c = [_case(150, 70, "plane", s) for s in (1, 2)]
    a, b = [_grid(x, cg.TILED) for x in c], [_grid(x, cg.DIRECT) for x in c]
    for _ in range(3):
        for g in (*a, *b):
            g.step(18)
    for x, y in zip(a, b):
        _same(x, y)


@pytest.mark.parametrize("metrics", [("plane", "plane", "plane"), ("sphere", "plane", "sphere"),
                                     ("plane", "stretched", "sphere")])
def test_batched_whole_steps_match_sweeps(metrics):
    """Uneven grids in one batch, by steps of odd and even length."""
    sizes = [(3, 40), (65, 31), (190, 97 if metrics[2] == "plane" else 2100)]
    cs = [_case(nx, ny, m, nx) for (nx, ny), m in zip(sizes, metrics)]
    a, b = [_grid(c, cg.TILED) for c in cs], [_grid(c, cg.DIRECT) for c in cs]
    batch = pkg.Batch(a)
    for graph_steps in (8, 5):
        batch.set_plan(cg.GRAPH, graph_steps=graph_steps)
        for steps in (21, 2, 7):
            batch.step(steps)
            for g in b:
                g.step(steps)
    for x, y in zip(a, b):
        _same(x, y)
    batch.close()
