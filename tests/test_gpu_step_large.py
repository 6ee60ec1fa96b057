"""Whole steps beyond the sizes of test_gpu_step.py, against a launch per sweep
(CLIFFS_SWEEP_DIRECT), bit for bit: batches on 64 x 30 tiles (more than 608 of
them); single grids beyond 3648 tiles, which run by bands; and a line whose
forcing ends, which goes on in one launch."""
import importlib

import numpy as np
import pytest

from test_gpu_step import _case, _grid, _same

pytestmark = pytest.mark.gpu
pkg = importlib.import_module("cliffs-src_gb300")
cg = pkg.cliffs_gpu


@pytest.mark.parametrize("metrics", [("plane", "plane"), ("sphere", "plane"), ("plane", "stretched")])
@pytest.mark.parametrize("sizes", [((1103, 701), (1090, 722)), ((3301, 2203), (3, 40))])
def test_batches_on_large_tiles(sizes, metrics):
    cs = [_case(nx, ny, m, nx) for (nx, ny), m in zip(sizes, metrics)]
    a, b = [_grid(c, cg.TILED) for c in cs], [_grid(c, cg.DIRECT) for c in cs]
    batch = pkg.Batch(a)
    batch.set_plan(cg.GRAPH, graph_steps=4)
    for steps in (7, 2):
        batch.step(steps)
        for g in b:
            g.step(steps)
    for x, y in zip(a, b):
        _same(x, y)
    batch.close()


@pytest.mark.parametrize("nx,ny,metric", [(3301, 2203, "plane"), (3329, 2189, "sphere"), (3277, 2311, "stretched")])
def test_grids_by_bands(nx, ny, metric):
    c = _case(nx, ny, metric, nx)
    a, b = _grid(c, cg.TILED), _grid(c, cg.DIRECT)
    for steps in (5, 3):
        a.step(steps)
        b.step(steps)
    _same(a, b)


@pytest.mark.parametrize("along", ["x", "y"])
def test_line_whose_forcing_ends(along):
    n = 600
    rng = np.random.default_rng(4)
    d = 0.3 * rng.uniform(-0.6, 1.0, n)
    d[: n // 3] += 1.5
    d = d.astype(np.float32).astype(np.float64)[None, :]
    h = np.maximum(d + 0.1 * rng.uniform(-0.5, 0.5, (1, n)), 0.0)
    t = np.arange(6) * 1.5
    rec = [0.05 * np.sin(t[:, None, None] + k + np.arange(3)[None, :, None]) for k in range(2)]
    grids = []
    for kind in (cg.TILED, cg.DIRECT):
        kw = dict(ground=0.01, crough=0.000625, dt=0.15)
        if along == "x":
            g = pkg.GpuGrid(d, dx=np.full(n - 1, 10.0), **kw)
            g.set_initial(h)
            g.set_feed(t, west=rec[0], east=rec[1], irec=1, freeze=False)
        else:
            g = pkg.GpuGrid(d.T.copy(), dy=np.full(n - 1, 10.0), **kw)
            g.set_initial(h.T.copy())
            g.set_feed(t, south=rec[0], north=rec[1], irec=1, freeze=False)
        g.set_sweep_kernel(kind)
        for steps in (13, 60, 25):  # forced, past the last record, and on without forcing
            g.step(steps)
        grids.append(g)
    _same(*grids)
