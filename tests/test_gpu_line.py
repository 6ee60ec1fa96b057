"""Many steps of a one-dimensional grid in one launch (line_kernel, a cluster
of blocks that holds the line in shared memory) against a launch per sweep
(CLIFFS_SWEEP_DIRECT): bit-identical states, max-wave fields and status.

Lines along x and y of sizes around the blocks' and the cluster's (one block up
to 252 cells, two up to 504, four up to 1008, eight beyond; 7648 at most), with
a rough bed of ponds and islands across all block edges, uniform and stretched
spacing, a row factor, a metric term, and a passive second line.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
pkg = importlib.import_module("cliffs-src_gb300")
cg = pkg.cliffs_gpu


def _grids(n, along, lines, stretched, metric, seed=None, depth=0.0):
    rng = np.random.default_rng(n if seed is None else seed)
    d = 0.3 * rng.uniform(-0.6, 1.0, (lines, n)) + depth
    d[:, : n // 3] += 1.5
    d = d.astype(np.float32).astype(np.float64)
    h = np.maximum(d + 0.1 * rng.uniform(-0.5, 0.5, (lines, n)), 0.0)
    dx = rng.uniform(8.0, 12.0, n - 1) if stretched else np.full(n - 1, 10.0)
    kw = dict(ground=0.01, crough=0.000625, dt=0.15)
    if along == "x":
        kw.update(dx=dx, row_scale=np.full(lines, 0.8) if metric else None)
    else:
        d, h = d.T.copy(), h.T.copy()
        kw.update(dy=dx, zeta=1e-4 * np.sin(np.arange(n)) if metric else None)
    out = []
    for kind in (cg.TILED, cg.DIRECT):
        g = pkg.GpuGrid(d, **kw)
        g.set_initial(h)
        g.set_sweep_kernel(kind)
        out.append(g)
    return out


def _same(a, b):
    for x, y in zip((*a.download_state(), *a.maxwave()), (*b.download_state(), *b.maxwave())):
        assert np.array_equal(x, y)
    assert a.status() == b.status() and a.courant() == b.courant()
    assert np.isfinite(a.download_state()[0]).all()


@pytest.mark.parametrize("n", [3, 4, 31, 252, 253, 504, 505, 1008, 1009, 2000, 2017, 6001, 7648, 7649])
@pytest.mark.parametrize("along", ["x", "y"])
def test_line_matches_sweeps(n, along):
    a, b = _grids(n, along, 1, n % 2 == 1, n % 3 == 0)
    for steps in (1, 40, 7):
        a.step(steps)
        b.step(steps)
    _same(a, b)


@pytest.mark.parametrize("along", ["x", "y"])
def test_passive_second_line(along):
    a, b = _grids(300, along, 2, False, True)
    for g in (a, b):
        g.step(25)
    _same(a, b)


@pytest.mark.parametrize("depth", [-1.0, -0.35])
def test_drying_line(depth):
    """Little or no water: lines that fall dry, remainders far from any wet cell."""
    a, b = _grids(700, "x", 1, False, False, seed=5, depth=depth)
    for _ in range(20):
        a.step(9)
        b.step(9)
    _same(a, b)


def test_turns_between_line_and_sweeps():
    """Single sweeps, sources and uploads between the launches."""
    a, b = _grids(600, "x", 1, False, False)
    x = np.arange(600) * 10.0
    for g in (a, b):
        g.step(11)
        g.sweep(1)
        g.step(5)
        g.add_source(x, np.zeros(1), x0=900.0, y0=0.0, ax=300.0, ay=50.0, amp=0.1, rise_time=1.0)
        g.step(30)
        cel, u, v = g.download_state()
        g.upload_state(cel, 0.9 * u, v)
        g.step(12)
    _same(a, b)
