"""Whole steps in one kernel where most cells take the full wet/dry rules, against
a launch per sweep (CLIFFS_SWEEP_DIRECT): the same bits, at about the same cost.

Land that keeps a remainder: velocities left on cells whose row and column hold
no water stay as they are (cliffs.f:113), step after step, and every such cell
has its column looked through.  A sea floor of random depths, a third of it land:
flooded and drying cells all over.  And a rough beach after a wave."""
import importlib
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
pkg = importlib.import_module("cliffs-src_gb300")
cg = pkg.cliffs_gpu


def _grids(nx, ny, columns):
    """Water in the low quarter, land elsewhere, a velocity on the high quarter's columns."""
    d = np.full((ny, nx), -5.0)
    d[: ny // 2, : nx // 2] = 20.0
    h = np.maximum(d, 0.0)
    u = np.zeros((ny, nx))
    u[ny // 2 + 8:, nx // 2 + 8: nx // 2 + 8 + columns] = 0.1
    u[ny // 2 + 8::3, nx // 4] = 0.2  # and one column whose remainders the next y-sweep clears
    out = []
    for kind in (cg.TILED, cg.DIRECT):
        g = pkg.GpuGrid(d, dx=np.full(nx - 1, 100.0), dy=np.full(ny - 1, 100.0), ground=0.05, crough=0.0, dt=1.0)
        g.set_initial(h, u, np.zeros_like(u))
        g.set_sweep_kernel(kind)
        out.append(g)
    return out


@pytest.mark.parametrize("nx,ny", [(61, 73), (512, 500), (1300, 320), (1700, 800)])
def test_remainders_match_sweeps(nx, ny):
    a, b = _grids(nx, ny, nx)
    for steps in (3, 4, 2):
        a.step(steps)
        b.step(steps)
    for x, y in zip((*a.download_state(), *a.maxwave()), (*b.download_state(), *b.maxwave())):
        assert np.array_equal(x, y)
    assert a.status() == b.status()
    assert np.count_nonzero(a.download_state()[1][ny // 2 + 8:, nx // 2 + 8:]) > 0  # they were kept


def _step_time(g):
    t = []
    g.step(9)
    for _ in range(7):
        g.sync()
        t0 = time.perf_counter()
        g.step(16)
        g.sync()
        t.append(time.perf_counter() - t0)
    return sorted(t)[3]


def test_remainders_cost_no_more_than_sweeps():
    """At most half as much again as a launch per sweep (a scan for each cell: four times as much)."""
    took = [_step_time(g) for g in _grids(512, 512, 512)]
    assert took[0] <= 1.5 * took[1], took


@pytest.mark.parametrize("nx,ny", [(1003, 777), (2048, 1100)])
def test_rough_floors_cost_no_more_than_sweeps(nx, ny):
    """At most two fifths more than a launch per sweep (with flooded cells taken as they come: about twice)."""
    rng = np.random.default_rng(1)
    d = 0.3 * rng.uniform(-0.6, 1.0, (ny, nx))
    d[:, : nx // 3] += 1.5
    d = d.astype(np.float32).astype(np.float64)
    h = np.maximum(d + 0.1 * rng.uniform(-0.5, 0.5, (ny, nx)), 0.0)
    took, state = [], []
    for kind in (cg.TILED, cg.DIRECT):
        g = pkg.GpuGrid(d, dx=np.full(nx - 1, 10.0), dy=np.full(ny - 1, 10.0), ground=0.01, crough=0.000625, dt=0.15)
        g.set_initial(h)
        g.set_sweep_kernel(kind)
        took.append(_step_time(g))
        state.append(g.download_state())
    assert all(np.array_equal(x, y) for x, y in zip(*state))
    assert took[0] <= 1.4 * took[1], took


def test_runup_on_a_rough_beach_costs_no_more_than_sweeps():
    """0.5 m of noise on a 1:100 slope, while the wave is on the beach and as it leaves: at most a twentieth more
    than a launch per sweep (with a column looked through for every remainder: up to a seventh)."""
    nx = ny = 600
    rng = np.random.default_rng(0)
    x = np.arange(nx)[None, :]
    d = np.clip(0.9 * nx - x, -5.0, 200.0) + 0.5 * rng.standard_normal((ny, nx))
    d = d.astype(np.float32).astype(np.float64)
    h = np.where(d > 0, d + np.exp(-(((x - nx / 2) / 20.0) ** 2)), 0.0)
    took, state = [], []
    for kind in (cg.TILED, cg.DIRECT):
        g = pkg.GpuGrid(d, dx=np.full(nx - 1, 100.0), dy=np.full(ny - 1, 100.0), ground=0.05, crough=0.000625, dt=1.5)
        g.set_initial(h)
        g.set_sweep_kernel(kind)
        g.step(1089)
        took.append(_step_time(g))
        state.append(g.download_state())
    assert all(np.array_equal(x, y) for x, y in zip(*state))
    assert took[0] <= 1.05 * took[1], took
