"""The Courant check of the line ends where one axis is uniform and the other
stretched: whole steps read both axes' geometry from tables there, and a uniform
axis counts its end cells as it does in a launch per sweep.  One column (row) of
deep still water at each end is the only place with a number above 1."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
pkg = importlib.import_module("cliffs-src_gb300")
cg = pkg.cliffs_gpu


@pytest.mark.parametrize("uniform", ["x", "y"])
@pytest.mark.parametrize("nx,ny", [(50, 40), (900, 700), (1700, 800)])  # each of the tiles
def test_ends_of_a_uniform_axis_are_counted(nx, ny, uniform):
    rng = np.random.default_rng(nx)
    d = np.full((ny, nx), 0.5)
    if uniform == "x":
        d[:, [0, -1]] = 500.0  # 70 m/s: 1.05 at 10 m and 0.15 s
    else:
        d[[0, -1]] = 500.0
    dx = np.full(nx - 1, 10.0) if uniform == "x" else rng.uniform(11.0, 12.0, nx - 1)
    dy = np.full(ny - 1, 10.0) if uniform == "y" else rng.uniform(11.0, 12.0, ny - 1)
    seen = []
    for kind in (cg.TILED, cg.DIRECT):
        g = pkg.GpuGrid(d, dx=dx, dy=dy, ground=0.01, crough=0.0, dt=0.15)
        g.set_initial(d)
        g.set_sweep_kernel(kind)
        g.step(1)  # a fresh state's first step runs a launch per sweep
        assert g.status()[1] != 0 and g.status()[1] == 0  # told once
        g.step(2)
        seen.append((g.status(), g.courant(), g.download_state()))
    assert seen[0][0][1] != 0
    assert seen[0][0] == seen[1][0] and seen[0][1] == seen[1][1] > 1.0
    for x, y in zip(seen[0][2], seen[1][2]):
        assert np.array_equal(x, y)
