"""The kernel and bytes that the ensemble's bench line names follow the plan that
its autotuner kept."""
import importlib
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
bench = importlib.import_module("bench")
cg = importlib.import_module("cliffs-src_gb300").cliffs_gpu


@pytest.mark.parametrize("mode,x_rows,y_groups,whole", [
    (cg.GRAPH, 1, 1, True), (cg.GRAPH, 0, 0, True), (cg.GRAPH, 2, 1, False), (cg.GRAPH, 1, 4, False),
    (cg.PERSISTENT, 1, 1, False)])
def test_kernel_and_bytes_of_a_plan(mode, x_rows, y_groups, whole):
    name, per_cell = bench.batch_step_kernel(dict(mode=mode, ctas_per_sm=1, graph_steps=32, x_rows=x_rows,
                                                  y_groups=y_groups))
    assert ("batch_step_kernel" in name) == whole
    assert per_cell == (44 if whole else 72)
