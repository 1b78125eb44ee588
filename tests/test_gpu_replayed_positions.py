"""Positions that a replayed graph moves after a grid's update are the ones that
the lists see, as with the procedure called."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu


def scene():
    from prtcl_gb300.core import DeviceScene
    sc = scenes.dam_break(fluid_cells=(9, 8, 7), spacing=0.025, box=(0.5, 0.4, 0.3))
    d = DeviceScene()
    driver.setup_dam_break(d, sc, dict(driver.DAM_BREAK_27K, time_step=0.02))
    d.set_varying("f", "velocity", np.random.default_rng(2).normal(0, 0.3, sc["fluid"].shape).astype(np.float32))
    d.update()
    d.run("density", "compute_density")
    d.run("symplectic_euler", "integrate_position")
    return d


@pytest.mark.parametrize("list_split", [0, 1])
def test_lists_after_a_replay(list_split):
    import torch
    eager, graphed = scene(), scene()
    s = torch.cuda.ExternalStream(graphed.model.stream_handle())
    graphed.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        graphed.run("symplectic_euler", "integrate_position")
    for d in (eager, graphed):
        d.model.tune_set("list_split", list_split)
        d.update()
    eager.run("symplectic_euler", "integrate_position")
    with torch.cuda.stream(s):
        g.replay()
    for d in (eager, graphed):
        d.run("density", "compute_density")
    n = len(eager.get_varying("f", "density"))
    for name, nc in (("position", 3), ("density", 1)):
        assert_bitwise(graphed.get_varying("f", name, nc), eager.get_varying("f", name, nc), name)
    for k in range(2):
        a, b = graphed.nhood.neighbor_lists(1, k, n), eager.nhood.neighbor_lists(1, k, n)
        assert_bitwise(a[0], b[0], "offsets")
        assert_bitwise(a[1], b[1], "indices")
