"""The first Jacobi iteration's zero sums rest on the pressure that set-up
wrote: a captured graph that runs an iteration between set-up and solve, which
the host does not see, must not be taken for none."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu

FIELDS = [("pressure", 1), ("acceleration", 3), ("iisph_right_hand_side", 1)]


def prepared():
    from prtcl_gb300.core import DeviceScene
    sc = scenes.dam_break(fluid_cells=(9, 8, 7), spacing=0.025, box=(0.5, 0.4, 0.3))
    d = DeviceScene()
    driver.setup_dam_break(d, sc, dict(driver.DAM_BREAK_27K, max_iters=3, eta=1e-9))
    v = np.random.default_rng(2).normal(0, 0.3, sc["fluid"].shape).astype(np.float32)
    d.set_varying("f", "velocity", v)
    d.update()
    d.run("density", "compute_density")
    d.run("iisph", "setup")
    iteration(d)
    return d


def iteration(d):
    d.run("iisph", "iteration_pressure_acceleration")
    d.run("iisph", "iteration_pressure")


def test_captured_iteration_between_setup_and_solve():
    import torch
    eager, graphed = prepared(), prepared()
    s = torch.cuda.ExternalStream(graphed.model.stream_handle())
    graphed.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        iteration(graphed)
    for d in (eager, graphed):
        d.run("iisph", "setup")
    iteration(eager)
    with torch.cuda.stream(s):
        g.replay()
    for d in (eager, graphed):
        d.run("iisph", "solve_pressure")
    for name, nc in FIELDS:
        assert_bitwise(graphed.get_varying("f", name, nc), eager.get_varying("f", name, nc), name)
