"""The first Jacobi iteration's zero sums rest on the densities that set-up
found: a replayed graph that computes others between set-up and solve, which
the host does not see, must not be taken for none."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu

FIELDS = [("pressure", 1), ("acceleration", 3), ("iisph_right_hand_side", 1)]


def scene():
    from prtcl_gb300.core import DeviceScene
    sc = scenes.dam_break(fluid_cells=(9, 8, 7), spacing=0.025, box=(0.5, 0.4, 0.3))
    d = DeviceScene()
    driver.setup_dam_break(d, sc, dict(driver.DAM_BREAK_27K, max_iters=1, eta=1e-9))
    d.set_varying("f", "velocity", np.random.default_rng(2).normal(0, 0.3, sc["fluid"].shape).astype(np.float32))
    d.update()
    d.run("density", "compute_density")
    d.run("iisph", "setup")
    d.run("iisph", "solve_pressure")
    return d


@pytest.mark.parametrize("unroll", [1, 2])
@pytest.mark.parametrize("h", [1e30, 0.0])
def test_densities_replayed_between_setup_and_solve(h, unroll):
    """Densities of zero and not-a-number, by a smoothing scale that is there
    for the replay alone."""
    import torch
    eager, graphed = scene(), scene()
    s = torch.cuda.ExternalStream(graphed.model.stream_handle())
    graphed.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
        graphed.run("density", "compute_density")
    own = eager.get_global("smoothing_scale")
    for d in (eager, graphed):
        d.model.tune_set("jacobi_unroll", unroll)
        d.run("density", "compute_density")
        d.run("iisph", "setup")
        d.set_global("smoothing_scale", h)
        if d is eager:
            d.run("density", "compute_density")
        else:
            with torch.cuda.stream(s):
                g.replay()
            d.synchronize()
        d.set_global("smoothing_scale", own)
    for d in (eager, graphed):
        d.run("iisph", "solve_pressure")
    assert not np.isfinite(eager.get_varying("f", "acceleration", 3)).all()
    for name, nc in FIELDS:
        assert_bitwise(graphed.get_varying("f", name, nc), eager.get_varying("f", name, nc), name)
