"""integrate_position writes the sweeps' packed records with the positions and
raises the maximum speed in place: fields and maximum equal the oracle's, with
masses that change before and after, and whatever the maximum starts from."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise, both_scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("start", [-3.0, -0.0, 0.0, 0.5, 1e9, float("nan"), float("inf")])
@pytest.mark.parametrize("mass", ["same", "before", "after"])
def test_integrate_then_density(oracle_mod, start, mass):
    sc = scenes.dam_break(fluid_cells=(9, 8, 7), spacing=0.025, box=(0.5, 0.4, 0.3))
    d, o = both_scenes(sc, dict(driver.DAM_BREAK_27K), oracle_mod)
    rng = np.random.default_rng(1)
    n = len(sc["fluid"])
    v = rng.normal(0, 0.3, (n, 3)).astype(np.float32)
    m2 = (d.get_varying("f", "mass") * rng.uniform(0.5, 2.0, n)).astype(np.float32)
    for s in (d, o):
        s.set_varying("f", "velocity", v)
        s.update()
        s.run("density", "compute_density")
        s.set_global("maximum_speed", start)
        if mass == "before":
            s.set_varying("f", "mass", m2)
        s.run("symplectic_euler", "integrate_position")
        if mass == "after":
            s.set_varying("f", "mass", m2)
        s.update()
        s.run("density", "compute_density")
        s.run("symplectic_euler", "integrate_position")
        s.update()
        s.run("density", "compute_density")
    assert_bitwise(d.get_varying("f", "position", 3), o.get_varying("f", "position", 3), "position")
    assert_bitwise(d.get_varying("f", "density"), o.get_varying("f", "density", 1), "density")
    got, want = d.get_global("maximum_speed"), o.get_global("maximum_speed")
    if not np.isnan(start):
        assert got == want


@pytest.mark.parametrize("n", [39_990, 40_000, 40_001])
def test_adjacent_cells_at_the_limit(n):
    """A warp per cell up to 40,000 items of the grid, a thread per cell above."""
    from prtcl_gb300.core import DeviceScene
    from tests.helpers import point_scene
    rng = np.random.default_rng(n)
    x = (rng.random((n, 3)) * 2.0 - 0.7).astype(np.float32)
    rows = []
    for knob in (0, 1):
        d = DeviceScene()
        point_scene(d, [("p", "fluid", x, [])], 0.06)
        d.model.tune_set("grid_sort", knob)
        for _ in range(2):
            d.update()
        rows.append(d.nhood.neighbor_lists(0, 0, n))
    assert_bitwise(rows[1][0], rows[0][0], "offsets")
    assert_bitwise(rows[1][1], rows[0][1], "indices")
