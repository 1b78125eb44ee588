"""The PCG loop of a small scene as one cooperative launch gives the velocity
change, the acceleration and the iteration count of the launches one by one
(driven from the host, as with profiling on), with and without gradient correction, at item
counts around a block and at the largest it takes, up to the iteration cap."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu


def scene(n, **params):
    from prtcl_gb300.core import DeviceScene
    k = max(2, int(np.ceil(n ** (1 / 3))))
    sc = scenes.dam_break(fluid_cells=(k, k, k), spacing=0.025, box=(k * 0.03, k * 0.03, k * 0.03))
    sc["fluid"] = np.ascontiguousarray(sc["fluid"][:n])
    d = DeviceScene()
    driver.setup_dam_break(d, sc, dict(driver.DAM_BREAK_27K, **{"viscosity": True, **params}))
    rng = np.random.default_rng(n)
    d.set_varying("f", "position", (sc["fluid"] + rng.normal(0, 5e-4, (n, 3))).astype(np.float32))
    d.set_varying("f", "velocity", rng.normal(0, 0.3, (n, 3)).astype(np.float32))
    d.update()
    d.run("density", "compute_density")
    return d


def solve(d, scheme, singly):
    d.run(scheme, "compute_diagonal")
    d.model.profile(singly)
    d.run(scheme, "accumulate_acceleration")
    d.model.profile(False)
    return ([d.get_varying("f", "wkbb18_velocity_delta", 3), d.get_varying("f", "acceleration", 3)],
            d.get_uniform("f", "wkbb18_iterations"))


def check(d, gc, iterations=None):
    if gc:
        d.scheme("correction")
        d.scheme("wkbb18_gc")
        d.run("correction", "compute_gradient_correction")
    scheme = "wkbb18_gc" if gc else "wkbb18"
    a, b = solve(d, scheme, False), solve(d, scheme, True)
    for x, y in zip(a[0], b[0]):
        assert_bitwise(x, y)
    assert a[1] == b[1] >= 0
    if iterations is not None:
        assert a[1] == iterations


@pytest.mark.parametrize("gc", [False, True])
@pytest.mark.parametrize("n", [1, 127, 128, 129, 5003, 152 * 4 * 128, 152 * 4 * 128 + 1])
def test_one_launch_matches_the_launches(n, gc):
    check(scene(n), gc)


@pytest.mark.parametrize("gc", [False, True])
@pytest.mark.parametrize("cap", [0, 1, 7])
def test_iteration_cap(gc, cap):
    check(scene(3000, wkbb18_maximum_iterations=cap, wkbb18_maximum_error=1e-9), gc)


@pytest.mark.parametrize("gc", [False, True])
def test_at_rest(gc):
    d = scene(700)
    d.set_varying("f", "velocity", np.zeros((700, 3), np.float32))
    check(d, gc)
