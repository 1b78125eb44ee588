"""The first Jacobi iteration's zero sums where rest density times volume
overflows, with densities of set-up's sums finite and not: the fields of the
iteration in full (taken where the pressure was written again)."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu

FIELDS = [("pressure", 1), ("acceleration", 3), ("iisph_right_hand_side", 1)]


@pytest.mark.parametrize("density", ["computed", "set"])
@pytest.mark.parametrize("volume", [1e30, 3e35, 4e35, 1e36])  # 3.4e38 / 1000 lies between
def test_large_volumes(volume, density):
    from prtcl_gb300.core import DeviceScene
    sc = scenes.dam_break(fluid_cells=(6, 6, 6), spacing=0.025, box=(0.2, 0.2, 0.2))
    n, nb = len(sc["fluid"]), len(sc["boundary"])
    d = DeviceScene()
    driver.setup_dam_break(d, sc, dict(driver.DAM_BREAK_27K, max_iters=1))
    d.set_varying("b", "volume", np.full(nb, volume, np.float32))
    d.update()
    d.run("density", "compute_density")
    if density == "set":
        d.set_varying("f", "density", np.full(n, 1000.0, np.float32))
    got = []
    for written_again in (False, True):
        d.run("iisph", "setup")
        if written_again:
            d.set_varying("f", "pressure", d.get_varying("f", "pressure"))
        d.run("iisph", "solve_pressure")
        got.append([d.get_varying("f", name, nc) for name, nc in FIELDS])
    for a, b, (name, _) in zip(*got, FIELDS):
        assert_bitwise(a, b, name)
