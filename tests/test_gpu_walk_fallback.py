"""Rows that the branch-free walk does not take: densities and volumes at
smoothing scales outside of the prepared divisors, accelerations and pressures
after the scale changed under the lists, explicit viscosity where every row
divides below 2^-40, at row lengths around 8 and 16 entries.  Fields equal the
oracle's."""
import numpy as np
import pytest

from prtcl_gb300 import driver
from tests.helpers import assert_bitwise, both_scenes
from tests.test_gpu_walk_forms import cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16, 17, 130])
@pytest.mark.parametrize("h,h2", [(5e-6, None), (2.0 ** -13, None), (0.05, 0.051), (2.0 ** 12 * 1.5, None)])
def test_fields(oracle_mod, m, h, h2):
    sc, v = cloud(m, h, m, walls=m + 3)
    d, o = both_scenes(sc, dict(driver.DAM_BREAK_27K, smoothing_scale=h), oracle_mod)
    for s in (d, o):
        if s is d:
            s.scheme("viscosity")
        s.set_varying("f", "velocity", (v * np.float32(h)).astype(np.float32))
        s.update()
        s.run("aiast12", "compute_volume")
        s.run("density", "compute_density")
        if h2 is not None:
            s.set_global("smoothing_scale", h2)
        s.run("iisph", "setup")
        for _ in range(2):
            s.set_global("iisph_aprde", 0.0)
            s.run("iisph", "iteration_pressure_acceleration")
            s.run("iisph", "iteration_pressure")
        s.run("gravity", "initialize_acceleration")
        s.run("viscosity", "accumulate_acceleration")
    assert_bitwise(d.get_varying("b", "volume"), o.get_varying("b", "volume", 1), "volume")
    for name, nc in (("density", 1), ("pressure", 1), ("iisph_right_hand_side", 1), ("acceleration", 3)):
        assert_bitwise(d.get_varying("f", name, nc), o.get_varying("f", name, nc), name)
