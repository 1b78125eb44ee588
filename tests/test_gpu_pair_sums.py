"""Sums taken two at a time (PCG's r.r and r.y, and b.b beside them) keep the
trees of the single ones: a scene alone in a batch, whose tiles of 128 items
sum in warps of 32, and the plain path agree as they did, and the velocity
change is the oracle's at item counts around a warp and a block."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import both_scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 2000])
def test_velocity_change_matches_the_oracle(oracle_mod, n):
    k = max(2, int(np.ceil(n ** (1 / 3))))
    sc = scenes.dam_break(fluid_cells=(k, k, k), spacing=0.025, box=(k * 0.03, k * 0.03, k * 0.03))
    sc["fluid"] = np.ascontiguousarray(sc["fluid"][:n])
    d, o = both_scenes(sc, dict(driver.DAM_BREAK_27K, viscosity=True), oracle_mod)
    v = np.random.default_rng(n).normal(0, 0.3, (n, 3)).astype(np.float32)
    for s in (d, o):
        s.set_varying("f", "velocity", v)
        s.update()
        s.run("density", "compute_density")
        s.run("wkbb18", "compute_diagonal")
        s.run("wkbb18", "accumulate_acceleration")
    # (the sums' trees differ from the oracle's order: alpha and beta may round
    # to the next float now and then)
    a, b = d.get_varying("f", "wkbb18_velocity_delta", 3), o.get_varying("f", "wkbb18_velocity_delta", 3)
    scale = float(np.abs(b).max()) or 1.0
    assert float(np.abs(a - b).max()) <= 1e-5 * scale
    assert d.get_uniform("f", "wkbb18_iterations") == o.get_uniform("f", "wkbb18_iterations")
