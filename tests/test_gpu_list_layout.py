"""The storage of the neighbour lists (units of 32 items per chunk plane) and
its readers at the edges of a unit span: item counts around multiples of 32,
rows of several chunks.  Every field of the sweeps that read the lists equals
the oracle's bit for bit."""
import numpy as np
import pytest

from prtcl_gb300 import driver
from tests.helpers import assert_bitwise, both_scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,nb", [(1, 1), (31, 33), (32, 32), (33, 31), (64, 1), (97, 65), (1025, 500)])
def test_sweeps_at_unit_edges(oracle_mod, nf, nb):
    # points in a cube of 3 h: rows of up to a few hundred entries
    h = 0.05
    rng = np.random.default_rng(nf * 1000 + nb)
    sc = {"fluid": (rng.random((nf, 3)) * 3.0 * h).astype(np.float32),
          "boundary": (rng.random((nb, 3)) * 3.0 * h).astype(np.float32)}
    p = dict(driver.DAM_BREAK_27K, smoothing_scale=h, viscosity=True)
    d, o = both_scenes(sc, p, oracle_mod)
    v = (rng.standard_normal((nf, 3)) * 0.1).astype(np.float32)
    for m in (d, o):
        m.set_varying("f", "velocity", v)
        m.update()
        m.run("density", "compute_density")
        m.run("iisph", "setup")
        m.set_global("iisph_aprde", 0.0)
        m.run("iisph", "iteration_pressure_acceleration")
        m.run("iisph", "iteration_pressure")
        m.run("iisph", "iteration_pressure_acceleration")
        m.run("wkbb18", "compute_diagonal")
    assert_bitwise(d.get_varying("b", "volume"), o.get_varying("b", "volume", 1), "volume")
    for name, nc in [("density", 1), ("iisph_helper_c", 3), ("iisph_source_term", 1), ("iisph_diagonal_element", 1),
                     ("iisph_right_hand_side", 1), ("pressure", 1), ("acceleration", 3),
                     ("wkbb18_system_diagonal", 9)]:
        assert_bitwise(d.get_varying("f", name, nc), o.get_varying("f", name, nc), name)
