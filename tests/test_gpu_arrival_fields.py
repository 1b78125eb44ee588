"""What a scene's arrival in a batch writes beside positions and masses: its
time of birth, one second before it came, and (by the densities that rest on
them) its walls; and integrate_position leaves a maximum speed that is not a
number as it is."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise
from tests.test_gpu_batch_arrival import P, scene

pytestmark = pytest.mark.gpu


def test_time_of_birth_and_walls():
    from prtcl_gb300.batch import Batch
    sizes = [(300, 200), (1, 40), (257, 0), (64, 300)]
    dt, t = float(np.float32(P["time_step"])), 0.0
    bt, ids, born = Batch(P), [], []
    for k, (nf, nb) in enumerate(sizes):
        ids.append(bt.add_scene(*scene(nf, nb, k)))
        born.append(np.float32(np.float32(t) - np.float32(1.0)))
        bt.step(k + 1)
        for _ in range(k + 1):
            t += dt
    for k, (nf, nb) in enumerate(sizes):
        assert_bitwise(bt.download(ids[k], "time_of_birth"), np.full(nf, born[k], np.float32), f"scene {k}")
        alone = Batch(P)
        i = alone.add_scene(*scene(nf, nb, k))
        alone.step(sum(range(k + 1, len(sizes) + 1)))
        for name in ("density", "velocity", "position"):
            assert_bitwise(bt.download(ids[k], name), alone.download(i, name), f"scene {k} {name}")


def test_maximum_speed_not_a_number():
    from prtcl_gb300.core import DeviceScene
    sc = scenes.dam_break(fluid_cells=(9, 8, 7), spacing=0.025, box=(0.5, 0.4, 0.3))
    d = DeviceScene()
    driver.setup_dam_break(d, sc, dict(driver.DAM_BREAK_27K))
    d.set_varying("f", "velocity", np.full(sc["fluid"].shape, 0.5, np.float32))
    d.set_global("maximum_speed", float("nan"))
    d.run("symplectic_euler", "integrate_position")
    assert np.isnan(d.get_global("maximum_speed"))
    d.set_global("maximum_speed", 0.0)
    d.run("symplectic_euler", "integrate_position")
    assert d.get_global("maximum_speed") == np.float32(np.sqrt(np.float32(0.75)))
