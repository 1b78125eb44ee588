"""The cell-tile product (pcg_q 4) reads raw -> sorted, which is made where a
reader asks for it: a solve whose launches went into a capture, whether that
takes them or not, made nothing, and the solve after it makes it."""
import ctypes

import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu


def test_solve_after_a_captured_one():
    from prtcl_gb300 import _lib
    from prtcl_gb300.core import DeviceScene
    sc = scenes.dam_break(fluid_cells=(12, 11, 10), spacing=0.025, box=(0.5, 0.4, 0.3))
    v = np.random.default_rng(3).normal(0, 0.3, sc["fluid"].shape).astype(np.float32)
    d = DeviceScene()
    driver.setup_dam_break(d, sc, dict(driver.DAM_BREAK_27K, viscosity=True))
    d.set_varying("f", "velocity", v)

    def solve(knob):
        d.model.tune_set("pcg_q", knob)
        d.run("wkbb18", "accumulate_acceleration")

    def prepare():
        d.update()
        d.run("density", "compute_density")
        d.run("wkbb18", "compute_diagonal")

    prepare()
    solve(0)
    want = d.get_varying("f", "wkbb18_velocity_delta", 3)
    prepare()
    d.synchronize()
    cu = ctypes.CDLL("libcuda.so.1")
    stream, graph = ctypes.c_void_p(d.model.stream_handle()), ctypes.c_void_p()
    assert cu.cuStreamBeginCapture_v2(stream, 2) == 0  # relaxed
    try:
        solve(4)
    except _lib.PrtclGpuError:
        pass
    cu.cuStreamEndCapture(stream, ctypes.byref(graph))
    if graph.value:
        cu.cuGraphDestroy(graph)
    try:
        solve(4)  # (a refused launch's error shows up in the next check of the launches too)
    except _lib.PrtclGpuError:
        solve(4)
    assert_bitwise(d.get_varying("f", "wkbb18_velocity_delta", 3), want)
