"""The forms of the neighbour walk: every shape of the sweeps (the small-scene
shape, without branches between the entries; the others) gives the same bits,
and those of the oracle, at row lengths around the 8 entries held together, at
smoothing scales inside and outside of the range of the prepared divisors, with
operands that the branch-free divisions pass on to the row's second walk, and
after the smoothing scale changed under the lists."""
import numpy as np
import pytest

from tests.helpers import assert_bitwise, both_scenes
from prtcl_gb300 import driver

pytestmark = pytest.mark.gpu

SWEEPS = ["density", "iisph_setup", "iisph_accel", "iisph_pressure", "wkbb18_diag", "pcg_init", "pcg_q"]
FIELDS = [("density", 1), ("iisph_helper_c", 3), ("iisph_source_term", 1), ("iisph_diagonal_element", 1),
          ("iisph_right_hand_side", 1), ("pressure", 1), ("acceleration", 3), ("wkbb18_system_diagonal", 9)]


def sweeps(m, h2=None):
    m.run("density", "compute_density")
    if h2 is not None:
        m.set_global("smoothing_scale", h2)
        m.run("density", "compute_density")
    m.run("iisph", "setup")
    for _ in range(2):
        m.set_global("iisph_aprde", 0.0)
        m.run("iisph", "iteration_pressure_acceleration")
        m.run("iisph", "iteration_pressure")
    m.run("iisph", "iteration_pressure_acceleration")
    m.run("wkbb18", "compute_diagonal")


def check(oracle_mod, sc, p, v, h2=None):
    d, o = both_scenes(sc, p, oracle_mod)
    first = None
    for m in (d, o):
        m.set_varying("f", "velocity", v)
        m.update()
    for knob in range(4):
        for k in SWEEPS:
            d.model.tune_set(k, knob)
        for m in (d, o) if knob == 0 else (d,):
            m.set_global("smoothing_scale", float(np.float32(p["smoothing_scale"])))
            sweeps(m, h2)
        if knob == 0:
            for name, nc in FIELDS:
                assert_bitwise(d.get_varying("f", name, nc), o.get_varying("f", name, nc), name)
        d.run("wkbb18", "accumulate_acceleration")
        got = [d.get_varying("f", name, nc) for name, nc in FIELDS] + [d.get_varying("f", "wkbb18_velocity_delta", 3)]
        first = first or got
        for a, b in zip(got, first):
            assert_bitwise(a, b, f"shape {knob}")


def cloud(m, h, seed, walls=20):
    rng = np.random.default_rng(seed)
    f = (rng.random((m, 3)) * 2.0 * h).astype(np.float32)
    f = np.concatenate([f, (rng.random((5, 3)) * 2.0 * h + [2.0 * h, 0, 0]).astype(np.float32)])
    b = (rng.random((walls, 3)) * [4.0 * h, 2.0 * h, 2.0 * h]).astype(np.float32)
    return {"fluid": f, "boundary": b}, rng.normal(0.0, 1.0, f.shape).astype(np.float32)


@pytest.mark.parametrize("m", [1, 7, 8, 9, 15, 16, 17, 33, 130])
def test_row_lengths(oracle_mod, m):
    h = 0.05
    sc, v = cloud(m, h, m, walls=m + 3)
    check(oracle_mod, sc, dict(driver.DAM_BREAK_27K, smoothing_scale=h), v)


# below and above 2^-12 and 2^12, and their neighbours inside
@pytest.mark.parametrize("h", [2.0 ** -13, 2.0 ** -12, 0.3, 2.0 ** 12, 2.0 ** 12 * 1.5])
def test_smoothing_scales(oracle_mod, h):
    sc, v = cloud(40, h, 3)
    check(oracle_mod, sc, dict(driver.DAM_BREAK_27K, smoothing_scale=h), v * np.float32(h))


# numerators below 2^-100 (and zero), subnormal ones, and large ones
@pytest.mark.parametrize("speed", [0.0, 1e-25, 1e-38, 1e15])
def test_rows_walked_again(oracle_mod, speed):
    h = 0.05
    sc, v = cloud(40, h, 4)
    check(oracle_mod, sc, dict(driver.DAM_BREAK_27K, smoothing_scale=h), v * np.float32(speed))


def test_smoothing_scale_changed_under_the_lists(oracle_mod):
    h = 0.05
    sc, v = cloud(40, h, 5)
    check(oracle_mod, sc, dict(driver.DAM_BREAK_27K, smoothing_scale=h), v, h2=0.051)


# one item more than the small-scene shape takes
@pytest.mark.parametrize("n", [152 * 4 * 128, 152 * 4 * 128 + 1])
def test_small_scene_limit(oracle_mod, n):
    rng = np.random.default_rng(n)
    h = 0.025
    k = 43
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    f = ((g + 0.2 * rng.random(g.shape)) * h).astype(np.float32)
    b = (rng.random((500, 3)) * [k * h, k * h, 0.1] - [0, 0, 0.11]).astype(np.float32)
    check(oracle_mod, {"fluid": f, "boundary": b}, dict(driver.DAM_BREAK_27K, smoothing_scale=h),
          rng.normal(0.0, 0.1, f.shape).astype(np.float32))
