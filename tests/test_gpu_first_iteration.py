"""The relaxed-Jacobi loop takes zero sums in the first iteration after a
set-up (p = 0).  The loop as one procedure must give the fields of the
iteration procedures driven from the host, which take every iteration in
full, bit for bit: also where masses, volumes or densities are not finite,
and where something changed between set-up and solve."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from prtcl_gb300.core import DeviceScene

pytestmark = pytest.mark.gpu

FIELDS = [("acceleration", 3), ("pressure", 1), ("iisph_right_hand_side", 1)]


def scene(seed, change):
    sc = scenes.dam_break(fluid_cells=(9, 8, 7), spacing=0.025, box=(0.5, 0.4, 0.3))
    p = dict(driver.DAM_BREAK_27K, max_iters=7, eta=1e-3)
    d = DeviceScene()
    driver.setup_dam_break(d, sc, p)
    rng = np.random.default_rng(seed)
    n, nb = len(sc["fluid"]), len(sc["boundary"])
    x = d.get_varying("f", "position")
    d.set_varying("f", "position", (x + rng.normal(0, 2e-4, x.shape)).astype(np.float32))
    d.set_varying("f", "velocity", rng.normal(0, 0.2, (n, 3)).astype(np.float32))
    m, V = d.get_varying("f", "mass"), d.get_varying("b", "volume")
    if change == "mass_inf":
        m[n // 2] = np.inf
    if change == "mass_nan":
        m[3] = np.nan
    if change == "mass_zero":
        m[::5] = 0.0
    if change == "mass_negative":
        m[::7] *= -1.0
    if change == "volume_inf":
        V[nb // 3] = np.inf
    if change == "isolated":
        x[0] = (0.45, 0.35, 0.25)
        d.set_varying("f", "position", x)
    d.set_varying("f", "mass", m)
    d.set_varying("b", "volume", V)
    d.update()
    d.run("density", "compute_density")
    rho = d.get_varying("f", "density")
    if change == "density_zero":
        rho[n // 3] = 0.0
    if change == "density_inf":
        rho[n // 3] = np.inf
    if change == "density_nan":
        rho[n // 3] = np.nan
    if change.startswith("density_"):
        d.set_varying("f", "density", rho)
    d.run("iisph", "setup")
    if change == "pressure_after":
        d.set_varying("f", "pressure", rng.random(n).astype(np.float32) * 1000)
    if change == "mass_after":
        m[n // 2] = np.inf
        d.set_varying("f", "mass", m)
    if change == "h_after":
        d.set_global("smoothing_scale", float(np.float32(0.03)))
    if change == "rho0_after":
        d.set_uniform("f", "rest_density", float("inf"))
    if change == "radius_after":
        d.set_radius(0.07)
        d.update()
    if change == "cap_1":
        d.set_global("iisph_maximum_iterations", 1)
    return d


def host_loop(d, cap, eta):
    nprde = d.get_global("iisph_nprde")
    for it in range(1, cap + 1):
        d.set_global("iisph_aprde", 0.0)
        d.run("iisph", "iteration_pressure_acceleration")
        d.run("iisph", "iteration_pressure")
        if it >= 2 and d.get_global("iisph_aprde") / nprde < eta:
            break
    return it


@pytest.mark.parametrize("change", ["", "mass_inf", "mass_nan", "mass_zero", "mass_negative", "volume_inf", "isolated",
                                    "density_zero", "density_inf", "density_nan", "pressure_after", "mass_after",
                                    "h_after", "rho0_after", "radius_after", "cap_1"])
def test_loop_equals_full_iterations(change):
    a, b = scene(5, change), scene(5, change)
    a.run("iisph", "solve_pressure")
    it = host_loop(b, 1 if change == "cap_1" else 7, np.float32(1e-3))
    assert a.get_global("iisph_iterations") == it
    for name, nc in FIELDS:
        u, v = a.get_varying("f", name, nc).view(np.uint32), b.get_varying("f", name, nc).view(np.uint32)
        assert np.array_equal(u, v), (name, np.count_nonzero(u != v))


def test_second_solve_starts_from_the_first():
    a, b = scene(6, ""), scene(6, "")
    for _ in range(2):
        a.run("iisph", "solve_pressure")
        host_loop(b, 7, np.float32(1e-3))
        for name, nc in FIELDS:
            u, v = a.get_varying("f", name, nc).view(np.uint32), b.get_varying("f", name, nc).view(np.uint32)
            assert np.array_equal(u, v), name
