"""Many items that were not permuted take another walk in the density and the
diagonal: the same items in the same order, once uploaded in it and once
permuted into it (which moves none), give the same bits, at the least such
count, one item fewer and a ragged one."""
import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu

FIELDS = [("density", 1), ("wkbb18_system_diagonal", 9), ("acceleration", 3)]


@pytest.mark.parametrize("gc", [False, True])
@pytest.mark.parametrize("n", [499_999, 500_000, 500_077])
def test_both_walks(n, gc):
    from prtcl_gb300.core import DeviceScene
    sc = scenes.dam_break(fluid_cells=(80, 80, 79), spacing=0.025, box=(2.1, 2.1, 2.1))
    rng = np.random.default_rng(n)
    sc["fluid"] = (sc["fluid"][:n] + rng.normal(0, 2e-3, (n, 3))).astype(np.float32)
    v = rng.normal(0, 0.3, (n, 3)).astype(np.float32)
    wkbb18 = "wkbb18_gc" if gc else "wkbb18"

    def scene(x):
        d = DeviceScene()
        driver.setup_dam_break(d, dict(sc, fluid=sc["fluid"][:1]), dict(driver.DAM_BREAK_27K, viscosity=True))
        mass = d.get_varying("f", "mass")[0]
        for name in ("viscosity", "correction", wkbb18):
            d.scheme(name)
        d.resize("f", n)
        d.set_varying("f", "position", x)
        d.set_varying("f", "velocity", v)
        d.set_varying("f", "mass", np.full(n, mass, np.float32))
        d.update()
        return d

    def sweep(d):
        d.run("density", "compute_density")
        if gc:
            d.run("correction", "compute_gradient_correction")
        d.run(wkbb18, "compute_diagonal")
        d.run("gravity", "initialize_acceleration")
        d.run("viscosity", "accumulate_acceleration")
        return [d.get_varying("f", name, nc) for name, nc in FIELDS]

    first = scene(sc["fluid"])
    first.permute()
    x = first.get_varying("f", "position", 3)
    uploaded, permuted = scene(x), scene(x)
    permuted.permute()
    assert_bitwise(permuted.get_varying("f", "position", 3), x)
    for a, b, (name, _) in zip(sweep(uploaded), sweep(permuted), FIELDS):
        assert np.isfinite(a).all()
        assert_bitwise(a, b, name)
