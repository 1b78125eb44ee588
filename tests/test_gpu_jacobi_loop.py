"""The relaxed-Jacobi loop of a small scene as one cooperative launch gives the
fields, the iteration count and the statistics of the launches sweep by sweep
(taken with a repeat count of 2), at item counts around a block and at the
largest it takes, up to the iteration cap, with nothing to iterate, and with
two models solving at the same time."""
import threading

import numpy as np
import pytest

from prtcl_gb300 import driver, scenes
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu

FIELDS = [("pressure", 1), ("acceleration", 3), ("iisph_right_hand_side", 1)]


def scene(n, seed, **params):
    from prtcl_gb300.core import DeviceScene
    k = max(2, int(np.ceil(n ** (1 / 3))))
    sc = scenes.dam_break(fluid_cells=(k, k, k), spacing=0.025, box=(k * 0.03, k * 0.03, k * 0.03))
    sc["fluid"] = np.ascontiguousarray(sc["fluid"][:n])
    d = DeviceScene()
    driver.setup_dam_break(d, sc, dict(driver.DAM_BREAK_27K, **params))
    rng = np.random.default_rng(seed)
    d.set_varying("f", "position", (sc["fluid"] + rng.normal(0, 5e-4, (n, 3))).astype(np.float32))
    d.set_varying("f", "velocity", rng.normal(0, 0.3, (n, 3)).astype(np.float32))
    d.update()
    d.run("density", "compute_density")
    return d


def solve(d, unroll, again=False):
    d.model.tune_set("jacobi_unroll", unroll)
    d.run("iisph", "setup")
    d.run("iisph", "solve_pressure")
    if again:  # from the pressure that is there: no zero sums
        d.run("iisph", "solve_pressure")
    out = [d.get_varying("f", name, nc) for name, nc in FIELDS]
    return out, d.get_global("iisph_iterations"), d.get_global("iisph_aprde")


def same(a, b):
    for x, y in zip(a[0], b[0]):
        assert_bitwise(x, y)
    assert a[1] == b[1] and a[2] == b[2]
    assert a[1] >= 0


@pytest.mark.parametrize("n", [1, 127, 128, 129, 5003, 152 * 4 * 128, 152 * 4 * 128 + 1])
@pytest.mark.parametrize("again", [False, True])
def test_one_launch_matches_the_sweeps(n, again):
    d = scene(n, n)
    same(solve(d, 1, again), solve(d, 2, again))


@pytest.mark.parametrize("params", [dict(max_iters=1), dict(max_iters=9, eta=1e-9), dict(eta=10.0)])
def test_ends(params):
    d = scene(3000, 7, **params)
    same(solve(d, 1), solve(d, 2))


def test_nothing_to_iterate():
    d = scene(300, 8)
    d.run("iisph", "setup")
    before = d.get_varying("f", "pressure")
    d.set_global("iisph_nprde", 0)
    d.run("iisph", "solve_pressure")
    assert d.get_global("iisph_iterations") == 0
    assert_bitwise(d.get_varying("f", "pressure"), before)


def test_two_models_at_the_same_time():
    ds = [scene(27_000, k, max_iters=20, eta=1e-9) for k in (1, 2)]
    want = [solve(d, 2) for d in ds]
    got = [None, None]

    def work(k):
        for _ in range(10):
            got[k] = solve(ds[k], 1)

    ts = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for a, b in zip(got, want):
        same(a, b)
