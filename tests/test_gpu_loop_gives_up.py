"""A barrier of a one-launch solver loop that gives up (no polls allowed, so
that the first block to arrive does) is an error where the host sees it first.
Velocities, positions and the viscosity solve's results are those from before,
and the next solve, with or without a set-up before it, runs as usual."""
import numpy as np
import pytest

from tests import test_gpu_jacobi_loop as jacobi, test_gpu_pcg_loop as pcg
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu

N = 152 * 4 * 128  # 608 blocks: the first to arrive never finds the others there
DEFAULT = 1 << 21


def fails(d, procedures, then):
    """The procedures, none of whose barriers may poll, then a reader: some call
    of these fails, and the error is raised once."""
    from prtcl_gb300 import _lib
    d.model.solver_polls(0)
    with pytest.raises(_lib.PrtclGpuError, match="did not meet"):
        for scheme, procedure in procedures:
            d.run(scheme, procedure)
        then()
    d.synchronize()
    d.model.solver_polls(DEFAULT)


@pytest.mark.parametrize("reader", ["synchronize", "field", "global", "lists"])
def test_pressure(reader):
    d = jacobi.scene(N, 3, max_iters=20, eta=1e-9)
    d.scheme("symplectic_euler")
    want = jacobi.solve(d, 2)
    keep = {f: d.get_varying("f", f, 3) for f in ("velocity", "position")}
    then = {"synchronize": d.synchronize, "field": lambda: d.get_varying("f", "pressure"),
            "global": lambda: d.get_global("iisph_aprde"), "lists": lambda: (d.update(), d.nhood.query(0))}[reader]
    d.model.tune_set("jacobi_unroll", 1)
    fails(d, [("iisph", "setup"), ("iisph", "solve_pressure"),
              ("symplectic_euler", "integrate_velocity_with_hard_fade"), ("symplectic_euler", "integrate_position")],
          then)
    for f, v in keep.items():
        assert_bitwise(d.get_varying("f", f, 3), v, f)
    d.run("density", "compute_density")
    jacobi.same(jacobi.solve(d, 1), want)


def test_solve_without_a_set_up_after_it():
    d = jacobi.scene(N, 4, max_iters=5, eta=1e-9)
    start = jacobi.solve(d, 2)[0][0]
    d.model.tune_set("jacobi_unroll", 1)
    fails(d, [("iisph", "solve_pressure")], d.synchronize)
    got = []
    for unroll in (2, 1):
        d.set_varying("f", "pressure", start)
        d.model.tune_set("jacobi_unroll", unroll)
        d.run("iisph", "solve_pressure")
        got.append([d.get_varying("f", name, nc) for name, nc in jacobi.FIELDS])
    for a, b in zip(*got):
        assert_bitwise(a, b)


@pytest.mark.parametrize("gc", [False, True])
def test_viscosity(gc):
    d = pcg.scene(N, wkbb18_maximum_iterations=12, wkbb18_maximum_error=1e-9)
    scheme = "wkbb18_gc" if gc else "wkbb18"
    if gc:
        d.scheme("correction")
        d.scheme("wkbb18_gc")
        d.run("correction", "compute_gradient_correction")
    want = pcg.solve(d, scheme, True)
    mark = np.random.default_rng(1).normal(0, 1, (N, 3)).astype(np.float32)
    for f in ("acceleration", "wkbb18_velocity_delta"):
        d.set_varying("f", f, mark)
    v = d.get_varying("f", "velocity", 3)
    fails(d, [(scheme, "accumulate_acceleration"), ("symplectic_euler", "integrate_velocity_with_hard_fade")],
          d.synchronize)
    for f in ("acceleration", "wkbb18_velocity_delta"):
        assert_bitwise(d.get_varying("f", f, 3), mark, f)
    assert_bitwise(d.get_varying("f", "velocity", 3), v)
    got = pcg.solve(d, scheme, False)
    for a, b in zip(got[0], want[0]):
        assert_bitwise(a, b)
    assert got[1] == want[1]
