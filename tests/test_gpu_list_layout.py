"""The storage of the neighbour lists (units of 32 items per chunk plane), its
readers and its builder at their edges: item counts around multiples of 32,
rows of several chunks, cells around the builder's unit and portion sizes.
Lists, and every field of the sweeps that read them, equal the oracle's bit
for bit."""
import numpy as np
import pytest

from prtcl_gb300 import driver
from tests.helpers import assert_bitwise, both_scenes, point_scene

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


def check_lists(d, o, names, counts):
    for q in range(len(names)):
        for g in range(len(names)):
            od, idd = d.nhood.neighbor_lists(q, g, counts[q])
            oo, ido = o.neighbor_lists(q, g, counts[q], cap=int(od[-1]) + 16)
            assert_bitwise(od, oo, f"offsets {q}->{g}")
            assert_bitwise(idd, ido, f"indices {q}->{g}")


# queries of a cell around the 16 of a unit, candidates around the 320 of a
# portion and past several, rows past the first capacity of 48
@pytest.mark.parametrize("knob", [0, 1])
@pytest.mark.parametrize("m", [1, 15, 16, 17, 32, 33, 319, 320, 321, 700])
def test_list_build_cell_sizes(oracle_mod, m, knob):
    h = 0.05
    rng = np.random.default_rng(m)
    cell = 2.0 * h
    # m fluid items in one cell, a few in the next, walls in both
    f = np.concatenate([rng.random((m, 3)) * cell, rng.random((5, 3)) * cell + [cell, 0, 0]]).astype(np.float32)
    b = (rng.random((20, 3)) * [2.0 * cell, cell, cell]).astype(np.float32)
    sc = {"fluid": f, "boundary": b}
    p = dict(driver.DAM_BREAK_27K, smoothing_scale=h)
    d, o = both_scenes(sc, p, oracle_mod)
    d.model.tune_set("list_split", knob)
    for s in (d, o):
        s.update()
        s.run("density", "compute_density")
        s.run("iisph", "setup")
    check_lists(d, o, ["b", "f"], [20, m + 5])
    for name, nc in [("density", 1), ("iisph_helper_c", 3), ("iisph_diagonal_element", 1)]:
        assert_bitwise(d.get_varying("f", name, nc), o.get_varying("f", name, nc), name)


def test_row_turns_wide_in_a_later_portion(oracle_mod):
    """A cell of 400 low indices beside one of 400 high indices: a row's
    first portion of candidates fits 16-bit offsets, a later one does not."""
    from prtcl_gb300.core import DeviceScene
    n, r = 70_000, 0.1
    rng = np.random.default_rng(3)
    x = np.empty((n, 3))
    x[:400] = rng.random((400, 3)) * r
    x[400:n - 400] = rng.random((n - 800, 3)) * [4.0, 4.0, 4.0] + 1.0
    x[n - 400:] = rng.random((400, 3)) * r + [r, 0.0, 0.0]
    x = x.astype(np.float32)
    d, o = DeviceScene(), oracle_mod.Scene(np.float32)
    for s in (d, o):
        point_scene(s, [("p", "fluid", x, [])], r)
        s.update()
    check_lists(d, o, ["p"], [n])


@pytest.mark.parametrize("groups", [3, 4])
def test_list_build_more_groups(oracle_mod, groups):
    """More than two neighbour groups take the thread-per-query form."""
    from prtcl_gb300.core import DeviceScene
    rng = np.random.default_rng(groups)
    gs = [("abcd"[k], "fluid", (rng.random((300 + k, 3)) * 0.3).astype(np.float32), []) for k in range(groups)]
    d, o = DeviceScene(), oracle_mod.Scene(np.float32)
    for s in (d, o):
        point_scene(s, gs, 0.06)
        s.update()
    check_lists(d, o, [g[0] for g in gs], [len(g[2]) for g in gs])


def test_lists_after_a_group_grew(oracle_mod):
    """A group that grew since the grid's update: its new items have no
    neighbours until the next update."""
    from prtcl_gb300.core import DeviceScene
    rng = np.random.default_rng(9)
    x = (rng.random((500, 3)) * 0.3).astype(np.float32)
    d = DeviceScene()
    point_scene(d, [("p", "fluid", x, [])], 0.06)
    d.update()
    before, idx = d.nhood.neighbor_lists(0, 0, 500)
    d.resize("p", 600)
    d.nhood.load(d.model)
    offs, idx2 = d.nhood.neighbor_lists(0, 0, 600)
    assert_bitwise(offs[:501], before, "offsets")
    assert (offs[501:] == before[500]).all()
    assert_bitwise(idx2, idx, "indices")
