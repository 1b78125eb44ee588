"""The grid built by counting (grid_sort 1, short cell keys) at its edges:
cells around the size it ranks, key bits that are informative on one axis
only, layouts that change between updates, tables that grow, tile and run
boundaries.  Grid and lists equal the oracle's, as with the radix sort
(grid_sort 0)."""
import numpy as np
import pytest

from prtcl_gb300 import scenes
from tests.helpers import assert_bitwise, point_scene
from tests.test_gpu_grid import make
from tests.test_gpu_list_layout import check_lists

pytestmark = pytest.mark.gpu


def grid_equal(d, o):
    gd, go = d.nhood.grid(), o.grid()
    for k in ("cell_gi", "cell_range", "cell_adj", "sorted"):
        assert_bitwise(gd[k], go[k], k)


def compare(d, o, groups):
    grid_equal(d, o)
    check_lists(d, o, [g[0] for g in groups], [len(g[2]) for g in groups])


@pytest.mark.parametrize("knob", [0, 1])
@pytest.mark.parametrize("m", [1, 2, 255, 256, 257, 1000])
def test_cell_sizes(oracle_mod, m, knob):
    """m items in one cell (more than 256 go to the radix sort), few around;
    then fewer again, at the same and at another radius."""
    rng = np.random.default_rng(m)
    pts = np.concatenate([rng.random((m, 3)) * 0.1, rng.random((300, 3)) * [2.0, 0.3, 0.1] + 0.1]).astype(np.float32)
    rng.shuffle(pts)
    b = (rng.random((77, 3)) * 0.3).astype(np.float32)
    d, o = make(oracle_mod, [("f", "fluid", pts, []), ("w", "boundary", b, [])], 0.1, {"grid_sort": knob})
    grid_equal(d, o)
    for r in (0.1, 0.05, 0.1):
        pts = (pts + rng.random(pts.shape) * np.float32(0.02)).astype(np.float32)
        for s in (d, o):
            s.set_varying("f", "position", pts)
            s.set_radius(r)
            s.update()
        grid_equal(d, o)


@pytest.mark.parametrize("scale", [(1, 1, 1), (40, 3, 1), (1, 40, 3), (3, 1, 200), (900, 900, 1)])
@pytest.mark.parametrize("shift", [0.0, -1.7, 5.3, -0.05])
def test_flat_domains(oracle_mod, scale, shift):
    """Axes that span different numbers of cells, across and beside zero."""
    rng = np.random.default_rng(scale[0] + 7 * scale[1])
    pts = (rng.random((3000, 3)) * scale * 0.1 + shift).astype(np.float32)
    groups = [("p", "fluid", pts, [])]
    d, o = make(oracle_mod, groups, 0.1)
    compare(d, o, groups)


def test_axis_layout_changes(oracle_mod):
    """x spans many cells throughout, so the bits that are informative on any
    axis stay the same while y and z come to need them too: the table's layout
    is another one, and back."""
    rng = np.random.default_rng(4)
    base = rng.random((5000, 3))
    d = o = None
    for sy, sz in [(2, 2), (50, 2), (50, 60), (2, 2), (3, 60)]:
        pts = (base * [60.0, sy, sz] * 0.1 + 0.3).astype(np.float32)
        pts[0], pts[1] = (0.11, 0.31, 0.31), (6.29, 0.31, 0.31)
        groups = [("p", "fluid", pts, [])]
        if d is None:
            d, o = make(oracle_mod, groups, 0.1)
        else:
            for s in (d, o):
                s.set_varying("p", "position", pts)
                s.update()
        compare(d, o, groups)


def test_positions_changed_after_update(oracle_mod):
    """The update leaves the sorted positions for the list build; positions
    set after it are the ones the lists see."""
    rng = np.random.default_rng(8)
    pts = (rng.random((2000, 3)) * 0.5).astype(np.float32)
    groups = [("p", "fluid", pts, [])]
    d, o = make(oracle_mod, groups, 0.05)
    compare(d, o, groups)
    moved = (pts + rng.normal(0, 0.002, pts.shape)).astype(np.float32)
    for s in (d, o):
        s.set_varying("p", "position", moved)
    od, idd = d.nhood.neighbor_lists(0, 0, 2000)
    oo, ido = o.neighbor_lists(0, 0, 2000)
    assert_bitwise(od, oo, "offsets")
    assert_bitwise(idd, ido, "indices")


@pytest.mark.parametrize("n", [4096, 60000, 300000])
def test_counted_equals_sorted(n):
    """Random order, blobs and a shuffled lattice: the counted grid is the
    sorted one, table by table, over several updates."""
    from prtcl_gb300.core import DeviceScene
    rng = np.random.default_rng(n)
    x = np.concatenate([scenes.search_points(n // 2, "blobs", seed=3),
                        rng.random((n - n // 2, 3)).astype(np.float32)]).astype(np.float32)
    got = []
    for knob in (0, 1):
        d = DeviceScene()
        d.model.tune_set("grid_sort", knob)
        point_scene(d, [("a", "fluid", x[: n // 3], []), ("b", "boundary", x[n // 3:], [])], 0.02)
        out = []
        for k in range(3):
            d.set_varying("a", "position", (x[: n // 3] + np.float32(0.01 * k)).astype(np.float32))
            d.update()
            out.append(d.nhood.grid())
            if k == 1:
                d.permute()
                out.append(d.nhood.grid())
        got.append(out)
    for g0, g1 in zip(*got):
        for k in g0:
            assert_bitwise(g0[k], g1[k], k)
