"""Which updates count and which sort, told apart by their launches: a layout
that was mispredicted does not send a grid without crowded cells to the sort."""
import numpy as np
import pytest

from tests.helpers import assert_bitwise, point_scene

pytestmark = pytest.mark.gpu

R = 0.1
N = 500


def scene(x, knob=1):
    from prtcl_gb300.core import DeviceScene
    d = DeviceScene()
    d.model.tune_set("grid_sort", knob)
    point_scene(d, [("p", "fluid", x, [])], R)
    return d


def move(d, x):
    """The launches of the update after the points moved, and the grid."""
    from prtcl_gb300._lib import load
    d.set_varying("p", "position", x)
    before = load().prtcl_gpu_launch_count()
    d.update()
    launches = load().prtcl_gpu_launch_count() - before
    return launches, d.nhood.grid()


def points(rng, cells):
    """Along x in the given cells, one after the other."""
    x = (rng.random((N, 3)) * 0.8 * R + 0.1 * R).astype(np.float32)
    x[:, 0] += (np.asarray(cells)[np.arange(N) % len(cells)] * R).astype(np.float32)
    return x


def launches_of(knob, x):
    d = scene(x, knob)
    move(d, x)
    return move(d, x)[0]


def test_mispredicted_layout_is_no_crowd():
    rng = np.random.default_rng(2)
    two = points(rng, [0, 1])                 # one informative bit, 250 a cell
    even = points(rng, np.arange(0, 120, 2))  # 8 or 9 a cell; by that bit, all of them in one entry
    counted, sorted_ = launches_of(1, even), launches_of(0, even)
    assert counted != sorted_
    d, o = scene(two), scene(two, 0)
    for x in (two, even, even):
        launches, g = move(d, x)
        want = move(o, x)[1]
        for k in want:
            assert_bitwise(g[k], want[k], k)
    assert launches == counted


@pytest.mark.parametrize("m", [257, 400])
def test_counts_again_once_a_crowd_is_gone(m):
    """A cell too full to count, one that is nearly so, then none: sorted while
    it lasts and once more, counted after that."""
    rng = np.random.default_rng(m)
    even = points(rng, np.arange(0, 120, 2))

    def crowd(k):
        x = even.copy()
        x[:k] = (rng.random((k, 3)) * 0.8 * R + 0.1 * R).astype(np.float32)
        return x

    counted, sorted_ = launches_of(1, even), launches_of(0, even)
    d, o = scene(even), scene(even, 0)
    took = []
    for x in (even, even, crowd(m), crowd(m), crowd(230), crowd(230), even, even, even):
        launches, g = move(d, x)
        want = move(o, x)[1]
        for k in want:
            assert_bitwise(g[k], want[k], k)
        took.append(launches)
    cluster = took[3]  # (the cluster sort, where the radix sort's passes are the knob's other side)
    assert cluster != counted
    assert took[1] == counted and took[3:7] == [cluster] * 4 and took[7:] == [counted] * 2
