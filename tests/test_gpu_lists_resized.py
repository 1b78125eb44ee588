"""Lists of groups resized since the grid's update, from nothing and to
nothing: items that the grid does not hold have no neighbours, those that are
gone are nobody's; in both forms of the list build, one to three groups."""
import numpy as np
import pytest

from tests.helpers import assert_bitwise, point_scene

pytestmark = pytest.mark.gpu


def rows(d, q, g, n):
    o, i = d.nhood.neighbor_lists(q, g, n)
    return [list(i[o[k]:o[k + 1]]) for k in range(n)]


@pytest.mark.parametrize("knob", [0, 1])
@pytest.mark.parametrize("before,after", [(0, 1), (0, 300), (500, 600), (500, 5000), (500, 499), (500, 33), (500, 0)])
@pytest.mark.parametrize("others", [[], [200], [200, 0]])
def test_resized(before, after, others, knob):
    from prtcl_gb300.core import DeviceScene
    rng = np.random.default_rng(before + after)
    counts = [before] + others
    groups = [("abc"[k], "fluid", (rng.random((m, 3)) * 0.3).astype(np.float32), []) for k, m in enumerate(counts)]
    d = DeviceScene()
    d.model.tune_set("list_split", knob)
    point_scene(d, groups, 0.06)
    d.update()
    G = range(len(counts))
    want = [[rows(d, q, g, counts[q]) for g in G] for q in G]
    d.resize("a", after)
    d.nhood.load(d.model)
    now = [after] + others
    for q in G:
        for g in G:
            got = rows(d, q, g, now[q])
            for k, row in enumerate(got):
                old = want[q][g][k] if k < counts[q] else []
                assert row == [j for j in old if j < now[g]], (q, g, k)
    d.update()
    fresh = DeviceScene()
    point_scene(fresh, [(n, t, d.get_varying(n, "position", 3), []) for n, t, _, _ in groups], 0.06)
    fresh.update()
    for q in G:
        for g in G:
            a, b = d.nhood.neighbor_lists(q, g, now[q]), fresh.nhood.neighbor_lists(q, g, now[q])
            assert_bitwise(a[0], b[0], "offsets")
            assert_bitwise(a[1], b[1], "indices")
