"""A grid whose layout and fullest cell both turn out wrong at the read-back:
the update that replaces it is confirmed too before the grid is read or
permutes, so cells keep (group, raw index) order, as with the radix sort."""
import numpy as np
import pytest

from tests.helpers import assert_bitwise, point_scene

pytestmark = pytest.mark.gpu


def contracted(knob, read):
    """Points over about 128 cells an axis (keys too long to count 2000 items
    by), then most of them in one cell."""
    from prtcl_gb300.core import DeviceScene
    rng = np.random.default_rng(5)
    n, r = 2000, 0.05
    wide = (rng.random((n, 3)) * 128.0 * r).astype(np.float32)
    tight = (rng.random((n, 3)) * 3.0 * r).astype(np.float32)
    crowd = rng.permutation(n)[:1200]
    tight[crowd] = (rng.random((1200, 3)) * 0.9 * r).astype(np.float32)
    d = DeviceScene()
    d.model.tune_set("grid_sort", knob)
    point_scene(d, [("p", "fluid", wide, [])], r)
    d.update()
    d.set_varying("p", "position", tight)
    d.update()
    if read == "permute":
        d.permute()
        return d.get_varying("p", "position", 3), d.nhood.grid()["sorted"]
    g = d.nhood.grid()
    return tuple(g[k] for k in ("sorted", "cell_gi", "cell_range", "cell_adj"))


@pytest.mark.parametrize("read", ["grid", "permute"])
def test_both_predictions_wrong(read):
    for a, b in zip(contracted(1, read), contracted(0, read)):
        assert_bitwise(a, b, read)
