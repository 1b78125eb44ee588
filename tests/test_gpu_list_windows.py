"""The list build's windows: rows around the item counts at which the window
changes, and cells that fill or straddle windows of every size, equal those of
the build with a thread per query."""
import numpy as np
import pytest

from tests.helpers import assert_bitwise, point_scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [39_999, 40_000, 40_001, 199_999, 200_000, 200_001])
@pytest.mark.parametrize("mean", [3.0, 30.0])
def test_rows_at_window_limits(n, mean):
    from prtcl_gb300.core import DeviceScene
    rng = np.random.default_rng(n)
    x = rng.random((n, 3)).astype(np.float32)
    x[: n // 100] = x[: n // 100] * np.float32(0.02) + np.float32(0.4)  # some full cells
    r = float(np.float32((mean / n / 4.18879) ** (1.0 / 3.0)))
    rows = []
    for knob in (0, 1):
        d = DeviceScene()
        point_scene(d, [("p", "fluid", x, [])], r)
        d.model.tune_set("list_split", knob)
        d.update()
        rows.append(d.nhood.neighbor_lists(0, 0, n))
    assert_bitwise(rows[1][0], rows[0][0], "offsets")
    assert_bitwise(rows[1][1], rows[0][1], "indices")
