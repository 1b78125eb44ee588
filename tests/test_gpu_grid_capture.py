"""Grid updates that are captured into a graph and replayed."""
import numpy as np
import pytest

from tests.helpers import assert_bitwise, point_scene

pytestmark = pytest.mark.gpu

R = 0.1


def scene(x, knob):
    from prtcl_gb300.core import DeviceScene
    d = DeviceScene()
    d.model.tune_set("grid_sort", knob)
    point_scene(d, [("p", "fluid", x, [])], R)
    return d


def captured(d):
    import torch
    s = torch.cuda.ExternalStream(d.model.stream_handle())
    d.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
        d.update()

    def replay():
        with torch.cuda.stream(s):
            g.replay()
    return replay


def equal(d, x):
    o = scene(x, 0)
    o.update()
    got, want = d.nhood.grid(), o.nhood.grid()
    for k in want:
        assert_bitwise(got[k], want[k], k)


def test_without_a_table():
    """Sorted so far, so there is no table to count in, and none can be
    allocated during a capture: the captured update sorts."""
    x = (np.random.default_rng(1).random((3000, 3)) * 0.9).astype(np.float32)
    d = scene(x, 0)
    for _ in range(2):
        d.update()
    d.model.tune_set("grid_sort", 1)
    replay = captured(d)
    replay()
    equal(d, x)


@pytest.mark.parametrize("m", [0, 300, 1500])
def test_cells_that_fill_between_replays(m):
    """Cells of any size come out in (group, raw index) order, at the first
    replay and at later ones, whose cells the host does not look at."""
    rng = np.random.default_rng(m)
    x = (rng.random((3000, 3)) * 0.9).astype(np.float32)
    x[:2] = (0.05, 0.05, 0.05), (0.85, 0.85, 0.85)  # (the key bits stay the same)
    d = scene(x, 1)
    for _ in range(2):
        d.update()
    replay = captured(d)
    replay()
    equal(d, x)
    full = x.copy()
    full[rng.permutation(np.arange(2, 3000))[:m]] = (rng.random((m, 3)) * 0.08 + 0.41).astype(np.float32)
    d.set_varying("p", "position", full)
    replay()
    equal(d, full)
