"""Scenes that arrive in a batch: empty groups, single items and slots around
a block's 256 items, scenes taken out again before they are set up, and host
buffers (pageable and pinned) that are written again once add_scene returns."""
import numpy as np
import pytest

from prtcl_gb300 import driver
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu

P = dict(driver.DAM_BREAK_27K, viscosity=True)


def scene(nf, nb, seed):
    rng = np.random.default_rng(seed)
    k = max(2, int(np.ceil(max(nf, 1) ** (1 / 3))))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:nf]
    f = (g * 0.025 + rng.normal(0, 1e-3, (nf, 3))).astype(np.float32)
    b = (rng.random((nb, 3)) * [k * 0.025, 0.05, k * 0.025] - [0, 0.06, 0]).astype(np.float32)
    return f, b


def alone(f, b, steps):
    from prtcl_gb300.batch import Batch
    bt = Batch(P)
    i = bt.add_scene(f, b)
    bt.step(steps)
    return bt.download(i, "position"), bt.download(i, "mass"), bt.download(i, "time_of_birth")


@pytest.mark.parametrize("pinned", [False, True])
def test_arrivals(pinned):
    import torch

    from prtcl_gb300.batch import Batch
    sizes = [(1, 0), (0, 5), (255, 1), (256, 300), (0, 0), (257, 256), (700, 0), (64, 33)]
    bt = Batch(P)
    ids = []

    def add(f, b):
        bufs = [torch.empty(a.shape, dtype=torch.float32, pin_memory=pinned).numpy() for a in (f, b)]
        for buf, a in zip(bufs, (f, b)):
            buf[...] = a
        i = bt.add_scene(*bufs)
        for buf in bufs:
            buf[...] = np.nan
        return i

    for k, (nf, nb) in enumerate(sizes):
        if k == 4:
            bt.step(2)  # the first ones are under way
            bt.remove_scene(ids[2])
        gone = add(*scene(100, 50, 99))
        ids.append(add(*scene(nf, nb, k)))
        bt.remove_scene(gone)
    bt.step(6)
    for k, (nf, nb) in enumerate(sizes):
        if k == 2 or nf == 0:
            continue
        for got, want in zip((bt.download(ids[k], n) for n in ("position", "mass")),
                             alone(*scene(nf, nb, k), 8 if k < 4 else 6)):
            assert_bitwise(got, want, f"scene {k}")
