"""The barriers of the one-launch solver loops: scenes at the largest size they
take, whose launches do not fit the chip together, solving at the same time
from threads of their own give what each gives alone, many times over."""
import threading

import pytest

from tests import test_gpu_jacobi_loop as jacobi, test_gpu_pcg_loop as pcg
from tests.helpers import assert_bitwise

pytestmark = pytest.mark.gpu

LARGEST = 152 * 4 * 128


def at_the_same_time(works):
    bad = []

    def call(w):
        try:
            w()
        except Exception as e:  # shown by the test's own thread
            bad.append(e)

    ts = [threading.Thread(target=call, args=(w,)) for w in works]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    if bad:
        raise bad[0]


def test_largest_scenes_at_the_same_time():
    js = [jacobi.scene(LARGEST, k, max_iters=30, eta=1e-9) for k in (1, 2)]
    ps = [pcg.scene(LARGEST, wkbb18_maximum_iterations=12, wkbb18_maximum_error=1e-9)]
    want_j = [jacobi.solve(d, 2) for d in js]
    want_p = [pcg.solve(d, "wkbb18", True) for d in ps]

    def jacobi_work(d, want):
        def work():
            for _ in range(20):
                jacobi.same(jacobi.solve(d, 1), want)
        return work

    def pcg_work(d, want):
        def work():
            for _ in range(20):
                got = pcg.solve(d, "wkbb18", False)
                for x, y in zip(got[0], want[0]):
                    assert_bitwise(x, y)
                assert got[1] == want[1]
        return work

    at_the_same_time([jacobi_work(d, w) for d, w in zip(js, want_j)] + [pcg_work(d, w) for d, w in zip(ps, want_p)])
