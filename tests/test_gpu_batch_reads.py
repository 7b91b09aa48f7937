"""psba_batch_get_params: a few reads bring over what they ask for and no more;
many are served from one copy of all problems, with the same values, and a solve
or a reset between reads, or beside them, leaves nothing of an older state."""
import threading

import numpy as np
import pytest

import psba_gb300 as P
from psba_gb300 import scenes
from psba_gb300.batch import Batch

pytestmark = pytest.mark.gpu


def _batch(n=40):
    return Batch([scenes.arc_scene(seed=q, n_cams=4 + q % 3, n_pts=20 + q, arc_deg=12.0, min_views=3) for q in range(n)])


def _all(b, n=40):
    return [b.get_params(q) for q in range(n)]


def _same(x, y):
    return all(np.array_equal(a, c) and np.array_equal(b, d) for (a, b), (c, d) in zip(x, y))


def test_a_few_reads_launch_nothing():
    with _batch() as b:
        b.levmar(allow_switch=0, max_iter=4)
        k = P.kernel_launches()
        first, again = b.get_params(7), b.get_params(7)
        assert P.kernel_launches() == k
        assert _same([first], [again])


def test_reads_in_any_number_and_order_agree():
    with _batch() as b:
        start = _all(b)
        b.levmar(allow_switch=0, max_iter=4)
        solved = _all(b)  # single reads first, then the copy
        assert not _same(start, solved)
        assert _same(solved, [b.get_params(q) for q in reversed(range(40))][::-1])
        b.reset()
        assert _same(start, _all(b))
        b.levmar(allow_switch=0, max_iter=4)
        assert _same(solved, _all(b))


def test_reads_beside_a_solve_leave_nothing_stale():
    with _batch() as b:
        b.levmar(allow_switch=0, max_iter=4)
        solved = _all(b)
        for _ in range(5):
            b.reset()
            stop = threading.Event()

            def reader():
                while not stop.is_set():
                    _all(b)

            t = threading.Thread(target=reader)
            t.start()
            b.levmar(allow_switch=0, max_iter=4)
            stop.set()
            t.join()
            assert _same(solved, _all(b))
