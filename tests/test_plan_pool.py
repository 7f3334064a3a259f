"""The pool of spectral plans (host logic, no GPU), on stand-ins for plans: no
two streams share workspaces, batches grow, the pool is bounded."""

import threading
import time

import pytest

from finitevolx_b200._lib import FvxError
from finitevolx_b200.solvers.spectral import _PlanPool


class Plan:
    def __init__(self, key, batch, fp64):
        self.key, self.batch_max, self.fp64 = key, batch, fp64


def test_streams_have_their_own_plans():
    pool = _PlanPool(Plan)
    a = pool.get("p", 0, 2, True, False)
    assert pool.get("p", 0, 1, True, False) is a
    b = pool.get("p", 7, 2, True, False)
    assert b is not a and pool.get("p", 7, 2, True, False) is b
    assert pool.get("other", 0, 2, True, False) not in (a, b)
    grown = pool.get("p", 0, 5, True, False)
    assert grown.batch_max == 5 and pool.get("p", 0, 2, True, False) is grown
    assert pool.get("p", 7, 2, True, False) is b


def test_threads_create_one_plan():
    made = []

    def make(*args):
        time.sleep(0.02)
        made.append(Plan(*args))
        return made[-1]

    pool = _PlanPool(make)
    got = []
    threads = [threading.Thread(target=lambda: got.append(pool.get("p", 0, 1, True, False))) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(made) == 1 and all(p is made[0] for p in got) and len(got) == 8


def test_bounded_oldest_first():
    pool = _PlanPool(Plan)
    plans = [pool.get("p", s, 1, True, False) for s in range(_PlanPool.STREAMS)]
    extra = pool.get("p", 100, 1, True, False)
    assert pool.get("p", 100, 1, True, False) is extra
    assert all(pool.get("p", s, 1, True, False) is plans[s] for s in range(2, _PlanPool.STREAMS))
    assert pool.get("p", 0, 1, True, False) is not plans[0]


def test_memory_of_other_streams_is_given_back():
    room = [2]

    def make(key, batch, fp64):
        if room[0] == 0:
            room[0] = 2  # what the pool drops is free again
            raise FvxError("memory")
        room[0] -= 1
        return Plan(key, batch, fp64)

    pool = _PlanPool(make)
    a, b = pool.get("p", 0, 1, True, False), pool.get("p", 1, 1, True, False)
    c = pool.get("p", 2, 1, True, False)
    assert pool.get("p", 2, 1, True, False) is c
    assert pool.get("p", 0, 1, True, False) is not a

    def never(*args):
        raise FvxError("memory")

    with pytest.raises(FvxError):
        _PlanPool(never).get("p", 0, 1, True, False)


def test_capture_uses_a_plan_made_before():
    pool = _PlanPool(Plan)
    a = pool.get("p", 0, 2, True, False)
    assert pool.get("p", 9, 2, True, True) is a


def test_fp64_is_part_of_the_request():
    pool = _PlanPool(Plan)
    a = pool.get("p", 0, 4, False, False)
    b = pool.get("p", 0, 1, True, False)
    assert b.fp64 and b.batch_max == 4
    assert pool.get("p", 0, 4, False, False) is b and pool.get("p", 0, 2, True, False) is b and a is not b
    pool.get("p", 1, 1, False, False)
    assert pool.get("p", 2, 1, True, True) is b  # a capture takes one that has it
