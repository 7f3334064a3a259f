"""The pool of spectral plans (host logic, no GPU), on stand-ins for plans: no
two streams share workspaces, no graph shares them with anything, batches grow,
the pool is bounded."""

import threading
import time

import pytest

from finitevolx_b200._lib import FvxError
from finitevolx_b200.solvers.spectral import _PlanPool


class Plan:
    def __init__(self, key, batch, fp64):
        self.key, self.batch_max, self.fp64, self.graphs = key, batch, fp64, 0

    def hold(self, stream):
        self.graphs += 1

    def holds(self):
        return self.graphs


def test_streams_have_their_own_plans():
    pool = _PlanPool(Plan)
    a = pool.get("p", 0, 2, True)
    assert pool.get("p", 0, 1, True) is a
    b = pool.get("p", 7, 2, True)
    assert b is not a and pool.get("p", 7, 2, True) is b
    assert pool.get("other", 0, 2, True) not in (a, b)
    grown = pool.get("p", 0, 5, True)
    assert grown.batch_max == 5 and pool.get("p", 0, 2, True) is grown
    assert pool.get("p", 7, 2, True) is b


def test_threads_create_one_plan():
    made = []

    def make(*args):
        time.sleep(0.02)
        made.append(Plan(*args))
        return made[-1]

    pool = _PlanPool(make)
    got = []
    threads = [threading.Thread(target=lambda: got.append(pool.get("p", 0, 1, True))) for _ in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(made) == 1 and all(p is made[0] for p in got) and len(got) == 8


def test_bounded_oldest_first():
    pool = _PlanPool(Plan)
    plans = [pool.get("p", s, 1, True) for s in range(_PlanPool.STREAMS)]
    extra = pool.get("p", 100, 1, True)
    assert pool.get("p", 100, 1, True) is extra
    assert all(pool.get("p", s, 1, True) is plans[s] for s in range(2, _PlanPool.STREAMS))
    assert pool.get("p", 0, 1, True) is not plans[0]


def test_memory_of_other_streams_is_given_back():
    room = [2]

    def make(key, batch, fp64):
        if room[0] == 0:
            room[0] = 2  # what the pool drops is free again
            raise FvxError("memory")
        room[0] -= 1
        return Plan(key, batch, fp64)

    pool = _PlanPool(make)
    a, b = pool.get("p", 0, 1, True), pool.get("p", 1, 1, True)
    c = pool.get("p", 2, 1, True)
    assert pool.get("p", 2, 1, True) is c
    assert pool.get("p", 0, 1, True) is not a

    def never(*args):
        raise FvxError("memory")

    with pytest.raises(FvxError):
        _PlanPool(never).get("p", 0, 1, True)


def test_fp64_is_part_of_the_request():
    pool = _PlanPool(Plan)
    a = pool.get("p", 0, 4, False)
    b = pool.get("p", 0, 1, True)
    assert b.fp64 and b.batch_max == 4
    assert pool.get("p", 0, 4, False) is b and pool.get("p", 0, 2, True) is b and a is not b


def test_graphs_have_their_own_plans():
    pool = _PlanPool(Plan)
    eager = pool.get("p", 0, 1, True)
    g = pool.get("p", 9, 1, True, capture=4)
    assert g is not eager and g.graphs == 1
    assert pool.get("p", 9, 1, True, capture=4) is g and g.graphs == 1
    fork = pool.get("p", 8, 1, True, capture=4)  # another stream of the same capture
    other = pool.get("p", 9, 1, True, capture=5)
    assert len({id(p) for p in (eager, g, fork, other)}) == 4
    # outgrown in its capture and outside: still there for the replay
    grown = pool.get("p", 9, 3, True, capture=4)
    assert grown is not g and pool.get("p", 0, 3, True) is not eager
    assert {id(p) for _, p in pool._held} == {id(p) for p in (g, fork, other, grown)}
    assert pool.get("p", 0, 1, True).graphs == 0


def test_a_graphs_plan_goes_with_it():
    pool = _PlanPool(Plan)
    g, h = pool.get("p", 9, 1, True, capture=4), pool.get("p", 9, 1, True, capture=5)
    g.graphs = 0  # destroyed: free for the next capture
    assert pool.get("q", 9, 1, True, capture=6) is not g and pool.get("p", 9, 2, True, capture=6) is not g
    assert pool.get("p", 9, 1, True, capture=7) is g and g.graphs == 1
    g.graphs = 0
    pool.get("p", 0, 1, True)  # a plan is made outside: what no graph holds goes
    assert h in [p for _, p in pool._held] and g not in [p for _, p in pool._held]


def test_a_graph_takes_a_plan_over_when_memory_is_short():
    room = [1]

    def make(key, batch, fp64):
        if not room[0]:
            raise FvxError("memory")
        room[0] -= 1
        return Plan(key, batch, fp64)

    pool = _PlanPool(make)
    a = pool.get("p", 0, 2, True)
    assert pool.get("p", 9, 1, True, capture=4) is a and a.graphs == 1
    room[0] = 1
    assert pool.get("p", 0, 2, True) is not a
    with pytest.raises(FvxError):
        pool.get("p", 9, 8, True, capture=6)
