"""CPU tests of the serving loop's slots with a stand-in executor: a cached
handle of any earlier request of a finished slot is found again, and requests
that ran one after another count neither as running together nor as memory in
use at the same time."""
import time

from mittet_main_b200.serving import MittetServer, Request


class FakeWL:
    pass


def make(rid, arrival, size=10, key=None, work=0.01):
    r = Request(rid, arrival, FakeWL())
    r.size, r.key, r.work = size, key, work
    return r


def test_a_finished_slot_keeps_the_handles_of_all_its_grids():
    """Slot 1 serves grid A, then grid B; A's next request finds A's handle
    there although slot 0 is free and B was the slot's last grid."""
    made = []

    def execu(cache, req):
        if req.key not in cache:
            cache[req.key] = object()
            made.append(req.key)
        time.sleep(req.work)

    reqs = [make(0, 0.0, key="X", work=0.15), make(1, 0.03, key="A"), make(2, 0.4, key="B"),
            make(3, 0.6, key="A"), make(4, 0.8, key="C")]
    srv = MittetServer(n_slots=2, hbm_budget=1000, executor=execu, estimator=lambda r: r.size, keyer=lambda r: r.key)
    res = srv.run(reqs)
    assert all(r.error is None for r in res)
    assert res[1].slot == res[2].slot == res[3].slot
    assert made.count("A") == 1 and srv.reuses == 1


def test_requests_one_after_another_do_not_count_as_overlapping():
    reqs = [make(i, 0.15 * i, size=30) for i in range(4)]
    srv = MittetServer(n_slots=3, hbm_budget=100, executor=lambda c, r: time.sleep(r.work), estimator=lambda r: r.size)
    srv.run(reqs)
    assert srv.max_running == 1
    assert srv.peak_in_use == 30


def test_requests_that_overlap_are_counted():
    reqs = [make(i, 0.001 * i, size=30, work=0.3) for i in range(4)]
    srv = MittetServer(n_slots=4, hbm_budget=100, executor=lambda c, r: time.sleep(r.work), estimator=lambda r: r.size)
    srv.run(reqs)
    assert srv.max_running == 3  # the budget holds three of them
    assert srv.peak_in_use == 90
