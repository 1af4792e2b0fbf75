"""hbx_serve_stats.peak_bytes is an upper bound of the device memory that batches
held: with left strings over 256 symbols and a key domain above 2^20, with
outputs that grow, pairs sorted on the device, plans of several rules, and
several batches at once.  The same pairs when the budget leaves the device's
sort no room."""
import ctypes

import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from tests import _util

pytestmark = pytest.mark.gpu

PLANS = [[synth.rule_yaml([3, 4], [(1, 0.5)])],  # 1,101 x 1,001 keys
         [synth.rule_yaml([], [(1, 0.1)])],
         [synth.rule_yaml([3, 4], [(1, 0.5)]), synth.rule_yaml([4], [(2, 0.0)]),
          synth.rule_yaml([], [(2, 0.3), (1, 0.2)])]]


@pytest.fixture(scope="module")
def tables():
    rng = np.random.Generator(np.random.PCG64(6))
    base = bytes(rng.choice(list(b"abcdefgh"), size=400).tolist())

    def rows(n, longest):
        s = [base[:int(rng.integers(1, longest))] for _ in range(n)]
        return [[b"%d" % i for i in range(n)], s, s[::-1], [b"%d" % (i % 1101) for i in range(n)],
                [b"%d" % (i % 1001) for i in range(n)]]

    return rows(3303, 40), rows(300, 60), rows(300, 400), rows(3, 400)


def _pool_peak(c, reset):
    f = hb.lib().hbx_internal_pool_peak
    f.restype, f.argtypes = ctypes.c_uint64, [ctypes.c_void_p, ctypes.c_int]
    return f(c.h, reset)


def _serve(c, resident, jobs, **kw):
    """Pairs of every job, the pool's high-water mark above the resident
    table, the server's peak_bytes."""
    plans = [hb.Plan.from_yaml(d, c) for d in PLANS]
    with hb.Server(c, plans, hb.Table.from_columns(resident, c), **kw) as srv:
        _pool_peak(c, 1)
        before = _pool_peak(c, 0)
        for k, (plan, rows) in enumerate(jobs):
            srv.submit(k, plan, rows)
        got = {}
        for _ in jobs:
            r = srv.poll(60000)
            assert r["status"] == hb.OK
            got[r["id"]] = r["pairs"]
        return got, _pool_peak(c, 0) - before, srv.stats().peak_bytes


@pytest.mark.parametrize("jobs", [[(0, 1)], [(0, 2)], [(0, 3)], [(1, 1)], [(1, 2)], [(2, 1)], [(2, 2)],
                                  [(0, 1), (1, 2), (2, 3), (0, 2), (1, 1), (2, 2)]])
@pytest.mark.parametrize("inflight,rows", [(1, 0), (3, 64)])
def test_peak_covers_what_batches_take(built, tables, jobs, inflight, rows):
    c = hb.Context(0)
    jobs = [(plan, tables[k]) for plan, k in jobs]
    _, used, peak = _serve(c, tables[0], jobs, max_inflight=inflight, max_batch_rows=rows)
    assert 0 < used <= peak
    c.close()


def test_no_room_for_the_sort(built, tables):
    c = hb.Context(0)
    jobs = [(1, tables[1]), (1, tables[2])]
    want, _, _ = _serve(c, tables[0], jobs)
    got, used, peak = _serve(c, tables[0], jobs, budget_bytes=4 << 20)
    assert len(want[0]) > 500000  # their output alone is above the budget
    for k in want:
        assert np.array_equal(got[k], want[k])
        assert np.array_equal(_util.sorted_pairs(got[k]), got[k])
    assert used <= peak
    c.close()
