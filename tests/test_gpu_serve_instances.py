"""More rule instances (requests x rules of their plans) waiting than a batch
may hold: 1,200 requests of one record under a plan of 64 rules, queued behind a
request that takes a while."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu

STRICT = [synth.rule_yaml([3, 4], [(1, round(0.99 - 0.001 * k, 4))]) for k in range(64)]
LOOSE = [synth.rule_yaml([3], [(1, 0.6)])]


def test_many_small_requests(built):
    rng = np.random.Generator(np.random.PCG64(64))
    words = [bytes(rng.choice(list(b"abcd"), size=int(rng.integers(6, 12))).tolist()) for _ in range(40)]

    def cells(n):
        return [[b"%d" % i for i in range(n)], [words[int(k)] for k in rng.integers(0, 40, size=n)],
                [b"x"] * n, [b"%d" % int(k) for k in rng.integers(0, 3, size=n)],
                [b"%d" % int(k) for k in rng.integers(0, 2, size=n)]]

    resident = cells(600)
    long = [c[:] for c in resident]
    pad = cells(200_000)
    pad[3] = [b"far"] * 200_000  # partners of the slow request alone
    for c in range(5):
        long[c] += pad[c]
    records = [[[c[k]] for c in cells(8)] for k in range(8)]
    slow = cells(4096)
    slow[3] = [b"far"] * 4096

    def oracle(docs, cols):
        plan = rules.serialize(rules.sort_rules([rules.decode_rule(rules.parse_yaml(d)) for d in docs]))
        return api.run_block(api.CTable(cols), api.CTable(resident), plan, 1).pairs

    want = {(p, k): oracle(d, records[k]) for p, d in ((0, STRICT), (1, LOOSE)) for k in range(8)}
    assert len(want[1, 0]) > len(want[0, 0])
    c = hb.Context(0)
    plans = [hb.Plan.from_yaml(d, c) for d in (STRICT, LOOSE)]
    with hb.Server(c, plans, hb.Table.from_columns(long, c), max_inflight=1) as srv:
        srv.submit(10_000, 1, slow)
        for i in range(1200):
            srv.submit(i, 1 if i % 100 == 99 else 0, records[i % 8])
        most = 0
        for _ in range(1201):
            r = srv.poll(60000)
            assert r["status"] == hb.OK
            if r["id"] == 10_000:
                continue
            most = max(most, r["batch_requests"])
            assert np.array_equal(r["pairs"], want[r["plan"], r["id"] % 8]), (r["id"], r["batch_requests"])
    print("largest batch", most)
    c.close()
