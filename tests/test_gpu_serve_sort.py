"""Serving results are sorted on the device from kDeviceSortPairs pairs per
batch on, on the host below: batches around that size, requests of several
chunks among them, give the oracle's pairs in (record, resident row) order."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 7, 8, 9, 64, 300])
@pytest.mark.parametrize("chunk", [0, 5])
def test_results_in_order_at_any_size(ctx, rows, chunk):
    # about 256 pairs per record: 8 records make 2,048
    cl, cr = _util.random_tables(3, 300, 512, b"ab", 12, n_eq_values=2)
    docs = [synth.rule_yaml([3], [(1, 0.0)])]
    plan = rules.serialize(rules.sort_rules([rules.decode_rule(rules.parse_yaml(d)) for d in docs]))
    request = [c[1:1 + rows] for c in cl]
    want = api.run_block(api.CTable([[b"\x01"] + c for c in request]), api.CTable(cr), plan, 1).pairs
    want = want[want[:, 0] > 0] - np.array([1, 0], np.uint32)
    right = hb.Table.from_columns(cr, ctx)
    with hb.Server(ctx, [hb.Plan.from_yaml(docs, ctx)], right, max_batch_rows=chunk) as srv:
        for k in range(3):
            srv.submit(k, 0, request)
        for _ in range(3):
            got = srv.poll(20000)
            assert got["status"] == hb.OK
            assert np.array_equal(got["pairs"], _util.sorted_pairs(want))
