"""The equality join (k_join_count, k_join_scan, k_join_scatter) where its
pieces meet: key domains at the edges of the scan's chunks (4,096 keys), with
more chunks than one warp adds up, and rules that share their equalities (one
of them counts the comparisons of all)."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu

RULES = [synth.rule_yaml([3], [(1, 0.6)]), synth.rule_yaml([3, 4], [(1, 0.7), (2, 0.5)]),
         synth.rule_yaml([4, 3], [(2, 0.6), (1, 0.55)]), synth.rule_yaml([3], [(2, 0.8)])]


@pytest.mark.parametrize("n_keys", [4095, 4096, 4097, 32 * 4096 + 1, 35 * 4096])
@pytest.mark.parametrize("docs", [RULES[:1], RULES[1:3], RULES])
def test_domains_at_chunk_edges(ctx, n_keys, docs):
    cl, cr = _util.random_tables(n_keys, 300, n_keys - 1, b"abc", 10)
    # every key occurs on the right (the header row holds one of its own);
    # the last keys occur on the left
    cr[3][1:] = [b"%d" % i for i in range(n_keys - 1)]
    cl[3][1:] = [b"%d" % max(0, n_keys - 2 - 7 * i) for i in range(300)]
    want = api.run_block(api.CTable(cl), api.CTable(cr), rules.serialize(rules.sort_rules(
        [rules.decode_rule(rules.parse_yaml(d)) for d in docs])), 1)
    assert len(want.pairs) > 10
    plan = hb.Plan.from_yaml(docs, ctx)
    left, right = hb.Table.from_columns(cl, ctx), hb.Table.from_columns(cr, ctx)
    for mode in ("plain", "batched"):
        got, st = hb.block(ctx, plan, left, right, 1, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
        assert st.pair_comparisons == want.pair_comparisons, mode
