"""hbx_stats.pair_comparisons, every (rule, left, right) triple whose
equalities hold, for rule sets in which rules have the same equalities: one of
them counts for all in the batched form, whatever their order in the plan."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu

COLS = "[%d, 0, 1, 2, 3, 4, 5, 6]"


def _rule(eq, sims):
    doc = synth.rule_yaml(eq, sims)
    for t in (0, 1):
        doc = doc.replace("[%d, 0, 1, 2, 3, 4]" % t, COLS % t)
    return doc


def _tables(seed, n_l=160, n_r=230):
    rng = np.random.Generator(np.random.PCG64(seed))
    cl, cr = _util.random_tables(seed, n_l, n_r, b"abcd", 12, n_eq_values=3)
    for t, n in ((cl, n_l), (cr, n_r)):
        for k in (2, 4):
            t.append([b"k"] + [b"%d" % int(x) for x in rng.integers(0, k, size=n)])
    return cl, cr


def _random_rules(seed):
    rng = np.random.Generator(np.random.PCG64(1000 + seed))
    # few sets of equalities, so that several rules have the same one
    sets = [sorted(rng.choice([3, 4, 5, 6], size=int(rng.integers(1, 4)), replace=False).tolist())
            for _ in range(int(rng.integers(1, 4)))]
    docs = []
    for _ in range(int(rng.integers(2, 10))):
        eq = list(sets[int(rng.integers(0, len(sets)))])
        rng.shuffle(eq)
        cols = rng.permutation([1, 2])[:int(rng.integers(1, 3))]
        docs.append(_rule(eq, [(int(c), round(float(rng.uniform(0.5, 0.9)), 3)) for c in cols]))
    return docs


MEMBER_FIRST = [_rule([3, 4], [(1, 0.6)]), _rule([3, 4], [(2, 0.7)]), _rule([3], [(1, 0.8)])]
RULE_SETS = [MEMBER_FIRST, MEMBER_FIRST[::-1],
             MEMBER_FIRST + [_rule([4, 3], [(1, 0.9), (2, 0.5)]), _rule([3], [(2, 0.9)])],
             [_rule([3, 4, 5], [(1, 0.6)]), _rule([5, 4, 3], [(2, 0.6)]), _rule([3, 5, 4], [(1, 0.5)]),
              _rule([4], [(1, 0.8)])]] + [_random_rules(s) for s in range(12)]


@pytest.mark.parametrize("k", range(len(RULE_SETS)))
def test_every_form_counts_every_triple(ctx, k):
    docs = RULE_SETS[k]
    cl, cr = _tables(k)
    want = api.run_block(api.CTable(cl), api.CTable(cr), rules.serialize(rules.sort_rules(
        [rules.decode_rule(rules.parse_yaml(d)) for d in docs])), 3)
    plan = hb.Plan.from_yaml(docs, ctx)
    left, right = hb.Table.from_columns(cl, ctx), hb.Table.from_columns(cr, ctx)
    for mode in ("plain", "batched"):
        got, st = hb.block(ctx, plan, left, right, 3, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
        assert st.pair_comparisons == want.pair_comparisons, mode
    got, st = hb.block_streamed(ctx, plan, left, right, 3, 1 << 16)
    assert np.array_equal(_util.sorted_pairs(got), want.pairs)
    assert st.pair_comparisons == want.pair_comparisons
