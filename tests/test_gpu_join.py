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


def _rule8(eq_cols, sims):
    return synth.rule_yaml(eq_cols, sims).replace("[0, 0, 1, 2, 3, 4]", "[0, 0, 1, 2, 3, 4, 5, 6, 7]") \
        .replace("[1, 0, 1, 2, 3, 4]", "[1, 0, 1, 2, 3, 4, 5, 6, 7]")


# rules that share pairs only where the other's equalities hold: one slot, two,
# more than the two that are compared, the same ones, and more rules than are
# listed (every pair then goes through the duplicate set)
ROOTS = [
    [([3], 1), ([4], 2)],
    [([3], 1), ([4, 5], 1), ([5, 6, 7], 2)],
    [([3], 1), ([3], 2), ([4], 1)],
    [([], 1), ([4], 2)],
    [([3], 1), ([4], 2), ([5], 1), ([6], 2), ([7], 1), ([3, 5], 2)],
]


@pytest.mark.parametrize("thr", [0.55, 0.0])
@pytest.mark.parametrize("roots", range(len(ROOTS)))
def test_pairs_of_several_rules_are_reported_once(built, roots, thr):
    """At threshold 0 a quarter to all of 350,000 pairs match, more than the
    first run's duplicate set holds."""
    rng = np.random.Generator(np.random.PCG64(roots))
    cl, cr = _util.random_tables(40 + roots, 499, 701, b"abc", 9, n_eq_values=2)
    for t, n in ((cl, 499), (cr, 701)):
        for k in (2, 3, 2):
            t.append([b"k"] + [b"%d" % int(x) for x in rng.integers(0, k, size=n)])
    docs = [_rule8(eq, [(col, thr)]) for eq, col in ROOTS[roots]]
    want = api.run_block(api.CTable(cl), api.CTable(cr), rules.serialize(rules.sort_rules(
        [rules.decode_rule(rules.parse_yaml(d)) for d in docs])), 1)
    c = hb.Context(0)
    plan = hb.Plan.from_yaml(docs, c)
    left, right = hb.Table.from_columns(cl, c), hb.Table.from_columns(cr, c)
    for mode in ("plain", "batched"):
        got, st = hb.block(c, plan, left, right, 1, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
        assert st.pair_comparisons == want.pair_comparisons, mode
    got, _ = hb.block_streamed(c, plan, left, right, 1, 1 << 18)
    assert np.array_equal(_util.sorted_pairs(got), want.pairs)
    with hb.Server(c, [plan], right) as srv:
        srv.submit(1, 0, [col[1:] for col in cl])
        got = srv.poll(20000)["pairs"]
    served = want.pairs[want.pairs[:, 0] > 0] - np.array([1, 0], np.uint32)
    assert np.array_equal(got, served)
    c.close()


@pytest.mark.parametrize("n_keys", [413696, 417793, 421888, 425985])
def test_domains_around_the_wide_chunks(ctx, n_keys):
    """Three scans of 101 to 105 chunks of 4,096 keys: one wave of blocks takes
    304, so the larger sizes take chunks of 8,192."""
    cl, cr = _util.random_tables(n_keys, 300, 2000, b"abc", 10)
    n = n_keys // 4
    cr[3][1:] = [b"%d" % (i * 37 % n) for i in range(2000)]
    cl[3][1:] = [b"%d" % (n - 1 - 7 * i) for i in range(300)]
    # 4 partitions and a filler column value per key: the right table lists them all
    for c in range(len(cr)):
        cr[c] += [b"%d" % i for i in range(n - 1)] if c == 3 else [b"zz"] * (n - 1)
    docs = RULES[:1]
    want = api.run_block(api.CTable(cl), api.CTable(cr), rules.serialize(rules.sort_rules(
        [rules.decode_rule(rules.parse_yaml(d)) for d in docs])), 4)
    plan = hb.Plan.from_yaml(docs, ctx)
    left, right = hb.Table.from_columns(cl, ctx), hb.Table.from_columns(cr, ctx)
    for mode in ("plain", "batched"):
        got, st = hb.block(ctx, plan, left, right, 4, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
        assert st.pair_comparisons == want.pair_comparisons, mode
