"""The device encoder where its launches split: more equality slots, string
columns and copied pieces than one launch takes, and scans at the limit of the
single-launch form (2,048 chunks of 4,096 values)."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu


def _plan(docs):
    return rules.serialize(rules.sort_rules([rules.decode_rule(rules.parse_yaml(d)) for d in docs]))


@pytest.mark.parametrize("n_cols", [7, 8, 9, 17])
@pytest.mark.parametrize("ingest", [0, 1])
def test_many_columns(built, n_cols, ingest):
    rng = np.random.Generator(np.random.PCG64(n_cols))
    width = 1 + 2 * n_cols  # id, equality columns, string columns

    def table(n):
        t = [[b"id"] + [b"%d" % i for i in range(n)]]
        t += [[b"k"] + [b"%d" % int(x) for x in rng.integers(0, 2 + c % 3, size=n)]
              for c in range(n_cols)]
        t += [[b"s"] + [bytes(rng.choice(list(b"abcde"), size=int(rng.integers(0, 40))).tolist())
                        for _ in range(n)] for _ in range(n_cols)]
        return t

    cl, cr = table(90), table(140)
    cols = ", ".join(str(c) for c in range(width))
    docs = [synth.rule_yaml([1 + k], [(1 + n_cols + k, 0.62)])
            .replace("[0, 0, 1, 2, 3, 4]", f"[0, {cols}]").replace("[1, 0, 1, 2, 3, 4]", f"[1, {cols}]")
            for k in range(n_cols)]
    want = api.run_block(api.CTable(cl), api.CTable(cr), _plan(docs), 3)
    assert len(want.pairs) > 10
    c = hb.Context(0, ingest=ingest)
    plan = hb.Plan.from_yaml(docs, c)
    got, st = hb.block(c, plan, hb.Table.from_columns(cl, c), hb.Table.from_columns(cr, c), 3)
    assert np.array_equal(_util.sorted_pairs(got), want.pairs)
    assert st.pair_comparisons == want.pair_comparisons
    assert st.pairs_covered == want.pairs_covered
    c.close()


@pytest.mark.parametrize("cards", [(64, 64), (65, 64), (2048, 4096), (2049, 4096)])
def test_resident_key_domains_at_the_scan_limit(ctx, cards):
    """The resident join's offsets are scanned over the product of the two
    columns' distinct values: 1, 2, 2,048 and 2,049 chunks."""
    n = 6000
    _, cr = _util.random_tables(cards[0], 5, n, b"abc", 12)
    cr[3][1:] = [b"%d" % (i % (cards[0] - 1)) for i in range(n)]  # the header row is a value too
    cr[4][1:] = [b"%d" % (i % (cards[1] - 1)) for i in range(n)]
    docs = [synth.rule_yaml([3, 4], [(1, 0.3)])]
    request = [[c[1 + 97 * i % n] for i in range(40)] for c in cr]
    want = api.run_block(api.CTable([[b"\x01"] + c for c in request]), api.CTable(cr), _plan(docs), 1)
    pairs = want.pairs[want.pairs[:, 0] > 0] - np.array([1, 0], np.uint32)
    assert len(pairs) > 30
    with hb.Server(ctx, [hb.Plan.from_yaml(docs, ctx)], hb.Table.from_columns(cr, ctx)) as srv:
        srv.submit(1, 0, request)
        got = srv.poll(20000)
    assert np.array_equal(got["pairs"], _util.sorted_pairs(pairs))
