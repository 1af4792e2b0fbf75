"""Work items larger than a staging buffer (tile_right above 128: pieces of 96
right rows), with right blocks at the pieces' and items' edges, beside a rule
of equalities only."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 32, 95, 96, 97, 128, 159, 160, 161, 191, 192, 193, 287, 288, 289, 320, 321, 385]


@pytest.mark.parametrize("tile", [128, 160, 192, 288, 320])
@pytest.mark.parametrize("variant", [1, 2])
def test_pieces_of_an_item(built, tile, variant):
    cl, cr = _util.random_tables(12, 3 * len(SIZES), sum(SIZES), b"abcd", 20)
    cl[3][1:] = [b"%d" % (i % len(SIZES)) for i in range(3 * len(SIZES))]
    cr[3][1:] = [b"%d" % k for k, n in enumerate(SIZES) for _ in range(n)]
    cl[4][1:] = [b"%d" % (i % 50) for i in range(3 * len(SIZES))]
    cr[4][1:] = [b"%d" % (i % 997) for i in range(sum(SIZES))]
    docs = [synth.rule_yaml([3], [(1, 0.62), (2, 0.6)]), synth.rule_yaml([3, 4], []),
            synth.rule_yaml([3, 4], [(1, 0.3)])]
    want = api.run_block(api.CTable(cl), api.CTable(cr), rules.serialize(rules.sort_rules(
        [rules.decode_rule(rules.parse_yaml(d)) for d in docs])), 2)
    assert len(want.pairs) > 100
    c = hb.Context(0, tile_right=tile, eval_variant=variant)
    plan = hb.Plan.from_yaml(docs, c)
    left, right = hb.Table.from_columns(cl, c), hb.Table.from_columns(cr, c)
    for mode in ("plain", "batched"):
        got, st = hb.block(c, plan, left, right, 2, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
        assert st.pair_comparisons == want.pair_comparisons
    c.close()
