"""The planner's order from counts made on the device (k_sample) equals the
one from the host's, strings at the ends of its range (empty, 256 and more
symbols: counted on the host) among the sampled ones.  The order shows in the
number of pairs that reach a scan."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from tests import _util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[0, 5, 40], [255, 256], [256, 257, 300], [16, 17, 31, 32, 33, 64]])
def test_order_is_the_hosts(built, lens):
    rng = np.random.Generator(np.random.PCG64(len(lens)))

    def table(n):
        def s(alphabet):
            return [bytes(rng.choice(list(alphabet), size=lens[int(rng.integers(0, len(lens)))]).tolist())
                    for _ in range(n)]
        return [[b"id"] + [b"%d" % i for i in range(n)], [b"s1"] + s(b"ab"), [b"s2"] + s(b"abcdefghijklm"),
                [b"k1"] + [b"0"] * n, [b"k2"] + [b"1"] * n]

    cl, cr = table(150), table(220)
    docs = [synth.rule_yaml([3], [(1, 0.6), (2, 0.75)]), synth.rule_yaml([4], [(2, 0.2), (1, 0.97)]),
            synth.rule_yaml([3], [(1, 0.9), (2, 0.9)])]
    seen = {}
    for ingest in (0, 1):
        c = hb.Context(0, ingest=ingest, tile_right=96, eval_variant=2)
        plan = hb.Plan.from_yaml(docs, c)
        left, right = hb.Table.from_columns(cl, c), hb.Table.from_columns(cr, c)
        got, st = hb.block(c, plan, left, right, 1, _util.INT_MAX, "plain")
        again, st2 = hb.block(c, plan, left, right, 1, _util.INT_MAX, "plain")  # the memoised order
        assert (st.pairs_scanned, st.rest_scans) == (st2.pairs_scanned, st2.rest_scans)
        seen[ingest] = (_util.sorted_pairs(got).tolist(), st.pairs_scanned, st.rest_scans)
        assert _util.sorted_pairs(again).tolist() == seen[ingest][0]
        c.close()
    assert seen[0] == seen[1]
