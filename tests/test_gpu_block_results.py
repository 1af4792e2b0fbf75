"""hbx_block's pairs on their way to the host: up to 65,536 come with the
run's counters, more through page-locked chunks that grow with the results.
Counts around both limits, in one context, larger after smaller and back."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from tests import _util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["plain", "batched"])
def test_every_pair_arrives(built, mode):
    c = hb.Context(0)
    plan = hb.Plan.from_yaml([synth.rule_yaml([3], [(1, 0.0)])], c)

    def table(n):
        return hb.Table.from_columns([[b"%d" % i for i in range(n)], [b"a"] * n, [b"a"] * n,
                                      [b"k"] * n], c)

    for n_l, n_r in [(1, 1), (3, 683), (1, 65535), (256, 256), (1, 65537), (2, 131072), (1, 262145),
                     (3, 300001), (5, 7), (2, 32768), (7, 40001)]:
        got, st = hb.block(c, plan, table(n_l), table(n_r), 1, _util.INT_MAX, mode)
        assert st.n_matches == n_l * n_r
        want = np.stack((np.repeat(np.arange(n_l), n_r), np.tile(np.arange(n_r), n_l)), 1)
        assert np.array_equal(_util.sorted_pairs(got), want), (n_l, n_r)
    c.close()
