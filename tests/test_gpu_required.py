"""n_required of a call whose buffer is too small when the duplicate set fills up
in the same run: at least the distinct pairs, at most the matches of all rules
(a pair reported once and taken through the set is one of them, not two)."""
import ctypes

import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from tests import _util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["plain", "batched"])
@pytest.mark.parametrize("second", [[3], [4]])  # every pair is shared, a third of the pairs are
def test_bound_of_a_full_duplicate_set(built, mode, second):
    c = hb.Context(0)
    plan = hb.Plan.from_yaml([synth.rule_yaml([3], [(1, 0.0)]), synth.rule_yaml(second, [(2, 0.0)])], c)

    def table(n):
        return hb.Table.from_columns([[b"%d" % i for i in range(n)], [b"a"] * n, [b"b"] * n, [b"k"] * n,
                                      [b"%d" % (i % 3) for i in range(n)]], c)

    n_l, n_r = 900, 1200
    left, right = table(n_l), table(n_r)
    distinct = n_l * n_r
    matches = 2 * distinct if second == [3] else distinct + distinct // 3
    p = hb.Pairs(np.zeros(8, np.uint32).ctypes.data, np.zeros(8, np.uint32).ctypes.data, 8, 0, 0)
    st = hb.Stats()
    assert hb.lib().hbx_block(c.h, plan.h, left.h, right.h, 1, hb.INT_MAX, hb._mode(mode), ctypes.byref(p),
                              ctypes.byref(st), None) == hb.ERR_CAPACITY
    assert distinct <= p.n_required <= matches
    s = hb.Session(c, plan, left, right)
    assert distinct <= s.count(mode) <= matches
    got, st = hb.block(c, plan, left, right, 1, _util.INT_MAX, mode)
    assert st.n_matches == len(got) == distinct
    s.close()
    c.close()
