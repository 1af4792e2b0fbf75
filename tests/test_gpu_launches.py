"""hbx_stats.n_launches counts every kernel of a run."""
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from tests import _util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("longest,extra", [(20, 0), (300, 1)])
def test_launches_of_a_run(built, longest, extra):
    """Batched: reset, three of the join, evaluation, report, and the long
    left strings' where there are some.  Plain (one partition, one rule): the
    same and the gathering of its bounds; long left strings twice, their work
    items and the pairs deferred to them."""
    cl, cr = _util.random_tables(5, 40, 60, b"ab", 16, n_eq_values=1)
    cl[1][3] = b"ab" * (longest // 2)
    c = hb.Context(0)
    plan = hb.Plan.from_yaml([synth.rule_yaml([3], [(1, 0.7)])], c)
    left, right = hb.Table.from_columns(cl, c), hb.Table.from_columns(cr, c)
    assert hb.block(c, plan, left, right, 1, _util.INT_MAX, "batched")[1].n_launches == 6 + extra
    assert hb.block(c, plan, left, right, 1, _util.INT_MAX, "plain")[1].n_launches == 7 + 2 * extra
    s = hb.Session(c, plan, left, right)
    for mode, n in (("batched", 6 + extra), ("plain", 7 + 2 * extra), ("batched", 6 + extra)):
        s.count(mode)  # the last one replays the graph of the first
        assert s.stats().n_launches == n, mode
    s.close()
    c.close()
