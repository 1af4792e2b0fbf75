"""A streamed call's predicate order comes from the device's count of the
planner's sample, and is the order the host's count gives (it shows in the
number of pairs that reach a scan)."""
import ctypes

import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from tests import _util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lens", [[0, 5, 40], [256, 257, 300]])
def test_order_is_counted_on_the_device(built, lens):
    rng = np.random.Generator(np.random.PCG64(len(lens)))

    def table(n):
        def s(alphabet):
            return [bytes(rng.choice(list(alphabet), size=lens[int(rng.integers(0, len(lens)))]).tolist())
                    for _ in range(n)]
        return [[b"id"] + [b"%d" % i for i in range(n)], [b"s1"] + s(b"ab"), [b"s2"] + s(b"abcdefghijklm"),
                [b"k1"] + [b"%d" % (i % 3) for i in range(n)], [b"k2"] + [b"1"] * n]

    cl, cr = table(150), table(220)
    docs = [synth.rule_yaml([3], [(1, 0.6), (2, 0.75)]), synth.rule_yaml([4], [(2, 0.2), (1, 0.97)])]
    f = hb.lib().hbx_internal_sampled_on_device
    f.restype, f.argtypes = ctypes.c_int, [ctypes.c_void_p]
    seen = {}
    for ingest in (0, 1):
        c = hb.Context(0, ingest=ingest, tile_right=96, eval_variant=2)
        plan = hb.Plan.from_yaml(docs, c)
        left, right = hb.Table.from_columns(cl, c), hb.Table.from_columns(cr, c)
        got, st = hb.block_streamed(c, plan, left, right, 3, 1 << 16, _util.INT_MAX, "plain")
        assert f(c.h) == 1 - ingest
        seen[ingest] = (_util.sorted_pairs(got).tolist(), st.pairs_scanned, st.rest_scans)
        c.close()
    assert seen[0] == seen[1]
