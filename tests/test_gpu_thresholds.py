"""Thresholds around and above 1 with common prefixes around and above 10:
the prefix has no cap, so the Jaro-Winkler value would pass 1 from there on,
and the reference cuts it at 1 before it compares (device_func.cuh:228-230)."""
import ctypes

import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu

PREFIXES = (9, 10, 11, 17, 100)


def _tables(length):
    """Strings of about `length` symbols; a left and a right one have one of
    PREFIXES in common, or all."""
    rng = np.random.Generator(np.random.PCG64(length))
    base = rng.choice(list(b"abcdefghij"), size=length + 4).astype(np.uint8)

    def table(mark):
        rows = []
        for p in PREFIXES + (length + 4,):
            for cut in (0, 3):  # equal lengths, and not
                s = base[:length + 4 - cut].copy()
                if p < len(s):
                    s[p] = ord(mark)
                rows.append(s.tobytes())
        n = len(rows)
        return [[b"id"] + [b"%d" % i for i in range(n)], [b"s1"] + rows, [b"s2"] + rows[::-1],
                [b"k1"] + [b"1"] * n, [b"k2"] + [b"%d" % (i % 2) for i in range(n)]]

    return table("x"), table("y")


@pytest.mark.parametrize("thr", [0.9999, 1.0, 1.00005, 1.05, 2.0])
@pytest.mark.parametrize("length", [20, 60, 120, 250, 300, 600])
@pytest.mark.parametrize("group", [False, True])
def test_against_the_oracle(ctx, thr, length, group):
    import torch

    docs = [synth.rule_yaml([3], [(1, thr)])]
    if group:  # members at their own thresholds, on the first and on a later column
        docs += [synth.rule_yaml([3, 4], [(1, 0.97), (2, thr)]), synth.rule_yaml([4, 3], [(1, 0.995), (2, 0.98)])]
    cl, cr = _tables(length)
    want = api.run_block(api.CTable(cl), api.CTable(cr), rules.serialize(rules.sort_rules(
        [rules.decode_rule(rules.parse_yaml(d)) for d in docs])), 1).pairs
    assert group or (len(want) > 0) == (thr <= 1.0)
    plan = hb.Plan.from_yaml(docs, ctx)
    left, right = hb.Table.from_columns(cl, ctx), hb.Table.from_columns(cr, ctx)
    for mode in ("plain", "batched"):
        got, _ = hb.block(ctx, plan, left, right, 1, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want), mode
    got, _ = hb.block_streamed(ctx, plan, left, right, 1, 1 << 14)
    assert np.array_equal(_util.sorted_pairs(got), want)
    with hb.Server(ctx, [plan], right) as srv:
        srv.submit(1, 0, [c[1:] for c in cl])
        got = srv.poll(20000)["pairs"]
    served = want[want[:, 0] > 0] - np.array([1, 0], np.uint32)
    assert np.array_equal(got, served)
    out = torch.empty((2, 1024), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    p = hb.Pairs(out[0].data_ptr(), out[1].data_ptr(), 1024, 0, 0)
    assert hb.lib().hbx_block_static(0, plan.h, left.h, right.h, 1, hb.INT_MAX, ctypes.byref(p),
                                     None, None) == hb.OK
    got = out[:, :p.n_written].cpu().numpy().view(np.uint32).T
    assert np.array_equal(_util.sorted_pairs(got), want)
