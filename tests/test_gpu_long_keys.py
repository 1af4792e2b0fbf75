"""Left keys of strings without a Peq table (dev::Rule::ranked): one per join
key, or one per row where there are at least twice as many join keys as left
rows; the state of a large key domain is not doubled by a few long strings."""
import ctypes

import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu

ONE = [synth.rule_yaml([3], [(1, 0.7)])]
# a group on s1 whose root is the rule on k1, and rules of their own
SET = [synth.rule_yaml([3], [(1, 0.75)]), synth.rule_yaml([3, 4], [(1, 0.6), (2, 0.5)]),
       synth.rule_yaml([4], [(2, 0.8)]), synth.rule_yaml([3, 4], [(2, 0.55)])]


def _tables(n_l, n_r, n_keys, long_rows):
    """n_keys values of k1 with the header's; every n-th left string long."""
    rng = np.random.Generator(np.random.PCG64(n_keys))
    base = bytes(rng.choice(list(b"abc"), size=400).tolist())

    def table(n, prefix, long_every):
        s = [base[:int(rng.integers(257, 400))] if long_every and i % long_every == 0 else
             bytes(rng.choice(list(b"abc"), size=int(rng.integers(0, 14))).tolist()) for i in range(n)]
        k = rng.integers(0, 40, size=n) * (n_keys - 2) // 39  # the matching keys lie far apart
        return [[b"id"] + [b"%s%d" % (prefix, i) for i in range(n)], [b"s1"] + s,
                [b"s2"] + s[1:] + s[:1], [b"k1"] + [b"%d" % int(x) for x in k],
                [b"k2"] + [b"%d" % int(x) for x in rng.integers(0, 2, size=n)]]

    left, right = table(n_l, b"l", long_rows), table(n_r, b"r", 7)
    for c in range(5):  # the right table lists every key
        right[c] += [b"%d" % i for i in range(n_keys - 1)] if c == 3 else [b"b"] * (n_keys - 1)
    return left, right


def _oracle(docs, cl, cr, n_part):
    plan = rules.serialize(rules.sort_rules([rules.decode_rule(rules.parse_yaml(d)) for d in docs]))
    return api.run_block(api.CTable(cl), api.CTable(cr), plan, n_part)


# 100 left rows (with the header): 2 partitions x 99, 100 and 101 keys are on
# either side of the rule
@pytest.mark.parametrize("n_keys", [50, 99, 100, 101, 5000, 20001])
@pytest.mark.parametrize("long_rows", [1, 9])
@pytest.mark.parametrize("docs", [ONE, SET])
def test_every_form(ctx, n_keys, long_rows, docs):
    import torch

    cl, cr = _tables(99, 180, n_keys, long_rows)
    want = _oracle(docs, cl, cr, 2)
    assert len(want.pairs) > 5
    plan = hb.Plan.from_yaml(docs, ctx)
    left, right = hb.Table.from_columns(cl, ctx), hb.Table.from_columns(cr, ctx)
    for mode in ("plain", "batched"):
        got, st = hb.block(ctx, plan, left, right, 2, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
        assert st.pair_comparisons == want.pair_comparisons, mode
    s = hb.Session(ctx, plan, left, right, 2)  # runs after runs start from no ranks
    for mode in ("batched", "plain", "batched"):
        assert s.count(mode) == len(want.pairs)
    s.close()
    for mode in ("plain", "batched"):
        got, st = hb.block_streamed(ctx, plan, left, right, 2, 1 << 19, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
        assert st.pair_comparisons == want.pair_comparisons, mode
    out = torch.empty((2, 40000), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    p = hb.Pairs(out[0].data_ptr(), out[1].data_ptr(), 40000, 0, 0)
    st = hb.Stats()
    assert hb.lib().hbx_block_static(0, plan.h, left.h, right.h, 2, hb.INT_MAX, ctypes.byref(p),
                                     None, ctypes.byref(st)) == hb.OK
    got = out[:, :p.n_written].cpu().numpy().view(np.uint32).T
    assert np.array_equal(_util.sorted_pairs(got), want.pairs)
    assert st.pair_comparisons == want.pair_comparisons
    request = [c[1:] for c in cl]
    want = _oracle(docs, [[b"\x01"] + c for c in request], cr, 1).pairs
    want = want[want[:, 0] > 0] - np.array([1, 0], np.uint32)
    with hb.Server(ctx, [plan], right) as srv:
        srv.submit(1, 0, request)
        srv.submit(2, 0, [c[:11] for c in request])
        got = {r["id"]: r["pairs"] for r in (srv.poll(20000), srv.poll(20000))}
    assert np.array_equal(got[1], want)
    assert np.array_equal(got[2], want[want[:, 0] < 11])


def test_memory_of_a_large_domain(built):
    """16 partitions x 1,001 x 1,001 keys, 500 left rows: 32 bytes a join key
    (histogram, cursor and offset of both tables, work items of the left)."""
    L = hb.lib()
    L.hbx_internal_pool_peak.restype = ctypes.c_uint64
    L.hbx_internal_pool_peak.argtypes = [ctypes.c_void_p, ctypes.c_int]
    cl, cr = _tables(500, 300, 1001, 9)
    for c in (cl, cr):
        c[4] = [b"%d" % (i % 1000) for i in range(len(c[4]))]
    cr[4][0] = b"k2"
    c = hb.Context(0)
    plan = hb.Plan.from_yaml([synth.rule_yaml([3, 4], [(1, 0.5)])], c)
    left, right = hb.Table.from_columns(cl, c), hb.Table.from_columns(cr, c)
    L.hbx_internal_pool_peak(c.h, 1)
    _, st = hb.block(c, plan, left, right, 16)
    assert 0 < L.hbx_internal_pool_peak(c.h, 0) < 33 * 16 * 1001 * 1001 + (300 << 20)
    c.close()
