"""Left strings without a Peq table (k_eval_long): lengths at the table's end
(256), at the reference loops' last position, at the filters' limit (1,024)
and beyond, counts that do not fit a signature byte, and a long string in a
first, second or both columns, in every execution form, against the oracle."""
import ctypes

import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu

LENS = [0, 1, 16, 17, 100, 255, 256, 257, 258, 271, 272, 288, 300, 400, 512, 513, 1023, 1024, 1025,
        1100]
ONE = [synth.rule_yaml([3], [(1, 0.75), (2, 0.7)])]
# a group: its members share s1, add k2, and go on with s2 at their own thresholds
GROUP = [synth.rule_yaml([3], [(1, 0.9)]), synth.rule_yaml([3, 4], [(1, 0.8), (2, 0.72)]),
         synth.rule_yaml([4, 3], [(2, 0.85), (1, 0.7)]), synth.rule_yaml([4], [(2, 0.93)])]


def _tables(alphabet, n_l=110, n_r=150):
    rng = np.random.Generator(np.random.PCG64(len(alphabet)))
    base = bytes(rng.choice(list(alphabet), size=1200).tolist())

    def string():
        n = LENS[int(rng.integers(0, len(LENS)))]
        s = bytearray(base[:n]) if rng.random() < 0.5 else \
            bytearray(rng.choice(list(alphabet), size=n).tolist())
        for i in rng.integers(0, max(n, 1), size=n // 12):  # near copies pass
            s[int(i)] = alphabet[int(rng.integers(0, len(alphabet)))]
        return bytes(s)

    def table(n, prefix):
        return [[b"id"] + [f"{prefix}{i}".encode() for i in range(n)],
                [b"s1"] + [string() for _ in range(n)], [b"s2"] + [string() for _ in range(n)],
                [b"k1"] + [b"%d" % (i % 2) for i in range(n)],
                [b"k2"] + [b"%d" % int(x) for x in rng.integers(0, 2, size=n)]]

    return table(n_l, "l"), table(n_r, "r")


def _oracle(docs, cl, cr, n_part):
    plan = rules.serialize(rules.sort_rules([rules.decode_rule(rules.parse_yaml(d)) for d in docs]))
    return api.run_block(api.CTable(cl), api.CTable(cr), plan, n_part)


@pytest.mark.parametrize("alphabet", [b"ab", b"abcdefghijklmnopqrstuvwxyz ,"])
@pytest.mark.parametrize("docs", [ONE, GROUP])
def test_session_forms(ctx, docs, alphabet):
    cl, cr = _tables(alphabet)
    want = _oracle(docs, cl, cr, 2)
    assert len(want.pairs) > 50
    plan = hb.Plan.from_yaml(docs, ctx)
    left, right = hb.Table.from_columns(cl, ctx), hb.Table.from_columns(cr, ctx)
    for mode in ("plain", "batched"):
        got, st = hb.block(ctx, plan, left, right, 2, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
        assert st.pair_comparisons == want.pair_comparisons
        assert st.long_string_pairs > 0
    got, st = hb.block_streamed(ctx, plan, left, right, 2, 1 << 17)
    assert st.n_windows > 1
    assert np.array_equal(_util.sorted_pairs(got), want.pairs)


def test_host_encoding(built):
    cl, cr = _tables(b"ab")
    c = hb.Context(0, ingest=1)
    plan = hb.Plan.from_yaml(GROUP, c)
    got, _ = hb.block(c, plan, hb.Table.from_columns(cl, c), hb.Table.from_columns(cr, c), 3)
    assert np.array_equal(_util.sorted_pairs(got), _oracle(GROUP, cl, cr, 3).pairs)
    c.close()


@pytest.mark.parametrize("docs", [ONE, GROUP])
def test_serving_and_static(ctx, docs):
    import torch

    cl, cr = _tables(b"abcd")
    plan = hb.Plan.from_yaml(docs, ctx)
    right = hb.Table.from_columns(cr, ctx)
    request = [col[1:] for col in cl]  # records carry no header row
    want = _oracle(docs, [[b"\x01"] + c for c in request], cr, 1).pairs
    want = want[want[:, 0] > 0] - np.array([1, 0], np.uint32)
    with hb.Server(ctx, [plan], right) as srv:
        srv.submit(1, 0, request)
        srv.submit(2, 0, [c[:7] for c in request])
        got = {r["id"]: r["pairs"] for r in (srv.poll(20000), srv.poll(20000))}
    assert np.array_equal(got[1], want)
    assert np.array_equal(got[2], want[want[:, 0] < 7])
    out = torch.empty((2, 40000), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    p = hb.Pairs(out[0].data_ptr(), out[1].data_ptr(), 40000, 0, 0)
    st = hb.Stats()
    left = hb.Table.from_columns(cl, ctx)
    assert hb.lib().hbx_block_static(0, plan.h, left.h, right.h, 1, hb.INT_MAX, ctypes.byref(p),
                                     None, ctypes.byref(st)) == hb.OK
    got = out[:, :p.n_written].cpu().numpy().view(np.uint32).T
    assert np.array_equal(_util.sorted_pairs(got), _oracle(docs, cl, cr, 1).pairs)


@pytest.mark.parametrize("docs", [ONE, GROUP])
def test_more_pairs_than_the_list_of_deferred_ones_holds(ctx, docs):
    """Every pair passes a short first string and meets a long second one: 9,600 pairs for a list
    of 1,024 + 4 x 200; the others are decided in their lanes."""
    rng = np.random.Generator(np.random.PCG64(3))
    base = bytes(rng.choice(list(b"abcdefgh"), size=300).tolist())

    def table(n, prefix):
        s2 = [base[:257 + i % 40] + bytes(rng.choice(list(b"ab"), size=3 * (i % 9)).tolist())
              for i in range(n)]
        return [[b"id"] + [f"{prefix}{i}".encode() for i in range(n)],
                [b"s1"] + [b"abcd"] * n, [b"s2"] + s2,
                [b"k1"] + [b"1"] * n, [b"k2"] + [b"%d" % (i % 2) for i in range(n)]]

    cl, cr = table(80, "l"), table(120, "r")
    want = _oracle(docs, cl, cr, 1)
    assert len(want.pairs) > 1000
    plan = hb.Plan.from_yaml(docs, ctx)
    left, right = hb.Table.from_columns(cl, ctx), hb.Table.from_columns(cr, ctx)
    for mode in ("plain", "batched"):
        got, _ = hb.block(ctx, plan, left, right, 1, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
