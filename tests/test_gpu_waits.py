"""What a block of a single-launch scan or of the pair sort does when its wait
for the blocks before it gives up: it counts what lies before it itself, and
the results are the same.  HBX_TEST_SCAN_GIVE_UP=1 lets every wait give up at
once; HBX_TEST_SORT_WIDE=1 sorts with the 64-bit words that 2^30 pairs take."""
import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from oracle import api, rules
from tests import _util

pytestmark = pytest.mark.gpu

DOCS = [synth.rule_yaml([3], [(1, 0.6)]), synth.rule_yaml([3, 4], [(1, 0.7), (2, 0.5)]),
        synth.rule_yaml([3], [(2, 0.8)])]


@pytest.fixture
def give_up(built, monkeypatch):
    monkeypatch.setenv("HBX_TEST_SCAN_GIVE_UP", "1")
    c = hb.Context(0)
    yield c
    c.close()


def _oracle(docs, cl, cr, n_part):
    plan = rules.serialize(rules.sort_rules([rules.decode_rule(rules.parse_yaml(d)) for d in docs]))
    return api.run_block(api.CTable(cl), api.CTable(cr), plan, n_part)


# chunks of the join's scans: one, two, 35 and (8,192 keys each) 104 a task
@pytest.mark.parametrize("n_keys", [4096, 4097, 35 * 4096, 104 * 8192])
@pytest.mark.parametrize("longest", [10, 300])
def test_join(give_up, n_keys, longest):
    cl, cr = _util.random_tables(n_keys, 300, 2000, b"abc", 10)
    n = n_keys // 4
    cr[3][1:] = [b"%d" % (i * 37 % n) for i in range(2000)]
    cl[3][1:] = [b"%d" % (n - 1 - 7 * i) if i % 2 else b"%d" % i for i in range(300)]
    for k in range(1, 300, 9):  # long left strings have keys of their own
        cl[1][k] = (cl[1][k] + b"abc" * 100)[:longest]
    for c in range(len(cr)):  # the right table lists every key
        cr[c] += [b"%d" % i for i in range(n - 1)] if c == 3 else [b"ab"] * (n - 1)
    want = _oracle(DOCS, cl, cr, 4)
    assert len(want.pairs) > 10
    plan = hb.Plan.from_yaml(DOCS, give_up)
    left, right = hb.Table.from_columns(cl, give_up), hb.Table.from_columns(cr, give_up)
    for mode in ("plain", "batched"):
        got, st = hb.block(give_up, plan, left, right, 4, _util.INT_MAX, mode)
        assert np.array_equal(_util.sorted_pairs(got), want.pairs), mode
        assert st.pair_comparisons == want.pair_comparisons, mode


def test_served_join_and_encoder(give_up):
    n = 9000
    _, cr = _util.random_tables(3, 5, n, b"abc", 12)
    cr[3][1:] = [b"%d" % (i % 4500) for i in range(n)]
    docs = [synth.rule_yaml([3], [(1, 0.3)])]
    request = [[c[1 + 97 * i % n] for i in range(40)] for c in cr]
    want = _oracle(docs, [[b"\x01"] + c for c in request], cr, 1).pairs
    want = want[want[:, 0] > 0] - np.array([1, 0], np.uint32)
    assert len(want) > 30
    with hb.Server(give_up, [hb.Plan.from_yaml(docs, give_up)], hb.Table.from_columns(cr, give_up)) as srv:
        srv.submit(1, 0, request)
        got = srv.poll(20000)
    assert got["status"] == hb.OK
    assert np.array_equal(got["pairs"], want)


# pairs around a tile of 2,048 (8 keys a thread) and of 4,096 (16), 32-bit
# words with 16 keys a thread only in the last of them
@pytest.mark.parametrize("n_l,n_r", [(1, 300), (2, 1024), (3, 683), (1, 4096), (17, 241), (129, 257),
                                     (2, 70001), (1201, 1101)])
@pytest.mark.parametrize("wide,polls", [("1", "0"), ("1", "1"), ("0", "1")])
def test_sort(built, monkeypatch, tmp_path, n_l, n_r, wide, polls):
    monkeypatch.setenv("HBX_TEST_SORT_WIDE", wide)
    monkeypatch.setenv("HBX_TEST_SCAN_GIVE_UP", polls)

    def write(path, n):
        path.write_text("".join(f"{i},a,a,k\n" for i in range(n)))
        return str(path)

    folder = tmp_path / "rules"
    folder.mkdir()
    (folder / "0.yaml").write_text(synth.rule_yaml([3], [(1, 0.0)]))
    out = tmp_path / "pairs.csv"
    assert hb.run_cli(["run_hyperblocker_exec", "-data_l", write(tmp_path / "l.csv", n_l), "-data_r",
                       write(tmp_path / "r.csv", n_r), "-rule_dir", str(folder), "-n_partitions", "1",
                       "-o", str(out)]) == 0
    got = np.array(out.read_bytes().replace(b"\n", b",").rstrip(b",").split(b","), dtype=np.int64)
    want = np.stack((np.repeat(np.arange(n_l), n_r), np.tile(np.arange(n_r), n_l)), 1)
    assert np.array_equal(got.reshape(-1, 2), want)
