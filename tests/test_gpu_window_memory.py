"""Device memory of a streamed call's windows: no more than window_bytes and what
hbx.h says comes on top; the dictionary of one equality at a time, so that eight
equalities instead of one take their columns and codes more, not seven more
tables."""
import ctypes

import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth

pytestmark = pytest.mark.gpu

N_L, N_R = 10, 132_000  # a dictionary has 2^19 slots, 16 bytes each


def _peak(c, slots):
    """Most device memory of a window over all rows (few pairs: small output)."""
    cols = ", ".join(str(k) for k in range(10))
    doc = synth.rule_yaml(list(range(2, 2 + slots)), [(1, 0.9)]) \
        .replace("[0, 0, 1, 2, 3, 4]", f"[0, {cols}]").replace("[1, 0, 1, 2, 3, 4]", f"[1, {cols}]")

    def table(n):
        rng = np.random.Generator(np.random.PCG64(n))
        key = [(rng.integers(48, 50, size=n, dtype=np.uint8), np.arange(n + 1)) for _ in range(9)]
        return hb.Table.from_columns(
            [key[0], (rng.integers(97, 117, size=4 * n, dtype=np.uint8), 4 * np.arange(n + 1))] + key[1:], c)

    left, right = table(N_L), table(N_R)
    plan = hb.Plan.from_yaml([doc], c)
    _, st = hb.block_streamed(c, plan, left, right, 1, 40 << 20)
    assert st.n_windows == 1
    f = hb.lib().hbx_internal_window_peak
    f.restype, f.argtypes = ctypes.c_uint64, [ctypes.c_void_p]
    return f(c.h)


def test_one_dictionary_at_a_time(built):
    c = hb.Context(0)
    one, eight = _peak(c, 1), _peak(c, 8)
    # a column more: 1 byte, its 8-byte offset and a 4-byte code a row
    assert eight - one <= 7 * 13 * (N_L + N_R) + (4 << 20)
    c.close()


@pytest.mark.parametrize("n_rules", [1, 3])
@pytest.mark.parametrize("longest", [24, 200, 300])
@pytest.mark.parametrize("window", [1 << 22, 1 << 26])
def test_window_bytes_and_what_comes_on_top(built, n_rules, longest, window):
    rng = np.random.Generator(np.random.PCG64(longest))
    n_l, n_r, n_keys, n_part = 8000, 12000, 300, 5

    def table(n):
        def strings():
            size = np.where(rng.random(n) < 0.1, longest, rng.integers(1, 24, size=n))
            off = np.concatenate(([0], np.cumsum(size))).astype(np.int64)
            return rng.integers(97, 117, size=int(off[-1]), dtype=np.uint8), off
        key = b"".join(b"%03d" % int(x) for x in rng.integers(0, n_keys, size=n))
        return hb.Table.from_columns([(np.frombuffer(key, np.uint8), 3 * np.arange(n + 1)), strings(), strings(),
                                      (np.frombuffer(key, np.uint8), 3 * np.arange(n + 1)),
                                      (np.frombuffer(key, np.uint8), 3 * np.arange(n + 1))])

    docs = [synth.rule_yaml([3], [(1, 0.9)]), synth.rule_yaml([4], [(2, 0.9)]),
            synth.rule_yaml([3], [(2, 0.8), (1, 0.8)])][:n_rules]
    c = hb.Context(0)
    _, st = hb.block_streamed(c, hb.Plan.from_yaml(docs, c), table(n_l), table(n_r), n_part, window)
    assert (st.n_windows == 1) == (window == 1 << 26)
    f = hb.lib().hbx_internal_window_peak
    f.restype, f.argtypes = ctypes.c_uint64, [ctypes.c_void_p]
    pairs = max(window // 8, 1 << 16)
    on_top = (pairs * (8 + (32 if n_rules > 1 else 0))  # output, set of reported pairs
              + 32 * 21 * n_l * 2  # masks: 20 symbols and the padding, two strings
              + 32 * n_part * (n_keys + 1) * n_rules  # key states
              + 64 * (n_l + n_r) + 64 * n_r * n_rules)  # a dictionary, records in join order
    assert 0 < f(c.h) <= window + on_top + (2 << 20)
    c.close()
