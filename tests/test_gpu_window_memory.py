"""Windows of a streamed call build the dictionary of one equality at a time:
eight equalities instead of one take their columns and codes more, not seven
more tables."""
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
