"""The entry point without allocation near the end of its 64 MiB: what the
encoder needs only while it runs is given back before the join is placed."""
import ctypes

import numpy as np
import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth
from tests import _util

pytestmark = pytest.mark.gpu


def test_many_rules_over_eight_strings(ctx):
    """57,000 left rows, eight string columns of eight characters and 16 rules
    over them: 57,432 rows were the most while the units and offsets of the
    left table's arenas lay below the right table's."""
    import torch

    cols = ", ".join(str(c) for c in range(10))
    docs = [synth.rule_yaml([1], [(2 + (c + q) % 8, 0.9) for c in range(8)])
            .replace("[0, 0, 1, 2, 3, 4]", f"[0, {cols}]").replace("[1, 0, 1, 2, 3, 4]", f"[1, {cols}]")
            for q in range(16)]
    rng = np.random.Generator(np.random.PCG64(16))

    def table(n):
        key = b"".join(b"%d" % (i % 10) for i in range(n))
        return hb.Table.from_columns(
            [(np.frombuffer(key, np.uint8), np.arange(n + 1))] * 2 +
            [(rng.integers(97, 99, size=8 * n, dtype=np.uint8), 8 * np.arange(n + 1)) for _ in range(8)], ctx)

    left, right = table(57_000), table(50)
    plan = hb.Plan.from_yaml(docs, ctx)
    want, _ = hb.block(ctx, plan, left, right, 1)
    assert len(want) > 0
    out = torch.empty((2, 1 << 16), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    p = hb.Pairs(out[0].data_ptr(), out[1].data_ptr(), 1 << 16, 0, 0)
    assert hb.lib().hbx_block_static(0, plan.h, left.h, right.h, 1, hb.INT_MAX, ctypes.byref(p),
                                     None, None) == hb.OK, hb.lib().hbx_static_last_error()
    got = out[:, :p.n_written].cpu().numpy().view(np.uint32).T
    assert np.array_equal(_util.sorted_pairs(got), _util.sorted_pairs(want))
