"""A session whose buffers grow: after a growth that found no device memory the
next run has them again, and buffers that grew during a run on a caller's stream
outlive that stream."""
import ctypes

import pytest

import hyperblocker_gb300 as hb
from hyperblocker_gb300 import synth

pytestmark = pytest.mark.gpu

N_L, N_R = 900, 1200


@pytest.fixture
def session(built):
    """Two rules that both accept every pair: the set of reported pairs, of
    131,072 slots at first, grows to the 2 x 1,080,000 reports."""
    c = hb.Context(0, tile_right=96, eval_variant=2)
    plan = hb.Plan.from_yaml([synth.rule_yaml([3], [(1, 0.0)]), synth.rule_yaml([3], [(2, 0.0)])], c)

    def table(n):
        return hb.Table.from_columns([[b"%d" % i for i in range(n)], [b"a"] * n, [b"b"] * n, [b"k"] * n], c)

    s = hb.Session(c, plan, table(N_L), table(N_R))
    yield s
    s.close()
    c.close()


def _run(s, mode, stream=None):
    import torch

    out = torch.empty((2, N_L * N_R), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    n = s.run_device(mode, out[0].data_ptr(), out[1].data_ptr(), N_L * N_R, stream)
    keys = out[0, :n].long() * N_R + out[1, :n].long()
    return n, int(keys.unique().numel())


@pytest.mark.parametrize("mode", ["batched", "plain"])
def test_growth_without_memory(session, monkeypatch, mode):
    monkeypatch.setenv("HBX_TEST_ALLOC_LIMIT", str(4 << 20))
    for _ in range(2):
        with pytest.raises(hb.HbxError) as e:
            _run(session, mode)
        assert e.value.status == hb.ERR_OOM
    monkeypatch.delenv("HBX_TEST_ALLOC_LIMIT")
    for _ in range(2):
        assert _run(session, mode) == (N_L * N_R, N_L * N_R)


@pytest.mark.parametrize("mode", ["batched", "plain"])
def test_growth_on_a_stream_that_goes(session, mode):
    import torch

    torch.cuda.synchronize()  # the runtime is loaded
    rt = ctypes.CDLL("libcudart.so.%s" % torch.version.cuda.split(".")[0])
    stream = ctypes.c_void_p()
    assert rt.cudaStreamCreate(ctypes.byref(stream)) == 0
    assert _run(session, mode, stream.value) == (N_L * N_R, N_L * N_R)
    assert rt.cudaStreamDestroy(stream) == 0
    assert _run(session, mode) == (N_L * N_R, N_L * N_R)
