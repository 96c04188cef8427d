"""What a prepared executor keeps between calls, on the CPU: a stand-in for the native step call records what it is made
from and launched with.  Nothing here touches a GPU."""
import types

import pytest
import torch

from r2omni_b200 import build
from r2omni_b200.sspa import executor as X
from r2omni_b200.sspa.cache import PackedArenas


def _arenas(heads=1, tokens=128):
    z = lambda *s, dtype=torch.uint8: torch.zeros(s, dtype=dtype)  # noqa: E731
    i64 = lambda n: z(1, n, dtype=torch.int64)  # noqa: E731
    return PackedArenas(
        dtype=torch.bfloat16, page_size=32, k_block=32, v2_group=32, flush=128, k_packed=z(1, heads, 256, 64),
        k_scale=z(1, heads, 8, 128, dtype=torch.float16), k_zero=z(1, heads, 8, 128), k_active=tokens, k_offsets=(0, 0, tokens),
        fp_v=z(1, heads, 0, 128, dtype=torch.bfloat16), i4_packed=z(1, heads, tokens, 64),
        i4_scale=z(1, heads, tokens, 1, dtype=torch.float32), i2_packed=z(1, heads, 128, 32),
        i2_scale=z(1, heads, 128, 4, 1, dtype=torch.float16), i2_zero=z(1, heads, 128, 4, 1), i2_active=0,
        recent_k=z(1, heads, 128, 128, dtype=torch.bfloat16), recent_v=z(1, heads, 128, 128, dtype=torch.bfloat16),
        recent_len_device=z(1, dtype=torch.int32), recent_global=i64(128), recent_logical=i64(128), recent_page_lengths=i64(4),
        recent_len=0, i2_global=i64(128), i2_logical=i64(128), fp_global=i64(0), fp_logical=i64(0), i4_global=i64(tokens),
        i4_logical=i64(tokens), evicted_global=i64(0))


@pytest.fixture
def prepared(monkeypatch):
    made, used = [], []

    class Step:
        def __init__(self, *args):
            made.append(self)

        def plain(self, *args):
            used.append((self, args))

        append = plain

    monkeypatch.setattr(X, "host", lambda: types.SimpleNamespace(Step=Step))
    monkeypatch.setattr(X, "_stream_ptr", lambda device: 0)
    ws = X.SplitKWorkspace(torch.zeros(1024, dtype=torch.uint8), torch.zeros(1, 2, 128, dtype=torch.bfloat16), None, 128, 1, 2)
    ex = X.SplitKExecutor(_arenas(), ws)
    ex._decode = lambda *args: 0
    ex._decode_host = lambda *args: 0
    return ex, made, used


@pytest.mark.parametrize("between", ["nothing", "decode_f32", "decode_state", "step_host"])
def test_native_step_follows_a_renewed_view_whoever_sees_it_first(prepared, between):
    ex, made, used = prepared
    query = torch.zeros(1, 2, 128, dtype=torch.bfloat16)
    ex(query)
    ex.arenas.k_packed = ex.arenas.k_packed.clone()
    ex.arenas._view = None   # the tensors' addresses are taken again
    if between == "step_host":
        ex.step_host(query.flatten(), torch.empty_like(query))
    elif between != "nothing":
        getattr(ex, between)(query)
    ex(query)
    assert len(made) == 2 and used[-1][0] is made[1], "launched with the addresses of the old view"
    ex(query)
    assert len(made) == 2


def test_host_step_takes_the_addresses_its_tensors_have_now(prepared):
    ex, _, _ = prepared
    calls = []
    ex._decode_host = lambda *args: calls.append(args) or 0
    host_in, host_out = torch.zeros(256, dtype=torch.bfloat16), torch.zeros(1, 2, 128, dtype=torch.bfloat16)
    ex.step_host(host_in, host_out)
    ex.step_host(host_in, host_out)
    moved_in, moved_out = torch.zeros(512, dtype=torch.bfloat16), torch.zeros(1, 2, 128, dtype=torch.bfloat16)
    host_in.set_(moved_in)
    host_out.set_(moved_out)
    ex.step_host(host_in, host_out)
    assert [c[2] for c in calls[1:]] == [calls[0][2], moved_in.data_ptr()]
    assert [c[8] for c in calls[1:]] == [calls[0][8], moved_out.data_ptr()]
    host_out.resize_(1, 2, 64)
    with pytest.raises(ValueError):
        ex.step_host(host_in, host_out)


def test_host_module_of_another_torch_or_python_is_stale(monkeypatch):
    build.build_library()
    assert not build.host_stale()
    monkeypatch.setattr(torch, "__version__", torch.__version__ + ".other")
    assert build.host_stale()
