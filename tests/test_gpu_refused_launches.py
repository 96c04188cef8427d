"""A launch that the runtime refuses is reported by its own call and by no later one."""
import ctypes as C

import pytest
import torch

from r2omni_b200 import _lib as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("refused", ["transform", "rotation", "merge", "rows"])
def test_next_call_does_not_report_it(refused):
    rt = pytest.importorskip("cuda.bindings.runtime")
    lib, done = L.lib(), rt.cudaError_t.cudaSuccess
    heads, tokens = 2, 32
    x = torch.randn(1, heads, tokens, 128, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    out, other, tables, states = torch.zeros_like(x), torch.zeros_like(x), torch.zeros(3, 1, tokens, 128, device="cuda"), torch.zeros(4, 130, device="cuda")
    index = torch.arange(tokens - 1, -1, -1, device="cuda")
    ptr, n64 = (lambda t: C.c_void_p(t.data_ptr())), C.c_int64
    strides = (C.c_int64 * 4)(*tables.stride())
    calls = {
        "transform": lambda st: lib.r2k_fwht128(ptr(x), ptr(out), L.DTYPE_BF16, n64(heads * tokens), st),
        "rotation": lambda st: lib.r2k_qk_mrope(ptr(x), ptr(x), ptr(out), ptr(other), L.DTYPE_BF16, 1, heads, heads, tokens, ptr(tables), ptr(tables), 2,
                                                strides, strides, 16, 24, 0, st),
        "merge": lambda st: lib.r2k_merge_states(ptr(states), 1, n64(4 * 130), 4, L.DTYPE_BF16, ptr(out), C.c_uint32(0), st),
        "rows": lambda st: lib.r2k_gather_rows(ptr(x), heads, n64(tokens), ptr(index), n64(tokens), ptr(out), n64(tokens), n64(0), st)}
    plain = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    for call in calls.values():   # whatever a first call sets up
        assert call(plain) == L.OK
    torch.cuda.synchronize()

    # a stream whose capture has been given up (it was waited for meanwhile) takes no launch
    side = torch.cuda.Stream()
    assert rt.cudaStreamBeginCapture(side.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeRelaxed)[0] == done
    assert rt.cudaStreamSynchronize(side.cuda_stream)[0] != done
    status = calls[refused](C.c_void_p(side.cuda_stream))
    assert rt.cudaStreamEndCapture(side.cuda_stream)[0] != done
    rt.cudaGetLastError()
    assert status == L.ERR_CUDA

    out.zero_()
    assert calls["rows"](plain) == L.OK
    assert torch.equal(out, x.flip(2))
