"""The last head of a request to finish raises the residual window's length, which every CTA of every head has read before: each step's
rows of all heads go to one row of the window, however many CTAs share a head and whichever of them have a window tile."""
import pytest
import torch

from gpu_helpers import make_executor
from test_gpu_decode import both_caches, seeded_classes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hkv,cap", [(1, None), (2, None), (24, None), (24, 24), (24, 60), (24, 5), (2, 9)])
def test_rows_of_all_heads_go_to_one_row(hkv, cap, monkeypatch):
    pages, steps, hq = 60, 128, 2 * hkv
    _, cache, _, _, _ = both_caches(hkv, hq=hq, hkv=hkv, tokens=pages * 32, page=32, classes=seeded_classes(pages, 3), appends=1)
    if cap:
        monkeypatch.setenv("R2K_GRID_CAP", str(cap))
    ex, a = make_executor(cache, hq), cache.arenas
    g = torch.Generator(device="cuda").manual_seed(hkv)
    k, v = (torch.randn(steps, 1, hkv, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2))
    q = torch.randn(steps, 1, hq, 128, generator=g, device="cuda").to(torch.bfloat16)

    def run(wait):
        for t in (a.recent_k, a.recent_v):
            t.fill_(float("nan"))
        a.recent_len_device.zero_()
        a.recent_len = 0
        outs = torch.empty(steps, 1, hq, 130, device="cuda")
        torch.cuda.synchronize()
        for i in range(steps):
            ex.decode_state(q[i], out=outs[i], append=(k[i], v[i], i, 2 * i))
            a.recent_len = i + 1
            if wait:
                torch.cuda.synchronize()
                assert int(a.recent_len_device) == i + 1
        return outs

    want = run(True)
    got = run(False)
    assert torch.isfinite(want).all() and torch.equal(got, want)
    assert torch.equal(a.recent_k[0], k[:, 0].transpose(0, 1)) and torch.equal(a.recent_v[0], v[:, 0].transpose(0, 1))
    assert torch.equal(a.recent_global[0].cpu(), torch.arange(steps)) and torch.equal(a.recent_logical[0].cpu(), 2 * torch.arange(steps))
    assert int(a.recent_len_device) == steps and ex.device_status() == 0
