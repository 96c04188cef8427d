"""Small caches (one cluster of CTAs per head) fetch the residual window whole, whatever its length: rows behind the last one must
not reach the result, whatever they hold."""
import pytest
import torch

from gpu_helpers import assert_close, build_gpu_cache, make_executor
from oracle import sspa_oracle as O
from test_gpu_decode import both_caches, seeded_classes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("length", [0, 1, 15, 16, 17, 63, 64, 65, 80, 127, 128])
def test_rows_behind_the_window_do_not_count(length, dtype):
    pages, heads = 9, 3
    _, cache, new_k, new_v, queries = both_caches(7, hq=5 * heads, hkv=heads, tokens=pages * 32, page=32,
                                                  classes=seeded_classes(pages, 3), appends=128, dtype=dtype, append_capacity=256)
    ex = make_executor(cache, 5 * heads)
    a, q = cache.arenas, queries[0].cuda()
    rows_k, rows_v = (t.transpose(0, 1).unsqueeze(0).cuda() for t in (new_k, new_v))   # [1, heads, 128, 128]

    def fill(rest):
        a.recent_k.fill_(rest)
        a.recent_v.fill_(rest)
        a.recent_k[:, :, :length], a.recent_v[:, :, :length] = rows_k[:, :, :length], rows_v[:, :, :length]
        a.recent_len_device.fill_(length)
        a.recent_len = length

    fill(0.0)
    want = ex.decode_f32(q).clone()
    fill(float("nan"))
    assert torch.isfinite(want).all() and torch.equal(ex.decode_f32(q), want)
    if length < 128:   # the appended row takes the place of the first of them
        outs = []
        for rest in (0.0, float("nan")):
            fill(rest)
            step = (new_k[length].unsqueeze(0).cuda().contiguous(), new_v[length].unsqueeze(0).cuda().contiguous(), 500, 500)
            outs.append(ex(q, append=step).clone())
            assert int(a.recent_len_device) == length + 1
            assert torch.equal(a.recent_k[:, :, length], rows_k[:, :, length]) and torch.equal(a.recent_v[:, :, length], rows_v[:, :, length])
        assert torch.isfinite(outs[0].float()).all() and torch.equal(outs[0], outs[1])
    assert ex.device_status() == 0


@pytest.mark.parametrize("ring", [192, 1024])   # three tiles, and more than a cluster has CTAs
@pytest.mark.parametrize("length", [0, 1, 63, 64, 65, 128, 150, 191])
def test_long_windows_of_small_caches(length, ring):
    """Windows of more than two tiles come without the tiles behind their length; the appended row may open a tile."""
    pages, heads = 9, 3
    g = torch.Generator().manual_seed(ring + length)
    key, value = (torch.randn(heads, pages * 32, 128, generator=g).to(torch.bfloat16) for _ in range(2))
    rows_k, rows_v = (torch.randn(1, heads, length + 1, 128, generator=g).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(1, 5 * heads, 128, generator=g).to(torch.bfloat16)
    classes = seeded_classes(pages, 3)
    ocache = O.build_cache(key, value, classes, page_size=32, recent_capacity=ring, append_capacity=256)
    cache = build_gpu_cache(key, value, classes, page_size=32, recent_capacity=ring, append_capacity=256)
    a, ex = cache.arenas, make_executor(cache, 5 * heads)
    for t, rows in ((a.recent_k, rows_k), (a.recent_v, rows_v)):
        t.fill_(float("nan"))
        t[:, :, :length] = rows[:, :, :length].cuda()
    for i in range(length):
        O.append_token(ocache, rows_k[0, :, i], rows_v[0, :, i], 500 + i, 500 + i)
    a.recent_len_device.fill_(length)
    a.recent_len = length
    assert_close(ex.decode_f32(q.cuda()), O.decode_fp32(q.float(), ocache), "window")
    O.append_token(ocache, rows_k[0, :, length], rows_v[0, :, length], 900, 900)
    step = tuple(t[:, :, length].cuda().contiguous() for t in (rows_k, rows_v))
    assert_close(ex.decode_f32(q.cuda(), append=(*step, 900, 900)), O.decode_fp32(q.float(), ocache), "appended")
    assert int(a.recent_len_device) == length + 1 and torch.equal(a.recent_k[:, :, length], step[0]) and torch.equal(a.recent_v[:, :, length], step[1])
    assert ex.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("heads,cap", [(3, 3), (3, 20), (24, None)])   # a CTA per head, several, a grid of more heads than clusters
@pytest.mark.parametrize("length", [0, 1, 15, 16, 17, 63, 64, 65, 127])
def test_rows_behind_the_window_of_the_general_launch(length, heads, cap, dtype, monkeypatch):
    """A window's tile comes whole in every launch, and the memory behind its last row is the caller's."""
    pages = 9
    _, cache, new_k, new_v, queries = both_caches(7, hq=5 * heads, hkv=heads, tokens=pages * 32, page=32,
                                                  classes=seeded_classes(pages, 3), appends=length + 1, dtype=dtype, append_capacity=256)
    if cap:
        monkeypatch.setenv("R2K_GRID_CAP", str(cap))
    ex, a, q = make_executor(cache, 5 * heads), cache.arenas, queries[0].cuda()
    rows = [t.transpose(0, 1).unsqueeze(0)[:, :, :length].cuda() for t in (new_k, new_v)]
    step = (new_k[length].unsqueeze(0).cuda().contiguous(), new_v[length].unsqueeze(0).cuda().contiguous(), 500, 500)
    for append in (None, step):
        outs = []
        for rest in (0.0, float("inf"), float("nan")):
            for t, r in zip((a.recent_k, a.recent_v), rows):
                t.fill_(rest)
                t[:, :, :length] = r
            a.recent_len_device.fill_(length)
            a.recent_len = length
            outs.append(ex.decode_f32(q, append=append).clone())
        assert torch.isfinite(outs[0]).all() and torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    assert ex.device_status() == 0
