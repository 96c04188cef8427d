"""The one-launch cache build against the pack entry points it replaces (r2k_pack_*, r2k_gather_rows over token-index
arrays): every arena and index array bit for bit, at odd page counts, lengths and mixes; and the row transforms on
rows and tables that do not allow 16-byte accesses."""
import ctypes as C

import pytest
import torch

import r2omni_b200 as R
from oracle import sspa_oracle as O
from r2omni_b200 import _lib as L
from r2omni_b200.sspa.cache import dtype_code, tier_sorted_tokens

pytestmark = pytest.mark.gpu
RING = 128


def _plan(classes, lengths, positions=None):
    classes, lengths = torch.as_tensor(classes), torch.as_tensor(lengths)
    total = int(lengths.sum())
    pos = torch.arange(total) if positions is None else positions
    sel = lambda c: (classes == c).nonzero().flatten()  # noqa: E731
    return R.LayerCompressionPlan(
        layer_id=0, fp_pages=sel(1), int4_pages=sel(2), int2_pages=sel(5), evicted_pages=sel(0),
        protected_pages=torch.empty(0, dtype=torch.long), recent_fp_capacity=RING, logical_positions=pos,
        global_token_indices=pos * 3 + 1, page_offsets=lengths.cumsum(0) - lengths, page_lengths=lengths, page_classes=classes)


def _by_entry_points(key, value, plan, arenas, k_block, group):
    """What the separate launches write, in zeroed arenas of the same shapes."""
    out = {n: torch.zeros_like(getattr(arenas, n)) for n in ("k_packed", "k_scale", "k_zero", "fp_v", "i4_packed", "i4_scale",
                                                             "i2_packed", "i2_scale", "i2_zero")}
    fp, i4, i2, _ = (t.cuda() for t in tier_sorted_tokens(plan))
    lib, h, rows, dt = L.lib(), key.shape[0], C.c_int64(key.shape[1]), dtype_code(key.dtype)
    ptr, n64, zero, st = (lambda t: C.c_void_p(t.data_ptr())), C.c_int64, C.c_int64(0), C.c_void_p(torch.cuda.current_stream().cuda_stream)
    order = torch.cat((fp, i4, i2))
    if order.numel():
        L.check(lib.r2k_pack_k_int4(ptr(key), dt, h, rows, ptr(order), n64(order.numel()), ptr(out["k_packed"]), ptr(out["k_scale"]),
                                    ptr(out["k_zero"]), n64(out["k_packed"].shape[2]), k_block, zero, st), "k")
    if fp.numel():
        L.check(lib.r2k_gather_rows(ptr(value), h, rows, ptr(fp), n64(fp.numel()), ptr(out["fp_v"]), n64(fp.numel()), zero, st), "fp")
    if i4.numel():
        L.check(lib.r2k_pack_v_int4(ptr(value), dt, h, rows, ptr(i4), n64(i4.numel()), ptr(out["i4_packed"]), ptr(out["i4_scale"]),
                                    n64(i4.numel()), zero, st), "i4")
    if i2.numel():
        L.check(lib.r2k_pack_v_int2(ptr(value), dt, h, rows, ptr(i2), n64(i2.numel()), ptr(out["i2_packed"]), ptr(out["i2_scale"]),
                                    ptr(out["i2_zero"]), n64(out["i2_packed"].shape[2]), group, zero, st), "i2")
    torch.cuda.synchronize()
    return out


CASES = [   # page size, page lengths, page classes
    (16, [16, 3, 16, 0, 1, 16, 7], [5, 2, 1, 1, 2, 0, 5]),
    (32, [31], [2]),
    (32, [32] * 5, [0] * 5),
    (64, [64] * 9 + [1], [1, 2, 5, 2, 0, 5, 1, 2, 5, 1]),
    (64, [64, 64, 1], [5, 5, 5]),
    (16, [16] * 8 + [15] * 3, [1] * 11),
]


@pytest.mark.parametrize("page,lengths,classes", CASES)
@pytest.mark.parametrize("k_block,group,heads,dtype", [(32, 32, 2, torch.bfloat16), (64, 128, 1, torch.float16),
                                                       (128, 64, 3, torch.bfloat16)])
@pytest.mark.parametrize("form", ["plain", "scattered", "device", "special"])
def test_build_equals_the_pack_entry_points(page, lengths, classes, k_block, group, heads, dtype, form):
    total = sum(lengths)
    g = torch.Generator().manual_seed(total + heads)
    key, value = (torch.randn(heads, total, 128, generator=g).to(dtype) for _ in range(2))
    if form == "special":   # infinities, NaN, the type's lowest value, rows without any range
        for t in (key, value):
            t[:, 0, 5], t[:, total // 2, 7], t[:, total - 1, 9] = float("inf"), float("nan"), torch.finfo(dtype).min
            t[:, total // 3] = 0
    plan = _plan(classes, lengths, torch.randperm(total, generator=g) if form == "scattered" else None)
    if form == "device":
        for name in ("logical_positions", "global_token_indices", "page_offsets", "page_lengths", "page_classes"):
            object.__setattr__(plan, name, getattr(plan, name).cuda())
    key, value = key.cuda(), value.cuda()
    # memory that the cache's allocation is likely to reuse holds no zeros
    junk = torch.full((1 << 22,), 0xA5, dtype=torch.uint8, device="cuda")
    del junk
    cache = R.build_three_precision_cache(key, value, plan, page_size=page, key_quantization_superblock=k_block, int2_group_size=group,
                                          compact_key_append_capacity=200, recent_flush_size=128)
    a = cache.arenas
    want = _by_entry_points(key, value, plan, a, k_block, group)
    for name, t in want.items():
        assert torch.equal(getattr(a, name).view(torch.uint8), t.view(torch.uint8)), name
    fp, i4, i2, evicted = tier_sorted_tokens(plan)
    glob, logi = plan.global_token_indices.cpu(), plan.logical_positions.cpu()
    for name, rows in (("fp", fp), ("i4", i4), ("i2", i2)):
        for kind, source in (("global", glob), ("logical", logi)):
            got = getattr(a, f"{name}_{kind}")[0].cpu()
            assert torch.equal(got[:rows.numel()], source[rows]) and bool((got[rows.numel():] == -1).all()), (name, kind)
    assert torch.equal(a.evicted_global[0].cpu(), glob[evicted])
    assert int(a.recent_len_device) == 0 and not a.recent_k.any() and not a.recent_v.any() and not a.recent_page_lengths.any()
    assert bool((a.recent_global == -1).all()) and bool((a.recent_logical == -1).all())


def test_a_cache_without_tokens_is_cleared():
    empty = torch.empty(2, 0, 128, dtype=torch.bfloat16, device="cuda")
    for _ in range(2):
        junk = torch.full((1 << 22,), 0xA5, dtype=torch.uint8, device="cuda")
        del junk
        a = R.build_three_precision_cache(empty, empty, _plan(torch.empty(0, dtype=torch.long), torch.empty(0, dtype=torch.long)),
                                          page_size=32, compact_key_append_capacity=128).arenas
        assert int(a.recent_len_device) == 0 and bool((a.recent_global == -1).all())
        assert not a.k_packed.any() and not a.k_scale.any() and not a.i2_packed.any() and not a.recent_k.any()


def test_query_of_several_tokens_decodes_its_first():
    g = torch.Generator().manual_seed(5)
    key, value = (torch.randn(1, 96, 128, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    cache = R.build_three_precision_cache(key, value, _plan([2, 2, 5], [32, 32, 32]), page_size=32)
    ex = R.prepare_splitk_executor(cache, R.allocate_splitk_workspace(cache, num_query_heads=1))
    query = torch.randn(1, 1, 3, 128, generator=g).to(torch.bfloat16).cuda()
    assert torch.equal(ex(query).clone(), ex(query[:, :, 0]))


@pytest.mark.parametrize("sections", [(16, 24, 24), (15, 26, 23)])   # the second ends an axis inside an eight-channel word
@pytest.mark.parametrize("shift", [0, 4])                            # rows on 16-byte boundaries and 8 bytes off them
@pytest.mark.parametrize("batch,hq,hkv,tokens", [(1, 3, 1, 5), (3, 16, 2, 67), (1, 2, 1, 4099)])
def test_rotation_of_unaligned_rows_and_ragged_sections(sections, shift, batch, hq, hkv, tokens):
    g = torch.Generator().manual_seed(tokens + shift)

    def rows(heads):
        n = batch * heads * tokens * 128
        flat = torch.randn(n + 8, generator=g).to(torch.bfloat16).cuda()
        return flat[shift:shift + n].view(batch, heads, tokens, 128)

    q, k = rows(hq), rows(hkv)
    angle = torch.rand(3, batch, tokens, 128, generator=g) * 6.2831853
    cos, sin = angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)
    want = O.qk_mrope(q.cpu(), k.cpu(), cos, sin, sections, True)
    got = R.qwen_qk_mrope(q, k, cos.cuda(), sin.cuda(), sections, apply_hadamard=True)
    for a, b in zip(got, want):
        assert torch.equal(a.cpu().view(torch.int16), b.view(torch.int16))
    assert torch.equal(R.triton_fwht_128(k).cpu().view(torch.int16), R.triton_fwht_128(k.clone()).cpu().view(torch.int16))


@pytest.mark.parametrize("key_dtype,value_dtype", [(torch.bfloat16, torch.float16), (torch.float16, torch.bfloat16)])
def test_values_of_the_other_element_type(key_dtype, value_dtype):
    """Keys and values of different 16-bit types: each is read as what it is; bf16 pages hold the values rounded to the
    cache's (the keys') type."""
    lengths, classes = [16, 3, 16, 16, 1, 16, 7, 16], [5, 2, 1, 1, 2, 0, 5, 2]
    total, plan = sum(lengths), _plan(classes, lengths)
    g = torch.Generator().manual_seed(total)
    key = torch.randn(2, total, 128, generator=g).to(key_dtype).cuda()
    value = torch.randn(2, total, 128, generator=g).to(value_dtype).cuda()
    a = R.build_three_precision_cache(key, value, plan, page_size=16).arenas
    same = R.build_three_precision_cache(value, value, plan, page_size=16).arenas
    keys = R.build_three_precision_cache(key, key, plan, page_size=16).arenas
    for name in ("k_packed", "k_scale", "k_zero"):
        assert torch.equal(getattr(a, name), getattr(keys, name)), name
    for name in ("i4_packed", "i4_scale", "i2_packed", "i2_scale", "i2_zero"):
        assert torch.equal(getattr(a, name), getattr(same, name)), name
    fp = tier_sorted_tokens(plan)[0]
    assert a.fp_v.dtype == key_dtype and torch.equal(a.fp_v[0].cpu(), value.cpu()[:, fp].to(key_dtype))


def test_values_of_no_cache_type_are_refused():
    plan = _plan([2, 1], [16, 16])
    key = torch.zeros(1, 32, 128, dtype=torch.bfloat16, device="cuda")
    for value in (key.float(), key.double()):
        with pytest.raises(ValueError):
            R.build_three_precision_cache(key, value, plan, page_size=16)


def test_values_on_another_device_are_refused():
    plan = _plan([2, 1], [16, 16])
    key = torch.zeros(1, 32, 128, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(ValueError):
        R.build_three_precision_cache(key, key.cpu(), plan, page_size=16)


def _many_short_pages(n, page):
    lengths = torch.ones(n, dtype=torch.long)
    lengths[n // 2] = page   # one whole page between runs of one-token pages
    return lengths


def test_pages_of_one_token():
    n = 3000
    lengths = _many_short_pages(n, 64)
    lengths[::7] = 0
    classes = torch.tensor([2, 5, 1, 0, 2])[torch.arange(n) % 5]
    plan, total = _plan(classes, lengths), int(lengths.sum())
    key = torch.randn(1, total, 128, generator=torch.Generator().manual_seed(2)).to(torch.bfloat16).cuda()
    a = R.build_three_precision_cache(key, key, plan, page_size=64).arenas
    for name, t in _by_entry_points(key, key, plan, a, 32, 32).items():
        assert torch.equal(getattr(a, name).view(torch.uint8), t.view(torch.uint8)), name
    fp, i4, i2, evicted = tier_sorted_tokens(plan)
    for name, rows in (("fp", fp), ("i4", i4), ("i2", i2)):
        assert torch.equal(getattr(a, f"{name}_global")[0].cpu()[:rows.numel()], plan.global_token_indices[rows]), name


def test_build_time_does_not_grow_with_the_square_of_the_pages():
    """One-token pages cost a search per row, not a walk over the table: 262144 of them take less than 20 ms (2.5 measured,
    most of it host work; a walk of up to 262144 * 63 / 64 steps per row took 97.9)."""
    n = 262144
    plan = _plan(torch.full((n,), 2), torch.ones(n, dtype=torch.long))
    key = torch.zeros(1, n, 128, dtype=torch.bfloat16, device="cuda")
    times = []
    for _ in range(3):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        begin.record()
        R.build_three_precision_cache(key, key, plan, page_size=64)
        end.record()
        torch.cuda.synchronize()
        times.append(begin.elapsed_time(end))
    assert min(times) < 20.0, times


def test_pages_without_tokens_may_start_anywhere():
    plan = _plan([2, 1, 5], [16, 0, 16])
    object.__setattr__(plan, "page_offsets", torch.tensor([0, 4711, 16]))
    key = torch.randn(1, 32, 128, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    a = R.build_three_precision_cache(key, key, plan, page_size=16).arenas
    b = R.build_three_precision_cache(key, key, _plan([2, 1, 5], [16, 0, 16]), page_size=16).arenas
    assert torch.equal(a.k_packed, b.k_packed) and torch.equal(a.i2_packed, b.i2_packed) and torch.equal(a.i4_packed, b.i4_packed)


@pytest.mark.parametrize("mode", ["global", "thread_local", "relaxed"])
def test_build_is_refused_while_a_graph_is_captured(mode):
    """The page table is uploaded from a block that the call gives back: a replay would read whatever lies there then."""
    plan = _plan([2, 1], [16, 16])
    key = torch.zeros(1, 32, 128, dtype=torch.bfloat16, device="cuda")
    R.build_three_precision_cache(key, key, plan, page_size=16)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(torch.cuda.CUDAGraph(), capture_error_mode=mode):
            R.build_three_precision_cache(key, key, plan, page_size=16)
    torch.cuda.synchronize()
    assert int(R.build_three_precision_cache(key, key, plan, page_size=16).arenas.recent_len_device) == 0
