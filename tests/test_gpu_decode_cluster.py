"""The decode launch of small caches (few tiles per head, few heads: one cluster of eight CTAs per head, merged through
distributed shared memory) against the oracle and against the general launch, which a grid limit brings back."""
import ctypes as C

import pytest
import torch

import r2omni_b200 as R
from r2omni_b200 import _lib as L
from gpu_helpers import assert_close, make_executor
from oracle import sspa_oracle as O
from test_gpu_decode import both_caches, seeded_classes

pytestmark = pytest.mark.gpu


# from one tile in all (most of a cluster's CTAs idle) past the longest cache that takes clusters; one to eight heads;
# every group width at its ends
@pytest.mark.parametrize("hq,hkv,pages,page", [(16, 2, 1, 16), (16, 2, 3, 32), (7, 1, 11, 64), (2, 2, 20, 32), (28, 4, 16, 64),
                                               (4, 4, 37, 16), (16, 2, 64, 64), (16, 2, 100, 64), (5, 5, 16, 64), (8, 8, 12, 64)])
@pytest.mark.parametrize("dtype,hadamard", [(torch.bfloat16, False), (torch.float16, True)])
def test_small_caches_through_a_flush(hq, hkv, pages, page, dtype, hadamard, monkeypatch):
    tokens = pages * page
    ocache, gcache, new_k, new_v, queries = both_caches(31 + pages, hq=hq, hkv=hkv, tokens=tokens, page=page,
                                                        classes=seeded_classes(pages, pages), appends=131, dtype=dtype,
                                                        append_capacity=256)
    ex = make_executor(gcache, hq, output_hadamard=hadamard)
    stats = R.DynamicCacheStats()
    k, v, q = new_k.cuda(), new_v.cuda(), queries[0].cuda()
    for i in range(131):
        O.append_token(ocache, new_k[i], new_v[i], tokens + i, tokens + i)
        ring = gcache.recent_fp_pool
        if ring.active_length == ring.capacity:
            R.flush_recent(gcache.arenas, stats)
        ex(q, append=(k[i].unsqueeze(0).contiguous(), v[i].unsqueeze(0).contiguous(), tokens + i, tokens + i))
        ring.active_length += 1
        if i in (0, 63, 64, 127, 128, 130) and not hadamard:
            assert_close(ex.decode_f32(q), O.decode_fp32(queries[0].float(), ocache), f"step {i}")
    assert stats.flushed_tokens == 128 and int(gcache.arenas.recent_len_device) == ocache.recent_len
    assert torch.equal(gcache.arenas.recent_global[0, :3].cpu(), torch.arange(tokens + 128, tokens + 131))
    here = ex(queries[1].cuda()).float().clone()
    monkeypatch.setenv("R2K_GRID_CAP", str(7 * hkv))   # below eight CTAs per head: the general launch
    assert_close(here, ex(queries[1].cuda()).float(), "cluster against general launch")
    assert ex.device_status() == 0


def test_replayed_from_a_graph():
    pages = 12
    ocache, gcache, _, _, queries = both_caches(3, hq=16, hkv=2, tokens=pages * 64, page=64, classes=seeded_classes(pages, 3), appends=1)
    ex = make_executor(gcache, 16)
    q = queries[0].cuda()
    eager = ex(q).clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        ex(q)
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for _ in range(4):
            out = ex(q)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, eager)


@pytest.mark.parametrize("tail", [1, 2, 3, 13])   # INT4 pool lengths off multiples of four: scales of the later heads unaligned
@pytest.mark.parametrize("pages,cap", [(9, None), (70, None), (70, 4)])
def test_heads_behind_an_odd_int4_pool(tail, pages, cap, monkeypatch):
    page, heads = 16, 4
    lengths = torch.full((pages + 1,), page)
    lengths[-1] = tail
    classes = torch.cat((seeded_classes(pages, pages), torch.tensor([2])))
    total = int(lengths.sum())
    g = torch.Generator().manual_seed(total)
    key, value = (torch.randn(heads, total, 128, generator=g).to(torch.bfloat16).cuda() for _ in range(2))
    query = torch.randn(1, heads * 7, 128, generator=g).to(torch.bfloat16).cuda()
    sel = lambda c: (classes == c).nonzero().flatten()  # noqa: E731

    def decode(rows, q):
        plan = R.LayerCompressionPlan(
            layer_id=0, fp_pages=sel(1), int4_pages=sel(2), int2_pages=sel(5), evicted_pages=sel(0),
            protected_pages=torch.empty(0, dtype=torch.long), recent_fp_capacity=128, logical_positions=torch.arange(total),
            global_token_indices=torch.arange(total), page_offsets=torch.arange(pages + 1) * page, page_lengths=lengths,
            page_classes=classes)
        cache = R.build_three_precision_cache(key[rows].contiguous(), value[rows].contiguous(), plan, page_size=page)
        return make_executor(cache, q.shape[1]).decode_f32(q.contiguous())

    want = torch.cat([decode(slice(h, h + 1), query[:, 7 * h:7 * h + 7]) for h in range(heads)], dim=1)   # one head: its INT4 scales are aligned
    if cap:
        monkeypatch.setenv("R2K_GRID_CAP", str(cap))   # one CTA per head streams all of its tiles
    assert_close(decode(slice(None), query), want.cpu(), "all heads against one at a time")


@pytest.mark.parametrize("hq,hkv,pages,page,clusters", [(16, 2, 1, 16, True), (16, 2, 3, 32, True), (7, 1, 11, 64, True),
                                                        (28, 4, 16, 64, True), (16, 2, 64, 64, True), (5, 5, 16, 64, True),
                                                        (8, 8, 12, 64, True), (16, 2, 100, 64, False)])
def test_which_small_caches_take_clusters(hq, hkv, pages, page, clusters, monkeypatch):
    """The sizes of the tests above on this device: clusters up to about 5000 tokens x 2 heads, none with a grid limit."""
    _, gcache, _, _, _ = both_caches(31 + pages, hq=hq, hkv=hkv, tokens=pages * page, page=page, classes=seeded_classes(pages, pages),
                                     appends=1, append_capacity=256)

    def layout():
        ctas, cluster = C.c_int32(), C.c_int32()
        geom = gcache.arenas.geom(hq)
        L.check(L.lib().r2k_decode_plan(C.byref(geom), C.c_uint32(0), 1, 0, 0, C.byref(ctas), C.byref(cluster)), "r2k_decode_plan")
        return ctas.value, cluster.value

    assert (layout() == (8 * hkv, 8)) == clusters
    monkeypatch.setenv("R2K_GRID_CAP", str(7 * hkv))
    assert layout()[1] == 0


# Pool lengths and offsets off every power of two, INT2 metadata rows of one, two and four bytes (groups of 128, 64 and 32
# channels): rows of scales and zero points at every offset inside their 16-byte granules, in full and in ragged tiles
@pytest.mark.parametrize("group", [32, 64, 128])
@pytest.mark.parametrize("tails", [(1, 1, 1), (3, 7, 5), (16, 2, 13), (9, 16, 15)])   # rows of the last page of each pool
@pytest.mark.parametrize("pages,cap,dtype", [(9, None, torch.bfloat16), (130, None, torch.float16), (130, 3, torch.bfloat16)])
def test_odd_pools_against_the_oracle(group, tails, pages, cap, dtype, monkeypatch):
    page, heads = 16, 3
    lengths = torch.cat((torch.full((pages,), page), torch.tensor(tails)))
    classes = torch.cat((seeded_classes(pages, pages, 0.2, 0.35), torch.tensor([1, 2, 5])))
    total = int(lengths.sum())
    g = torch.Generator().manual_seed(total + group)
    key, value = (torch.randn(heads, total, 128, generator=g).to(dtype) for _ in range(2))
    query = torch.randn(1, heads * 5, 128, generator=g).to(dtype)
    offsets = lengths.cumsum(0) - lengths
    ocache = O.build_cache(key, value, classes, page_size=page, page_offsets=offsets, page_lengths=lengths, v2_group=group)
    sel = lambda c: (classes == c).nonzero().flatten()  # noqa: E731
    plan = R.LayerCompressionPlan(
        layer_id=0, fp_pages=sel(1), int4_pages=sel(2), int2_pages=sel(5), evicted_pages=sel(0),
        protected_pages=torch.empty(0, dtype=torch.long), recent_fp_capacity=128, logical_positions=torch.arange(total),
        global_token_indices=torch.arange(total), page_offsets=offsets, page_lengths=lengths, page_classes=classes)
    cache = R.build_three_precision_cache(key.cuda(), value.cuda(), plan, page_size=page, int2_group_size=group)
    if cap:
        monkeypatch.setenv("R2K_GRID_CAP", str(cap))   # one CTA per head streams all of its tiles
    got = make_executor(cache, heads * 5).decode_f32(query.cuda())
    assert_close(got, O.decode_fp32(query.float(), ocache, round_int4_values=False), "odd pools")
