"""A decode launch reads the packed pools before it waits for the kernel in front of it, and a rotation lets it in as soon as it has
come in itself.  So whatever writes the pools (a pack entry point, a flush, a build, a stacked copy) lets no launch in early:
writer, rotation and decode, queued together, give what they give one at a time.  The pools hold other values before."""
import ctypes as C

import pytest
import torch

import r2omni_b200 as R
from gpu_helpers import build_gpu_cache, make_executor
from r2omni_b200 import _lib as L
from r2omni_b200.sspa.cache import dtype_code, tier_sorted_tokens
from test_gpu_cache_build import _plan
from test_gpu_decode import seeded_classes

pytestmark = pytest.mark.gpu
HQ, HKV, PAGE = 16, 2, 32


def queue(wait):
    """The calls behind this one are all on the stream before the first of them starts (or run one at a time)."""
    torch.cuda.synchronize()
    if not wait:
        torch.cuda._sleep(40_000_000)


def settle(wait):
    if wait:
        torch.cuda.synchronize()


class Rows:
    """A step's projections and tables, and the buffers its rotated rows go to."""

    def __init__(self, seed, batch=1):
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.rows = [torch.randn(batch, h, 128, generator=g, device="cuda").to(torch.bfloat16) for h in (HQ, HKV, HKV)]
        angle = torch.rand(3, batch, 1, 128, generator=g, device="cuda")
        self.cos, self.sin = angle.cos(), angle.sin()
        self.made = tuple(torch.zeros(batch, h, 1, 128, device="cuda", dtype=torch.bfloat16) for h in (HQ, HKV, HKV))

    def rotate(self):
        q, k, v = R.qwen_qkv_prologue(*self.rows, self.cos, self.sin, (16, 24, 24), key_hadamard=True, value_hadamard=True, output=self.made)
        return q.squeeze(2), k.squeeze(2), v.squeeze(2)


def random_rows(seed, tokens):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return [torch.randn(HKV, tokens, 128, generator=g, device="cuda").to(torch.bfloat16) for _ in range(2)]


@pytest.mark.parametrize("last", ["keys", "values", "int4", "int2"])
@pytest.mark.parametrize("pages", [12, 700])   # a cluster per head, and the whole grid
def test_pack_entry_points(pages, last):
    tokens, steps = pages * PAGE, 6
    plan = _plan(seeded_classes(pages, 3), [PAGE] * pages)
    sources = [random_rows(s, tokens) for s in (1, 2)]
    cache = R.build_three_precision_cache(*sources[0], plan, page_size=PAGE)
    a, ex, rows = cache.arenas, make_executor(cache, HQ), Rows(3)
    fp, i4, i2, _ = (t.cuda() for t in tier_sorted_tokens(plan))
    order = torch.cat((fp, i4, i2))
    lib, n64, dt = L.lib(), C.c_int64, dtype_code(torch.bfloat16)
    ptr, zero = (lambda t: C.c_void_p(t.data_ptr())), C.c_int64(0)

    def repack(key, value, wait):
        st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
        writers = {
            "keys": lambda: lib.r2k_pack_k_int4(ptr(key), dt, HKV, n64(tokens), ptr(order), n64(tokens), ptr(a.k_packed), ptr(a.k_scale),
                                                ptr(a.k_zero), n64(a.k_packed.shape[2]), a.k_block, zero, st),
            "values": lambda: lib.r2k_gather_rows(ptr(value), HKV, n64(tokens), ptr(fp), n64(fp.numel()), ptr(a.fp_v), n64(fp.numel()), zero, st),
            "int4": lambda: lib.r2k_pack_v_int4(ptr(value), dt, HKV, n64(tokens), ptr(i4), n64(i4.numel()), ptr(a.i4_packed), ptr(a.i4_scale),
                                                n64(i4.numel()), zero, st),
            "int2": lambda: lib.r2k_pack_v_int2(ptr(value), dt, HKV, n64(tokens), ptr(i2), n64(i2.numel()), ptr(a.i2_packed), ptr(a.i2_scale),
                                                ptr(a.i2_zero), n64(a.i2_packed.shape[2]), a.v2_group, zero, st)}
        for name in [n for n in writers if n != last] + [last]:
            L.check(writers[name](), name)
            settle(wait)

    def run(wait):
        repack(*sources[1], True)
        outs = torch.zeros(steps, 1, HQ, 130, device="cuda")
        queue(wait)
        for i in range(steps):
            repack(*sources[i % 2], wait)
            q, _, _ = rows.rotate()
            settle(wait)
            ex.decode_state(q, out=outs[i])
            settle(wait)
        return outs

    want = run(True)
    assert torch.isfinite(want).all() and not torch.equal(want[0], want[1])
    assert torch.equal(run(False), want)


@pytest.mark.parametrize("pages", [12, 700])
def test_flush(pages):
    """A full window becomes packed rows, and the rotated step behind it attends to them."""
    tokens = pages * PAGE
    cache = build_gpu_cache(*random_rows(5, tokens), seeded_classes(pages, 5), page_size=PAGE, append_capacity=256)
    a, ex, rows = cache.arenas, make_executor(cache, HQ), Rows(7)
    g = torch.Generator(device="cuda").manual_seed(8)
    for t in (a.recent_k, a.recent_v):
        t.copy_(torch.randn(t.shape, generator=g, device="cuda"))
    a.recent_len = 128
    a.recent_len_device.fill_(128)
    before = {n: t.clone() for n, t in a.tensors().items()}
    lengths = a.k_active, a.i2_active, a.recent_len

    def run(wait):
        for n, t in a.tensors().items():
            t.copy_(before[n])
        a.k_active, a.i2_active, a.recent_len = lengths
        outs = torch.zeros(2, 1, HQ, 130, device="cuda")
        queue(wait)
        R.flush_recent(a, R.DynamicCacheStats())
        settle(wait)
        for i in range(2):
            q, k, v = rows.rotate()
            settle(wait)
            ex.decode_state(q, out=outs[i], append=(k, v, tokens + 128 + i, tokens + 128 + i))
            a.recent_len += 1
            settle(wait)
        return outs, {n: t.clone() for n, t in a.tensors().items()}

    (want, arenas), (got, arenas_got) = run(True), run(False)
    assert torch.isfinite(want).all() and torch.equal(got, want)
    assert a.recent_len == 2 and int(a.recent_len_device) == 2 and a.k_active == lengths[0] + 128
    for n, t in arenas.items():
        assert torch.equal(t.view(torch.uint8), arenas_got[n].view(torch.uint8)), n


@pytest.mark.parametrize("pages", [12, 700])
def test_build(pages):
    """Each cache takes the memory of the one before it."""
    tokens, steps = pages * PAGE, 4
    plan = _plan(seeded_classes(pages, 3), [PAGE] * pages)
    sources = [random_rows(s, tokens) for s in (1, 2)]
    rows, ws = Rows(3), None

    def run(wait):
        nonlocal ws
        cache = R.build_three_precision_cache(*sources[1], plan, page_size=PAGE)
        ws = ws or R.allocate_splitk_workspace(cache, num_query_heads=HQ)
        outs = torch.zeros(steps, 1, HQ, 130, device="cuda")
        queue(wait)
        for i in range(steps):
            ex = cache = None
            cache = R.build_three_precision_cache(*sources[i % 2], plan, page_size=PAGE)
            ex = R.prepare_splitk_executor(cache, ws)
            settle(wait)
            q, _, _ = rows.rotate()
            settle(wait)
            ex.decode_state(q, out=outs[i])
            settle(wait)
        torch.cuda.synchronize()
        return outs

    want = run(True)
    assert torch.isfinite(want).all() and not torch.equal(want[0], want[1])
    assert torch.equal(run(False), want)


@pytest.mark.parametrize("pages", [12, 300])
def test_copied_arenas(pages):
    """Arenas that a copy on the stream (as the one that stacks requests) has just written."""
    tokens, steps = pages * PAGE, 4
    classes = seeded_classes(pages, 3)
    images = [{n: t.clone() for n, t in build_gpu_cache(*random_rows(s, tokens), classes, page_size=PAGE).arenas.tensors().items()} for s in (1, 2)]
    cache = build_gpu_cache(*random_rows(4, tokens), classes, page_size=PAGE)
    a, ex, rows = cache.arenas, make_executor(cache, HQ), Rows(3)

    def run(wait):
        for n, t in a.tensors().items():
            t.copy_(images[1][n])
        outs = torch.zeros(steps, 1, HQ, 130, device="cuda")
        queue(wait)
        for i in range(steps):
            for n, t in a.tensors().items():
                t.copy_(images[i % 2][n])
            settle(wait)
            q, _, _ = rows.rotate()
            settle(wait)
            ex.decode_state(q, out=outs[i])
            settle(wait)
        return outs

    want = run(True)
    assert torch.isfinite(want).all() and not torch.equal(want[0], want[1])
    assert torch.equal(run(False), want)


def layers(cache, seed, steps):
    """Steps of rotation, shard state, merge and transform, each launch behind the one whose rows it reads."""
    sharded, rows = R.SequenceShardedExecutor(make_executor(cache, HQ)), [Rows(seed + i) for i in range(steps)]
    outs, turned = (torch.zeros(steps, 1, HQ, 128, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    a = cache.arenas

    def run(wait):
        for i in range(steps):
            q, k, v = rows[i].rotate()
            settle(wait)
            sharded.output = outs[i]   # nothing between a merge and the next step's launches
            sharded(q, append=(k, v, i, i))
            a.recent_len = i + 1
            settle(wait)
            R.triton_fwht_128(outs[i], output=turned[i])
            settle(wait)

    def clear():
        for t in (a.recent_k, a.recent_v, outs, turned):
            t.fill_(float("nan"))
        a.recent_len_device.zero_()
        a.recent_len = 0

    def result():
        torch.cuda.synchronize()
        assert int(a.recent_len_device) == steps
        return [t.clone() for t in (outs, turned, a.recent_k[:, :, :steps], a.recent_v[:, :, :steps])]

    return run, clear, result


@pytest.mark.parametrize("pages", [12, 700])
def test_steps_behind_each_other(pages):
    cache = build_gpu_cache(*random_rows(9, pages * PAGE), seeded_classes(pages, 9), page_size=PAGE)
    run, clear, result = layers(cache, 20, 24)
    results = []
    for wait in (True, False):
        clear()
        queue(wait)
        run(wait)
        results.append(result())
    for want, got in zip(*results):
        assert torch.isfinite(want.float()).all() and torch.equal(got, want)


@pytest.mark.parametrize("pages", [12, 700])
def test_steps_in_a_graph(pages):
    """The same launches captured: their early starts become edges of the graph."""
    cache = build_gpu_cache(*random_rows(9, pages * PAGE), seeded_classes(pages, 9), page_size=PAGE)
    run, clear, result = layers(cache, 20, 24)
    clear()
    run(True)
    want = result()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(False)
    for _ in range(2):
        clear()
        graph.replay()
        for one, other in zip(want, result()):
            assert torch.isfinite(one.float()).all() and torch.equal(other, one)


def test_captured_behind_joins_and_copies():
    """What stands in front of an early launch in a graph: a fill, a copy, two streams that meet, nothing at all."""
    tokens = 12 * PAGE
    cache = build_gpu_cache(*random_rows(9, tokens), seeded_classes(12, 9), page_size=PAGE)
    sharded, rows, side = R.SequenceShardedExecutor(make_executor(cache, HQ)), Rows(31), torch.cuda.Stream()
    source = [t.clone() for t in rows.rows]
    turned = torch.zeros(1, HQ, 128, device="cuda", dtype=torch.bfloat16)

    def front(kind):
        main = torch.cuda.current_stream()
        if kind == "copy":
            for t, s in zip(rows.rows, source):
                t.copy_(s)
        elif kind == "fill":
            for t in (*rows.made, sharded.state):
                t.zero_()
        elif kind == "join":
            side.wait_stream(main)
            with torch.cuda.stream(side):
                rows.rows[0].mul_(2)
            rows.rows[1].mul_(2)
            main.wait_stream(side)

    def steps():
        outs = []
        for kind in ("none", "copy", "join", "fill"):
            front(kind)
            q, _, _ = rows.rotate()
            front(kind)
            sharded.output = torch.empty(1, HQ, 128, device="cuda", dtype=torch.bfloat16)
            out = sharded(q)
            front(kind)
            outs += [out, R.triton_fwht_128(out, output=turned).clone()]
        return outs

    def reset():
        for t, s in zip(rows.rows, source):
            t.copy_(s)
        torch.cuda.synchronize()

    reset()
    want = [t.clone() for t in steps()]
    reset()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = steps()
    for _ in range(2):
        reset()
        graph.replay()
        torch.cuda.synchronize()
        for one, other in zip(want, got):
            assert torch.isfinite(one.float()).all() and torch.equal(one, other)


@pytest.mark.parametrize("pages", [12, 700])
def test_decode_directly_behind_a_build(pages):
    """No launch in between: each cache takes the memory of the one before it."""
    tokens, steps = pages * PAGE, 6
    plan = _plan(seeded_classes(pages, 3), [PAGE] * pages)
    sources, q = [random_rows(s, tokens) for s in (1, 2)], Rows(3).rows[0]
    ws = R.allocate_splitk_workspace(R.build_three_precision_cache(*sources[1], plan, page_size=PAGE), num_query_heads=HQ)

    def run(wait):
        outs = torch.zeros(steps, 1, HQ, 130, device="cuda")
        queue(wait)
        for i in range(steps):
            ex = cache = None
            cache = R.build_three_precision_cache(*sources[i % 2], plan, page_size=PAGE)
            settle(wait)
            ex = R.prepare_splitk_executor(cache, ws)
            ex.decode_state(q, out=outs[i])
            settle(wait)
        torch.cuda.synchronize()
        return outs

    want = run(True)
    assert torch.isfinite(want).all() and not torch.equal(want[0], want[1])
    assert torch.equal(run(False), want)
