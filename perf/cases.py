"""The work that users of the packed-KV path have it do, as timed cases.

Kinds of case:

* ``step``: one generated token through the attention of ``layers`` decoder layers: per layer a decode launch with
  its fused append and, when the residual window is full, the quantize-and-pack flush in front of it.
* ``shard``: the decode step of one rank's slice of a sequence-sharded cache (state, then merge).
* ``host``: a decode step whose query, new rows and result are in pinned host memory.
* ``block``: a decoder layer's attention block as the attention manager runs it (projections, rotation, append,
  attention, output projection).
* ``build``: packing the keys and values of a prefill into a cache.
* ``rotate``: rotating a prefill's query and key rows and transforming its value rows before they are packed.

Head shapes and cache sizes are the ones of ``bench.py`` and the tests.
"""
from __future__ import annotations

import types

import torch

import r2omni_b200 as R

D, RING = 128, 128
HORIZON = 512   # generated tokens a cache has room for; then the next request starts on the same prefilled cache
SECTIONS = (16, 24, 24)
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}


def _cache(**kw):
    """Cache options: page mix as shares of bf16, INT4 and evicted pages, the rest is INT2."""
    c = dict(batch=1, hq=16, hkv=2, tokens=4096, page=64, p_fp=0.25, p_i4=0.5, p_evict=0.0, k_block=32, v2_group=32,
             dtype="bf16", hadamard=False)
    c.update(kw)
    return c


def listed():
    return [
        # a short chat turn, one request: 36 layers, a few hundred cached tokens of an odd count; launches count
        dict(name="step_short_b1", kind="step", layers=36, **_cache(tokens=701, page=32)),
        # one request, 4096 INT4-value tokens: interactive use
        dict(name="step_4k_b1", kind="step", layers=36, **_cache(tokens=4096, page=32, p_fp=0.0, p_i4=1.0)),
        # a batch of eight 32K-token contexts, all three value formats: the ordinary serving step
        dict(name="step_32k_b8", kind="step", layers=4, **_cache(batch=8, tokens=32768)),
        # the wider model's head shape, sixteen 64K-token contexts: the largest launch
        dict(name="step_64k_b16", kind="step", layers=1, **_cache(batch=16, hq=28, hkv=4, tokens=65536)),
        # everything off the common path: fp16, seven heads a group, 16-token pages, coarse blocks, evicted pages, Hadamard
        dict(name="step_odd_b3_fp16", kind="step", layers=8,
             **_cache(batch=3, hq=28, hkv=4, tokens=9001, page=16, p_evict=0.1, k_block=64, v2_group=64, dtype="fp16",
                      hadamard=True)),
        # one million tokens of one request on one GPU: long audio/video sessions
        dict(name="shard_1m_b1", kind="shard", **_cache(tokens=1048576, p_fp=0.0)),
        # an eighth of it: one rank's slice on an eight-GPU box
        dict(name="shard_128k_b1", kind="shard", **_cache(tokens=131072, p_fp=0.0)),
        # a runtime that keeps its activations on the host
        dict(name="host_32k_b8", kind="host", **_cache(batch=8, tokens=32768)),
        # a layer's attention block in the batch-32 decoder
        dict(name="block_16k_b32", kind="block", hidden=2048, **_cache(batch=32, tokens=16384)),
        # the end of a 32K-token prefill: one layer's keys and values packed
        dict(name="build_32k", kind="build", **_cache(tokens=32768)),
        # the end of a short prompt's prefill
        dict(name="build_short_fp16", kind="build", **_cache(tokens=777, page=16, p_evict=0.1, dtype="fp16")),
        # rotation of a 16K-token prefill with Hadamard preconditioning
        dict(name="rotate_16k", kind="rotate", batch=1, hq=16, hkv=2, tokens=16384, dtype="bf16"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choices(("step", "shard", "host", "block", "build", "rotate"), (8, 2, 2, 2, 3, 2))[0]
    hq, hkv = rng.choice(((16, 2), (16, 2), (28, 4), (28, 4), (12, 2), (8, 2), (7, 1), (16, 4)))
    dtype = rng.choice(("bf16", "bf16", "bf16", "fp16"))
    if kind == "rotate":
        return dict(kind=kind, batch=rng.choice((1, 1, 2, 4)), hq=hq, hkv=hkv, tokens=_log(rng, 200, 16384), dtype=dtype)
    p_fp, p_i4 = rng.choice(((0.25, 0.5), (0.25, 0.5), (0.0, 1.0), (0.0, 0.5), (0.1, 0.3), (0.5, 0.5)))
    c = _cache(hq=hq, hkv=hkv, page=rng.choice((16, 32, 64)), p_fp=p_fp, p_i4=p_i4, p_evict=rng.choice((0.0, 0.0, 0.1)),
               k_block=rng.choice((32, 32, 32, 64, 128)), v2_group=rng.choice((32, 32, 32, 64, 128)), dtype=dtype)
    if kind == "build":
        c.update(tokens=_log(rng, 300, 65536))
    elif kind == "shard":
        c.update(tokens=_log(rng, 20000, 1048576 * 2 // hkv))
    else:
        # batch x tokens x kv heads within the largest listed launch
        c.update(batch=_log(rng, 1, 32))
        c.update(tokens=_log(rng, 300, min(131072, 16 * 65536 * 4 // (c["batch"] * hkv))))
    if kind == "step":
        small = c["batch"] * c["tokens"] * hkv
        c.update(layers=rng.randint(8, 36) if small < 40000 else rng.randint(2, 4) if small < 1000000 else 1,
                 hadamard=rng.random() < 0.25)
    elif kind == "block":
        c.update(hidden=hq * D)
    elif kind == "host":
        c.update(dtype="bf16")
    return dict(kind=kind, **c)


# ---------------------------------------------------------------- inputs
def _pages(case):
    """Page classes of a cache, the same for every seed, so that work() can count its tokens."""
    n = -(-case["tokens"] // case["page"])
    r = torch.rand(n, generator=torch.Generator().manual_seed(17))
    classes = torch.full((n,), 5)
    edge = case["p_evict"]
    for cls, share in ((0, 0.0), (1, case["p_fp"] * (1 - case["p_evict"])), (2, case["p_i4"] * (1 - case["p_evict"]))):
        classes[(r >= (0.0 if cls == 0 else edge)) & (r < edge + share)] = cls
        edge += share
    lengths = torch.full((n,), case["page"])
    lengths[-1] = case["tokens"] - (n - 1) * case["page"]
    return classes, lengths


def _plan(case):
    classes, lengths = _pages(case)
    pos = torch.arange(case["tokens"])
    sel = lambda c: (classes == c).nonzero().flatten()  # noqa: E731
    return R.LayerCompressionPlan(
        layer_id=0, fp_pages=sel(1), int4_pages=sel(2), int2_pages=sel(5), evicted_pages=sel(0),
        protected_pages=torch.empty(0, dtype=torch.long), recent_fp_capacity=RING, logical_positions=pos,
        global_token_indices=pos.clone(), page_offsets=torch.arange(classes.numel()) * case["page"], page_lengths=lengths,
        page_classes=classes)


def _kv(case, gen):
    """Keys with outlier channels (lognormal factors), normal values."""
    shape, dtype = (case["hkv"], case["tokens"], D), DTYPES[case["dtype"]]
    factor = torch.exp(torch.randn(case["hkv"], 1, D, generator=gen, device="cuda"))
    key = (torch.randn(shape, generator=gen, device="cuda") * factor).to(dtype)
    return key, torch.randn(shape, generator=gen, device="cuda").to(dtype)


def _build(case, key, value, plan):
    return R.build_three_precision_cache(key, value, plan, page_size=case["page"],
                                         key_quantization_superblock=case["k_block"], int2_group_size=case["v2_group"],
                                         compact_key_append_capacity=HORIZON, recent_flush_size=RING)


def _caches(case, gen, plan):
    return [_build(case, *_kv(case, gen), plan) for _ in range(case["batch"])]


def _executor(case, gen, plan):
    singles = [R.prepare_splitk_executor(c, R.allocate_splitk_workspace(c, num_query_heads=case["hq"]),
                                         output_hadamard=case["hadamard"]) for c in _caches(case, gen, plan)]
    return singles[0] if len(singles) == 1 else R.stack_homogeneous_splitk_executors(singles)


def _fill_window(case, arenas, gen):
    """A full residual window: the tokens generated since the last flush."""
    for t in (arenas.recent_k, arenas.recent_v):
        t.copy_(torch.randn(t.shape, generator=gen, device="cuda"))
    pos = torch.arange(case["tokens"], case["tokens"] + RING, device="cuda")
    arenas.recent_global.copy_(pos.expand_as(arenas.recent_global))
    arenas.recent_logical.copy_(pos.expand_as(arenas.recent_logical))
    arenas.recent_page_lengths.fill_(arenas.page_size)
    arenas.recent_len_device.fill_(RING)
    arenas.recent_len = RING


def _rows(case, gen, heads, host=False):
    x = torch.randn(case["batch"], heads, D, generator=gen, device="cuda").to(DTYPES[case["dtype"]])
    return x.cpu() if host else x


class _Layer:
    """One layer's executor, its inputs of a step and where its sequence began."""

    def __init__(self, case, gen, plan):
        self.executor = _executor(case, gen, plan)
        arenas = self.executor.arenas
        _fill_window(case, arenas, gen)
        self.base = (arenas.k_active, arenas.i2_active)
        self.query, self.key, self.value = (_rows(case, gen, h) for h in (case["hq"], case["hkv"], case["hkv"]))
        self.position = case["tokens"] + RING


def _begin_again(arenas, base):
    """The next request on the same prefilled cache: what was generated is dropped."""
    arenas.k_active, arenas.i2_active = base
    arenas.recent_len_device.zero_()
    arenas.recent_len = 0


def _make_room(arenas, base, stats):
    """Called with a full window: flush it, or start the next request when the horizon is reached."""
    if arenas.k_active + RING > base[0] + HORIZON:
        _begin_again(arenas, base)
    else:
        R.flush_recent(arenas, stats)


def _arena_outputs(a):
    names = ("k_packed", "k_scale", "k_zero", "i2_packed", "i2_scale", "i2_zero", "recent_k", "recent_v", "recent_len_device",
             "recent_global", "recent_logical", "recent_page_lengths", "i2_global", "i2_logical")
    return [getattr(a, n) for n in names]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    s = types.SimpleNamespace(case=case, kind=case["kind"], stats=R.DynamicCacheStats())
    if s.kind == "rotate":
        dtype = DTYPES[case["dtype"]]
        b, t = case["batch"], case["tokens"]
        s.query, s.key, s.value = (torch.randn(b, h, t, D, generator=gen, device="cuda").to(dtype)
                                   for h in (case["hq"], case["hkv"], case["hkv"]))
        angle = torch.rand(3, b, t, D // 2, generator=gen, device="cuda").mul_(6.2831853)
        angle = torch.cat((angle, angle), dim=-1)
        s.cos, s.sin = angle.cos().to(dtype), angle.sin().to(dtype)
        return s
    plan = _plan(case)
    if s.kind == "build":
        s.plan = plan
        s.key, s.value = _kv(case, gen)
    elif s.kind == "step":
        s.layers = [_Layer(case, gen, plan) for _ in range(case["layers"])]
    elif s.kind == "shard":
        s.executor = R.SequenceShardedExecutor(_executor(case, gen, plan))
        _fill_window(case, s.executor.local.arenas, gen)
        s.query = _rows(case, gen, case["hq"])
    elif s.kind == "host":
        s.layer = _Layer(case, gen, plan)
        rows = [_rows(case, gen, h, host=True).flatten() for h in (case["hq"], case["hkv"], case["hkv"])]
        s.host_in = torch.cat(rows).pin_memory()
        s.host_out = torch.empty(case["batch"], case["hq"], D, dtype=DTYPES[case["dtype"]]).pin_memory()
    elif s.kind == "block":
        _prepare_block(s, case, gen, plan)
    return s


def _prepare_block(s, case, gen, plan):
    dtype, hidden, b = DTYPES[case["dtype"]], case["hidden"], case["batch"]

    def linear(n_out, n_in):
        w = (torch.randn(n_out, n_in, generator=gen, device="cuda") * 0.02).to(dtype)
        return lambda x: torch.nn.functional.linear(x, w)

    s.module = types.SimpleNamespace(head_dim=D, qkv_proj=linear((case["hq"] + 2 * case["hkv"]) * D, hidden),
                                     o_proj=linear(hidden, case["hq"] * D))
    s.manager = R.PackedKVAttentionManager(num_query_heads=case["hq"], mrope_section=SECTIONS)
    s.layer = s.manager.adopt_layer(0, _caches(case, gen, plan), case["tokens"] + RING)
    s.arenas = s.layer.fourq_executor.arenas
    _fill_window(case, s.arenas, gen)
    s.base = (s.arenas.k_active, s.arenas.i2_active)
    s.hidden = torch.randn(b, 1, hidden, generator=gen, device="cuda").to(dtype)
    angle = torch.rand(3, b, 1, D // 2, generator=gen, device="cuda").mul_(6.2831853)
    angle = torch.cat((angle, angle), dim=-1)
    s.rotary = (angle.cos().to(dtype), angle.sin().to(dtype))


# ---------------------------------------------------------------- one pass
def run(s):
    if s.kind == "step":
        return _run_step(s)
    if s.kind == "shard":
        return s.executor(s.query)
    if s.kind == "host":
        layer = s.layer
        a = layer.executor.arenas
        if a.recent_len == a.recent_capacity:
            _make_room(a, layer.base, s.stats)
        layer.executor.step_host(s.host_in, s.host_out, append_indices=(layer.position, layer.position))
        if not layer.executor.batched:
            a.recent_len += 1
        layer.position += 1
        return [s.host_out] + _arena_outputs(a)
    if s.kind == "block":
        a = s.arenas
        if a.recent_len == a.recent_capacity:
            if a.k_active + RING > s.base[0] + HORIZON:
                _begin_again(a, s.base)
            else:
                s.manager.flush_if_full(0)
        out = s.manager.active_forward(0, s.module, s.hidden, s.rotary)
        return [out] + _arena_outputs(a)
    if s.kind == "build":
        a = _build(s.case, s.key, s.value, s.plan).arenas
        return [a.fp_v, a.i4_packed, a.i4_scale, a.fp_global, a.i4_global, a.evicted_global] + _arena_outputs(a)
    q, k = R.qwen_qk_mrope(s.query, s.key, s.cos, s.sin, SECTIONS, apply_hadamard=True)
    return [q, k, R.triton_fwht_128(s.value)]


def _run_step(s):
    outs = []
    for layer in s.layers:
        a = layer.executor.arenas
        if a.recent_len == a.recent_capacity:
            _make_room(a, layer.base, s.stats)
        outs.append(layer.executor(layer.query, append=(layer.key, layer.value, layer.position, layer.position)))
        if not layer.executor.batched:
            a.recent_len += 1
        layer.position += 1
    return outs + _arena_outputs(s.layers[0].executor.arenas)


# ---------------------------------------------------------------- what a pass cannot do without
def _pool_tokens(case):
    classes, lengths = _pages(case)
    return [int(lengths[classes == c].sum()) for c in (1, 2, 5, 0)]


def work(case):
    hq, hkv, b = case["hq"], case["hkv"], case["batch"]
    if case["kind"] == "rotate":
        rows = b * (hq + 2 * hkv) * case["tokens"]
        tables = 2 * b * case["tokens"] * D * 2   # each channel needs one of the three axes
        return {"bytes": rows * 512 + tables, "flops": rows * (7 * D + 4 * D)}
    n_fp, n_i4, n_i2, n_ev = _pool_tokens(case)
    kept = n_fp + n_i4 + n_i2
    k_meta, v_meta = 3 * D // case["k_block"], 3 * D // case["v2_group"]
    packed = kept * 64 + -(-kept // case["k_block"]) * 3 * D + n_fp * 256 + n_i4 * 68 + n_i2 * (32 + v_meta)
    if case["kind"] == "build":
        return {"bytes": hkv * (kept * 512 + packed), "flops": hkv * kept * D * 8}
    # attention over the packed tokens and, on average, a half-filled window
    ring = RING // 2 if case["kind"] != "shard" else RING
    moved = b * (hkv * (packed + ring * 512) + 4 * hq * D + 8 * hkv * D)
    # the window's quantization, once in RING tokens
    moved += b * hkv * (512 + 64 + k_meta + 32 + v_meta)
    flops = b * hq * (kept + ring) * D * 4
    if case["kind"] == "block":
        weights = case["hidden"] * D * (2 * hq + 2 * hkv)
        moved += weights * 2 + b * case["hidden"] * 4
        flops += 2 * b * weights
    layers = case.get("layers", 1)
    return {"bytes": layers * moved, "flops": layers * flops}


def tolerance(case):
    """Packed bytes, scales and copied rows are the same to the bit; attention and rotation results are rounded to
    16 bits (bf16 has 8 significant bits)."""
    if case["kind"] == "build":
        return "exact"
    if case["dtype"] == "fp16" and case["kind"] == "rotate":
        return {"rel": 1e-3}
    return {"rel": 5e-3}
