"""Launches that come in while the kernel in front of them is still running (the state merge, the Hadamard transform): a chain of
them without a synchronisation gives what the same calls give one at a time."""
import pytest
import torch

import r2omni_b200 as R
from gpu_helpers import make_executor
from test_gpu_decode import both_caches, seeded_classes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pages", [4, 700])   # a cluster per head, and the whole grid
def test_state_and_merge_in_a_chain(pages):
    _, cache, new_k, new_v, _ = both_caches(11, hq=16, hkv=2, tokens=pages * 32, page=32, classes=seeded_classes(pages, 3), appends=40,
                                            append_capacity=256)
    ex = R.SequenceShardedExecutor(make_executor(cache, 16))
    queries = torch.randn(40, 1, 16, 128, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    k, v, a = new_k.cuda(), new_v.cuda(), cache.arenas

    def steps(wait):
        a.recent_len_device.zero_()
        a.recent_len = 0
        outs = []
        for i in range(40):   # each step attends to the rows that the steps before it appended
            out = ex(queries[i], append=(k[i:i + 1].contiguous(), v[i:i + 1].contiguous(), i, i))
            a.recent_len = i + 1
            outs.append(out.clone() if wait or i % 3 else out.float().to(out.dtype))
            if wait:
                torch.cuda.synchronize()
        return torch.stack(outs)

    want = steps(True)
    assert torch.equal(steps(False), want) and int(a.recent_len_device) == 40


@pytest.mark.parametrize("rows", [1, 15, 4096, 300000])
def test_transforms_in_a_chain(rows):
    x = torch.randn(rows, 128, generator=torch.Generator(device="cuda").manual_seed(rows), device="cuda").to(torch.bfloat16)
    want = x.clone()
    for _ in range(6):
        want = R.triton_fwht_128(want)
        torch.cuda.synchronize()
    got = x.clone()
    for _ in range(6):
        R.triton_fwht_128(got, output=got)   # in place: each reads what the one in front of it writes
    assert torch.equal(got, want)


@pytest.mark.parametrize("tokens", [1, 37, 9000])
def test_rotations_in_a_chain(tokens):
    """Each rotation reads what the launch in front of it (a rotation, a transform, a matrix product) has just written."""
    g = torch.Generator(device="cuda").manual_seed(tokens)
    q, k = (torch.randn(2, h, tokens, 128, generator=g, device="cuda").to(torch.bfloat16) for h in (7, 2))
    angle = torch.rand(3, 2, tokens, 128, generator=g, device="cuda")
    cos, sin = angle.cos().to(torch.bfloat16), angle.sin().to(torch.bfloat16)
    weight = torch.randn(128, 128, generator=g, device="cuda").to(torch.bfloat16) * 0.05

    def steps(wait):
        a, b = q, k
        for _ in range(5):
            for step in (lambda: R.qwen_qk_mrope(a, b, cos, sin, (16, 24, 24), apply_hadamard=True),
                         lambda: (torch.nn.functional.linear(a, weight), R.triton_fwht_128(b)),
                         lambda: R.qwen_qk_mrope(a, b, cos, sin, (16, 24, 24))):
                a, b = step()
                if wait:
                    torch.cuda.synchronize()
        return a, b

    for want, got in zip(steps(True), steps(False)):
        assert torch.equal(want, got)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("tokens", [1, 37, 9000])
def test_tables_written_in_front(tokens, dtype):
    """Each rotation takes its cosines from the rows that the rotation in front of it has just written, in buffers that held
    others before."""
    g = torch.Generator(device="cuda").manual_seed(tokens)
    q, k = ((1.6 * torch.rand(1, h, tokens, 128, generator=g, device="cuda") - 0.8).to(dtype) for h in (3, 1))
    # |row| <= 0.8 |cos| + 0.8 |sin| <= 0.8 |row in front| + 0.8: never above 4
    angle = torch.rand(3, 1, tokens, 128, generator=g, device="cuda")
    cos, sin = angle.cos().to(dtype), angle.sin().to(dtype)
    turns = [tuple(torch.empty_like(t) for t in (q, k)) for _ in range(3)]

    def steps(wait):
        table, rows = cos, []
        for i in range(9):   # three query heads: the table's three axes
            out = R.qwen_qk_mrope(q, k, table, sin, (16, 24, 24), output=turns[i % 3])
            table = out[0][0].unsqueeze(1)
            if wait:
                torch.cuda.synchronize()
            if i >= 6:
                rows.append(out[0].clone() if wait else out[0])
        return rows

    want = steps(True)
    for got, wanted in zip(steps(False), want):
        assert torch.isfinite(wanted).all() and torch.equal(got, wanted)


def test_query_and_new_rows_written_in_front():
    """Decode launches whose query and appended rows the rotation in front of each has just written."""
    pages, steps = 40, 24
    _, cache, _, _, _ = both_caches(11, hq=16, hkv=2, tokens=pages * 32, page=32, classes=seeded_classes(pages, 3), appends=1,
                                    append_capacity=256)
    ex, a = make_executor(cache, 16), cache.arenas
    g = torch.Generator(device="cuda").manual_seed(5)
    rows = [torch.randn(steps, 1, h, 128, generator=g, device="cuda").to(torch.bfloat16) for h in (16, 2, 2)]
    angle = torch.rand(steps, 3, 1, 1, 128, generator=g, device="cuda")
    cos, sin = angle.cos(), angle.sin()
    made = tuple(torch.empty(1, h, 1, 128, device="cuda", dtype=torch.bfloat16) for h in (16, 2, 2))   # rows take the place of the last step's

    def run(wait):
        for t in (a.recent_k, a.recent_v):
            t.fill_(float("nan"))
        a.recent_len_device.zero_()
        a.recent_len = 0
        outs = torch.empty(steps, 1, 16, 130, device="cuda")
        torch.cuda.synchronize()
        for i in range(steps):
            q, k, v = R.qwen_qkv_prologue(*(t[i] for t in rows), cos[i], sin[i], (16, 24, 24), key_hadamard=True, value_hadamard=True, output=made)
            if wait:
                torch.cuda.synchronize()
            ex.decode_state(q.squeeze(2), out=outs[i], append=(k.squeeze(2), v.squeeze(2), i, i))
            a.recent_len = i + 1
            if wait:
                torch.cuda.synchronize()
        return outs, a.recent_k[:, :, :steps].clone(), a.recent_v[:, :, :steps].clone()

    for want, got in zip(run(True), run(False)):
        assert torch.isfinite(want).all() and torch.equal(got, want)
    assert int(a.recent_len_device) == steps
