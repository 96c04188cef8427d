"""The one-launch cache build where its eight-row warps meet pool ends and the last token, and its bookkeeping where a page's token
indices are consecutive but for one."""
import dataclasses

import pytest
import torch

import r2omni_b200 as R
from r2omni_b200.sspa.cache import tier_sorted_tokens
from test_gpu_cache_build import _by_entry_points, _plan

pytestmark = pytest.mark.gpu


def _pools(fp, i4, i2):
    lengths, classes = [], []
    for cls, n in ((5, i2), (2, i4), (1, fp)):   # the order of the pools is not that of the pages
        while n > 0:
            lengths.append(min(16, n))
            classes.append(cls)
            n -= 16
    return lengths, classes


@pytest.mark.parametrize("rows", [(8, 8, 8), (7, 9, 16), (1, 1, 1), (0, 0, 7), (128, 120, 8), (4, 4, 121), (129, 7, 0), (0, 3, 5), (16, 0, 113),
                                  (3, 250, 4)])
@pytest.mark.parametrize("k_block,group,dtype", [(32, 32, torch.bfloat16), (64, 64, torch.float16), (128, 128, torch.bfloat16)])
def test_pools_that_end_inside_a_warp(rows, k_block, group, dtype):
    lengths, classes = _pools(*rows)
    g = torch.Generator().manual_seed(sum(rows))
    key, value = (torch.randn(2, sum(lengths), 128, generator=g).to(dtype).cuda() for _ in range(2))
    plan = _plan(classes, lengths)
    got = R.build_three_precision_cache(key, value, plan, page_size=16, key_quantization_superblock=k_block, int2_group_size=group).arenas
    want = _by_entry_points(key, value, plan, got, k_block, group)
    n = {"k_packed": sum(rows), "k_scale": -(-sum(rows) // k_block), "k_zero": -(-sum(rows) // k_block), "fp_v": rows[0], "i4_packed": rows[1],
         "i4_scale": rows[1], "i2_packed": rows[2], "i2_scale": rows[2], "i2_zero": rows[2]}
    for name, used in n.items():
        a, b = (t[:, :, :used].contiguous().view(torch.uint8) for t in (getattr(got, name), want[name]))
        assert torch.equal(a, b), name


@pytest.mark.parametrize("odd", [None, 0, 1, 7, 8, 62, 63, 64, 500, 1023])
def test_indices_consecutive_but_for_one(odd):
    pages, page = 16, 64
    classes = torch.tensor([1, 2, 5, 0] * 4)
    key, value = (torch.randn(1, pages * page, 128, device="cuda").to(torch.bfloat16) for _ in range(2))
    plan = _plan(classes, [page] * pages)
    glob, logical = torch.arange(pages * page) + (1 << 40), torch.arange(pages * page)
    if odd is not None:
        glob[odd] += 1 << 33
        logical[-1 - odd] -= 5
    plan = dataclasses.replace(plan, global_token_indices=glob, logical_positions=logical)
    got = R.build_three_precision_cache(key, value, plan, page_size=page).arenas
    fp, i4, i2, evicted = tier_sorted_tokens(plan)
    for order, name in ((fp, "fp"), (i4, "i4"), (i2, "i2")):
        assert torch.equal(getattr(got, name + "_global")[0, :order.numel()].cpu(), glob[order])
        assert torch.equal(getattr(got, name + "_logical")[0, :order.numel()].cpu(), logical[order])
    assert torch.equal(got.evicted_global[0].cpu(), glob[evicted])
