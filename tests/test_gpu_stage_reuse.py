"""One or two CTAs walk every head's tiles through the same four stages of shared memory: what plain stores left in a stage (the
appended row, ragged rows of a pool) is followed by bulk copies of later tiles and of the next heads'."""
import pytest
import torch

import r2omni_b200 as R
from gpu_helpers import assert_close, make_executor
from oracle import sspa_oracle as O
from test_gpu_decode import both_caches, seeded_classes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("cap", [1, 2])
@pytest.mark.parametrize("row", [0, 15, 63, 64, 127])   # window row of the appended token: at the ends of slices and tiles
def test_stages_behind_plain_stores(row, cap, dtype, monkeypatch):
    pages, page, heads = 37, 16, 5   # pools of a few ragged tiles each
    ocache, gcache, new_k, new_v, queries = both_caches(row, hq=3 * heads, hkv=heads, tokens=pages * page, page=page,
                                                        classes=seeded_classes(pages, 5), appends=row + 1, dtype=dtype, append_capacity=256)
    stats = R.DynamicCacheStats()
    k, v, q = new_k.cuda(), new_v.cuda(), queries[0].cuda()
    for i in range(row + 1):
        O.append_token(ocache, new_k[i], new_v[i], 600 + i, 600 + i)
        if i < row:
            R.append_generated_token(gcache, k[i].unsqueeze(1), v[i].unsqueeze(1), global_token_index=600 + i, logical_position=600 + i,
                                     stats=stats)
    ex = make_executor(gcache, 3 * heads)
    monkeypatch.setenv("R2K_GRID_CAP", str(cap))
    got = ex.decode_f32(q, append=(k[row].unsqueeze(0).contiguous(), v[row].unsqueeze(0).contiguous(), 600 + row, 600 + row))
    assert_close(got, O.decode_fp32(queries[0].float(), ocache), "appended in the launch")
    gcache.arenas.recent_len = row + 1
    assert_close(ex.decode_f32(q), O.decode_fp32(queries[0].float(), ocache), "appended before it")
    assert ex.device_status() == 0 and int(gcache.arenas.recent_len_device) == row + 1
