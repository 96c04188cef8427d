"""A call that waits for room in the launch queue leaves the interpreter to the other threads."""
import threading
import time

import pytest
import torch

import r2omni_b200 as R
from gpu_helpers import build_gpu_cache, make_executor, make_plan

pytestmark = pytest.mark.gpu


def _calls():
    key = torch.randn(1, 256, 128, generator=torch.Generator().manual_seed(1)).to(torch.bfloat16).cuda()
    classes = torch.tensor([2, 1, 5, 2])
    ex = make_executor(build_gpu_cache(key, key, classes, page_size=64), 4)
    q = torch.zeros(1, 4, 128, dtype=torch.bfloat16, device="cuda")
    row = torch.zeros(1, 1, 128, dtype=torch.bfloat16, device="cuda")
    rows4 = torch.zeros(1, 4, 1, 128, dtype=torch.bfloat16, device="cuda")
    table = torch.zeros(3, 1, 1, 128, dtype=torch.bfloat16, device="cuda")
    plan = make_plan(classes, 64, 128)
    return {"step": lambda: ex(q), "step with append": lambda: ex(q, append=(row, row, 0, 0)), "fwht": lambda: R.triton_fwht_128(rows4),
            "rotation": lambda: R.qwen_qk_mrope(rows4, rows4, table, table, (16, 24, 24)),
            "prologue": lambda: R.qwen_qkv_prologue(rows4, rows4, rows4, table, table, (16, 24, 24)),
            "build": lambda: R.build_three_precision_cache(key, key, plan, page_size=64)}


@pytest.mark.parametrize("name", ["step", "step with append", "fwht", "rotation", "prologue", "build"])
def test_other_threads_run_while_a_launch_waits(name):
    call = _calls()[name]
    call()
    torch.cuda.synchronize()
    ticks, done = [], threading.Event()

    def tick():
        while not done.is_set():
            ticks.append(time.perf_counter())
            time.sleep(0.001)

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(1_500_000_000)   # about 0.8 s in which the queue (about a thousand launches) fills up
        begin = time.perf_counter()
        slowest = 0.0
        for _ in range(1500):
            t = time.perf_counter()
            call()
            slowest = max(slowest, time.perf_counter() - t)
        end = time.perf_counter()
    finally:
        done.set()
        thread.join()
        torch.cuda.synchronize()
    assert slowest > 0.2, f"no call waited (the slowest took {slowest:.3f} s)"
    inside = [begin] + [t for t in ticks if begin < t < end] + [end]
    assert max(b - a for a, b in zip(inside, inside[1:])) < slowest / 2
