"""Which kernels let the next launch of the stream in early, read from their source: a decode launch reads the packed pools before its own
wait, so a kernel that lets it in has waited for the kernel in front of itself, which may have written them."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "r2omni_b200", "csrc")


def kernels():
    for name in ("pack_kernels.cuh", "build_kernel.cuh", "decode_kernel.cuh"):
        with open(os.path.join(CSRC, name)) as f:
            text = re.sub(r"//[^\n]*", "", f.read())
        for part in re.split(r"__global__ void", text)[1:]:
            yield re.search(r"(\w+_kernel)\(", part).group(1), part[: part.index("\n}\n")]


def test_who_lets_the_next_launch_in():
    bodies = dict(kernels())
    assert {"decode_kernel", "mrope_rows_kernel", "fwht128_kernel", "merge_states_kernel", "build_cache_kernel"} <= set(bodies)
    early = {n for n, b in bodies.items() if re.search(r"(?<!\) )\blaunch_dependents\(\)", b)}
    assert early == {"decode_kernel", "mrope_rows_kernel", "host_block_copy_kernel"}   # none of them writes the pools
    rotation = bodies["mrope_rows_kernel"]
    assert rotation.index("grid_dependency_wait()") < rotation.index("launch_dependents()")
    for name in ("fwht128_kernel", "merge_states_kernel", "flush_ring_kernel", "build_cache_kernel", "gather_rows_kernel", "pack_v_int4_kernel"):
        assert "launch_dependents" not in bodies[name]
    for name in ("pack_k_int4_kernel", "pack_v_int2_kernel"):   # in a flush alone: its last launch waits for both
        assert re.findall(r"[^;{}]*launch_dependents\(\)", bodies[name])[0].strip() == "if (a.in_flush) launch_dependents()"


def test_pool_writers_publish_what_they_wrote():
    """A decode launch behind one of them may come in when its CTAs have left, before the grid counts as completed."""
    bodies = dict(kernels())
    for name in ("pack_k_int4_kernel", "pack_v_int4_kernel", "pack_v_int2_kernel", "gather_rows_kernel"):
        assert bodies[name].count("publish_pools()") == 1, name
    build = bodies["build_cache_kernel"]   # its rows and its fills; the token bookkeeping is not read by a decode launch
    assert re.search(r"build_values<[^;]*;\s*publish_pools\(\);\s*return;", build) and build.rstrip().endswith("publish_pools();\n    return;\n  }")
