"""What the kernels do when a bounded wait has run out, as far as their source shows it.

The warps of the GEMM kernels leave their loops each on its own.  A hardware barrier between some of a CTA's warps would
then be waited for, without any limit, by those that are left: the kernels must have none.  What remains is the whole CTA's
(`__syncthreads`) and the cluster's, which every path comes to, and mbarriers with bounded waits.

Copies that were waited for in vain may still be in flight: a kernel that starts asynchronous copies into shared memory
gives them time to land (`drain_after_abort`) before it hands the memory back."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warpforge_b200", "csrc")
SOURCES = sorted(f for f in os.listdir(CSRC) if f.endswith((".cu", ".cuh")))


def _code(name):
    return re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())


@pytest.mark.parametrize("name", ["wf_gemm_core.cuh", "wf_gemm_pair.cuh", "wf_gemm_split.cuh"])
def test_no_barrier_between_some_warps(name):
    assert not re.findall(r"\bbar(?:rier)?(?:\.cta)?\.(?:sync|arrive|red)\b", _code(name))
    # a wait that is not one of the bounded ones would be a loop around try_wait
    assert len(re.findall(r"mbarrier\.(?:try|test)_wait", _code(name))) == (1 if name == "wf_gemm_core.cuh" else 0)


def _kernels():
    for name in SOURCES:
        code = _code(name)
        for m in re.finditer(r"__global__ void (?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\([^;{]*\{", code):
            depth, end = 1, m.end()
            while depth:
                depth += {"{": 1, "}": -1}.get(code[end], 0)
                end += 1
            yield name, m.group(1), code[m.end():end]


COPIES = ("tma_load_2d(", "bulk_load(", "stage_x_slice_bulk(", "produce_share<", "st_async_16(")


def test_kernels_with_copies_in_flight_drain():
    copying = {k: body for _, k, body in _kernels() if any(c in body for c in COPIES)}
    assert {"gemm_pair_kernel", "gemm_split_kernel", "gemvn_kernel", "gemv1_group_kernel", "gather_bulk_kernel"} <= set(copying)
    for kernel, body in copying.items():
        assert "drain_after_abort()" in body, kernel
