"""Every rank has to choose the same way for a row-sharded projection's gather: the choice (csrc/wf_gather_route.h, host
arithmetic only, compiled here by itself) sees nothing but values that are equal on all ranks -- not the weight, whose
shards may differ in what the local kernels can take of them -- and the collective takes its route from nowhere else."""
import ctypes
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warpforge_b200", "csrc")
STORES, LOADS, NCCL = range(3)
LAND, STAGE = 32 << 20, 128 << 20


@pytest.fixture(scope="module")
def route(tmp_path_factory):
    d = tmp_path_factory.mktemp("route")
    (d / "route.cpp").write_text('#include "wf_gather_route.h"\nextern "C" int route(int peers, int world, long long land, long long stage, '
                                 "int f32, long long m, long long rows) { return wf::gather_route(wf::GatherRoom{peers != 0, world, land, stage}, f32 != 0, m, rows); }\n")
    so = str(d / "route.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(d / "route.cpp"), "-o", so], check=True)
    f = ctypes.CDLL(so).route
    f.argtypes = [ctypes.c_int, ctypes.c_int, ctypes.c_longlong, ctypes.c_longlong, ctypes.c_int, ctypes.c_longlong, ctypes.c_longlong]
    return f


@pytest.mark.parametrize("f32,m,want", [(0, 1, STORES), (0, 32, STORES), (0, 33, LOADS), (1, 1, STORES), (1, 10, STORES), (1, 11, LOADS), (1, 300, LOADS)])
def test_route_by_token_count(route, f32, m, want):
    for world in (2, 3, 8):
        assert route(1, world, LAND, STAGE, f32, m, 1024) == want
        assert route(0, world, LAND, STAGE, f32, m, 1024) == NCCL
    assert route(1, 1, LAND, STAGE, f32, m, 1024) == NCCL


def test_buffers_that_are_too_small(route):
    rows = LAND // 2 // 8 // 2 // 4  # two ranks, four tokens: exactly one half of the landing buffer
    assert route(1, 2, LAND, STAGE, 0, 4, rows) == STORES
    assert route(1, 2, LAND, STAGE, 0, 4, rows + 1) == LOADS
    assert route(1, 2, LAND, STAGE, 0, 64, STAGE // 4 // 64) == LOADS
    assert route(1, 2, LAND, STAGE, 0, 64, STAGE // 4 // 64 + 1) == NCCL


def test_the_collective_asks_nothing_else():
    code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, "wf_comm.cu")).read())
    body = code[code.index("int wf_qlinear_allgather"):]
    assert body.count("gather_route(") == 1 and "gemm_supported" not in code and "beyond_fp16" not in code
    # nothing is enqueued before the local projection's scratch is there
    assert body.index("qlinear_reserve") < body.index("gather_wait_done_kernel<<<")
