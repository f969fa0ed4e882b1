"""The warps of the GEMM kernels leave their loops each on its own when a wait has run out.  A hardware barrier between some
of a CTA's warps would then be waited for, without any limit, by those that are left: the kernels must have none.  What
remains is the whole CTA's (`__syncthreads`) and the cluster's, which every path comes to, and mbarriers with bounded waits."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "warpforge_b200", "csrc")


@pytest.mark.parametrize("name", ["wf_gemm_core.cuh", "wf_gemm_pair.cuh", "wf_gemm_split.cuh"])
def test_no_barrier_between_some_warps(name):
    code = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    assert not re.findall(r"\bbar(?:rier)?(?:\.cta)?\.(?:sync|arrive|red)\b", code)
    # a wait that is not one of the bounded ones would be a loop around try_wait
    assert len(re.findall(r"mbarrier\.(?:try|test)_wait", code)) == (1 if name == "wf_gemm_core.cuh" else 0)
