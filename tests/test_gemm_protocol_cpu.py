"""The hand-overs between the roles of the K-quant product, checked from its source: what a run shows only when a wait runs out or a copy is late."""
import os
import re

SRC = os.path.join(os.path.dirname(__file__), "..", "mesh_llm_b200", "csrc", "kq_gemm_tc.cu")


def source():
    with open(SRC) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def kernel_body():
    s = source()
    at = s.index("gemm_kq_kernel(")
    return s[at:s.index("\n}", at)]


def test_no_barrier_that_a_warp_can_miss_by_giving_up():
    """the waits of the roles give up one warp at a time, so warps may meet only behind all of them: between the start of the roles and the
    kernel's last barrier there is none, and a warp that gave up takes no part in counting the parts of a cut tile"""
    body = kernel_body()
    roles = body[body.index("if (warp >= 12)"):]
    assert roles.count("__syncthreads") == 1
    assert not re.search(r"\bbar\.sync\b|barrier\.sync|__syncthreads_|named_barrier", roles)
    drain = roles[roles.index("setmaxnreg.inc"):roles.index("__syncthreads")]
    assert drain.index("if (!ok) break;") < drain.index("atomicAdd")
