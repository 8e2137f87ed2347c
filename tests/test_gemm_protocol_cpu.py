"""The hand-overs between the roles of the K-quant product, checked from its source: what a run shows only when a wait runs out or a copy is late."""
import os
import re

import numpy as np
import pytest

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


def test_a_wait_orders_memory_for_the_whole_warp():
    """one lane asks for a barrier, all lanes read what it guards, and an elected lane hands it on by an arrival of its own: behind every wait that
    succeeds the warp meets in a way that orders memory, which a vote does not"""
    s = source()
    wait = s[s.index("bool wait_on("):]
    wait = wait[:wait.index("\n}")]
    succeeds = list(re.finditer(r"return true;", wait))
    assert succeeds and all(re.search(r"__syncwarp\(\);\s*$", wait[:m.start()]) for m in succeeds)
    body = kernel_body()
    assert "try_wait(" not in body  # every wait goes through wait_on
    assert body.index("wait_on(bar, par") < body.index("bar_arrive(&acc_full[w])")


def constants(q6):
    """the sizes of the rings of one instance"""
    s = source()
    v = dict(re.findall(r"\b(DA_RING|SC_RING) = (\d+)", s))
    for name in ("RAW_STAGES", "B_STAGES"):
        a, b = re.search(name + r" = Q6 \? (\d+) : (\d+)", s).groups()
        v[name] = a if q6 else b
    return {k: int(n) for k, n in v.items()}


def drained_when_issued(q):
    """the last chunk that is known to be drained when the MMAs of chunk q are issued (they wait for its accumulator)"""
    return q - 2


@pytest.mark.parametrize("q6", [False, True], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("chunks", [1, 2, 3, 4])
def test_waits_by_parity_are_unambiguous(q6, chunks):
    """a wait by parity for phase n of a barrier is right only if phase n - 1 is known to be over: the waiting warp has waited for it, or for
    something that comes behind it, before it tries.  Walks the waits of the two issuing warps on the token stages"""
    c, body = constants(q6), kernel_body()
    acc_first = c["B_STAGES"] % 2 == 0 or "C::B_STAGES % 2 && q >= 2 && !(ok = wait(&acc_empty[w]" in body
    for w in (0, 1):
        seen = {}
        for q in range(w, 64 * chunks, 2):  # a warp issues every second chunk of the whole walk, whatever the blocks
            s, phase = q % c["B_STAGES"], q // c["B_STAGES"]
            known = seen.get(s, -1)
            if acc_first and q >= 2:  # every chunk up to q - 2 has been drained, so it had been loaded
                d = drained_when_issued(q)
                known = max(known, max((p // c["B_STAGES"] for p in range(d + 1) if p % c["B_STAGES"] == s), default=-1))
            assert known >= phase - 1
            seen[s] = phase


@pytest.mark.parametrize("q6", [False, True], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("chunks", [1, 2, 3, 4])
def test_rings_without_an_empty_barrier(q6, chunks):
    """the scales of tokens and of weight blocks are overwritten only when their last reader is known to be through"""
    c = constants(q6)
    for q in range(200):
        # token scales of chunk q are requested when the MMAs of chunk q - B_STAGES are over: then their place's former chunk is drained
        assert q - c["DA_RING"] <= drained_when_issued(q - c["B_STAGES"])
        # scales of block u are written when the MMAs of block u - 2 are over
        u = q
        last = (u - 2) * chunks + chunks - 1  # its last chunk
        assert (u - c["SC_RING"]) * chunks + chunks - 1 <= drained_when_issued(last)


def test_decoded_q4_weights_are_exact_in_f16():
    """sc q - k by the two multiply-adds of the decoder, for every scale and code: the integer itself, at most 512, so that 256 of them times
    a code of 128 stay within 2^24; and k, exact"""
    h = np.float16
    decoder = source()[source().index("auto k = [&](__half2 sc)"):]
    assert re.findall(r"__floats2half2_rn\((-?[\d.]+)f, (-?[\d.]+)f\)", decoder)[:2] == [("-1024.", "0."), ("1032.", "8.")]
    assert re.findall(r"__float2half2_rn\((-?[\d.]+)f\)", decoder)[:3] == ["-1032.", "0.0625", "-72."]
    fma = lambda a, b, c: h(float(a) * float(b) + float(c))  # one rounding: product and sum are exact in double
    for sc in range(64):
        o0, o1 = h(h(sc) * h(-1032.0)), h(h(sc) * h(-72.0))
        k0, k1 = fma(h(sc), h(-1024.0), h(h(sc) * h(1032.0))), h(h(sc) * h(8.0))
        assert np.isfinite(o0) and float(o0) == -1024 * sc - float(k0) and float(o1) == -72 * sc and float(k1) == 8 * sc
        for q in range(16):
            low, high = fma(h(1024 + q), h(sc), o0), fma(h(1024 + 16 * q), h(h(sc) * h(0.0625)), o1)
            assert float(low) == sc * q - float(k0) and float(high) == sc * q - float(k1)
            assert max(abs(float(low)), abs(float(high))) * 128 * 256 <= 2 ** 24


def test_warps_of_the_decode_product_divide_among_the_tokens(tmp_path):
    """its warps are dealt out to up to 8 tokens; a number that leaves some over, which a build may ask for, would have them write behind the last token: refused"""
    import shutil
    import subprocess

    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    src = os.path.join(os.path.dirname(SRC), "kq_gemv_stream.cu")
    r = subprocess.run([nvcc, "-cuda", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr", "-DKQ_GEMV_WARPS=12", "-x", "cu", src,
                        "-o", str(tmp_path / "x.ii")], capture_output=True, text=True)
    assert r.returncode != 0 and "a warp past the last token" in r.stderr + r.stdout
