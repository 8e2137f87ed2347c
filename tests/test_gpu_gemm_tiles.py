"""The tensor-core product with K-quant weights at the edges of its tiles, shares and rings, against the oracle's integer block
sums and a combination in 64 bits.

Per block the kernel forms da (dw si - dmin sm) with three roundings and adds it to an f32 sum of at most K / 256 terms (a tile that
was cut adds a few more), so |error| <= (K / 256 + 8) 2^-23 sum_b da (|dw si| + |dmin sm|)."""
import numpy as np
import pytest

from oracle import binding as orc

pytestmark = pytest.mark.gpu

# rows: part of a tile, several; K: one block, odd counts, Q6_K groups with an odd tail
SHAPES = [(1, 256), (100, 512), (129, 2816), (264, 768)]
TOKENS = [9, 16, 17, 64, 65, 128, 129, 193, 256, 257]


def blocks_of(ty, N, K, seed):
    rng = np.random.default_rng(seed)
    blk = rng.integers(0, 256, size=(N * K // 256, 144 if ty == orc.TYPE_Q4_K else 210), dtype=np.uint8)
    half = lambda lo, hi: rng.uniform(lo, hi, len(blk)).astype(np.float16)[:, None].view(np.uint8)
    if ty == orc.TYPE_Q4_K:
        blk[:, 0:2], blk[:, 2:4] = half(1e-4, 1e-3), half(1e-4, 1e-3)
    else:
        blk[:, 208:210] = half(1e-5, 1e-4)
    return blk.reshape(N, -1)


def exact(ty, W, x, N, K):
    """-> y and the sum of the magnitudes of its terms, both in 64 bits"""
    q, d, bs = orc.quantize_act(x)
    si, sm = orc.block_sums(ty, W, q, bs, N, K)
    b = np.ascontiguousarray(W).reshape(N, K // 256, -1)
    f16 = lambda at: np.ascontiguousarray(b[:, :, at:at + 2]).view(np.float16)[..., 0].astype(np.float64)
    main = si.reshape(-1, N, K // 256) * (f16(0) if ty == orc.TYPE_Q4_K else f16(208))
    low = sm.reshape(-1, N, K // 256) * f16(2) if ty == orc.TYPE_Q4_K else np.zeros_like(main)
    d = d.reshape(-1, 1, K // 256).astype(np.float64)
    return ((main - low) * d).sum(-1), ((np.abs(main) + np.abs(low)) * d).sum(-1)


def check(got, want, size, K):
    bound = (K // 256 + 8) * 2.0 ** -23 * size + 1e-30
    assert np.all(np.abs(got.astype(np.float64) - want) <= bound)


@pytest.mark.parametrize("ty", [orc.TYPE_Q4_K, orc.TYPE_Q6_K], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("N,K", SHAPES)
def test_dense(ty, N, K):
    import torch

    from mesh_llm_b200 import capi, ops

    W = blocks_of(ty, N, K, N + K)
    dev = ops.upload_weights(ty, W, N, K)
    for M in TOKENS:
        x = np.random.default_rng(M).standard_normal((M, K)).astype(np.float32)
        want, size = exact(ty, W, x, N, K)
        got = ops.mul_mat(ty, dev, torch.from_numpy(x).cuda(), N, K).cpu().numpy()
        assert capi.lib().b200_check_device_waits() == 0
        check(got, want, size, K)


@pytest.mark.parametrize("ty,N,K,M", [(orc.TYPE_Q4_K, 20000, 4096, 16), (orc.TYPE_Q6_K, 20000, 4096, 16), (orc.TYPE_Q6_K, 6000, 2816, 200)])
def test_long_shares_and_cut_tiles(ty, N, K, M):
    """a CTA walks through more blocks than any ring has stages, and through parts of tiles"""
    import torch

    from mesh_llm_b200 import capi, ops

    W = blocks_of(ty, N, K, 5)
    dev = ops.upload_weights(ty, W, N, K)
    x = np.random.default_rng(6).standard_normal((M, K)).astype(np.float32)
    want, size = exact(ty, W, x, N, K)
    xd = torch.from_numpy(x).cuda()
    got = [ops.mul_mat(ty, dev, xd, N, K) for _ in range(3)]
    assert capi.lib().b200_check_device_waits() == 0
    assert torch.equal(got[0], got[1]) and torch.equal(got[0], got[2]) # the order of additions does not depend on the timing
    check(got[0].cpu().numpy(), want, size, K)


@pytest.mark.parametrize("ty", [orc.TYPE_Q4_K, orc.TYPE_Q6_K], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("N,K,M", [(6000, 2816, 257), (6000, 2816, 400), (6000, 2816, 500), (3000, 512, 513), (1024, 5120, 77), (70, 27648, 1100)])
def test_widths_of_token_tiles(ty, N, K, M):
    """sizes whose tokens are cut into tiles of one to four chunks, with a shorter last one, and into slabs (rows of 27648)"""
    import torch

    from mesh_llm_b200 import capi, ops

    W = blocks_of(ty, N, K, 11)
    x = np.random.default_rng(12).standard_normal((M, K)).astype(np.float32)
    want, size = exact(ty, W, x, N, K)
    got = ops.mul_mat(ty, ops.upload_weights(ty, W, N, K), torch.from_numpy(x).cuda(), N, K).cpu().numpy()
    assert capi.lib().b200_check_device_waits() == 0
    check(got, want, size, K)


def extreme_blocks(ty, kind, N, rng):
    """blocks of one scale factor 1 whose sums are as large as the format allows, or pass through such sums on their way to a small one"""
    blk = np.zeros((N, 144 if ty == orc.TYPE_Q4_K else 210), np.uint8)
    one = np.array([1.0], np.float16).view(np.uint8)
    top = kind != "near" # "near": every scale and code near its end of the range
    if ty == orc.TYPE_Q4_K:
        sc, q = (np.full((N, 8), 63), np.full((N, 256), 15)) if top else (rng.integers(56, 64, (N, 8)), rng.integers(12, 16, (N, 256)))
        blk[:, 0:2] = one
        blk[:, 4:8] = sc[:, :4] | (sc[:, 4:] >> 4) << 6
        blk[:, 12:16] = sc[:, 4:] & 15
        q = q.reshape(N, 4, 2, 32)
        blk[:, 16:] = (q[:, :, 0] | q[:, :, 1] << 4).reshape(N, 128)
    else:
        sc, q = (np.full((N, 16), -128), np.zeros((N, 256), int)) if top else (rng.integers(-128, -119, (N, 16)), rng.integers(0, 4, (N, 256)))
        q = q.reshape(N, 2, 2, 2, 32)  # [half][low or high nibble][32 of 64][..]
        blk[:, :128] = ((q[:, :, 0] & 15) | (q[:, :, 1] & 15) << 4).reshape(N, 128)
        quarters = q.reshape(N, 2, 4, 32) >> 4
        blk[:, 128:192] = (quarters[:, :, 0] | quarters[:, :, 1] << 2 | quarters[:, :, 2] << 4 | quarters[:, :, 3] << 6).reshape(N, 64)
        blk[:, 192:208] = sc.astype(np.int8).view(np.uint8)
        blk[:, 208:210] = one
    return blk


@pytest.mark.parametrize("ty", [orc.TYPE_Q4_K, orc.TYPE_Q6_K], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("kind", ["top", "near", "cancelling"])
@pytest.mark.parametrize("M", [1, 8, 9, 77, 300])
def test_largest_block_sums(ty, kind, M):
    """one block, scale factors 1: the result is the block's integer sum, up to 3.1e7 (Q4_K) or 1.3e8 (Q6_K), rounded to f32 once: off by
    half a spacing of f32 at most, and not at all below 2^24"""
    import torch

    from mesh_llm_b200 import ops

    rng = np.random.default_rng(M)
    N, K = 130, 256
    W = extreme_blocks(ty, kind, N, rng)
    x = np.full((M, K), 127.0, np.float32) if kind == "top" else rng.integers(120, 128, (M, K)).astype(np.float32)
    x[:, 0] = 127.0  # the Q8 scale is 1
    if kind == "cancelling":
        x[:, 128:] *= -1
    x[1::2] *= -1
    q, d, bs = orc.quantize_act(x)
    assert np.all(d == 1.0) and np.array_equal(q.astype(np.float32), x)
    si, _ = orc.block_sums(ty, W, q, bs, N, K)
    want = si.astype(np.float64).reshape(M, N)
    assert kind == "cancelling" or np.abs(want).min() > 2.0 ** 24
    got = ops.mul_mat(ty, ops.upload_weights(ty, W, N, K), torch.from_numpy(x).cuda(), N, K).cpu().numpy()
    assert np.all(np.abs(got.astype(np.float64) - want) <= np.where(np.abs(want) < 2.0 ** 24, 0.0, np.spacing(np.abs(want).astype(np.float32)) / 2))


def test_more_tokens_than_a_slab():
    import torch

    from mesh_llm_b200 import ops

    N, K, M = 130, 256, 4100
    W = blocks_of(orc.TYPE_Q4_K, N, K, 7)
    x = np.random.default_rng(8).standard_normal((M, K)).astype(np.float32)
    want, size = exact(orc.TYPE_Q4_K, W, x, N, K)
    got = ops.mul_mat(orc.TYPE_Q4_K, ops.upload_weights(orc.TYPE_Q4_K, W, N, K), torch.from_numpy(x).cuda(), N, K).cpu().numpy()
    check(got, want, size, K)


@pytest.mark.parametrize("ty", [orc.TYPE_Q4_K, orc.TYPE_Q6_K], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("rows,ku,E,N,K", [(5, 2, 3, 100, 768), (300, 2, 4, 192, 512), (16, 8, 128, 64, 256)])
def test_experts(ty, rows, ku, E, N, K):
    """experts without pairs, with one, and with more than a tile; rows of an expert that end inside a tile"""
    import torch

    from mesh_llm_b200 import capi, ops

    rng = np.random.default_rng(rows)
    W = blocks_of(ty, E * N, K, 9)
    x = rng.standard_normal((rows, K)).astype(np.float32)
    ids = rng.integers(0, E, rows * ku).astype(np.int32)
    ids[ids == 1] = 0
    ids[-1] = 1
    got = ops.mul_mat_id(ty, ops.upload_weights(ty, W, E * N, K), E, torch.from_numpy(x).cuda(), torch.from_numpy(ids).cuda(), N, K).cpu().numpy()
    assert capi.lib().b200_check_device_waits() == 0
    for e in range(E):
        at = np.nonzero(ids == e)[0]
        if len(at):
            want, size = exact(ty, W[e * N:(e + 1) * N], x[at // ku], N, K)
            check(got[at], want, size, K)


@pytest.mark.parametrize("h", [4, 64, 128, 132, 256])
def test_norm_of_short_rows(h):
    """a warp per row up to 128 values, a CTA above; the sum of squares is taken in double, then three f32 roundings"""
    import torch

    from mesh_llm_b200 import ops

    x = np.random.default_rng(h).standard_normal((37, h)).astype(np.float32)
    w = np.random.default_rng(h + 1).standard_normal(h).astype(np.float32)
    got = ops.rms_norm(torch.from_numpy(x).cuda(), torch.from_numpy(w).cuda(), 1e-6).cpu().numpy()
    want = x.astype(np.float64) / np.sqrt((x.astype(np.float64) ** 2).mean(-1, keepdims=True) + 1e-6) * w
    assert np.all(np.abs(got - want) <= 2.0 ** -21 * np.abs(want))


@pytest.mark.parametrize("M", [300, 900, 1000])
@pytest.mark.parametrize("N,K", [(3072, 128), (3000, 200), (6200, 64)])
def test_bf16_tiles(M, N, K):
    """sizes around the tiles (every width: test_gpu_bf16_tiles.py); bf16 operands, f32 sums of at most 200 terms (truncating: 2^-22 each)"""
    import torch

    from mesh_llm_b200 import ops

    g = torch.Generator(device="cuda").manual_seed(M + N)
    w = torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16).float()
    got = ops.mul_mat_bf16(ops.upload_bf16(w), x, N, K).double()
    want = x.double() @ w.double().T
    size = x.double().abs() @ w.double().abs().T
    assert ((got - want).abs() <= K * 2.0 ** -22 * size).all()


@pytest.mark.parametrize("n", [1, 3, 4, 255, 2048, 2052, 32001, 151936, 152064])
def test_greedy_token(n):
    """the first of the largest values, at the edges of the slices, with infinities and NaN; the same as the statistics' most likely token"""
    import torch

    from mesh_llm_b200 import capi

    rng = np.random.default_rng(n)
    x = rng.standard_normal((5, n)).astype(np.float32)
    x[1, rng.integers(0, n)] = x[1, n - 1] = 9.0
    x[2] = -np.inf
    x[3, :] = np.float32(-3.4028235e38)
    x[4, rng.integers(0, n)] = np.inf
    if n > 4:
        x[0, 2] = np.nan
    L, xd, out = capi.lib(), torch.from_numpy(x).cuda(), torch.empty(5, dtype=torch.int32, device="cuda")
    scratch = torch.zeros(L.b200_logit_signals_scratch_bytes(5), dtype=torch.uint8, device="cuda")
    for _ in range(2): # the counters are left as they were found
        capi.check(L.b200_logit_signals(capi.ptr(xd), 5, n, None, None, capi.ptr(out), capi.ptr(scratch), scratch.numel(), capi.cur_stream()))
    got = out.cpu().numpy()
    assert np.array_equal(got, [int(np.argmax(np.where(np.isnan(r), -np.inf, r))) for r in x])


MEMORY = """
import torch
from mesh_llm_b200 import capi, ops
from oracle import binding as orc

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]

def product(M, K, N=128):
    W = torch.zeros(N * K // 256 * 144, dtype=torch.uint8, device="cuda")
    q, d = torch.ones((M, K), dtype=torch.int8, device="cuda"), torch.ones((M, K // 256), device="cuda")
    bs, y = torch.full((M, K // 16), 16, dtype=torch.int16, device="cuda"), torch.full((M, N), 7.0, device="cuda")
    return lambda: ops.mul_mat_q8(orc.TYPE_Q4_K, W, q, d, bs, N, K, out=y)

MB = 1 << 20
first = product(16, 256)
first()
"""
GROWTH = MEMORY + """
calls = [product(M, 8192) for M in (256, 512, 1024, 2048, 3000)]
before = free()
for c in calls:
    c()
used = before - free()
# 3000 tokens x 32 blocks x 544 bytes and their scales, in allocations of 2 MB
assert used <= 3000 * 32 * (544 + 4) + 6 * MB, used
"""
NO_ROOM = MEMORY + """
import ctypes
c = product(3000, 8192)
cu, at = ctypes.CDLL("libcuda.so.1"), ctypes.c_uint64()
take = lambda n: cu.cuMemAlloc_v2(ctypes.byref(at), ctypes.c_size_t(n)) == 0
assert take(16 * MB)
hole, size = at.value, 1 << 34
while size >= 2 * MB:
    if not take(size):
        size //= 2
assert cu.cuMemFree_v2(ctypes.c_uint64(hole)) == 0 and not take(3000 * 32 * 544)
y = c()
torch.cuda.synchronize()
assert capi.lib().b200_check_device_waits() == 0 and bool((y == 0).all())
"""


@pytest.mark.parametrize("script", [GROWTH, NO_ROOM], ids=["growth", "no_room"])
def test_memory_of_images(script):
    """calls of growing size leave the device with the largest one's images, not with all of them; and where the images of a call do not fit,
    it takes fewer tokens at a time"""
    import os
    import subprocess
    import sys

    r = subprocess.run([sys.executable, "-c", script], cwd=os.path.join(os.path.dirname(__file__), ".."), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


def test_experts_in_slabs():
    """images of more than 256 MB: the tiles of the routed pairs in several launches"""
    import torch

    from mesh_llm_b200 import capi, ops

    ty, rows, ku, E, N, K = orc.TYPE_Q4_K, 1200, 8, 256, 128, 7168
    rng = np.random.default_rng(13)
    W = np.tile(blocks_of(ty, 2 * N, K, 14), (E // 2, 1))  # two matrices in turn
    x = rng.standard_normal((rows, K)).astype(np.float32)
    ids = rng.integers(0, E, rows * ku).astype(np.int32)
    dev, xd = ops.upload_weights(ty, W, E * N, K), torch.from_numpy(x).cuda()
    got = ops.mul_mat_id(ty, dev, E, xd, torch.from_numpy(ids).cuda(), N, K).cpu().numpy()
    assert capi.lib().b200_check_device_waits() == 0
    for e in (0, 1, 100, 201, 254, 255):
        at = np.nonzero(ids == e)[0]
        want, size = exact(ty, W[e * N:(e + 1) * N], x[at // ku], N, K)
        check(got[at], want, size, K)


@pytest.mark.parametrize("ty", [orc.TYPE_Q4_K, orc.TYPE_Q6_K], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("N,K", [(20000, 512), (2000, 2816)])
def test_tiles_of_one_two_and_four_chunks(ty, N, K):
    """every edge between tiles of one chunk (two warpgroups decode in turn), of two and of four, with many and with few row tiles"""
    import torch

    from mesh_llm_b200 import capi, ops

    W = blocks_of(ty, N, K, 21)
    dev = ops.upload_weights(ty, W, N, K)
    x = np.random.default_rng(22).standard_normal((260, K)).astype(np.float32)
    want, size = exact(ty, W, x, N, K)
    for M in (9, 31, 33, 49, 64, 65, 97, 128, 129, 192, 193, 255, 260):
        got = ops.mul_mat(ty, dev, torch.from_numpy(x[:M]).cuda(), N, K).cpu().numpy()
        assert capi.lib().b200_check_device_waits() == 0
        check(got, want[:M], size[:M], K)


@pytest.mark.parametrize("ty", [orc.TYPE_Q4_K, orc.TYPE_Q6_K], ids=["q4_k", "q6_k"])
@pytest.mark.parametrize("pairs", [9, 47, 48 * 5, 48 * 5 + 1, 700])
def test_experts_with_narrow_and_wide_tiles(ty, pairs):
    """five experts, one of them without a pair and one with most of them, on both sides of the number of pairs from which tiles are wide"""
    import torch

    from mesh_llm_b200 import capi, ops

    E, N, K = 5, 200, 768
    rng = np.random.default_rng(pairs)
    W = blocks_of(ty, E * N, K, 23)
    ids = rng.choice([0, 1, 3, 4], pairs, p=[0.7, 0.1, 0.15, 0.05]).astype(np.int32)
    x = rng.standard_normal((pairs, K)).astype(np.float32)
    want, size = exact(ty, W, x, E * N, K)
    pick = lambda v: v.reshape(pairs, E, N)[np.arange(pairs), ids]
    got = ops.mul_mat_id(ty, ops.upload_weights(ty, W, E * N, K), E, torch.from_numpy(x).cuda(), torch.from_numpy(ids[:, None]).cuda(), N, K).cpu().numpy()
    assert capi.lib().b200_check_device_waits() == 0
    check(got.reshape(pairs, N), pick(want), pick(size), K)
