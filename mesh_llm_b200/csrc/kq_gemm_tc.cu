// Products of more than a few tokens with K-quant weights on the 5th-generation tensor cores:
// y[m][n] = sum_k W[n][k] x[m][k], W in Q4_K / Q6_K blocks, x in Q8 blocks of 256.
//
// The integer scale of a sub-block is folded into the weight, and the products of a 256-element block are added up as integers.
// Q4_K: w' = sc_j q goes in as sc_j q - k_j, |.| <= 512, with k_j about 8 sc_j: exact in f16, as a Q8 code is, so one
// tcgen05.mma of kind::f16 per 16 elements adds up  sum_j sum_i (sc_j q_ij - k_j) a_ij  in f32, and no partial sum exceeds 2^24: exact.
// One more MMA (K = 16) adds sum_j k_j bsum_j, which makes it the block's integer sum: above 2^24 that one addition rounds, by half a
// spacing at most as a conversion from int32 would.  The min term sum_j m_j bsum_j is another MMA into an
// accumulator of its own.  Per block an output then takes y += d_a (d_w main - d_min min) in f32.
// Q6_K: w' = sc (q - 32) has 14 bits with its sign, w' = 64 hi + lo with |hi| <= 64 and 0 <= lo < 64.  Both are bytes, and two tcgen05.mma of
// kind::i8 per 32 elements, each into an int32 accumulator of its own, give the sum of the block whatever its size; it is rounded once, to f32.
//
// A tile is 128 weight rows x up to 256 tokens.  Weight rows are the M of the MMA (TMEM lanes), tokens its N in chunks of
// up to 64.  Packed blocks arrive by TMA; a warpgroup (a thread per row) decodes them into TMEM, two bytes per weight in both types, from where
// the MMAs take them as their A operand, so that decoded weights never pass through shared memory.  The token operand is an image that
// act_image_kernel, or the kernel that makes the tokens, writes (f16 codes and sums of 16 for Q4_K, the codes themselves for Q6_K): one bulk copy per chunk and block.  Two warps issue MMAs in turn, each with an accumulator of its own;
// the draining warps add the accumulators to the running f32 result, which stays in registers for the whole tile.  Lanes of a
// warp hold neighbouring rows of W, so results leave in full lines.
// With tiles of two or four chunks one warpgroup decodes and two drain, half of every chunk each.  Narrow tiles are one chunk: their blocks take the decoding longer
// than anything else, so two warpgroups decode, block by block in turn, and one drains.
//
// Up to three matrices that read the same tokens (q / k / v, gate / up) share the image and, type by type, the launch: the small ones would
// leave most of the GPU idle (256 x 2048 at 77 tokens: 19 us alone, two of them in the launch of q: none).
// The (tile, block) pairs are dealt out to the CTAs in equal contiguous shares, so that any number of tiles fills the GPU.  A tile
// that was cut is added up, in the order of its parts, by the CTA that arrives last, each draining warp its own rows and tokens of the
// tile; nobody waits, and no barrier stands between a wait that can give up and the end of the kernel.
//
// What bounds it.  Wide tiles: a chunk of 64 tokens takes 756 clocks of MMAs in either type (18 of 42; 32 would be the tensor rate) and about 1000 in fact: an accumulator
// goes round MMAs, drain (300) and two hand-overs, and TMEM has room for two beside the two decoded blocks.  28672 x 8192 at 512 tokens: 250 us in Q4_K (960 TFLOP/s),
// 271 in Q6_K; 316 and 349 while the loop over the blocks also held the end of the tile and unrolled chunks, whose turn cost a draining warp a thousand clocks beside
// the additions, and while it waited for the scales' barriers beside the accumulator's.  Narrow tiles: the decoding, 1100 clocks a block and warpgroup in Q4_K and twice that in Q6_K, and
// the way of a decoded block's place through decoding and MMAs: 16 tokens 49 us in Q4_K, 78 in Q6_K (one decoding warpgroup: 67 and 110), 64 tokens 58 and 87 (78 and 117).
// A thread takes all its codes into registers before it waits for the place of the decoded block (64 tokens 68 -> 64 us), and stores of 16 registers let the next
// ones be computed meanwhile.  A wait tries its barrier 64 times before it looks at the clock (250 against 255 us).  Not kept: chunks to the draining warpgroups in turn (263), a
// packed block's place given back as soon as its codes are in registers (64 -> 68 us with 64 tokens), sleeps between tries.
// Q4_K: two int8 planes per weight out of shared memory (the form before this one) took 1659 us where this takes 1204, for 2048 tokens x 28672 x
// 8192, 547 against 317 at 512 tokens, 169 against 67 at 16 (without the k_j, exact below 2^24 only: 1201, 316, 66).  Q6_K, whose two planes came from shared memory as well: 1637 against 1324,
// 624 against 351, 248 against 110; as two f16 addends into one f32 accumulator, with the decoded operand in a single buffer, it
// took 2125, 512 and 155, and was exact only below 2^24.
// Every wait is bounded; on a time-out the kernel records an error, lets its copies and MMAs end, frees its TMEM and returns.
#include "kq_tc.cuh"

#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>

namespace {

constexpr int NTHREADS = 512, CHUNK = 64, MAX_CHUNKS = 4, ROWS = 128, DA_RING = 8, SC_RING = 8;
// bytes of a token and block in an image: 256 f16 codes and 16 f16 sums (Q4_K), or 256 codes (Q6_K); eight tokens are [chunks of 16 bytes][8 tokens]
constexpr int TOK16 = KQ_TOK16, TOK8 = KQ_TOK8;
constexpr int TILE_OUT = MAX_CHUNKS * CHUNK * ROWS; // outputs of a tile
constexpr int MAX_CTAS = 256, MAX_DEVICES = 16, DRAIN_WARPS = 8;
constexpr uint64_t LIMIT = 5 * KQ_WAIT_LIMIT_NS;

// NARROW: tiles of one chunk.  Their blocks take the decoding longer than anything else, so two warpgroups decode, block by block in turn, and one drains;
// otherwise one decodes and each of two drains half of every chunk.
template <bool Q6, bool NARROW>
struct Cfg {
    static constexpr int DRAIN_WG = NARROW ? 1 : 2, DECODE_WG = 3 - DRAIN_WG;
    static constexpr int GROUPS = NARROW ? 4 : 8; // groups of 16 tokens whose results a draining thread holds
    static constexpr int REG_DRAIN = NARROW ? 184 : 208, REG_DECODE = NARROW ? 144 : 56, REG_REST = 40;
    static constexpr int REG_SUM = DRAIN_WG * REG_DRAIN + DECODE_WG * REG_DECODE + REG_REST;
    static_assert(REG_SUM <= 512, "registers of 512 threads, 128 each at the launch");
    static constexpr int RAW_BYTES = Q6 ? 13 * ROWS * 32 : ROWS * KQ_Q4K_BYTES; // Q6_K: two blocks of each row
    static constexpr int TOK_BYTES = Q6 ? TOK8 : TOK16, B_BYTES = CHUNK * TOK_BYTES;
    static constexpr int RAW_STAGES = Q6 ? 2 : 3, B_STAGES = Q6 ? 6 : 4;
    static constexpr int AMIN_BYTES = 8192; // Q4_K, per block: the operands m_j and k_j for the sums of 16, each twice
    static constexpr int SM_B = 0, SM_RAW = B_STAGES * B_BYTES, SM_AMIN = SM_RAW + RAW_STAGES * RAW_BYTES,
                         SM_DA = SM_AMIN + (Q6 ? 0 : 2 * AMIN_BYTES), SM_SC = SM_DA + DA_RING * CHUNK * 4, SMEM = SM_SC + SC_RING * ROWS * 4;
    static_assert(SM_RAW % 128 == 0 && RAW_BYTES % 128 == 0 && SM_AMIN % 16 == 0, "TMA destinations are 128-byte aligned");
    static_assert(SMEM <= 226 * 1024, "shared memory of a CTA");
    // the two issuing warps take alternate chunks: with an even number a stage is always the same warp's, which then waits for every phase of it
    static_assert(B_STAGES % 2 == 0, "a wait by parity must not miss a phase");
    // the one before it on its accumulator, q - 2, has been drained when chunk q is issued, and a stage is filled again when its chunk's MMAs are over: what the rings without
    // barriers of their own rely on
    static_assert(DA_RING >= B_STAGES + 2 && SC_RING >= 4, "rings");
};

__device__ int g_gemm_error;
// Parts of a cut tile that have been written, by the CTA that holds its first block and the draining warp; one set for each of the two launches
// (Q4_K, Q6_K) that may read an image, cleared by the launch that writes the image, so that a call which gave up leaves nothing behind.
__device__ int4 g_parts_done[2 * MAX_CTAS * DRAIN_WARPS / 4];

constexpr int MAX_SEGS = 3;
struct Seg { // one of the matrices that share the tokens
    float *y;
    const float *bias;
    const uint8_t *W;
    int32_t N, tile_end; // rows; row tiles up to this matrix's last
};
struct Params {
    CUtensorMap w[2 * MAX_SEGS]; // packed blocks; Q6_K: rows' full groups of eight blocks, then their last, smaller group
    Seg seg[MAX_SEGS];
    const uint8_t *img;    // token images [block][groups of 8 tokens]
    const float *da;       // activation scales [block][m_pad]
    float *part;
    const float *residual; // with one matrix only
    int32_t M, nb, m_pad, row_tiles, tok_tiles, tile_tok, min_share;
    int64_t w_row;
    // products with experts: token tile t belongs to expert tile_expert[t] and holds the tile_count[t] pairs row_src[tile_tok t ..]
    const int32_t *row_src, *tile_expert, *tile_count, *n_tiles;
    int32_t first_tile; // of the token tiles that n_tiles counts, the one that is tile 0 of this launch
};

// n tokens as c chunks of cw: one, or an even number, so that each accumulator and its issuing warp have the chunks of one parity
__host__ __device__ __forceinline__ void chunks_of(bool narrow, int n, int &c, int &cw) {
    c = narrow ? 1 : n <= 2 * CHUNK ? 2 : 4;
    cw = ((n + c - 1) / c + 15) & ~15;
}

struct TilePos {
    int n0, t0, n, c, cw, expert, seg;
};
// selects, not indexing: parameters indexed by a variable are read through generic loads
__device__ __forceinline__ int seg_rows(const Params &p, int s) { return s == 0 ? p.seg[0].N : s == 1 ? p.seg[1].N : p.seg[2].N; }
template <bool NARROW>
__device__ __forceinline__ TilePos tile_at(const Params &p, int tile) {
    TilePos t;
    const int tt = tile / p.row_tiles, rt = tile - tt * p.row_tiles;
    t.seg = (rt >= p.seg[0].tile_end) + (rt >= p.seg[1].tile_end);
    t.n0 = (rt - (t.seg == 0 ? 0 : t.seg == 1 ? p.seg[0].tile_end : p.seg[1].tile_end)) * ROWS;
    t.t0 = tt * p.tile_tok;
    if (p.row_src) t.n = p.tile_count[tt], t.expert = p.tile_expert[tt];
    else t.n = min(p.tile_tok, p.M - t.t0), t.expert = 0;
    chunks_of(NARROW, t.n, t.c, t.cw);
    return t;
}

__device__ __forceinline__ uint64_t nosw_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr & 0x3FFFF) >> 4) | (uint64_t)(lbo >> 4) << 16 | (uint64_t)(sbo >> 4) << 32 | (uint64_t)1 << 46;
}
__device__ __forceinline__ __half2 h2(uint32_t v) { return *reinterpret_cast<__half2 *>(&v); }
__device__ __forceinline__ uint32_t u2(__half2 v) { return *reinterpret_cast<uint32_t *>(&v); }
// byte b of v as an f16 pair, 1024 + byte in both halves
__device__ __forceinline__ __half2 byte_pair(uint32_t v, int b) { return h2(__byte_perm(v, 0x64646464u, 0x4040u | (b << 8) | b)); }
// bytes b and b + 1 of v as f16
__device__ __forceinline__ __half2 two_bytes(uint32_t v, int b) { return __hsub2(h2(__byte_perm(v, 0x64646464u, 0x4040u | ((b + 1) << 8) | b)), __float2half2_rn(1024.f)); }

#define TMEM_LD8(taddr, r)                                                                                              \
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"                                \
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])       \
                 : "r"(taddr)                                                                                           \
                 : "memory")
__device__ __forceinline__ void tmem_ld(uint32_t at, uint32_t (&r)[8]) { TMEM_LD8(at, r); }
__device__ __forceinline__ void tmem_ld(uint32_t at, uint32_t (&r)[16]) { TMEM_LD16(at, r); }
#define TMEM_ST4(taddr, r) \
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]) : "memory")

// kind::i8, A in TMEM (four elements to a column), s32 accumulators, B signed
__device__ __forceinline__ constexpr uint32_t idesc_i8(int m, int n, bool a_signed) {
    return (2u << 4) | ((a_signed ? 1u : 0u) << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void mma_i8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}"
                 :
                 : "r"(d_tmem), "r"(a_tmem), "l"(b), "r"(id), "r"(acc)
                 : "memory");
}

__device__ __forceinline__ void bar_init(uint64_t *b, int count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count)); }
__device__ __forceinline__ void bar_arrive(uint64_t *b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory"); }
__device__ __forceinline__ void bar_expect(uint64_t *b, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_in(uint32_t dst, const void *src, int bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(smem_u32(bar))
                 : "memory");
}

// Waits of a whole warp for up to three barriers: lane i < n asks for (bar, parity) of its own, the others ask for nothing (a try of
// 32 lanes takes 85 clocks even when the phase is over).  No time hint: with one, a warp wakes up to 900 clocks late (2048 tokens x
// 28672 x 8192: 1252 us with a hint of a millisecond, 1166 without, 1222 with a spin on test_wait).
__device__ __forceinline__ bool try_wait(uint32_t bar, uint32_t parity, int lane, int n) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p, a;\n\tsetp.lt.s32 a, %3, %4;\n\tsetp.ge.s32 p, %3, %4;\n\t"
                 "@a mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity), "r"(lane), "r"(n)
                 : "memory");
    return __all_sync(0xffffffffu, ok) != 0;
}
// What its lanes have waited for is there for every lane behind it, and for whom one of them then arrives for: a vote brings lanes together, but only
// __syncwarp orders their accesses to memory.
__device__ __forceinline__ bool wait_on(uint32_t bar, uint32_t parity, int lane, int n, volatile int *give_up, int code) {
    uint64_t t0 = 0;
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 64; i++)
            if (try_wait(bar, parity, lane, n)) {
                __syncwarp();
                return true;
            }
        const uint64_t now = kq_globaltimer_ns();
        if (!t0) t0 = now;
        const bool late = now - t0 > LIMIT;
        if (__any_sync(0xffffffffu, *give_up || late)) {
            *give_up = 1;
            if (late) atomicExch(&g_gemm_error, code);
            return false;
        }
    }
}

template <bool Q6, bool NARROW>
__global__ void __launch_bounds__(NTHREADS, 1) gemm_kq_kernel(const __grid_constant__ Params p) {
    using C = Cfg<Q6, NARROW>;
    constexpr int RAW_FULL = !Q6 && NARROW ? 2 * C::RAW_STAGES : C::RAW_STAGES; // blocks decoded in turn: a barrier per stage and warpgroup, which then sees each phase of its own
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t raw_full[RAW_FULL], raw_empty[C::RAW_STAGES], b_full[C::B_STAGES], b_empty[C::B_STAGES];
    __shared__ uint64_t a_full[2], a_empty[2], acc_full[2], acc_empty[2], s_end[2];
    __shared__ uint32_t s_tmem;
    __shared__ int s_abort;
    KQ_PDL_TRIGGER();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) {
        for (int i = 0; i < RAW_FULL; i++) bar_init(&raw_full[i], 1);
        for (int i = 0; i < C::RAW_STAGES; i++) bar_init(&raw_empty[i], Q6 && NARROW ? 8 : 4); // Q6_K: both warpgroups read a pair of blocks
        for (int i = 0; i < C::B_STAGES; i++) bar_init(&b_full[i], 1), bar_init(&b_empty[i], 1);
        for (int i = 0; i < 2; i++) // acc_full: the MMAs, and the issuing warp for the scales that it has waited for
            bar_init(&a_full[i], 4), bar_init(&a_empty[i], NARROW ? 1 : 2), bar_init(&acc_full[i], 2), bar_init(&acc_empty[i], 4 * C::DRAIN_WG), bar_init(&s_end[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        s_abort = 0;
    }
    KQ_PDL_WAIT(); // before the TMEM allocation: a CTA that starts early must not hold columns its predecessor needs
    if (warp == 15) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    // this CTA's share of the (tile, block) pairs: per pairs, one more for the first rem CTAs
    const int nb = p.nb;
    const uint32_t units = (uint32_t)(p.row_src ? max(0, min(*p.n_tiles - p.first_tile, p.tok_tiles)) : p.tok_tiles) * p.row_tiles * nb;
    const uint32_t ctas = max(1u, min(gridDim.x, units / p.min_share)), per = units / ctas, rem = units - per * ctas;
    const uint32_t u0 = blockIdx.x * per + min(blockIdx.x, rem);
    const int total = blockIdx.x < ctas ? per + (blockIdx.x < rem) : 0, tile0 = total ? u0 / nb : 0, b0 = u0 - tile0 * nb;
    auto wait = [&](uint64_t *bar, uint32_t parity, int code) { return wait_on(smem_u32(bar), parity, lane, 1, &s_abort, code); };

    if (warp >= 12) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::REG_REST));
        const bool lead = tc_elect();
        int tile = tile0, b = b0, k = 0;
        TilePos t = {};
        if (total) t = tile_at<NARROW>(p, tile);
        bool ok = true;
        if (warp == 12) { // packed weights
            for (int u = 0; u < total; u++) {
                if (!Q6 || u == 0 || b % 2 == 0) { // Q6_K: the two blocks of a pair come together
                    const int s = k % C::RAW_STAGES, round = k / C::RAW_STAGES;
                    if (round > 0 && !(ok = wait(&raw_empty[s], (round - 1) & 1, 1))) break;
                    if (lead) {
                        uint64_t *full = &raw_full[k % RAW_FULL];
                        bar_expect(full, C::RAW_BYTES);
                        const uint32_t dst = smem_u32(smem + C::SM_RAW + s * C::RAW_BYTES), bar = smem_u32(full);
                        const int row = t.expert * seg_rows(p, t.seg) + t.n0;
                        if (Q6) {
                            const int grp = b / KQ_Q6_GROUP, full = nb / KQ_Q6_GROUP, x = (b % KQ_Q6_GROUP) / 2 * 32;
                            const CUtensorMap *m = p.w + 2 * t.seg + (grp < full ? 0 : 1);
                            asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
                                         "l"(m), "r"(x), "r"(row), "r"(0), "r"(grp < full ? grp : 0), "r"(bar)
                                         : "memory");
                        } else {
                            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
                                         "l"(p.w + 2 * t.seg), "r"(b * KQ_Q4K_BYTES), "r"(row), "r"(bar)
                                         : "memory");
                        }
                    }
                    __syncwarp();
                    k++;
                }
                if (++b == nb) {
                    b = 0;
                    if (u + 1 < total) t = tile_at<NARROW>(p, ++tile);
                }
            }
            if (!ok && lead) // copies that were posted must land before the CTA goes away
                for (int i = max(0, k - C::RAW_STAGES); i < k; i++) kq_mbar_wait(smem_u32(&raw_full[i % RAW_FULL]), (i / RAW_FULL) & 1, KQ_WAIT_LIMIT_NS);
        } else if (warp == 13) { // token images and scales
            const int64_t block_bytes = (int64_t)p.m_pad * C::TOK_BYTES;
            for (int u = 0; u < total && ok; u++) {
                for (int c = 0; c < t.c; c++, k++) {
                    const int s = k % C::B_STAGES, round = k / C::B_STAGES;
                    if (round > 0 && !(ok = wait(&b_empty[s], (round - 1) & 1, 2))) break;
                    if (lead) {
                        const int tok = t.t0 + c * t.cw, d = k % DA_RING;
                        bar_expect(&b_full[s], t.cw * (C::TOK_BYTES + 4));
                        bulk_in(smem_u32(smem + C::SM_B + s * C::B_BYTES), p.img + b * block_bytes + (int64_t)tok * C::TOK_BYTES, t.cw * C::TOK_BYTES, &b_full[s]);
                        bulk_in(smem_u32(smem + C::SM_DA + d * CHUNK * 4), p.da + (int64_t)b * p.m_pad + tok, t.cw * 4, &b_full[s]);
                    }
                    __syncwarp();
                }
                if (++b == nb) {
                    b = 0;
                    if (u + 1 < total) t = tile_at<NARROW>(p, ++tile);
                }
            }
            if (!ok && lead)
                for (int i = max(0, k - C::B_STAGES); i < k; i++) kq_mbar_wait(smem_u32(&b_full[i % C::B_STAGES]), (i / C::B_STAGES) & 1, KQ_WAIT_LIMIT_NS);
        } else { // MMAs: a warp per accumulator, for the chunks of its parity (NARROW: blocks of its parity)
            const int w = warp & 1;
            int n = 0; // chunks this warp has issued
            for (int u = 0; u < total && ok; u++) {
                const uint32_t id = Q6 ? idesc_i8(128, t.cw, true) : tc_idesc(128, t.cw, false, false), sa = u & 1, pa = (u >> 1) & 1;
                for (int c = NARROW ? (sa ^ w) : w; c < t.c; c += 2, n++) {
                    const int q = k + c, s = q % C::B_STAGES;
                    // tokens with their scales, the accumulator (free from the start), and once a block the decoded weights
                    const uint32_t bar = smem_u32(lane == 1 && n ? &acc_empty[w] : lane == 2 ? &a_full[sa] : &b_full[s]);
                    const uint32_t par = lane == 1 && n ? (n - 1) & 1 : lane == 2 ? pa : (q / C::B_STAGES) & 1;
                    if (!(ok = wait_on(bar, par, lane, NARROW || c == w ? 3 : 2, &s_abort, 3))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t bd = nosw_desc(smem_u32(smem + C::SM_B + s * C::B_BYTES), 128, 8 * C::TOK_BYTES);
                    const uint32_t acc = tmem + 256 + w * 2 * CHUNK, a = tmem + sa * 128;
                    if (lead) {
                        bar_arrive(&acc_full[w]); // hands on what this warp has waited for: the scales of the tokens and of the weights
                        if (Q6) {
#pragma unroll 4
                            for (int i = 0; i < 8; i++) mma_i8_ts(acc, a + i * 8, bd + i * 16, id, i > 0);
                            const uint32_t id_lo = idesc_i8(128, t.cw, false);
#pragma unroll 4
                            for (int i = 0; i < 8; i++) mma_i8_ts(acc + CHUNK, a + 64 + i * 8, bd + i * 16, id_lo, i > 0);
                        } else {
#pragma unroll 4
                            for (int i = 0; i < 16; i++) tc_mma_ts(acc, a + i * 8, bd + i * 16, id, i > 0);
                            const uint32_t mins = smem_u32(smem + C::SM_AMIN + sa * C::AMIN_BYTES);
                            tc_mma_ss(acc, nosw_desc(mins + 4096, 2048, 128), bd + 256, id, 1); // last: the others are exact
                            tc_mma_ss(acc + CHUNK, nosw_desc(mins, 2048, 128), bd + 256, id, 0);
                        }
                        tc_commit(smem_u32(&acc_full[w]));
                        if (c + 2 >= t.c) tc_commit(smem_u32(&a_empty[sa])); // this warp's last use of the decoded weights
                        tc_commit(smem_u32(&b_empty[s]));
                    }
                    __syncwarp();
                }
                k += t.c;
                if (++b == nb) {
                    b = 0;
                    if (u + 1 < total) t = tile_at<NARROW>(p, ++tile);
                }
            }
            if (!ok && lead) { // MMAs in flight end before TMEM is freed
                tc_commit(smem_u32(&s_end[w]));
                kq_mbar_wait(smem_u32(&s_end[w]), 0, KQ_WAIT_LIMIT_NS);
            }
        }
        __syncwarp();
    } else if (warp >= 4 * C::DRAIN_WG) { // decode the packed blocks into TMEM, a thread per row
        if (NARROW) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::REG_DECODE));
        else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::REG_DECODE));
        const int row = tid & 127, turn = NARROW ? (warp >> 2) - 1 : 0; // NARROW: this warpgroup takes the blocks of its parity
        const uint32_t tl = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        if (!Q6) {
            const __half2 k1024 = __float2half2_rn(1024.f);
            for (int u = turn; u < total; u += C::DECODE_WG) {
                const int s = u % C::RAW_STAGES, sa = u & 1;
                if (!wait(&raw_full[u % RAW_FULL], (u / RAW_FULL) & 1, 6)) break;
                const uint8_t *blk = smem + C::SM_RAW + s * C::RAW_BYTES + row * KQ_Q4K_BYTES;
                const uint4 hdr = *reinterpret_cast<const uint4 *>(blk);
                const uint32_t sc_lo = hdr.y & 0x3F3F3F3Fu, sc_hi = (hdr.w & 0x0F0F0F0Fu) | ((hdr.y >> 2) & 0x30303030u);
                uint4 codes[8];
                if (NARROW)
#pragma unroll
                    for (int i = 0; i < 8; i++) codes[i] = *reinterpret_cast<const uint4 *>(blk + 16 + 16 * i);
                // the place of the decoded blocks (free from the start)
                if (u >= 2 && !wait(&a_empty[sa], ((u >> 1) - 1) & 1, 7)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                { // m_j, then k_j, in order of j, for the sums of 16 of even and of odd place
                    const uint32_t m_lo = hdr.z & 0x3F3F3F3Fu, m_hi = ((hdr.w >> 4) & 0x0F0F0F0Fu) | ((hdr.z >> 2) & 0x30303030u);
                    uint4 *am = reinterpret_cast<uint4 *>(smem + C::SM_AMIN + sa * C::AMIN_BYTES + (row >> 3) * 128 + (row & 7) * 16);
                    am[0] = am[128] = make_uint4(u2(two_bytes(m_lo, 0)), u2(two_bytes(m_lo, 2)), u2(two_bytes(m_hi, 0)), u2(two_bytes(m_hi, 2)));
                    auto k = [&](__half2 sc) { // what the decoding below takes off two neighbouring sub-blocks
                        return u2(__hfma2(sc, __floats2half2_rn(-1024.f, 0.f), __hmul2(sc, __floats2half2_rn(1032.f, 8.f))));
                    };
                    am[256] = am[384] = make_uint4(k(two_bytes(sc_lo, 0)), k(two_bytes(sc_lo, 2)), k(two_bytes(sc_hi, 0)), k(two_bytes(sc_hi, 2)));
                    *reinterpret_cast<uint32_t *>(smem + C::SM_SC + ((u % SC_RING) * ROWS + row) * 4) = hdr.x;
                }
#pragma unroll (NARROW ? 4 : 1)
                for (int g = 0; g < 4; g++) { // 64 elements: sub-block 2g in the low nibbles, 2g + 1 in the high ones
                    const uint32_t scw = (g < 2 ? sc_lo : sc_hi) >> (16 * (g & 1));
                    const __half2 s0 = __hsub2(byte_pair(scw, 0), k1024), s1 = __hsub2(byte_pair(scw, 1), k1024);
                    // (1024 + q) sc - f16(1032 sc) and (1024 + 16 q) sc / 16 - 72 sc: one rounding, of an exact result.  f16(1032 sc) - 1024 sc = k is
                    // within 16 of 8 sc and a multiple of 32 from sc = 32 on: -512 <= sc q - k <= 441 for every scale
                    const __half2 o0 = __hmul2(s0, __float2half2_rn(-1032.f)), t1 = __hmul2(s1, __float2half2_rn(0.0625f)),
                                  o1 = __hmul2(s1, __float2half2_rn(-72.f));
                    uint32_t o[32];
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const uint4 w4 = NARROW ? codes[2 * g + h] : *reinterpret_cast<const uint4 *>(blk + 16 + 32 * g + 16 * h);
                        const uint32_t w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                        for (int i = 0; i < 4; i++) {
                            const uint32_t v = w[i] >> 8;
                            o[8 * h + 2 * i] = u2(__hfma2(h2((w[i] & 0x000F000Fu) | 0x64006400u), s0, o0));
                            o[8 * h + 2 * i + 1] = u2(__hfma2(h2((v & 0x000F000Fu) | 0x64006400u), s0, o0));
                            o[16 + 8 * h + 2 * i] = u2(__hfma2(h2((w[i] & 0x00F000F0u) | 0x64006400u), t1, o1));
                            o[16 + 8 * h + 2 * i + 1] = u2(__hfma2(h2((v & 0x00F000F0u) | 0x64006400u), t1, o1));
                        }
                    }
                    TMEM_ST16(tl + sa * 128 + g * 32, o);
                    TMEM_ST16(tl + sa * 128 + g * 32 + 16, (o + 16));
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // the min operand, for the MMA
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) bar_arrive(&a_full[sa]), bar_arrive(&raw_empty[s]);
            }
        } else {
            int tile = tile0, b = b0, k = -1;
            uint4 dv = make_uint4(0, 0, 0, 0); // block scales of the row's group of eight blocks
            const uint8_t *wr = nullptr;
            for (int u = 0; u < total; u++) {
                const int sa = u & 1;
                if (u == 0 || b == 0) {
                    const TilePos t = tile_at<NARROW>(p, tile);
                    const int n = seg_rows(p, t.seg);
                    wr = (t.seg == 0 ? p.seg[0].W : t.seg == 1 ? p.seg[1].W : p.seg[2].W) + ((int64_t)t.expert * n + min(t.n0 + row, n - 1)) * p.w_row;
                }
                if (u == 0 || b % KQ_Q6_GROUP == 0)
                    dv = __ldg(reinterpret_cast<const uint4 *>(wr + kq_q6_addr(nb, b / KQ_Q6_GROUP * KQ_Q6_GROUP).d));
                if (u == 0 || b % 2 == 0) {
                    k++;
                    if (!wait(&raw_full[k % C::RAW_STAGES], (k / C::RAW_STAGES) & 1, 6)) break;
                }
                const int s = k % C::RAW_STAGES;
                if (!NARROW || sa == turn) {
                    if (u >= 2 && !wait(&a_empty[sa], ((u >> 1) - 1) & 1, 7)) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint8_t *blk = smem + C::SM_RAW + s * C::RAW_BYTES + row * 32 + (b & 1) * 16; // chunk i of the block 4096 i further
                    const uint4 sc4 = *reinterpret_cast<const uint4 *>(blk + 12 * 4096);
                    const int b8 = b % KQ_Q6_GROUP;
                    const uint32_t dw = b8 < 2 ? dv.x : b8 < 4 ? dv.y : b8 < 6 ? dv.z : dv.w;
                    *reinterpret_cast<uint32_t *>(smem + C::SM_SC + ((u % SC_RING) * ROWS + row) * 4) = (b8 & 1 ? dw >> 16 : dw) & 0xFFFFu;
#pragma unroll (NARROW ? 2 : 1)
                    for (int hh = 0; hh < 2; hh++) { // 128 elements
                        const uint32_t sc_a = hh ? sc4.z : sc4.x, sc_b = hh ? sc4.w : sc4.y;
                        uint32_t wide_hi[NARROW ? 32 : 4], wide_lo[NARROW ? 32 : 4]; // NARROW: 128 elements at a time, for more independent work
#pragma unroll (NARROW ? 2 : 1)
                        for (int h = 0; h < 2; h++) { // elements 128 hh + 32 q + 16 h + ..
                            const uint4 a4 = *reinterpret_cast<const uint4 *>(blk + (4 * hh + h) * 4096), c4 = *reinterpret_cast<const uint4 *>(blk + (4 * hh + 2 + h) * 4096),
                                        q4 = *reinterpret_cast<const uint4 *>(blk + (8 + 2 * hh + h) * 4096);
                            const uint32_t a[4] = {a4.x, a4.y, a4.z, a4.w}, c[4] = {c4.x, c4.y, c4.z, c4.w}, qh[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                            for (int q = 0; q < 4; q++) { // 16 elements: scale group 8 hh + 2 q + h
                                // Two codes to a register, 16 bits each: 4 (sc (q - 32) + 8192) is between 16384 and 49152, so neither half reaches into the
                                // other.  Its upper byte is hi + 128, its lower one 4 lo.
                                const int sc = (int)((q < 2 ? sc_a : sc_b) << (24 - 8 * ((2 * q) & 3) - 8 * h)) >> 24;
                                const uint32_t k4 = 4u * (uint32_t)sc, base = 0x80008000u - 0x00800080u * (uint32_t)sc;
                                uint32_t *hi = wide_hi + (NARROW ? 8 * q + 4 * h : 0), *lo = wide_lo + (NARROW ? 8 * q + 4 * h : 0);
#pragma unroll
                                for (int i = 0; i < 4; i++) {
                                    const uint32_t n = q & 1 ? c[i] : a[i], top = q == 0 ? qh[i] << 4 : q == 1 ? qh[i] << 2 : q == 2 ? qh[i] : qh[i] >> 2;
                                    const uint32_t code = ((q & 2 ? n >> 4 : n) & 0x0F0F0F0Fu) | (top & 0x30303030u);
                                    const uint32_t even = (code & 0x00FF00FFu) * k4 + base, odd = ((code >> 8) & 0x00FF00FFu) * k4 + base;
                                    hi[i] = __byte_perm(even, odd, 0x7351) ^ 0x80808080u;
                                    lo[i] = __byte_perm(even, odd, 0x6240);
                                }
                                const uint32_t at = tl + sa * 128 + 32 * hh + 8 * q + 4 * h;
                                if (!NARROW) {
                                    TMEM_ST4(at, hi);
                                    TMEM_ST4(at + 64, lo);
                                }
                            }
                        }
                        if constexpr (NARROW) {
                            TMEM_ST32(tl + sa * 128 + 32 * hh, wide_hi);
                            TMEM_ST32(tl + sa * 128 + 32 * hh + 64, wide_lo);
                        }
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) bar_arrive(&a_full[sa]);
                }
                if (lane == 0 && (b % 2 == 1 || b == nb - 1)) bar_arrive(&raw_empty[s]);
                if (++b == nb) b = 0, tile++;
            }
        }
        __syncwarp();
    } else { // add the accumulators to the running result
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::REG_DRAIN));
        const int row = tid & 127, half = NARROW ? 0 : (warp >> 2) * (CHUNK / 2); // of two warpgroups each takes half of every chunk
        const uint32_t tl = tmem + 256 + ((uint32_t)((warp & 3) * 32) << 16);
        constexpr int STEP = 16, PART = CHUNK / C::DRAIN_WG;
        float y[C::GROUPS][16]; // [chunk, group of its part][token]
        int tile = tile0, b = b0, n = 0, u = 0;
        bool ok = true;
        while (u < total) { // a tile, or this CTA's part of it
            const TilePos t = tile_at<NARROW>(p, tile);
            const int end = u + min(nb - b, total - u);
            const bool whole = b == 0 && end - u == nb;
#pragma unroll
            for (int i = 0; i < C::GROUPS * 16; i++) y[i / 16][i % 16] = 0.f;
            // the loop over the blocks holds nothing else: with the tile's end inside it a turn took a thousand clocks more
#pragma unroll 1
            for (; u < end; u++) {
#pragma unroll
                for (int c = 0; c < (NARROW ? 1 : MAX_CHUNKS); c++) {
                    if (c >= t.c) break;
                    const int slot = n & 1;
                    if (!(ok = wait(&acc_full[slot], (n >> 1) & 1, 9))) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t ta = tl + slot * 2 * CHUNK + half;
                    const float *da = reinterpret_cast<const float *>(smem + C::SM_DA + n % DA_RING * CHUNK * 4) + half;
                    uint32_t m[2][STEP], l[2][STEP]; // two steps: one on its way while the other is added
                    tmem_ld(ta, m[0]);
                    tmem_ld(ta + CHUNK, l[0]);
                    float2 df = __half22float2(h2(*reinterpret_cast<const uint32_t *>(smem + C::SM_SC + ((u % SC_RING) * ROWS + row) * 4))); // d_w, d_min
                    if (Q6) df.x *= 0.25f; // the sums come four times
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int st = 0; st < PART / STEP; st++) { // y += d_a (d_w main - d_min min), or d_a d_w (64 hi + lo)
                        if (half + st * STEP >= t.cw) break;
                        if (st + 1 < PART / STEP) { // behind the last step it loads what nobody uses
                            tmem_ld(ta + (st + 1) * STEP, m[(st + 1) & 1]);
                            tmem_ld(ta + (st + 1) * STEP + CHUNK, l[(st + 1) & 1]);
                        }
                        const uint32_t(&mv)[STEP] = m[st & 1], (&lv)[STEP] = l[st & 1];
#pragma unroll
                        for (int j = 0; j < STEP; j += 4) {
                            const float4 da4 = *reinterpret_cast<const float4 *>(da + st * STEP + j);
                            float *acc = &y[c * (PART / 16) + st][j];
#pragma unroll
                            for (int e = 0; e < 4; e += 2) { // two tokens per instruction: 28672 x 8192 at 512 tokens 325 -> 316 us
                                const float2 main = Q6 ? make_float2(__int2float_rn((int)(mv[j + e] * 256u + lv[j + e])), __int2float_rn((int)(mv[j + e + 1] * 256u + lv[j + e + 1])))
                                                       : make_float2(__uint_as_float(mv[j + e]), __uint_as_float(mv[j + e + 1]));
                                float2 v = __fmul2_rn(make_float2(df.x, df.x), main);
                                if (!Q6) v = __ffma2_rn(make_float2(-df.y, -df.y), make_float2(__uint_as_float(lv[j + e]), __uint_as_float(lv[j + e + 1])), v);
                                const float2 r = __ffma2_rn(e ? make_float2(da4.z, da4.w) : make_float2(da4.x, da4.y), v, make_float2(acc[e], acc[e + 1]));
                                acc[e] = r.x, acc[e + 1] = r.y;
                            }
                        }
                        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    }
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) bar_arrive(&acc_empty[slot]);
                    n++;
                }
                if (!ok) break;
            }
            if (!ok) break;
            { // the end of this CTA's part of the tile
                const uint32_t first = (uint32_t)tile * nb, big = rem * (per + 1);
                // the CTAs that hold the tile's first and last block
                auto cta_of = [&](uint32_t v) { return v < big ? v / (per + 1) : rem + (v - big) / per; };
                const uint32_t c0 = cta_of(first), c1 = cta_of(first + nb - 1);
                // 16 tokens of this thread's row, from token col0 of the tile on
                const Seg &sg = t.seg == 0 ? p.seg[0] : t.seg == 1 ? p.seg[1] : p.seg[2];
                const int N = sg.N;
                float *const y_out = sg.y;
                const float *const bias_in = sg.bias;
                auto put = [&](float (&v)[16], int col0) {
                    const int n = t.n0 + row, live = t.n - col0;
                    if (n >= N) return;
                    if (p.row_src) {
                        const int32_t *src = p.row_src + t.t0 + col0;
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            if (j < live) y_out[(int64_t)src[j] * N + n] = v[j];
                        return;
                    }
                    const int64_t o = (int64_t)(t.t0 + col0) * N + n;
                    if (bias_in) {
                        const float bias = bias_in[n];
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] += bias;
                    }
                    if (p.residual) {
                        const float *src = p.residual + o;
#pragma unroll
                        for (int j = 0; j < 16; j++, src += N)
                            if (j < live) v[j] += *src;
                    }
                    float *dst = y_out + o;
#pragma unroll
                    for (int j = 0; j < 16; j++, dst += N)
                        if (j < live) *dst = v[j];
                };
#pragma unroll 1
                for (int i = 0; i < C::GROUPS; i++) { // one copy of this code for all of y: it runs once per tile
                    const int c = i / (PART / 16), g16 = half + i % (PART / 16) * 16, col0 = c * t.cw + g16;
                    if (c >= t.c || g16 >= t.cw || col0 >= t.n) continue;
                    float v[16];
#define TAKE(I) case I: { _Pragma("unroll") for (int j = 0; j < 16; j++) v[j] = y[I][j]; } break
                    switch (i) {
                        TAKE(0);
                        TAKE(1);
                        TAKE(2);
                        TAKE(3);
                    default:
                        if constexpr (!NARROW)
                            switch (i) {
                                TAKE(4);
                                TAKE(5);
                                TAKE(6);
                                TAKE(7);
                            }
                    }
#undef TAKE
                    if (whole) {
                        put(v, col0);
                    } else {
                        float *dst = p.part + ((int64_t)blockIdx.x * 2 + (first >= u0 ? 1 : 0)) * TILE_OUT + (c * CHUNK + g16) * ROWS + row;
#pragma unroll
                        for (int j = 0; j < 16; j++) __stcg(dst + j * ROWS, v[j]);
                    }
                }
                if (!whole) {
                    __threadfence();
                    __syncwarp();
                    int before = 0;
                    if (lane == 0) before = atomicAdd(reinterpret_cast<int *>(g_parts_done) + ((Q6 ? MAX_CTAS : 0) + c0) * DRAIN_WARPS + warp, 1);
                    before = __shfl_sync(0xffffffffu, before, 0);
                    if (before == (int)(c1 - c0)) { // this warp's part of the tile is complete
                        __threadfence();
#pragma unroll 1
                        for (int i = 0; i < C::GROUPS; i++) {
                            const int c = i / (PART / 16), g16 = half + i % (PART / 16) * 16, col0 = c * t.cw + g16;
                            if (c >= t.c || g16 >= t.cw || col0 >= t.n) continue;
                            float v[16];
#pragma unroll
                            for (int j = 0; j < 16; j++) v[j] = 0.f;
                            const float *src = p.part + ((int64_t)c0 * 2 + 1) * TILE_OUT + (c * CHUNK + g16) * ROWS + row;
                            // the first CTA's second part, then the first parts of the others; eight at a time, so that their trips to L2 overlap
#pragma unroll 1
                            for (uint32_t cc = c0; cc <= c1; cc += 8) {
                                float part[8][16];
#pragma unroll
                                for (int r = 0; r < 8; r++) {
                                    const float *from = src + (cc + r == c0 ? 0 : (int64_t)(2 * (cc + r - c0) - 1) * TILE_OUT);
#pragma unroll
                                    for (int j = 0; j < 16; j++) part[r][j] = cc + r <= c1 ? __ldcg(from + j * ROWS) : 0.f;
                                }
#pragma unroll
                                for (int r = 0; r < 8; r++)
                                    if (cc + r <= c1)
#pragma unroll
                                        for (int j = 0; j < 16; j++) v[j] += part[r][j];
                            }
                            put(v, col0);
                        }
                    }
                }
            }
            b = 0, tile++;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 15) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}


// Q8 rows -> the token operand, in the forms that the call's matrices read.  A thread writes 16 bytes of a token: eight codes (or sums of 16) as
// f16, in the order in which Q4_K weights are decoded (0 2 1 3 of every four), or 16 codes.  grid (runs of 16 tokens, blocks); tokens past
// the last are zeros.  The first CTA clears the counters of cut tiles for the products that read this image.
struct ImageParams {
    const int8_t *q;
    const float *d;
    const int16_t *bs;
    uint8_t *img16, *img8; // null: not wanted
    float *da;
    int32_t M, nb, m_pad, act_div;
    const int32_t *row_src, *tile_count, *n_tiles; // products with experts
    int32_t first_tile, tile_tok, narrow;
};
__global__ void __launch_bounds__(288) act_image_kernel(const __grid_constant__ ImageParams p) {
    KQ_PDL_ENTER();
    if (blockIdx.x == 0 && blockIdx.y == 0)
        for (int i = threadIdx.x; i < 2 * MAX_CTAS * DRAIN_WARPS / 4; i += blockDim.x) g_parts_done[i] = make_int4(0, 0, 0, 0);
    const int b = blockIdx.y, base = blockIdx.x * 16;
    int n_live = p.M - base; // tokens of this run
    if (p.row_src) {
        const int tile = base / p.tile_tok, at = base - tile * p.tile_tok;
        if (tile >= *p.n_tiles - p.first_tile) return;
        const int n = p.tile_count[tile];
        int c, cw;
        chunks_of(p.narrow, n, c, cw);
        if (at >= c * cw) return;
        n_live = n - at;
    }
    const __half2 k1152 = __float2half2_rn(1152.f);
    auto source_row = [&](int at) { return (int64_t)(p.row_src ? p.row_src[base + at] / p.act_div : base + at) * p.nb + b; };
    if (threadIdx.x < 16) p.da[(int64_t)b * p.m_pad + base + threadIdx.x] = (int)threadIdx.x < n_live ? p.d[source_row(threadIdx.x)] : 0.f;
    if (p.img16) {
        for (int i = threadIdx.x; i < 2 * 34 * 8; i += blockDim.x) {
            const int r = i & 7, kc = (i >> 3) % 34, g = i / 272, at = g * 8 + r; // token at of the run
            uint4 o = make_uint4(0, 0, 0, 0);
            if (at < n_live) {
                const int64_t m = source_row(at);
                if (kc < 32) {
                    const uint2 v = *reinterpret_cast<const uint2 *>(p.q + m * 256 + kc * 8);
                    const uint32_t x = v.x ^ 0x80808080u, y = v.y ^ 0x80808080u;
                    o.x = u2(__hsub2(h2((x & 0x00FF00FFu) | 0x64006400u), k1152));
                    o.y = u2(__hsub2(h2(((x >> 8) & 0x00FF00FFu) | 0x64006400u), k1152));
                    o.z = u2(__hsub2(h2((y & 0x00FF00FFu) | 0x64006400u), k1152));
                    o.w = u2(__hsub2(h2(((y >> 8) & 0x00FF00FFu) | 0x64006400u), k1152));
                } else { // |sum of 16| <= 2048: exact.  Those of even place, then those of odd place
                    const int4 *sums = reinterpret_cast<const int4 *>(p.bs + m * 16);
                    const int4 s8[2] = {sums[0], sums[1]};
                    const int16_t *s = reinterpret_cast<const int16_t *>(&s8[0]);
                    __half h[8];
#pragma unroll
                    for (int j = 0; j < 8; j++) h[j] = __int2half_rn((int)(kc == 32 ? s[2 * j] : s[2 * j + 1]));
                    o = *reinterpret_cast<uint4 *>(&h[0]);
                }
            }
            *reinterpret_cast<uint4 *>(p.img16 + ((int64_t)b * p.m_pad + base) * TOK16 + g * 8 * TOK16 + kc * 128 + r * 16) = o;
        }
    }
    if (p.img8) {
        for (int i = threadIdx.x; i < 2 * 16 * 8; i += blockDim.x) {
            const int r = i & 7, kc = (i >> 3) & 15, g = i >> 7, at = g * 8 + r;
            uint4 o = make_uint4(0, 0, 0, 0);
            if (at < n_live) o = *reinterpret_cast<const uint4 *>(p.q + source_row(at) * 256 + kc * 16);
            *reinterpret_cast<uint4 *>(p.img8 + ((int64_t)b * p.m_pad + base) * TOK8 + g * 8 * TOK8 + kc * 128 + r * 16) = o;
        }
    }
}

// ---- expert-major order of the (token, slot) pairs of a routed batch (MUL_MAT_ID with many tokens) ----
// A stable counting sort by expert: the pairs of expert e, in pair order, become the rows of that
// expert's token tiles; every expert starts on a tile boundary, the rows behind its last pair are
// padding (-1).  One CTA of 16 warps; warp w walks a contiguous range of the pairs 32 at a time, so the
// order inside an expert is the pair order whatever the timing (with 8 warps and a serial table of tiles 55 us
// for 8192 pairs and 128 experts, with 16 and a parallel table 27, with the experts asked for ahead and compared once 17).  Output: n_tiles, the expert of each
// tile, and for each tile row the pair it holds.
constexpr int SORT_WARPS = 16, SORT_MAX_E = 256;
__global__ void __launch_bounds__(SORT_WARPS * 32) moe_sort_kernel(const int32_t *ids, int n_pairs, int E, int TM,
                                                                   int32_t *n_tiles_out, int32_t *tile_expert, int32_t *row_src,
                                                                   int32_t *tile_count) {
    KQ_PDL_ENTER();
    __shared__ int cnt[SORT_WARPS][SORT_MAX_E]; // pass 1: pairs of expert e in warp w's range; then the range's offset inside the expert
    __shared__ int tile_start[SORT_MAX_E];
    __shared__ int s_tiles, s_warp[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = threadIdx.x; i < SORT_WARPS * SORT_MAX_E; i += blockDim.x) (&cnt[0][0])[i] = 0;
    __syncthreads();
    const int chunk = ((n_pairs + SORT_WARPS - 1) / SORT_WARPS + 31) & ~31;
    const int begin = min(n_pairs, warp * chunk), end = min(n_pairs, begin + chunk);
    // experts of the warp's pairs from i on, AHEAD runs of 32: asked for together, since a run's own trip to L2 would take longer than its work
    constexpr int AHEAD = 16;
    int ex[AHEAD];
    unsigned mates[AHEAD]; // the run's pairs of the same expert: found once, by pairs that fit (with some thirty experts in a run it takes longer than the rest)
    const bool once = end - begin <= AHEAD * 32;
    auto fetch = [&](int i) {
#pragma unroll
        for (int j = 0; j < AHEAD; j++) {
            const int pr = i + j * 32 + lane;
            const int e = pr < end ? ids[pr] : -1;
            ex[j] = e < E ? max(e, -1) : -1; // not an expert of this table: the pair is dropped
        }
    };
    for (int i0 = begin; i0 < end; i0 += AHEAD * 32) {
        fetch(i0);
#pragma unroll
        for (int j = 0; j < AHEAD; j++) {
            if (i0 + j * 32 >= end) break;
            const int e = ex[j];
            const unsigned same = mates[j] = __match_any_sync(0xffffffffu, e);
            if (e >= 0 && lane == __ffs(same) - 1) cnt[warp][e] += __popc(same);
            __syncwarp();
        }
    }
    __syncthreads();
    if ((int)threadIdx.x < E) {
        int run = 0;
        for (int w = 0; w < SORT_WARPS; w++) {
            const int c = cnt[w][threadIdx.x];
            cnt[w][threadIdx.x] = run;
            run += c;
        }
        tile_start[threadIdx.x] = run; // the expert's pair count, for the moment
    }
    __syncthreads();
    if (warp < 8) { // tiles in front of every expert's first: a scan over the warp, then over the warps
        const int e = threadIdx.x, n = e < E ? tile_start[e] : 0, nt = (n + TM - 1) / TM;
        int incl = nt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        if (lane == 31) s_warp[warp] = incl;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        int t = incl - nt;
        for (int w = 0; w < warp; w++) t += s_warp[w];
        if (e < E) {
            tile_start[e] = t;
            for (int k = 0; k < nt; k++) tile_expert[t + k] = e, tile_count[t + k] = min(TM, n - k * TM);
            if (e == E - 1) {
                s_tiles = t + nt;
                *n_tiles_out = t + nt;
            }
        }
    }
    __syncthreads();
    const int live = s_tiles * TM;
    if (((uintptr_t)row_src & 15) == 0) {
        for (int i = threadIdx.x; i < live / 4; i += blockDim.x) reinterpret_cast<int4 *>(row_src)[i] = make_int4(-1, -1, -1, -1);
    } else {
        for (int i = threadIdx.x; i < live; i += blockDim.x) row_src[i] = -1;
    }
    __syncthreads();
    for (int i0 = begin; i0 < end; i0 += AHEAD * 32) {
        if (!once) fetch(i0);
#pragma unroll
        for (int j = 0; j < AHEAD; j++) {
            if (i0 + j * 32 >= end) break;
            const int e = ex[j];
            const unsigned same = once ? mates[j] : __match_any_sync(0xffffffffu, e);
            const int leader = __ffs(same) - 1;
            int base = 0;
            if (e >= 0 && lane == leader) base = cnt[warp][e];
            base = __shfl_sync(0xffffffffu, base, leader);
            if (e >= 0) row_src[tile_start[e] * TM + base + __popc(same & ((1u << lane) - 1u))] = i0 + j * 32 + lane;
            __syncwarp();
            if (e >= 0 && lane == leader) cnt[warp][e] = base + __popc(same);
            __syncwarp();
        }
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                  const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
} // namespace

// Generic tiled tensor map for other kernels (the type lives in <cuda.h>; callers pass 128 bytes).
// elem_bytes 1, 2 or 8; swizzle128 selects the 128-byte swizzle (inner box extent <= 128 bytes).
b200_status kq_tmap_encode(void *map128, int elem_bytes, int rank, const void *base, const uint64_t *dims,
                           const uint64_t *strides_bytes, const uint32_t *box, int swizzle128) {
    static EncodeTiledFn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qr = cudaDriverEntryPointSymbolNotFound;
        KQ_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qr));
        KQ_REQUIRE(fn && qr == cudaDriverEntryPointSuccess, "the driver does not export cuTensorMapEncodeTiled");
        encode = (EncodeTiledFn)fn;
    }
    cuuint64_t d[5], sb[4];
    cuuint32_t bx[5], es[5];
    for (int i = 0; i < rank; i++) {
        d[i] = dims[i];
        bx[i] = box[i];
        es[i] = 1;
        if (i + 1 < rank) sb[i] = strides_bytes[i];
    }
    const CUresult rc = encode((CUtensorMap *)map128, elem_bytes == 8 ? CU_TENSOR_MAP_DATA_TYPE_UINT64 : elem_bytes == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8,
                               (cuuint32_t)rank, const_cast<void *>(base), d, sb, bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                               swizzle128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    KQ_REQUIRE(rc == CUDA_SUCCESS, "tensor map encode failed (%d)", (int)rc);
    return B200_OK;
}

namespace {
// Images, scales and parts of cut tiles, per device.  Launches that share them are ordered by the library's rule (one stream per device
// at a time).  A buffer grows to what is needed and the old one is given back, unless a stream was being captured when it was handed out: the graph
// holds its address, so it is kept, and the next one is twice as large (up to the largest that a call asks for), so that all that are kept
// stay below that size together.
constexpr int64_t SLAB_BYTES = 64 << 20, GROUP_BYTES = 256 << 20; // images of one launch: dense products, products with experts

struct Scratch {
    uint8_t *img16, *img8;
    float *da, *part;
    int4 *parts_done;
    int dev;
};
b200_status scratch(int dev, size_t img16_bytes, size_t img8_bytes, size_t da_bytes, cudaStream_t st, Scratch *out) {
    static std::mutex mu;
    static void *buf[MAX_DEVICES][4];
    static size_t cap[MAX_DEVICES][4];
    static bool captured[MAX_DEVICES][4];
    static int4 *parts_done[MAX_DEVICES];
    std::lock_guard<std::mutex> lock(mu);
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    KQ_CUDA(cudaStreamIsCapturing(st, &cs));
    const bool capturing = cs != cudaStreamCaptureStatusNone;
    const size_t need[4] = {img16_bytes, img8_bytes, da_bytes, (size_t)kq_sm_count() * 2 * TILE_OUT * 4};
    for (int i = 0; i < 4; i++) {
        if (need[i] > cap[dev][i]) {
            // an allocation is no work of the stream that is being captured
            cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
            KQ_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
            size_t bytes = need[i];
            cudaError_t e = cudaSuccess;
            if (buf[dev][i]) {
                if (captured[dev][i] || capturing) {
                    bytes = std::max(bytes, std::min(2 * cap[dev][i], (size_t)GROUP_BYTES));
                } else {
                    e = cudaDeviceSynchronize();
                    if (e == cudaSuccess) e = cudaFree(buf[dev][i]);
                }
                buf[dev][i] = nullptr;
                cap[dev][i] = 0;
                captured[dev][i] = false;
            }
            if (e == cudaSuccess) e = cudaMalloc(&buf[dev][i], bytes);
            if (e != cudaSuccess && bytes > need[i]) {
                cudaGetLastError();
                e = cudaMalloc(&buf[dev][i], bytes = need[i]);
            }
            cudaThreadExchangeStreamCaptureMode(&mode);
            if (e != cudaSuccess) {
                cudaGetLastError();
                buf[dev][i] = nullptr;
                kq_set_error("gemm: cudaMalloc(%zu) failed: %s", need[i], cudaGetErrorString(e));
                return B200_ERR_ALLOC;
            }
            cap[dev][i] = bytes;
        }
        if (need[i] && capturing) captured[dev][i] = true;
    }
    if (!parts_done[dev]) {
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed; // no work of a stream that is being captured either
        KQ_CUDA(cudaThreadExchangeStreamCaptureMode(&mode));
        const cudaError_t e = cudaGetSymbolAddress((void **)&parts_done[dev], g_parts_done);
        cudaThreadExchangeStreamCaptureMode(&mode);
        KQ_CUDA(e);
    }
    *out = {img16_bytes ? (uint8_t *)buf[dev][0] : nullptr, img8_bytes ? (uint8_t *)buf[dev][1] : nullptr, (float *)buf[dev][2], (float *)buf[dev][3], parts_done[dev], dev};
    return B200_OK;
}

// bytes of a token's images in the forms that the matrices read
int64_t token_bytes(const KqGemvSeg *segs, int nseg, int64_t nb, bool q6) {
    for (int i = 0; i < nseg; i++)
        if ((segs[i].type == B200_TYPE_Q6_K) == q6) return nb * (q6 ? TOK8 : TOK16);
    return 0;
}
b200_status scratch_for(int dev, const KqGemvSeg *segs, int nseg, int64_t m_pad, int64_t nb, cudaStream_t st, Scratch *out) {
    return scratch(dev, (size_t)(m_pad * token_bytes(segs, nseg, nb, false)), (size_t)(m_pad * token_bytes(segs, nseg, nb, true)), (size_t)(m_pad * nb * 4), st, out);
}

b200_status add_seg(Params &p, int i, const KqGemvSeg &g, int64_t experts, int64_t K) {
    CUtensorMap *w = p.w + 2 * i;
    const int64_t rows = g.n_rows * experts;
    const uint64_t row = (uint64_t)kq_device_row_bytes(g.type, K);
    p.w_row = (int64_t)row;
    if (g.type == B200_TYPE_Q4_K) {
        const uint64_t dims[2] = {row, (uint64_t)rows}, str[1] = {row};
        const uint32_t box[2] = {KQ_Q4K_BYTES, ROWS};
        KQ_TRY(kq_tmap_encode(w, 1, 2, g.W, dims, str, box, 0));
    } else {
        const int full = (int)(K / 256 / KQ_Q6_GROUP), tail = (int)(K / 256 % KQ_Q6_GROUP);
        const uint32_t box[4] = {32, ROWS, 13, 1}; // two blocks' 16-byte chunks: 8 of low nibbles, 4 of high bits, the scales
        if (full) {
            const uint64_t dims[4] = {KQ_Q6_GROUP * 16, (uint64_t)rows, 13, (uint64_t)full}, str[3] = {row, KQ_Q6_GROUP * 16, KQ_Q6_GROUP_BYTES};
            KQ_TRY(kq_tmap_encode(w, 1, 4, g.W, dims, str, box, 0));
        }
        if (tail) {
            const uint64_t dims[4] = {(uint64_t)tail * 16, (uint64_t)rows, 13, 1}, str[3] = {row, (uint64_t)tail * 16, row};
            KQ_TRY(kq_tmap_encode(w + 1, 1, 4, g.W + (int64_t)full * KQ_Q6_GROUP_BYTES, dims, str, box, 0));
        }
    }
    p.row_tiles += (int)kq_div_up(g.n_rows, ROWS);
    p.seg[i] = {g.y, g.bias, g.W, g.n_rows, p.row_tiles};
    for (int k = i + 1; k < MAX_SEGS; k++) p.seg[k].tile_end = 0x7fffffff;
    return B200_OK;
}

// Blocks of a CTA at least, in products with experts: shorter shares are shorter chains, but more parts to add up.
constexpr int MIN_SHARE = 2;

// Token tiles of a dense product and the least share of a CTA, by the time they should take, in hundredths of a microsecond.  A (tile, block) pair
// costs its decoding or its MMAs, whichever is longer, and the drains' turns (28672 x 8192, the pairs of a CTA one after another: Q4_K 0.9 us with 16 tokens,
// 1.1 with 64, 1.6 with 128, 2.5 with 256; Q6_K 1.5, 1.7, 2.3, 2.7).  A tile that was cut is added up by its last CTA: a trip to L2 for every
// eight parts and 16 tokens of a warp, and its parts come in at the rate of one SM.  Wide tiles decode a weight less often; narrow ones are more pairs, hence fewer parts and a shorter end where
// a product is too small to keep the GPU busy: 1024 x 5120 in Q4_K with 512 tokens 41 us as tiles of 256, 25 as tiles of 128; 5120 x 5120
// with 1024 tokens 81 and 86, with 64 tokens 24 as a tile of two chunks and 22 as one of one.
struct TokTiles {
    int n, tok;
    bool narrow;
    int min_share;
};
TokTiles token_tiles(bool q6, int64_t M, int64_t row_tiles, int64_t nb) {
    const int sms = kq_sm_count();
    TokTiles best = {0, 0, false, 0};
    int64_t best_cost = INT64_MAX;
    for (int chunks = MAX_CHUNKS; chunks >= 1; chunks /= 2) {
        const bool narrow = chunks == 1;
        int c, cw;
        chunks_of(narrow, (int)kq_div_up(M, kq_div_up(M, chunks * CHUNK)), c, cw);
        const int64_t tok = c * cw, tiles = kq_div_up(M, tok), pairs = tiles * row_tiles * nb;
        const int64_t per_pair = narrow ? (q6 ? 130 + tok / 4 : 80 + tok / 4) : c == 2 ? (q6 ? 175 : 110) + tok * 3 / 10 : (q6 ? 240 + tok / 7 : 178 + tok * 2 / 7);
        const int64_t groups = narrow ? cw / 16 : c * kq_div_up(std::min(cw, CHUNK / 2), 16); // of 16 tokens that a draining warp has
        int64_t before = 0;
        for (const int min_share : {2, 3, 4, 6, 8}) {
            const int64_t ctas = std::max<int64_t>(1, std::min<int64_t>(sms, pairs / min_share)), share = kq_div_up(pairs, ctas);
            if (ctas == before) continue; // enough pairs for all SMs: nothing to choose
            before = ctas;
            const int64_t parts = pairs % ctas == 0 && nb % share == 0 ? nb / share : kq_div_up(nb - 1, share) + 1;
            const int64_t cost = share * per_pair + (pairs % ctas == 0 && share % nb == 0 ? 0 : 150 + 50 * groups * kq_div_up(parts, 8) + parts * tok * (narrow ? 50 : 40) / CHUNK);
            if (cost < best_cost) best_cost = cost, best = {(int)tiles, (int)tok, narrow, min_share};
        }
    }
    return best;
}
// the same for a call's matrices of one type; none: no tiles
TokTiles token_tiles_of(uint32_t type, const KqGemvSeg *segs, int nseg, int64_t M, int64_t nb) {
    int64_t row_tiles = 0;
    for (int i = 0; i < nseg; i++)
        if (segs[i].type == type) row_tiles += kq_div_up(segs[i].n_rows, ROWS);
    return row_tiles ? token_tiles(type == B200_TYPE_Q6_K, M, row_tiles, nb) : TokTiles{0, 0, false, 0};
}

struct CallTiles {
    TokTiles q4, q6;
};
CallTiles call_tiles(const KqGemvSeg *segs, int nseg, int64_t M, int64_t nb) {
    return {token_tiles_of(B200_TYPE_Q4_K, segs, nseg, M, nb), token_tiles_of(B200_TYPE_Q6_K, segs, nseg, M, nb)};
}

template <bool Q6, bool NARROW>
b200_status launch(int dev, int grid, cudaStream_t st, const Params &p) {
    using C = Cfg<Q6, NARROW>;
    static std::atomic<uint32_t> ready; // devices on which this instance may have its shared memory; an instance that nobody uses is not loaded
    if (!(ready.load() >> dev & 1)) {
        cudaFuncAttributes a;
        KQ_CUDA(cudaFuncSetAttribute(gemm_kq_kernel<Q6, NARROW>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
        KQ_CUDA(cudaFuncGetAttributes(&a, gemm_kq_kernel<Q6, NARROW>));
        // setmaxnreg moves registers of the launch between the warpgroups: more than it was launched with would wait for ever
        KQ_REQUIRE(4 * a.numRegs >= C::REG_SUM, "gemm: built with %d registers", a.numRegs);
        ready |= 1u << dev;
    }
    KQ_CUDA(kq_launch(gemm_kq_kernel<Q6, NARROW>, dim3(grid), dim3(NTHREADS), C::SMEM, st, p));
    return B200_OK;
}

// one launch per weight type for the matrices that read the images in sc; dense products cut the tokens by type
b200_status launch_segs(Params p, bool narrow, const CallTiles *tiles, const Scratch &sc, const KqGemvSeg *segs, int nseg, int64_t experts, int64_t K, cudaStream_t st) {
    for (const uint32_t type : {(uint32_t)B200_TYPE_Q4_K, (uint32_t)B200_TYPE_Q6_K}) {
        int n = 0;
        p.row_tiles = 0;
        if (!p.row_src) {
            const TokTiles &t = type == B200_TYPE_Q4_K ? tiles->q4 : tiles->q6;
            p.tok_tiles = t.n, p.tile_tok = t.tok, p.min_share = t.min_share, narrow = t.narrow;
        }
        p.img = type == B200_TYPE_Q4_K ? sc.img16 : sc.img8, p.da = sc.da, p.part = sc.part;
        for (int i = 0; i < nseg; i++)
            if (segs[i].type == type) KQ_TRY(add_seg(p, n++, segs[i], experts, K));
        if (!n) continue;
        const int64_t units = (int64_t)p.tok_tiles * p.row_tiles * p.nb;
        KQ_REQUIRE(units < (int64_t)1 << 31, "gemm: bad shape");
        // with experts the number of tiles is known on the device only
        const int grid = p.row_src ? kq_sm_count() : (int)std::min<int64_t>(kq_sm_count(), std::max<int64_t>(1, units / p.min_share));
        const bool q6 = type == B200_TYPE_Q6_K;
        if (narrow) KQ_TRY((q6 ? launch<true, true>(sc.dev, grid, st, p) : launch<false, true>(sc.dev, grid, st, p)));
        else KQ_TRY((q6 ? launch<true, false>(sc.dev, grid, st, p) : launch<false, false>(sc.dev, grid, st, p)));
        KQ_COUNT_LAUNCH();
        KQ_LAUNCH_CHECK();
    }
    return B200_OK;
}

b200_status check_segs(const KqGemvSeg *segs, int nseg, const int8_t *q, int64_t K, int *dev) {
    KQ_REQUIRE(nseg >= 1 && nseg <= MAX_SEGS && K > 0 && K % 256 == 0 && ((uintptr_t)q & 15) == 0, "gemm: bad shape");
    for (int i = 0; i < nseg; i++) {
        KQ_REQUIRE(segs[i].type == B200_TYPE_Q4_K || segs[i].type == B200_TYPE_Q6_K, "gemm: weight type %u", segs[i].type);
        KQ_REQUIRE(segs[i].n_rows > 0, "gemm: bad shape");
        KQ_REQUIRE(((uintptr_t)segs[i].W & 15) == 0, "gemm: operands must be 16-byte aligned");
    }
    KQ_CUDA(cudaGetDevice(dev));
    KQ_REQUIRE(*dev >= 0 && *dev < MAX_DEVICES, "gemm: device %d out of range", *dev);
    return B200_OK;
}

} // namespace

int kq_gemm_error_fetch() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, g_gemm_error, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(g_gemm_error, &zero, sizeof(int));
    return v;
}

// Tokens whose images are held at a time: every row tile reads the images again, so they should stay in L2 (126 MB) beside the weights that
// stream by.  2048 and 4096 tokens x 8192 x 28672 in Q4_K, 125 and 250 MB at once: 1363 and 2788 us; in slabs of 62 MB 1200 and 2406.
constexpr int64_t SLAB_MIN = MAX_CHUNKS * CHUNK;
static int64_t slab_tokens(int64_t per_token) { return std::max(SLAB_MIN, SLAB_BYTES / per_token / SLAB_MIN * SLAB_MIN); }
// the tokens that the images of a call hold, in whole tiles of either type
static int32_t padded_tokens(const CallTiles &t) { return std::max(t.q4.n * t.q4.tok, t.q6.n * t.q6.tok); }

b200_status kq_gemm_image(const KqGemvSeg *segs, int nseg, int64_t M, int64_t K, cudaStream_t st, KqTokenImage *im) {
    *im = KqTokenImage{};
    int dev = 0;
    KQ_TRY(check_segs(segs, nseg, nullptr, K, &dev));
    const int64_t nb = K / 256;
    if (M > slab_tokens(token_bytes(segs, nseg, nb, false) + token_bytes(segs, nseg, nb, true))) return B200_OK; // in slabs
    const int32_t pad = padded_tokens(call_tiles(segs, nseg, M, nb));
    Scratch sc;
    const b200_status rc = scratch_for(dev, segs, nseg, pad, nb, st, &sc);
    if (rc != B200_OK) return rc == B200_ERR_ALLOC ? B200_OK : rc;
    *im = {sc.img16, sc.img8, sc.da, sc.parts_done, 2 * MAX_CTAS * DRAIN_WARPS / 4, pad, (int32_t)M};
    return B200_OK;
}

b200_status kq_launch_gemm_image(const KqGemvSeg *segs, int nseg, const KqTokenImage &im, int64_t K, const float *residual, cudaStream_t st) {
    int dev = 0;
    KQ_TRY(check_segs(segs, nseg, nullptr, K, &dev));
    KQ_REQUIRE(im.n_tok > 0 && (im.img16 || im.img8) && (!residual || nseg == 1), "gemm: bad shape");
    Params p = {};
    p.M = im.n_tok, p.nb = (int32_t)(K / 256), p.m_pad = im.m_pad, p.residual = residual;
    Scratch sc;
    KQ_TRY(scratch_for(dev, segs, nseg, im.m_pad, p.nb, st, &sc)); // the buffers that kq_gemm_image gave
    KQ_REQUIRE(sc.img16 == im.img16 && sc.img8 == im.img8 && sc.da == im.da, "gemm: another call came between a token image and its product");
    const CallTiles tiles = call_tiles(segs, nseg, p.M, p.nb);
    return launch_segs(p, false, &tiles, sc, segs, nseg, 1, K, st);
}

b200_status kq_launch_gemm_tc(const KqGemvSeg *segs, int nseg, const int8_t *q, const float *d, const int16_t *bs, int64_t M, int64_t K,
                              const float *residual, cudaStream_t st) {
    int dev = 0;
    KQ_TRY(check_segs(segs, nseg, q, K, &dev));
    KQ_REQUIRE(M > 0 && (!residual || nseg == 1), "gemm: bad shape");
    const int64_t nb = K / 256;
    const int64_t per_token = token_bytes(segs, nseg, nb, false) + token_bytes(segs, nseg, nb, true);
    int64_t slab = slab_tokens(per_token);
    for (int64_t m0 = 0, mc; m0 < M; m0 += mc) {
        mc = kq_div_up(M - m0, kq_div_up(M - m0, slab)); // of equal size
        if (mc < M - m0) mc = kq_div_up(mc, SLAB_MIN) * SLAB_MIN;
        Params p = {};
        p.M = (int32_t)mc, p.nb = (int32_t)nb;
        const CallTiles tiles = call_tiles(segs, nseg, mc, nb);
        p.m_pad = padded_tokens(tiles);
        Scratch sc;
        const b200_status rc = scratch_for(dev, segs, nseg, p.m_pad, nb, st, &sc);
        if (rc == B200_ERR_ALLOC && mc > SLAB_MIN) { // no room for these images: fewer at a time
            slab = kq_div_up(mc, 2 * SLAB_MIN) * SLAB_MIN;
            mc = 0;
            continue;
        }
        KQ_TRY(rc);
        const ImageParams ip = {q + m0 * K, d + m0 * nb, bs + m0 * nb * 16, sc.img16, sc.img8, sc.da, (int32_t)mc, (int32_t)nb, p.m_pad, 1, nullptr, nullptr, nullptr, 0, 0, 0};
        KQ_CUDA(kq_launch(act_image_kernel, dim3((unsigned)(p.m_pad / 16), (unsigned)nb), dim3(288), 0, st, ip));
        KQ_COUNT_LAUNCH();
        KqGemvSeg sg[MAX_SEGS];
        for (int i = 0; i < nseg; i++) {
            sg[i] = segs[i];
            sg[i].y += m0 * sg[i].n_rows;
        }
        p.residual = residual ? residual + m0 * segs[0].n_rows : nullptr;
        KQ_TRY(launch_segs(p, false, &tiles, sc, sg, nseg, 1, K, st));
    }
    return B200_OK;
}

// ---- MUL_MAT_ID over many tokens: pairs gathered per expert, one grouped launch of the tensor-core kernel ----
// Scratch of the sort, in int32 words: [0] number of live tiles, [1 .. 1 + max_tiles) expert per tile,
// [1 + max_tiles ..) pair per tile row, then pairs per tile; with t = moe_tile(n_pairs, n_expert) pairs a tile, max_tiles = ceil(n_pairs / t) + n_expert bounds sum_e ceil(c_e / t).
// So the places in it depend on both numbers: sort and products are given the same.
// Pairs of a tile: with few pairs an expert narrow tiles, whose blocks two warpgroups decode; from about as many as fill one, wide ones, where most experts are one
// tile.  Narrow / wide, us, with 8, 48, 64 and 96 pairs an expert: 128 experts 768 x 2048 in Q4_K 63 / 87, 113 / 133, 151 / 148, 208 / 183; 2048 x 768 in Q6_K 87 / 103, 143 / 161, 202 / 170, 272 / 197;
// 8 experts 14336 x 4096 in Q4_K 94 / 135, 128 / 165, 179 / 170, 231 / 178; 256 experts 2048 x 2048 in Q6_K 301 / 429, 463 / 576, 659 / 617, 874 / 689; fourteen such tables alike.  Narrow tiles
// need no more room for the sort than wide ones: at most 48 E / 64 + E tiles of 64 rows against E of 128.
static inline int moe_tile(int64_t n_pairs, int64_t E) { return n_pairs <= 48 * E ? CHUNK : 2 * CHUNK; }
static inline int64_t moe_max_tiles(int64_t n_pairs, int64_t E) { return kq_div_up(n_pairs, moe_tile(n_pairs, E)) + E; }

size_t kq_moe_sort_scratch_bytes(int64_t n_pairs, int64_t E) {
    const int64_t mt = moe_max_tiles(n_pairs, E);
    return (size_t)(1 + mt + mt * moe_tile(n_pairs, E) + mt + 64) * sizeof(int32_t);
}

b200_status kq_moe_sort(const int32_t *ids, int64_t n_pairs, int64_t E, int32_t *scratch, size_t scratch_bytes, cudaStream_t st) {
    KQ_REQUIRE(ids && scratch && n_pairs >= 1 && E >= 1 && E <= SORT_MAX_E, "moe_sort: n_pairs >= 1, 1 <= experts <= %d", SORT_MAX_E);
    KQ_REQUIRE(scratch_bytes >= kq_moe_sort_scratch_bytes(n_pairs, E), "moe_sort: scratch of %zu bytes, %zu needed", scratch_bytes,
               kq_moe_sort_scratch_bytes(n_pairs, E));
    const int64_t mt = moe_max_tiles(n_pairs, E);
    const int TM = moe_tile(n_pairs, E);
    kq_launch(moe_sort_kernel, 1, SORT_WARPS * 32, 0, st, ids, (int)n_pairs, (int)E, TM, scratch, scratch + 1, scratch + 1 + mt,
              scratch + 1 + mt + mt * TM);
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}

// y[pair][N] = W[expert of the pair] . x[pair / act_div] for up to three expert-packed matrices: q / d / bs are the quantised
// activations of the n_pairs / act_div source rows, sorted = the scratch kq_moe_sort left for these pairs.
b200_status kq_launch_gemm_grouped(const KqGemvSeg *segs, int nseg, const KqGroupedRows &rows, int act_div,
                                   int64_t n_pairs, int64_t E, int64_t K, const int32_t *sorted, cudaStream_t st) {
    int dev = 0;
    KQ_TRY(check_segs(segs, nseg, rows.q, K, &dev));
    KQ_REQUIRE(n_pairs > 0 && act_div >= 1 && (!rows.g || act_div == 1), "grouped gemm: bad shape");
    for (int i = 0; i < nseg; i++)
        KQ_REQUIRE(segs[i].expert_stride == kq_device_row_bytes(segs[i].type, K) * segs[i].n_rows && segs[i].expert_stride % 16 == 0,
                   "grouped gemm: expert matrices must be contiguous and 16-byte aligned");
    const int64_t nb = K / 256, mt = moe_max_tiles(n_pairs, E);
    const int TM = moe_tile(n_pairs, E);
    const bool narrow = TM == CHUNK;
    const int64_t per_token = token_bytes(segs, nseg, nb, false) + token_bytes(segs, nseg, nb, true);
    int64_t slab = std::max<int64_t>(1, GROUP_BYTES / (per_token * TM));
    for (int64_t t0 = 0, tc; t0 < mt; t0 += tc) {
        tc = kq_div_up(mt - t0, kq_div_up(mt - t0, slab));
        Params p = {};
        p.M = p.m_pad = (int32_t)(tc * TM), p.nb = (int32_t)nb, p.tok_tiles = (int)tc, p.first_tile = (int)t0, p.tile_tok = TM, p.min_share = MIN_SHARE;
        Scratch sc;
        const b200_status rc = scratch_for(dev, segs, nseg, p.m_pad, nb, st, &sc);
        if (rc == B200_ERR_ALLOC && tc > 1) {
            slab = kq_div_up(tc, 2);
            tc = 0;
            continue;
        }
        KQ_TRY(rc);
        p.n_tiles = sorted, p.tile_expert = sorted + 1 + t0, p.row_src = sorted + 1 + mt + t0 * TM, p.tile_count = sorted + 1 + mt + mt * TM + t0;
        if (rows.g) {
            const KqTokenImage im = {sc.img16, sc.img8, sc.da, sc.parts_done, 2 * MAX_CTAS * DRAIN_WARPS / 4, p.m_pad, 0};
            KQ_TRY(kq_act_image_tiles(rows.g, rows.u, K, im, {p.row_src, p.tile_count, p.n_tiles, p.first_tile, TM, narrow}, st));
        } else {
            const ImageParams ip = {rows.q, rows.d, rows.bs, sc.img16, sc.img8, sc.da, 0, (int32_t)nb, p.m_pad, act_div, p.row_src, p.tile_count, p.n_tiles, p.first_tile, TM, narrow};
            KQ_CUDA(kq_launch(act_image_kernel, dim3((unsigned)(p.m_pad / 16), (unsigned)nb), dim3(288), 0, st, ip));
            KQ_COUNT_LAUNCH();
        }
        KQ_TRY(launch_segs(p, narrow, nullptr, sc, segs, nseg, E, K, st));
    }
    return B200_OK;
}
