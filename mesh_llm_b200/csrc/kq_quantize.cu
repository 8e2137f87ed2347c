// Activation quantiser (f32 -> Q8 blocks of 256), its fused forms (RMSNorm -> Q8), the Q6_K
// device repack, and the on-device generator of synthetic Q4_K_M weights.
#include "kq_common.cuh"

#include <cuda_bf16.h>

namespace {

__global__ void __launch_bounds__(128) quantize_act_kernel(const float *x, int64_t nblocks,
                                                           int8_t *q, float *d, int16_t *bs) {
    KQ_PDL_ENTER();
    const int lane = threadIdx.x & 31;
    const int64_t blk = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (blk >= nblocks) return;
    const float4 *xp = reinterpret_cast<const float4 *>(x + blk * 256 + lane * 8);
    const float4 a = xp[0], b = xp[1];
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    kq_quantize_block_warp(v, lane, q + blk * 256, d + blk, bs + blk * 16);
}

// SwiGLU and the Q8 quantiser of its result in one pass (the input of the down projection in a prefill): one warp
// per 256-element block, lane l on elements 8l .. 8l+7; y (f32, may alias g) is written when it is not null.
// Same expression and same quantiser as the separate kernels, so codes and values are theirs.
__global__ void __launch_bounds__(128) swiglu_quantize_kernel(const float *g, const float *u, int64_t nblocks, float *y, int8_t *q,
                                                              float *d, int16_t *bs) {
    KQ_PDL_ENTER();
    const int lane = threadIdx.x & 31;
    const int64_t blk = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (blk >= nblocks) return;
    const int64_t o = blk * 256 + lane * 8;
    const float4 g0 = *reinterpret_cast<const float4 *>(g + o), g1 = *reinterpret_cast<const float4 *>(g + o + 4);
    const float4 u0 = *reinterpret_cast<const float4 *>(u + o), u1 = *reinterpret_cast<const float4 *>(u + o + 4);
    const float a[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w}, b[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = (a[i] / (1.0f + expf(-a[i]))) * b[i];
    if (y) {
        *reinterpret_cast<float4 *>(y + o) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4 *>(y + o + 4) = make_float4(v[4], v[5], v[6], v[7]);
    }
    kq_quantize_block_warp(v, lane, q + blk * 256, d + blk, bs + blk * 16);
}

// The same for the tensor-core product: eight tokens of a block per CTA, a warp each, gathered in shared memory so that the image is written in full lines.
// With UP silu(x) * up.  A pass over the codes and a launch less than codes first, image then.
// TILES: the rows of a product with experts, gathered; chunks of a tile are one (narrow) or two.
template <bool UP, bool TILES>
__global__ void __launch_bounds__(256) act_to_image_kernel(const float *x, const float *up, float *y, int64_t K, const __grid_constant__ KqTokenImage im,
                                                           const __grid_constant__ KqTileRows rows) {
    KQ_PDL_ENTER();
    constexpr int PITCH = 144; // chunks of 128 bytes, 16 further apart: a warp's stores fall on different banks
    __shared__ __align__(16) uint8_t s16[34 * PITCH], s8[16 * PITCH];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, b = blockIdx.y, t0 = blockIdx.x * 8, t = t0 + warp;
    if (blockIdx.x == 0 && b == 0)
        for (int i = tid; i < im.n_parts; i += 256) im.parts[i] = make_int4(0, 0, 0, 0);
    int live = im.n_tok;
    int64_t row = t;
    if (TILES) {
        const int tile = t0 / rows.tile_tok, first = tile * rows.tile_tok;
        row = rows.row_src[t]; // asked for before it is known whether there is one: the table has all of them
        if (tile >= *rows.n_tiles - rows.first_tile) return;
        const int n = rows.tile_count[tile], padded = rows.narrow ? (n + 15) & ~15 : 2 * (((n + 1) / 2 + 15) & ~15);
        if (t0 - first >= padded) return;
        live = first + n;
    }
    float v[8] = {};
    if (t < live) {
        const int64_t at = row * K + b * 256 + lane * 8;
        const float4 x0 = *reinterpret_cast<const float4 *>(x + at), x1 = *reinterpret_cast<const float4 *>(x + at + 4);
        v[0] = x0.x, v[1] = x0.y, v[2] = x0.z, v[3] = x0.w, v[4] = x1.x, v[5] = x1.y, v[6] = x1.z, v[7] = x1.w;
        if (UP) {
            const float4 u0 = *reinterpret_cast<const float4 *>(up + at), u1 = *reinterpret_cast<const float4 *>(up + at + 4);
            const float u[8] = {u0.x, u0.y, u0.z, u0.w, u1.x, u1.y, u1.z, u1.w};
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = (v[i] / (1.0f + expf(-v[i]))) * u[i];
            if (y) {
                *reinterpret_cast<float4 *>(y + at) = make_float4(v[0], v[1], v[2], v[3]);
                *reinterpret_cast<float4 *>(y + at + 4) = make_float4(v[4], v[5], v[6], v[7]);
            }
        }
    }
    const KqQ8Codes o = kq_quantize_codes_warp(v); // of zeros: zeros
    kq_image_put(im.img16 ? s16 + warp * 16 : nullptr, im.img8 ? s8 + warp * 16 : nullptr, PITCH, lane, o);
    if (lane == 0) im.da[(int64_t)b * im.m_pad + t] = o.d;
    __syncthreads();
    const int64_t group = (int64_t)b * im.m_pad + t0;
    if (im.img16)
        for (int i = tid; i < 34 * 8; i += 256)
            *reinterpret_cast<uint4 *>(im.img16 + group * KQ_TOK16 + i * 16) = *reinterpret_cast<const uint4 *>(s16 + (i >> 3) * PITCH + (i & 7) * 16);
    if (im.img8)
        for (int i = tid; i < 16 * 8; i += 256)
            *reinterpret_cast<uint4 *>(im.img8 + group * KQ_TOK8 + i * 16) = *reinterpret_cast<const uint4 *>(s8 + (i >> 3) * PITCH + (i & 7) * 16);
}

// RMSNorm and Q8 of a row, W warps: a warp holds up to R of the row's blocks in registers, so that the row is read once.  PRE, for few rows: the weights as well, asked for before the
// kernel waits for the one that writes the row; many rows would rather have the registers (512 rows of 5120 8.9 us with, 7.0 without).  Outputs: f32 (y), Q8 (q, d, bs), an image; rows past im.n_tok are zeros of the image.  The sum of squares is
// carried in double so that the scale does not depend on the order of the reduction: the normalised values, and with them the Q8 codes, are then
// reproducible.
template <int W, int R, bool PRE>
__global__ void __launch_bounds__(W * 32) rms_norm_q8_kernel(const float *x, const float *w, int h, float eps, float *y, int8_t *q, float *d, int16_t *bs,
                                                             int64_t x_row_stride, const __grid_constant__ KqTokenImage im) {
    __shared__ double part[W];
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nb = h / 256;
    const bool image = im.img16 || im.img8, live = !image || row < im.n_tok;
    const float *xr = x + (int64_t)row * x_row_stride;
    KQ_PDL_TRIGGER();
    float g[PRE ? R : 1][8], v[R][8];
    auto load = [&](const float *p, int b, float (&o)[8]) {
        const float4 a = *reinterpret_cast<const float4 *>(p + b * 256 + lane * 8), c = *reinterpret_cast<const float4 *>(p + b * 256 + lane * 8 + 4);
        o[0] = a.x, o[1] = a.y, o[2] = a.z, o[3] = a.w, o[4] = c.x, o[5] = c.y, o[6] = c.z, o[7] = c.w;
    };
    auto weights = [&](int b, float (&o)[8]) {
#pragma unroll
        for (int i = 0; i < 8; i++) o[i] = 1.0f;
        if (w && b < nb) load(w, b, o);
    };
    if constexpr (PRE) {
#pragma unroll
        for (int r = 0; r < R; r++) weights(warp + r * W, g[r]);
    }
    KQ_PDL_WAIT();
    if (image && row == 0)
        for (int i = tid; i < im.n_parts; i += W * 32) im.parts[i] = make_int4(0, 0, 0, 0);
    double ss = 0.0;
#pragma unroll
    for (int r = 0; r < R; r++) {
#pragma unroll
        for (int i = 0; i < 8; i++) v[r][i] = 0.f;
        if (live && warp + r * W < nb) load(xr, warp + r * W, v[r]);
    }
    auto add = [&](const float (&u)[8]) {
#pragma unroll
        for (int i = 0; i < 8; i++) ss += (double)u[i] * u[i];
    };
#pragma unroll
    for (int r = 0; r < R; r++) add(v[r]);
    if (live)
        for (int b = warp + R * W; b < nb; b += W) {
            float u[8];
            load(xr, b, u);
            add(u);
        }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) part[warp] = ss;
    __syncthreads();
    double t = 0.0;
#pragma unroll
    for (int i = 0; i < W; i++) t += part[i];
    const float scale = 1.0f / sqrtf((float)(t / (double)h) + eps);
    auto emit = [&](int b, const float (&u)[8], const float (&f)[8]) {
        float n[8];
#pragma unroll
        for (int i = 0; i < 8; i++) n[i] = live ? u[i] * scale * f[i] : 0.f;
        if (y && live) {
            float *yo = y + (int64_t)row * h + b * 256 + lane * 8;
            *reinterpret_cast<float4 *>(yo) = make_float4(n[0], n[1], n[2], n[3]);
            *reinterpret_cast<float4 *>(yo + 4) = make_float4(n[4], n[5], n[6], n[7]);
        }
        const KqQ8Codes o = kq_quantize_codes_warp(n);
        const int64_t gb = (int64_t)row * nb + b;
        if (q && live) {
            *reinterpret_cast<uint2 *>(q + gb * 256 + lane * 8) = o.pk;
            if ((lane & 1) == 0) bs[gb * 16 + (lane >> 1)] = (int16_t)o.sum;
            if (lane == 0) d[gb] = o.d;
        }
        if (image) {
            const int64_t group = (int64_t)b * im.m_pad + (row & ~7);
            kq_image_put(im.img16 ? im.img16 + group * KQ_TOK16 + (row & 7) * 16 : nullptr, im.img8 ? im.img8 + group * KQ_TOK8 + (row & 7) * 16 : nullptr, 128, lane, o);
            if (lane == 0) im.da[(int64_t)b * im.m_pad + row] = o.d;
        }
    };
#pragma unroll
    for (int r = 0; r < R; r++)
        if (warp + r * W < nb) {
            if constexpr (!PRE) weights(warp + r * W, g[0]);
            emit(warp + r * W, v[r], g[PRE ? r : 0]);
        }
    for (int b = warp + R * W; b < nb; b += W) {
        float u[8] = {}, f[8];
        if (live) load(xr, b, u);
        weights(b, f);
        emit(b, u, f);
    }
}

// RMSNorm (x * rsqrt(mean(x^2) + eps) * w) of rows of any length, f32 output.  One CTA of 256 threads per row.
__global__ void __launch_bounds__(256) rms_norm_kernel(const float *x, const float *w, int h, float eps, float *y, int64_t x_row_stride) {
    KQ_PDL_ENTER();
    __shared__ double part[8];
    __shared__ float s_scale;
    const int row = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *xr = x + (int64_t)row * x_row_stride;
    // the sum of squares is carried in double so that the scale does not depend on the order of
    // the reduction: the normalised values, and with them the Q8 codes, are then reproducible
    double ss = 0.0;
    for (int i = tid * 4; i < h; i += 1024) {
        const float4 v = *reinterpret_cast<const float4 *>(xr + i);
        ss += (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) part[warp] = ss;
    __syncthreads();
    if (tid == 0) {
        double t = 0.0;
        for (int i = 0; i < 8; i++) t += part[i];
        s_scale = 1.0f / sqrtf((float)(t / (double)h) + eps);
    }
    __syncthreads();
    const float scale = s_scale;
    for (int i = tid; i < h; i += 256) y[(int64_t)row * h + i] = xr[i] * scale * (w ? w[i] : 1.0f);
}

// Rows of up to 128 values (one head), f32 output only: a warp per row, with the sums in the order of the kernel above, which gives such a row
// 256 threads and two barriers.  32768 rows of 128: 52 -> 9 us.  Rows from `rows` on, rows2 of them, are those of a second pair of arrays (the heads of
// q and of k in one launch: one token through four layers of experts 183 -> 179 us).
struct HeadRows {
    const float *x, *w;
    float *y;
    int64_t ldx;
};
__global__ void __launch_bounds__(256) rms_norm_head_kernel(HeadRows a, int64_t rows, HeadRows b, int64_t rows2, int h, float eps) {
    KQ_PDL_ENTER();
    const int lane = threadIdx.x & 31;
    int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= rows + rows2) return;
    const bool second = row >= rows;
    if (second) row -= rows;
    const float *x = second ? b.x : a.x, *w = second ? b.w : a.w;
    float *y = second ? b.y : a.y;
    const int64_t x_row_stride = second ? b.ldx : a.ldx;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (lane * 4 < h) v = *reinterpret_cast<const float4 *>(x + row * x_row_stride + lane * 4);
    double ss = (double)v.x * v.x + (double)v.y * v.y + (double)v.z * v.z + (double)v.w * v.w;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float scale = 1.0f / sqrtf((float)(ss / (double)h) + eps);
    if (lane * 4 < h) {
        float f[4] = {1.f, 1.f, 1.f, 1.f};
        if (w) {
#pragma unroll
            for (int i = 0; i < 4; i++) f[i] = w[lane * 4 + i];
        }
        *reinterpret_cast<float4 *>(y + row * h + lane * 4) = make_float4(v.x * scale * f[0], v.y * scale * f[1], v.z * scale * f[2], v.w * scale * f[3]);
    }
}

// ---- Q6_K repack: GGUF block-interleaved rows <-> device rows [ql | qh | scales | d | pad] ------
__global__ void repack_q6k_kernel(const uint16_t *src, uint16_t *dst,
                                  int64_t n_rows, int nb, int64_t dst_row_u16, int inverse) {
    KQ_PDL_ENTER();
    const int64_t per_row = (int64_t)nb * 105;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_rows * per_row) return;
    const int64_t row = i / per_row;
    const int r = (int)(i % per_row), b = r / 105, o = r % 105; // u16 index inside the block
    const KqQ6Addr qa = kq_q6_addr(nb, b);
    int64_t dev; // u16 offset inside the device row
    if (o < 64) dev = (qa.ql + ((2 * o) >> 4) * qa.cs + ((2 * o) & 15)) / 2;
    else if (o < 96) dev = (qa.qh + ((2 * (o - 64)) >> 4) * qa.cs + ((2 * (o - 64)) & 15)) / 2;
    else if (o < 104) dev = qa.sc / 2 + (o - 96);
    else dev = qa.d / 2;
    const int64_t g = row * per_row + r, dv = row * dst_row_u16 + dev;
    if (inverse) dst[g] = src[dv];
    else dst[dv] = src[g];
}

// ---- synthetic weights ------------------------------------------------------------------------
__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ float gauss_at(uint64_t key, uint64_t i) {
    const uint64_t r = mix64(key + i * 0xD1342543DE82EF95ull);
    const float u1 = ((float)((uint32_t)(r >> 32) >> 8) + 1.0f) * (1.0f / 16777216.0f);
    const float u2 = (float)((uint32_t)r >> 8) * (1.0f / 16777216.0f);
    return sqrtf(-2.0f * __logf(u1)) * __cosf(6.28318530717958647692f * u2);
}

// One warp per 256-element block; writes the block in device layout.
__global__ void __launch_bounds__(128) synth_kquant_kernel(uint32_t type, uint8_t *W, int64_t n_rows,
                                                           int nb, uint64_t key, float sigma) {
    KQ_PDL_ENTER();
    __shared__ uint8_t codes[4][256];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t gb = (int64_t)blockIdx.x * 4 + warp;
    if (gb >= n_rows * nb) return;
    const int64_t row = gb / nb;
    const int b = (int)(gb % nb);
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = sigma * gauss_at(key, (uint64_t)(gb * 256 + lane * 8 + i));
    uint8_t *rp = W + row * kq_device_row_bytes(type, (int64_t)nb * 256);
    uint8_t *cd = codes[warp];
    if (type == B200_TYPE_Q4_K) {
        float lo = 0.f, hi = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) { lo = fminf(lo, v[i]); hi = fmaxf(hi, v[i]); }
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, 1));
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, 2));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, 1));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, 2));
        const float scale = (hi - lo) / 15.0f, mn = -lo;
        const __half dh = __float2half_rn(kq_warp_max(scale) / 63.0f);
        const __half mh = __float2half_rn(kq_warp_max(mn) / 63.0f);
        const float d = __half2float(dh), dmin = __half2float(mh);
        const int sc = d > 0.f ? max(0, min(63, __float2int_rn(scale / d))) : 0;
        const int mc = dmin > 0.f ? max(0, min(63, __float2int_rn(mn / dmin))) : 0;
        const float dl = d * (float)sc, ml = dmin * (float)mc;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int qv = dl > 0.f ? __float2int_rn((v[i] + ml) / dl) : 0;
            cd[lane * 8 + i] = (uint8_t)max(0, min(15, qv));
        }
        __syncwarp();
        uint8_t *blk = rp + (int64_t)b * KQ_Q4K_BYTES;
        // 128 quant bytes: lane writes bytes 4l .. 4l+3
        uint32_t pk = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int byte = lane * 4 + i, g = byte >> 5, k = byte & 31;
            pk |= (uint32_t)(cd[64 * g + k] | (cd[64 * g + 32 + k] << 4)) << (8 * i);
        }
        *reinterpret_cast<uint32_t *>(blk + 16 + lane * 4) = pk;
        // header: gather the 8 scale / min codes (sub-block j lives in lanes 4j..4j+3)
        int scj[8], mcj[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            scj[j] = __shfl_sync(0xffffffffu, sc, 4 * j);
            mcj[j] = __shfl_sync(0xffffffffu, mc, 4 * j);
        }
        if (lane == 0) {
            uint8_t s[12];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                s[j] = (uint8_t)(scj[j] | ((scj[j + 4] >> 4) << 6));
                s[j + 4] = (uint8_t)(mcj[j] | ((mcj[j + 4] >> 4) << 6));
                s[j + 8] = (uint8_t)((scj[j + 4] & 0xF) | ((mcj[j + 4] & 0xF) << 4));
            }
            uint4 hdr;
            hdr.x = (uint32_t)__half_as_ushort(dh) | ((uint32_t)__half_as_ushort(mh) << 16);
            hdr.y = s[0] | (s[1] << 8) | (s[2] << 16) | ((uint32_t)s[3] << 24);
            hdr.z = s[4] | (s[5] << 8) | (s[6] << 16) | ((uint32_t)s[7] << 24);
            hdr.w = s[8] | (s[9] << 8) | (s[10] << 16) | ((uint32_t)s[11] << 24);
            *reinterpret_cast<uint4 *>(blk) = hdr;
        }
    } else { // Q6_K, symmetric per 16 elements (2 lanes)
        float am = 0.f;
#pragma unroll
        for (int i = 0; i < 8; i++) am = fmaxf(am, fabsf(v[i]));
        am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, 1));
        const float scale = am / 31.0f;
        const __half dh = __float2half_rn(kq_warp_max(scale) / 127.0f);
        const float d = __half2float(dh);
        const int sc = d > 0.f ? max(0, min(127, __float2int_rn(scale / d))) : 0;
        const float dl = d * (float)sc;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int qv = dl > 0.f ? __float2int_rn(v[i] / dl) : 0;
            cd[lane * 8 + i] = (uint8_t)(max(-32, min(31, qv)) + 32);
        }
        __syncwarp();
        // ql: 128 bytes, lane writes bytes 4l..4l+3; byte 64h+k = elem 128h+k | elem 128h+64+k << 4
        uint32_t pk = 0;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int byte = lane * 4 + i, h = byte >> 6, k = byte & 63;
            pk |= (uint32_t)((cd[128 * h + k] & 0xF) | ((cd[128 * h + 64 + k] & 0xF) << 4)) << (8 * i);
        }
        const KqQ6Addr qa = kq_q6_addr(nb, b);
        *reinterpret_cast<uint32_t *>(rp + qa.ql + ((lane * 4) >> 4) * qa.cs + ((lane * 4) & 15)) = pk;
        // qh: 64 bytes, lane writes bytes 2l, 2l+1; byte 32h+k = hi2 of elems 128h+k+{0,32,64,96}
        uint16_t ph = 0;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int byte = lane * 2 + i, h = byte >> 5, k = byte & 31;
            const uint32_t v8 = (cd[128 * h + k] >> 4) | ((cd[128 * h + 32 + k] >> 4) << 2) |
                                ((cd[128 * h + 64 + k] >> 4) << 4) | ((cd[128 * h + 96 + k] >> 4) << 6);
            ph |= (uint16_t)(v8 << (8 * i));
        }
        *reinterpret_cast<uint16_t *>(rp + qa.qh + ((lane * 2) >> 4) * qa.cs + ((lane * 2) & 15)) = ph;
        if ((lane & 1) == 0) rp[qa.sc + (lane >> 1)] = (uint8_t)(int8_t)sc;
        if (lane == 0) *reinterpret_cast<uint16_t *>(rp + qa.d) = __half_as_ushort(dh);
    }
}

__global__ void synth_f32_kernel(float *w, int64_t n, uint64_t key, float mean, float sigma) {
    KQ_PDL_ENTER();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) w[i] = mean + sigma * gauss_at(key, (uint64_t)i);
}

// bf16 rows of K values padded with zeros to ld
__global__ void synth_bf16_kernel(uint16_t *w, int64_t n_rows, int64_t K, int64_t ld, uint64_t key, float mean, float sigma) {
    KQ_PDL_ENTER();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_rows * ld) return;
    const int64_t r = i / ld, k = i % ld;
    w[i] = k < K ? __bfloat16_as_ushort(__float2bfloat16_rn(mean + sigma * gauss_at(key, (uint64_t)(r * K + k)))) : 0;
}

} // namespace

b200_status kq_synth_weights(uint32_t type, void *W, int64_t n_rows, int64_t K, uint64_t key,
                             float mean, float sigma, cudaStream_t st) {
    if (type == B200_TYPE_F32) {
        const int64_t n = n_rows * K;
        kq_launch(synth_f32_kernel, (unsigned)kq_div_up(n, 256), 256, 0, st, (float *)W, n, key, mean, sigma);
    } else if (type == B200_TYPE_BF16) {
        const int64_t ld = kq_device_row_bytes(type, K) / 2, n = n_rows * ld;
        kq_launch(synth_bf16_kernel, (unsigned)kq_div_up(n, 256), 256, 0, st, (uint16_t *)W, n_rows, K, ld, key, mean, sigma);
    } else {
        KQ_REQUIRE(type == B200_TYPE_Q4_K || type == B200_TYPE_Q6_K, "synth: type %u", type);
        KQ_REQUIRE(K % 256 == 0, "synth: K %% 256");
        const int64_t blocks = n_rows * (K / 256);
        kq_launch(synth_kquant_kernel, (unsigned)kq_div_up(blocks, 4), 128, 0, st, type, (uint8_t *)W, n_rows,
                                                                           (int)(K / 256), key, sigma);
    }
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}

// few rows: 8 warps for up to 4096 values, 16 for more, so that a row is one round of loads; many: 8
static b200_status norm_q8(const float *x, const float *w, int64_t rows, int64_t h, float eps, float *y, int8_t *q, float *d, int16_t *bs, int64_t ldx,
                           const KqTokenImage &im, cudaStream_t st) {
    auto go = [&](auto kernel, int warps) { kq_launch(kernel, (unsigned)rows, warps * 32, 0, st, x, w, (int)h, eps, y, q, d, bs, ldx, im); };
    if (rows > 2 * kq_sm_count()) { // in registers up to 8192 values
        if (h <= 2048) go(rms_norm_q8_kernel<8, 1, false>, 8);
        else if (h <= 4096) go(rms_norm_q8_kernel<8, 2, false>, 8);
        else if (h <= 6144) go(rms_norm_q8_kernel<8, 3, false>, 8);
        else go(rms_norm_q8_kernel<8, 4, false>, 8);
    } else {
        if (h <= 2048) go(rms_norm_q8_kernel<8, 1, true>, 8);
        else if (h <= 4096) go(rms_norm_q8_kernel<8, 2, true>, 8);
        else go(rms_norm_q8_kernel<16, 2, true>, 16);
    }
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}
b200_status kq_rms_norm_image(const float *x, const float *w, int64_t h, float eps, const KqTokenImage &im, cudaStream_t st) {
    KQ_REQUIRE(h > 0 && h % 256 == 0 && im.m_pad > 0, "rms_norm: bad shape");
    return norm_q8(x, w, im.m_pad, h, eps, nullptr, nullptr, nullptr, nullptr, h, im, st);
}
b200_status kq_act_image(const float *x, const float *up, float *y, int64_t K, const KqTokenImage &im, cudaStream_t st) {
    KQ_REQUIRE(K > 0 && K % 256 == 0 && im.m_pad % 8 == 0 && ((uintptr_t)x & 15) == 0 && (((uintptr_t)up | (uintptr_t)y) & 15) == 0, "act_image: bad shape");
    const dim3 grid((unsigned)(im.m_pad / 8), (unsigned)(K / 256));
    if (up) kq_launch(act_to_image_kernel<true, false>, grid, dim3(256), 0, st, x, up, y, K, im, KqTileRows{});
    else kq_launch(act_to_image_kernel<false, false>, grid, dim3(256), 0, st, x, up, y, K, im, KqTileRows{});
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}

b200_status kq_rms_norm(const float *x, const float *w, int64_t T, int64_t h, float eps, float *y,
                        int8_t *q, float *d, int16_t *bs, cudaStream_t st, int64_t x_row_stride) {
    KQ_REQUIRE(T > 0 && h > 0 && h % 4 == 0, "rms_norm: bad shape");
    KQ_REQUIRE(!q || h % 256 == 0, "rms_norm: Q8 output needs h %% 256 == 0");
    KQ_REQUIRE(y || q, "rms_norm: no output");
    const int64_t ldx = x_row_stride ? x_row_stride : h;
    if (!q && h <= 128 && ldx % 4 == 0 && (((uintptr_t)x | (uintptr_t)y) & 15) == 0) {
        kq_launch(rms_norm_head_kernel, (unsigned)kq_div_up(T, 8), 256, 0, st, HeadRows{x, w, y, ldx}, T, HeadRows{}, (int64_t)0, (int)h, eps);
        KQ_COUNT_LAUNCH();
        KQ_LAUNCH_CHECK();
        return B200_OK;
    }
    if (q) return norm_q8(x, w, T, h, eps, y, q, d, bs, ldx, KqTokenImage{}, st);
    kq_launch(rms_norm_kernel, (unsigned)T, 256, 0, st, x, w, (int)h, eps, y, ldx);
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}

b200_status kq_act_image_tiles(const float *x, const float *up, int64_t K, const KqTokenImage &im, const KqTileRows &rows, cudaStream_t st) {
    KQ_REQUIRE(up && K > 0 && K % 256 == 0 && im.m_pad % 8 == 0 && rows.tile_tok % 8 == 0 && (((uintptr_t)x | (uintptr_t)up) & 15) == 0, "act_image: bad shape");
    kq_launch(act_to_image_kernel<true, true>, dim3((unsigned)(im.m_pad / 8), (unsigned)(K / 256)), dim3(256), 0, st, x, up, (float *)nullptr, K, im, rows);
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}

// the heads of q and of k in place, rows of h <= 128 values
b200_status kq_rms_norm_heads(float *q, const float *wq, int64_t q_rows, float *k, const float *wk, int64_t k_rows, int64_t h, float eps, cudaStream_t st) {
    if (h > 128 || h % 4 != 0 || (((uintptr_t)q | (uintptr_t)k) & 15)) {
        KQ_TRY(kq_rms_norm(q, wq, q_rows, h, eps, q, nullptr, nullptr, nullptr, st, 0));
        return kq_rms_norm(k, wk, k_rows, h, eps, k, nullptr, nullptr, nullptr, st, 0);
    }
    kq_launch(rms_norm_head_kernel, (unsigned)kq_div_up(q_rows + k_rows, 8), 256, 0, st, HeadRows{q, wq, q, h}, q_rows, HeadRows{k, wk, k, h}, k_rows, (int)h, eps);
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}

// y = silu(g) * u for [M][K] and its Q8 form; K a multiple of 256, pointers 16-byte aligned; y may be null or alias g
b200_status kq_swiglu_quantize(const float *g, const float *u, int64_t M, int64_t K, float *y, int8_t *q, float *d, int16_t *bs,
                               cudaStream_t st) {
    KQ_REQUIRE(M > 0 && K > 0 && K % 256 == 0, "swiglu_quantize: K must be a multiple of 256");
    KQ_REQUIRE((((uintptr_t)g | (uintptr_t)u | (uintptr_t)y | (uintptr_t)q) & 15) == 0, "swiglu_quantize: alignment");
    const int64_t nblocks = M * (K / 256);
    kq_launch(swiglu_quantize_kernel, (unsigned)kq_div_up(nblocks, 4), 128, 0, st, g, u, nblocks, y, q, d, bs);
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}

extern "C" b200_status b200_quantize_act(const float *x, int64_t M, int64_t K, int8_t *q, float *d,
                                         int16_t *bsum16, void *stream) {
    KQ_REQUIRE(M > 0 && K > 0 && K % 256 == 0, "quantize_act: K must be a multiple of 256");
    KQ_REQUIRE(((uintptr_t)x & 15) == 0 && ((uintptr_t)q & 15) == 0, "quantize_act: alignment");
    const int64_t nblocks = M * (K / 256);
    kq_launch(quantize_act_kernel, (unsigned)kq_div_up(nblocks, 4), 128, 0, (cudaStream_t)stream, x, nblocks, q, d,
                                                                                        bsum16);
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}

extern "C" b200_status b200_rms_norm(const float *x, const float *w, int64_t T, int64_t h, float eps,
                                     float *y, void *stream) {
    return kq_rms_norm(x, w, T, h, eps, y, nullptr, nullptr, nullptr, (cudaStream_t)stream, 0);
}

static b200_status repack(const void *src, void *dst, int64_t n_rows, int64_t k, int inverse,
                          cudaStream_t st) {
    KQ_REQUIRE(n_rows > 0 && k > 0 && k % 256 == 0, "repack_q6k: bad shape");
    const int nb = (int)(k / 256);
    const int64_t total = n_rows * nb * 105;
    kq_launch(repack_q6k_kernel, (unsigned)kq_div_up(total, 256), 256, 0, st, 
        (const uint16_t *)src, (uint16_t *)dst, n_rows, nb, kq_device_row_bytes(B200_TYPE_Q6_K, k) / 2,
        inverse);
    KQ_COUNT_LAUNCH();
    KQ_LAUNCH_CHECK();
    return B200_OK;
}

extern "C" b200_status b200_repack_q6k(const void *gguf_rows_dev, void *device_rows, int64_t n_rows,
                                       int64_t k, void *stream) {
    return repack(gguf_rows_dev, device_rows, n_rows, k, 0, (cudaStream_t)stream);
}
extern "C" b200_status b200_unpack_q6k(const void *device_rows, void *gguf_rows_dev, int64_t n_rows,
                                       int64_t k, void *stream) {
    return repack(device_rows, gguf_rows_dev, n_rows, k, 1, (cudaStream_t)stream);
}
