// Prefill contraction (M > 8 tokens): dispatch between the tensor-core kernel and, as a fall-back
// that can be forced with B200_GEMM_TC=0, a walk over the token batch in slabs of 8 through the
// decode kernel (identical results token for token, but weight-stream bound).
#include "kq_common.cuh"

#include <stdlib.h>

b200_status kq_launch_gemm_tc(const KqGemvSeg *segs, int nseg, const int8_t *q, const float *d, const int16_t *bs, int64_t M, int64_t K,
                              const float *residual, cudaStream_t st);

bool kq_gemm_takes_images() { // the tensor-core product is on
    static int use_tc = -1;
    if (use_tc < 0) {
        const char *v = getenv("B200_GEMM_TC");
        use_tc = !(v && v[0] == '0');
    }
    return use_tc != 0;
}

b200_status kq_launch_gemm(const KqGemvSeg *segs, int nseg, const int8_t *q, const float *d, const int16_t *bs, int64_t M, int64_t K,
                           const float *residual, cudaStream_t st) {
    if (kq_gemm_takes_images()) return kq_launch_gemm_tc(segs, nseg, q, d, bs, M, K, residual, st);
    const int64_t nb = K / 256;
    for (int i = 0; i < nseg; i++)
        for (int64_t m0 = 0; m0 < M; m0 += 8) {
            const int mc = (int)(M - m0 < 8 ? M - m0 : 8);
            KqGemvSeg sg = segs[i];
            sg.y += m0 * sg.n_rows;
            KQ_TRY(kq_launch_gemv(&sg, 1, q + m0 * K, d + m0 * nb, bs + m0 * nb * 16, mc, K, residual ? residual + m0 * sg.n_rows : nullptr, 0,
                                  nullptr, st));
        }
    return B200_OK;
}
