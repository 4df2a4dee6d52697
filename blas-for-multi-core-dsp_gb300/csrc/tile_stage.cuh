// tile_stage.cuh -- shared-memory staging of a C tile's operands for the
// kernels that sum on the CUDA cores (gemm_ordered.cu, grouped.cu): slices of
// 16 k of op(A) (TM rows) and op(B) (TN columns), k-major, two buffers, the
// next slice's loads held in registers while the current one is summed.
#pragma once

#include <stdint.h>

namespace gb {

constexpr int STAGE_K = 16;

// rows padded by 16 bytes: aligned vector reads, spread banks
template <typename T, int TM, int TN>
struct Stage {
    static constexpr int PAD = 16 / (int)sizeof(T);
    T A[2][STAGE_K][TM + PAD], B[2][STAGE_K][TN + PAD];
};

// One thread's share (of NT threads) of a slice.  P: M, N, lda, ldb, ta, tb of the product.
template <typename T, int TM, int TN, int NT>
struct StageLoader {
    static constexpr int BK = STAGE_K, NA = TM * BK / NT, NB = TN * BK / NT;
    static_assert(TM * BK % NT == 0 && TN * BK % NT == 0, "whole elements a thread");
    T a[NA], b[NB];

    // k in [k0, min(k0 + 16, kend)) of the tile at (m0, n0); k past kend as zeros.  Rows past M
    // (columns past N) repeat the last one: their products are never stored.
    template <typename P>
    __device__ __forceinline__ void fetch(const T *__restrict__ A, const T *__restrict__ B, const P &p, int64_t m0,
                                          int64_t n0, int64_t k0, int64_t kend) {
#pragma unroll
        for (int r = 0; r < NA; r++) {
            const int l = (int)threadIdx.x + r * NT;
            const int mm = p.ta ? l % TM : l / BK, kk = p.ta ? l / TM : l % BK;
            const int64_t m = m0 + mm < p.M ? m0 + mm : p.M - 1, k = k0 + kk;
            a[r] = k < kend ? (p.ta ? A[k * p.lda + m] : A[m * p.lda + k]) : T(0);
        }
#pragma unroll
        for (int r = 0; r < NB; r++) {
            const int l = (int)threadIdx.x + r * NT;
            const int nn = p.tb ? l / BK : l % TN, kk = p.tb ? l % BK : l / TN;
            const int64_t n = n0 + nn < p.N ? n0 + nn : p.N - 1, k = k0 + kk;
            b[r] = k < kend ? (p.tb ? B[n * p.ldb + k] : B[k * p.ldb + n]) : T(0);
        }
    }

    // into buffer `buf`, each value as fa / fb returns it
    template <typename P, typename FA, typename FB>
    __device__ __forceinline__ void store(Stage<T, TM, TN> &s, int buf, const P &p, FA fa, FB fb) const {
#pragma unroll
        for (int r = 0; r < NA; r++) {
            const int l = (int)threadIdx.x + r * NT;
            s.A[buf][p.ta ? l / TM : l % BK][p.ta ? l % TM : l / BK] = fa(a[r]);
        }
#pragma unroll
        for (int r = 0; r < NB; r++) {
            const int l = (int)threadIdx.x + r * NT;
            s.B[buf][p.tb ? l % BK : l / TN][p.tb ? l / BK : l % TN] = fb(b[r]);
        }
    }
};

}  // namespace gb
