// gemm_ordered.cu -- GEMM in the reference's summation order, bit-exact.
//
// Every C element is computed exactly as the reference's host check loop
// computes it, so results are bit-identical to those loops:
//   two-level sum (dgemm_release_V1.1/host_code/dgemm_demo.c:233-252,
//   sgemm_release_V1.3.2/host_code/sgemm_demo.c:214-242,
//   irr_*_V0.0 demos :205-222): per K block of k_block (K_G = 512): tmp = 0,
//   tmp = fma(a, b, tmp) ascending in k, c += tmp; then the tail block the
//   same way (always added); scalar beta added last;
//   three-level sum (irr_thinB_sgemm_release_V1.2/host_code/
//   irr_thinB_sgemm_demo.c:217-239): slabs of k_slab (K_A) inside blocks of
//   k_block (K_G), tmp_i += tmp_s, tmp_o += tmp_i, c = c0 + (tmp_o + beta).
// FP32 products use the double-precision fma() on float operands rounded
// back to float, as those C loops do (fma() is the double libm function).
//
// Tiling: a CTA owns a TM x TN tile of C, a thread RM x RN neighbouring
// elements, K is staged through double-buffered shared memory 16 at a time
// with the next step's loads in flight.  The tiling does not change the
// per-element order.
//
// FP64 is bound by the FP64 pipe (2 DFMA per clock and SM, ~1.1 TFLOP/s); it
// is also the library's plain DGEMM.  FP32 would be too, and by the
// conversions around each double fma; it runs on the FP32 pipe instead (see
// fmac_step below).
#include <math.h>

#include "gb_common.cuh"
#include "sm100_ptx.cuh"
#include "tile_stage.cuh"

namespace gb {
namespace {

constexpr int BK = STAGE_K;

template <typename T>
struct Ord;

template <>
struct Ord<double> {
    __device__ static double fmac(double a, double b, double t) { return __fma_rn(a, b, t); }
    __device__ static double add(double a, double b) { return __dadd_rn(a, b); }
    __device__ static double mul(double a, double b) { return __dmul_rn(a, b); }
    // the same product, never computed ahead of the branch around it: an unused multiply of every
    // staged value would take 4-6 % of the FP64 pipe
    __device__ static double scaled(double a, double b) {
        double v;
        asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(v) : "d"(a), "d"(b));
        return v;
    }
    __device__ static bool plain(double) { return true; }
};

template <>
struct Ord<float> {
    // (float) fma((double)a, (double)b, (double)t): the reference's double fma
    __device__ static float fmac(float a, float b, float t) {
        return __double2float_rn(__fma_rn((double)a, (double)b, (double)t));
    }
    __device__ static float add(float a, float b) { return __fadd_rn(a, b); }
    __device__ static float mul(float a, float b) { return __fmul_rn(a, b); }
    __device__ static float scaled(float a, float b) { return mul(a, b); }
    // zero, or a magnitude in [2^-40, 2^45] (see fmac_step)
    __device__ static bool plain(float v) {
        const unsigned u = __float_as_uint(v) & 0x7fffffffu;
        return u == 0u || u - 0x2B800000u <= 0x56000000u - 0x2B800000u;
    }
};

// One k of a thread's RM x RN products: t = fmac(a, b, t).
template <typename T, int RM, int RN>
struct Micro {
    T a[RM], b[RN];
    __device__ __forceinline__ void load(const T *As, const T *Bs) {
#pragma unroll
        for (int i = 0; i < RM; i++) a[i] = As[i];
#pragma unroll
        for (int j = 0; j < RN; j++) b[j] = Bs[j];
    }
    __device__ __forceinline__ void exact(T (&t)[RM][RN]) const {
#pragma unroll
        for (int i = 0; i < RM; i++)
#pragma unroll
            for (int j = 0; j < RN; j++) t[i][j] = Ord<T>::fmac(a[i], b[j], t[i][j]);
    }
};

// FP32 without the FP64 pipe.  The wanted value is x = a b + t rounded to 53
// bits and then to 24.  r = fmaf(a, b, t) rounds x once; the two differ only
// if the first rounding lands on the midpoint of two floats and x does not.
// With p + q = a b exactly (q by an fma):
//  - 2^-22 |p| <= |t| < 16 |p|: x has at most 53 significant bits, the first
//    rounding changes nothing and r is the result;
//  - |t| >= 16 |p|: the distance e = x - r = (p - (r - t)) + q is formed in
//    FP32 (r - t and p - (r - t) are exact, the sum rounds once).  If the two
//    differ, x lies within 2^-28 of half a spacing of the midpoint, and r + (1 + 2^-21) e
//    rounds away from r;
//  - |t| < 2^-22 |p|: not decided here.
// A thread that finds a product undecided or near a midpoint (5.6e-7 of random
// products; every tie) redoes its products of that k with the double fma.
// All this holds while nothing nears the ends of FP32's range: operands are
// checked as they are staged to be zero or in [2^-40, 2^45], so that products
// and sums are multiples of 2^-126 below 2^122; a chain with any other operand
// (Inf and NaN too) runs on the double fma from that slice on.
// Nine FP32 operations (packed in pairs) and four compares a product in place
// of a DFMA and its conversions (the FP64 pipe serves 2 lanes a clock and SM,
// the FP32 pipe 128): 768 x 1000 x 1536
// takes 0.70 ms, with the double fma 12.0.
template <int RM, int RN>
__device__ __forceinline__ void fmac_step(const Micro<float, RM, RN> &m, float (&t)[RM][RN]) {
    static_assert(RN % 2 == 0, "packed pairs of columns");
    const uint64_t minus1 = ptx::f2_pack(-1.f, -1.f), grow = ptx::f2_pack(1.f + 0x1p-21f, 1.f + 0x1p-21f);
    const uint64_t p16 = ptx::f2_pack(16.f, 16.f), ptiny = ptx::f2_pack(0x1p-22f, 0x1p-22f);
    float r[RM][RN];
    bool redo = false;
#pragma unroll
    for (int j = 0; j < RN; j += 2) {
        const uint64_t b2 = ptx::f2_pack(m.b[j], m.b[j + 1]), nb2 = ptx::f2_pack(-m.b[j], -m.b[j + 1]);
#pragma unroll
        for (int i = 0; i < RM; i++) {
            const uint64_t a2 = ptx::f2_pack(m.a[i], m.a[i]), t2 = ptx::f2_pack(t[i][j], t[i][j + 1]);
            const uint64_t p2 = ptx::f2_mul(a2, b2);
            const uint64_t nq2 = ptx::f2_fma_rn(a2, nb2, p2);       // -q
            const uint64_t r2 = ptx::f2_fma_rn(a2, b2, t2);
            const uint64_t z2 = ptx::f2_fma_rn(t2, minus1, r2);     // r - t
            const uint64_t w2 = ptx::f2_fma_rn(z2, minus1, p2);     // p - (r - t)
            const uint64_t e2 = ptx::f2_fma_rn(nq2, minus1, w2);    // + q
            const uint64_t s2 = ptx::f2_fma_rn(e2, grow, r2);
            float s[2], big[2], tiny[2];
            ptx::f2_unpack(s2, s[0], s[1]);
            ptx::f2_unpack(r2, r[i][j], r[i][j + 1]);
            ptx::f2_unpack(ptx::f2_mul(p2, p16), big[0], big[1]);
            ptx::f2_unpack(ptx::f2_mul(p2, ptiny), tiny[0], tiny[1]);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float at = fabsf(t[i][j + h]);
                redo = redo || (at >= fabsf(big[h]) && s[h] != r[i][j + h]) || at < fabsf(tiny[h]);
            }
        }
    }
    if (redo) {
        m.exact(t);
    } else {
#pragma unroll
        for (int i = 0; i < RM; i++)
#pragma unroll
            for (int j = 0; j < RN; j++) t[i][j] = r[i][j];
    }
}

// The first k of a chain: a b rounded to 53 bits (exact) and to 24.
template <int RM, int RN>
__device__ __forceinline__ void first_step(const Micro<float, RM, RN> &m, float (&t)[RM][RN]) {
#pragma unroll
    for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) t[i][j] = __fmaf_rn(m.a[i], m.b[j], 0.f);
}
template <int RM, int RN>
__device__ __forceinline__ void first_step(const Micro<double, RM, RN> &m, double (&t)[RM][RN]) {
    m.exact(t);
}

template <int RM, int RN>
__device__ __forceinline__ void fmac_step(const Micro<double, RM, RN> &m, double (&t)[RM][RN]) {
    m.exact(t);
}

struct OrdParams {
    int64_t M, N, K, lda, ldb, ldc;
    int ta, tb;
    int64_t kg, ka;       // block and slab (ka == 0: two-level)
    int start_from_c;     // c starts from C_in (else +0)
    int scale_a, scale_b; // alpha pre-scales op(A) / op(B)
    int scalar_beta;      // add beta as a scalar at the end
    int blas_general;     // C = alpha*c + beta*C_in after the sum
};

// Stage a slice, scaled; whether an operand is outside the FP32 path's range.
template <typename T, int TM, int TN, int NT>
__device__ __forceinline__ bool stage(const StageLoader<T, TM, TN, NT> &ld, Stage<T, TM, TN> &s, int buf,
                                      const OrdParams &p, T alpha) {
    bool odd = false;
    auto put = [&](T v, int scale) {
        if (scale) v = Ord<T>::scaled(alpha, v);
        odd = odd || !Ord<T>::plain(v);
        return v;
    };
    ld.store(s, buf, p, [&](T v) { return put(v, p.scale_a); }, [&](T v) { return put(v, p.scale_b); });
    return odd;
}

// Sum op(A)op(B) over k in [ks, ke) into t (a fresh chain, t starts at 0).
template <typename T, int TM, int TN, int RM, int RN>
__device__ __forceinline__ void chain(const T *__restrict__ A, const T *__restrict__ B, Stage<T, TM, TN> &s,
                                      const OrdParams &p, int64_t m0, int64_t n0, int64_t ks, int64_t ke, T alpha,
                                      T (&t)[RM][RN]) {
    constexpr int NT = TM / RM * (TN / RN);
    constexpr int KU = sizeof(T) == 4 ? 2 : 4;   // unrolled steps
    const int tx = threadIdx.x % (TN / RN), ty = threadIdx.x / (TN / RN);
#pragma unroll
    for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) t[i][j] = T(0);
    if (ks >= ke) return;
    StageLoader<T, TM, TN, NT> ld;
    ld.fetch(A, B, p, m0, n0, ks, ke);
    int buf = 0;
    // a chain's first buffer was last read before the previous chain's last barrier
    bool odd = __syncthreads_or(stage(ld, s, 0, p, alpha));
    for (int64_t k0 = ks; k0 < ke; k0 += BK, buf ^= 1) {
        const bool more = k0 + BK < ke;
        if (more) ld.fetch(A, B, p, m0, n0, k0 + BK, ke);
        const int kn = (int)(ke - k0 < BK ? ke - k0 : BK);
        Micro<T, RM, RN> m;
        int kk = 0;
        if (odd) {
            for (; kk < kn; kk++) {
                m.load(&s.A[buf][kk][ty * RM], &s.B[buf][kk][tx * RN]);
                m.exact(t);
            }
        } else if (k0 == ks) {
            m.load(&s.A[buf][0][ty * RM], &s.B[buf][0][tx * RN]);
            first_step(m, t);
            kk = 1;
        }
        if (kk == 0 && kn == BK) {
#pragma unroll KU
            for (int k = 0; k < BK; k++) {
                m.load(&s.A[buf][k][ty * RM], &s.B[buf][k][tx * RN]);
                fmac_step(m, t);
            }
        } else {
#pragma unroll 1
            for (; kk < kn; kk++) {
                m.load(&s.A[buf][kk][ty * RM], &s.B[buf][kk][tx * RN]);
                fmac_step(m, t);
            }
        }
        const bool next_odd = more && stage(ld, s, buf ^ 1, p, alpha);
        odd = __syncthreads_or(next_odd) || odd;
    }
}

// 512 threads an SM at least.  FP32, two CTAs of 64 x 64 and 128 registers a thread: 4.5 TFLOP/s
// at 2048 x 2048 x 1024, 3.8 with one.  FP64 in slabs would take 136 registers and one CTA:
// 297 x 1876 x 3122 in slabs of 512 3577 us, 3369 with two.  (FP32 in slabs needs its 222.)
template <typename T, int TM, int TN, int RM, int RN, bool SLABS>
__global__ void __launch_bounds__(TM / RM * (TN / RN), sizeof(T) == 8 || !SLABS ? 512 * RM * RN / (TM * TN) : 1)
    gemm_ordered_kernel(const T *__restrict__ A, const T *__restrict__ B, T *__restrict__ C, OrdParams p, T alpha,
                        T beta, unsigned tiles_n) {
    __shared__ __align__(16) Stage<T, TM, TN> s;
    const int tx = threadIdx.x % (TN / RN), ty = threadIdx.x / (TN / RN);
    const int64_t m0 = (int64_t)(blockIdx.x / tiles_n) * TM, n0 = (int64_t)(blockIdx.x % tiles_n) * TN;

    T c[RM][RN], t[RM][RN];
#pragma unroll
    for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) {
            const int64_t m = m0 + ty * RM + i, n = n0 + tx * RN + j;
            c[i][j] = (p.start_from_c && m < p.M && n < p.N) ? C[m * p.ldc + n] : T(0);
        }

    if (!SLABS) {
        // two-level: full K blocks, then the (possibly empty) tail block
        const int64_t kfull = p.K - p.K % p.kg;
        for (int64_t kb = 0; kb <= kfull; kb += p.kg) {
            chain<T, TM, TN, RM, RN>(A, B, s, p, m0, n0, kb, kb < kfull ? kb + p.kg : p.K, alpha, t);
#pragma unroll
            for (int i = 0; i < RM; i++)
#pragma unroll
                for (int j = 0; j < RN; j++) c[i][j] = Ord<T>::add(c[i][j], t[i][j]);
        }
        if (p.scalar_beta) {
#pragma unroll
            for (int i = 0; i < RM; i++)
#pragma unroll
                for (int j = 0; j < RN; j++) c[i][j] = Ord<T>::add(c[i][j], beta);
        }
    } else {
        // three-level: slabs of ka inside blocks of kg (min-sized at the end)
        T to[RM][RN], ti[RM][RN];
#pragma unroll
        for (int i = 0; i < RM; i++)
#pragma unroll
            for (int j = 0; j < RN; j++) to[i][j] = T(0);
        for (int64_t ko = 0; ko < p.K; ko += p.kg) {
            int64_t kgc = p.kg < p.K - ko ? p.kg : p.K - ko;
#pragma unroll
            for (int i = 0; i < RM; i++)
#pragma unroll
                for (int j = 0; j < RN; j++) ti[i][j] = T(0);
            for (int64_t ki = 0; ki < kgc; ki += p.ka) {
                int64_t kac = p.ka < kgc - ki ? p.ka : kgc - ki;
                chain<T, TM, TN, RM, RN>(A, B, s, p, m0, n0, ko + ki, ko + ki + kac, alpha, t);
#pragma unroll
                for (int i = 0; i < RM; i++)
#pragma unroll
                    for (int j = 0; j < RN; j++) ti[i][j] = Ord<T>::add(ti[i][j], t[i][j]);
            }
#pragma unroll
            for (int i = 0; i < RM; i++)
#pragma unroll
                for (int j = 0; j < RN; j++) to[i][j] = Ord<T>::add(to[i][j], ti[i][j]);
        }
#pragma unroll
        for (int i = 0; i < RM; i++)
#pragma unroll
            for (int j = 0; j < RN; j++) {
                const T v = p.scalar_beta ? Ord<T>::add(to[i][j], beta) : to[i][j];
                c[i][j] = Ord<T>::add(c[i][j], v);
            }
    }

#pragma unroll
    for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) {
            const int64_t m = m0 + ty * RM + i, n = n0 + tx * RN + j;
            if (m < p.M && n < p.N) {
                T v = c[i][j];
                if (p.blas_general) {
                    T bc = (beta == T(0)) ? T(0) : Ord<T>::mul(beta, C[m * p.ldc + n]);
                    v = Ord<T>::add(Ord<T>::mul(alpha, v), bc);
                }
                C[m * p.ldc + n] = v;
            }
        }
}

template <typename T, int TM, int TN, int RM, int RN>
gb_status launch_tile(const GemmArgs &g, const OrdParams &p) {
    const int64_t tn = ceil_div(g.N, TN), tiles = ceil_div(g.M, TM) * tn;
    if (tiles > 0x7fffffff) return set_status(GB_ERR_UNSUPPORTED, "ordered gemm: C too large");
    const int nt = TM / RM * (TN / RN);
    auto kernel = p.ka > 0 ? gemm_ordered_kernel<T, TM, TN, RM, RN, true> : gemm_ordered_kernel<T, TM, TN, RM, RN, false>;
    kernel<<<(unsigned)tiles, nt, 0, g.stream>>>((const T *)g.A, (const T *)g.B, (T *)g.C, p, (T)g.alpha, (T)g.beta,
                                                 (unsigned)tn);
    GB_LAUNCH_CHECK("gemm_ordered_kernel");
    return ok();
}

// Estimated time (ns) of one k with this tiling: the SM with the most tiles
// decides, each tile costs `tile`, and an SM with few of them still waits out
// a step's latency, `least`.
inline double step_ns(const GemmArgs &g, int tm, int tn, double least, double tile, double once = 0.0) {
    const double tiles = (double)ceil_div(g.M, tm) * (double)ceil_div(g.N, tn);
    const double t = ceil(tiles / sm_count()) * tile + once;
    return t > least ? t : least;
}

template <typename T>
gb_status launch(const GemmArgs &g) {
    OrdParams p;
    p.M = g.M; p.N = g.N; p.K = g.K;
    p.lda = g.lda; p.ldb = g.ldb; p.ldc = g.ldc;
    p.ta = g.ta; p.tb = g.tb;
    p.kg = g.k_block > 0 ? g.k_block : 512;
    p.ka = g.k_slab > 0 ? g.k_slab : 0;
    p.start_from_c = 0; p.scale_a = 0; p.scale_b = 0; p.scalar_beta = 0; p.blas_general = 0;
    if (g.semantics == GB_SEM_BLAS) {
        if (g.alpha == 1.0 && g.beta == 1.0) {
            p.start_from_c = 1;                 // C += op(A)op(B), the reference update
        } else {
            p.blas_general = 1;                 // C = alpha*sum + beta*C
        }
    } else {
        p.scalar_beta = 1;
        p.start_from_c = (g.semantics == GB_SEM_ACCUM_SCALAR_BETA);
        if (g.alpha_on_b) p.scale_b = 1; else p.scale_a = 1;
    }
    if (g.M == 0 || g.N == 0) return ok();
    if (ceil_div(g.M, 64) > 65535)
        return set_status(GB_ERR_UNSUPPORTED, "ordered gemm: M too large (%lld)", (long long)g.M);
    // The tiling of least estimated time; the constants are measured (a k of
    // FP32 64 x 64 / 32 x 64 / 32 x 32: 340 / 280 / 165 ns alone on an SM, 268 /
    // 140 / 87 a tile when there are many; FP64 32 x 32 / 16 x 16: 310 / 120 and 256 /
    // 78).  FP32 768 x 1000 x 1536: 703 us in 32 x 64, 796 in 32 x 32, 839 in
    // 64 x 64; 256^3: 75 / 43 / 92; 2048 x 2048 x 512: 1004 / 1182 / 961.  FP64 256^3:
    // 81 us in 32 x 32, 50 in 16 x 16; 128 x 200 x 300: 96 / 36; 512^3: 273 / 292 (64 x 64:
    // 283, 328 and 554).
    if constexpr (sizeof(T) == 8) {
        const double t32 = step_ns(g, 32, 32, 310, 256), t16 = step_ns(g, 16, 16, 120, 78, 40);
        if (t16 < t32) return launch_tile<T, 16, 16, 1, 1>(g, p);
        return launch_tile<T, 32, 32, 2, 2>(g, p);
    } else {
        const double t64 = step_ns(g, 64, 64, 340, 268), t48 = step_ns(g, 32, 64, 280, 140, 40),
                     t32 = step_ns(g, 32, 32, 165, 87);
        if (t32 < t48 && t32 < t64) return launch_tile<T, 32, 32, 2, 2>(g, p);
        if (t48 < t64) return launch_tile<T, 32, 64, 4, 4>(g, p);
        return launch_tile<T, 64, 64, 4, 4>(g, p);
    }
}

}  // namespace

gb_status launch_gemm_ordered_f64(const GemmArgs &g) { return launch<double>(g); }
gb_status launch_gemm_ordered_f32(const GemmArgs &g) { return launch<float>(g); }

}  // namespace gb
