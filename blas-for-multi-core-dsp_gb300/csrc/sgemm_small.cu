// sgemm_small.cu -- plain FP32 SGEMM for products that cannot fill the GPU
// with 128 x 128 tiles (the serving mix starts at 256^3, four such tiles).
//
// The same reference kernels as sgemm_simt.cu (sgemm_release_V1.3.2/
// device_code/sgemm_kernel.c:984-2474 and the drivers :2476-4043).  What
// bounds a small product is latency: the steps along K one after the other,
// and the loads before the first.  So C is cut into TM x TN tiles and K into
// S x G parts: G groups of threads of one CTA and the S CTAs of a cluster each
// sum their part of K (16 k a stage, four stages of cp.async in flight), the
// groups' sums are added in shared memory and the CTAs' through distributed
// shared memory, each CTA finishing TM / S rows of the tile.  Fixed order, no
// workspace.  Within a part the FMAs run in k order, two outputs of a row in
// one packed FP32x2 instruction.
#include <cooperative_groups.h>
#include <math.h>

#include "gb_common.cuh"
#include "sm100_ptx.cuh"

namespace cg = cooperative_groups;

namespace gb {
namespace {

constexpr int BK = 16, ST = 4;

struct SmallParams {
    int64_t M, N, K, lda, ldb, ldc;
    int ta, tb;
    float alpha, beta;
    int semantics;
    int64_t kpart;   // k of a part, a multiple of BK
    unsigned tiles_n;
};

__device__ __forceinline__ void cp_async4(float *dst, const float *src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(ptx::smem_u32(dst)), "l"(src), "r"(live ? 4u : 0u)
                 : "memory");
}

template <int TM, int TN, int G>
struct SmallCfg {
    static constexpr int RM = 4, RN = 4, NG = TM / RM * (TN / RN), NT = NG * G;   // threads of a group, of the CTA
    static constexpr int LA = TM + 4, LB = TN + 4;                                 // padded slice rows
    static constexpr int STAGE = BK * (LA + LB);                                   // floats
    static constexpr int SMEM = (ST * G * STAGE > TM * LB * G ? ST * G * STAGE : TM * LB * G) * 4;
};

template <int TM, int TN, int G>
__global__ void __launch_bounds__(SmallCfg<TM, TN, G>::NT)
    sgemm_small_kernel(const float *__restrict__ A, const float *__restrict__ B, float *__restrict__ C, SmallParams p) {
    using F = SmallCfg<TM, TN, G>;
    extern __shared__ __align__(16) float sm[];
    cg::cluster_group cluster = cg::this_cluster();
    const int S = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const unsigned tile = blockIdx.x / (unsigned)S;
    const int64_t m0 = (int64_t)(tile / p.tiles_n) * TM, n0 = (int64_t)(tile % p.tiles_n) * TN;
    const int grp = threadIdx.x / F::NG, tid = threadIdx.x % F::NG;
    const int tx = tid % (TN / F::RN), ty = tid / (TN / F::RN);
    const int64_t ks = (int64_t)(rank * G + grp) * p.kpart;
    float *st = sm + grp * ST * F::STAGE;

    // This thread's elements of a slice: element r of op(A) sits r * NG / TM steps of k (stored K x M) or
    // r * NG / 16 rows (stored M x K) after its first; the same for op(B).  Outside the operand: zeros.
    const int ak = p.ta ? tid / TM : tid % BK, am = p.ta ? tid % TM : tid / BK;
    const int bk = p.tb ? tid % BK : tid / TN, bn = p.tb ? tid / BK : tid % TN;
    const int adk = p.ta ? F::NG / TM : 0, adm = p.ta ? 0 : F::NG / BK;
    const int bdk = p.tb ? 0 : F::NG / TN, bdn = p.tb ? F::NG / BK : 0;
    const float *ap = A + (p.ta ? (ks + ak) * p.lda + m0 + am : (m0 + am) * p.lda + ks + ak);
    const float *bp = B + (p.tb ? (n0 + bn) * p.ldb + ks + bk : (ks + bk) * p.ldb + n0 + bn);
    const int64_t ar = p.ta ? adk * p.lda : adm * p.lda, as_step = p.ta ? BK * p.lda : BK;
    const int64_t br = p.tb ? bdn * p.ldb : bdk * p.ldb, bs_step = p.tb ? BK : BK * p.ldb;
    const int mlim = (int)(p.M - m0 < TM ? p.M - m0 : TM), nlim = (int)(p.N - n0 < TN ? p.N - n0 : TN);
    int64_t kleft = p.K - ks;   // k of this part that lie inside, from the next slice on
    auto fetch = [&](int slot) {
        float *as = st + slot * F::STAGE + ak * F::LA + am, *bs = st + slot * F::STAGE + BK * F::LA + bk * F::LB + bn;
        const int klim = (int)(kleft < BK ? kleft : BK);
#pragma unroll
        for (int r = 0; r < TM * BK / F::NG; r++) {
            const bool live = ak + r * adk < klim && am + r * adm < mlim;
            cp_async4(as + r * adk * F::LA + r * adm, live ? ap + r * ar : A, live);
        }
#pragma unroll
        for (int r = 0; r < TN * BK / F::NG; r++) {
            const bool live = bk + r * bdk < klim && bn + r * bdn < nlim;
            cp_async4(bs + r * bdk * F::LB + r * bdn, live ? bp + r * br : B, live);
        }
        ap += as_step;
        bp += bs_step;
        kleft -= BK;
    };
    const int steps = (int)(p.kpart / BK);
#pragma unroll
    for (int i = 0; i < ST - 1; i++) {
        if (i < steps) fetch(i);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }

    uint64_t acc[F::RM][F::RN / 2];
#pragma unroll
    for (int i = 0; i < F::RM; i++)
#pragma unroll
        for (int j = 0; j < F::RN / 2; j++) acc[i][j] = 0ull;
    for (int i = 0; i < steps; i++) {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();
        if (i + ST - 1 < steps) fetch((i + ST - 1) % ST);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float *as = st + i % ST * F::STAGE + ty * F::RM, *bs = st + i % ST * F::STAGE + BK * F::LA + tx * F::RN;
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            const float4 a = *reinterpret_cast<const float4 *>(as + kk * F::LA);
            const float4 b = *reinterpret_cast<const float4 *>(bs + kk * F::LB);
            const uint64_t b01 = ptx::f2_pack(b.x, b.y), b23 = ptx::f2_pack(b.z, b.w);
            const float av[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const uint64_t a2 = ptx::f2_pack(av[r], av[r]);
                acc[r][0] = ptx::f2_fma_rn(a2, b01, acc[r][0]);
                acc[r][1] = ptx::f2_fma_rn(a2, b23, acc[r][1]);
            }
        }
    }

    // the groups' sums to shared memory, added group by group into group 0's
    __syncthreads();
    float *sum = sm + grp * TM * F::LB;
#pragma unroll
    for (int r = 0; r < F::RM; r++) {
        float4 v;
        ptx::f2_unpack(acc[r][0], v.x, v.y);
        ptx::f2_unpack(acc[r][1], v.z, v.w);
        *reinterpret_cast<float4 *>(sum + (ty * F::RM + r) * F::LB + tx * F::RN) = v;
    }
    __syncthreads();
    if (G > 1) {
        for (int e = threadIdx.x; e < TM * TN / 4; e += F::NT) {
            float4 *o = reinterpret_cast<float4 *>(sm + e / (TN / 4) * F::LB + e % (TN / 4) * 4);
            float4 v = *o;
#pragma unroll
            for (int g = 1; g < G; g++) {
                const float4 w = o[g * TM * F::LB / 4];
                v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
            }
            *o = v;
        }
    }
    if (S > 1) cluster.sync();
    else __syncthreads();

    // rows of this CTA: the CTAs' sums in rank order (all loads in flight at once), then the epilogue
    const int rows = TM / S;
    for (int e = threadIdx.x; e < rows * TN / 4; e += F::NT) {
        const int rr = rank * rows + e / (TN / 4), cc = e % (TN / 4) * 4;
        float *o = sm + rr * F::LB + cc;
        float4 part[8];
#pragma unroll
        for (int s = 0; s < 8; s++)
            if (s < S) part[s] = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(o, s));
#pragma unroll
        for (int s = 1; s < 8; s++)
            if (s < S) {
                part[0].x += part[s].x; part[0].y += part[s].y;
                part[0].z += part[s].z; part[0].w += part[s].w;
            }
        const int64_t m = m0 + rr;
        const float acc4[4] = {part[0].x, part[0].y, part[0].z, part[0].w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int64_t n = n0 + cc + j;
            if (m >= p.M || n >= p.N) continue;
            float *cp = C + m * p.ldc + n;
            float v = p.alpha * acc4[j];
            if (p.semantics == GB_SEM_BLAS) {
                if (p.beta != 0.f) v = fmaf(p.beta, *cp, v);
            } else if (p.semantics == GB_SEM_SCALAR_BETA) {
                v = v + p.beta;
            } else {
                v = *cp + (v + p.beta);
            }
            *cp = v;
        }
    }
    if (S > 1) cluster.sync();   // the others may still read this CTA's sums
}

template <int TM, int TN, int G>
gb_status launch_small(const GemmArgs &g, SmallParams p, int S) {
    using F = SmallCfg<TM, TN, G>;
    auto kernel = sgemm_small_kernel<TM, TN, G>;
    static std::atomic<uint64_t> attr{0};
    if (device_setup_needed(attr)) {
        GB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F::SMEM));
        device_setup_done(attr);
    }
    const int64_t tn = ceil_div(g.N, TN), tiles = ceil_div(g.M, TM) * tn;
    p.tiles_n = (unsigned)tn;
    p.kpart = ceil_div(ceil_div(g.K, (int64_t)S * G), BK) * BK;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)S;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * S));
    cfg.blockDim = dim3(F::NT);
    cfg.dynamicSmemBytes = F::SMEM;
    cfg.stream = g.stream;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, (const float *)g.A, (const float *)g.B, (float *)g.C, p));
    GB_LAUNCH_CHECK("sgemm_small_kernel");
    return ok();
}

}  // namespace

// Estimated times in us, fitted to measurements on GB300 (n CTAs on the
// busiest SM): a launch and its first loads, each CTA's start and store, and
// the staged steps one after the other.
//
//                        32x32, G 4     64x64, G 1     128x128 (sgemm_simt.cu)
//   256^3                6.2 (S 2)      8.2 (S 4)      31.9
//   512^3                14.6 (S 1)     14.4 (S 4)     57.4
//   64 x 64 x 4096       11.3 (S 8)     26.7 (S 8)     440
//   100 x 700 x 900      14.4 (S 4)     14.4 (S 8)     100
//   1024 x 1024 x 128    16.4 (S 1)     14.4 (S 1)     18.5
//   2000 x 2000 x 32     32.8 (S 1)     16.5 (S 1)     14.4
//   1024^3                              78   (S 1)     117
//   1500^3                              216  (S 1)     211
//   2048^3                              480  (S 1)     401
//   4096^3                              3514 (S 1)     2585
static double small_us(const GemmArgs &g, int tm, int tn, int S, double kstep, double cta, double step, double per_cta) {
    const double ctas = (double)ceil_div(g.M, tm) * (double)ceil_div(g.N, tn) * S;
    const double n = ceil(ctas / sm_count()), steps = ceil((double)g.K / (kstep * S));
    return 3.0 + n * cta + steps * (step + per_cta * n) + (S > 1 ? 1.0 : 0.0);
}

// The plan of least estimated time; tile 0: 128 x 128 tiles.  K is split for
// the products GB_ALGO_AUTO sends here (at most 2^27 multiply-adds, or K <
// 64); larger ones, which only ask for plain FFMA sums to compare with, keep
// one sum per output in k order, and a 64 x 64 tile's step takes 0.48 us there
// (the shared-memory reads of its four rows and columns a thread).
SmallPlan sgemm_small_plan(const GemmArgs &g) {
    const double n128 = ceil((double)ceil_div(g.M, 128) * (double)ceil_div(g.N, 128) / sm_count());
    const double step = 0.69 * n128 > 0.9 ? 0.69 * n128 : 0.9;
    SmallPlan best{0, 0};
    double t = 3.0 + 2.0 * n128 + ceil((double)g.K / 8.0) * step;
    const bool split = g.K < 64 || (double)g.M * (double)g.N * (double)g.K <= 134217728.0;
    for (int S = 1; S <= (split ? 8 : 1); S *= 2) {
        const double t32 = small_us(g, 32, 32, S, 64, 1.0, 0.45, 0.35), t64 = small_us(g, 64, 64, S, 16, 1.2, 0.4, split ? 0.27 : 0.48);
        if (split && t32 < t) { t = t32; best = SmallPlan{32, S}; }
        if (t64 < t) { t = t64; best = SmallPlan{64, S}; }
    }
    return best;
}

gb_status launch_sgemm_small(const GemmArgs &g, SmallPlan plan) {
    SmallParams p{g.M, g.N, g.K, g.lda, g.ldb, g.ldc, g.ta, g.tb, (float)g.alpha, (float)g.beta, g.semantics, 0, 0};
    return plan.tile == 32 ? launch_small<32, 32, 4>(g, p, plan.split) : launch_small<64, 64, 1>(g, p, plan.split);
}

}  // namespace gb
