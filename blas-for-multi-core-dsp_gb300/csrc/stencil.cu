// stencil.cu -- 5-point Jacobi on padded grids, with temporal blocking.
//
// Replaces stencil_vector / stencil_scalar
// (stencil_2d_V1.2/device_code/kernel_stencil.c:1042, :14): one sweep
// B = 0.2 * (N + S + E + W + C) over an (M+2) x (N+2) padded grid with a
// fixed halo.  The reference streams 128x128 (+1 halo) tiles through AM;
// here FP32 grids are streamed through registers several sweeps a pass
// (temporal blocking: HBM traffic per sweep drops to about (1 + halo
// overhead) / t of a read plus a write), FP64 grids one sweep a pass through
// shared-memory tiles.  Every interior point is computed from the same
// neighbours in the same add order as the unblocked recurrence, so results
// are bit-identical for any number of sweeps a pass.
#include <math.h>

#include "gb_common.cuh"
#include "sm100_ptx.cuh"

namespace gb {
namespace {

template <typename T>
struct SOps;
template <>
struct SOps<double> {
    __device__ static double add(double a, double b) { return __dadd_rn(a, b); }
    __device__ static double mul(double a, double b) { return __dmul_rn(a, b); }
    __device__ static double fifth() { return 0.2; }
};
// The three reference add orders (see gbblas.h, gb_stencil_order).
template <typename T, int ORDER>
__device__ __forceinline__ T update(T top, T left, T right, T down, T mid, int64_t row) {
    using O = SOps<T>;
    if (ORDER == GB_STENCIL_HOST)
        return O::mul(O::add(O::add(O::add(O::add(top, left), right), down), mid), O::fifth());
    if (ORDER == GB_STENCIL_SCALAR)
        return O::mul(O::fifth(), O::add(O::add(O::add(O::add(top, mid), down), left), right));
    if ((row & 1) == 0) return O::mul(O::add(right, O::add(O::add(left, top), O::add(mid, down))), O::fifth());
    return O::mul(O::add(right, O::add(O::add(left, down), O::add(top, mid))), O::fifth());
}

constexpr int NT = 256;            // 32 columns x 8 row bands
constexpr int TH = 32, TW = 64;    // output tile

// FP64 form: one CTA per TH x TW output tile, loaded with a halo of one cell
// into shared memory.  Warp w walks row band w of the tile and lane l the
// columns l and l+32; a thread keeps (top, middle, down) of its column in
// registers while it moves down the band, so a point costs three shared loads
// (down, left, right).  Bound by the FP64 pipe, where the halos of several
// sweeps a pass would only be computed twice: one sweep per launch (the FP32
// form's streaming measured slower, 1.38 against 1.64 TB/s at 8192 x 8192).
template <typename T, int ORDER>
__global__ void __launch_bounds__(NT) stencil_tb_kernel(const T *__restrict__ src, T *__restrict__ dst, int64_t M,
                                                        int64_t N) {
    constexpr int H = TH + 2, W = TW + 2, ROWS = TH / (NT / 32);
    __shared__ T tile[H * W];
    const int64_t ld = N + 2;
    const int64_t R0 = (int64_t)blockIdx.y * TH;   // padded coords of the halo's corner
    const int64_t C0 = (int64_t)blockIdx.x * TW;
    const int lane = threadIdx.x % 32, band = threadIdx.x / 32;

    for (int lr = band; lr < H; lr += NT / 32) {
        const int64_t r = R0 + lr;
        if (r > M + 1) break;
        const T *srow = src + r * ld;
        for (int lc = lane; lc < W; lc += 32) {
            const int64_t c = C0 + lc;
            if (c <= N + 1) tile[lr * W + lc] = srow[c];
        }
    }
    __syncthreads();

    const int lr0 = 1 + band * ROWS;
    for (int lc = 1 + lane; lc <= TW; lc += 32) {
        const int64_t c = C0 + lc;
        if (c > N) break;
        const T *cp = tile + lr0 * W + lc;
        T top = cp[-W], mid = cp[0];
        T *out = dst + (R0 + lr0) * ld + c;
        for (int64_t r = R0 + lr0; r < R0 + lr0 + ROWS && r <= M; r++, cp += W, out += ld) {
            const T down = cp[W];
            *out = update<T, ORDER>(top, cp[-1], cp[1], down, mid, r - 1);
            top = mid;
            mid = down;
        }
    }
}

// FP32 form, no shared memory: register-streamed temporal blocking.  A warp
// owns a strip of 128 columns and walks a segment of rows top to bottom, one
// input row per step.  Sweep level l = 1..T keeps the last two rows of level
// l-1 in registers; when level l-1 produces row rho+1, level l computes row
// rho from (rho-1, rho, rho+1).  The level-T rows are written out.  Each
// level loses one column at each strip edge and one row at each segment end,
// so a strip writes 128 - 2T columns and a segment of `seg` rows reads T rows
// of halo above and below.  Every point gets the same neighbours in the same
// add order as one sweep at a time, so results are bit-identical.
//
// Bound by FP32 issue.  Lane l holds columns 2l, 2l+1 and 64+2l, 65+2l as the
// two packed FP32x2 values (2l, 64+2l) and (2l+1, 65+2l): every add and multiply serves two
// points, the neighbours of a pair are again pairs (the other pair of the
// lane, or the adjacent lane's, rotated once around the strip), and the ring
// of two rows per level is indexed by the unrolled row, so no value is moved
// from register to register.  Rows are loaded four steps before they are used
// (a warp alone on a scheduler would otherwise wait for L2 at every row).
// Only warps whose window touches the grid's boundary (EDGE) test for fixed
// cells.
constexpr int RS_W = 128, RS_T = 6, RS_U = 4;   // strip, most sweeps a pass, rows unrolled
constexpr int RS_WARPS = 16;   // warps an SM holds

template <int ORDER, int PAR>
__device__ __forceinline__ uint64_t update2(uint64_t top, uint64_t left, uint64_t right, uint64_t down, uint64_t mid,
                                            uint64_t fifth) {
    using ptx::f2_add;
    if (ORDER == GB_STENCIL_HOST)
        return ptx::f2_mul(f2_add(f2_add(f2_add(f2_add(top, left), right), down), mid), fifth);
    if (ORDER == GB_STENCIL_SCALAR)
        return ptx::f2_mul(fifth, f2_add(f2_add(f2_add(f2_add(top, mid), down), left), right));
    if (PAR == 0) return ptx::f2_mul(f2_add(right, f2_add(f2_add(left, top), f2_add(mid, down))), fifth);
    return ptx::f2_mul(f2_add(right, f2_add(f2_add(left, down), f2_add(top, mid))), fifth);
}

template <int T, int ORDER, bool EDGE>
__device__ __forceinline__ void rs_walk(const float *__restrict__ src, float *__restrict__ dst, int64_t M, int64_t N,
                                        int64_t c0, int64_t out_r0, int64_t out_r1) {
    const int lane = threadIdx.x % 32;
    const int64_t ld = N + 2;
    const int64_t cl = c0 + 2 * lane;   // this lane's columns: cl, cl + 1, cl + 64, cl + 65
    const int lprev = (lane + 31) & 31, lnext = (lane + 1) & 31;
    // bit q + 2h: column cl + q + 64h is inside the padded grid / fixed / written
    unsigned cload = 0, cfix = 0, cstore = 0;
#pragma unroll
    for (int b = 0; b < 4; b++) {
        const int d = (b & 1) + 64 * (b >> 1);
        const int64_t gc = cl + d;
        if (gc >= 0 && gc <= N + 1) cload |= 1u << b;
        if (gc <= 0 || gc >= N + 1) cfix |= 1u << b;
        if (2 * lane + d >= T && 2 * lane + d < RS_W - T && gc >= 1 && gc <= N) cstore |= 1u << b;
    }
    const uint64_t fifth = ptx::f2_pack(0.2f, 0.2f);

    uint64_t R[2][T][2];   // [ring slot][level][pair]
#pragma unroll
    for (int l = 0; l < T; l++)
#pragma unroll
        for (int q = 0; q < 2; q++) R[0][l][q] = R[1][l][q] = 0ull;

    // input rows i0 + k, k = 0 .. kn - 1, up to row out_r1 + T - 1; i0 even so that a row's parity is
    // known when unrolled
    const int64_t i0 = (out_r0 - T) & ~(int64_t)1;
    const int kn = (int)(out_r1 + T - i0), ks = (int)(out_r0 + T - i0);   // row k - T is written from k = ks
    const int klo = (int)(-i0 > -(1 << 30) ? -i0 : -(1 << 30));                                           // rows k < klo lie above the grid
    const int khi = (int)(M + 2 - i0 < kn ? M + 2 - i0 : kn);              // rows k >= khi below it, or unused
    const int kend = (int)(M + 1 - i0 < (1 << 30) ? M + 1 - i0 : 1 << 30); // row M + 1, fixed like row 0
    const float *pin = src + i0 * ld + cl;
    float *pout = dst + (i0 - T) * ld + cl;
    float f[RS_U][4];
    auto load = [&](float (&x)[4], int k) {   // row k, at pin
        if (EDGE) {
            const unsigned m = k >= klo && k < khi ? cload : 0u;
#pragma unroll
            for (int b = 0; b < 4; b++) x[b] = (m >> b) & 1u ? ptx::ld_after_wait(pin + (b & 1) + 64 * (b >> 1)) : 0.f;
        } else if (k < kn) {
#pragma unroll
            for (int b = 0; b < 4; b++) x[b] = ptx::ld_after_wait(pin + (b & 1) + 64 * (b >> 1));
        }
        pin += ld;
    };
#pragma unroll
    for (int u = 0; u < RS_U; u++) {
#pragma unroll
        for (int b = 0; b < 4; b++) f[u][b] = 0.f;
        load(f[u], u);
    }

    for (int kb = 0; kb < kn; kb += RS_U) {
#pragma unroll
        for (int u = 0; u < RS_U; u++) {
            const int k = kb + u;
            uint64_t x[2] = {ptx::f2_pack(f[u][0], f[u][2]), ptx::f2_pack(f[u][1], f[u][3])};
            load(f[u], k + RS_U);
#pragma unroll
            for (int l = 0; l < T; l++) {
                // level l+1, row k - l - 1: top R[slot], middle R[slot ^ 1], down x
                uint64_t(&top)[2] = R[u & 1][l];
                const uint64_t(&mid)[2] = R[(u & 1) ^ 1][l];
                float m0l, m0h, m1l, m1h;
                ptx::f2_unpack(mid[0], m0l, m0h);
                ptx::f2_unpack(mid[1], m1l, m1h);
                // column 2l - 1 from the previous lane's second pair; the high half of lane 0 follows
                // the low half of lane 31
                const float al = __shfl_sync(0xffffffffu, m1l, lprev), ah = __shfl_sync(0xffffffffu, m1h, lprev);
                const uint64_t left0 = ptx::f2_pack(al, lane == 0 ? al : ah);
                const float bl = __shfl_sync(0xffffffffu, m0l, lnext), bh = __shfl_sync(0xffffffffu, m0h, lnext);
                const uint64_t right1 = ptx::f2_pack(lane == 31 ? bh : bl, bh);
                uint64_t v[2];
                if ((u + l) & 1) {   // (row - 1) is odd
                    v[0] = update2<ORDER, 1>(top[0], left0, mid[1], x[0], mid[0], fifth);
                    v[1] = update2<ORDER, 1>(top[1], mid[0], right1, x[1], mid[1], fifth);
                } else {
                    v[0] = update2<ORDER, 0>(top[0], left0, mid[1], x[0], mid[0], fifth);
                    v[1] = update2<ORDER, 0>(top[1], mid[0], right1, x[1], mid[1], fifth);
                }
                if (EDGE) {
                    const int kr = k - l - 1;
                    const unsigned m = kr <= klo || kr >= kend ? 15u : cfix;
                    float w0l, w0h, w1l, w1h;
                    ptx::f2_unpack(v[0], w0l, w0h);
                    ptx::f2_unpack(v[1], w1l, w1h);
                    v[0] = ptx::f2_pack(m & 1u ? m0l : w0l, m & 4u ? m0h : w0h);
                    v[1] = ptx::f2_pack(m & 2u ? m1l : w1l, m & 8u ? m1h : w1h);
                }
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    top[q] = x[q];
                    x[q] = v[q];
                }
            }
            if (k >= ks && k < kn) {   // x: level T, row k - T
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    float lo, hi;
                    ptx::f2_unpack(x[q], lo, hi);
                    if ((cstore >> q) & 1u) pout[q] = lo;
                    if ((cstore >> (q + 2)) & 1u) pout[q + 64] = hi;
                }
            }
            pout += ld;
        }
    }
}

// One warp per CTA, 16 of them resident per SM (128 registers), so that a
// grid that does not fill the GPU spreads evenly.  A pass after the first is
// launched as a programmatic dependent.  No pass triggers its dependent early
// (1000 x 1500, 60 sweeps: 145 us with a trigger, 125 without the attribute,
// 105 with it and the wait alone), so it starts when the last CTA of the pass
// before has exited, and what is saved is the gap of a plain launch.
template <int T, int ORDER>
__global__ void __launch_bounds__(32, T > RS_T ? 12 : RS_WARPS) stencil_rs_kernel(const float *__restrict__ src,
                                                                  float *__restrict__ dst, int64_t M, int64_t N,
                                                                  int strips, int seg) {
    ptx::pdl_wait();   // returns at once when not launched as a dependent
    const int64_t sx = blockIdx.x % (unsigned)strips, sy = blockIdx.x / (unsigned)strips;
    const int64_t c0 = 1 + sx * (RS_W - 2 * T) - T;   // padded column of the strip's first
    const int64_t r0 = 1 + sy * seg;                   // padded rows written: [r0, r1)
    const int64_t r1 = r0 + seg < M + 1 ? r0 + seg : M + 1;
    // every load inside the grid, and no fixed cell among those that the rows and columns written
    // come from: a boundary column may be the window's outermost, whose sweeps only reach the strip's
    // halo, which is not written
    const bool inside = c0 >= 0 && c0 + RS_W <= N + 2 && r0 - T - 1 >= 0 && r1 + T <= M + 2;
    if (inside) rs_walk<T, ORDER, false>(src, dst, M, N, c0, r0, r1);
    else rs_walk<T, ORDER, true>(src, dst, M, N, c0, r0, r1);
}

template <int T>
cudaError_t launch_rs(const float *src, float *dst, int64_t M, int64_t N, int seg, int order, bool dependent,
                      cudaStream_t st) {
    const int64_t strips = ceil_div(N, RS_W - 2 * T);
    cudaLaunchAttribute pdl;
    pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(strips * ceil_div(M, seg)));
    cfg.blockDim = dim3(32);
    cfg.stream = st;
    cfg.attrs = &pdl;
    cfg.numAttrs = dependent ? 1 : 0;
    auto kernel = order == GB_STENCIL_HOST ? stencil_rs_kernel<T, 0>
                  : order == GB_STENCIL_SCALAR ? stencil_rs_kernel<T, 1> : stencil_rs_kernel<T, 2>;
    return cudaLaunchKernelEx(&cfg, kernel, src, dst, M, N, (int)strips, seg);
}

// 9-point stencil with a 3x3 weight window (w[0..2] the row above, w[3..5]
// the row, w[6..8] the row below): r = w0*a_tl, then eight fused
// multiply-adds in window order.  Same register-streaming scheme as the
// 5-point kernel; every row that enters a level's window brings the left /
// right neighbours of its edge columns (two shuffles per row and level).
template <typename E>
struct W9 {
    E w[9];
};

template <typename E>
struct Row4 {
    E v[4];
    E lft, rgt;   // column 4*lane - 1 and 4*lane + 4
};

template <typename E>
__device__ __forceinline__ E fma_rn(E a, E b, E c);
template <>
__device__ __forceinline__ float fma_rn<float>(float a, float b, float c) { return __fmaf_rn(a, b, c); }
template <>
__device__ __forceinline__ double fma_rn<double>(double a, double b, double c) { return __fma_rn(a, b, c); }

template <typename E>
__device__ __forceinline__ E mul_rn(E a, E b);
template <>
__device__ __forceinline__ float mul_rn<float>(float a, float b) { return __fmul_rn(a, b); }
template <>
__device__ __forceinline__ double mul_rn<double>(double a, double b) { return __dmul_rn(a, b); }

constexpr int R9_SEG = 256, R9_NT = 256;

template <typename E, int T>
__global__ void __launch_bounds__(R9_NT) stencil9_rs_kernel(const E *__restrict__ src, E *__restrict__ dst,
                                                            int64_t M, int64_t N, int strips, int segs, W9<E> w) {
    const int lane = threadIdx.x % 32;
    const int64_t wid = (int64_t)blockIdx.x * (R9_NT / 32) + threadIdx.x / 32;
    if (wid >= (int64_t)strips * segs) return;   // whole warp
    const int sx = (int)(wid % strips), sy = (int)(wid / strips);
    const int64_t ld = N + 2;
    const int64_t c0 = 1 + (int64_t)sx * (RS_W - 2 * T) - T;
    const int64_t out_r0 = 1 + (int64_t)sy * R9_SEG;
    const int64_t out_r1 = out_r0 + R9_SEG < M + 1 ? out_r0 + R9_SEG : M + 1;
    const int64_t cl = c0 + 4 * lane;

    bool cfix[4], cload[4], cstore[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        const int64_t gc = cl + q;
        const int lc = 4 * lane + q;
        cfix[q] = gc <= 0 || gc >= N + 1;
        cload[q] = gc >= 0 && gc <= N + 1;
        cstore[q] = lc >= T && lc < RS_W - T && gc >= 1 && gc <= N;
    }

    Row4<E> p2[T], p1[T];
#pragma unroll
    for (int l = 0; l < T; l++) {
#pragma unroll
        for (int q = 0; q < 4; q++) p2[l].v[q] = p1[l].v[q] = E(0);
        p2[l].lft = p2[l].rgt = p1[l].lft = p1[l].rgt = E(0);
    }

    for (int64_t i = out_r0 - T - 1; i < out_r1 + T; i++) {
        Row4<E> x;
#pragma unroll
        for (int q = 0; q < 4; q++) x.v[q] = E(0);
        if (i >= 0 && i <= M + 1) {
            const E *row = src + i * ld + cl;
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (cload[q]) x.v[q] = __ldg(row + q);
        }
#pragma unroll
        for (int l = 0; l < T; l++) {
            x.lft = __shfl_up_sync(0xffffffffu, x.v[3], 1);
            x.rgt = __shfl_down_sync(0xffffffffu, x.v[0], 1);
            const int64_t gr = i - l - 1;
            const bool rfix = gr <= 0 || gr >= M + 1;
            const Row4<E> &t = p2[l], &m = p1[l];
            Row4<E> v;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const E tl = q == 0 ? t.lft : t.v[q - 1], tr = q == 3 ? t.rgt : t.v[q + 1];
                const E ml = q == 0 ? m.lft : m.v[q - 1], mr = q == 3 ? m.rgt : m.v[q + 1];
                const E dl = q == 0 ? x.lft : x.v[q - 1], dr = q == 3 ? x.rgt : x.v[q + 1];
                E r = mul_rn(w.w[0], tl);
                r = fma_rn(w.w[1], t.v[q], r);
                r = fma_rn(w.w[2], tr, r);
                r = fma_rn(w.w[3], ml, r);
                r = fma_rn(w.w[4], m.v[q], r);
                r = fma_rn(w.w[5], mr, r);
                r = fma_rn(w.w[6], dl, r);
                r = fma_rn(w.w[7], x.v[q], r);
                r = fma_rn(w.w[8], dr, r);
                v.v[q] = (rfix || cfix[q]) ? m.v[q] : r;
            }
            p2[l] = p1[l];
            p1[l] = x;
            x = v;
        }
        const int64_t ro = i - T;
        if (ro >= out_r0 && ro < out_r1) {
            E *row = dst + ro * ld + cl;
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (cstore[q]) row[q] = x.v[q];
        }
    }
}

template <typename E, int T>
void launch_rs9(const E *src, E *dst, int64_t M, int64_t N, const W9<E> &w, cudaStream_t st) {
    const int strips = (int)ceil_div(N, RS_W - 2 * T);
    const int segs = (int)ceil_div(M, R9_SEG);
    const unsigned blocks = (unsigned)ceil_div((int64_t)strips * segs, R9_NT / 32);
    stencil9_rs_kernel<E, T><<<blocks, R9_NT, 0, st>>>(src, dst, M, N, strips, segs, w);
}

template <typename E>
gb_status stencil9(int64_t M, int64_t N, E *A, E *B, int iters, const E *w_host, void *stream) {
    GB_CHECK_ARG(M >= 0 && N >= 0, "stencil9: negative size");
    GB_CHECK_ARG(iters >= 0, "stencil9: negative iteration count");
    if (M == 0 || N == 0 || iters == 0) return ok();
    GB_CHECK_ARG(A && B && A != B, "stencil9: A and B must be distinct device buffers");
    GB_CHECK_ARG(w_host != nullptr, "stencil9: null weight window");
    GB_CHECK_ARG((M + R9_SEG - 1) / R9_SEG < (1 << 30), "stencil9: M too large");
    W9<E> w;
    for (int i = 0; i < 9; i++) w.w[i] = w_host[i];
    // FP32: 4 sweeps per pass (the window rows of 4 levels fill the register
    // budget); FP64 is bound by the FP64 pipe: one sweep per pass
    const int tmax = sizeof(E) == 4 ? 4 : 1;
    int L = (int)ceil_div(iters, tmax);
    if ((L & 1) != (iters & 1)) L += 1;   // result in B for odd iters, in A for even
    cudaStream_t st = as_stream(stream);
    int done = 0;
    for (int l = 0; l < L; l++) {
        int t = (iters - done) / (L - l);
        if ((iters - done) % (L - l)) t += 1;
        const E *src = (l % 2 == 0) ? A : B;
        E *dst = (l % 2 == 0) ? B : A;
        switch (t) {
            case 1: launch_rs9<E, 1>(src, dst, M, N, w, st); break;
            case 2: launch_rs9<E, (sizeof(E) == 4 ? 2 : 1)>(src, dst, M, N, w, st); break;
            case 3: launch_rs9<E, (sizeof(E) == 4 ? 3 : 1)>(src, dst, M, N, w, st); break;
            default: launch_rs9<E, (sizeof(E) == 4 ? 4 : 1)>(src, dst, M, N, w, st); break;
        }
        GB_LAUNCH_CHECK("stencil9_rs_kernel");
        done += t;
    }
    return ok();
}

// Sweeps per pass and rows per segment of the FP32 form: the plan of least
// estimated time.  A warp's row of t sweeps costs about (t + 1.2) (46 + 28 k)
// cycles with k warps on its scheduler (measured, t = 6: 89 / 120 / 153 / 191 a sweep at
// k = 1 / 2 / 3 / 4; 146 in waves of four that other waves follow; the 1.2
// are the row's loads and stores), a pass about 6000 cycles besides (launch,
// first rows).  Long segments waste few halo rows, short ones fill the GPU:
// 1000 x 1500, 60 sweeps, measures 112 us in segments of 12 rows (105 against
// 116 in 24 and 120 in 16, before the loads behind the wait were made coherent);
// 8192 x 8192, 48 sweeps, 1115 us in segments of 84, 1136 in 112, 1153 in 64
// (segments of 256 whatever the grid: 2311 and 2620 us).
struct RsPlan {
    int launches, seg;
};
RsPlan rs_plan(int64_t M, int64_t N, int iters, int parity) {
    RsPlan best{1, 8};
    double best_cost = 1e300;
    const double sched = 4.0 * sm_count(), wave = (double)RS_WARPS * sm_count();
    for (int t = RS_T < iters ? RS_T : iters; t >= 1; t--) {
        int launches = (int)ceil_div(iters, t);
        if ((launches & 1) != parity) launches++;   // the result lands in B for odd iters, in A for even
        const int tt = (int)ceil_div(iters, launches);
        const double strips = (double)ceil_div(N, RS_W - 2 * tt);
        for (int seg = 8; seg <= 256; seg += seg < 64 ? 4 : 8) {
            const double warps = strips * (double)ceil_div(M, seg);
            if (warps > 2147483647.0) continue;
            const double full = floor(warps / wave), rest = ceil((warps - full * wave) / sched);
            const double level = full * 122.0 + (rest > 0 ? 46.0 + 28.0 * rest : 0.0);
            const double cost = launches * (6000.0 + level * (tt + 1.2) * (seg + 2 * tt));
            if (cost < best_cost) {
                best_cost = cost;
                best = RsPlan{launches, seg};
            }
        }
        if (t <= RS_T - 2) break;   // fewer sweeps a pass only add passes (and, on large grids, HBM traffic)
    }
    return best;
}

template <typename T>
gb_status stencil(int64_t M, int64_t N, T *A, T *B, int iters, int order, void *stream) {
    GB_CHECK_ARG(M >= 0 && N >= 0, "stencil2d: negative size");
    GB_CHECK_ARG(iters >= 0, "stencil2d: negative iteration count");
    GB_CHECK_ARG(order >= 0 && order <= 2, "stencil2d: order %d not in 0..2", order);
    if (M == 0 || N == 0 || iters == 0) return ok();
    GB_CHECK_ARG(A && B && A != B, "stencil2d: A and B must be distinct device buffers");
    cudaStream_t st = as_stream(stream);
    if (sizeof(T) == 4) {
        GB_CHECK_ARG(ceil_div(M, 64) <= 65535, "stencil2d: M too large");
        // An odd number of sweeps ends with a pass of its own: it leaves in A the sweep that an even
        // spread over an odd number of passes of at most eight does (seven at the end at most), which
        // is what a caller that passes the same A again starts from.  The passes before it are as for
        // an even number.
        int last = 0;
        if (iters & 1) {
            const int passes = (int)ceil_div(iters, 8);
            last = iters / (passes + 1 - (passes & 1));
        }
        const int rest = iters - last;
        RsPlan pl = rs_plan(M, N, rest > 0 ? rest : last, rest > 0 ? 0 : 1);
        if (rest == 0) pl.launches = 0;
        // captured launches keep plain stream order
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        GB_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
        int done = 0;
        for (int l = 0; l < pl.launches + (last > 0); l++) {
            const int t = l < pl.launches ? (int)ceil_div(rest - done, pl.launches - l) : last;   // spread evenly
            const float *src = (const float *)(l % 2 == 0 ? A : B);
            float *dst = (float *)(l % 2 == 0 ? B : A);
            const bool dep = l > 0 && cap == cudaStreamCaptureStatusNone;
            cudaError_t e;
            switch (t) {
                case 1: e = launch_rs<1>(src, dst, M, N, pl.seg, order, dep, st); break;
                case 2: e = launch_rs<2>(src, dst, M, N, pl.seg, order, dep, st); break;
                case 3: e = launch_rs<3>(src, dst, M, N, pl.seg, order, dep, st); break;
                case 4: e = launch_rs<4>(src, dst, M, N, pl.seg, order, dep, st); break;
                case 5: e = launch_rs<5>(src, dst, M, N, pl.seg, order, dep, st); break;
                case 6: e = launch_rs<6>(src, dst, M, N, pl.seg, order, dep, st); break;
                default: e = launch_rs<7>(src, dst, M, N, pl.seg, order, dep, st); break;
            }
            GB_CUDA_TRY(e);
            GB_LAUNCH_CHECK("stencil_rs_kernel");
            done += t;
        }
        return ok();
    }
    dim3 grid((unsigned)ceil_div(N, TW), (unsigned)ceil_div(M, TH));
    GB_CHECK_ARG(grid.y <= 65535u, "stencil2d: M too large");
    for (int l = 0; l < iters; l++) {
        const double *src = (const double *)(l % 2 == 0 ? A : B);
        double *dst = (double *)(l % 2 == 0 ? B : A);
        switch (order) {
            case 0: stencil_tb_kernel<double, 0><<<grid, NT, 0, st>>>(src, dst, M, N); break;
            case 1: stencil_tb_kernel<double, 1><<<grid, NT, 0, st>>>(src, dst, M, N); break;
            default: stencil_tb_kernel<double, 2><<<grid, NT, 0, st>>>(src, dst, M, N); break;
        }
        GB_LAUNCH_CHECK("stencil_tb_kernel");
    }
    return ok();
}

}  // namespace
}  // namespace gb

extern "C" {

gb_status gb_stencil2d_f64(int64_t M, int64_t N, double *A, double *B, int iters, int order, void *stream) {
    return gb::stencil<double>(M, N, A, B, iters, order, stream);
}

gb_status gb_stencil2d_f32(int64_t M, int64_t N, float *A, float *B, int iters, int order, void *stream) {
    return gb::stencil<float>(M, N, A, B, iters, order, stream);
}

gb_status gb_stencil9_f32(int64_t M, int64_t N, float *A, float *B, int iters, const float *w, void *stream) {
    return gb::stencil9<float>(M, N, A, B, iters, w, stream);
}

gb_status gb_stencil9_f64(int64_t M, int64_t N, double *A, double *B, int iters, const double *w, void *stream) {
    return gb::stencil9<double>(M, N, A, B, iters, w, stream);
}

}  // extern "C"
