// gemm_ozaki.cu -- DGEMM from exact integer slices on the tcgen05 tensor cores
// (Ozaki scheme: Ozaki, Ogita, Oishi & Rump, "Error-free transformations of
// matrix multiplication by using fast routines of matrix multiplication and
// its applications", Numer. Algorithms 59, 2012; integer-slice form as in
// Ootomo, Ozaki & Yokota, "DGEMM on integer matrix multiplication unit",
// IJHPCA 2024).  Precision form of the reference's DGEMM
// (dgemm_release_V1.1/device_code/dgemm_kernel.c:1994-3170); it has no
// counterpart in the reference.
//
// Each row i of op(A) is scaled by 2^-e_i (e_i: max_k |a_ik| < 2^e_i) and
// written as s balanced base-256 digits, a_ik = 2^(e_i+1) * sum_t v_ikt 2^-8t
// (+ a remainder of at most half of 2^(e_i+1-8s)), v in [-128, 127] (the leading digit
// in [-128, 128]); columns of op(B) likewise with exponents f_j and digits w.
// Then
//     C_ij ~= 2^(e_i+f_j+2) sum_{t+u <= s+1} 2^-8(t+u) (V_t W_u^T)_ij .
// The digits are integers that BF16 holds exactly (|v| <= 128), so each slice
// product runs on tcgen05.mma kind::f16 with an FP32 accumulator in TMEM, and
// every partial sum of a 1024-long K chunk is an integer of magnitude at most
// 1024*128^2 = 2^24: exact.  Eight bits per slice (balanced digits keep the
// products within 2^14 although they carry a full byte) give FP64-level
// results with 7 slices (28 slice products) and no worse than native FP64
// with 8 (36, the default).  Chunk sums are added exactly in int32 registers (up to 127 chunks),
// and FP64 appears only in the per-pair scaled sum kept in TMEM and in the
// final 2^(e_i+f_j), alpha, beta epilogue.  (sm_103a has no kind::i8 MMA, so
// the INT8 products are carried in BF16; products and sums stay exact.)
//
// Kernels: row/column exponents (integer max of |x| bit patterns), digit
// extraction (integer shifts of the FP64 mantissa; the transpose modes are
// absorbed here, slices are written K-major), and a persistent GEMM: one CTA
// per SM over 128 x 128 C tiles, per tile a loop over slice pairs and K
// chunks; warp 0 issues TMA (one digit tile of V_t and one of W_u per 64-wide
// K block), warp 1 issues the MMAs into one of two FP32 accumulators
// (alternating per chunk), warps 2-9 drain them into int32 registers and the
// FP64 sum in TMEM, and write C.  The FP64 pipe (2 lanes a clock and SM) gets one
// addition an output and diagonal, and alpha and beta: conversions and
// powers of two are made on the integer pipes.
#include <cuda.h>
#include <limits.h>
#include <math.h>
#include <cuda_bf16.h>

#include "gb_common.cuh"
#include "sm100_ptx.cuh"

namespace gb {

bool make_tmap_bf16(CUtensorMap *map, const void *base, uint64_t inner, uint64_t outer, uint64_t row_bytes,
                    uint32_t box_inner, uint32_t box_outer, int swizzle_bytes);

int ozaki_pick_slices(double target_err, int64_t K) {
    // Each input is truncated at 2^(1-8s) of its row (column) maximum, so a
    // product term errs by at most ~2^(2-8s) |a||b|; FP64's own rounding is
    // u = 2^-53 per term, and both grow like sqrt(K) over a dot product.
    // target_err 0 (FP64-equivalent): no worse than native FP64, s = 8
    // (measured on 8192^3 with entries u*2^e, e in [-20, 20]: 8.3e-19 against
    // native 7.5e-18; s = 7 measured 7.56e-18, a little worse than native).
    // A target: the smallest s with 2^(2-8s) sqrt(K) * 4 <= target.
    if (target_err <= 0) return 8;
    double logk = 0;
    for (int64_t k = K; k > 1; k >>= 1) logk += 0.5;
    for (int s = 2; s <= 9; s++)
        if (2.0 - 8.0 * s + logk + 2.0 <= __builtin_log2(target_err)) return s;
    return 9;
}

namespace {

constexpr int BM = 128, BN = 128, BK = 64, STAGES = 7, GROUP_M = 8;
constexpr int KCHUNK_BLOCKS = 16;              // 1024-long exact FP32 chunk
constexpr int MAX_CHUNKS_INT32 = 127;          // chunk sums per int32 accumulator
constexpr int MAXS = 9, MAXPAIRS = MAXS * (MAXS + 1) / 2;
constexpr int TILE_BYTES = BM * BK * 2;        // 16 KB (BM == BN)
constexpr int STAGE_BYTES = 2 * TILE_BYTES;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + 256;
static_assert(SMEM_BYTES <= 232448, "shared memory");
constexpr int EWARPS = 8, NT = 64 + 32 * EWARPS;
constexpr uint32_t TMEM_COLS = 512;            // [0,256): two FP32 accumulators, [256,512): FP64 sum

// ------------------------------------------------------------- exponents
// (exp_of_maxbits: the line exponent from the maximum |x| bit pattern)

// Largest |x| of every row of op(A) and column of op(B), as bits, by atomicMax
// from blocks of 64 lines x 16 `steps` k, both operands in one launch (out
// cleared before).  Element (r, k): trans ? X[k*ldx + r] : X[r*ldx + k].
struct MaxOp {
    const double *X;
    int64_t ldx, rows, tiles_k, tiles;
    int trans;
    unsigned long long *out;
};
struct MaxArgs {
    MaxOp op[2];
    int64_t K;
    int steps;
};

__global__ void __launch_bounds__(256) maxbits64_kernel(const __grid_constant__ MaxArgs a) {
    __shared__ unsigned long long red[16][65];
    int64_t b = blockIdx.x;
    const int w = b < a.op[0].tiles ? 0 : 1;
    if (w) b -= a.op[0].tiles;
    const MaxOp &o = a.op[w];
    const int64_t r0 = (b / o.tiles_k) * 64, kb0 = (b % o.tiles_k) * (16 * a.steps);
    const int t = threadIdx.x, c4 = 4 * (t % 16), rl = t / 16;
    const unsigned long long *X = reinterpret_cast<const unsigned long long *>(o.X);
    auto top = [](unsigned long long m, unsigned long long v) {
        v &= 0x7FFFFFFFFFFFFFFFull;
        return v > m ? v : m;
    };
    unsigned long long m[4] = {0, 0, 0, 0};
    if (!o.trans) {   // 16 threads (a half warp) per row, 16 rows apart
#pragma unroll 4
        for (int sb = 0; sb < a.steps; sb++) {
            const int64_t k = kb0 + 16 * sb + t % 16;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int64_t r = r0 + rl + 16 * i;
                if (r < o.rows && k < a.K) m[i] = top(m[i], __ldg(X + r * o.ldx + k));
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
#pragma unroll
            for (int s = 8; s >= 1; s >>= 1) m[i] = top(m[i], __shfl_xor_sync(0xffffffffu, m[i], s));
            const int64_t r = r0 + rl + 16 * i;
            if ((t & 15) == 0 && r < o.rows) atomicMax(o.out + r, m[i]);
        }
    } else {          // 4 consecutive rows, every 16th k
#pragma unroll 4
        for (int sb = 0; sb < a.steps; sb++) {
            const int64_t k = kb0 + 16 * sb + rl, r = r0 + c4;
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (k < a.K && r + q < o.rows) m[q] = top(m[q], __ldg(X + k * o.ldx + r + q));
        }
#pragma unroll
        for (int q = 0; q < 4; q++) red[rl][c4 + q] = m[q];
        __syncthreads();
        if (t < 64 && r0 + t < o.rows) {
            unsigned long long mm = 0;
#pragma unroll
            for (int j = 0; j < 16; j++) mm = top(mm, red[j][t]);
            atomicMax(o.out + r0 + t, mm);
        }
    }
}

// ---------------------------------------------------------------- digits
// s balanced base-256 digits of x (|x| < 2^e): N = +-round(|x| 2^(8s-1-e))
// (to nearest: the representation error is half a unit of the last digit
// either way, where truncation erred up to a whole unit toward zero),
// |N| <= 2^(8s-1), cut from the least significant digit up (d = N mod 256 in
// [-128, 127], N = (N - d) / 256), so x ~= 2^(e+1) sum_t d_t 2^-8t; the
// leading digit is in [-128, 128].  Written as BF16, most significant first.
__device__ __forceinline__ void digits(double x, int e, int s, unsigned short *out, int64_t stride) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int E = (int)((b >> 52) & 0x7FF);
    unsigned long long m = b & 0xFFFFFFFFFFFFFull;
    int ex;
    if (E == 0) {
        ex = -1074;
    } else {
        m |= 1ull << 52;
        ex = E - 1075;
    }
    const int shift = ex + 8 * s - 1 - e;   // F = m * 2^shift <= 2^(8s-1) <= 2^71, rounded to nearest
    unsigned __int128 F = 0;
    if (m != 0 && shift > -64) {
        if (shift >= 0) {
            F = (unsigned __int128)m << shift;
        } else {   // half a unit of the last digit added first: the dropped part errs both ways
            const int rs = -shift;
            F = (unsigned __int128)((m + (1ull << (rs - 1))) >> rs);
        }
    }
    __int128 N = (b >> 63) ? -(__int128)F : (__int128)F;
    for (int t = s; t >= 1; t--) {
        const int d = (int)(((long long)N + 128) & 255) - 128;
        N = (N - d) >> 8;
        const int v = t == 1 ? d + 256 * (int)N : d;   // the leading digit takes what is left (|v| <= 128)
        const unsigned short h = v ? __bfloat16_as_ushort(__float2bfloat16_rn((float)v)) : 0;
        out[(int64_t)(t - 1) * stride] = h;
    }
}

// The bytes of the digits of four values at once (s <= 8, the same digits as
// above).  N' = N 2^(64-8s) has the digits of N above zeros; adding 128 to
// every byte below the top one carries exactly as cutting the digits one by
// one does, so byte i is digit i plus 128 and what is left above is the
// leading digit.  |N'| <= 2^63: the sum is formed in two words.
struct Digits8 {
    uint32_t lo, hi;   // bytes 0-3, and 4-6: digit + 128
    int top;           // [-128, 128]
};

__device__ __forceinline__ Digits8 digits8(double x, int e, int s) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(x);
    const int E = (int)((b >> 52) & 0x7FF);
    unsigned long long m = b & 0xFFFFFFFFFFFFFull;
    if (E) m |= 1ull << 52;
    const int shift = (E ? E - 1075 : -1074) + 8 * s - 1 - e;
    unsigned long long F = 0;
    if (shift >= 0) F = m << (shift & 63);               // m 2^shift < 2^(8s-1); m == 0 whatever the shift
    else if (shift > -64) F = (m + (1ull << (-shift - 1))) >> -shift;
    F <<= 64 - 8 * s;
    const bool neg = (long long)b < 0;
    const unsigned long long U = neg ? 0ull - F : F;
    const uint32_t lo = (uint32_t)U, hi = (uint32_t)(U >> 32);
    Digits8 d;
    d.lo = lo + 0x80808080u;
    const long long h = (neg ? (long long)(int)hi : (long long)hi) + 0x00808080 + (d.lo < lo ? 1 : 0);
    d.hi = (uint32_t)h;
    d.top = (int)(h >> 24);
    return d;
}

// byte `sel` of w, minus 128, as a float: 2^23 + byte, minus 2^23 + 128 (exact)
__device__ __forceinline__ float digit_float(uint32_t w, int sel) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 | sel)) - 8388736.0f;
}

__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}

// s slices of an operand, rows_p x kp each (K-major, most significant first).
// Source element (r, k): trans ? X[k*ldx + r] : X[r*ldx + k]; padding rows
// and columns are zero.
struct SliceOp {
    const double *X;
    int64_t ldx, rows, rows_p, tiles_k, tiles;
    int trans;
    const unsigned long long *maxbits;   // largest |x| of each line, as bits
    int *e;                              // the lines' exponents, written here for the epilogue
    unsigned short *out;
};
struct SliceArgs {
    SliceOp op[2];
    int64_t K, kp;
    int s;
};

// four consecutive k of row r
__device__ __forceinline__ void store_slices(const SliceArgs &a, const SliceOp &o, int64_t r, int64_t k,
                                             const double (&v)[4]) {
    const int e = r < o.rows ? exp_of_maxbits(o.maxbits[r]) : 0;
    const int64_t stride = o.rows_p * a.kp;
    unsigned short *out = o.out + r * a.kp + k;
    if (a.s > 8) {
        for (int j = 0; j < 4; j++) digits(v[j], e, a.s, out + j, stride);
        return;
    }
    Digits8 d[4];
#pragma unroll
    for (int j = 0; j < 4; j++) d[j] = digits8(v[j], e, a.s);
    *reinterpret_cast<uint2 *>(out) =
        make_uint2(bf16x2((float)d[0].top, (float)d[1].top), bf16x2((float)d[2].top, (float)d[3].top));
#pragma unroll
    for (int t = 1; t < 8; t++) {   // slice t + 1: digit 7 - t
        if (t >= a.s) break;
        const int i = 7 - t;
        float f[4];
#pragma unroll
        for (int j = 0; j < 4; j++) f[j] = digit_float(i < 4 ? d[j].lo : d[j].hi, i & 3);
        *reinterpret_cast<uint2 *>(out + t * stride) = make_uint2(bf16x2(f[0], f[1]), bf16x2(f[2], f[3]));
    }
}

// Both operands in one launch; a CTA cuts a 64 x 64 block of (row, k), a thread
// four consecutive k at a time (8-byte stores, 128 bytes of a slice row per
// half warp).  Bound by HBM: 8 bytes read and 2 s written a value (two
// operands of 8192^2, s = 8: 0.565 ms, 5.7 TB/s; cut one value a thread in
// 128-bit integers: 1.80 ms).
__global__ void __launch_bounds__(256) slice_kernel(const __grid_constant__ SliceArgs a) {
    __shared__ double tile[32][65];
    ptx::pdl_wait();   // the line maxima (returns at once when not launched as a dependent)
    int64_t b = blockIdx.x;
    const int w = b < a.op[0].tiles ? 0 : 1;
    if (w) b -= a.op[0].tiles;
    const SliceOp &o = a.op[w];
    const int64_t r0 = (b / o.tiles_k) * 64, k0 = (b % o.tiles_k) * 64;
    const int t = threadIdx.x, c4 = 4 * (t % 16), rl = t / 16;
    if (k0 == 0 && t < 64 && r0 + t < o.rows_p) o.e[r0 + t] = r0 + t < o.rows ? exp_of_maxbits(o.maxbits[r0 + t]) : 0;
    if (!o.trans) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int64_t r = r0 + rl + 16 * i, k = k0 + c4;
            if (r >= o.rows_p) continue;
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            if (r < o.rows) {
                const double *src = o.X + r * o.ldx + k;
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (k + j < a.K) v[j] = __ldg(src + j);
            }
            store_slices(a, o, r, k, v);
        }
        return;
    }
    // row-contiguous source: two halves of 32 k through tile[k][r]
    const int kw = 4 * (t % 8), rw = t / 8;   // writer: four consecutive k of row rw (+ 32)
#pragma unroll
    for (int h = 0; h < 2; h++) {
        if (h) __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int kl = rl + 16 * i;
            const int64_t k = k0 + 32 * h + kl, r = r0 + c4;
            const double *src = o.X + k * o.ldx + r;
#pragma unroll
            for (int j = 0; j < 4; j++) tile[kl][c4 + j] = k < a.K && r + j < o.rows ? __ldg(src + j) : 0.0;
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int rr = rw + 32 * i;
            if (r0 + rr >= o.rows_p) continue;
            const double v[4] = {tile[kw][rr], tile[kw + 1][rr], tile[kw + 2][rr], tile[kw + 3][rr]};
            store_slices(a, o, r0 + rr, k0 + 32 * h + kw, v);
        }
    }
}

// ------------------------------------------------------------------ gemm
struct OzParams {
    double *C;
    int64_t M, N, ldc;
    double alpha, beta;
    int semantics;
    int num_kb;                    // K blocks of 64
    int chunk_kb;                  // K blocks summed in one accumulator, at most KCHUNK_BLOCKS
    int tiles_m, tiles_n;
    int64_t mp, np;                // padded rows of one V / W slice
    int npairs;
    signed char pt[MAXPAIRS], pu[MAXPAIRS];   // 1-based digit indices per pair
    int s, parts;                  // 128 x 128 form: CTAs that share a tile's chunks
    int *sums;                     // parts > 1: int32 sums, [tile][level + part][128 x 128]
    const int *erow, *fcol;
    int *err;
    // operands, for the outputs that a non-finite row or column reaches
    const double *A, *B;
    int64_t lda, ldb, K;
    int ta, tb;
};

__device__ __forceinline__ void tile_coords(int t, int tiles_m, int tiles_n, int &tm, int &tn) {
    const int per_group = GROUP_M * tiles_n;
    const int g = t / per_group;
    const int first_m = g * GROUP_M;
    const int gm = min(GROUP_M, tiles_m - first_m);
    const int r = t - g * per_group;
    tm = first_m + r % gm;
    tn = r / gm;
}

// C = alpha 2^(e_i + f_j) sum (+ beta ...) for eight consecutive columns of a
// row, their C loads in flight together.
__device__ __forceinline__ void store_outputs(const OzParams &p, int64_t row, int64_t col0, int erow,
                                              const double (&sum)[8]) {
    const bool needc = p.semantics == GB_SEM_ACCUM_SCALAR_BETA || (p.semantics == GB_SEM_BLAS && p.beta != 0.0);
    const bool rowok = row < p.M;
    double *crow = p.C + row * p.ldc;
    double cv[8];
#pragma unroll
    for (int j = 0; j < 8; j++) cv[j] = (rowok && needc && col0 + j < p.N) ? crow[col0 + j] : 0.0;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int64_t col = col0 + j;
        if (!rowok || col >= p.N) continue;
        const int fc = ptx::ld_after_wait(p.fcol + col);
        double v;
        if (fc == kNonFiniteLineExp || erow == kNonFiniteLineExp)
            v = p.alpha * native_dot_cold(p.A, p.lda, p.ta, row, p.B, p.ldb, p.tb, col, p.K);
        else
            v = p.alpha * scale_pow2(scale_pow2(sum[j], erow), fc);
        if (p.semantics == GB_SEM_BLAS) {
            if (p.beta != 0.0) v = fma(p.beta, cv[j], v);
        } else if (p.semantics == GB_SEM_SCALAR_BETA) {
            v = v + p.beta;
        } else {
            v = cv[j] + (v + p.beta);
        }
        crow[col] = v;
    }
}

// First unit (a chunk of a digit pair) of part j of a tile.
__device__ __forceinline__ int part_start(int units, int parts, int j) { return (int)((int64_t)units * j / parts); }

// Diagonal t + u of the pair that unit u belongs to.
__device__ __forceinline__ int unit_level(const OzParams &p, int u, int nchunks) {
    const int q = u / nchunks;
    return q < p.npairs ? p.pt[q] + p.pu[q] : 0;
}

__global__ void __launch_bounds__(NT, 1)
    ozaki_gemm_kernel(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmW, OzParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES * STAGE_BYTES);
    uint64_t *empty = full + STAGES;
    uint64_t *acc_full = empty + STAGES;
    uint64_t *acc_empty = acc_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int items = p.tiles_m * p.tiles_n * p.parts;
    const int nchunks = (p.num_kb + p.chunk_kb - 1) / p.chunk_kb, units = p.npairs * nchunks;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; s++) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            ptx::mbar_init(&acc_full[b], 1);
            ptx::mbar_init(&acc_empty[b], EWARPS);
        }
        ptx::fence_mbar_init();
        ptx::tma_prefetch_desc(&tmV);
        ptx::tma_prefetch_desc(&tmW);
    }
    if (warp == 1) ptx::tmem_alloc(tmem_slot, TMEM_COLS);
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    ptx::pdl_wait();   // the slices (and everything before them on the stream)

    if (warp == 0) {
        if (lane == 0) {   // TMA producer: per tile, per pair, every K block
            int kbg = 0;
            bool go = true;
            for (int it = blockIdx.x; it < items && go; it += gridDim.x) {
                int tm, tn;
                tile_coords(it / p.parts, p.tiles_m, p.tiles_n, tm, tn);
                const int u1 = part_start(units, p.parts, it % p.parts + 1);
                for (int u = part_start(units, p.parts, it % p.parts); u < u1 && go; u++) {
                    const int q = u / nchunks, c = u - q * nchunks;
                    const int vrow = (int)((p.pt[q] - 1) * p.mp + (int64_t)tm * BM);
                    const int wrow = (int)((p.pu[q] - 1) * p.np + (int64_t)tn * BN);
                    const int kb_end = min(p.num_kb, (c + 1) * p.chunk_kb);
                    for (int kb = c * p.chunk_kb; kb < kb_end; kb++, kbg++) {
                        const int s = kbg % STAGES;
                        if (kbg >= STAGES && !ptx::mbar_wait(&empty[s], ((kbg / STAGES) & 1) ^ 1, p.err, 11)) {
                            go = false;
                            break;
                        }
                        uint8_t *st = smem + s * STAGE_BYTES;
                        ptx::mbar_arrive_expect_tx(&full[s], STAGE_BYTES);
                        ptx::tma_load_2d(st, &tmV, &full[s], kb * BK, vrow);
                        ptx::tma_load_2d(st + TILE_BYTES, &tmW, &full[s], kb * BK, wrow);
                    }
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {   // MMA issuer: one accumulator per K chunk of a pair
            constexpr uint32_t idesc = ptx::idesc_bf16_f32(BM, BN);
            int kbg = 0, gi = 0;
            bool go = true;
            for (int it = blockIdx.x; it < items && go; it += gridDim.x) {
                const int u1 = part_start(units, p.parts, it % p.parts + 1);
                for (int u = part_start(units, p.parts, it % p.parts); u < u1 && go; u++, gi++) {
                    const int c = u % nchunks;
                    const int b = gi & 1;
                    if (gi >= 2 && !ptx::mbar_wait(&acc_empty[b], ((gi >> 1) & 1) ^ 1, p.err, 12)) {
                        go = false;
                        break;
                    }
                    ptx::tc_fence_after();
                    const uint32_t acc = tmem + (uint32_t)(b * BN);
                    const int kb_end = min(p.num_kb, (c + 1) * p.chunk_kb);
                    for (int kb = c * p.chunk_kb; kb < kb_end; kb++, kbg++) {
                        const int s = kbg % STAGES;
                        if (!ptx::mbar_wait(&full[s], (kbg / STAGES) & 1, p.err, 13)) {
                            go = false;
                            break;
                        }
                        ptx::tc_fence_after();
                        const uint32_t st = ptx::smem_u32(smem + s * STAGE_BYTES);
                        const uint64_t vd = ptx::sdesc_kmajor_sw128(st);
                        const uint64_t wd = ptx::sdesc_kmajor_sw128(st + TILE_BYTES);
#pragma unroll
                        for (int k = 0; k < BK / 16; k++) {
                            const uint64_t dk = (uint64_t)((k * 32) >> 4);
                            ptx::umma_f16(acc, vd + dk, wd + dk, idesc, (kb != c * p.chunk_kb) || (k != 0));
                        }
                        ptx::umma_commit(&empty[s]);
                    }
                    if (go) ptx::umma_commit(&acc_full[b]);
                }
            }
        }
    } else {   // epilogue warps 2..9: TMEM lane quarter warp % 4, columns 64 * ((warp - 2) / 4) + 0..63
        const int q = warp % 4, half = (warp - 2) / 4;
        const uint32_t lane_base = (uint32_t)(q * 32) << 16;
        const uint32_t tot = tmem + 256u + lane_base + (uint32_t)(half * 128);   // FP64 sums: two columns each
        int gi = 0;
        bool go = true;
        for (int it = blockIdx.x; it < items && go; it += gridDim.x) {
            const int t = it / p.parts, part = it % p.parts;
            bool first_flush = true;
            // exact int32 sums of the chunk sums of consecutive pairs on one diagonal t + u (one
            // scale): one FP64 flush per diagonal, or after MAX_CHUNKS_INT32 chunk sums
            int iacc[64];
#pragma unroll
            for (int j = 0; j < 64; j++) iacc[j] = 0;
            int nacc = 0;
            const int u1 = part_start(units, p.parts, part + 1);
            for (int u = part_start(units, p.parts, part); u < u1; u++, gi++) {
                const int lev = unit_level(p, u, nchunks);
                const bool lev_ends = u == u1 - 1 || unit_level(p, u + 1, nchunks) != lev;
                const int b = gi & 1;
                if (!ptx::mbar_wait(&acc_full[b], (gi >> 1) & 1, p.err, 14)) { go = false; break; }
                ptx::tc_fence_after();
                uint32_t r0[32], r1[32];
                const uint32_t acc = tmem + (uint32_t)(b * BN + half * 64) + lane_base;
                ptx::tmem_ld_32x32b_x32(acc, r0);
                ptx::tmem_ld_32x32b_x32(acc + 32u, r1);
                ptx::tmem_ld_wait();
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&acc_empty[b]);
#pragma unroll
                for (int j = 0; j < 32; j++) {
                    iacc[j] += __float2int_rn(__uint_as_float(r0[j]));
                    iacc[32 + j] += __float2int_rn(__uint_as_float(r1[j]));
                }
                if (p.parts > 1) {   // a level's sum, or this part's share of it, to the join
                    if (!lev_ends) continue;
                    int4 *dst = reinterpret_cast<int4 *>(p.sums) +
                                ((size_t)t * (p.s + p.parts - 1) + (p.s + 1 - lev + part)) * (BM * BN / 4) +
                                (size_t)(half * 4 + q) * 16 * 32 + lane;
#pragma unroll
                    for (int g = 0; g < 16; g++) {
                        __stcg(dst + g * 32, make_int4(iacc[4 * g], iacc[4 * g + 1], iacc[4 * g + 2], iacc[4 * g + 3]));
                        iacc[4 * g] = iacc[4 * g + 1] = iacc[4 * g + 2] = iacc[4 * g + 3] = 0;
                    }
                    continue;
                }
                const bool flush = lev_ends || ++nacc == MAX_CHUNKS_INT32;
                if (flush) {   // FP64 sum += 2^(2-8(t+u)) * iacc (exact scaling, one rounding)
                    nacc = 0;
#pragma unroll
                    for (int cb = 0; cb < 8; cb++) {
                        uint32_t r[16];
                        if (!first_flush) {
                            ptx::tmem_ld_32x32b_x16(tot + (uint32_t)(cb * 16), r);
                            ptx::tmem_ld_wait();
                        }
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            double v = int_pow2(iacc[cb * 8 + j], 2 - 8 * lev);
                            if (!first_flush) v = __dadd_rn(__hiloint2double((int)r[2 * j + 1], (int)r[2 * j]), v);
                            r[2 * j] = (uint32_t)__double2loint(v);
                            r[2 * j + 1] = (uint32_t)__double2hiint(v);
                            iacc[cb * 8 + j] = 0;
                        }
                        ptx::tmem_st_32x32b_x16(tot + (uint32_t)(cb * 16), r);
                    }
                    ptx::tmem_st_wait();
                    first_flush = false;
                }
            }
            if (!go) break;
            if (p.parts > 1) continue;
            // C = alpha * 2^(e_i + f_j) * sum (+ beta ...): this lane's row, 64 columns
            int tm, tn;
            tile_coords(t, p.tiles_m, p.tiles_n, tm, tn);
            const int64_t row = (int64_t)tm * BM + q * 32 + lane;
            const int64_t c0 = (int64_t)tn * BN + half * 64;
            const int erow = row < p.M ? p.erow[row] : 0;
#pragma unroll 1
            for (int cb = 0; cb < 8; cb++) {
                uint32_t r[16];
                ptx::tmem_ld_32x32b_x16(tot + (uint32_t)(cb * 16), r);
                ptx::tmem_ld_wait();
                double sum[8];
#pragma unroll
                for (int j = 0; j < 8; j++) sum[j] = __hiloint2double((int)r[2 * j + 1], (int)r[2 * j]);
                store_outputs(p, row, c0 + cb * 8, erow, sum);
            }
            ptx::tc_fence_before();
        }
    }

    ptx::tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(tmem, TMEM_COLS);
    }
}

// The parts' int32 sums of every level, added up and taken into FP64 level by level:
// the same integers, order and roundings as one CTA's flushes, so the same bits.
// A thread has eight columns of a row.  Bound by the FP64 pipe's additions (2 a clock
// and SM), which here all SMs share.
__global__ void __launch_bounds__(256) ozaki_join_kernel(const __grid_constant__ OzParams p) {
    const int nchunks = (p.num_kb + p.chunk_kb - 1) / p.chunk_kb, units = p.npairs * nchunks;
    const int t = blockIdx.x / 8, e = (blockIdx.x % 8) * 256 + threadIdx.x;   // eight CTAs a tile
    const int lane = e % 32, cb = e / 32 % 8, q = e / 256 % 4, half = e / 1024;
    const int4 *src = reinterpret_cast<const int4 *>(p.sums) + (size_t)t * (p.s + p.parts - 1) * (BM * BN / 4) +
                      (size_t)(half * 4 + q) * 16 * 32 + cb * 2 * 32 + lane;
    ptx::pdl_wait();
    double sum[8];
    int acc[8], level = 0;   // level 0: nothing yet
    bool first = true;
#pragma unroll
    for (int j = 0; j < 8; j++) { acc[j] = 0; sum[j] = 0.0; }
    for (int part = 0; part < p.parts; part++) {
        const int last = unit_level(p, part_start(units, p.parts, part + 1) - 1, nchunks);
        for (int lev = unit_level(p, part_start(units, p.parts, part), nchunks); lev >= last; lev--) {
            const int4 *at = src + (size_t)(p.s + 1 - lev + part) * (BM * BN / 4);
            const int4 x = __ldcg(at), y = __ldcg(at + 32);
            const int v[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
            if (lev != level && level) {
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const double d = int_pow2(acc[j], 2 - 8 * level);
                    sum[j] = first ? d : __dadd_rn(sum[j], d);
                    acc[j] = 0;
                }
                first = false;
            }
            level = lev;
#pragma unroll
            for (int j = 0; j < 8; j++) acc[j] += v[j];
        }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const double d = int_pow2(acc[j], 2 - 8 * level);
        sum[j] = first ? d : __dadd_rn(sum[j], d);
    }
    int tm, tn;
    tile_coords(t, p.tiles_m, p.tiles_n, tm, tn);
    const int64_t row = (int64_t)tm * BM + q * 32 + lane;
    store_outputs(p, row, (int64_t)tn * BN + half * 64 + cb * 8, row < p.M ? p.erow[row] : 0, sum);
}

// ------------------------------------------------------------ wide form
// 128 x 256 C tiles of one CTA (CG = 1), or 256 x 256 of a cluster of two (CG = 2).
// What bounds it is operand bytes into the SM's shared memory, about 64 a clock:
// a k-block of 128 x 256 brings 48 KB for 1024 clocks of MMA at most.  Two CTAs on
// one tile (cta_group::2) hold half of W each, 32 KB a k-block for the same work,
// and six stages fit.  4096^3, s = 8: 4106 us one CTA, 3596 two.  8192^3 runs at the
// power limit and gains little or nothing: 26.7 and 25.5 ms in a loop, 28.25 and
// 28.04 timed side by side, entries of U[-1, 1] (u 2^e: 22.8).  One CTA stays where
// tiles of 256 rows would waste a wave.  The two FP32 accumulators take all 512 TMEM
// columns, so the FP64 running sum of each diagonal flush lives in a per-CTA
// scratch array in global memory (256 KB per CTA, L2-resident, interleaved so that
// a warp's access to one pair of a lane's values is 512 contiguous bytes).  Warps:
// 0 TMA, 1 MMA (of a pair's first CTA), 2-9 epilogue (two per TMEM lane quarter,
// 128 columns each).  The arithmetic is that of ozaki_gemm_kernel (same chunk sums,
// flush order, exact scalings and rounding), so the results are the same bit for bit.
namespace wide {
constexpr int BN_W = 256, EW = 8, NT_W = 64 + 32 * EW;
// per CTA of a unit of CG: 48 KB a stage, or 32 KB with half of W's rows
template <int CG> struct Stg {
    static constexpr int BYTES = TILE_BYTES + BN_W / CG * BK * 2, N = CG == 2 ? 6 : 4, SMEM = N * BYTES + 1024 + 256;
};
static_assert(Stg<1>::SMEM <= 232448 && Stg<2>::SMEM <= 232448, "shared memory");
constexpr size_t SCRATCH_DOUBLES = (size_t)EW * 32 * 128;   // per CTA
}  // namespace wide

template <int CG>
__global__ void __launch_bounds__(wide::NT_W, 1)
    ozaki_wide_kernel(const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmW, OzParams p,
                      double *scratch) {
    using namespace wide;
    constexpr int STAGES_W = Stg<CG>::N, STAGE_W = Stg<CG>::BYTES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + STAGES_W * STAGE_W);
    uint64_t *empty = full + STAGES_W;
    uint64_t *acc_full = empty + STAGES_W;
    uint64_t *acc_empty = acc_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int rank = CG == 2 ? (int)ptx::cluster_ctarank() : 0, unit = blockIdx.x / CG, units = gridDim.x / CG;
    const int num_tiles = p.tiles_m * p.tiles_n;
    const int nchunks = (p.num_kb + p.chunk_kb - 1) / p.chunk_kb;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES_W; s++) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; b++) {
            ptx::mbar_init(&acc_full[b], 1);
            ptx::mbar_init(&acc_empty[b], CG * EW);
        }
        ptx::fence_mbar_init();
        ptx::tma_prefetch_desc(&tmV);
        ptx::tma_prefetch_desc(&tmW);
    }
    if (warp == 1) {
        if (CG == 2) ptx::tmem_alloc_pair(tmem_slot, TMEM_COLS);
        else ptx::tmem_alloc(tmem_slot, TMEM_COLS);
    }
    __syncwarp();
    ptx::tc_fence_before();
    if (CG == 2) ptx::cluster_sync_all();
    else __syncthreads();
    ptx::tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    ptx::pdl_wait();   // the slices (and everything before them on the stream)

    if (warp == 0) {
        if (lane == 0) {   // TMA producer: per tile, per pair, every K block
            int kbg = 0;
            bool go = true;
            for (int t = unit; t < num_tiles && go; t += units) {
                int tm, tn;
                tile_coords(t, p.tiles_m, p.tiles_n, tm, tn);
                for (int q = 0; q < p.npairs && go; q++) {
                    const int vrow = (int)((p.pt[q] - 1) * p.mp + ((int64_t)tm * CG + rank) * BM);
                    const int wrow = (int)((p.pu[q] - 1) * p.np + (int64_t)tn * BN_W + rank * (BN_W / CG));
                    for (int kb = 0; kb < p.num_kb; kb++, kbg++) {
                        const int s = kbg % STAGES_W;
                        if (kbg >= STAGES_W && !ptx::mbar_wait(&empty[s], ((kbg / STAGES_W) & 1) ^ 1, p.err, 11)) {
                            go = false;
                            break;
                        }
                        uint8_t *st = smem + s * STAGE_W;
                        if (rank == 0) ptx::mbar_arrive_expect_tx(&full[s], CG * STAGE_W);
                        if (CG == 2) {   // the first CTA's barrier counts both CTAs' bytes
                            const uint32_t bar = ptx::cluster_addr(&full[s], 0);
                            ptx::tma_load_2d_pair(st, &tmV, bar, kb * BK, vrow);
                            ptx::tma_load_2d_pair(st + TILE_BYTES, &tmW, bar, kb * BK, wrow);
                        } else {
                            ptx::tma_load_2d(st, &tmV, &full[s], kb * BK, vrow);
                            ptx::tma_load_2d(st + TILE_BYTES, &tmW, &full[s], kb * BK, wrow);
                        }
                    }
                }
            }
            if (CG == 2) {   // neither CTA may leave while copies or arrivals of the other are under way
                for (int i = max(0, kbg - STAGES_W); i < kbg && go; i++)
                    go = ptx::mbar_wait(&empty[i % STAGES_W], (i / STAGES_W) & 1, p.err, 15);
                for (int i = 0; i < 64 && !go; i++) __nanosleep(2000);
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {   // MMA issuer: one accumulator per K chunk of a pair
            constexpr uint32_t idesc = ptx::idesc_bf16_f32(CG * BM, BN_W);
            int kbg = 0, gi = 0;
            bool go = true;
            for (int t = unit; t < num_tiles && go; t += units) {
                for (int q = 0; q < p.npairs && go; q++) {
                    for (int c = 0; c < nchunks && go; c++, gi++) {
                        const int b = gi & 1;
                        if (gi >= 2 && !ptx::mbar_wait(&acc_empty[b], ((gi >> 1) & 1) ^ 1, p.err, 12)) {
                            go = false;
                            break;
                        }
                        ptx::tc_fence_after();
                        const uint32_t acc = tmem + (uint32_t)(b * BN_W);
                        const int kb_end = min(p.num_kb, (c + 1) * p.chunk_kb);
                        for (int kb = c * p.chunk_kb; kb < kb_end; kb++, kbg++) {
                            const int s = kbg % STAGES_W;
                            if (!ptx::mbar_wait(&full[s], (kbg / STAGES_W) & 1, p.err, 13)) {
                                go = false;
                                break;
                            }
                            ptx::tc_fence_after();
                            const uint32_t st = ptx::smem_u32(smem + s * STAGE_W);
                            const uint64_t vd = ptx::sdesc_kmajor_sw128(st);
                            const uint64_t wd = ptx::sdesc_kmajor_sw128(st + TILE_BYTES);
#pragma unroll
                            for (int k = 0; k < BK / 16; k++) {
                                const uint64_t dk = (uint64_t)((k * 32) >> 4);
                                const uint32_t add = (kb != c * p.chunk_kb) || (k != 0);
                                if (CG == 2) ptx::umma_f16_pair(acc, vd + dk, wd + dk, idesc, add);
                                else ptx::umma_f16(acc, vd + dk, wd + dk, idesc, add);
                            }
                            if (CG == 2) ptx::umma_commit_pair(&empty[s]);
                            else ptx::umma_commit(&empty[s]);
                        }
                        if (!go) break;
                        if (CG == 2) ptx::umma_commit_pair(&acc_full[b]);
                        else ptx::umma_commit(&acc_full[b]);
                    }
                }
            }
        }
    } else {   // epilogue warps 2..9: TMEM lane quarter warp % 4, columns 128 * ((warp - 2) / 4) + 0..127
        const int w = warp - 2, q = warp % 4;
        // this lane's value pair jp at scr[jp * 32] (formed where used: registers are tight here)
#define OZ_SCR (reinterpret_cast<double2 *>(scratch + (size_t)blockIdx.x * SCRATCH_DOUBLES) + \
                (size_t)(threadIdx.x / 32 - 2) * 64 * 32 + threadIdx.x % 32)
        int gi = 0;
        bool go = true;
        for (int t = unit; t < num_tiles && go; t += units) {
            bool first_flush = true;
            int iacc[128];
#pragma unroll
            for (int j = 0; j < 128; j++) iacc[j] = 0;
            int nacc = 0;
            for (int qq = 0; qq < p.npairs && go; qq++) {
                const int lev = p.pt[qq] + p.pu[qq];
                const bool lev_ends = qq == p.npairs - 1 || p.pt[qq + 1] + p.pu[qq + 1] != lev;
                for (int c = 0; c < nchunks; c++, gi++) {
                    const int b = gi & 1;
                    if (!ptx::mbar_wait(&acc_full[b], (gi >> 1) & 1, p.err, 14)) { go = false; break; }
                    ptx::tc_fence_after();
#pragma unroll
                    for (int cb = 0; cb < 8; cb++) {   // 16 columns per load
                        uint32_t r[16];
                        ptx::tmem_ld_32x32b_x16(tmem + (uint32_t)(b * BN_W) + ((uint32_t)(q * 32) << 16) +
                                                    (uint32_t)((w / 4) * 128 + cb * 16), r);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 16; j++) iacc[cb * 16 + j] += __float2int_rn(__uint_as_float(r[j]));
                    }
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        if (CG == 2) ptx::mbar_arrive_cluster(ptx::cluster_addr(&acc_empty[b], 0));
                        else ptx::mbar_arrive(&acc_empty[b]);
                    }
                    const bool flush = (c == nchunks - 1 && lev_ends) || ++nacc == MAX_CHUNKS_INT32;
                    if (flush) {   // FP64 sum += 2^(2-8(t+u)) * iacc (exact scaling, one rounding)
                        nacc = 0;
                        double2 *scr = OZ_SCR;
                        if (first_flush) {
#pragma unroll
                            for (int jp = 0; jp < 64; jp++)
                                scr[jp * 32] = make_double2(int_pow2(iacc[2 * jp], 2 - 8 * lev),
                                                            int_pow2(iacc[2 * jp + 1], 2 - 8 * lev));
                        } else {
#pragma unroll
                            for (int g8 = 0; g8 < 64; g8 += 4) {   // four pairs' loads in flight
                                double2 v[4];
#pragma unroll
                                for (int i = 0; i < 4; i++) v[i] = __ldcg(scr + (g8 + i) * 32);
#pragma unroll
                                for (int i = 0; i < 4; i++) {
                                    v[i].x = __dadd_rn(v[i].x, int_pow2(iacc[2 * (g8 + i)], 2 - 8 * lev));
                                    v[i].y = __dadd_rn(v[i].y, int_pow2(iacc[2 * (g8 + i) + 1], 2 - 8 * lev));
                                    __stcg(scr + (g8 + i) * 32, v[i]);
                                }
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 128; j++) iacc[j] = 0;
                        first_flush = false;
                    }
                }
            }
            if (!go) break;
            // C = alpha * 2^(e_i + f_j) * sum (+ beta ...): this lane's row, 128 columns
            int tm, tn;
            tile_coords(t, p.tiles_m, p.tiles_n, tm, tn);
            const int64_t row = ((int64_t)tm * CG + rank) * BM + q * 32 + lane;
            const int64_t c0 = (int64_t)tn * BN_W + (w / 4) * 128;
            const int erow = row < p.M ? p.erow[row] : 0;
            const double2 *scr = OZ_SCR;
#pragma unroll 1
            for (int g8 = 0; g8 < 64; g8 += 4) {
                double2 sm[4];
#pragma unroll
                for (int i = 0; i < 4; i++) sm[i] = __ldcg(scr + (g8 + i) * 32);
                const double sum[8] = {sm[0].x, sm[0].y, sm[1].x, sm[1].y, sm[2].x, sm[2].y, sm[3].x, sm[3].y};
                store_outputs(p, row, c0 + 2 * g8, erow, sum);
            }
        }
    }

#undef OZ_SCR
    __syncwarp();
    ptx::tc_fence_before();
    if (CG == 2) ptx::cluster_sync_all();
    else __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        if (CG == 2) ptx::tmem_dealloc_pair(tmem, TMEM_COLS);
        else ptx::tmem_dealloc(tmem, TMEM_COLS);
    }
}

}  // namespace

static gb_status ozaki_one(const GemmArgs &g, int s);

// Slices of both operands take s * (Mp + Np) * Kp * 2 bytes of workspace.
// Past kWorkspaceCap the K range is cut into chunks, each sliced and
// multiplied on its own and accumulated into C (beta applied by the first
// chunk, later chunks add with beta = 1); each chunk gets its own row and
// column exponents.
constexpr double kWorkspaceCap = 4.0 * (1ull << 30);

gb_status launch_dgemm_ozaki(const GemmArgs &g, int slices) {
    if (g.M == 0 || g.N == 0) return ok();
    const int s = slices > 0 ? slices : ozaki_pick_slices(0.0, g.K);
    if (s < 2 || s > MAXS) return set_status(GB_ERR_INVALID_ARG, "ozaki: slices %d not in 2..%d", s, MAXS);
    const double per_k = (double)s * (double)(ceil_div(g.M, BM) * BM + ceil_div(g.N, BN) * BN) * 2.0;
    int64_t kc = (int64_t)(kWorkspaceCap / per_k) / (KCHUNK_BLOCKS * BK) * (KCHUNK_BLOCKS * BK);
    if (kc < KCHUNK_BLOCKS * BK) kc = KCHUNK_BLOCKS * BK;
    if (g.K <= kc) return ozaki_one(g, s);
    for (int64_t k0 = 0; k0 < g.K; k0 += kc) {
        GemmArgs c = g;
        c.K = (g.K - k0) < kc ? (g.K - k0) : kc;
        c.A = (const double *)g.A + (g.ta ? k0 * g.lda : k0);
        c.B = (const double *)g.B + (g.tb ? k0 : k0 * g.ldb);
        if (k0 > 0) {   // later chunks: C += alpha * A_k B_k
            c.semantics = GB_SEM_BLAS;
            c.beta = 1.0;
        }
        gb_status st = ozaki_one(c, s);
        if (st != GB_OK) return st;
    }
    return ok();
}

static gb_status ozaki_one(const GemmArgs &g, int s) {
    // 128 x 128 tiles, 128 x 256 ones of one CTA, or 256 x 256 ones of two, whichever takes the least
    // time: waves of tiles times (a k-block of a digit pair, us, and the part of a level's flush that
    // the next chunk does not hide, which decides for short K).  GB_OZAKI_WIDE=0 keeps 128 x 128.
    // Measured, us:             128 x 128   one CTA   two CTAs
    //   4096x1024x4096              1435      1103       997
    //   3301x4098x3621              3628      2855      2574
    //   4000x1270x2000              1082      1073      1010
    //   384x12800x1024               485       483       710
    //   2305x2305x1300               770       826       805
    //   3900x1293x605                436       515       527
    //   1500x1500x1500               313       441       430
    const char *wv = getenv("GB_OZAKI_WIDE");
    const double pair_kbs = 0.5 * s * (s + 1) * (double)ceil_div(g.K, BK);
    auto cost = [&](int bm, int bn, int ctas, double kb_us, double level_us) {
        const double waves = ceil((double)ceil_div(g.M, bm) * (double)ceil_div(g.N, bn) / (sm_count() / ctas));
        return waves * (pair_kbs * kb_us + s * level_us);
    };
    const double c128 = cost(BM, BN, 1, 0.27, 3.5), c256 = cost(BM, wide::BN_W, 1, 0.41, 8.75);
    const double cpair = g.M > BM ? cost(2 * BM, wide::BN_W, 2, 0.36, 10.6) : 1e30;
    // 128 x 128 tiles that leave SMs idle are shared by several CTAs, each with an equal part of the
    // (pair, chunk) units, and joined by a launch of its own.  The parts' sums take no more than the
    // wide form's scratch and stay exact in 32 bits; a part has 1.5 us for each level that it stores.
    // GB_OZAKI_SPLIT=0 keeps one CTA per tile.  Measured, us (tiles; whole call):
    //   512^3 (16)            150 whole   76 two   48 six   45 nine   56 nineteen
    //   800^3 (49)            198        117      102 three 125 four
    //   1000^3 (64)           228        151
    //   300x300x4000 (9)      722        375      124 nine   99 sixteen  117 thirty-three
    //   1000x1000x4000 (64)   766        440
    const char *ord = getenv("GB_OZAKI_PAIR_ORDER"), *sv = getenv("GB_OZAKI_SPLIT");
    const bool by_w = ord && ord[0] == 'w';
    // even chunks: the accumulator of a short last one would be drained slower than it fills
    const int num_kb = (int)ceil_div(g.K, BK), chunk_kb = (int)ceil_div(num_kb, ceil_div(num_kb, KCHUNK_BLOCKS));
    const int nchunks = (int)ceil_div(num_kb, chunk_kb), units = s * (s + 1) / 2 * nchunks;
    const int64_t tiles128 = ceil_div(g.M, BM) * ceil_div(g.N, BN);
    const double unit_us = 0.27 * chunk_kb;
    double csplit = 1e30;
    int parts = 1;
    for (int n = 2; !by_w && !(sv && sv[0] == '0') && s * nchunks <= MAX_CHUNKS_INT32 && n <= units; n++) {
        if ((double)tiles128 * (s + n - 1) * (BM * BN * 4) > (double)sm_count() * wide::SCRATCH_DOUBLES * 8) break;
        const double waves = ceil((double)tiles128 * n / sm_count());
        const double c = waves * (ceil((double)units / n) * unit_us + (1.0 + (double)s / n) * 1.5) + 6.0 +
                         (double)g.M * (double)g.N * (s + 2) / (2.0 * 1900.0 * sm_count());
        if (c < csplit) { csplit = c; parts = n; }
    }
    if (csplit >= std::min(c128, std::min(c256, cpair))) parts = 1;
    const bool wide = parts == 1 && !(wv && wv[0] == '0') && g.N >= wide::BN_W && std::min(c256, cpair) <= c128;
    const int cg = wide && cpair <= c256 ? 2 : 1;   // CTAs per tile
    const int bn = wide ? wide::BN_W : BN;
    const int64_t kp = ceil_div(g.K, BK) * BK;
    const int64_t mp = ceil_div(g.M, BM) * BM, np = ceil_div(g.N, bn) * bn;
    if (s * mp > 0x7fffffff || s * np > 0x7fffffff || kp > 0x7fffffff)
        return set_status(GB_ERR_UNSUPPORTED, "ozaki: problem too large for 32-bit TMA coordinates");
    const size_t ebytes = ((size_t)(mp + np) * sizeof(int) + 255) / 256 * 256;
    const size_t vbytes = (size_t)s * mp * kp * 2, wbytes = (size_t)s * np * kp * 2;
    const int64_t tiles_total = ceil_div(mp, cg * BM) * (np / bn);
    int grid = cg * (int)std::min<int64_t>(tiles_total * parts, sm_count() / cg);
    const size_t sums = (size_t)tiles_total * (s + parts - 1) * (BM * BN * 4);
    size_t sbytes = wide ? (size_t)grid * wide::SCRATCH_DOUBLES * sizeof(double) : parts > 1 ? sums : 0;
    const size_t mbytes = (size_t)(mp + np) * sizeof(unsigned long long);
    const StatusKeeper before;
    uint8_t *ws = (uint8_t *)workspace(vbytes + wbytes + ebytes + sbytes + mbytes + 4096, g.stream);
    if (!ws && parts > 1) {   // no room for the parts' sums
        before.restore();
        parts = 1;
        sbytes = 0;
        grid = (int)std::min<int64_t>(tiles_total, sm_count());
        ws = (uint8_t *)workspace(vbytes + wbytes + ebytes + mbytes + 4096, g.stream);
    }
    if (!ws) return (gb_status)gb_get_last_status();
    unsigned short *V = (unsigned short *)ws;
    unsigned short *W = (unsigned short *)(ws + vbytes);
    int *erow = (int *)(ws + vbytes + wbytes);
    int *fcol = erow + mp;
    unsigned long long *maxbits = (unsigned long long *)(ws + vbytes + wbytes + ebytes + sbytes);
    double *scratch = wide ? (double *)(ws + vbytes + wbytes + ebytes) : nullptr;   // 256-byte aligned
    int *err = error_word();
    if (!err) return set_status(GB_ERR_OOM, "ozaki: no device error word");

    // line maxima: rows of op(A), columns of op(B)
    const double *A = (const double *)g.A, *B = (const double *)g.B;
    GB_CUDA_TRY(cudaMemsetAsync(maxbits, 0, (size_t)(mp + np) * sizeof(unsigned long long), g.stream));
    // blocks of 256 k, or of 64 while those would leave an SM fewer than eight
    const int steps = (ceil_div(g.M, 64) + ceil_div(g.N, 64)) * ceil_div(g.K, 256) < 8 * sm_count() ? 4 : 16;
    const int64_t mk = ceil_div(g.K, 16 * steps), sk = kp / 64;
    if (ceil_div(mp, 32) > 65535 || ceil_div(np, 32) > 65535)
        return set_status(GB_ERR_UNSUPPORTED, "ozaki: M or N too large");
    MaxArgs ma;
    ma.K = g.K;
    ma.steps = steps;
    ma.op[0] = MaxOp{A, g.lda, g.M, mk, ceil_div(g.M, 64) * mk, g.ta ? 1 : 0, maxbits};
    ma.op[1] = MaxOp{B, g.ldb, g.N, mk, ceil_div(g.N, 64) * mk, g.tb ? 0 : 1, maxbits + mp};
    const int64_t mblocks = ma.op[0].tiles + ma.op[1].tiles;
    // digits: V_t = digits of op(A) rows (M x K), W_u = digits of op(B)^T rows (N x K)
    SliceArgs sa;
    sa.K = g.K; sa.kp = kp; sa.s = s;
    sa.op[0] = SliceOp{A, g.lda, g.M, mp, sk, ceil_div(mp, 64) * sk, g.ta ? 1 : 0, maxbits, erow, V};
    sa.op[1] = SliceOp{B, g.ldb, g.N, np, sk, ceil_div(np, 64) * sk, g.tb ? 0 : 1, maxbits + mp, fcol, W};
    const int64_t sblocks = sa.op[0].tiles + sa.op[1].tiles;
    if (mblocks > 0x7fffffff || sblocks > 0x7fffffff)
        return set_status(GB_ERR_UNSUPPORTED, "ozaki: operands too large");
    maxbits64_kernel<<<(unsigned)mblocks, 256, 0, g.stream>>>(ma);
    GB_LAUNCH_CHECK("ozaki line maxima");
    // the slices and the GEMM are launched as programmatic dependents of the kernel before: it
    // triggers nothing early, so they start when its last CTA has exited, without the gap of a plain
    // launch (captured launches keep plain stream order)
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    GB_CUDA_TRY(cudaStreamIsCapturing(g.stream, &cap));
    cudaLaunchAttribute attrs[2];
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)sblocks);
    cfg.blockDim = dim3(256);
    cfg.stream = g.stream;
    cfg.attrs = attrs;
    cfg.numAttrs = cap == cudaStreamCaptureStatusNone ? 1 : 0;
    GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, slice_kernel, sa));
    GB_LAUNCH_CHECK("ozaki slices");

    CUtensorMap tV, tW;
    if (!make_tmap_bf16(&tV, V, kp, (uint64_t)s * mp, kp * 2, BK, BM, 128) ||
        !make_tmap_bf16(&tW, W, kp, (uint64_t)s * np, kp * 2, BK, bn / cg, 128))
        return set_status(GB_ERR_CUDA, "ozaki: cuTensorMapEncodeTiled failed");

    OzParams p{};
    p.C = (double *)g.C; p.M = g.M; p.N = g.N; p.ldc = g.ldc;
    p.alpha = g.alpha; p.beta = g.beta; p.semantics = g.semantics;
    p.num_kb = (int)(kp / BK);
    p.chunk_kb = chunk_kb;
    p.tiles_m = (int)ceil_div(mp, cg * BM); p.tiles_n = (int)(np / bn);
    p.mp = mp; p.np = np;
    p.erow = erow; p.fcol = fcol; p.err = err;
    p.A = A; p.B = B; p.lda = g.lda; p.ldb = g.ldb; p.K = g.K; p.ta = g.ta ? 1 : 0; p.tb = g.tb ? 1 : 0;
    // slice pairs t + u <= s + 1, diagonal by diagonal, least significant
    // first: the pairs of a diagonal share a scale, so the epilogue sums them
    // exactly in int32 and flushes to FP64 once per diagonal (GB300's FP64
    // pipe made one flush per pair the limiter).  GB_OZAKI_PAIR_ORDER=w
    // groups the pairs by the W digit u instead: the tiles in flight (8 tile
    // rows x 19 tile columns) keep W_u's panels hot in L2, halving the DRAM
    // reads, at one flush per pair.
    int n = 0;
    if (!by_w) {
        for (int d = s + 1; d >= 2; d--)
            for (int t = 1; t <= s; t++) {
                int u = d - t;
                if (u >= 1 && u <= s) { p.pt[n] = (signed char)t; p.pu[n] = (signed char)u; n++; }
            }
    } else {
        for (int u = s; u >= 1; u--)
            for (int t = s + 1 - u; t >= 1; t--) { p.pt[n] = (signed char)t; p.pu[n] = (signed char)u; n++; }
    }
    p.npairs = n;
    p.s = s;
    p.parts = parts;
    p.sums = parts > 1 ? (int *)(ws + vbytes + wbytes + ebytes) : nullptr;

    static std::atomic<uint64_t> attr{0};
    if (device_setup_needed(attr)) {
        GB_CUDA_TRY(cudaFuncSetAttribute(ozaki_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
        GB_CUDA_TRY(cudaFuncSetAttribute(ozaki_wide_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         wide::Stg<1>::SMEM));
        GB_CUDA_TRY(cudaFuncSetAttribute(ozaki_wide_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         wide::Stg<2>::SMEM));
        device_setup_done(attr);
    }
    cfg.gridDim = dim3((unsigned)grid);
    if (wide) {
        cfg.blockDim = dim3(wide::NT_W);
        cfg.dynamicSmemBytes = cg == 2 ? wide::Stg<2>::SMEM : wide::Stg<1>::SMEM;
        if (cg == 2) {
            attrs[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
            attrs[cfg.numAttrs].val.clusterDim.x = 2;
            attrs[cfg.numAttrs].val.clusterDim.y = attrs[cfg.numAttrs].val.clusterDim.z = 1;
            cfg.numAttrs++;
        }
        GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, cg == 2 ? ozaki_wide_kernel<2> : ozaki_wide_kernel<1>, tV, tW, p, scratch));
        GB_LAUNCH_CHECK("ozaki_wide_kernel");
    } else {
        cfg.blockDim = dim3(NT);
        cfg.dynamicSmemBytes = SMEM_BYTES;
        GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, ozaki_gemm_kernel, tV, tW, p));
        GB_LAUNCH_CHECK("ozaki_gemm_kernel");
        if (parts > 1) {
            cfg.gridDim = dim3((unsigned)(8 * tiles_total));
            cfg.blockDim = dim3(256);
            cfg.dynamicSmemBytes = 0;
            GB_CUDA_TRY(cudaLaunchKernelEx(&cfg, ozaki_join_kernel, p));
            GB_LAUNCH_CHECK("ozaki_join_kernel");
        }
    }
    return ok();
}

}  // namespace gb
