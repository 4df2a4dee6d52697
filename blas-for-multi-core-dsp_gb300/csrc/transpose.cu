// transpose.cu -- out-of-place matrix transpose, bit-exact copy.
//
// Replaces transpose_float_32x32_dbuf / transpose_16x16_dbuf
// (transpose/device_code/kernel.c:2002, :1167) and the ld-aware
// transpose_A2B (dgemm_release_V1.1/device_code/dgemm_kernel.c:974): B (N x M,
// ldb) = A^T with A M x N (lda).  The reference moves 128x128 tiles through
// on-chip AM with double-buffered DMA and transposes 32x32 / 16x16 blocks in
// registers; here a CTA stages a 64x64 (or 32x32) tile through padded shared memory
// so both the HBM read (rows of A) and the write (rows of B) are coalesced.
// HBM-bound: 2*M*N*sizeof(T) bytes.
#include "gb_common.cuh"

namespace gb {
namespace {

// One TILE x TILE block of A per CTA, ADD: B += A^T.  Bound by HBM: what counts
// is loads in flight, so 256 threads issue all their reads (16 each for 64 x 64)
// before the first goes to shared memory, and four CTAs share an SM (64
// registers; B's 16 values for ADD spill a few, and still 12345 x 6789 FP64 takes
// 324 us with four CTAs, 361 with three and 412 with two).  Against 1024 threads
// with four values each: 12345 x 6789 FP64 199 us, 6.73 TB/s (225), with ADD 324
// (396); FP32 of odd leading dimensions, 20001 x 9001, 255 us (332), with ADD 413
// (630).
constexpr int NT = 256;

// LARGE (FP64 operands that do not fit the L2): A is read and B written as
// streams, 199 us against 212.  Not for FP32, whose tiles share sectors along the
// edges of unaligned rows: 276 us against 255 at 20001 x 9001.
template <typename T, int TILE, bool ADD, bool LARGE>
__global__ void __launch_bounds__(NT, 4) transpose_kernel(const T *__restrict__ A, int64_t lda, T *__restrict__ B,
                                                          int64_t ldb, int64_t M, int64_t N) {
    constexpr int NV = TILE * TILE / NT, STEP = NT / TILE;
    __shared__ T tile[TILE][TILE + 1];
    const int tx = threadIdx.x % TILE, ty = threadIdx.x / TILE;
    const int64_t r0 = (int64_t)blockIdx.y * TILE, c0 = (int64_t)blockIdx.x * TILE;
    // rows r0.. of A, coalesced along its columns c0..
    T v[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int64_t r = r0 + ty + i * STEP, c = c0 + tx;
        v[i] = T(0);
        if (r < M && c < N) v[i] = LARGE ? __ldcs(A + r * lda + c) : A[r * lda + c];
    }
#pragma unroll
    for (int i = 0; i < NV; i++) tile[ty + i * STEP][tx] = v[i];
    __syncthreads();
    // rows c0.. of B, coalesced along its columns r0..
    if (ADD) {
#pragma unroll
        for (int i = 0; i < NV; i++) {
            const int64_t br = c0 + ty + i * STEP, bc = r0 + tx;
            v[i] = br < N && bc < M ? B[br * ldb + bc] : T(0);
        }
    }
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int64_t br = c0 + ty + i * STEP, bc = r0 + tx;
        const T t = tile[tx][ty + i * STEP];
        if (br >= N || bc >= M) continue;
        const T out = ADD ? v[i] + t : t;
        if (LARGE) __stcs(B + br * ldb + bc, out);
        else B[br * ldb + bc] = out;
    }
}

// Blocks of 32 x 32 where 64 x 64 would not fill the SMs twice (700 x 900 FP64:
// 4.0 us against 5.2), and for FP64 ADD within the L2, where eight smaller CTAs per
// SM hide more than longer rows give (2000 x 2000: 12.3 us against 18.8).
template <typename T, bool ADD>
void launch_tiles(int64_t M, int64_t N, const T *A, int64_t lda, T *B, int64_t ldb, cudaStream_t st) {
    const bool large = sizeof(T) == 8 && 2.0 * (double)M * (double)N * sizeof(T) > 128e6;
    const bool small = ceil_div(M, 64) * ceil_div(N, 64) < 2 * (int64_t)sm_count();
    if (small || (ADD && sizeof(T) == 8 && !large && ceil_div(M, 32) <= 65535)) {
        const dim3 grid((unsigned)ceil_div(N, 32), (unsigned)ceil_div(M, 32));
        transpose_kernel<T, 32, ADD, false><<<grid, NT, 0, st>>>(A, lda, B, ldb, M, N);
        return;
    }
    const dim3 grid((unsigned)ceil_div(N, 64), (unsigned)ceil_div(M, 64));
    if (large)
        transpose_kernel<T, 64, ADD, sizeof(T) == 8><<<grid, NT, 0, st>>>(A, lda, B, ldb, M, N);
    else
        transpose_kernel<T, 64, ADD, false><<<grid, NT, 0, st>>>(A, lda, B, ldb, M, N);
}

// FP32: each thread moves 2 x 2 blocks, so the global reads (two rows of A)
// and writes (two rows of B) are 8-byte accesses like the FP64 kernel's.
// Needs lda, ldb even and 8-byte aligned bases; edges fall back to scalars.
constexpr int T2 = 64;
__global__ void __launch_bounds__(256) transpose2x2_kernel(const float *__restrict__ A, int64_t lda,
                                                           float *__restrict__ B, int64_t ldb, int64_t M, int64_t N) {
    __shared__ float tile[T2][T2 + 1];
    const int tx = threadIdx.x % 32, ty = threadIdx.x / 32;   // 32 x 8
    const int64_t r0 = (int64_t)blockIdx.y * T2, c0 = (int64_t)blockIdx.x * T2;
    const bool full = r0 + T2 <= M && c0 + T2 <= N;
    if (full) {   // all eight loads before the first goes to shared memory
        float2 u[T2 / 16], v[T2 / 16];
        const float *src = A + (r0 + ty * 2) * lda + c0 + tx * 2;
#pragma unroll
        for (int i = 0; i < T2 / 16; i++) {
            u[i] = *reinterpret_cast<const float2 *>(src + (int64_t)(16 * i) * lda);
            v[i] = *reinterpret_cast<const float2 *>(src + (int64_t)(16 * i + 1) * lda);
        }
#pragma unroll
        for (int i = 0; i < T2 / 16; i++) {
            const int rr = ty * 2 + 16 * i, cc = tx * 2;
            tile[rr][cc] = u[i].x; tile[rr][cc + 1] = u[i].y;
            tile[rr + 1][cc] = v[i].x; tile[rr + 1][cc + 1] = v[i].y;
        }
    } else {
        for (int i = 0; i < T2; i += 16) {
            const int rr = ty * 2 + i, cc = tx * 2;
            const int64_t r = r0 + rr, c = c0 + cc;
#pragma unroll
            for (int a = 0; a < 2; a++)
#pragma unroll
                for (int b = 0; b < 2; b++)
                    if (r + a < M && c + b < N) tile[rr + a][cc + b] = A[(r + a) * lda + c + b];
        }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < T2; i += 16) {
        const int bc = ty * 2 + i, br = tx * 2;   // B row c0+bc (+1), columns r0+br (+1)
        const int64_t row = c0 + bc, col = r0 + br;
        if (full) {
            *reinterpret_cast<float2 *>(B + row * ldb + col) = make_float2(tile[br][bc], tile[br + 1][bc]);
            *reinterpret_cast<float2 *>(B + (row + 1) * ldb + col) = make_float2(tile[br][bc + 1], tile[br + 1][bc + 1]);
        } else {
#pragma unroll
            for (int a = 0; a < 2; a++)
#pragma unroll
                for (int b = 0; b < 2; b++)
                    if (row + a < N && col + b < M) B[(row + a) * ldb + col + b] = tile[br + b][bc + a];
        }
    }
}

template <typename T>
gb_status transpose_add(int64_t M, int64_t N, const T *A, int64_t lda, T *B, int64_t ldb, void *stream) {
    GB_CHECK_ARG(M >= 0 && N >= 0, "transpose_add: negative size");
    GB_CHECK_ARG(lda >= N || M == 0, "transpose_add: lda (%lld) < N (%lld)", (long long)lda, (long long)N);
    GB_CHECK_ARG(ldb >= M || N == 0, "transpose_add: ldb (%lld) < M (%lld)", (long long)ldb, (long long)M);
    if (M == 0 || N == 0) return ok();
    GB_CHECK_ARG(A && B, "transpose_add: null pointer");
    GB_CHECK_ARG((const void *)A != (const void *)B, "transpose_add: A and B must not be the same buffer");
    GB_CHECK_ARG(ceil_div(M, 64) <= 65535, "transpose_add: M too large");
    launch_tiles<T, true>(M, N, A, lda, B, ldb, as_stream(stream));
    GB_LAUNCH_CHECK("transpose_kernel (add)");
    return ok();
}

template <typename T>
gb_status transpose(int64_t M, int64_t N, const T *A, int64_t lda, T *B, int64_t ldb, void *stream) {
    GB_CHECK_ARG(M >= 0 && N >= 0, "transpose: negative size");
    GB_CHECK_ARG(lda >= N || M == 0, "transpose: lda (%lld) < N (%lld)", (long long)lda, (long long)N);
    GB_CHECK_ARG(ldb >= M || N == 0, "transpose: ldb (%lld) < M (%lld)", (long long)ldb, (long long)M);
    if (M == 0 || N == 0) return ok();
    GB_CHECK_ARG(A && B, "transpose: null pointer");
    GB_CHECK_ARG((const void *)A != (const void *)B, "transpose: in-place transpose is not supported");
    dim3 grid((unsigned)ceil_div(N, T2), (unsigned)ceil_div(M, T2));
    GB_CHECK_ARG(grid.y <= 65535u, "transpose: M too large");
    if (sizeof(T) == 4 && (int64_t)grid.x * grid.y >= 2 * (int64_t)sm_count() && lda % 2 == 0 && ldb % 2 == 0 &&
        (uintptr_t)A % 8 == 0 && (uintptr_t)B % 8 == 0) {
        transpose2x2_kernel<<<grid, 256, 0, as_stream(stream)>>>((const float *)A, lda, (float *)B, ldb, M, N);
        GB_LAUNCH_CHECK("transpose2x2_kernel");
        return ok();
    }
    launch_tiles<T, false>(M, N, A, lda, B, ldb, as_stream(stream));
    GB_LAUNCH_CHECK("transpose_kernel");
    return ok();
}

}  // namespace
}  // namespace gb

extern "C" {

gb_status gb_transpose_f32(int64_t M, int64_t N, const float *A, int64_t lda, float *B, int64_t ldb, void *stream) {
    return gb::transpose<float>(M, N, A, lda, B, ldb, stream);
}

gb_status gb_transpose_f64(int64_t M, int64_t N, const double *A, int64_t lda, double *B, int64_t ldb,
                           void *stream) {
    return gb::transpose<double>(M, N, A, lda, B, ldb, stream);
}

gb_status gb_transpose_add_f32(int64_t M, int64_t N, const float *A, int64_t lda, float *B, int64_t ldb,
                               void *stream) {
    return gb::transpose_add<float>(M, N, A, lda, B, ldb, stream);
}

gb_status gb_transpose_add_f64(int64_t M, int64_t N, const double *A, int64_t lda, double *B, int64_t ldb,
                               void *stream) {
    return gb::transpose_add<double>(M, N, A, lda, B, ldb, stream);
}

}  // extern "C"
