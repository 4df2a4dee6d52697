// grouped.cu -- one persistent kernel over many independent GEMMs.
//
// A batch of GEMMs of uneven shapes, transpose modes, semantics and dtypes
// (FP32 and FP64 mixed) is described by a device work list; a persistent
// grid of CTAs pulls C tiles from the whole list through one atomic counter,
// so small problems that could not fill the GPU alone share it.  FP64 tiles,
// 16 x 16 or 32 x 32, come first, those of the longest K before the others:
// the FP64 pipe (2 FMAs a clock and SM) bounds a mixed batch, and it is busy to
// the end only if the last tiles are small.  FP32 tiles, 64 x 64, follow.
// The reference runs one problem at a time per DSP cluster; this is the
// GB300 batching layer of the serving path and has no reference counterpart.
//
// The work list travels host -> device with one copy per batch from a pinned
// staging buffer; each staging slot owns its device list, an event guarding
// reuse, and (optionally) a CUDA graph of [copy, kernel] captured once and
// replayed for every batch that uses the slot.
#include <string.h>

#include <mutex>
#include <vector>

#include "gb_common.cuh"
#include "gb_internal.h"
#include "sm100_ptx.cuh"
#include "tile_stage.cuh"

namespace gb {
namespace {

constexpr int NT = 256, T32 = 64, PER_SM = 2;   // threads of a CTA; side of an FP32 tile; CTAs of an SM

struct alignas(16) GItem {
    const void *A, *B;
    void *C;
    int64_t M, N, K, lda, ldb, ldc;
    double alpha, beta;
    int16_t bits, tile;                 // C tiles of side `tile`
    int32_t ta, tb, semantics;
    int32_t tiles_n, tile_base;
};
static_assert(sizeof(GItem) == 112, "128 bytes cost the host 64 us more for 4096 items");

struct alignas(16) GHeader {
    int32_t count, total_tiles, counter, pad;
};

// One k of a thread's RM x RN outputs, FMAs in k order.
template <int RM, int RN>
__device__ __forceinline__ void fma_step(const double *As, const double *Bs, double (&acc)[RM][RN]) {
    double a[RM], b[RN];
#pragma unroll
    for (int i = 0; i < RM; i++) a[i] = As[i];
#pragma unroll
    for (int j = 0; j < RN; j++) b[j] = Bs[j];
#pragma unroll
    for (int i = 0; i < RM; i++)
#pragma unroll
        for (int j = 0; j < RN; j++) acc[i][j] = fma(a[i], b[j], acc[i][j]);
}
// FP32: two outputs of a row in one packed FMA.
__device__ __forceinline__ void fma_step(const float *As, const float *Bs, float (&acc)[4][4]) {
    const float4 a = *reinterpret_cast<const float4 *>(As), b = *reinterpret_cast<const float4 *>(Bs);
    const float av[4] = {a.x, a.y, a.z, a.w};
    const uint64_t b01 = ptx::f2_pack(b.x, b.y), b23 = ptx::f2_pack(b.z, b.w);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint64_t a2 = ptx::f2_pack(av[i], av[i]);
        ptx::f2_unpack(ptx::f2_fma_rn(a2, b01, ptx::f2_pack(acc[i][0], acc[i][1])), acc[i][0], acc[i][1]);
        ptx::f2_unpack(ptx::f2_fma_rn(a2, b23, ptx::f2_pack(acc[i][2], acc[i][3])), acc[i][2], acc[i][3]);
    }
}

template <typename T, int TILE>
__device__ __forceinline__ void tile_gemm(const GItem &g, int tm, int tn, unsigned char *smem) {
    constexpr int R = TILE / 16;   // 16 x 16 threads, R x R neighbouring outputs each
    Stage<T, TILE, TILE> &s = *reinterpret_cast<Stage<T, TILE, TILE> *>(smem);
    const T *A = (const T *)g.A, *B = (const T *)g.B;
    T *C = (T *)g.C;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int64_t m0 = (int64_t)tm * TILE, n0 = (int64_t)tn * TILE;
    T acc[R][R];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < R; j++) acc[i][j] = T(0);
    StageLoader<T, TILE, TILE, NT> ld;
    const auto same = [](T v) { return v; };
    if (g.K > 0) {
        ld.fetch(A, B, g, m0, n0, 0, g.K);
        ld.store(s, 0, g, same, same);
    }
    __syncthreads();
    int buf = 0;
    for (int64_t k0 = 0; k0 < g.K; k0 += STAGE_K, buf ^= 1) {
        const bool more = k0 + STAGE_K < g.K;
        if (more) ld.fetch(A, B, g, m0, n0, k0 + STAGE_K, g.K);
        if (g.K - k0 >= STAGE_K) {
#pragma unroll
            for (int kk = 0; kk < STAGE_K; kk++) fma_step(&s.A[buf][kk][ty * R], &s.B[buf][kk][tx * R], acc);
        } else {
            for (int kk = 0; kk < (int)(g.K - k0); kk++)
                fma_step(&s.A[buf][kk][ty * R], &s.B[buf][kk][tx * R], acc);
        }
        if (more) ld.store(s, buf ^ 1, g, same, same);
        __syncthreads();
    }
    // every load of C before the first store (one output after the other took a tile of a short
    // K longer than its sums: 268 of 180 x 9 x 11, 37 us a call, 26 so)
    const bool rc = g.semantics == GB_SEM_ACCUM_SCALAR_BETA || (g.semantics == GB_SEM_BLAS && g.beta != 0.0);
    T *const c0 = C + (m0 + ty * R) * g.ldc + n0 + tx * R;
    const int ml = (int)(g.M - m0 - ty * R < R ? g.M - m0 - ty * R : R);
    const int nl = (int)(g.N - n0 - tx * R < R ? g.N - n0 - tx * R : R);
    T c[R][R];
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < R; j++) c[i][j] = rc && i < ml && j < nl ? c0[i * g.ldc + j] : T(0);
#pragma unroll
    for (int i = 0; i < R; i++)
#pragma unroll
        for (int j = 0; j < R; j++) {
            if (i >= ml || j >= nl) continue;
            T v = (T)g.alpha * acc[i][j];
            if (g.semantics == GB_SEM_BLAS) {
                if (g.beta != 0.0) v = fma((T)g.beta, c[i][j], v);
            } else if (g.semantics == GB_SEM_SCALAR_BETA) {
                v = v + (T)g.beta;
            } else {
                v = c[i][j] + (v + (T)g.beta);
            }
            c0[i * g.ldc + j] = v;
        }
}

__global__ void __launch_bounds__(NT, PER_SM) grouped_gemm_kernel(GHeader *hdr, const GItem *items) {
    __shared__ __align__(16) unsigned char smem[sizeof(Stage<double, 32, 32>)];
    static_assert(sizeof(Stage<float, T32, T32>) <= sizeof(smem), "both tile types share the buffer");
    __shared__ int s_tile;
    const int count = hdr->count, total = hdr->total_tiles;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_tile = atomicAdd(&hdr->counter, 1);
        __syncthreads();
        const int t = s_tile;
        if (t >= total) break;
        // item whose tile range holds t (tile_base is increasing)
        int lo = 0, hi = count - 1;
        while (lo < hi) {
            int mid = (lo + hi + 1) / 2;
            if (items[mid].tile_base <= t) lo = mid; else hi = mid - 1;
        }
        const GItem g = items[lo];
        const int local = t - g.tile_base;
        const int tm = local / g.tiles_n, tn = local - tm * g.tiles_n;
        if (g.bits == 32) tile_gemm<float, T32>(g, tm, tn, smem);
        else if (g.tile == 16) tile_gemm<double, 16>(g, tm, tn, smem);
        else tile_gemm<double, 32>(g, tm, tn, smem);
    }
}

// Indices of the GEMMs with outputs, FP64 before FP32, long K before short (to an
// eighth of an octave), equal ones as given; *tiles32: their FP64 tiles of 32 x 32.  By
// counting, and as given where that is the order already: a comparison sort takes the
// host longer than the kernel takes (4096 GEMMs of 16^3: 181 us a call, 80 so, where
// the items' size has the other part).
constexpr int MAX_GROUP = 4096;   // GEMMs of a launch

int work_order(const gb_gemm_desc *d, int n, uint16_t *order, int64_t *tiles32) {
    constexpr int BINS = 2 * 64 * 8;
    uint16_t bin[MAX_GROUP];
    int live = 0, last = 0;
    int64_t t32 = 0;
    bool sorted = true;
    for (int i = 0; i < n; i++) {
        if (d[i].M == 0 || d[i].N == 0) continue;
        if (d[i].dtype_bits == 64) t32 += ceil_div(d[i].M, 32) * ceil_div(d[i].N, 32);
        const unsigned long long K = (unsigned long long)d[i].K + 1;
        const int e = 63 - __builtin_clzll(K), f = (int)((e >= 3 ? K >> (e - 3) : K << (3 - e)) & 7);
        const int b = BINS - 1 - ((d[i].dtype_bits == 64 ? 512 : 0) + 8 * e + f);
        sorted = sorted && b >= last;
        last = b;
        bin[live] = (uint16_t)b;
        order[live++] = (uint16_t)i;
    }
    *tiles32 = t32;
    if (sorted) return live;
    int start[BINS + 1] = {0};
    uint16_t given[MAX_GROUP];
    for (int i = 0; i < live; i++) start[bin[i] + 1]++, given[i] = order[i];
    for (int b = 0; b < BINS; b++) start[b + 1] += start[b];
    for (int i = 0; i < live; i++) order[start[bin[i]]++] = given[i];
    return live;
}

// A pinned staging buffer + device work list + reuse event (+ graph).
struct Slot {
    unsigned char *host = nullptr;
    unsigned char *dev = nullptr;
    size_t cap = 0;
    cudaEvent_t done = nullptr;
    cudaGraphExec_t graph = nullptr;
    cudaStream_t graph_stream = nullptr;
    int graph_grid = 0;
};

}  // namespace

struct GroupRunner {
    std::mutex mu;
    std::vector<Slot> slots;
    size_t next = 0;
    int max_items;

    explicit GroupRunner(int nslots, int max_items_) : slots(nslots), max_items(max_items_) {}

    ~GroupRunner() {
        for (auto &s : slots) {
            if (s.done) cudaEventSynchronize(s.done);
            if (s.graph) cudaGraphExecDestroy(s.graph);
            if (s.done) cudaEventDestroy(s.done);
            if (s.host) cudaFreeHost(s.host);
            if (s.dev) cudaFree(s.dev);
        }
    }

    gb_status prepare(Slot &s) {
        const size_t need = sizeof(GHeader) + sizeof(GItem) * (size_t)max_items;
        if (s.cap >= need) return ok();
        GB_CUDA_TRY(cudaHostAlloc((void **)&s.host, need, cudaHostAllocDefault));
        GB_CUDA_TRY(cudaMalloc((void **)&s.dev, need));
        GB_CUDA_TRY(cudaEventCreateWithFlags(&s.done, cudaEventDisableTiming));
        s.cap = need;
        return ok();
    }

    // Build the work list for n descriptors; launch on `stream`.
    gb_status run(const gb_gemm_desc *d, int n, cudaStream_t stream, bool use_graph) {
        if (n > max_items || n > MAX_GROUP) return set_status(GB_ERR_INVALID_ARG, "gb_gemm_batch: %d GEMMs > capacity %d", n, max_items < MAX_GROUP ? max_items : MAX_GROUP);
        Slot *sp;
        {
            std::lock_guard<std::mutex> lk(mu);
            sp = &slots[next];
            next = (next + 1) % slots.size();
        }
        Slot &s = *sp;
        gb_status st = prepare(s);
        if (st != GB_OK) return st;
        GB_CUDA_TRY(cudaEventSynchronize(s.done));   // previous batch in this slot finished reading it
        GHeader *h = reinterpret_cast<GHeader *>(s.host);
        GItem *it = reinterpret_cast<GItem *>(s.host + sizeof(GHeader));
        // FP64 before FP32, long K first; FP64 in 16 x 16 tiles where 32 x 32 would leave an SM
        // fewer than four.  Mixed batches, us (16 / 32): 1.6 tiles of 32 x 32 an SM 109 / 152, 2.0
        // 104 / 116, 4.1 311 / 301, 5.6 281 / 265 (the FP64 pipe alone: 60, 36, 219, 201; 64 x 64
        // tiles in the order given: 448, 367, 762, 615)
        uint16_t order[MAX_GROUP];
        int count = 0;
        int64_t tiles32 = 0;
        const int live = work_order(d, n, order, &tiles32);
        const int log64 = tiles32 < 4 * (int64_t)sm_count() ? 4 : 5;
        int64_t tiles = 0;
        for (int i = 0; i < live; i++) {
            const gb_gemm_desc &q = d[order[i]];
            GItem &g = it[count++];
            g.A = q.A; g.B = q.B; g.C = q.C;
            g.M = q.M; g.N = q.N; g.K = q.K; g.lda = q.lda; g.ldb = q.ldb; g.ldc = q.ldc;
            g.alpha = q.alpha; g.beta = q.beta;
            g.bits = (int16_t)q.dtype_bits; g.ta = is_trans(q.transA); g.tb = is_trans(q.transB); g.semantics = q.semantics;
            const int log2 = q.dtype_bits == 64 ? log64 : 6;   // shifts: a division is most of an item's work here
            g.tile = (int16_t)(1 << log2);
            g.tiles_n = (int)((q.N + g.tile - 1) >> log2);
            g.tile_base = (int)tiles;
            tiles += ((q.M + g.tile - 1) >> log2) * g.tiles_n;
            if (tiles > 0x7fffffff) return set_status(GB_ERR_UNSUPPORTED, "gb_gemm_batch: too many tiles");
        }
        h->count = count;
        h->total_tiles = (int)tiles;
        h->counter = 0;
        h->pad = 0;
        if (count == 0) return ok();
        const int grid = PER_SM * sm_count();
        if (use_graph) {   // the captured copy takes any batch: the whole list
            const size_t bytes = sizeof(GHeader) + sizeof(GItem) * (size_t)max_items;
            if (!s.graph || s.graph_stream != stream) {
                if (s.graph) cudaGraphExecDestroy(s.graph);
                s.graph = nullptr;
                cudaStream_t cap;
                GB_CUDA_TRY(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
                cudaGraph_t gr;
                cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
                cudaMemcpyAsync(s.dev, s.host, bytes, cudaMemcpyHostToDevice, cap);
                grouped_gemm_kernel<<<grid, NT, 0, cap>>>(reinterpret_cast<GHeader *>(s.dev),
                                                          reinterpret_cast<const GItem *>(s.dev + sizeof(GHeader)));
                cudaError_t e = cudaStreamEndCapture(cap, &gr);
                cudaStreamDestroy(cap);
                if (e != cudaSuccess) return cuda_status(e, "grouped graph capture");
                e = cudaGraphInstantiate(&s.graph, gr, 0);
                cudaGraphDestroy(gr);
                if (e != cudaSuccess) return cuda_status(e, "grouped graph instantiate");
                s.graph_stream = stream;
                s.graph_grid = grid;
            }
            count_launch();
            GB_CUDA_TRY(cudaGraphLaunch(s.graph, stream));
        } else {
            GB_CUDA_TRY(cudaMemcpyAsync(s.dev, s.host, sizeof(GHeader) + sizeof(GItem) * (size_t)count,
                                        cudaMemcpyHostToDevice, stream));
            grouped_gemm_kernel<<<grid, NT, 0, stream>>>(reinterpret_cast<GHeader *>(s.dev),
                                                         reinterpret_cast<const GItem *>(s.dev + sizeof(GHeader)));
            GB_LAUNCH_CHECK("grouped_gemm_kernel");
        }
        GB_CUDA_TRY(cudaEventRecord(s.done, stream));
        return ok();
    }
};

GroupRunner *group_runner_create(int nslots, int max_items) { return new GroupRunner(nslots, max_items); }
void group_runner_destroy(GroupRunner *r) { delete r; }
gb_status group_runner_run(GroupRunner *r, const gb_gemm_desc *d, int n, void *stream, int use_graph) {
    return r->run(d, n, as_stream(stream), use_graph != 0);
}

gb_status check_desc(const gb_gemm_desc &q, int i) {
    GB_CHECK_ARG(q.dtype_bits == 32 || q.dtype_bits == 64, "gemm %d: dtype_bits must be 32 or 64", i);
    GB_CHECK_ARG(is_mode(q.transA) && is_mode(q.transB), "gemm %d: transA/transB must be 'N' or 'T'", i);
    GB_CHECK_ARG(q.M >= 0 && q.N >= 0 && q.K >= 0, "gemm %d: negative dimension", i);
    GB_CHECK_ARG(q.semantics >= 0 && q.semantics <= 2, "gemm %d: unknown semantics", i);
    const int64_t acols = is_trans(q.transA) ? q.M : q.K, bcols = is_trans(q.transB) ? q.K : q.N;
    GB_CHECK_ARG(q.lda >= (acols > 1 ? acols : 1) && q.ldb >= (bcols > 1 ? bcols : 1) && q.ldc >= (q.N > 1 ? q.N : 1),
                 "gemm %d: leading dimension too small", i);
    if (q.M > 0 && q.N > 0) {
        GB_CHECK_ARG(q.C != nullptr, "gemm %d: C is null", i);
        if (q.K > 0) GB_CHECK_ARG(q.A && q.B, "gemm %d: A or B is null", i);
    }
    GB_CHECK_ARG(ceil_div(q.M, 64) * ceil_div(q.N, 64) < (1ll << 30), "gemm %d: too many tiles", i);
    return ok();
}

}  // namespace gb

static std::mutex g_batch_mu;
static gb::GroupRunner *g_batch_runner = nullptr;

extern "C" gb_status gb_gemm_batch(const gb_gemm_desc *descs, int n, void *stream) {
    using namespace gb;
    GB_CHECK_ARG(n >= 0, "gb_gemm_batch: negative count");
    if (n == 0) return ok();
    GB_CHECK_ARG(descs != nullptr, "gb_gemm_batch: null descriptor array");
    GB_CHECK_ARG(n <= 4096, "gb_gemm_batch: at most 4096 GEMMs per batch");
    int64_t tiles = 0;
    for (int i = 0; i < n; i++) {
        gb_status st = check_desc(descs[i], i);
        if (st != GB_OK) return st;
        tiles += ceil_div(descs[i].M, 64) * ceil_div(descs[i].N, 64);
    }
    GB_CHECK_ARG(tiles < (1ll << 30), "gb_gemm_batch: too many tiles in one batch");
    std::lock_guard<std::mutex> lk(g_batch_mu);
    if (!g_batch_runner) g_batch_runner = group_runner_create(4, 4096);
    return group_runner_run(g_batch_runner, descs, n, stream, 0);
}

// Strided batch: GEMM i uses A + i*strideA, B + i*strideB, C + i*strideC
// (strides in elements), all with the same shape, modes and scalars; run as
// grouped launches of up to 4096 GEMMs.
extern "C" gb_status gb_gemm_strided_batched(int dtype_bits, char transA, char transB, int64_t M, int64_t N,
                                             int64_t K, double alpha, const void *A, int64_t lda, int64_t strideA,
                                             const void *B, int64_t ldb, int64_t strideB, double beta, void *C,
                                             int64_t ldc, int64_t strideC, int64_t batch, int semantics,
                                             void *stream) {
    using namespace gb;
    GB_CHECK_ARG(dtype_bits == 32 || dtype_bits == 64, "gb_gemm_strided_batched: dtype_bits must be 32 or 64");
    GB_CHECK_ARG(batch >= 0, "gb_gemm_strided_batched: negative batch count");
    GB_CHECK_ARG(strideA >= 0 && strideB >= 0 && strideC >= 0, "gb_gemm_strided_batched: negative stride");
    if (batch == 0) return ok();
    // distinct C matrices must not overlap: strideC covers one C (rows x ldc)
    GB_CHECK_ARG(batch == 1 || strideC >= (M > 0 ? (M - 1) * ldc + N : 0),
                 "gb_gemm_strided_batched: strideC %lld smaller than one C", (long long)strideC);
    const size_t es = dtype_bits / 8;
    std::vector<gb_gemm_desc> d((size_t)(batch < 4096 ? batch : 4096));
    for (int64_t b0 = 0; b0 < batch; b0 += 4096) {
        const int n = (int)(batch - b0 < 4096 ? batch - b0 : 4096);
        for (int i = 0; i < n; i++) {
            gb_gemm_desc &q = d[i];
            memset(&q, 0, sizeof(q));
            q.dtype_bits = dtype_bits; q.transA = transA; q.transB = transB; q.semantics = semantics;
            q.M = M; q.N = N; q.K = K; q.alpha = alpha; q.beta = beta;
            q.A = (const char *)A + (size_t)(b0 + i) * strideA * es; q.lda = lda;
            q.B = (const char *)B + (size_t)(b0 + i) * strideB * es; q.ldb = ldb;
            q.C = (char *)C + (size_t)(b0 + i) * strideC * es; q.ldc = ldc;
        }
        gb_status st = gb_gemm_batch(d.data(), n, stream);
        if (st != GB_OK) return st;
    }
    return ok();
}
