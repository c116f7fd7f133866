// Stage 1: fused bandwidth-calibration pair sums and the pair-distance median.
//
// The reference writes every strict-lower-triangle distance to HBM
// (dmat_comp, ks_bandwidth.cu:181-232) and re-reads the whole buffer once per
// bandwidth (kernelsum_comp x 36, :276-325, :566-572).  Here each 128 x 128
// pair tile is evaluated once into registers and every scale of the sweep is
// accumulated from those registers in the same pass: no distance buffer, one
// read of X (L2-resident), and the work is bound by the exp2 (MUFU) rate.
//
// Tiles cover the lower triangle ti >= tj of the 128-row tile grid; pairs with
// i <= l, or outside [0, N), are masked to D = +inf (exp2(-inf) = 0).  Each
// CTA is persistent over a contiguous range of tiles and keeps one FP64
// accumulator per scale; warp partials are FP32 (<= 2048 terms of <= 1).  The
// per-CTA FP64 partials go to a scratch array and a second kernel reduces them
// in a fixed order, so the result is deterministic.
#include "kevd_internal.cuh"
#include "kevd_pairtile.cuh"

#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

namespace kevd {

constexpr int kCalTile = 128;
constexpr int kCalMaxScales = 256;
constexpr int kCalMaxD = 1024;
constexpr int kFC = 64;            // feature chunk staged in shared memory
constexpr int kFP = kFC + 1;       // its row pitch (bank-conflict padding)

// Tile index t of the lower-triangular tile grid -> (ti, tj), ti >= tj.
__device__ __forceinline__ void tri_tile(int64_t t, int64_t& ti, int64_t& tj) {
    int64_t i = (int64_t)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while (i * (i + 1) / 2 > t) --i;
    while ((i + 1) * (i + 2) / 2 <= t) ++i;
    ti = i;
    tj = t - i * (i + 1) / 2;
}

// Loads features [c0, c0 + w) of rows [r0, r0+128) of X into a [128][kFP]
// shared tile (zeros past N).
__device__ __forceinline__ void load_chunk(const float* __restrict__ X, int64_t N, int d, int64_t r0, int c0,
                                           int w, float* dst) {
    for (int e = threadIdx.x; e < kCalTile * w; e += blockDim.x) {
        const int rr = e / w, kk = e - rr * w;
        const int64_t r = r0 + rr;
        dst[rr * kFP + kk] = (r < N) ? X[r * d + c0 + kk] : 0.f;
    }
}

// Group p of the grid (four per CTA) takes a contiguous range of half tiles, so
// that its i rows stay staged along a row of tiles.
__global__ void __launch_bounds__(kPtThreads, 1)
calibrate_tiles_kernel(const float* __restrict__ X, int64_t N, int d,
                       const float* __restrict__ c2, int n_scales, int64_t n_tiles,
                       double* __restrict__ partial) {
    extern __shared__ __align__(16) float smem[];
    const int g = pt_group();
    float* sm = smem + g * kPtSmemFloats;
    float* cs = smem + kPtGroups * kPtSmemFloats;                 // n_scales
    float* red = cs + kCalMaxScales + g * kPtWarps * kCalMaxScales;   // 4 warps x n_scales
    for (int j = threadIdx.x; j < n_scales; j += kPtThreads) cs[j] = c2[j];
    __syncthreads();
    constexpr int kPer = kCalMaxScales / kPtGroup;
    double acc[kPer] = {};   // thread t of a group owns scales t, t + 128
    const int64_t part = (int64_t)blockIdx.x * kPtGroups + g, parts = (int64_t)gridDim.x * kPtGroups;
    const int64_t u0 = 2 * n_tiles * part / parts, u1 = 2 * n_tiles * (part + 1) / parts;
    PtUnit unit = pt_unit(u0);
    int64_t staged = -1;
    for (int64_t u = u0; u < u1; ++u, pt_next(unit)) {
        f32x2 D[8][4];
        pt_dist(X, N, d, unit, sm, staged, D);
        pt_mask(N, unit, D);
        pt_exp_sums(D, cs, n_scales, red, kCalMaxScales);
        pt_sync();
#pragma unroll
        for (int i = 0; i < kPer; ++i) {
            const int j = pt_tid() + i * kPtGroup;
            if (j < n_scales) {
                double w = 0.0;
#pragma unroll
                for (int q = 0; q < kPtWarps; ++q) w += (double)red[q * kCalMaxScales + j];
                acc[i] += w;
            }
        }
    }
    __syncthreads();
    double* accs = reinterpret_cast<double*>(smem);   // over the tiles
#pragma unroll
    for (int i = 0; i < kPer; ++i) accs[g * kCalMaxScales + pt_tid() + i * kPtGroup] = acc[i];
    __syncthreads();
    for (int j = threadIdx.x; j < n_scales; j += kPtThreads) {
        double w = 0.0;
#pragma unroll
        for (int q = 0; q < kPtGroups; ++q) w += accs[q * kCalMaxScales + j];
        partial[(int64_t)blockIdx.x * n_scales + j] = w;
    }
}

__global__ void reduce_partials_kernel(const double* __restrict__ partial, int n_parts,
                                       int n_scales, double* __restrict__ out) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n_scales) return;
    double s = 0.0;
    for (int p = 0; p < n_parts; ++p) s += partial[(int64_t)p * n_scales + j];
    out[j] = s;
}

// Plain FP64 form of the same pass (FP64 direct distances, FP64 exp): the
// precision reference of the fused FP32 / exp2 kernel above.  Same tiles and
// masking; 64 FP64 distances per thread, so one CTA per SM.
__global__ void __launch_bounds__(256, 1)
calibrate_tiles_fp64_kernel(const float* __restrict__ X, int64_t N, int d, const double* __restrict__ sc,
                            int n_scales, int64_t n_tiles, double* __restrict__ partial) {
    extern __shared__ float sm[];
    float* xi = sm;
    float* xj = sm + kCalTile * kFP;
    double* cs = reinterpret_cast<double*>(xj + kCalTile * kFP + 2);   // 8-byte aligned (2 x 128 x kFP floats is even)
    double* red = cs + kCalMaxScales;                                   // 8 warps x n_scales
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int j = threadIdx.x; j < n_scales; j += blockDim.x) cs[j] = sc[j];
    double acc = 0.0;
    for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        int64_t ti, tj;
        tri_tile(t, ti, tj);
        double D[8][8];
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int b = 0; b < 8; ++b) D[a][b] = 0.0;
        for (int c0 = 0; c0 < d; c0 += kFC) {
            const int w = min(kFC, d - c0);
            __syncthreads();
            load_chunk(X, N, d, ti * kCalTile, c0, w, xi);
            load_chunk(X, N, d, tj * kCalTile, c0, w, xj);
            __syncthreads();
            for (int k = 0; k < w; ++k) {
                double vi[8], vj[8];
#pragma unroll
                for (int a = 0; a < 8; ++a) vi[a] = (double)xi[(ty + 16 * a) * kFP + k];
#pragma unroll
                for (int b = 0; b < 8; ++b) vj[b] = (double)xj[(tx + 16 * b) * kFP + k];
#pragma unroll
                for (int a = 0; a < 8; ++a)
#pragma unroll
                    for (int b = 0; b < 8; ++b) {
                        const double u = vi[a] - vj[b];
                        D[a][b] = fma(u, u, D[a][b]);
                    }
            }
        }
        const int64_t gi0 = ti * kCalTile + ty, gj0 = tj * kCalTile + tx;
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const int64_t gi = gi0 + 16 * a, gj = gj0 + 16 * b;
                if (!(gi < N && gi > gj)) D[a][b] = __longlong_as_double(0x7ff0000000000000ll);  // +inf
            }
        for (int j = 0; j < n_scales; ++j) {
            const double c = -cs[j];
            double s = 0.0;
#pragma unroll
            for (int a = 0; a < 8; ++a)
#pragma unroll
                for (int b = 0; b < 8; ++b) s += exp(D[a][b] * c);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (lane == 0) red[warp * kCalMaxScales + j] = s;
        }
        __syncthreads();
        if (threadIdx.x < n_scales) {
            double w = 0.0;
#pragma unroll
            for (int q = 0; q < 8; ++q) w += red[q * kCalMaxScales + threadIdx.x];
            acc += w;
        }
    }
    if (threadIdx.x < n_scales) partial[(int64_t)blockIdx.x * n_scales + threadIdx.x] = acc;
}

static size_t calib_smem_fp64(int d) {
    (void)d;
    return 2 * kCalTile * (size_t)kFP * sizeof(float) + 16 + 9 * kCalMaxScales * sizeof(double);
}

int run_calibrate_fp64(kevd_ctx* ctx, const float* X, int64_t N, int d, const double* scales, int n_scales,
                       double* sums, cudaStream_t s) {
    if (!X || !scales || !sums || N < 1 || d < 1 || d > kCalMaxD || n_scales < 1 || n_scales > kCalMaxScales)
        return set_error(ctx, KEVD_ERR_ARG, "calibrate_fp64: need N >= 1, 1 <= d <= %d, 1 <= n_scales <= %d",
                         kCalMaxD, kCalMaxScales);
    for (int j = 0; j < n_scales; ++j)
        if (!(scales[j] > 0.0)) return set_error(ctx, KEVD_ERR_ARG, "calibrate_fp64: scales must be positive");
    const int64_t nt = (N + kCalTile - 1) / kCalTile;
    const int64_t n_tiles = nt * (nt + 1) / 2;
    const int grid = (int)std::min<int64_t>(n_tiles, (int64_t)ctx->num_sms);
    int st = KEVD_OK;
    double* sc = arena_get<double>(ctx, "cal64.sc", kCalMaxScales, &st);
    double* partial = arena_get<double>(ctx, "cal64.partial", (size_t)grid * n_scales, &st);
    double* out = arena_get<double>(ctx, "cal64.out", kCalMaxScales, &st);
    if (st != KEVD_OK) return st;
    KEVD_CUDA(ctx, cudaMemcpyAsync(sc, scales, n_scales * sizeof(double), cudaMemcpyHostToDevice, s));
    const size_t smem = calib_smem_fp64(d);
    KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&calibrate_tiles_fp64_kernel), (int)smem));
    {
        ProfScope ps(ctx, "calibrate_tiles_fp64", s);
        calibrate_tiles_fp64_kernel<<<grid, 256, smem, s>>>(X, N, d, sc, n_scales, n_tiles, partial);
        KEVD_LAUNCH(ctx);
    }
    reduce_partials_kernel<<<1, kCalMaxScales, 0, s>>>(partial, grid, n_scales, out);
    KEVD_LAUNCH(ctx);
    KEVD_CUDA(ctx, cudaMemcpyAsync(sums, out, n_scales * sizeof(double), cudaMemcpyDeviceToHost, s));
    KEVD_CUDA(ctx, cudaStreamSynchronize(s));
    return KEVD_OK;
}

static size_t calib_smem(int d) {
    (void)d;
    return ((size_t)kPtGroups * kPtSmemFloats + (1 + kPtGroups * kPtWarps) * kCalMaxScales) * sizeof(float);
}

int run_calibrate(kevd_ctx* ctx, const float* X, int64_t N, int d, const double* scales,
                  int n_scales, double* sums, cudaStream_t s) {
    if (!X || !scales || !sums || N < 1 || d < 1 || d > kCalMaxD || n_scales < 1 ||
        n_scales > kCalMaxScales)
        return set_error(ctx, KEVD_ERR_ARG,
                         "calibrate: need N >= 1, 1 <= d <= %d, 1 <= n_scales <= %d", kCalMaxD,
                         kCalMaxScales);
    const int64_t nt = (N + kCalTile - 1) / kCalTile;
    const int64_t n_tiles = nt * (nt + 1) / 2;
    const int grid = (int)std::min<int64_t>(2 * n_tiles, ctx->num_sms);
    int st = KEVD_OK;
    float* c2 = arena_get<float>(ctx, "cal.c2", kCalMaxScales, &st);
    double* partial = arena_get<double>(ctx, "cal.partial", (size_t)grid * n_scales, &st);
    double* out = arena_get<double>(ctx, "cal.out", kCalMaxScales, &st);
    if (st != KEVD_OK) return st;
    std::vector<float> hc(n_scales);
    for (int j = 0; j < n_scales; ++j) {
        if (!(scales[j] > 0.0))
            return set_error(ctx, KEVD_ERR_ARG, "calibrate: scales must be positive");
        hc[j] = (float)(scales[j] * 1.4426950408889634);  // exp(-x s) = exp2(-x s log2 e)
    }
    KEVD_CUDA(ctx, cudaMemcpyAsync(c2, hc.data(), n_scales * sizeof(float),
                                   cudaMemcpyHostToDevice, s));
    const size_t smem = calib_smem(d);
    KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&calibrate_tiles_kernel), (int)smem));
    {
        ProfScope ps(ctx, "calibrate_tiles", s);
        calibrate_tiles_kernel<<<grid, kPtThreads, smem, s>>>(X, N, d, c2, n_scales, n_tiles, partial);
        KEVD_LAUNCH(ctx);
    }
    reduce_partials_kernel<<<1, kCalMaxScales, 0, s>>>(partial, grid, n_scales, out);
    KEVD_LAUNCH(ctx);
    KEVD_CUDA(ctx, cudaMemcpyAsync(sums, out, n_scales * sizeof(double), cudaMemcpyDeviceToHost, s));
    KEVD_CUDA(ctx, cudaStreamSynchronize(s));
    return KEVD_OK;
}

// ---- calibration without allocation -------------------------------------
// Some callers cannot allocate device memory: processes whose device memory is
// fully reserved by a pool they do not own (another framework's caching
// allocator, a host application that hands the plugin a fixed budget), and
// services that forbid allocation once they have started.  For them the
// pair-sum sweep has a variant whose scratch (per-CTA FP64 partials, the
// device copy of the scales and the reduced sums) lives in fixed file-scope
// device arrays instead of workspace buffers.  Limits: at most kNaMaxScales
// scales per call and a grid of at most kNaGrid CTAs (about 160 KB held by
// every GPU that loads the library, until the process exits).  Each call
// overwrites every entry it reads, so no entry has to start at zero; calls
// share the arrays, so calls that overlap on the GPU (different streams, or
// several host threads) race.
constexpr int kNaMaxScales = 64;
constexpr int kNaGrid = 304;
static __device__ __align__(256) double g_na_partial[kNaGrid * kNaMaxScales];
static __device__ __align__(256) float g_na_scales[kNaMaxScales];
static __device__ __align__(256) double g_na_sums[kNaMaxScales];

struct NoAllocScratch {
    double* partial = nullptr;
    float* scales = nullptr;
    double* sums = nullptr;
};

// The current CUDA context, through the driver entry point (no link against
// the driver library): the module holding the arrays is loaded once per
// context, so their device addresses are only valid in the context that
// resolved them.
using CtxGetCurrentFn = CUresult (*)(CUcontext*);
static CtxGetCurrentFn ctx_get_current() {
    static const CtxGetCurrentFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<CtxGetCurrentFn>(p);
        return (CtxGetCurrentFn) nullptr;
    }();
    return fn;
}

// Device addresses of the arrays, resolved with cudaGetSymbolAddress once per
// device and context, with that device current (a host-side use of the
// symbols is a host stand-in, not a device address).  A caller that switches
// to another context on the same device (cuCtxCreate) gets them resolved
// again for that context.
static int noalloc_scratch(NoAllocScratch* out) {
    constexpr int kMaxDevices = 64;
    static std::mutex mu;
    static CUcontext owner[kMaxDevices] = {};
    static NoAllocScratch table[kMaxDevices];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return KEVD_ERR_CUDA;
    CUcontext cur = nullptr;
    const CtxGetCurrentFn get = ctx_get_current();
    if (get && get(&cur) != CUDA_SUCCESS) cur = nullptr;
    std::lock_guard<std::mutex> lock(mu);
    if (owner[dev] == nullptr || owner[dev] != cur) {
        NoAllocScratch t;
        if (cudaGetSymbolAddress((void**)&t.partial, g_na_partial) != cudaSuccess ||
            cudaGetSymbolAddress((void**)&t.scales, g_na_scales) != cudaSuccess ||
            cudaGetSymbolAddress((void**)&t.sums, g_na_sums) != cudaSuccess)
            return KEVD_ERR_CUDA;
        // the first symbol access made the context current if none was
        if (get && cur == nullptr && get(&cur) != CUDA_SUCCESS) cur = nullptr;
        table[dev] = t;
        owner[dev] = cur;
    }
    *out = table[dev];
    return KEVD_OK;
}

int run_calibrate_noalloc(const float* X, int64_t N, int d, const double* scales, int n_scales, double* sums,
                          cudaStream_t s) {
    if (!X || !scales || !sums || N < 1 || d < 1 || d > kCalMaxD || n_scales < 1 || n_scales > kNaMaxScales)
        return KEVD_ERR_ARG;
    for (int j = 0; j < n_scales; ++j)
        if (!(scales[j] > 0.0)) return KEVD_ERR_ARG;
    // An error left pending by earlier work on this thread would make this
    // call's launch check ambiguous: report it and leave it in place.
    if (cudaPeekAtLastError() != cudaSuccess) return KEVD_ERR_CUDA;
    NoAllocScratch sc;
    if (noalloc_scratch(&sc) != KEVD_OK) {
        cudaGetLastError();   // this call's own failure
        return KEVD_ERR_CUDA;
    }
    float hc[kNaMaxScales];
    for (int j = 0; j < n_scales; ++j) hc[j] = (float)(scales[j] * 1.4426950408889634);
    const int64_t nt = (N + kCalTile - 1) / kCalTile;
    const int64_t n_tiles = nt * (nt + 1) / 2;
    const int grid = (int)std::min<int64_t>(2 * n_tiles, kNaGrid / 2);   // one CTA per SM
    const size_t smem = calib_smem(d);
    // hc lives on this stack frame: the copy is complete (pageable source) or
    // staged before cudaMemcpyAsync returns, and the stream is synchronised
    // below before the frame goes away
    if (cudaMemcpyAsync(sc.scales, hc, n_scales * sizeof(float), cudaMemcpyHostToDevice, s) != cudaSuccess ||
        raise_smem_limit(reinterpret_cast<const void*>(&calibrate_tiles_kernel), (int)smem) !=
            cudaSuccess) {
        cudaGetLastError();
        return KEVD_ERR_CUDA;
    }
    calibrate_tiles_kernel<<<grid, kPtThreads, smem, s>>>(X, N, d, sc.scales, n_scales, n_tiles, sc.partial);
    reduce_partials_kernel<<<1, kCalMaxScales, 0, s>>>(sc.partial, grid, n_scales, sc.sums);
    if (cudaPeekAtLastError() != cudaSuccess ||
        cudaMemcpyAsync(sums, sc.sums, n_scales * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        cudaGetLastError();   // nothing was pending on entry: the error is this call's
        return KEVD_ERR_CUDA;
    }
    return KEVD_OK;
}

// ---- pair-distance median by selection over FP32 bit patterns --------------
//
// Non-negative floats order like their uint32 bit patterns.  The general form is
// a radix selection: three passes histogram bits [31:20], [19:8], [7:0] of the
// distances whose higher bits match the prefix found so far, and the host walks
// each histogram to the bin holding the wanted rank.  Every pass recomputes the
// distances.  Counts are 64-bit: from N = 92,683 on there are more than 2^32 pairs,
// and one bin may hold most of them.  A CTA counts in 32 bits and adds its counts to
// the 64-bit ones at its end, so a launch gives it at most kHistUnits half tiles.
//
// Over all pairs the distances are nearly the whole cost, so one pass has to do
// (run_bracketed_median): the distances of random pairs give a bracket that holds
// the median and 1 to 2 % of all pairs; the pass counts the distances below it and
// collects those inside, and the exact rank is selected among these.  A bracket
// that misses (by the exact counts) leaves the call to the radix selection, and so
// does one that by the sample holds more pairs than fit the buffer (many ties),
// before the pass.  N = 20,000, d = 64: 1.25 ms, in three passes 3.08 ms.

constexpr int kHistBins = 4096;
using HistCount = unsigned long long;
constexpr int64_t kHistUnits = 1 << 18;   // half tiles of 8,192 pairs per CTA and launch: 2^31 counts

__device__ __forceinline__ void hist_add(unsigned* h, float D, int shift, unsigned mask,
                                         unsigned prefix, int hi_shift) {
    const unsigned u = __float_as_uint(D);
    const bool match = (hi_shift >= 32) ? true : ((u >> hi_shift) == prefix);
    if (match) atomicAdd(&h[(u >> shift) & mask], 1u);
}

__global__ void __launch_bounds__(kPtThreads, 1)
median_tiles_kernel(const float* __restrict__ X, int64_t N, int d, int64_t unit0, int64_t n_units, int shift,
                    unsigned mask, unsigned prefix, int hi_shift, HistCount* __restrict__ hist) {
    extern __shared__ __align__(16) float smem[];
    float* sm = smem + pt_group() * kPtSmemFloats;
    unsigned* h = reinterpret_cast<unsigned*>(smem + kPtGroups * kPtSmemFloats);
    for (int e = threadIdx.x; e < kHistBins; e += blockDim.x) h[e] = 0u;
    __syncthreads();
    const int64_t part = (int64_t)blockIdx.x * kPtGroups + pt_group(), parts = (int64_t)gridDim.x * kPtGroups;
    const int64_t u0 = unit0 + n_units * part / parts, u1 = unit0 + n_units * (part + 1) / parts;
    PtUnit unit = pt_unit(u0);
    int64_t staged = -1;
    for (int64_t u = u0; u < u1; ++u, pt_next(unit)) {
        f32x2 D[8][4];
        pt_dist(X, N, d, unit, sm, staged, D);
        const int64_t gi0 = unit.ti * kPtTile + 8 * unit.h + (pt_tid() >> 4);
        const int64_t gj0 = unit.tj * kPtTile + (pt_tid() & 15);
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int p = 0; p < 4; ++p) {
                const int64_t gi = gi0 + 16 * a, gj = gj0 + 32 * p;
                float x, y;
                unpack2(D[a][p], x, y);
                if (gi < N && gi > gj) hist_add(h, x, shift, mask, prefix, hi_shift);
                if (gi < N && gi > gj + 16) hist_add(h, y, shift, mask, prefix, hi_shift);
            }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kHistBins; e += blockDim.x)
        if (h[e]) atomicAdd(&hist[e], (HistCount)h[e]);
}

__global__ void median_pairs_kernel(const float* __restrict__ X, int d,
                                    const int64_t* __restrict__ pi, const int64_t* __restrict__ pl,
                                    int64_t n_pairs, int shift, unsigned mask, unsigned prefix,
                                    int hi_shift, HistCount* __restrict__ hist) {
    __shared__ unsigned h[kHistBins];
    for (int e = threadIdx.x; e < kHistBins; e += blockDim.x) h[e] = 0u;
    __syncthreads();
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n_pairs;
         p += (int64_t)gridDim.x * blockDim.x) {
        const float* a = X + pi[p] * d;
        const float* b = X + pl[p] * d;
        float D = 0.f;
        for (int k = 0; k < d; ++k) {
            const float t = a[k] - b[k];
            D = fmaf(t, t, D);
        }
        hist_add(h, D, shift, mask, prefix, hi_shift);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kHistBins; e += blockDim.x)
        if (h[e]) atomicAdd(&hist[e], (HistCount)h[e]);
}

// Distances of n pseudo-random pairs (i, j), i != j.
__global__ void __launch_bounds__(256) median_sample_kernel(const float* __restrict__ X, int64_t N, int d, int n,
                                                            unsigned* __restrict__ bits) {
    const int t = blockIdx.x * 256 + threadIdx.x;
    if (t >= n) return;
    uint64_t z = ((uint64_t)t + 1) * 0x9E3779B97F4A7C15ull;   // splitmix64
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    const int64_t i = (int64_t)((z & 0xffffffffu) * (uint64_t)N >> 32);
    int64_t j = (int64_t)((z >> 32) * (uint64_t)N >> 32);
    if (j == i) j = i + 1 < N ? i + 1 : 0;
    float D = 0.f;
    for (int k = 0; k < d; ++k) {
        const float u = X[i * d + k] - X[j * d + k];
        D = fmaf(u, u, D);
    }
    bits[t] = __float_as_uint(D);
}

// br[0], br[1]: the bits of the sample's order statistics r0 and r1 rounded down
// and up to multiples of 2^10 (two levels of 11 bits); br[2]: how many of the sample
// lie in [br[0], br[1]).  One CTA.
__global__ void __launch_bounds__(1024) median_bracket_kernel(const unsigned* __restrict__ bits, int n, int r0, int r1,
                                                              unsigned* __restrict__ br) {
    __shared__ unsigned h[2][2048];
    __shared__ unsigned pre[2];
    __shared__ int rank[2];
    __shared__ unsigned b01[2], inside;
    if (threadIdx.x < 2) rank[threadIdx.x] = threadIdx.x ? r1 : r0;
    if (threadIdx.x == 0) inside = 0u;
    for (int level = 0; level < 2; ++level) {
        for (int e = threadIdx.x; e < 2 * 2048; e += 1024) h[e >> 11][e & 2047] = 0u;
        __syncthreads();
        for (int t = threadIdx.x; t < n; t += 1024) {
            const unsigned b = bits[t];
            if (level == 0) {
                atomicAdd(&h[0][b >> 21], 1u);
            } else {
#pragma unroll
                for (int q = 0; q < 2; ++q)
                    if (b >> 21 == pre[q]) atomicAdd(&h[q][(b >> 10) & 2047], 1u);
            }
        }
        __syncthreads();
        if (threadIdx.x < 2) {
            const int q = threadIdx.x;
            const unsigned* hq = h[level ? q : 0];
            int r = rank[q], bin = 0;
            while (bin < 2047 && r >= (int)hq[bin]) r -= (int)hq[bin++];
            rank[q] = r;
            if (level == 0) pre[q] = (unsigned)bin;
            else br[q] = b01[q] = (((pre[q] << 11) | (unsigned)bin) + (unsigned)q) << 10;
        }
        __syncthreads();
    }
    unsigned in = 0u;
    for (int t = threadIdx.x; t < n; t += 1024) in += bits[t] >= b01[0] && bits[t] < b01[1];
    atomicAdd(&inside, in);
    __syncthreads();
    if (threadIdx.x == 0) br[2] = inside;
}

// One pass over all pairs: cnt[0] += distances below br[0], and those in
// [br[0], br[1]) appended to buf (in any order; cnt[1] counts them, also past cap).
// Nothing at all where more than max_inside of the sample lie in the bracket.
__global__ void __launch_bounds__(kPtThreads, 1)
median_collect_kernel(const float* __restrict__ X, int64_t N, int d, int64_t n_tiles, const unsigned* __restrict__ br,
                      unsigned max_inside, float* __restrict__ buf, unsigned long long cap,
                      unsigned long long* __restrict__ cnt) {
    if (br[2] > max_inside) return;
    extern __shared__ __align__(16) float smem[];
    float* sm = smem + pt_group() * kPtSmemFloats;
    const int lane = threadIdx.x & 31;
    const float lo = __uint_as_float(br[0]), hi = __uint_as_float(br[1]);
    const int64_t part = (int64_t)blockIdx.x * kPtGroups + pt_group(), parts = (int64_t)gridDim.x * kPtGroups;
    const int64_t u0 = 2 * n_tiles * part / parts, u1 = 2 * n_tiles * (part + 1) / parts;
    PtUnit unit = pt_unit(u0);
    int64_t staged = -1;
    unsigned long long below = 0;
    for (int64_t u = u0; u < u1; ++u, pt_next(unit)) {
        f32x2 D[8][4];
        pt_dist(X, N, d, unit, sm, staged, D);
        pt_mask(N, unit, D);   // pairs that do not count are +inf: above the bracket
        unsigned nb = 0, in[2] = {0u, 0u};
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            float x, y;
            unpack2(D[q >> 2][q & 3], x, y);
            nb += (x < lo) + (y < lo);
            if (x >= lo && x < hi) in[q >> 4] |= 1u << (2 * (q & 15));
            if (y >= lo && y < hi) in[q >> 4] |= 2u << (2 * (q & 15));
        }
        below += nb;
        const unsigned mine = __popc(in[0]) + __popc(in[1]);
        unsigned pre = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned v = __shfl_up_sync(0xffffffffu, pre, o);
            if (lane >= o) pre += v;
        }
        const unsigned total = __shfl_sync(0xffffffffu, pre, 31);
        if (total == 0) continue;
        unsigned long long at = 0;
        if (lane == 31) at = atomicAdd(cnt + 1, (unsigned long long)total);
        at = __shfl_sync(0xffffffffu, at, 31) + pre - mine;
        if (mine == 0) continue;
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            float x, y;
            unpack2(D[q >> 2][q & 3], x, y);
            if (in[q >> 4] >> (2 * (q & 15)) & 1u) {
                if (at < cap) buf[at] = x;
                ++at;
            }
            if (in[q >> 4] >> (2 * (q & 15)) & 2u) {
                if (at < cap) buf[at] = y;
                ++at;
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) below += __shfl_xor_sync(0xffffffffu, below, o);
    if (lane == 0 && below) atomicAdd(cnt, below);
}

// Histogram of (bits - lo) >> shift over the n collected distances with bits in
// [lo, lo + 2^(shift + 12)).
__global__ void __launch_bounds__(256) median_buffer_kernel(const float* __restrict__ buf, unsigned long long n,
                                                            unsigned lo, int shift, HistCount* __restrict__ hist) {
    __shared__ unsigned h[kHistBins];
    for (int e = threadIdx.x; e < kHistBins; e += 256) h[e] = 0u;
    __syncthreads();
    for (unsigned long long t = (unsigned long long)blockIdx.x * 256 + threadIdx.x; t < n;
         t += (unsigned long long)gridDim.x * 256) {
        const unsigned b = __float_as_uint(buf[t]);
        if (b >= lo && (b - lo) >> shift < (unsigned)kHistBins) atomicAdd(&h[(b - lo) >> shift], 1u);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < kHistBins; e += 256)
        if (h[e]) atomicAdd(&hist[e], (HistCount)h[e]);
}

// The median over all pairs in one pass; *found = false (the caller goes on with
// the radix selection) when there is no room for the bracket or it misses.
static int run_bracketed_median(kevd_ctx* ctx, const float* X, int64_t N, int d, uint64_t rank, HistCount* hist,
                                unsigned* bits, bool* found, cudaStream_t s) {
    *found = false;
    const int64_t nt = (N + kCalTile - 1) / kCalTile;
    const int64_t n_tiles = nt * (nt + 1) / 2;
    const uint64_t total = (uint64_t)N * (uint64_t)(N - 1) / 2;
    // +- 5 standard deviations of the sample's median: 2 % of the pairs with 2^16
    // samples, 0.5 % with 2^20, which the buffer (256 MiB) holds up to N = 160,000
    const int n = total > 400000000ull ? 1 << 20 : 1 << 16;
    const int half = (int)(2.5 * std::sqrt((double)n));
    const unsigned long long cap = (unsigned long long)std::min<uint64_t>((uint64_t)(0.06 * (double)total), 1ull << 26);
    int st = KEVD_OK;
    float* buf = arena_get<float>(ctx, "med.buf", cap, &st);
    unsigned* smp = arena_get<unsigned>(ctx, "med.smp", (size_t)n + 3, &st);
    unsigned long long* cnt = arena_get<unsigned long long>(ctx, "med.cnt", 2, &st);
    if (st != KEVD_OK) {
        for (const char* b : {"med.buf", "med.smp", "med.cnt"}) ctx->arena.idle(b);
        return KEVD_OK;
    }
    unsigned* br = smp + n;
    KEVD_CUDA(ctx, cudaMemsetAsync(cnt, 0, 2 * sizeof(*cnt), s));
    median_sample_kernel<<<n / 256, 256, 0, s>>>(X, N, d, n, smp);
    KEVD_LAUNCH(ctx);
    median_bracket_kernel<<<1, 1024, 0, s>>>(smp, n, n / 2 - half, n / 2 + half, br);
    KEVD_LAUNCH(ctx);
    const size_t smem = (size_t)kPtGroups * kPtSmemFloats * sizeof(float);
    KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&median_collect_kernel), (int)smem));
    const int grid = (int)std::min<int64_t>(2 * n_tiles, ctx->num_sms);
    median_collect_kernel<<<grid, kPtThreads, smem, s>>>(X, N, d, n_tiles, br,
                                                         (unsigned)((double)n * (double)cap / (double)total), buf, cap, cnt);
    KEVD_LAUNCH(ctx);
    unsigned hbr[2];
    unsigned long long hc[2];
    KEVD_CUDA(ctx, cudaMemcpyAsync(hbr, br, sizeof(hbr), cudaMemcpyDeviceToHost, s));
    KEVD_CUDA(ctx, cudaMemcpyAsync(hc, cnt, sizeof(hc), cudaMemcpyDeviceToHost, s));
    KEVD_CUDA(ctx, cudaStreamSynchronize(s));
    if (rank < hc[0] || rank - hc[0] >= hc[1] || hc[1] > cap) return KEVD_OK;
    uint64_t left = rank - hc[0];
    unsigned lo = hbr[0];
    std::vector<HistCount> hh(kHistBins);
    int shift = 0;   // the largest offset, hbr[1] - 1 - hbr[0], has a bin
    while ((hbr[1] - 1 - hbr[0]) >> shift >= (unsigned)kHistBins) ++shift;
    for (;;) {
        KEVD_CUDA(ctx, cudaMemsetAsync(hist, 0, kHistBins * sizeof(HistCount), s));
        median_buffer_kernel<<<(unsigned)std::min<unsigned long long>((hc[1] + 1023) / 1024, 2ull * ctx->num_sms), 256, 0,
                               s>>>(buf, hc[1], lo, shift, hist);
        KEVD_LAUNCH(ctx);
        KEVD_CUDA(ctx, cudaMemcpyAsync(hh.data(), hist, kHistBins * sizeof(HistCount), cudaMemcpyDeviceToHost, s));
        KEVD_CUDA(ctx, cudaStreamSynchronize(s));
        unsigned bin = 0;
        while (bin < (unsigned)kHistBins && left >= hh[bin]) left -= hh[bin++];
        if (bin == (unsigned)kHistBins) return KEVD_OK;
        lo += bin << shift;
        if (shift == 0) break;
        shift = std::max(0, shift - 12);
    }
    *bits = lo;
    *found = true;
    return KEVD_OK;
}

// Whether one pass with a bracket beats three.  A pass takes about 16 features' time a
// pair beside its d; the sample and its selection 100 us and 0.1 us a feature.  Times,
// three passes / bracket: N = 8,000, d = 3 176 / 201 us; 6,000, 16 189 / 199 and 8,000, 16
// 267 / 227; 5,000, 64 324 / 272; 3,000, 128 264 / 282 and 4,000, 128 396 / 317; 2,000,
// 1,024 832 / 850 and 3,000, 1,024 1,457 / 1,076.
static bool bracket_pays(int64_t N, int d) {
    return 0.5 * (double)N * (double)(N - 1) * (d + 16) >= 8e8 + 1.4e6 * d;
}

int run_pair_median(kevd_ctx* ctx, const float* X, int64_t N, int d, const int64_t* pi,
                    const int64_t* pl, int64_t n_pairs, double* median, cudaStream_t s) {
    if (!X || !median || N < 2 || d < 1 || d > kCalMaxD || n_pairs < 0 ||
        (n_pairs > 0 && (!pi || !pl)))
        return set_error(ctx, KEVD_ERR_ARG, "pair_median: bad arguments");
    const bool exact = (n_pairs == 0);
    const int64_t nt = (N + kCalTile - 1) / kCalTile;
    const int64_t n_tiles = nt * (nt + 1) / 2;
    const uint64_t total = exact ? (uint64_t)N * (uint64_t)(N - 1) / 2 : (uint64_t)n_pairs;
    uint64_t rank = (total - 1) / 2;  // lower median
    int st = KEVD_OK;
    HistCount* hist = arena_get<HistCount>(ctx, "med.hist", kHistBins, &st);
    if (st != KEVD_OK) return st;
    if (exact && bracket_pays(N, d) && N <= 160000) {
        bool found = false;
        unsigned bits = 0;
        KEVD_TRY(run_bracketed_median(ctx, X, N, d, rank, hist, &bits, &found, s));
        if (found) {
            float m;
            std::memcpy(&m, &bits, sizeof(float));
            *median = (double)m;
            return KEVD_OK;
        }
    }
    const size_t smem = (size_t)kPtGroups * kPtSmemFloats * sizeof(float) + kHistBins * sizeof(unsigned);
    KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&median_tiles_kernel), (int)smem));
    const int shifts[3] = {20, 8, 0};
    const unsigned masks[3] = {0xfffu, 0xfffu, 0xffu};
    unsigned prefix = 0;
    int hi_shift = 32;
    std::vector<HistCount> hh(kHistBins);
    for (int pass = 0; pass < 3; ++pass) {
        KEVD_CUDA(ctx, cudaMemsetAsync(hist, 0, kHistBins * sizeof(HistCount), s));
        if (exact) {
            for (int64_t u = 0; u < 2 * n_tiles; u += ctx->num_sms * kHistUnits) {
                const int64_t nu = std::min(2 * n_tiles - u, ctx->num_sms * kHistUnits);
                median_tiles_kernel<<<(int)std::min<int64_t>(nu, ctx->num_sms), kPtThreads, smem, s>>>(
                    X, N, d, u, nu, shifts[pass], masks[pass], prefix, hi_shift, hist);
                KEVD_LAUNCH(ctx);
            }
        } else {
            const int grid = (int)std::min<int64_t>((n_pairs + 255) / 256, (int64_t)ctx->num_sms * 4);
            median_pairs_kernel<<<grid, 256, 0, s>>>(X, d, pi, pl, n_pairs, shifts[pass],
                                                     masks[pass], prefix, hi_shift, hist);
            KEVD_LAUNCH(ctx);
        }
        KEVD_CUDA(ctx, cudaMemcpyAsync(hh.data(), hist, kHistBins * sizeof(HistCount),
                                       cudaMemcpyDeviceToHost, s));
        KEVD_CUDA(ctx, cudaStreamSynchronize(s));
        uint64_t cum = 0;
        int bin = -1;
        for (int b = 0; b <= (int)masks[pass]; ++b) {
            if (cum + hh[b] > rank) {
                bin = b;
                break;
            }
            cum += hh[b];
        }
        if (bin < 0) return set_error(ctx, KEVD_ERR_CUDA, "pair_median: histogram lost counts");
        rank -= cum;
        prefix = (hi_shift >= 32 ? 0u : (prefix << (hi_shift - shifts[pass]))) | (unsigned)bin;
        hi_shift = shifts[pass];
    }
    float m;
    unsigned bits = prefix;
    std::memcpy(&m, &bits, sizeof(float));
    *median = (double)m;
    return KEVD_OK;
}

}  // namespace kevd
