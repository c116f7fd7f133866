// Many uneven calibrations in one persistent launch.
//
// A batch of datasets (each its own X, N, d and eps sweep) is flattened into a
// device work queue of (dataset, tile range) items covering every dataset's
// lower-triangle 128 x 128 pair tiles.  One persistent grid (four groups per SM)
// takes items with an atomic counter, so the large datasets' items and the
// small datasets' items share the GPU without one launch per dataset and
// without idle SMs at the tail of a small dataset.  Each item writes its own
// FP64 partial per eps; a second kernel sums each dataset's items in item
// order, so the result does not depend on which CTA took which item.  The
// per-tile arithmetic is the single-dataset pass's (FP32 direct distances,
// ex2.approx, FP32 warp partials, FP64 accumulation).
//
// The launch sequence (counter reset, persistent kernel, reduction) has no host
// synchronisation or allocation once the queue is uploaded, so it can be
// captured in a CUDA graph and replayed.
#include "kevd_internal.cuh"
#include "kevd_pairtile.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace kevd {

namespace {

constexpr int kTile = 128;
constexpr int kMaxScalesB = 64;
constexpr int kMaxDB = 1024;

struct JobDesc {
    const float* X;
    int64_t N;
    int64_t n_tiles;
    int32_t d;
    int32_t n_scales;
    int32_t scale_off;   // into the flattened FP32 scale array (already x log2 e)
    int32_t item0;       // first item of the job
    int32_t n_items;
    int32_t pad;
};

struct Item {
    int32_t job;
    int32_t pad;
    int64_t u0, u1;      // range [u0, u1) of half tiles (pt_unit)
};

// Each group of a CTA takes items of its own.
__global__ void __launch_bounds__(kPtThreads, 1)
calibrate_queue_kernel(const JobDesc* __restrict__ jobs, const Item* __restrict__ items, int item_base,
                       int n_items, const float* __restrict__ c2all, int* __restrict__ counter,
                       double* __restrict__ partial) {
    extern __shared__ __align__(16) float smem[];
    __shared__ int cur[kPtGroups];
    static_assert(kMaxScalesB <= kPtGroup, "one thread per scale");
    const int g = pt_group(), gt = pt_tid();
    float* sm = smem + g * kPtSmemFloats;
    float* cs = smem + kPtGroups * kPtSmemFloats + g * (1 + kPtWarps) * kMaxScalesB;   // kMaxScalesB
    float* red = cs + kMaxScalesB;                                                    // 4 warps x kMaxScalesB
    while (true) {
        pt_sync();
        if (gt == 0) cur[g] = atomicAdd(counter, 1);
        pt_sync();
        if (cur[g] >= n_items) break;
        const int it = item_base + cur[g];
        const Item item = items[it];
        const JobDesc jb = jobs[item.job];
        if (gt < jb.n_scales) cs[gt] = c2all[jb.scale_off + gt];
        double acc = 0.0;   // thread j < n_scales of the group owns eps j
        PtUnit unit = pt_unit(item.u0);
        int64_t staged = -1;
        for (int64_t u = item.u0; u < item.u1; ++u, pt_next(unit)) {
            f32x2 D[8][4];
            pt_dist(jb.X, jb.N, jb.d, unit, sm, staged, D);
            pt_mask(jb.N, unit, D);
            pt_exp_sums(D, cs, jb.n_scales, red, kMaxScalesB);
            pt_sync();
            if (gt < jb.n_scales) {
                double w = 0.0;
#pragma unroll
                for (int q = 0; q < kPtWarps; ++q) w += (double)red[q * kMaxScalesB + gt];
                acc += w;
            }
        }
        if (gt < jb.n_scales) partial[(int64_t)it * kMaxScalesB + gt] = acc;
    }
}

// One CTA per job: 16 slices of its items in item order, then the slices in order.
constexpr int kReduceSlices = 16;
__global__ void __launch_bounds__(kReduceSlices * kMaxScalesB)
calibrate_queue_reduce_kernel(const JobDesc* __restrict__ jobs, const double* __restrict__ partial,
                              double* __restrict__ out) {
    __shared__ double part[kReduceSlices][kMaxScalesB];
    const int job = blockIdx.x, j = threadIdx.x % kMaxScalesB, sl = threadIdx.x / kMaxScalesB;
    const JobDesc& jb = jobs[job];
    const int n = jb.n_items, q0 = (int)((int64_t)n * sl / kReduceSlices), q1 = (int)((int64_t)n * (sl + 1) / kReduceSlices);
    double s = 0.0;
    if (j < jb.n_scales) {
#pragma unroll 8
        for (int q = q0; q < q1; ++q) s += partial[(int64_t)(jb.item0 + q) * kMaxScalesB + j];
    }
    part[sl][j] = s;
    __syncthreads();
    if (sl == 0 && j < jb.n_scales) {
        for (int t = 1; t < kReduceSlices; ++t) s += part[t][j];
        out[job * kMaxScalesB + j] = s;
    }
}

size_t queue_smem() {
    return (size_t)kPtGroups * (kPtSmemFloats + (1 + kPtWarps) * kMaxScalesB) * sizeof(float);
}

}  // namespace

int run_calibrate_batched(kevd_ctx* ctx, const kevd_calib_job* jobs, int n_jobs, int tiles_per_item,
                          cudaStream_t s) {
    if (!jobs || n_jobs < 1 || n_jobs > 4096 || tiles_per_item < 0)
        return set_error(ctx, KEVD_ERR_ARG, "calibrate_batched: need 1..4096 jobs");
    std::vector<JobDesc> hj(n_jobs);
    std::vector<Item> hi;
    std::vector<float> hc;
    int64_t total_tiles = 0;
    for (int q = 0; q < n_jobs; ++q) {
        const kevd_calib_job& j = jobs[q];
        if (!j.X || !j.scales || !j.sums || j.N < 1 || j.d < 1 || j.d > kMaxDB || j.n_scales < 1 ||
            j.n_scales > kMaxScalesB)
            return set_error(ctx, KEVD_ERR_ARG, "calibrate_batched: job %d needs N >= 1, 1 <= d <= %d, "
                             "1 <= n_scales <= %d", q, kMaxDB, kMaxScalesB);
        const int64_t nt = (j.N + kTile - 1) / kTile;
        total_tiles += nt * (nt + 1) / 2;
    }
    // item size in half tiles: about 8 items per group of threads over the whole
    // batch unless given
    const int64_t per = tiles_per_item > 0
                            ? 2 * (int64_t)tiles_per_item
                            : std::max<int64_t>(1, 2 * total_tiles / ((int64_t)ctx->num_sms * kPtGroups * 8));
    // features are staged kPtChunk at a time, so shared memory does not depend on d
    // and one persistent launch serves every dataset of the batch
    std::vector<int> order(n_jobs);
    for (int q = 0; q < n_jobs; ++q) order[q] = q;
    for (int oi = 0; oi < n_jobs; ++oi) {
        const int q = order[oi];
        const kevd_calib_job& j = jobs[q];
        const int64_t nt = (j.N + kTile - 1) / kTile;
        const int64_t tiles = nt * (nt + 1) / 2;
        JobDesc& d = hj[q];
        d.X = j.X;
        d.N = j.N;
        d.n_tiles = tiles;
        d.d = j.d;
        d.n_scales = j.n_scales;
        d.scale_off = (int32_t)hc.size();
        d.item0 = (int32_t)hi.size();
        for (int e = 0; e < j.n_scales; ++e) {
            if (!(j.scales[e] > 0.0)) return set_error(ctx, KEVD_ERR_ARG, "calibrate_batched: scales must be positive");
            hc.push_back((float)(j.scales[e] * 1.4426950408889634));
        }
        for (int64_t u0 = 0; u0 < 2 * tiles; u0 += per) hi.push_back(Item{q, 0, u0, std::min(2 * tiles, u0 + per)});
        d.n_items = (int32_t)hi.size() - d.item0;
        d.pad = 0;
    }
    if (hi.size() > (size_t)INT32_MAX / 2) return set_error(ctx, KEVD_ERR_ARG, "calibrate_batched: too many items");
    const int n_items = (int)hi.size();
    int st = KEVD_OK;
    JobDesc* dj = arena_get<JobDesc>(ctx, "cb.jobs", n_jobs, &st);
    Item* di = arena_get<Item>(ctx, "cb.items", n_items, &st);
    float* dc = arena_get<float>(ctx, "cb.c2", hc.size(), &st);
    int* counter = arena_get<int>(ctx, "cb.counter", 1, &st);
    double* partial = arena_get<double>(ctx, "cb.partial", (size_t)n_items * kMaxScalesB, &st);
    double* out = arena_get<double>(ctx, "cb.out", (size_t)n_jobs * kMaxScalesB, &st);
    if (st != KEVD_OK) return set_error(ctx, st, "calibrate_batched: out of device memory");
    KEVD_CUDA(ctx, cudaMemcpyAsync(dj, hj.data(), hj.size() * sizeof(JobDesc), cudaMemcpyHostToDevice, s));
    KEVD_CUDA(ctx, cudaMemcpyAsync(di, hi.data(), hi.size() * sizeof(Item), cudaMemcpyHostToDevice, s));
    KEVD_CUDA(ctx, cudaMemcpyAsync(dc, hc.data(), hc.size() * sizeof(float), cudaMemcpyHostToDevice, s));
    KEVD_CUDA(ctx, cudaMemsetAsync(counter, 0, sizeof(int), s));
    const size_t smem = queue_smem();
    KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&calibrate_queue_kernel), (int)smem));
    {
        ProfScope ps(ctx, "calibrate_queue", s);
        calibrate_queue_kernel<<<ctx->num_sms, kPtThreads, smem, s>>>(dj, di, 0, n_items, dc, counter, partial);
        KEVD_LAUNCH(ctx);
    }
    calibrate_queue_reduce_kernel<<<n_jobs, kReduceSlices * kMaxScalesB, 0, s>>>(dj, partial, out);
    KEVD_LAUNCH(ctx);
    std::vector<double> hout((size_t)n_jobs * kMaxScalesB);
    KEVD_CUDA(ctx, cudaMemcpyAsync(hout.data(), out, hout.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
    KEVD_CUDA(ctx, cudaStreamSynchronize(s));
    for (int q = 0; q < n_jobs; ++q)
        std::memcpy(jobs[q].sums, hout.data() + (size_t)q * kMaxScalesB, jobs[q].n_scales * sizeof(double));
    return KEVD_OK;
}

}  // namespace kevd
