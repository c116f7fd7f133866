// Fused out-of-sample evaluation (pass 4 of ks_kevd.cu:2246-2269 on new rows):
//
//   U(y)[c] = sum_j K(y, s_j) W[j][c] / sum_j K(y, s_j) W[j][k_out]
//
// K(y, s_j) is FP32 from direct differences summed over the features in
// increasing order (relative error about 1e-7).  W = L^{-T} [Z | c1] has large
// entries of both signs, so the sum over the landmarks needs FP64-like
// accuracy; the FP64 pipe (2 lanes per clock per SM) took 16 clocks per
// (state, landmark) for 33 columns.  Here W is an FP32 pair, every product
// K (hi + lo) keeps its rounding error (fma) and the running sum is a
// double-FP32 pair (two-sum): about 2^-46 of the partial sums, on the FP32
// pipe (11 operations, 3 clocks per (state, landmark)).
//
// The landmarks are cut into kGroups fixed groups (a function of r alone), one
// CTA of a 16-CTA cluster each; the groups' sums meet in FP64 through
// distributed shared memory, in group order (or one CTA walks through the groups, where
// landmarks are few for the batch).  A single state then occupies 16
// SMs instead of one, no workspace is needed (calls on any streams are
// independent, and the launch can be captured), and no thread ever combines
// two states: a state's values are bit-identical whatever batch it is in and
// wherever it sits there.
#include "kevd_internal.cuh"
#include "kevd_nystrom.cuh"
#include "kevd_pairtile.cuh"
#include "kevd_tc.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace kevd {

namespace {

namespace cg = cooperative_groups;

constexpr int kGroups = 16;     // landmark groups = CTAs per cluster
constexpr int kLm = 32;         // landmarks per step
constexpr int kLanesR = 8;      // thread rows of the K tile and of the sums
constexpr int kFeat = 128;      // features staged at a time
constexpr int kMinThreads = kLanesR * kLm;

// K tile: Q = 1 [state][landmark]; Q = 4 [landmark][thread row][q], so that the four
// states of a sum thread are one 16-byte read
constexpr int kKvPitch = kLanesR * 4 + 4;
template <int Q>
__host__ __device__ constexpr int kv_floats() { return Q == 4 ? kLm * kKvPitch : kLanesR * Q * (kLm + 1); }

__host__ __device__ inline int feat_pitch(int d) { return ((d < kFeat ? d : kFeat) + 3) / 4 * 4 + 4; }

// Shared memory of one CTA with Q states per thread row: two landmark tiles,
// the states, two W tiles, the K tile; the group's FP64 sums reuse the tiles.
template <int Q>
size_t smem_bytes(int d, int kc) {
    const size_t p = feat_pitch(d);
    const size_t tiles = (2 * kLm + kLanesR * Q) * p * sizeof(float);
    const size_t w = 2 * (size_t)kLm * kc * sizeof(float2);
    const size_t kv = (size_t)kv_floats<Q>() * sizeof(float);
    return std::max(tiles + w + kv, (size_t)kLanesR * Q * kc * sizeof(double));
}

// (s, c) += x * (w.x + w.y): the product's rounding error by fma, the sum's by
// two-sum.  The intrinsics keep the compiler from contracting the error terms.
__device__ __forceinline__ void pair_fma(float& s, float& c, float x, float2 w) {
    const float p = __fmul_rn(x, w.x);
    const float pe = __fmaf_rn(x, w.x, -p);
    const float t = __fadd_rn(s, p);
    const float z = __fsub_rn(t, s);
    const float e = __fadd_rn(__fsub_rn(s, __fsub_rn(t, z)), __fsub_rn(p, z));
    s = t;
    c = __fadd_rn(c, __fmaf_rn(x, w.y, __fadd_rn(pe, e)));
}

// The same for two states at once (packed pairs: half of the issue slots).  np = -x w.x,
// so that every difference is an FMA by -1, which rounds as the subtraction does.
__device__ __forceinline__ void pair_fma2(f32x2& s, f32x2& c, f32x2 x, f32x2 wx, f32x2 nwx, f32x2 wy) {
    const f32x2 m1 = pack2(-1.f, -1.f);
    const f32x2 np = mul2(x, nwx);
    const f32x2 pe = fma2(x, wx, np);
    const f32x2 t = fma2(np, m1, s);
    const f32x2 z = fma2(s, m1, t);
    const f32x2 e1 = fma2(fma2(z, m1, t), m1, s);
    const f32x2 e = fma2(add2(np, z), m1, e1);
    s = t;
    c = add2(c, fma2(x, wy, add2(pe, e)));
}

// 8-byte global -> shared copy; src_bytes 0 fills zeros.
__device__ __forceinline__ void cp_async8(void* dst, const void* src, uint32_t src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
}

// Rows [r0, r0 + rows) x features [f0, f0 + w) of a row-major n x d matrix into
// dst (pitch p), zeros past n and up to w rounded up to 4.
__device__ __forceinline__ void stage_rows(const float* __restrict__ src, int64_t n, int d, int64_t r0, int rows,
                                           int f0, int w, bool vec, float* dst, int p) {
    const int nq = (w + 3) >> 2;
    for (int e = threadIdx.x; e < rows * nq; e += blockDim.x) {
        const int rr = e / nq, k4 = (e - rr * nq) << 2;
        const int64_t row = r0 + rr;
        if (vec) {
            tc::cp_async16(dst + rr * p + k4, row < n ? src + row * d + f0 + k4 : src, row < n ? 16u : 0u);
        } else {
#pragma unroll
            for (int u = 0; u < 4; ++u)
                dst[rr * p + k4 + u] = (row < n && k4 + u < w) ? src[row * d + f0 + k4 + u] : 0.f;
        }
    }
}

// One cluster serves kLanesR * Q states, CTA rank g the landmarks of group g in
// steps of kLm: 256 threads form the K tile (state row warp + 8 q, landmark
// lane), then thread (rg, c) of 8 x kc adds the step's landmarks, in order, to
// the sums of states rg + 8 q and column c.  The next step's tiles are in
// flight meanwhile (cp.async).
// Q = 4 halves the W loads per product against Q = 1 and sums pairs of states in
// packed FP32 (16,384 states against 2,000 landmarks, 33 columns: 1,018 -> 903 us,
// two thirds of the FP32 pipe; fewer CTAs per 32 states with more landmark groups
// each is no faster: 923 to 956 us); Q = 1 is for batches
// that would leave SMs without a CTA otherwise.
//
// kOne: one CTA, without a cluster, takes all groups of its states in turn: the same
// sums in the same order, group by group.  Few landmarks leave a CTA of the cluster one
// step or none, and its start, its staging of the states and the hand-over cost more.
template <int Q, bool kOne>   // Q = 1 or 4
__global__ void __launch_bounds__(544)
nystrom_eval_kernel(const float* __restrict__ Y, int64_t n, const float* __restrict__ xs,
                    const float2* __restrict__ w, const int* __restrict__ ex, int64_t r, int d, int k_out,
                    ScalePair scale, float* __restrict__ Uy) {
    extern __shared__ __align__(16) unsigned char ny_smem[];
    constexpr int kRows = kLanesR * Q;
    const int kc = k_out + 1;
    const int p = feat_pitch(d);
    float* xt = reinterpret_cast<float*>(ny_smem);            // 2 x kLm x p
    float* ys = xt + 2 * kLm * p;                             // kRows x p
    float2* wt = reinterpret_cast<float2*>(ys + kRows * p);   // 2 x kLm x kc
    float* kv = reinterpret_cast<float*>(wt + 2 * kLm * kc);  // kv_floats
    const int group = kOne ? 0 : (int)cg::this_cluster().block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t row0 = (int64_t)(kOne ? blockIdx.x : blockIdx.x / kGroups) * kRows;
    const int64_t steps_all = (r + kLm - 1) / kLm;
    const int64_t per = (steps_all + kGroups - 1) / kGroups;
    const int64_t s0 = min(steps_all, group * per), s1 = kOne ? steps_all : min(steps_all, s0 + per);
    const int n_f = (d + kFeat - 1) / kFeat;   // feature chunks per step
    const bool vec = (d & 3) == 0 && ((uintptr_t)Y & 15) == 0;
    const bool vecx = (d & 3) == 0;            // xs is an allocation of its own

    // flat sequence of (landmark step, feature chunk); the states are staged
    // with the first chunk, and again for every chunk where there are several
    auto stage = [&](int64_t s, int f, int buf) {
        const int f0 = f * kFeat, wd = min(kFeat, d - f0);
        stage_rows(xs, r, d, s * kLm, kLm, f0, wd, vecx, xt + buf * kLm * p, p);
        if (f == 0) {
            const int64_t e0 = s * kLm * kc, e1 = min(r, (s + 1) * kLm) * kc;
            float2* dst = wt + (s & 1) * kLm * kc;
            for (int e = tid; e < kLm * kc; e += blockDim.x)
                cp_async8(dst + e, e0 + e < e1 ? w + e0 + e : w, e0 + e < e1 ? 8u : 0u);
        }
    };
    const int c = tid % kc, rg = tid / kc;
    float sum[Q], err[Q];
    f32x2 sum2[2] = {0, 0}, err2[2] = {0, 0};   // Q = 4: pairs of states
#pragma unroll
    for (int q = 0; q < Q; ++q) sum[q] = err[q] = 0.f;
    double total[Q];   // kOne: the groups so far
#pragma unroll
    for (int q = 0; q < Q; ++q) total[q] = 0.0;
    auto unpack_sums = [&] {
        if constexpr (Q == 4) {
            unpack2(sum2[0], sum[0], sum[1]);
            unpack2(sum2[1], sum[2], sum[3]);
            unpack2(err2[0], err[0], err[1]);
            unpack2(err2[1], err[2], err[3]);
        }
    };
    int64_t left = per;   // kOne: steps of this group still to come

    if (s0 < s1) {
        stage_rows(Y, n, d, row0, kRows, 0, min(kFeat, d), vec, ys, p);
        stage(s0, 0, 0);
        tc::cp_async_commit();
    }
    int buf = 0;
    for (int64_t s = s0; s < s1; ++s) {
        float dist[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) dist[q] = 0.f;
        for (int f = 0; f < n_f; ++f) {
            tc::cp_async_wait<0>();
            __syncthreads();   // this chunk is staged; everyone is past the buffers about to be filled
            if (f + 1 < n_f) stage(s, f + 1, buf ^ 1);
            else if (s + 1 < s1) stage(s + 1, 0, buf ^ 1);
            tc::cp_async_commit();
            if (warp < kLanesR) {
                const int nq = (min(kFeat, d - f * kFeat) + 3) >> 2;
                const float* xr = xt + buf * kLm * p + lane * p;
                for (int k4 = 0; k4 < nq; ++k4) {
                    const float4 b = *reinterpret_cast<const float4*>(xr + 4 * k4);
#pragma unroll
                    for (int q = 0; q < Q; ++q) {
                        const float4 a = *reinterpret_cast<const float4*>(ys + (warp + kLanesR * q) * p + 4 * k4);
                        float t = a.x - b.x;
                        dist[q] = fmaf(t, t, dist[q]);
                        t = a.y - b.y;
                        dist[q] = fmaf(t, t, dist[q]);
                        t = a.z - b.z;
                        dist[q] = fmaf(t, t, dist[q]);
                        t = a.w - b.w;
                        dist[q] = fmaf(t, t, dist[q]);
                    }
                }
            }
            buf ^= 1;
            if (n_f > 1) {   // the states' next chunk replaces this one
                __syncthreads();
                const int fn = (f + 1 < n_f) ? f + 1 : 0;
                if (fn != 0 || s + 1 < s1) {
                    stage_rows(Y, n, d, row0, kRows, fn * kFeat, min(kFeat, d - fn * kFeat), vec, ys, p);
                    tc::cp_async_commit();
                }
            }
        }
        if (warp < kLanesR) {
            float v[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) v[q] = (s * kLm + lane < r) ? kexp_scaled(dist[q], scale) : 0.f;
            if constexpr (Q == 4)
                *reinterpret_cast<float4*>(kv + lane * kKvPitch + 4 * warp) = make_float4(v[0], v[1], v[2], v[3]);
            else
                kv[warp * (kLm + 1) + lane] = v[0];
        }
        __syncthreads();
        if (rg < kLanesR) {
            const float2* wc = wt + (s & 1) * kLm * kc + c;
#pragma unroll 4
            for (int j = 0; j < kLm; ++j) {
                const float2 wv = wc[j * kc];
                if constexpr (Q == 4) {
                    const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(kv + j * kKvPitch + 4 * rg);
                    const f32x2 wx = pack2(wv.x, wv.x), nwx = pack2(-wv.x, -wv.x), wy = pack2(wv.y, wv.y);
                    pair_fma2(sum2[0], err2[0], x.x, wx, nwx, wy);
                    pair_fma2(sum2[1], err2[1], x.y, wx, nwx, wy);
                } else {
                    pair_fma(sum[0], err[0], kv[rg * (kLm + 1) + j], wv);
                }
            }
            if (kOne && (--left == 0 || s + 1 == s1)) {
                unpack_sums();
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    total[q] += (double)sum[q] + (double)err[q];
                    sum[q] = err[q] = 0.f;
                }
                sum2[0] = sum2[1] = err2[0] = err2[1] = 0;
                left = per;
            }
        }
    }
    if (!kOne) unpack_sums();
    tc::cp_async_wait<0>();
    __syncthreads();
    double* part = reinterpret_cast<double*>(ny_smem);   // kRows x kc, over the tiles
    if (rg < kLanesR) {
#pragma unroll
        for (int q = 0; q < Q; ++q)
            part[(rg + kLanesR * q) * kc + c] = kOne ? total[q] : (double)sum[q] + (double)err[q];
    }
    if constexpr (kOne) {
        __syncthreads();
        for (int e = tid; e < kRows * k_out; e += blockDim.x) {
            const int rr = e / k_out, cc = e - rr * k_out;
            if (row0 + rr < n)
                Uy[(row0 + rr) * k_out + cc] =
                    (float)ldexp(part[rr * kc + cc] / part[rr * kc + k_out], ex[cc] - ex[k_out]);
        }
        return;
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    // the cluster's CTAs share the outputs; every sum runs over the groups in order
    for (int e = group * blockDim.x + tid; e < kRows * k_out; e += kGroups * blockDim.x) {
        const int rr = e / k_out, cc = e - rr * k_out;
        if (row0 + rr >= n) continue;
        double num[kGroups], den[kGroups];
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            const double* pg = cluster.map_shared_rank(part, g) + rr * kc;
            num[g] = pg[cc];
            den[g] = pg[k_out];
        }
        double a = 0.0, b = 0.0;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            a += num[g];
            b += den[g];
        }
        Uy[(row0 + rr) * k_out + cc] = (float)ldexp(a / b, ex[cc] - ex[k_out]);
    }
    cluster.sync();   // no CTA leaves while its sums are read
}

// W column blockIdx.x: its binade and the FP32 pairs, scaled to 2^kWExp: K is as
// small as 2^-126 for a state far from every landmark, and with |W| < 1 the low parts
// of its products (2^-24 and 2^-48 of K W), then K W itself where the near landmarks
// have small entries, left the FP32 range.  A sum over r < 2^20 landmarks stays below
// 2^120, and the factor cancels in the quotient.
constexpr int kWExp = 100;
__global__ void __launch_bounds__(256) nystrom_pack_kernel(const double* __restrict__ zp, int64_t r, int kc,
                                                           float2* __restrict__ w, int* __restrict__ ex) {
    __shared__ double red[256];
    const int c = blockIdx.x;
    const double* col = zp + (int64_t)c * r;
    double m = 0.0;
    for (int64_t j = threadIdx.x; j < r; j += 256) m = fmax(m, fabs(col[j]));
    red[threadIdx.x] = m;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + o]);
        __syncthreads();
    }
    int e = kWExp;
    if (red[0] > 0.0 && isfinite(red[0])) frexp(red[0], &e);
    e -= kWExp;
    for (int64_t j = threadIdx.x; j < r; j += 256) {
        const double v = ldexp(col[j], -e);
        const float h = (float)v;
        w[j * kc + c] = make_float2(h, (float)(v - (double)h));
    }
    if (threadIdx.x == 0) ex[c] = e;
}

template <int Q, bool kOne>
int launch_eval(kevd_ctx* ctx, const Model& m, const float* Y, int64_t n, float* Uy, cudaStream_t s) {
    const int kc = m.k_out + 1;
    const int64_t blocks = (n + kLanesR * Q - 1) / (kLanesR * Q);
    const size_t smem = smem_bytes<Q>(m.d, kc);
    const void* fn = reinterpret_cast<const void*>(&nystrom_eval_kernel<Q, kOne>);
    KEVD_CUDA(ctx, raise_smem_limit(fn, std::max(smem, (size_t)48 * 1024)));
    // 16 CTAs per cluster is above the portable 8
    if (!kOne) KEVD_CUDA(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(kOne ? blocks : blocks * kGroups));
    cfg.blockDim = dim3((unsigned)std::max(kMinThreads, (kLanesR * kc + 31) / 32 * 32));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kGroups;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = kOne ? 0 : 1;
    KEVD_CUDA(ctx, cudaLaunchKernelEx(&cfg, &nystrom_eval_kernel<Q, kOne>, Y, n, (const float*)m.xs, (const float2*)m.w,
                                      (const int*)m.ex, m.r, m.d, m.k_out, split_scale(m.scale), Uy));
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

}  // namespace

int launch_nystrom_pack(kevd_ctx* ctx, const double* zp, const Model& m, cudaStream_t s) {
    nystrom_pack_kernel<<<m.k_out + 1, 256, 0, s>>>(zp, m.r, m.k_out + 1, m.w, m.ex);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

// Clusters split the landmarks 16 ways and start 16 CTAs for 32 states; one CTA walks
// through all of them.  Times in us, clusters / one CTA (d = 64, 8 columns): 100
// landmarks n = 1,000 27 / 23, 16,384 229 / 43; 300 1,000 27 / 48, 4,096 68 / 48, 65,536
// 905 / 319; 1,000 4,096 97 / 132, 16,384 335 / 292; 2,000 16,384 581 / 563 (32 columns 898
// / 992), 65,536 2,262 / 1,863.
static bool one_cta(int64_t r, int64_t n) {
    return 200 * ((r + kLm - 1) / kLm) <= std::min<int64_t>(n, 4096) + std::max<int64_t>(0, n - 4096) / 5;
}

// 32 states per cluster once those clusters give every SM a CTA (n > 300), or per CTA
// (one_cta); fewer states are served 8 per cluster.
int launch_nystrom_eval(kevd_ctx* ctx, const Model& m, const float* Y, int64_t n, float* Uy, cudaStream_t s) {
    constexpr int64_t kPiece = (int64_t)1 << 30;   // states per launch: the grid stays below 2^31 CTAs
    for (int64_t i = 0; i < n; i += kPiece) {
        const int64_t ni = std::min(kPiece, n - i);
        auto launch = ni <= 2 * ctx->num_sms ? &launch_eval<1, false>
                      : one_cta(m.r, ni)     ? &launch_eval<4, true>
                                             : &launch_eval<4, false>;
        KEVD_TRY(launch(ctx, m, Y + i * m.d, ni, Uy + i * m.k_out, s));
    }
    return KEVD_OK;
}

}  // namespace kevd
