// Stage 2: block randomly pivoted Cholesky with a stored factor.
//
// Semantics follow ks_arpclm.cu's round (propose, residual block, accept /
// reject + factor, residual-diagonal update, trace error), with the factor F
// kept in HBM instead of regenerating K(R, S) every round:
//
//   round:  sample   b proposals ~ d                    (1 CTA)
//           hgram    F(S',:) F(S',:)^T split over column chunks, and K(S',S')
//           factor   H = K(S',S') - F F^T, accept/reject, Cholesky, L_i^{-1}
//           update   G = (K(R,S_i) - F(R,:) F(S_i,:)^T) L_i^{-T} for every row
//                    block R; F(R, r:r+nacc) = G; d(R) -= rowsq(G), clamped;
//                    per-block sums of d for the next sampler
//
// All round state stays on the device: kernels read the rank and accepted
// count from a RoundState, and after the stop condition every kernel returns
// immediately, so the host enqueues rounds without a per-round sync (the
// reference synchronises and copies nacc to the host every round,
// ks_arpclm.cu:877-886).
//
// T = double is the plain FP64 form; T = float the mixed form (F, the F F^T
// products and G in FP32; H, its Cholesky and inverse, the residual diagonal
// and all sums in FP64).
#include "kevd_internal.cuh"
#include "kevd_rng.cuh"
#include "kevd_round.cuh"

#include <algorithm>
#include <cstring>
#include <vector>

namespace kevd {

bool update_tc_supported(const float* F, int64_t ldF, int d);
int reserve_update_tc(kevd_ctx* ctx, int64_t N, int64_t k_max);
int launch_update_tc(kevd_ctx* ctx, float* F, int64_t ldF, int64_t N, int64_t k_max, const float* X, int d,
                     double scale, const int64_t* sacc, const float* minv_f, int b, const void* round_state,
                     double* dvec, double* dblk, int* err, cudaStream_t s);

int launch_update_f32(kevd_ctx* ctx, float* F, int64_t ldF, const float* X, int64_t N, int d, double scale,
                      const int64_t* sacc, const float* minv_f, int b, const RoundState* st, double* dvec, double* dblk,
                      cudaStream_t s);

bool rpchol_small_supported(int b);
int64_t rpchol_small_blocks(int64_t N);
int launch_rpchol_small_init(kevd_ctx* ctx, double* dvec, double* dsub, int64_t N, RoundState* st, cudaStream_t s);
int launch_rpchol_small_propose(kevd_ctx* ctx, const double* F, int64_t ldF, const float* X, int64_t N, int d,
                                double scale, const double* dvec, const double* dsub, int round, int b, uint64_t seed,
                                const double* uniforms, double tol, int64_t k_max, int max_rounds, double err_target,
                                RoundState* st, double* minv, int64_t* sacc, int64_t* piv, double* err, int32_t* hm,
                                cudaStream_t s);
int launch_rpchol_small_update(kevd_ctx* ctx, double* F, int64_t ldF, const float* X, int64_t N, int d, double scale,
                               const int64_t* sacc, const double* minv, int b, const RoundState* st, double* dvec,
                               double* dsub, cudaStream_t s);

constexpr int kRowBlock = 128;   // rows per update CTA (= rows per d partial sum)
constexpr int kMaxBlock = 512;   // proposals per round (the reference's default BLK, ks_arpclm.cu:38)
constexpr int kGroup = 64;       // accepted columns per update pass: a round with more runs several passes
constexpr int kSmallBlock = 128; // rounds up to this size factor their block in shared memory
constexpr int kFactorThreads = 512;   // rp_factor_kernel: warp 0 decides, 15 warps update rows
constexpr int kBigFactorThreads = 1024;   // rp_factor_big_kernel: 32 x 32 threads
constexpr int kColChunk = 32;    // F columns per hgram CTA
constexpr int kFeat = 64;        // features staged at a time by the SIMT update
constexpr int kSampleThreads = 1024;

// Acceptance floor of the mixed form, relative to K(S',S')_ii (= 1 for the
// Gaussian kernel).  In the mixed form H = K(S',S') - F(S',:) F(S',:)^T is
// formed from the FP32 factor, whose rounding leaves noise of a few 1e-7 in
// H_ii; a proposal whose H_ii is at that level would be accepted on noise and
// give a column of noise / sqrt(noise).  The mixed form therefore rejects
// H_ii <= 16 u32 K_ii (u32 = 2^-24, about 9.5e-7) and stops once the trace
// error, the mean residual diagonal, has fallen below the same level.  The
// FP64 form keeps the reference's tolerance alone (ks_arpclm.cu:329-331).
constexpr double kMixedFloor = 16.0 / 16777216.0;

// Kernel values of a fixed pseudo-random sample of kDensityPairs pairs (i, j),
// i != j, counted when K(i, j) >= 2^-24.  A factorisation whose kernel is
// nearly diagonal (fewer than half the sampled values reach 2^-24) keeps the
// FP32 SIMT residual update: the tensor-core update splits F into f16 parts
// scaled to |F| <= 1, which hold F's tiny entries only to about 2^-39
// absolutely, and the bistochastic weights 1/dtil^2 of such kernels amplify
// exactly those rows (top-16 eigenvalue errors of 1e-6 .. 1e-5 against FP64
// on the same pivots, against at most 7e-7 with the SIMT update).
constexpr int kDensityPairs = 4096;

__device__ __forceinline__ uint64_t mix64(uint64_t z) {   // splitmix64 finaliser
    z ^= z >> 30;
    z *= 0xBF58476D1CE4E5B9ull;
    z ^= z >> 27;
    z *= 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void __launch_bounds__(256) kernel_density_kernel(const float* __restrict__ X, int64_t N, int d,
                                                              double scale, int* __restrict__ count) {
    int c = 0;
    for (int t = threadIdx.x; t < kDensityPairs; t += blockDim.x) {
        const int64_t i = (int64_t)(mix64(2 * (uint64_t)t + 1) % (uint64_t)N);
        int64_t j = (int64_t)(mix64(2 * (uint64_t)t + 2) % (uint64_t)N);
        if (j == i) j = (i + 1) % N;
        float d2 = 0.f;
        for (int f = 0; f < d; ++f) {
            const float u = X[i * d + f] - X[j * d + f];
            d2 = fmaf(u, u, d2);
        }
        c += (exp(-scale * (double)d2) >= 5.9604644775390625e-8) ? 1 : 0;   // 2^-24
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(count, c);
}

// Whether the kernel is nearly diagonal (see kernel_density_kernel); one
// small launch and a 4-byte copy.  Must not run inside a stream capture.
static int kernel_nearly_diagonal(kevd_ctx* ctx, const float* X, int64_t N, int d, double scale, cudaStream_t s,
                                  bool* out) {
    *out = false;
    if (N < 2) return KEVD_OK;
    int st = KEVD_OK;
    int* cnt = arena_get<int>(ctx, "rp.density", 1, &st);
    if (st != KEVD_OK) return set_error(ctx, st, "rpchol: out of device memory");
    KEVD_CUDA(ctx, cudaMemsetAsync(cnt, 0, sizeof(int), s));
    kernel_density_kernel<<<1, 256, 0, s>>>(X, N, d, scale, cnt);
    KEVD_LAUNCH(ctx);
    int* h = static_cast<int*>(ctx->pinned);
    KEVD_CUDA(ctx, cudaMemcpyAsync(h, cnt, sizeof(int), cudaMemcpyDeviceToHost, s));
    KEVD_CUDA(ctx, cudaStreamSynchronize(s));
    *out = 2 * *h < kDensityPairs;
    return KEVD_OK;
}

__global__ void rp_init_kernel(double* __restrict__ d, double* __restrict__ dblk, int64_t N,
                               int64_t nblk, RoundState* st) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N;
         i += (int64_t)gridDim.x * blockDim.x)
        d[i] = 1.0;
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nblk;
         b += (int64_t)gridDim.x * blockDim.x)
        dblk[b] = (double)min((int64_t)kRowBlock, N - b * kRowBlock);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->rank = 0;
        st->r_old = 0;
        st->nacc = 0;
        st->done = 0;
        st->rounds = 0;
        st->cur = 0;
        st->total = (double)N;
    }
}

// ---- sampler ---------------------------------------------------------------
// Inverse-CDF proposals (ks_arpclm.cu:197-224): pivot = smallest i with
// cumsum(d)[i] >= u * sum(d), else N - 1.  The prefix is hierarchical: a scan
// over per-thread chunks of the block sums, a sequential walk over the chunk,
// then a warp scan inside the 128-row block.  Also records the trace error of
// the previous round and decides the stop (the closing call, after the last
// round, always stops).
__global__ void __launch_bounds__(kSampleThreads)
rp_sample_kernel(const double* __restrict__ d, const double* __restrict__ dblk, int64_t N,
                 int64_t nblk, int closing, int b, uint64_t seed,
                 const double* __restrict__ uniforms, int64_t* __restrict__ props,
                 RoundState* st, int64_t k_max, int max_rounds, double err_target,
                 double err_floor, double* __restrict__ err) {
    __shared__ double incl[kSampleThreads];
    __shared__ int s_stop;
    if (st->done) return;
    const int round = st->cur;
    const int tid = threadIdx.x;
    const int64_t chunk = (nblk + kSampleThreads - 1) / kSampleThreads;
    const int64_t c0 = min(nblk, (int64_t)tid * chunk), c1 = min(nblk, c0 + chunk);
    double s = 0.0;
    for (int64_t q = c0; q < c1; ++q) s += dblk[q];
    incl[tid] = s;
    __syncthreads();
    for (int off = 1; off < kSampleThreads; off <<= 1) {
        const double v = (tid >= off) ? incl[tid - off] : 0.0;
        __syncthreads();
        incl[tid] += v;
        __syncthreads();
    }
    const double total = incl[kSampleThreads - 1];
    if (tid == 0) {
        const double e = total / (double)N;
        if (round > 0) err[round - 1] = e;
        st->total = total;
        const bool stop = closing || (round >= max_rounds) || (st->rank >= k_max) ||
                          (err_target > 0.0 && round > 0 && e <= err_target) ||
                          (err_floor > 0.0 && round > 0 && e <= err_floor);
        if (stop) {
            st->done = 1;
            st->rounds = round;
        }
        s_stop = stop;
    }
    __syncthreads();
    if (s_stop) return;
    const int lane = tid & 31, warp = tid >> 5;
    for (int t = warp; t < b; t += kSampleThreads / 32) {
        const double u = uniforms ? uniforms[((int64_t)round * 2) * b + t]
                                  : philox_uniform(seed, (uint32_t)round, 0u, (uint32_t)t);
        const double target = u * total;
        int64_t pick = N - 1;
        if (target <= total) {
            // smallest chunk owner c with incl[c] >= target
            int lo = 0, hi = kSampleThreads - 1;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (incl[mid] >= target) hi = mid; else lo = mid + 1;
            }
            double base = (lo > 0) ? incl[lo - 1] : 0.0;
            const int64_t q0 = min(nblk, (int64_t)lo * chunk), q1 = min(nblk, q0 + chunk);
            int64_t blk = q1 - 1;
            for (int64_t q = q0; q < q1; ++q) {
                const double nb = base + dblk[q];
                if (nb >= target) { blk = q; break; }
                base = nb;
            }
            if (blk >= q0) {
                // within block: lane l holds rows 4l..4l+3
                const int64_t r0 = blk * kRowBlock;
                double v[4], ls = 0.0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int64_t row = r0 + 4 * lane + j;
                    v[j] = (row < N) ? d[row] : 0.0;
                    ls += v[j];
                }
                double pre = ls;  // inclusive warp scan of lane sums
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double y = __shfl_up_sync(0xffffffffu, pre, o);
                    if (lane >= o) pre += y;
                }
                double cum = base + pre - ls;
                int hit = -1;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    cum += v[j];
                    if (hit < 0 && cum >= target && v[j] > 0.0) hit = j;
                }
                const unsigned m = __ballot_sync(0xffffffffu, hit >= 0);
                if (m) {
                    const int src = __ffs(m) - 1;
                    const int hj = __shfl_sync(0xffffffffu, hit, src);
                    pick = r0 + 4 * src + hj;
                } else {
                    // rounding left the target past this block's recomputed
                    // sum: take its last row with d > 0
                    const unsigned mz = __ballot_sync(0xffffffffu, ls > 0.0);
                    if (mz) {
                        const int src = 31 - __clz(mz);
                        int jj = 3;
                        double vv[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) vv[j] = __shfl_sync(0xffffffffu, v[j], src);
                        while (jj > 0 && !(vv[jj] > 0.0)) --jj;
                        pick = r0 + 4 * src + jj;
                    }
                }
            }
        }
        if (lane == 0) props[t] = min(pick, N - 1);
    }
}

// ---- proposal block: F(S',c-chunk) F(S',c-chunk)^T and K(S',S') -----------
constexpr int kHgramStageRows = 128;
template <typename T>
static size_t hgram_smem(int b) {
    const size_t f = (size_t)b * (kColChunk + 1) * sizeof(T);
    const size_t x = b <= kHgramStageRows ? (size_t)b * 129 * sizeof(float) : 0;
    return std::max(f, x);
}
template <typename T>
__global__ void __launch_bounds__(256)
rp_hgram_kernel(const T* __restrict__ F, int64_t ldF, const float* __restrict__ X, int d,
                double scale, const int64_t* __restrict__ props, int b, int n_split,
                const RoundState* st, double* __restrict__ hpart, double* __restrict__ kss) {
    if (st->done) return;
    // one buffer, used either for an F column chunk or for the X rows of S'
    extern __shared__ __align__(16) unsigned char raw[];
    T* fs = reinterpret_cast<T*>(raw);
    float* xs = reinterpret_cast<float*>(raw);
    const int tid = threadIdx.x;
    if ((int)blockIdx.x < n_split) {
        const int64_t r = st->rank;
        const int64_t c0 = (int64_t)blockIdx.x * kColChunk;
        if (c0 >= r) return;
        const int nc = (int)min((int64_t)kColChunk, r - c0);
        for (int e = tid; e < b * kColChunk; e += 256) {
            const int p = e / kColChunk, c = e - p * kColChunk;
            fs[p * (kColChunk + 1) + c] = (c < nc) ? F[props[p] * ldF + c0 + c] : (T)0;
        }
        __syncthreads();
        for (int e = tid; e < b * b; e += 256) {
            const int p = e / b, q = e - p * b;
            T acc = 0;
#pragma unroll 8
            for (int c = 0; c < kColChunk; ++c)
                acc += fs[p * (kColChunk + 1) + c] * fs[q * (kColChunk + 1) + c];
            hpart[((int64_t)blockIdx.x * b + p) * b + q] = (double)acc;
        }
    } else {
        // K(S', S') in FP64, rows split over the remaining CTAs
        const int nk = gridDim.x - n_split;
        const int part = blockIdx.x - n_split;
        // rows of S' staged in shared memory up to 128 features and 128
        // proposals, read from global memory (L2-resident, b rows) beyond;
        // same summation order
        const bool staged = d <= 128 && b <= kHgramStageRows;
        if (staged)
            for (int e = tid; e < b * d; e += 256) {
                const int p = e / d, k = e - p * d;
                xs[p * 129 + k] = X[props[p] * d + k];
            }
        __syncthreads();
        for (int e = tid; e < b * b; e += 256) {
            const int p = e / b, q = e - p * b;
            if (p % nk != part) continue;
            double acc = 0.0;
            if (staged) {
                for (int k = 0; k < d; ++k) {
                    const double t = (double)xs[p * 129 + k] - (double)xs[q * 129 + k];
                    acc += t * t;
                }
            } else {
                const float* xp = X + props[p] * d;
                const float* xq = X + props[q] * d;
                for (int k = 0; k < d; ++k) {
                    const double t = (double)__ldg(xp + k) - (double)__ldg(xq + k);
                    acc += t * t;
                }
            }
            kss[p * b + q] = exp(-scale * acc);
        }
    }
}

// ---- accept / reject, Cholesky, inverse of the compacted factor ------------
// ks_arpclm.cu:305-408.  One CTA; the b x b matrix lives in shared memory (b <=
// 32 Q).  An accepted proposal i (the m-th) with f = 1 / sqrt(H_ii) makes the
// scaled column l_j = H_ji f; right of it the trailing update is H_jk -= l_j l_k,
// and left of it, where the columns of accepted proposals have been used up, the
// same matrix collects S_jp = sum_e L_je Minv_ep, the sums of the forward
// substitution: row i of S gives row m of the inverse, Minv_mp = -f S_ip,
// Minv_mi = f, and S_jp += l_j Minv_mp.  So a step is one rank-1 update of the
// rows below i by v = (Minv_m, f, -l), with two barriers.
//
// What bounds a step is the FP64 pipe (2 lanes per clock on the one SM) and the
// chain decision -> 1 / sqrt -> scaled column.  Warp 0 keeps the diagonal in
// registers, tests all proposals at once (a rejected one costs nothing), and
// forms the next step's f while the other warps update; with every warp taking
// every decision and square root, one thread per column substituting forward at
// the end, and one load in flight per element of H, a round took 258 us at b = 64
// and 100 us at b = 32; now 104 and 38 us (N = 2M, k = 2000).
//
// Minv is b x b, row-major [a][e], zeros above the diagonal and beyond the
// accepted count.
template <int Q>
__global__ void __launch_bounds__(kFactorThreads)
rp_factor_kernel(const double* __restrict__ kss, const double* __restrict__ hpart, int b,
                 uint64_t seed, const double* __restrict__ uniforms, double tol,
                 double floor_rel, int64_t k_max, const int64_t* __restrict__ props, RoundState* st,
                 double* __restrict__ minv, float* __restrict__ minv_f,
                 int64_t* __restrict__ sacc, int64_t* __restrict__ piv,
                 int32_t* __restrict__ hm) {
    if (st->done) return;
    constexpr int B = 32 * Q;
    extern __shared__ double A[];     // b x (b + 1)
    __shared__ double thr[B], l[B], v[B];
    __shared__ int accpos[B];
    __shared__ double s_f;
    __shared__ int s_i;
    const int P = b + 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int round = st->cur;
    const int64_t r = st->rank;
    const int nz = (int)((r + kColChunk - 1) / kColChunk);
    // H = K(S',S') - sum of the column chunks' products, each element in chunk
    // order; kPer elements per thread and four chunks ahead keep 32 loads in flight
    constexpr int kPer = 8;
    for (int e0 = tid; e0 < b * b; e0 += kPer * kFactorThreads) {
        double x[kPer];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int e = e0 + j * kFactorThreads;
            x[j] = (e < b * b) ? kss[e] : 0.0;
        }
        int z = 0;
        for (; z + 4 <= nz; z += 4) {
            double y[4][kPer];
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int j = 0; j < kPer; ++j) {
                    const int e = e0 + j * kFactorThreads;
                    y[q][j] = (e < b * b) ? hpart[(int64_t)(z + q) * b * b + e] : 0.0;
                }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int j = 0; j < kPer; ++j) x[j] -= y[q][j];
        }
        for (; z < nz; ++z)
#pragma unroll
            for (int j = 0; j < kPer; ++j) {
                const int e = e0 + j * kFactorThreads;
                if (e < b * b) x[j] -= hpart[(int64_t)z * b * b + e];
            }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int e = e0 + j * kFactorThreads;
            if (e < b * b) {
                A[(e / b) * P + e % b] = x[j];
                minv[e] = 0.0;
                minv_f[e] = 0.f;
            }
        }
    }
    __syncthreads();
    // accepted iff H0_ii u < H_ii, H_ii > tol and H_ii above the rounding floor
    if (tid < b) {
        const double u = uniforms ? uniforms[((int64_t)round * 2 + 1) * b + tid]
                                  : philox_uniform(seed, (uint32_t)round, 1u, (uint32_t)tid);
        thr[tid] = fmax(fmax(A[tid * P + tid] * u, tol), floor_rel * kss[tid * b + tid]);
    }
    __syncthreads();
    const int cap = (int)min((int64_t)b, k_max - r);
    int m = 0;
    unsigned acc[Q];    // accepted proposals so far, 32 per word
    double dg[Q];       // warp 0: the diagonal, proposal lane + 32 q
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        acc[q] = 0u;
        dg[q] = (warp == 0 && lane + 32 * q < b) ? A[(lane + 32 * q) * P + lane + 32 * q] : 0.0;
    }
    // warp 0: the first acceptable proposal from i0 on (mm accepted before it)
    auto decide = [&](int i0, int mm) {
        int i = -1;
        double hii = 1.0;
#pragma unroll
        for (int q = Q - 1; q >= 0; --q) {
            const int p = lane + 32 * q;
            const unsigned ok = __ballot_sync(0xffffffffu, p >= i0 && p < b && mm < cap && dg[q] > thr[min(p, b - 1)]);
            if (ok) {
                i = 32 * q + __ffs(ok) - 1;
                hii = __shfl_sync(0xffffffffu, dg[q], __ffs(ok) - 1);
            }
        }
        const double f = rsqrt(hii);
        if (lane == 0) {
            s_i = i;
            s_f = f;
        }
    };
    if (warp == 0) decide(0, 0);
    __syncthreads();
    while (s_i >= 0) {
        const int i = s_i;
        const double f = s_f;
        if (tid < b) {
            const int c = tid;
            double vc = 0.0;
            if (c > i) {
                vc = -(A[c * P + i] * f);
            } else if (c == i || (acc[Q == 1 ? 0 : c >> 5] >> (c & 31) & 1u)) {
                vc = c == i ? f : -(f * A[i * P + c]);
                int t = 0;   // accepted before c
#pragma unroll
                for (int q = 0; q < Q; ++q)
                    t += __popc(q < (c >> 5) ? acc[q] : q == (c >> 5) ? acc[q] & ((1u << (c & 31)) - 1u) : 0u);
                minv[m * b + t] = vc;
                minv_f[m * b + t] = (float)vc;
            }
            l[c] = c > i ? -vc : 0.0;
            v[c] = vc;
        }
        if (tid == 0) accpos[m] = i;
        ++m;
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (q == i >> 5) acc[q] |= 1u << (i & 31);
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int p = lane + 32 * q;
                if (p > i && p < b) dg[q] = fma(-l[p], l[p], dg[q]);
            }
            decide(i + 1, m);
        } else {
            double vq[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) vq[q] = lane + 32 * q < b ? v[lane + 32 * q] : 0.0;
            for (int jj = i + warp; jj < b; jj += kFactorThreads / 32 - 1) {
                const double lj = l[jj];
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const int c = lane + 32 * q;
                    if (32 * q < jj && c < b)   // columns past jj are never read
                        A[jj * P + c] = fma(lj, vq[q], c == i ? 0.0 : A[jj * P + c]);
                }
            }
        }
        __syncthreads();
    }
    if (tid < m) {
        const int64_t sp = props[accpos[tid]];
        sacc[tid] = sp;
        piv[r + tid] = sp;
    }
    if (tid == 0) {
        st->r_old = r;
        st->nacc = m;
        st->rank = r + m;
        st->cur = round + 1;
        hm[round] = m;
    }
}

// Accept / reject, Cholesky and inverse for kSmallBlock < b <= kMaxBlock: with H, the compacted
// factor LC and the inverse MS in a global workspace (b^2 doubles each,
// L2-resident) instead of shared memory, and 32 x 32 threads over the
// trailing update.  __syncthreads orders the CTA's global accesses as it does
// its shared ones.
__global__ void __launch_bounds__(kBigFactorThreads)
rp_factor_big_kernel(const double* __restrict__ kss, const double* __restrict__ hpart, int b,
                     uint64_t seed, const double* __restrict__ uniforms, double tol,
                     double floor_rel, int64_t k_max, const int64_t* __restrict__ props, RoundState* st,
                     double* __restrict__ minv, float* __restrict__ minv_f,
                     int64_t* __restrict__ sacc, int64_t* __restrict__ piv,
                     int32_t* __restrict__ hm, double* H, double* MS, double* LC) {
    if (st->done) return;
    __shared__ double H0[kMaxBlock];
    __shared__ double us[kMaxBlock];
    __shared__ double kfl[kMaxBlock];
    __shared__ int accpos[kMaxBlock];
    __shared__ int s_dec, s_m;
    const int tid = threadIdx.x;
    const int nt = blockDim.x;
    const int round = st->cur;
    const int64_t r = st->rank;
    const int nz = (int)((r + kColChunk - 1) / kColChunk);
    for (int e = tid; e < b * b; e += nt) {
        double v = kss[e];
        for (int z = 0; z < nz; ++z) v -= hpart[(int64_t)z * b * b + e];
        H[e] = v;
    }
    __syncthreads();
    for (int p = tid; p < b; p += nt) {
        H0[p] = H[p * b + p];
        kfl[p] = floor_rel * kss[p * b + p];
        us[p] = uniforms ? uniforms[((int64_t)round * 2 + 1) * b + p] : philox_uniform(seed, (uint32_t)round, 1u, (uint32_t)p);
    }
    if (tid == 0) s_m = 0;
    __syncthreads();
    const int64_t cap = k_max - r;
    for (int i = 0; i < b; ++i) {
        __syncthreads();
        if (tid == 0) {
            const double u = us[i];
            const double hii = H[i * b + i];
            const int acc = (s_m < cap) && (H0[i] * u < hii) && (hii > tol) && (hii > kfl[i]);
            s_dec = acc;
            if (acc) accpos[s_m++] = i;
        }
        __syncthreads();
        if (s_dec) {
            const double f = 1.0 / sqrt(H[i * b + i]);
            __syncthreads();
            for (int j = i + tid; j < b; j += nt) H[j * b + i] *= f;
            __syncthreads();
            for (int jj = i + 1 + (tid >> 5); jj < b; jj += 32)
                for (int kk = i + 1 + (tid & 31); kk <= jj; kk += 32) H[jj * b + kk] -= H[jj * b + i] * H[kk * b + i];
            __syncthreads();
        }
    }
    const int nacc = s_m;
    for (int e = tid; e < b * b; e += nt) {
        MS[e] = 0.0;
        const int a = e / b, c = e - a * b;
        LC[e] = (a < nacc && c < nacc) ? H[accpos[a] * b + accpos[c]] : 0.0;
    }
    __syncthreads();
    if (tid < nacc) {
        const int t = tid;
        MS[t * b + t] = 1.0 / LC[t * b + t];
        for (int a = t + 1; a < nacc; ++a) {
            const double* la = LC + a * b;
            double sum = 0.0;
            for (int e = t; e < a; ++e) sum += la[e] * MS[e * b + t];
            MS[a * b + t] = -sum / la[a];
        }
    }
    __syncthreads();
    for (int e = tid; e < b * b; e += nt) {
        minv[e] = MS[e];
        minv_f[e] = (float)MS[e];
    }
    if (tid < nacc) {
        const int64_t sp = props[accpos[tid]];
        sacc[tid] = sp;
        piv[r + tid] = sp;
    }
    if (tid == 0) {
        st->r_old = r;
        st->nacc = nacc;
        st->rank = r + nacc;
        st->cur = round + 1;
        hm[round] = nacc;
    }
}

// ---- residual update over all row blocks -----------------------------------
// CTA = 128 rows x up to 64 accepted columns; thread (ty, tx) of 16 x 16 owns
// rows ty + 16i (i < 8) and columns tx + 16j (j < 4).
//
// A round that accepts more than 64 columns is updated in passes of 64
// (group g = columns r + 64g ...).  With L_i = [[L00, 0], [L10, L11]] the new
// columns satisfy G0 = T0 L00^{-T} and G1 = (T1 - G0 L10^T) L11^{-T}; pass g
// therefore runs the one-group update against the factor's first r + 64g
// columns (which include the previous passes' output, whose rows at S_g are
// L10) with the pivots of group g and the diagonal block g of L_i^{-1}.
__device__ __forceinline__ bool group_view(int64_t r_old, int nacc_all, int group, int64_t& r, int& nacc) {
    r = r_old + (int64_t)kGroup * group;
    nacc = min(kGroup, nacc_all - kGroup * group);
    return nacc > 0;
}
constexpr int kUpdCols = 32;   // factor columns staged at a time

__global__ void __launch_bounds__(256)
rp_update_kernel(double* __restrict__ F, int64_t ldF, const float* __restrict__ X, int64_t N, int d,
                 double scale, const int64_t* __restrict__ sacc, const double* __restrict__ minv, int b,
                 const RoundState* st, double* __restrict__ dvec, double* __restrict__ dblk, int group) {
    if (st->done) return;
    int64_t r;
    int nacc;
    if (!group_view(st->r_old, st->nacc, group, r, nacc)) return;
    {   // this pass's pivots and diagonal block of L_i^{-1} (leading dimension b)
        const int64_t o = (int64_t)kGroup * group;
        sacc += o;
        minv += o * b + o;
    }
    constexpr int KC = kUpdCols;
    extern __shared__ __align__(16) unsigned char smraw[];
    // region 1 (phase A: X rows, kFeat features at a time; phase B: F tiles),
    // then Tm, then Minv
    constexpr int dp = kFeat + 1;
    const size_t reg1_a = (size_t)(kRowBlock + kGroup) * dp * sizeof(float);
    const size_t reg1_b = (size_t)(kRowBlock + kGroup) * (KC + 1) * sizeof(double);
    const size_t reg1 = reg1_a > reg1_b ? reg1_a : reg1_b;
    float* xr = reinterpret_cast<float*>(smraw);
    float* xs = xr + kRowBlock * dp;
    double* At = reinterpret_cast<double*>(smraw);
    double* Bt = At + kRowBlock * (KC + 1);
    double* Tm = reinterpret_cast<double*>(smraw + ((reg1 + 15) / 16) * 16);   // 128 x (64+1)
    double* Mv = Tm + kRowBlock * (kGroup + 1);                         // 64 x (64+1)
    __shared__ double rowsq_s[kRowBlock];

    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int64_t row0 = (int64_t)blockIdx.x * kRowBlock;
    const int nrows = (int)min((int64_t)kRowBlock, N - row0);

    // phase A: K(R, S_i) into Tm
    for (int e = tid; e < nacc * nacc; e += 256) {
        const int a = e / nacc, q = e - a * nacc;
        Mv[a * (kGroup + 1) + q] = minv[a * b + q];
    }
    {
        double acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0;
        for (int c0 = 0; c0 < d; c0 += kFeat) {
            const int w = min(kFeat, d - c0);
            __syncthreads();
            for (int e = tid; e < kRowBlock * w; e += 256) {
                const int rr = e / w, k = e - rr * w;
                xr[rr * dp + k] = (rr < nrows) ? X[(row0 + rr) * d + c0 + k] : 0.f;
            }
            for (int e = tid; e < nacc * w; e += 256) {
                const int q = e / w, k = e - q * w;
                xs[q * dp + k] = X[sacc[q] * d + c0 + k];
            }
            __syncthreads();
            for (int k = 0; k < w; ++k) {
                double vr[8], vs[4];
#pragma unroll
                for (int i = 0; i < 8; ++i) vr[i] = (double)xr[(ty + 16 * i) * dp + k];
#pragma unroll
                for (int j = 0; j < 4; ++j) vs[j] = (double)xs[min(tx + 16 * j, kGroup - 1) * dp + k];
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const double t = vr[i] - vs[j];
                        acc[i][j] += t * t;
                    }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int c = tx + 16 * j;
                Tm[(ty + 16 * i) * (kGroup + 1) + c] = c < nacc ? exp(-scale * acc[i][j]) : 0.0;
            }
    }
    __syncthreads();

    // phase B: acc = F(R, 0:r) F(S_i, 0:r)^T
    double acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    for (int64_t c0 = 0; c0 < r; c0 += KC) {
        const int nc = (int)min((int64_t)KC, r - c0);
        for (int e = tid; e < kRowBlock * KC; e += 256) {
            const int rr = e / KC, c = e - rr * KC;
            At[rr * (KC + 1) + c] = (rr < nrows && c < nc) ? F[(row0 + rr) * ldF + c0 + c] : 0.0;
        }
        for (int e = tid; e < kGroup * KC; e += 256) {
            const int q = e / KC, c = e - q * KC;
            Bt[q * (KC + 1) + c] = (q < nacc && c < nc) ? F[sacc[q] * ldF + c0 + c] : 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int c = 0; c < KC; ++c) {
            double va[8], vb[4];
#pragma unroll
            for (int i = 0; i < 8; ++i) va[i] = At[(ty + 16 * i) * (KC + 1) + c];
#pragma unroll
            for (int j = 0; j < 4; ++j) vb[j] = Bt[(tx + 16 * j) * (KC + 1) + c];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] += va[i] * vb[j];
        }
        __syncthreads();
    }
    // phase C: Tm -= acc (own entries)
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) Tm[(ty + 16 * i) * (kGroup + 1) + tx + 16 * j] -= acc[i][j];
    __syncthreads();
    // phase D: G = Tm Minv^T
    double g[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) g[i][j] = 0;
    for (int e = 0; e < nacc; ++e) {
        double vt[8], vm[4];
#pragma unroll
        for (int i = 0; i < 8; ++i) vt[i] = Tm[(ty + 16 * i) * (kGroup + 1) + e];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int a = tx + 16 * j;
            vm[j] = (a < nacc) ? Mv[a * (kGroup + 1) + e] : 0.0;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) g[i][j] += vt[i] * vm[j];
    }
    // phase E: store the new columns, update d, block sum
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int rr = ty + 16 * i;
        double sq = 0.0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int a = tx + 16 * j;
            if (a < nacc && rr < nrows) {
                F[(row0 + rr) * ldF + r + a] = g[i][j];
                sq += g[i][j] * g[i][j];
            }
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        if (tx == 0) rowsq_s[rr] = sq;
    }
    __syncthreads();
    double nd = 0.0;
    if (tid < kRowBlock && tid < nrows) {
        const int64_t gi = row0 + tid;
        nd = fmax(dvec[gi] - rowsq_s[tid], 0.0);
        dvec[gi] = nd;
    }
    // block sum of the new d over the first 128 threads (4 warps)
    __shared__ double wsum[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nd += __shfl_xor_sync(0xffffffffu, nd, o);
    if ((tid & 31) == 0) wsum[tid >> 5] = nd;
    __syncthreads();
    if (tid == 0) dblk[blockIdx.x] = ((wsum[0] + wsum[1]) + (wsum[2] + wsum[3]));
}

static size_t update_smem() {
    const int dp = kFeat + 1;
    const size_t reg1_a = (size_t)(kRowBlock + kGroup) * dp * sizeof(float);
    const size_t reg1_b = (size_t)(kRowBlock + kGroup) * (kUpdCols + 1) * sizeof(double);
    const size_t reg1 = ((std::max(reg1_a, reg1_b) + 15) / 16) * 16;
    return reg1 + (size_t)kRowBlock * (kGroup + 1) * sizeof(double) +
           (size_t)kGroup * (kGroup + 1) * sizeof(double);
}

// One factorisation's buffers and launches.  setup() allocates (the sizes do not
// depend on the round count), init() starts the round state, round() enqueues one
// round (its index is in the round state, so the launches of every round are the
// same), closing() records the last round's error.
template <typename T>
struct RpRun {
    kevd_ctx* ctx;
    const float* X;
    int64_t N;
    int d;
    double scale;
    kevd_rpchol_params p;
    T* F;
    int64_t ldF;
    bool tc_allowed;

    int b = 0, n_split = 0;
    int64_t nblk = 0;
    bool small = false, use_tc = false;
    double floor_rel = 0.0;
    double *dvec = nullptr, *dblk = nullptr, *hpart = nullptr, *kss = nullptr, *minv = nullptr, *err = nullptr,
           *unif = nullptr, *hbig = nullptr;
    RoundState* rs = nullptr;
    int64_t *props = nullptr, *sacc = nullptr, *piv = nullptr;
    float* minv_f = nullptr;
    int32_t* hm = nullptr;
    int* tc_err = nullptr;
    size_t fsm = 0, hsm = 0, usm = 0;

    int setup() {
        b = p.block;
        floor_rel = sizeof(T) == 4 ? kMixedFloor : 0.0;
        nblk = (N + kRowBlock - 1) / kRowBlock;
        n_split = (int)((p.k_max + kColChunk - 1) / kColChunk);
        // few proposals in FP64: two kernels a round that touch the accepted columns
        // only (kevd_rpchol_small.cu).  The FP32 form keeps the general kernels: a
        // pivot sequence follows every rounding of its residual diagonal.
        small = sizeof(T) == 8 && rpchol_small_supported(b);
        int st = KEVD_OK;
        dvec = arena_get<double>(ctx, "rp.d", N, &st);
        dblk = arena_get<double>(ctx, "rp.dblk", small ? rpchol_small_blocks(N) : nblk, &st);
        rs = arena_get<RoundState>(ctx, "rp.state", 1, &st);
        props = arena_get<int64_t>(ctx, "rp.props", kMaxBlock, &st);
        sacc = arena_get<int64_t>(ctx, "rp.sacc", kMaxBlock, &st);
        piv = arena_get<int64_t>(ctx, "rp.piv", p.k_max, &st);
        hpart = arena_get<double>(ctx, "rp.hpart", (size_t)std::max(n_split, 1) * b * b, &st);
        kss = arena_get<double>(ctx, "rp.kss", (size_t)b * b, &st);
        minv = arena_get<double>(ctx, "rp.minv", (size_t)b * b, &st);
        minv_f = arena_get<float>(ctx, "rp.minvf", (size_t)b * b, &st);
        err = arena_get<double>(ctx, "rp.err", p.max_rounds, &st);
        hm = arena_get<int32_t>(ctx, "rp.hm", p.max_rounds, &st);
        tc_err = arena_get<int>(ctx, "rp.tcerr", 1, &st);
        if (p.uniforms) unif = arena_get<double>(ctx, "rp.unif", (size_t)p.max_rounds * 2 * b, &st);
        // H, the compacted factor and the inverse of a large block
        if (b > kSmallBlock) hbig = arena_get<double>(ctx, "rp.hbig", (size_t)3 * b * b, &st);
        if (st != KEVD_OK) return st;
        fsm = b > kSmallBlock ? 0 : (size_t)b * (b + 1) * sizeof(double);
        if (b <= kSmallBlock)
            KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(factor()), std::max(fsm, (size_t)1024)));
        hsm = hgram_smem<T>(b);
        KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&rp_hgram_kernel<T>), (int)hsm));
        usm = update_smem();
        if constexpr (sizeof(T) == 8)
            KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&rp_update_kernel), (int)usm));
        // FP32 factors take the tensor-core residual update when the layout allows
        // TMA and the kernel is not nearly diagonal (kernel_density_kernel)
        use_tc = sizeof(T) == 4 && tc_allowed && update_tc_supported(reinterpret_cast<const float*>(F), ldF, d);
        if (use_tc) KEVD_TRY(reserve_update_tc(ctx, N, p.k_max));
        return KEVD_OK;
    }

    int init(cudaStream_t s) {
        if (unif)
            KEVD_CUDA(ctx, cudaMemcpyAsync(unif, p.uniforms, (size_t)p.max_rounds * 2 * b * sizeof(double),
                                           cudaMemcpyHostToDevice, s));
        KEVD_CUDA(ctx, cudaMemsetAsync(err, 0, p.max_rounds * sizeof(double), s));
        KEVD_CUDA(ctx, cudaMemsetAsync(hm, 0, p.max_rounds * sizeof(int32_t), s));
        KEVD_CUDA(ctx, cudaMemsetAsync(tc_err, 0, sizeof(int), s));
        if (small) return launch_rpchol_small_init(ctx, dvec, dblk, N, rs, s);
        rp_init_kernel<<<ctx->num_sms * 4, 256, 0, s>>>(dvec, dblk, N, nblk, rs);
        KEVD_LAUNCH(ctx);
        return KEVD_OK;
    }

    // `index` is read by the two-kernel round alone
    int round(int index, cudaStream_t s) {
        if (small) {
            KEVD_TRY(propose_small(index, b, p.max_rounds, s));
            return launch_rpchol_small_update(ctx, (double*)F, ldF, X, N, d, scale, sacc, minv, b, rs, dvec, dblk, s);
        }
        {
            ProfScope ps(ctx, "rp_sample", s);
            sample(0, b, s);
            KEVD_LAUNCH(ctx);
        }
        {
            ProfScope ps(ctx, "rp_hgram", s);
            const int n_kss = 32;   // CTAs sharing the FP64 K(S', S') block
            rp_hgram_kernel<T><<<n_split + n_kss, 256, hsm, s>>>(F, ldF, X, d, scale, props, b, n_split, rs, hpart, kss);
            KEVD_LAUNCH(ctx);
        }
        {
            ProfScope ps(ctx, "rp_factor", s);
            if (hbig)
                rp_factor_big_kernel<<<1, kBigFactorThreads, 0, s>>>(kss, hpart, b, p.seed, unif, p.tol, floor_rel,
                                                                      p.k_max, props, rs, minv, minv_f, sacc, piv, hm,
                                                                      hbig, hbig + (size_t)b * b,
                                                                      hbig + (size_t)2 * b * b);
            else
                factor()<<<1, kFactorThreads, fsm, s>>>(kss, hpart, b, p.seed, unif, p.tol, floor_rel, p.k_max, props,
                                                        rs, minv, minv_f, sacc, piv, hm);
            KEVD_LAUNCH(ctx);
        }
        if (use_tc)
            return launch_update_tc(ctx, reinterpret_cast<float*>(F), ldF, N, p.k_max, X, d, scale, sacc, minv_f, b, rs,
                                    dvec, dblk, tc_err, s);
        ProfScope ps(ctx, "rp_update", s);
        if constexpr (sizeof(T) == 4) {
            KEVD_TRY(launch_update_f32(ctx, (float*)F, ldF, X, N, d, scale, sacc, minv_f, b, rs, dvec, dblk, s));
        } else {
            for (int g = 0; g < (b + kGroup - 1) / kGroup; ++g) {
                rp_update_kernel<<<(int)nblk, 256, usm, s>>>(F, ldF, X, N, d, scale, sacc, minv, b, rs, dvec, dblk, g);
                KEVD_LAUNCH(ctx);
            }
        }
        return KEVD_OK;
    }

    int closing(int rounds, cudaStream_t s) {
        if (small) return propose_small(rounds, 0, rounds, s);
        sample(1, 0, s);
        KEVD_LAUNCH(ctx);
        return KEVD_OK;
    }

    auto factor() const { return b <= 32 ? &rp_factor_kernel<1> : b <= 64 ? &rp_factor_kernel<2> : &rp_factor_kernel<4>; }
    void sample(int closing, int nb, cudaStream_t s) {
        rp_sample_kernel<<<1, kSampleThreads, 0, s>>>(dvec, dblk, N, nblk, closing, nb, p.seed, unif, props, rs, p.k_max,
                                                      p.max_rounds, p.err_target, floor_rel, err);
    }
    int propose_small(int round, int nb, int limit, cudaStream_t s) {
        return launch_rpchol_small_propose(ctx, (const double*)F, ldF, X, N, d, scale, dvec, dblk, round, nb, p.seed, unif,
                                           p.tol, p.k_max, limit, p.err_target, rs, minv, sacc, piv, err, hm, s);
    }
};

template <typename T>
static int rpchol_impl(kevd_ctx* ctx, const float* X, int64_t N, int d, double scale,
                       const kevd_rpchol_params* p, T* F, int64_t ldF, int64_t* piv_h,
                       double* err_h, int32_t* hm_h, kevd_rpchol_result* res, cudaStream_t s, bool tc_allowed = true) {
    RpRun<T> run{ctx, X, N, d, scale, *p, F, ldF, tc_allowed};
    KEVD_TRY(run.setup());
    KEVD_TRY(run.init(s));
    int* done_h = static_cast<int*>(ctx->pinned);
    // rounds between two reads of the done flag (each read waits for the stream):
    // a small round is short, and the rounds after the stop return at once
    const int poll = run.small ? 16 : 4;
    int round = 0;
    for (; round < p->max_rounds; ++round) {
        KEVD_TRY(run.round(round, s));
        if (round % poll == poll - 1) {
            KEVD_CUDA(ctx, cudaMemcpyAsync(done_h, &run.rs->done, sizeof(int), cudaMemcpyDeviceToHost, s));
            KEVD_CUDA(ctx, cudaStreamSynchronize(s));
            if (*done_h) break;
        }
    }
    KEVD_TRY(run.closing(std::min(round, p->max_rounds), s));
    RoundState hs;
    int herr = 0;
    KEVD_CUDA(ctx, cudaMemcpyAsync(&hs, run.rs, sizeof(RoundState), cudaMemcpyDeviceToHost, s));
    KEVD_CUDA(ctx, cudaMemcpyAsync(&herr, run.tc_err, sizeof(int), cudaMemcpyDeviceToHost, s));
    KEVD_CUDA(ctx, cudaStreamSynchronize(s));
    if (herr != 0)
        return set_error(ctx, KEVD_ERR_TIMEOUT, "rpchol: tensor-core update pipeline timed out (code %d)", herr);
    if (hs.rank > 0 && piv_h)
        KEVD_CUDA(ctx, cudaMemcpy(piv_h, run.piv, hs.rank * sizeof(int64_t), cudaMemcpyDeviceToHost));
    if (err_h) KEVD_CUDA(ctx, cudaMemcpy(err_h, run.err, hs.rounds * sizeof(double), cudaMemcpyDeviceToHost));
    if (hm_h) KEVD_CUDA(ctx, cudaMemcpy(hm_h, run.hm, hs.rounds * sizeof(int32_t), cudaMemcpyDeviceToHost));
    if (res) {
        res->rank = hs.rank;
        res->rounds = hs.rounds;
        res->trace_error = hs.total / (double)N;
    }
    return KEVD_OK;
}

int run_rpchol(kevd_ctx* ctx, const float* X, int64_t N, int d, double scale,
               const kevd_rpchol_params* p, void* F, int64_t ldF, int64_t* piv, double* err,
               int32_t* accepted, kevd_rpchol_result* res, cudaStream_t s) {
    if (!X || !p || !F || N < 1 || d < 1 || d > kMaxFeatures)
        return set_error(ctx, KEVD_ERR_ARG, "rpchol: need X, F, N >= 1 and 1 <= d <= %d", kMaxFeatures);
    if (p->block < 1 || p->block > kMaxBlock)
        return set_error(ctx, KEVD_ERR_ARG, "rpchol: block must be in [1, %d]", kMaxBlock);
    if (p->k_max < 1 || ldF < p->k_max || p->max_rounds < 1)
        return set_error(ctx, KEVD_ERR_ARG, "rpchol: need k_max >= 1, ldF >= k_max, max_rounds >= 1");
    if (p->precision == KEVD_FP64)
        return rpchol_impl<double>(ctx, X, N, d, scale, p, (double*)F, ldF, piv, err, accepted, res, s);
    if (p->precision == KEVD_MIXED) {
        bool diag = false;
        if (update_tc_supported((const float*)F, ldF, d)) KEVD_TRY(kernel_nearly_diagonal(ctx, X, N, d, scale, s, &diag));
        return rpchol_impl<float>(ctx, X, N, d, scale, p, (float*)F, ldF, piv, err, accepted, res, s, !diag);
    }
    return set_error(ctx, KEVD_ERR_ARG, "rpchol: unknown precision %d", p->precision);
}

// Many factorisations at once, each with a workspace and a stream of its own.
// With use_graph, kGraphRounds rounds of every job are captured as parallel
// branches of one CUDA graph (a round's launches do not depend on its index) and
// the graph is launched until every job has stopped; without, the same rounds are
// issued directly on the jobs' streams.  The host looks at a chunk's results while
// the next one runs.  Eight jobs of N = 14,000 .. 91,000 to rank 113 .. 981, b =
// 32: 13.6 ms a call, with and without the graph (31.3 ms with one graph of all
// max_rounds rounds, 136 for rank 1,000 of which about 35 do work: allocation,
// capture and instantiation took longer than the rounds).
//
// The jobs' workspaces, streams and pinned buffers stay with the context (grown to
// the largest batch seen) while they are at most kBatchKeepJobs and hold at most
// kBatchKeepBytes; beyond, and after an error, they are freed at the end of the call.
constexpr int kGraphRounds = 4;
constexpr size_t kBatchKeepBytes = (size_t)1 << 30;
constexpr int kBatchKeepJobs = 64;

struct BatchSlot {
    kevd_ctx* c = nullptr;
    cudaStream_t st = nullptr;
    cudaEvent_t ev = nullptr;            // joins the job's branch
    cudaEvent_t seen[2] = {};            // chunk's results copied (direct launches)
    RoundState* state_h = nullptr;       // pinned: two chunks' states, the error flag, the pivots
    int* tcerr_h = nullptr;
    int64_t* piv_h = nullptr;
    size_t pinned = 0;
};
struct BatchPool {
    std::vector<BatchSlot> slots;
    cudaStream_t cs = nullptr;           // capture stream
    cudaEvent_t fork = nullptr, seen[2] = {};
};

static void free_batch_slot(BatchSlot& x) {
    if (x.ev) cudaEventDestroy(x.ev);
    for (cudaEvent_t e : x.seen)
        if (e) cudaEventDestroy(e);
    if (x.st) cudaStreamDestroy(x.st);
    if (x.state_h) cudaFreeHost(x.state_h);
    if (x.c) {
        x.c->arena.release();
        delete x.c;
    }
    x = BatchSlot();
}

void free_batch_pool(kevd_ctx* ctx) {
    BatchPool* pool = static_cast<BatchPool*>(ctx->batch_pool);
    if (!pool) return;
    for (auto& x : pool->slots) free_batch_slot(x);
    if (pool->cs) cudaStreamDestroy(pool->cs);
    if (pool->fork) cudaEventDestroy(pool->fork);
    for (cudaEvent_t e : pool->seen)
        if (e) cudaEventDestroy(e);
    delete pool;
    ctx->batch_pool = nullptr;
}

// The pool with n ready slots, each with pinned room for its job's pivots.
static int batch_pool(kevd_ctx* ctx, const kevd_rpchol_job* jobs, int n, BatchPool** out) {
    if (!ctx->batch_pool) ctx->batch_pool = new BatchPool();
    BatchPool& pool = *static_cast<BatchPool*>(ctx->batch_pool);
    *out = &pool;
    auto event = [&](cudaEvent_t* e) { return *e ? cudaSuccess : cudaEventCreateWithFlags(e, cudaEventDisableTiming); };
    // the capture runs on a stream of its own (the caller's stream may be the
    // legacy default stream, which cannot be captured)
    if (!pool.cs) KEVD_CUDA(ctx, cudaStreamCreateWithFlags(&pool.cs, cudaStreamNonBlocking));
    KEVD_CUDA(ctx, event(&pool.fork));
    for (cudaEvent_t& e : pool.seen) KEVD_CUDA(ctx, event(&e));
    if ((int)pool.slots.size() < n) pool.slots.resize(n);
    for (int q = 0; q < n; ++q) {
        BatchSlot& x = pool.slots[q];
        if (!x.c) {
            x.c = new kevd_ctx();
            x.c->device = ctx->device;
            x.c->num_sms = ctx->num_sms;
        }
        if (!x.st) KEVD_CUDA(ctx, cudaStreamCreateWithFlags(&x.st, cudaStreamNonBlocking));
        KEVD_CUDA(ctx, event(&x.ev));
        for (cudaEvent_t& e : x.seen) KEVD_CUDA(ctx, event(&e));
        const size_t head = 2 * sizeof(RoundState) + 16, want = head + (size_t)jobs[q].k_max * sizeof(int64_t);
        if (x.pinned < want) {
            if (x.state_h) cudaFreeHost(x.state_h);
            x.state_h = nullptr;
            x.pinned = 0;
            KEVD_CUDA(ctx, cudaMallocHost(&x.state_h, want));
            x.pinned = want;
            x.tcerr_h = reinterpret_cast<int*>(x.state_h + 2);
            x.piv_h = reinterpret_cast<int64_t*>(reinterpret_cast<uint8_t*>(x.state_h) + head);
        }
    }
    return KEVD_OK;
}

static int rpchol_batched(kevd_ctx* ctx, kevd_rpchol_job* jobs, int n_jobs, bool use_graph, BatchPool& pool,
                          int* cnt, cudaGraph_t* graph, cudaGraphExec_t* exec, cudaStream_t s) {
    // the residual-update form of every job, decided before any capture
    KEVD_CUDA(ctx, cudaMemsetAsync(cnt, 0, n_jobs * sizeof(int), s));
    for (int q = 0; q < n_jobs; ++q) {
        const kevd_rpchol_job& j = jobs[q];
        if (j.N < 2 || !update_tc_supported((const float*)j.F, j.ldF, j.d)) continue;
        kernel_density_kernel<<<1, 256, 0, s>>>(j.X, j.N, j.d, j.scale, cnt + q);
        KEVD_LAUNCH(ctx);
    }
    std::vector<int> hcnt(n_jobs);
    KEVD_CUDA(ctx, cudaMemcpyAsync(hcnt.data(), cnt, n_jobs * sizeof(int), cudaMemcpyDeviceToHost, s));
    KEVD_CUDA(ctx, cudaStreamSynchronize(s));
    std::vector<RpRun<float>> runs;
    runs.reserve(n_jobs);
    auto job_error = [&](int q, int rc) {
        return set_error(ctx, rc, "rpchol_batched: job %d: %s", q, pool.slots[q].c->last_error.c_str());
    };
    for (int q = 0; q < n_jobs; ++q) {
        const kevd_rpchol_job& j = jobs[q];
        kevd_rpchol_params p;
        std::memset(&p, 0, sizeof(p));
        p.k_max = j.k_max;
        p.block = j.block;
        p.max_rounds = j.max_rounds;
        p.tol = 1e-10;
        p.seed = j.seed;
        p.precision = KEVD_MIXED;
        runs.push_back(RpRun<float>{pool.slots[q].c, j.X, j.N, j.d, j.scale, p, (float*)j.F, j.ldF,
                                    j.N < 2 || 2 * hcnt[q] >= kDensityPairs});
        int rc = runs[q].setup();
        if (rc == KEVD_OK) rc = runs[q].init(s);
        if (rc != KEVD_OK) return job_error(q, rc);
    }
    // one chunk of job q on its stream: kGraphRounds rounds and the state behind them
    auto chunk = [&](int q, int buf) -> int {
        BatchSlot& x = pool.slots[q];
        for (int i = 0; i < kGraphRounds; ++i) {
            const int rc = runs[q].round(0, x.st);
            if (rc != KEVD_OK) return job_error(q, rc);
        }
        ctx->launches += x.c->launches;
        x.c->launches = 0;
        KEVD_CUDA(ctx, cudaMemcpyAsync(x.state_h + buf, runs[q].rs, sizeof(RoundState), cudaMemcpyDeviceToHost, x.st));
        return KEVD_OK;
    };
    auto fork_from = [&](cudaStream_t root) -> int {
        KEVD_CUDA(ctx, cudaEventRecord(pool.fork, root));
        for (int q = 0; q < n_jobs; ++q) KEVD_CUDA(ctx, cudaStreamWaitEvent(pool.slots[q].st, pool.fork, 0));
        return KEVD_OK;
    };
    auto join_to = [&](cudaStream_t root) -> int {
        for (int q = 0; q < n_jobs; ++q) {
            KEVD_CUDA(ctx, cudaEventRecord(pool.slots[q].ev, pool.slots[q].st));
            KEVD_CUDA(ctx, cudaStreamWaitEvent(root, pool.slots[q].ev, 0));
        }
        return KEVD_OK;
    };
    // every job stops by itself in the round after its last one
    int max_rounds = 0;
    for (int q = 0; q < n_jobs; ++q) max_rounds = std::max(max_rounds, jobs[q].max_rounds);
    const int max_chunks = max_rounds / kGraphRounds + 1;
    if (use_graph) {
        const int64_t launched = ctx->launches;
        KEVD_CUDA(ctx, cudaStreamBeginCapture(pool.cs, cudaStreamCaptureModeRelaxed));
        int rc = fork_from(pool.cs);
        for (int q = 0; q < n_jobs && rc == KEVD_OK; ++q) rc = chunk(q, 0);
        if (rc == KEVD_OK) rc = join_to(pool.cs);
        const cudaError_t ce = cudaStreamEndCapture(pool.cs, graph);
        const int64_t captured = ctx->launches - launched;
        ctx->launches = launched;
        if (rc != KEVD_OK) return rc;
        if (ce != cudaSuccess) return set_error(ctx, KEVD_ERR_CUDA, "rpchol_batched: end capture: %s", cudaGetErrorString(ce));
        KEVD_CUDA(ctx, cudaGraphInstantiate(exec, *graph, 0));
        // launches alternate between two events; the states a launch copied are read
        // while the next one runs (a later copy can only show more jobs stopped)
        for (int c = 0; c < max_chunks; ++c) {
            KEVD_CUDA(ctx, cudaGraphLaunch(*exec, s));
            ctx->launches += captured;
            KEVD_CUDA(ctx, cudaEventRecord(pool.seen[c & 1], s));
            if (c == 0) continue;
            KEVD_CUDA(ctx, cudaEventSynchronize(pool.seen[(c - 1) & 1]));
            bool all = true;
            for (int q = 0; q < n_jobs; ++q)
                all = all && *reinterpret_cast<volatile int32_t*>(&pool.slots[q].state_h[0].done) != 0;
            if (all) break;
        }
    } else {
        KEVD_TRY(fork_from(s));
        std::vector<char> live(n_jobs, 1);
        int n_live = n_jobs;
        for (int c = 0; c < max_chunks && n_live > 0; ++c)
            for (int q = 0; q < n_jobs; ++q) {
                if (!live[q]) continue;
                BatchSlot& x = pool.slots[q];
                KEVD_TRY(chunk(q, c & 1));
                KEVD_CUDA(ctx, cudaEventRecord(x.seen[c & 1], x.st));
                if (c == 0) continue;
                KEVD_CUDA(ctx, cudaEventSynchronize(x.seen[(c - 1) & 1]));
                if (x.state_h[(c - 1) & 1].done) {
                    live[q] = 0;
                    --n_live;
                }
            }
        KEVD_TRY(join_to(s));
    }
    for (int q = 0; q < n_jobs; ++q) {
        BatchSlot& x = pool.slots[q];
        KEVD_CUDA(ctx, cudaMemcpyAsync(x.state_h, runs[q].rs, sizeof(RoundState), cudaMemcpyDeviceToHost, s));
        KEVD_CUDA(ctx, cudaMemcpyAsync(x.tcerr_h, runs[q].tc_err, sizeof(int), cudaMemcpyDeviceToHost, s));
        KEVD_CUDA(ctx, cudaMemcpyAsync(x.piv_h, runs[q].piv, jobs[q].k_max * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    }
    KEVD_CUDA(ctx, cudaStreamSynchronize(s));
    int rc = KEVD_OK;
    for (int q = 0; q < n_jobs; ++q) {
        const BatchSlot& x = pool.slots[q];
        kevd_rpchol_job& j = jobs[q];
        if (*x.tcerr_h != 0 && rc == KEVD_OK)
            rc = set_error(ctx, KEVD_ERR_TIMEOUT, "rpchol_batched: job %d tensor-core pipeline timed out", q);
        j.result.rank = x.state_h->rank;
        j.result.rounds = x.state_h->rounds;
        j.result.trace_error = x.state_h->total / (double)j.N;
        std::memcpy(j.piv, x.piv_h, (size_t)x.state_h->rank * sizeof(int64_t));
    }
    return rc;
}

int run_rpchol_batched(kevd_ctx* ctx, kevd_rpchol_job* jobs, int n_jobs, int use_graph, cudaStream_t s) {
    if (!jobs || n_jobs < 1 || n_jobs > 1024) return set_error(ctx, KEVD_ERR_ARG, "rpchol_batched: 1..1024 jobs");
    for (int q = 0; q < n_jobs; ++q) {
        const kevd_rpchol_job& j = jobs[q];
        if (!j.X || !j.F || !j.piv || j.N < 1 || j.d < 1 || j.d > kMaxFeatures || j.block < 1 || j.block > kMaxBlock ||
            j.k_max < 1 || j.ldF < j.k_max || j.max_rounds < 1 || !(j.scale > 0.0))
            return set_error(ctx, KEVD_ERR_ARG, "rpchol_batched: bad job %d", q);
    }
    BatchPool* pool = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    int rc = KEVD_OK;
    // before the pool is taken: an allocation of ctx may give the pool back
    int* cnt = arena_get<int>(ctx, "rp.density", n_jobs, &rc);
    if (rc != KEVD_OK) return set_error(ctx, rc, "rpchol_batched: out of device memory");
    // out of memory beside workspaces kept from earlier calls: once more without them
    for (bool kept = ctx->batch_pool != nullptr;; kept = false) {
        rc = batch_pool(ctx, jobs, n_jobs, &pool);
        if (rc == KEVD_OK) rc = rpchol_batched(ctx, jobs, n_jobs, use_graph != 0, *pool, cnt, &graph, &exec, s);
        if (rc != KEVD_OK) {
            // work may still be in flight on the caller's or the jobs' streams
            cudaStreamSynchronize(s);
            for (auto& x : pool->slots)
                if (x.st) cudaStreamSynchronize(x.st);
            cudaGetLastError();
        }
        if (exec) cudaGraphExecDestroy(exec);
        if (graph) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
        size_t held = 0;
        for (auto& x : pool->slots) held += x.c ? x.c->arena.total() : 0;
        if (held > kBatchKeepBytes || (int)pool->slots.size() > kBatchKeepJobs || rc != KEVD_OK) free_batch_pool(ctx);
        const bool idle = rc == KEVD_ERR_NOMEM && ctx->arena.reclaim();
        if (rc != KEVD_ERR_NOMEM || !(kept || idle)) return rc;
    }
}

// Gather rows idx of F (first ncols columns) into a column-major FP64 n x ncols
// matrix (ld n): used for L = F(S, :).
template <typename T>
__global__ void gather_rows_kernel(const T* __restrict__ F, int64_t ldF,
                                   const int64_t* __restrict__ idx, int64_t n, int64_t ncols,
                                   double* __restrict__ out) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n * ncols;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = e / n, q = e - c * n;
        out[e] = (double)F[idx[q] * ldF + c];
    }
}

int run_gather_rows(kevd_ctx* ctx, const void* F, int precision, int64_t ldF, const int64_t* idx,
                    int64_t n, int64_t ncols, double* out, cudaStream_t s) {
    const int grid = (int)std::min<int64_t>((n * ncols + 255) / 256, (int64_t)ctx->num_sms * 16);
    if (grid < 1) return KEVD_OK;
    if (precision == KEVD_FP64)
        gather_rows_kernel<double><<<grid, 256, 0, s>>>((const double*)F, ldF, idx, n, ncols, out);
    else
        gather_rows_kernel<float><<<grid, 256, 0, s>>>((const float*)F, ldF, idx, n, ncols, out);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

}  // namespace kevd
