// Plain FP64 rounds of few proposals (b <= 8): two kernels a round.
//
// The general round (kevd_rpchol.cu) updates 64 columns of every row block
// whatever the round accepted, so a round of one pivot does 64 times the FP64
// products it needs, and its sampler, proposal block and factorisation are
// three launches of latency.  Here a round is
//
//   rp_small_propose_kernel   sampler, H = K(S',S') - F F^T, accept / reject,
//                             Cholesky and inverse, in one CTA
//   rp_small_update_kernel    the accepted columns only, as dot products along
//                             the rows of F
//
// with the semantics of the general kernels (ks_arpclm.cu:197-224, :305-408,
// :933-995).  The FP64 pipe (2 lanes per clock per SM) bounds the update:
// nacc (r + 2 d) DFMA-class operations per row.  Sums along a row are spread
// over the 32 lanes of a warp, so their rounding differs from the general
// kernels' sequential sums (both are FP64).
#include "kevd_internal.cuh"
#include "kevd_rng.cuh"
#include "kevd_round.cuh"

#include <algorithm>

namespace kevd {

namespace {

constexpr int kSubRows = 16;        // rows per update CTA and per entry of the residual's block sums
constexpr int kUpdWarps = 4;
constexpr int kProposeThreads = 1024;
constexpr int kMaxSmallB = 8;

// (double)x without the FP64 pipe, which also runs the conversion: the
// exponent is rebiased in integer arithmetic (zero, subnormal and non-finite
// values take the conversion).
__device__ __forceinline__ double widen(float x) {
    const uint32_t u = __float_as_uint(x), m = u & 0x7fffffffu;
    if (m - 0x00800000u >= 0x7f000000u) return (double)x;
    return __hiloint2double((int)((u & 0x80000000u) | ((m >> 3) + 0x38000000u)), (int)(u << 29));
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ double warp_incl_scan(double v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

__global__ void rp_small_init_kernel(double* __restrict__ d, double* __restrict__ dsub, int64_t N, int64_t nsub,
                                     RoundState* st) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t i = t0; i < N; i += step) d[i] = 1.0;
    for (int64_t q = t0; q < nsub; q += step) dsub[q] = (double)min((int64_t)kSubRows, N - q * kSubRows);
    if (t0 == 0) *st = RoundState{0, 0, 0, 0, 0, 0, (double)N};
}

// One round up to L_i^{-1} (16 us a round at N = 20,000, b = 1; the general
// sampler, proposal block and factorisation 45 us).  Proposal t is the smallest i with
// cumsum(d)[i] >= u_t sum(d), found through the prefix over threads of block
// sums (kSubRows rows each), then the blocks of that thread, then the rows of
// that block.  b = 0 (the closing call) only records the last round's error.
__global__ void __launch_bounds__(kProposeThreads)
rp_small_propose_kernel(const double* __restrict__ F, int64_t ldF, const float* __restrict__ X, int d, double scale,
                        const double* __restrict__ dvec, const double* __restrict__ dsub, int64_t N, int64_t nsub,
                        int round, int b, uint64_t seed, const double* __restrict__ uniforms, double tol,
                        int64_t k_max, int max_rounds, double err_target, RoundState* st, double* __restrict__ minv,
                        int64_t* __restrict__ sacc, int64_t* __restrict__ piv, double* __restrict__ err,
                        int32_t* __restrict__ hm) {
    __shared__ double incl[kProposeThreads];
    __shared__ double wsum[32];
    __shared__ double part[kMaxSmallB * kMaxSmallB][32];
    __shared__ double kss[kMaxSmallB * kMaxSmallB];
    __shared__ double H[kMaxSmallB][kMaxSmallB + 1];
    __shared__ double H0[kMaxSmallB];
    __shared__ double MS[kMaxSmallB][kMaxSmallB + 1];
    __shared__ int64_t props[kMaxSmallB];
    __shared__ int accpos[kMaxSmallB];
    __shared__ int s_stop;
    if (st->done) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t r = st->rank;

    // prefix of the block sums over threads
    const int64_t chunk = (nsub + kProposeThreads - 1) / kProposeThreads;
    const int64_t c0 = min(nsub, (int64_t)tid * chunk), c1 = min(nsub, c0 + chunk);
    double s = 0.0;
    for (int64_t q = c0; q < c1; ++q) s += dsub[q];
    s = warp_incl_scan(s, lane);
    if (lane == 31) wsum[warp] = s;
    __syncthreads();
    if (warp == 0) wsum[lane] = warp_incl_scan(wsum[lane], lane);
    __syncthreads();
    incl[tid] = (warp > 0 ? wsum[warp - 1] : 0.0) + s;
    const double total = wsum[31];
    if (tid == 0) {
        const double e = total / (double)N;
        if (round > 0) err[round - 1] = e;
        st->total = total;
        const bool stop = (round >= max_rounds) || (r >= k_max) || (err_target > 0.0 && round > 0 && e <= err_target);
        if (stop) {
            st->done = 1;
            st->rounds = round;
        }
        s_stop = stop;
    }
    __syncthreads();
    if (s_stop) return;

    if (warp < b) {
        const double u = uniforms ? uniforms[((int64_t)round * 2) * b + warp]
                                  : philox_uniform(seed, (uint32_t)round, 0u, (uint32_t)warp);
        const double target = u * total;
        int64_t pick = N - 1;
        if (target <= total) {
            int lo = 0, hi = kProposeThreads - 1;   // smallest chunk owner with incl >= target
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (incl[mid] >= target) hi = mid; else lo = mid + 1;
            }
            double base = (lo > 0) ? incl[lo - 1] : 0.0;
            const int64_t q0 = min(nsub, (int64_t)lo * chunk), q1 = min(nsub, q0 + chunk);
            int64_t blk = q1 - 1;
            for (int64_t q = q0; q < q1; q += 32) {   // 32 blocks at a time
                const double v = (q + lane < q1) ? dsub[q + lane] : 0.0;
                const double pre = warp_incl_scan(v, lane);
                const unsigned m = __ballot_sync(0xffffffffu, q + lane < q1 && base + pre >= target);
                if (m) {
                    const int src = __ffs(m) - 1;
                    blk = q + src;
                    base += __shfl_sync(0xffffffffu, pre, src) - __shfl_sync(0xffffffffu, v, src);
                    break;
                }
                base += __shfl_sync(0xffffffffu, pre, 31);
            }
            if (blk >= q0) {
                const int64_t row = blk * kSubRows + lane;
                const double v = (lane < kSubRows && row < N) ? dvec[row] : 0.0;
                const double cum = base + warp_incl_scan(v, lane);
                unsigned m = __ballot_sync(0xffffffffu, v > 0.0 && cum >= target);
                // rounding can leave the target past the block's recomputed sum:
                // then its last row with d > 0
                if (m) {
                    pick = blk * kSubRows + __ffs(m) - 1;
                } else if ((m = __ballot_sync(0xffffffffu, v > 0.0)) != 0) {
                    pick = blk * kSubRows + 31 - __clz(m);
                }
            }
        }
        if (lane == 0) props[warp] = min(pick, N - 1);
    }
    __syncthreads();

    // H on the lower triangle: the 32 warps share the (pair, column range) products
    const int np = b * (b + 1) / 2;
    const int per = max(1, 32 / np);   // warps per pair
    for (int t = warp; t < np * per; t += 32) {
        const int pr = t / per, g = t - pr * per;
        int p = 0;
        while ((p + 1) * (p + 2) / 2 <= pr) ++p;
        const int q = pr - p * (p + 1) / 2;
        const double* fp = F + props[p] * ldF;
        const double* fq = F + props[q] * ldF;
        double acc = 0.0;
        for (int64_t c = g * 32 + lane; c < r; c += per * 32) acc += fp[c] * fq[c];
        acc = warp_sum(acc);
        if (lane == 0) part[pr][g] = acc;
        if (g == 0) {
            // p == q too: a state with an infinity or a NaN has no distance to itself, H is
            // NaN and it is rejected
            double d2 = 0.0;
            const float* xp = X + props[p] * d;
            const float* xq = X + props[q] * d;
            for (int k = lane; k < d; k += 32) {
                const double v = (double)xp[k] - (double)xq[k];
                d2 += v * v;
            }
            d2 = warp_sum(d2);
            if (lane == 0) kss[pr] = exp(-scale * d2);
        }
    }
    __syncthreads();
    if (warp != 0) return;
    for (int pr = lane; pr < np; pr += 32) {
        int p = 0;
        while ((p + 1) * (p + 2) / 2 <= pr) ++p;
        const int q = pr - p * (p + 1) / 2;
        double v = kss[pr];
        for (int g = 0; g < per; ++g) v -= part[pr][g];
        H[p][q] = v;
        if (p == q) H0[p] = v;
    }
    __syncwarp();
    // accept / reject and Cholesky by one warp: every lane takes the same
    // decisions, lane (jj, kk) pairs share the trailing update
    const int64_t cap = k_max - r;
    int m = 0;
    for (int i = 0; i < b; ++i) {
        const double hii = H[i][i];
        const double u = uniforms ? uniforms[((int64_t)round * 2 + 1) * b + i]
                                  : philox_uniform(seed, (uint32_t)round, 1u, (uint32_t)i);
        if (!(m < cap && H0[i] * u < hii && hii > tol && hii > 0.0)) continue;
        if (lane == 0) accpos[m] = i;
        ++m;
        const double f = 1.0 / sqrt(hii);
        __syncwarp();
        if (lane >= i && lane < b) H[lane][i] *= f;
        __syncwarp();
        for (int e = lane; e < b * b; e += 32) {
            const int jj = e / b, kk = e - jj * b;
            if (kk > i && kk <= jj) H[jj][kk] -= H[jj][i] * H[kk][i];
        }
        __syncwarp();
    }
    __syncwarp();
    // inverse of the compacted factor, one column per lane
    if (lane < m) {
        const int t = lane;
        const int64_t sp = props[accpos[t]];
        sacc[t] = sp;
        piv[r + t] = sp;
        for (int a = 0; a < t; ++a) MS[a][t] = 0.0;
        MS[t][t] = 1.0 / H[accpos[t]][accpos[t]];
        for (int a = t + 1; a < m; ++a) {
            double v = 0.0;
            for (int e = t; e < a; ++e) v += H[accpos[a]][accpos[e]] * MS[e][t];
            MS[a][t] = -v / H[accpos[a]][accpos[a]];
        }
        for (int a = 0; a < m; ++a) minv[a * b + t] = MS[a][t];
    }
    if (lane == 0) {
        st->r_old = r;
        st->nacc = m;
        st->rank = r + m;
        hm[round] = m;
    }
}

// Sums v[i] over the warp for every i < M (a power of two <= 32): the lanes
// halve the list at each exchange, so M sums cost M - 1 + log2(32 / M)
// additions instead of 5 M.  Lane l ends with the sum of index
// l >> (5 - log2 M).
template <int M>
__device__ __forceinline__ double warp_sums(double (&v)[M], int lane) {
    int o = 16;
#pragma unroll
    for (int half = M / 2; half > 0; half >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const double keep = up ? v[i + half] : v[i], give = up ? v[i] : v[i + half];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    }
    double s = v[0];
    for (; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// The accepted columns of 16 rows per CTA (4 warps): lanes run along the
// features and along the columns of F, R rows by NB pivots of sums per warp
// step; 128 threads then evaluate K - P, one (row, pivot) each, and 16 form
// G = T L_i^{-T}, F, d and the CTA's sum of d.  16 rows per CTA spread N =
// 20,000 over 1,250 CTAs (8.2 per SM, at most 9).
// N = 20,000, d = 64, k = 500, b = 1 (500 rounds): general kernels 904 ms of
// updates.
template <int NB>
__global__ void __launch_bounds__(32 * kUpdWarps)
rp_small_update_kernel(double* __restrict__ F, int64_t ldF, const float* __restrict__ X, int64_t N, int d,
                       double scale, const int64_t* __restrict__ sacc, const double* __restrict__ minv, int b,
                       const RoundState* st, double* __restrict__ dvec, double* __restrict__ dsub) {
    if (st->done) return;
    const int nacc = st->nacc;
    if (nacc == 0) return;
    const int64_t r = st->r_old;
    constexpr int R = NB <= 2 ? 4 : 8 / NB;   // rows per warp step
    constexpr int M = R * NB;
    static_assert((M & (M - 1)) == 0 && M <= 8, "sums per warp step");
    __shared__ double Ds[kSubRows][NB], Ps[kSubRows][NB];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row0 = (int64_t)blockIdx.x * kSubRows;
    const float* xs[NB];
    const double* fs[NB];
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        const int64_t sp = sacc[min(j, nacc - 1)];
        xs[j] = X + sp * d;
        fs[j] = F + sp * ldF;
    }
    for (int i0 = warp * (kSubRows / kUpdWarps); i0 < (warp + 1) * (kSubRows / kUpdWarps); i0 += R) {
        double dd[M], pp[M];
#pragma unroll
        for (int e = 0; e < M; ++e) dd[e] = pp[e] = 0.0;
        const float* xr[R];
        const double* fr[R];
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int64_t row = min(row0 + i0 + i, N - 1);
            xr[i] = X + row * d;
            fr[i] = F + row * ldF;
        }
        for (int k = lane; k < d; k += 32) {
            double vs[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j) vs[j] = widen(xs[j][k]);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const double vr = widen(xr[i][k]);
#pragma unroll
                for (int j = 0; j < NB; ++j) {
                    const double t = vr - vs[j];
                    dd[i * NB + j] = fma(t, t, dd[i * NB + j]);
                }
            }
        }
#pragma unroll 4
        for (int64_t c = lane; c < r; c += 32) {
            double vs[NB];
#pragma unroll
            for (int j = 0; j < NB; ++j) vs[j] = fs[j][c];
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const double vr = fr[i][c];
#pragma unroll
                for (int j = 0; j < NB; ++j) pp[i * NB + j] = fma(vr, vs[j], pp[i * NB + j]);
            }
        }
        const double ds = warp_sums<M>(dd, lane), ps = warp_sums<M>(pp, lane);
        if (lane % (32 / M) == 0) {
            const int e = lane / (32 / M);
            Ds[i0 + e / NB][e % NB] = ds;
            Ps[i0 + e / NB][e % NB] = ps;
        }
    }
    __syncthreads();
    // T = K - P in place of P
    for (int e = threadIdx.x; e < kSubRows * NB; e += 32 * kUpdWarps)
        Ps[e / NB][e % NB] = exp(-scale * Ds[e / NB][e % NB]) - Ps[e / NB][e % NB];
    __syncthreads();
    if (warp != 0) return;
    double nd = 0.0;
    const int64_t row = row0 + lane;
    if (lane < kSubRows && row < N) {
        double sq = 0.0;
        for (int a = 0; a < nacc; ++a) {
            double g = 0.0;
            for (int e = 0; e <= a; ++e) g = fma(Ps[lane][e], minv[a * b + e], g);
            F[row * ldF + r + a] = g;
            sq = fma(g, g, sq);
        }
        nd = fmax(dvec[row] - sq, 0.0);
        dvec[row] = nd;
    }
    nd = warp_sum(nd);
    if (lane == 0) dsub[blockIdx.x] = nd;
}

}  // namespace

bool rpchol_small_supported(int b) { return b <= kMaxSmallB; }

int64_t rpchol_small_blocks(int64_t N) { return (N + kSubRows - 1) / kSubRows; }

int launch_rpchol_small_init(kevd_ctx* ctx, double* dvec, double* dsub, int64_t N, RoundState* st, cudaStream_t s) {
    rp_small_init_kernel<<<ctx->num_sms * 4, 256, 0, s>>>(dvec, dsub, N, rpchol_small_blocks(N), st);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

int launch_rpchol_small_propose(kevd_ctx* ctx, const double* F, int64_t ldF, const float* X, int64_t N, int d,
                                double scale, const double* dvec, const double* dsub, int round, int b, uint64_t seed,
                                const double* uniforms, double tol, int64_t k_max, int max_rounds, double err_target,
                                RoundState* st, double* minv, int64_t* sacc, int64_t* piv, double* err, int32_t* hm,
                                cudaStream_t s) {
    ProfScope ps(ctx, "rp_propose", s);
    rp_small_propose_kernel<<<1, kProposeThreads, 0, s>>>(F, ldF, X, d, scale, dvec, dsub, N, rpchol_small_blocks(N),
                                                          round, b, seed, uniforms, tol, k_max, max_rounds, err_target,
                                                          st, minv, sacc, piv, err, hm);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

int launch_rpchol_small_update(kevd_ctx* ctx, double* F, int64_t ldF, const float* X, int64_t N, int d, double scale,
                               const int64_t* sacc, const double* minv, int b, const RoundState* st, double* dvec,
                               double* dsub, cudaStream_t s) {
    ProfScope ps(ctx, "rp_update", s);
    const unsigned grid = (unsigned)rpchol_small_blocks(N);
    auto go = [&](auto kern) { kern<<<grid, 32 * kUpdWarps, 0, s>>>(F, ldF, X, N, d, scale, sacc, minv, b, st, dvec, dsub); };
    if (b == 1) go(&rp_small_update_kernel<1>);
    else if (b == 2) go(&rp_small_update_kernel<2>);
    else if (b <= 4) go(&rp_small_update_kernel<4>);
    else go(&rp_small_update_kernel<8>);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

}  // namespace kevd
