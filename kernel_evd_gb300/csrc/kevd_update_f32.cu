// Residual update of one block-RPCholesky pass for an FP32 factor on the FP32
// pipe: layouts the tensor-core update cannot read by TMA (ldF not a multiple of
// 4) and nearly diagonal kernels.  The operations and their order are part of the
// result, because the pivots of a run follow every rounding of d:
//
//   P(i, q) = sum_c F(i, c) F(s_q, c)   one FMA chain in increasing c
//   T = K(i, s_q) - P                   direct distances in increasing feature order
//   G = T L_i^{-T}                      one FMA chain in increasing e
//   d(i) <- max(d(i) - sum_a G(i, a)^2, 0) in FP64, the squares added over a = t,
//           t + 16, .. first and then over t in a butterfly (8, 4, 2, 1)
//
// CTA = 128 threads on 128 rows x NC columns (NC = 32 or 64 by the block size b:
// with one width of 64 a block of 32 did twice the products it needs); thread
// (ty, tx) of 16 x 8 owns rows ty + 16 a and NC / 8 neighbouring columns as
// packed pairs (f32x2: subtraction and FMA take half the issue slots).  Operands
// are staged 32 terms at a time, term-major, so that a thread reads its rows and
// its columns in 16-byte loads; factor rows of any stride are read 8 terms of 4
// rows per warp load (32-byte pieces) and stored with the 4-row chunk index XOR-ed
// with the term, which spreads a warp's stores and its loads over all banks.
// FP32 pipe: nacc (r + 2 d + nacc) operations a row.  All updates of a run, here /
// 256 threads on 64 columns with one load per operand: N = 90,677, k = 898, b = 32
// 3.8 / 13.6 ms; N = 200,000, k = 1,001, b = 64 8.8 / 17.3 ms; k = 601, b = 16
// 7.4 / 26.9 ms (d = 64).
#include "kevd_internal.cuh"
#include "kevd_pairtile.cuh"
#include "kevd_round.cuh"

#include <algorithm>

namespace kevd {

namespace {

constexpr int kRows = 128;    // rows per CTA (= rows per d partial sum)
constexpr int kTerms = 32;    // features or factor columns staged at a time
constexpr int kPass = 64;     // accepted columns per pass
constexpr int kThreads = 128;

// Factor columns [c0, c0 + nc) of kPlaces rows (zeros past nc): loaded into
// registers (the next stage's while this one is multiplied), then stored to
// dst[term][place], chunk ch of 4 places at chunk ch ^ (term & 7).  row(place)
// gives a row pointer or nullptr.
template <int kPlaces>
struct FactorStage {
    static constexpr int kIter = kPlaces / 4 / (kThreads / 32);
    float v[kIter][kTerms / 8];
    template <class Row>
    __device__ __forceinline__ void load(Row row, int64_t c0, int nc) {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int k8 = lane >> 2, u = lane & 3;
#pragma unroll
        for (int j = 0; j < kIter; ++j) {
            const float* src = row(4 * (warp + j * (kThreads / 32)) + u);
#pragma unroll
            for (int q = 0; q < kTerms / 8; ++q) {
                v[j][q] = 0.f;
                if (src && 8 * q + k8 < nc)   // volatile: stays ahead of the products
                    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v[j][q]) : "l"(src + c0 + 8 * q + k8));
            }
        }
    }
    __device__ __forceinline__ void store(float* dst) const {
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        const int k8 = lane >> 2, u = lane & 3;
#pragma unroll
        for (int j = 0; j < kIter; ++j)
#pragma unroll
            for (int q = 0; q < kTerms / 8; ++q)
                dst[(8 * q + k8) * kPlaces + 4 * ((warp + j * (kThreads / 32)) ^ k8) + u] = v[j][q];
    }
};

// n consecutive places from 8-aligned place p0 (two 16-byte pieces; one for n = 4).
template <int n, int kPlaces, bool kSwizzled>
__device__ __forceinline__ void read_places(const float* tile, int k, int p0, float (&v)[n]) {
#pragma unroll
    for (int h = 0; h < n / 4; ++h) {
        const int ch = (p0 >> 2) + h;
        const float4 x =
            *reinterpret_cast<const float4*>(tile + k * kPlaces + 4 * (kSwizzled ? ch ^ (k & 7) : ch));
        v[4 * h] = x.x;
        v[4 * h + 1] = x.y;
        v[4 * h + 2] = x.z;
        v[4 * h + 3] = x.w;
    }
}

template <int NC>
struct Smem {
    static constexpr int kPitch = NC + 1;
    float a[kTerms * kRows];          // rows
    float b[kTerms * NC];             // columns
    float t[kRows * kPitch];          // P, then T, then G
    float mv[NC * NC];                // mv[e][a] = L_i^{-1}[a][e]
};

template <int NC>
__global__ void __launch_bounds__(kThreads, NC == 64 ? 2 : 3)
update_f32_kernel(float* __restrict__ F, int64_t ldF, const float* __restrict__ X, int64_t N, int d, double scale,
                  const int64_t* __restrict__ sacc, const float* __restrict__ minv_f, int b, const RoundState* st,
                  double* __restrict__ dvec, double* __restrict__ dblk, int group) {
    if (st->done) return;
    const int64_t r = st->r_old + (int64_t)kPass * group;
    const int nacc = min(kPass, st->nacc - kPass * group);
    if (nacc <= 0) return;
    {   // this pass's pivots and diagonal block of L_i^{-1} (leading dimension b)
        const int64_t o = (int64_t)kPass * group;
        sacc += o;
        minv_f += o * b + o;
    }
    constexpr int CP = NC / 8, NP = CP / 2;   // columns per thread, and as pairs
    constexpr int kPitch = Smem<NC>::kPitch;
    extern __shared__ __align__(16) unsigned char raw[];
    Smem<NC>& sm = *reinterpret_cast<Smem<NC>*>(raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = tid & 7, ty = tid >> 3;
    const int64_t row0 = (int64_t)blockIdx.x * kRows;
    const int nrows = (int)min((int64_t)kRows, N - row0);

    for (int e = tid; e < NC * NC; e += kThreads) {
        const int q = e / NC, a = e - q * NC;
        sm.mv[e] = (a < nacc && q < nacc) ? minv_f[(int64_t)a * b + q] : 0.f;
    }
    f32x2 acc[8][NP];
    auto zero = [&] {
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
            for (int p = 0; p < NP; ++p) acc[a][p] = 0ull;
    };

    // P = F(R, 0:r) F(S_i, 0:r)^T
    zero();
    FactorStage<kRows> fa;
    FactorStage<NC> fb;
    auto load = [&](int64_t c0) {
        const int nc = (int)max((int64_t)0, min((int64_t)kTerms, r - c0));
        fa.load([&](int place) {   // place 8 t + u is row t + 16 u
            const int rr = (place >> 3) + 16 * (place & 7);
            return rr < nrows ? F + (row0 + rr) * ldF : (const float*)nullptr;
        }, c0, nc);
        fb.load([&](int q) { return q < nacc ? F + sacc[q] * ldF : (const float*)nullptr; }, c0, nc);
    };
    load(0);
    for (int64_t c0 = 0; c0 < r; c0 += kTerms) {
        __syncthreads();
        fa.store(sm.a);
        fb.store(sm.b);
        __syncthreads();
        load(c0 + kTerms);
#pragma unroll 4
        for (int k = 0; k < kTerms; ++k) {
            float va[8], vb[CP];
            read_places<8, kRows, true>(sm.a, k, 8 * ty, va);
            read_places<CP, NC, true>(sm.b, k, CP * tx, vb);
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                const f32x2 v = pack2(va[a], va[a]);
#pragma unroll
                for (int p = 0; p < NP; ++p) acc[a][p] = fma2(v, pack2(vb[2 * p], vb[2 * p + 1]), acc[a][p]);
            }
        }
    }
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            float* t = sm.t + (ty + 16 * a) * kPitch + CP * tx + 2 * p;
            unpack2(acc[a][p], t[0], t[1]);
        }

    // T = K(R, S_i) - P (the thread's own entries)
    zero();
    for (int c0 = 0; c0 < d; c0 += kTerms) {
        const int w = min(kTerms, d - c0), w4 = (w + 3) & ~3;
        __syncthreads();
        pt_stage<kRows, false>(X, N, d, row0, c0, w, sm.a);
        for (int e = tid; e < NC * w4; e += kThreads) {
            const int q = e % NC, k = e / NC;
            sm.b[k * NC + q] = (q < nacc && k < w) ? -X[sacc[q] * d + c0 + k] : 0.f;
        }
        __syncthreads();
#pragma unroll 2
        for (int k = 0; k < w4; ++k) {
            float va[8], vb[CP];
            read_places<8, kRows, false>(sm.a, k, 8 * ty, va);
            read_places<CP, NC, false>(sm.b, k, CP * tx, vb);
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                const f32x2 v = pack2(va[a], va[a]);
#pragma unroll
                for (int p = 0; p < NP; ++p) {
                    const f32x2 u = add2(v, pack2(vb[2 * p], vb[2 * p + 1]));
                    acc[a][p] = fma2(u, u, acc[a][p]);
                }
            }
        }
    }
    const ScalePair sp = split_scale(scale);
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            float* t = sm.t + (ty + 16 * a) * kPitch + CP * tx + 2 * p;
            float x, y;
            unpack2(acc[a][p], x, y);
            const int c = CP * tx + 2 * p;
            t[0] = (c < nacc ? kexp_scaled(x, sp) : 0.f) - t[0];
            t[1] = (c + 1 < nacc ? kexp_scaled(y, sp) : 0.f) - t[1];
        }
    __syncthreads();

    // G = T L_i^{-T}
    zero();
#pragma unroll 2
    for (int e = 0; e < nacc; ++e) {
        float vm[CP];
        read_places<CP, NC, false>(sm.mv, e, CP * tx, vm);
#pragma unroll
        for (int a = 0; a < 8; ++a) {
            const float te = sm.t[(ty + 16 * a) * kPitch + e];
            const f32x2 v = pack2(te, te);
#pragma unroll
            for (int p = 0; p < NP; ++p) acc[a][p] = fma2(v, pack2(vm[2 * p], vm[2 * p + 1]), acc[a][p]);
        }
    }
    __syncthreads();   // every T has been read
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            float* t = sm.t + (ty + 16 * a) * kPitch + CP * tx + 2 * p;
            unpack2(acc[a][p], t[0], t[1]);
        }
    __syncthreads();

    // the new columns, a warp per row
    for (int rr = warp; rr < nrows; rr += kThreads / 32) {
        float* out = F + (row0 + rr) * ldF + r;
#pragma unroll
        for (int a = lane; a < NC; a += 32)
            if (a < nacc) out[a] = sm.t[rr * kPitch + a];
    }
    // sums of squares: lane t (of 16) holds the columns t, t + 16, .. of 16 rows, and
    // the butterfly over the 16 lanes halves the list of rows at each exchange
    // (15 FP64 additions for 16 rows instead of 64); lane t ends with row t
    double sq[16];
    {
        const int t16 = lane & 15, rb = 32 * warp + (lane & 16);
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            double s = 0.0;
#pragma unroll
            for (int j = 0; j < NC / 16; ++j)
                if (t16 + 16 * j < nacc) {
                    const double g = (double)sm.t[(rb + i) * kPitch + t16 + 16 * j];
                    s = fma(g, g, s);
                }
            sq[i] = s;
        }
#pragma unroll
        for (int half = 8; half > 0; half >>= 1) {
            const bool up = (lane & half) != 0;
#pragma unroll
            for (int i = 0; i < half; ++i) {
                const double keep = up ? sq[i + half] : sq[i], give = up ? sq[i] : sq[i + half];
                sq[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
            }
        }
    }
    double nd = 0.0;
    if (tid < nrows) {   // row 32 warp + lane = tid
        nd = fmax(dvec[row0 + tid] - sq[0], 0.0);
        dvec[row0 + tid] = nd;
    }
    __shared__ double wsum[kThreads / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nd += __shfl_xor_sync(0xffffffffu, nd, o);
    if (lane == 0) wsum[warp] = nd;
    __syncthreads();
    if (tid == 0) dblk[blockIdx.x] = ((wsum[0] + wsum[1]) + (wsum[2] + wsum[3]));
}

}  // namespace

// One round's update, in passes of 64 accepted columns; rounds of at most 32
// proposals compute 32 columns.
int launch_update_f32(kevd_ctx* ctx, float* F, int64_t ldF, const float* X, int64_t N, int d, double scale,
                      const int64_t* sacc, const float* minv_f, int b, const RoundState* st, double* dvec, double* dblk,
                      cudaStream_t s) {
    const unsigned grid = (unsigned)((N + kRows - 1) / kRows);
    auto go = [&](auto kern, size_t smem) -> int {
        KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(kern), smem));
        for (int g = 0; g < (b + kPass - 1) / kPass; ++g) {
            kern<<<grid, kThreads, smem, s>>>(F, ldF, X, N, d, scale, sacc, minv_f, b, st, dvec, dblk, g);
            KEVD_LAUNCH(ctx);
        }
        return KEVD_OK;
    };
    return b <= 32 ? go(&update_f32_kernel<32>, sizeof(Smem<32>)) : go(&update_f32_kernel<64>, sizeof(Smem<64>));
}

}  // namespace kevd
