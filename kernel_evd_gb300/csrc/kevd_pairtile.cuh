// FP32 squared distances of a 128 x 128 pair tile and the exponential sums over
// it, shared by the calibration kernels (single dataset, batched work queue)
// and the pair-distance median.
//
// A CTA holds four groups of 128 threads (8 ty x 16 tx), one CTA per SM; a group
// works on half tiles of its own, 64 x 128 pairs: half h covers rows ri0 + 8 h +
// ty + 16 a (a < 8) against rows rj0 + tx + 16 b (b < 8), 64 distances per thread
// as 32 packed pairs (b, b + 1).
//
// What bounds a sweep: per pair 2 d FP32 operations of distance, and per (pair,
// scale) a multiplication, an ex2 (8 lanes per clock per scheduler) and an
// addition: with d = 64 and 64 scales 2.0 clocks per pair and SM for the FMA
// pipe and as much for the ex2 unit.  The exponentials run at the ex2 unit's
// rate and the distances at 0.7 of the FMA pipe's; what is left is that they
// overlap little (3.0 clocks per pair).  Independent groups that share barriers
// with nobody overlap best: N = 200,000, d = 64, 64 scales takes 187 ms (190
// with two features of the distance loop unrolled, four are built); as four
// CTAs per SM 212 ms, with groups made to alternate between distances and
// exponentials 200 ms, with the next tile's distances woven into the exponentials
// (two tiles of registers, three groups) 214 to 231 ms, and as two CTAs of 256
// threads with scalar instructions 266 ms.  Distances and scalings are issued as
// packed FP32 pairs (f32x2), which halves their issue slots.
//
// Every distance is summed over the features in increasing order, FMA by FMA,
// and every scale's 64 terms per thread one after the other: the order of the
// sums is part of the result, packed or not.
//
// Features are staged 64 at a time, feature-major; the rows of a tile are
// placed so that a thread's eight i rows, and its eight j rows, are contiguous
// (row t + 16 u at 8 t + u): two 16-byte loads each.  j rows are staged
// negated, so that x_j - x_i is one packed addition.  A ragged last chunk is
// padded with zeros in both tiles, which adds exact zeros.
#pragma once

#include <cstdint>

namespace kevd {

constexpr int kPtTile = 128;
constexpr int kPtChunk = 64;
constexpr int kPtHalf = 64;                             // i rows of a group
constexpr int kPtGroup = 128;                           // threads of a group
constexpr int kPtGroups = 4;
constexpr int kPtThreads = kPtGroup * kPtGroups;
constexpr int kPtWarps = kPtGroup / 32;
constexpr int kPtSmemFloats = kPtChunk * (kPtHalf + kPtTile);   // i and j tiles of one group

using f32x2 = unsigned long long;   // two FP32 values, the first in the low word

__device__ __forceinline__ f32x2 pack2(float x, float y) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& x, float& y) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ int pt_group() { return threadIdx.x / kPtGroup; }
__device__ __forceinline__ int pt_tid() { return threadIdx.x % kPtGroup; }   // within the group
__device__ __forceinline__ void pt_sync() {                                 // the group's barrier
    asm volatile("bar.sync %0, %1;" ::"r"(1 + pt_group()), "n"(kPtGroup) : "memory");
}

// Half tiles of the lower-triangular tile grid, row of tiles by row of tiles,
// half 0 before half 1: unit u -> (ti, h, tj), tj <= ti.
struct PtUnit {
    int64_t ti, tj;
    int h;
};
__device__ __forceinline__ PtUnit pt_unit(int64_t u) {
    int64_t i = (int64_t)((sqrt(4.0 * (double)u + 1.0) - 1.0) * 0.5);
    while (i * (i + 1) > u) --i;
    while ((i + 1) * (i + 2) <= u) ++i;
    const int64_t rem = u - i * (i + 1);
    const int h = rem > i ? 1 : 0;
    return {i, rem - h * (i + 1), h};
}
__device__ __forceinline__ void pt_next(PtUnit& u) {
    if (++u.tj > u.ti) {
        u.tj = 0;
        if (u.h == 0) {
            u.h = 1;
        } else {
            u.h = 0;
            ++u.ti;
        }
    }
}

// Stage features [c0, c0 + w) of kRows rows into dst[feature][place] (zeros past
// N and past w, up to w rounded up to 4): place 8 t + u is row r0 + t + 16 u.  A
// lane takes a row, in the order of the places, so the transposed stores of a
// warp fall in distinct banks.
template <int kRows, bool kNegate>
__device__ __forceinline__ void pt_stage(const float* __restrict__ X, int64_t N, int d, int64_t r0, int c0, int w,
                                         float* dst) {
    const int lane = pt_tid() & 31, warp = pt_tid() >> 5;
    constexpr int kSets = kRows / 32;              // sets of 32 rows
    constexpr int kPar = kPtWarps / kSets;         // warps that share a set's features
    const int set = warp % kSets;
    const int64_t r = r0 + 4 * set + (lane >> 3) + 16 * (lane & 7);
    const bool in = r < N;
    const float* src = X + r * d + c0;
    const bool vec = (d & 3) == 0 && ((uintptr_t)X & 15) == 0;
    const int nq = (w + 3) >> 2;
#pragma unroll 8
    for (int q = warp / kSets; q < nq; q += kPar) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (in) {
            if (vec) {
                v = __ldg(reinterpret_cast<const float4*>(src) + q);
            } else {
                v.x = src[4 * q];
                if (4 * q + 1 < w) v.y = src[4 * q + 1];
                if (4 * q + 2 < w) v.z = src[4 * q + 2];
                if (4 * q + 3 < w) v.w = src[4 * q + 3];
            }
        }
        float* o = dst + 4 * q * kRows + 32 * set + lane;
        o[0] = kNegate ? -v.x : v.x;
        o[kRows] = kNegate ? -v.y : v.y;
        o[2 * kRows] = kNegate ? -v.z : v.z;
        o[3 * kRows] = kNegate ? -v.w : v.w;
    }
}

// Stage chunk c0 of unit u: i rows into sm, j rows behind them.  Two barriers:
// the tiles are free before, filled after.  staged: the (ti, h) whose rows are
// in place (-1: none), kept from unit to unit where the features fit one chunk.
__device__ __forceinline__ void pt_stage_unit(const float* __restrict__ X, int64_t N, int d, const PtUnit& u, int c0,
                                              float* sm, int64_t& staged) {
    const int w = min(kPtChunk, d - c0);
    pt_sync();
    if (staged != 2 * u.ti + u.h) pt_stage<kPtHalf, false>(X, N, d, u.ti * kPtTile + 8 * u.h, c0, w, sm);
    pt_stage<kPtTile, true>(X, N, d, u.tj * kPtTile, c0, w, sm + kPtChunk * kPtHalf);
    if (d <= kPtChunk) staged = 2 * u.ti + u.h;
    pt_sync();
}

// D[a][p] = squared distances of the unit's rows i = 128 ti + 8 h + ty + 16 a
// and the two rows j = 128 tj + tx + 16 (2 p), + 16 (2 p + 1).  Called by a
// whole group; sm: its tiles, 16-byte aligned.
__device__ __forceinline__ void pt_dist(const float* __restrict__ X, int64_t N, int d, const PtUnit& u, float* sm,
                                        int64_t& staged, f32x2 (&D)[8][4]) {
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int p = 0; p < 4; ++p) D[a][p] = 0ull;
    for (int c0 = 0; c0 < d; c0 += kPtChunk) {
        pt_stage_unit(X, N, d, u, c0, sm, staged);
        const int w4 = (min(kPtChunk, d - c0) + 3) & ~3;
        const float* xi = sm + 8 * (pt_tid() >> 4);
        const float* xj = sm + kPtChunk * kPtHalf + 8 * (pt_tid() & 15);
#pragma unroll 4
        for (int k = 0; k < w4; ++k) {
            const float4 i0 = *reinterpret_cast<const float4*>(xi + k * kPtHalf);
            const float4 i1 = *reinterpret_cast<const float4*>(xi + k * kPtHalf + 4);
            const ulonglong2 j0 = *reinterpret_cast<const ulonglong2*>(xj + k * kPtTile);
            const ulonglong2 j1 = *reinterpret_cast<const ulonglong2*>(xj + k * kPtTile + 4);
            const float vi[8] = {i0.x, i0.y, i0.z, i0.w, i1.x, i1.y, i1.z, i1.w};
            const f32x2 vj[4] = {j0.x, j0.y, j1.x, j1.y};
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                const f32x2 v = pack2(vi[a], vi[a]);
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const f32x2 t = add2(v, vj[p]);
                    D[a][p] = fma2(t, t, D[a][p]);
                }
            }
        }
    }
}

// Pairs that do not count (i <= l, or outside [0, N)) become +inf: exp2(-inf) = 0.
// Only tiles on the diagonal or at the ragged end hold any.
__device__ __forceinline__ void pt_mask(int64_t N, const PtUnit& u, f32x2 (&D)[8][4]) {
    if (u.tj < u.ti && (u.ti + 1) * kPtTile <= N) return;
    const int64_t gi0 = u.ti * kPtTile + 8 * u.h + (pt_tid() >> 4), gj0 = u.tj * kPtTile + (pt_tid() & 15);
    const float inf = __int_as_float(0x7f800000);
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int64_t gi = gi0 + 16 * a, gj = gj0 + 32 * p;
            float x, y;
            unpack2(D[a][p], x, y);
            if (!(gi < N && gi > gj)) x = inf;
            if (!(gi < N && gi > gj + 16)) y = inf;
            D[a][p] = pack2(x, y);
        }
}

// The sum of exp2(c D) over the thread's 64 pairs, in order.  Every product is
// formed one step before its exponentials and every exponential two steps before
// its addition; the statements are volatile to keep this order (left to the
// compiler, that sweep took 203 ms).
__device__ __forceinline__ float pt_exp_sum(const f32x2 (&D)[8][4], float c) {
    const f32x2 cc = pack2(c, c);
    float s = 0.f, ex[3], ey[3];
    f32x2 m;
    asm volatile("mul.rn.f32x2 %0, %1, %2;" : "=l"(m) : "l"(D[0][0]), "l"(cc));
#pragma unroll
    for (int q = 0; q < 34; ++q) {
        float x, y;
        if (q < 32) {
            unpack2(m, x, y);
            asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(ex[q % 3]) : "f"(x));
            if (q < 31) asm volatile("mul.rn.f32x2 %0, %1, %2;" : "=l"(m) : "l"(D[(q + 1) >> 2][(q + 1) & 3]), "l"(cc));
        }
        if (q >= 2) asm volatile("add.rn.f32 %0, %0, %1;" : "+f"(s) : "f"(ex[(q - 2) % 3]));
        if (q < 32) asm volatile("ex2.approx.ftz.f32 %0, %1;" : "=f"(ey[q % 3]) : "f"(y));
        if (q >= 2) asm volatile("add.rn.f32 %0, %0, %1;" : "+f"(s) : "f"(ey[(q - 2) % 3]));
    }
    return s;
}

// red[warp * pitch + j] = sum over the warp's 2,048 pairs of exp2(-cs[j] D) for
// every j < n (FP32).  cs[j] > 0 in shared memory.  Four j at a time: the four
// lane sums are reduced together (a lane halves the list at each of two
// exchanges: 6 shuffles instead of 20; the additions are those of a butterfly
// over lane distances 16, 8, 4, 2, 1).
__device__ __forceinline__ void pt_exp_sums(const f32x2 (&D)[8][4], const float* cs, int n, float* red, int pitch) {
    const int lane = pt_tid() & 31, warp = pt_tid() >> 5;
    for (int j = 0; j < n; j += 4) {
        float s[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            s[u] = 0.f;
            if (j + u < n) s[u] = pt_exp_sum(D, -cs[min(j + u, n - 1)]);   // a branch: uniform over the group
        }
#pragma unroll
        for (int half = 2, o = 16; half > 0; half >>= 1, o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int u = 0; u < half; ++u) {
                const float keep = up ? s[u + half] : s[u], give = up ? s[u] : s[u + half];
                s[u] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s[0] += __shfl_xor_sync(0xffffffffu, s[0], o);
        const int jj = j + (lane >> 3);   // lane bits 4, 3 chose halves of 2, 1
        if ((lane & 7) == 0 && jj < n) red[warp * pitch + jj] = s[0];
    }
}

}  // namespace kevd
