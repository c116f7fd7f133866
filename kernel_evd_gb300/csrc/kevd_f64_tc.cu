// FP64 products on the tensor cores in exact slices.
//
// The method is the error-free slicing of K. Ozaki, T. Ogita, S. Oishi and S. M. Rump,
// Error-free transformations of matrix multiplication by using fast routines of matrix
// multiplication, Numer. Algorithms 59 (2012), with digits in fixed point.
//
// The FP64 pipe of this GPU does 2 FMAs per clock and SM; the f16 tensor pipe
// does 4096.  A matrix entry is turned into fixed point relative to the largest
// entry of its row (of its column for a Gram), q = rn(x 2^(62 - e)) with
// |x| <= 2^e, and q into eight signed base-256 digits, q = sum_i a_i 256^(7-i)
// with |a_0| <= 64 and a_i in [-128, 127].  Digits are exact in f16, products of
// digits and their sums over a block of 192 terms are integers, exact in the FP32
// accumulators up to 2^24 (only S_6 and S_7 below can pass that, by a third at most,
// if the digits of all terms line up at +-128; they then lose units of 2^-60.  Squared
// distances, whose exact zeros matter, keep blocks of 128 terms: always exact).  The product of two entries is then
//
//   x y = 2^(ex + ey) sum_{i,j} a_i b_j 2^(-8 (i + j) - 12)
//
// of which the 36 digit pairs with i + j <= 7 are computed, one accumulator per
// i + j (what is left out is of the size of the last digit's rounding where the
// entries are of one size; see tail pairs below).  Every
// 192 terms the eight integer sums S_d leave Tensor Memory and are added, still
// exactly, to two 64-bit integers per output,
//
//   hi += S_0 2^24 + S_1 2^16 + S_2 2^8 + S_3,   lo likewise from S_4 .. S_7,
//
// so the long sum has no rounding at all; the result is rounded once to FP64.
// The error of an output is thus the fixed-point rounding of its inputs,
// 2^-63 of the row's (column's) largest entry each, and the pairs left out, against
// one FP64 rounding per product and per sum: an entry keeps its 53 bits down to 2^-10
// of the largest.
//
// Tail pairs (F from /linv).  There the entries of a row differ by orders of magnitude,
// an output's products may all be small against the rows' largest entries, and the 7
// pairs with i + j = 8 are 20 times the inputs' rounding.  They are added to the
// accumulator of i + j = 7.  For that the digits carry their weight, a_i 2^(-8 i), which
// f16 cannot hold and bf16 can (8 significant bits hold a digit): 14 more MMAs of 64
// columns a stage, and two more operations per pair of digits.  N = 20,000, r = 1,000,
// d = 64, errors of the entries of F relative to sum |K| |Linv|: rms 4.2e-16 without
// the pairs, 6.2e-17 with them (2.4e-16 on the FP64 pipe); N = 100,000, r = 1,024, the
// call 12.5 and 13.5 ms.
//
// CTA (512 threads): output tile 128 x 64, 32 terms per stage, two stages of
// shared memory (8 digit planes of A, 128 x 32 f16, and of B, 64 x 32 f16,
// SWIZZLE_64B, 96 KB), eight 64-column accumulators in Tensor Memory (all 512
// columns).  Warps 0-7 (A) and 8-11 (B) load packed digits (8 bytes per entry; the
// next stage's while this one is worked on) and write the f16 planes; every sixth
// stage all warps drain their part of the accumulators (warp w: lanes 32 (w % 4),
// columns 16 (w / 4)); a thread of warp 15 issues the MMAs of a stage, plane i of A
// against the 8 - i planes of B that it meets, side by side (24 MMAs of up to 256
// columns, 2,300 clocks, against 72 of 64 columns that each read A again).
// Accumulator i is complete after plane i, so the first ones of a block are
// drained while its last MMAs run.  Every wait is bounded and reports to an error
// flag.  Gram of 200,000 x 1,000 with its digits: 7.7 ms (FP64 pipe 204 ms); 11.7 with
// planes written by the issuing warp too, which then took planes and MMAs in turn,
// 8.6 with blocks of 128 terms.  A stage takes about 4,900 clocks: 2,800 for the MMAs,
// which read 240 KB of shared memory against 96 KB of stores, the rest mostly the
// drains, during which the tensor core has at most two stages to work on.
#include "kevd_internal.cuh"
#include "kevd_f64_tc.cuh"
#include "kevd_tc.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

namespace kevd {

namespace {

constexpr int kM = 128, kN = 64, kKs = 32;   // output tile, terms per stage
constexpr int kSlices = 8;
constexpr int kDiags = kSlices;              // digit pairs i + j = d, d < 8
constexpr int kBlockStages = 6;              // 192 terms per integer block (kernel blocks: 128)
constexpr int kAPlane = kM * kKs * 2, kBPlane = kN * kKs * 2;
constexpr int kStageBytes = kSlices * (kAPlane + kBPlane);
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kAWarps = 8, kBWarps = 4;      // expand the digits of A and of B
constexpr int kMmaWarp = kWarps - 1;         // its lane 0 issues the MMAs
constexpr uint32_t kTmemCols = 512;
constexpr uint64_t kTimeoutNs = 4000000000ull;
constexpr uint64_t kZeroDigits = 0x8080808080808080ull;   // q = 0: every digit byte holds digit + 128
static_assert(kStageBytes % 1024 == 0 && 2 * kStageBytes + 2048 <= 227 * 1024, "shared memory per CTA");
static_assert(kDiags * kN == (int)kTmemCols, "Tensor Memory");

struct Bars {
    uint64_t full[2], empty[2], accf[kDiags], acce[kDiags], done;
    uint32_t tmem_base;
};
constexpr size_t kSmem = 2 * (size_t)kStageBytes + sizeof(Bars) + 1024;

// D[tmem] (+)= A B^T, kind::f16, both operands in shared memory.
__device__ __forceinline__ void mma_f16_ss(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Packed digits of y, |y| <= 2^e: q = rn(y 2^(62 - e)) (ties away from zero), plus
// 128 in every digit's byte.
__device__ __forceinline__ uint64_t pack_digits(double y, int e) {
    const uint64_t b = (uint64_t)__double_as_longlong(y);
    const int ex = (int)(b >> 52) & 0x7ff;
    const int sh = 1023 + e - ex;                                                 // 0 at |y| = 2^e
    const uint64_t m = ((b & 0xfffffffffffffull) | 0x10000000000000ull) << 10;    // m / 2^62 in [1, 2)
    uint64_t q = 0;
    if (ex != 0 && sh >= 0 && sh < 64) q = sh == 0 ? m : (m + (1ull << (sh - 1))) >> sh;
    return ((b >> 63) ? 0ull - q : q) + kZeroDigits;
}

// Exponent e with |y| <= 2^e from the bits of |y| (0 for 0 and non-finite values).
__device__ __forceinline__ int digits_exp(uint64_t abs_bits) {
    const int ex = (int)(abs_bits >> 52);
    if (abs_bits == 0 || ex == 0x7ff) return 0;
    return ex - 1023 + ((abs_bits & 0xfffffffffffffull) ? 1 : 0);
}

// Two digits + 128, in bytes 0 and 2 of x, as two bf16 digits times 2^(-8 plane): u is
// 128 + (u & 127) minus 256 or, with bit 7, 128, which bf16 holds.
__device__ __forceinline__ uint32_t digits_bf16x2(uint32_t x, int plane) {
    const uint32_t w = (uint32_t)plane << 10;   // 8 plane in the exponent field
    const uint32_t hi = (x & 0x007f007fu) | ((0x4300u - w) * 0x10001u);
    const uint32_t lo = (x & 0x00800080u) ^ ((0x4380u - w) * 0x10001u);
    const __nv_bfloat162 d = __hsub2(*reinterpret_cast<const __nv_bfloat162*>(&hi), *reinterpret_cast<const __nv_bfloat162*>(&lo));
    return *reinterpret_cast<const uint32_t*>(&d);
}

// Eight packed entries along K -> the 16-byte piece of each plane: f16 digits, or
// (kTail) bf16 digits times 2^(-8 plane).
template <bool kTail>
__device__ __forceinline__ void store_planes(const uint64_t (&w)[8], uint8_t* planes, int plane_bytes, uint32_t off) {
    const __half2 bias = __half2half2(__ushort_as_half((unsigned short)0xE480));   // -1152
#pragma unroll
    for (int word = 0; word < 2; ++word) {   // digits 0 .. 3 in the high word, 4 .. 7 in the low one
        uint32_t h[4][4];
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const uint32_t x0 = (uint32_t)(w[2 * p] >> (word ? 0 : 32)), x1 = (uint32_t)(w[2 * p + 1] >> (word ? 0 : 32));
            // the same bytes of both entries side by side: two digits per register
            const uint32_t g[2] = {__byte_perm(x0, x1, 0x6273), __byte_perm(x0, x1, 0x4051)};
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                if constexpr (kTail) {
                    h[s][p] = digits_bf16x2(__byte_perm(g[s >> 1], 0u, (s & 1) ? 0x4342 : 0x4140), 4 * word + s);
                    continue;
                }
                // 0x64uu is the f16 1024 + u; minus 1152 leaves the digit u - 128
                const uint32_t v = __byte_perm(g[s >> 1], 0x64646464u, (s & 1) ? 0x4342 : 0x4140);
                const __half2 d = __hadd2(*reinterpret_cast<const __half2*>(&v), bias);
                h[s][p] = *reinterpret_cast<const uint32_t*>(&d);
            }
        }
#pragma unroll
        for (int s = 0; s < 4; ++s)
            *reinterpret_cast<uint4*>(planes + (4 * word + s) * plane_bytes + off) =
                make_uint4(h[s][0], h[s][1], h[s][2], h[s][3]);
    }
}

// Where the tile's operands come from.
//   Gram: both from the column-scaled digits of one panel, entry (column c, row i)
//         at q[i * ld + c]
//   rows: A from rows i0 .., B from rows n0 .., entry (row, k) at [row * ld + k]
struct Operand {
    const uint64_t* p;
    int64_t ld;
    int64_t first, count;   // first output row / column of the tile, and how many exist
};

// Loads that stay where they are written: left to the compiler, they sink to
// their first use behind the next stage's wait.
__device__ __forceinline__ uint64_t ld_here(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.global.nc.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void ld_here2(const uint64_t* p, uint64_t& a, uint64_t& b) {
    asm volatile("ld.global.nc.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p));
}

// Eight entries along K, from k0 on, of output row m of the tile (zeros from k1 on).
template <bool kGram>
__device__ __forceinline__ void load_words(const Operand& o, int m, int64_t k0, int64_t k1, uint64_t (&w)[8]) {
    constexpr int n = 8;
    const int left = m < o.count ? (int)max((int64_t)0, min((int64_t)n, k1 - k0)) : 0;
    if constexpr (kGram) {
        const uint64_t* src = o.p + k0 * o.ld + o.first + m;
        if (left == n) {
#pragma unroll
            for (int u = 0; u < n; ++u) w[u] = ld_here(src + u * o.ld);
        } else {
#pragma unroll
            for (int u = 0; u < n; ++u) w[u] = u < left ? ld_here(src + u * o.ld) : kZeroDigits;
        }
    } else {
        const uint64_t* src = o.p + (o.first + m) * o.ld + k0;
        if (left == n) {
#pragma unroll
            for (int u = 0; u < n; u += 2) ld_here2(src + u, w[u], w[u + 1]);
        } else {   // pairs: rows are padded to a multiple of 4 words
#pragma unroll
            for (int u = 0; u < n; u += 2) {
                w[u] = w[u + 1] = kZeroDigits;
                if (u < left) ld_here2(src + u, w[u], w[u + 1]);
            }
        }
    }
}

// One 128 x 64 tile: sums over k in [k0, k1) into (hi, lo) of the thread's 16
// outputs, row 32 (warp % 4) + lane, columns 16 (warp / 4) ...  Called by the
// whole CTA.  kTail: with the digit pairs i + j = 8.
template <bool kGram, int kBlockStages = ::kevd::kBlockStages, bool kTail = false>
__device__ __forceinline__ void tile_sums(const Operand& A, const Operand& B, int64_t k0, int64_t k1, uint8_t* base,
                                          Bars* bar, int* err, int64_t (&hi)[16], int64_t (&lo)[16]) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t n_st = k1 > k0 ? (k1 - k0 + kKs - 1) / kKs : 0;
    if (tid == 0) {
        for (int s = 0; s < 2; ++s) {
            tc::mbar_init(&bar->full[s], kAWarps + kBWarps);
            tc::mbar_init(&bar->empty[s], 1);
        }
        for (int d = 0; d < kDiags; ++d) {
            tc::mbar_init(&bar->accf[d], 1);
            tc::mbar_init(&bar->acce[d], kWarps);
        }
        tc::mbar_init(&bar->done, 1);
        tc::mbar_fence_init();
    }
    if (warp == kMmaWarp) {
        tc::tmem_alloc(&bar->tmem_base, kTmemCols);
        tc::tmem_relinquish();
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tbase = bar->tmem_base;
    const uint32_t tlane = tbase + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(16 * (warp >> 2));
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 16; ++c) hi[c] = lo[c] = 0;

    // the accumulators of block blk, each handed back as soon as it is read
    auto drain = [&](int64_t blk) {
#pragma unroll 1
        for (int half = 0; half < 2 && ok; ++half) {
#pragma unroll 1
            for (int d = 4 * half; d < 4 * half + 4; ++d) {
                if (!tc::mbar_wait(&bar->accf[d], (uint32_t)blk & 1u, kTimeoutNs)) {
                    atomicExch(err, 23);
                    ok = false;
                    break;
                }
                tc::tc_fence_after();
                float v[16];
                tc::tmem_ld16(tlane + (uint32_t)(d * kN), v);
                tc::tmem_wait_ld();
                tc::tc_fence_before();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&bar->acce[d]);
                const int w = 1 << (8 * (3 - (d & 3)));
                if constexpr (kTail) {   // the digits' weights: back to integers (i + j = 8 to the nearest)
                    const float up = __int_as_float((127 + 8 * d) << 23);
#pragma unroll
                    for (int c = 0; c < 16; ++c) v[c] *= up;
                }
                if (half == 0) {
#pragma unroll
                    for (int c = 0; c < 16; ++c) hi[c] += (int64_t)__float2int_rn(v[c]) * w;
                } else {
#pragma unroll
                    for (int c = 0; c < 16; ++c) lo[c] += (int64_t)__float2int_rn(v[c]) * w;
                }
            }
        }
    };
    // the MMAs of stage s (one thread)
    auto issue = [&](int64_t s) {
        const int slot = (int)(s & 1);
        const int64_t blk = s / kBlockStages;
        const bool first = s % kBlockStages == 0, last = s % kBlockStages == kBlockStages - 1 || s == n_st - 1;
        if (!tc::mbar_wait(&bar->full[slot], (uint32_t)(s >> 1) & 1u, kTimeoutNs)) {
            atomicExch(err, 21);
            return false;
        }
        tc::tc_fence_after();
        const uint32_t a0 = tc::smem_u32(base + (size_t)slot * kStageBytes);
        const uint64_t da = tc::desc_sw64(a0), db = tc::desc_sw64(a0 + kSlices * kAPlane);
        // plane i of A against planes 0 .. 7 - i of B, which lie one behind the other
        // like the accumulators i .. 7 they go to: MMAs of up to 256 columns
#pragma unroll
        for (int i = 0; i < kSlices; ++i) {
#pragma unroll
            for (int j = 0; j < kSlices - i; j += 4) {
                const int n = kN * min(4, kSlices - i - j);
                if (i == 0 && first && blk > 0) {   // the block before has left these accumulators
#pragma unroll 1
                    for (int d = j; d < j + 4; ++d)
                        if (!tc::mbar_wait(&bar->acce[d], (uint32_t)(blk - 1) & 1u, kTimeoutNs)) {
                            atomicExch(err, 22);
                            return false;
                        }
                    tc::tc_fence_after();
                }
#pragma unroll
                for (int ks = 0; ks < kKs / 16; ++ks)   // +32 bytes of K per MMA
                    mma_f16_ss(tbase + (uint32_t)((i + j) * kN), da + (uint64_t)((i * kAPlane + 32 * ks) >> 4),
                               db + (uint64_t)((j * kBPlane + 32 * ks) >> 4),
                               kTail ? tc::idesc_bf16(kM, n) : tc::idesc_f16(kM, n),
                               first && i == 0 && ks == 0 ? 0u : 1u);
            }
            if (kTail && i > 0) {   // plane 8 - i of B
#pragma unroll
                for (int ks = 0; ks < kKs / 16; ++ks)
                    mma_f16_ss(tbase + (uint32_t)((kDiags - 1) * kN), da + (uint64_t)((i * kAPlane + 32 * ks) >> 4),
                               db + (uint64_t)(((kSlices - i) * kBPlane + 32 * ks) >> 4), tc::idesc_bf16(kM, kN), 1u);
            }
            if (last) tc::mma_commit(&bar->accf[i]);   // accumulator i is complete
        }
        tc::mma_commit(&bar->empty[slot]);
        return true;
    };
    if (warp < kAWarps + kBWarps) {
        // this thread's share of a stage: two pieces of eight terms of a row of A or of B
        const bool is_a = warp < kAWarps;
        const Operand& O = is_a ? A : B;
        const int t = is_a ? tid : tid - 32 * kAWarps, rows = is_a ? kM : kN;
        const int m0 = kGram ? t & (rows - 1) : t >> 2, m1 = kGram ? m0 : m0 + rows / 2;
        const int g0 = kGram ? 8 * (t / rows) : 8 * (t & 3), g1 = kGram ? g0 + 16 : g0;
        const int plane = is_a ? kAPlane : kBPlane;
        uint8_t* planes = base + (is_a ? 0 : kSlices * kAPlane);
        const uint32_t off0 = tc::sw64_off16((uint32_t)m0, (uint32_t)g0), off1 = tc::sw64_off16((uint32_t)m1, (uint32_t)g1);
        uint64_t w0[8], w1[8];
        load_words<kGram>(O, m0, k0 + g0, k1, w0);
        load_words<kGram>(O, m1, k0 + g1, k1, w1);
        for (int64_t s = 0; s < n_st && ok; ++s) {
            const int slot = (int)(s & 1);
            if (!tc::mbar_wait(&bar->empty[slot], ((uint32_t)(s >> 1) & 1u) ^ 1u, kTimeoutNs)) {
                atomicExch(err, 24);
                ok = false;
                break;
            }
            const int64_t kn = k0 + (s + 1) * kKs;   // past the end: zeros, never used
            store_planes<kTail>(w0, planes + (size_t)slot * kStageBytes, plane, off0);
            load_words<kGram>(O, m0, kn + g0, k1, w0);
            store_planes<kTail>(w1, planes + (size_t)slot * kStageBytes, plane, off1);
            tc::fence_async_smem();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&bar->full[slot]);
            load_words<kGram>(O, m1, kn + g1, k1, w1);
            if (s % kBlockStages == 0 && s > 0) drain(s / kBlockStages - 1);
        }
    } else {
        for (int64_t s = 0; s < n_st && ok; ++s) {
            if (s % kBlockStages == 0 && s > 0) drain(s / kBlockStages - 1);
            if (warp == kMmaWarp) {
                if (lane == 0 && ok) ok = issue(s);
                ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
            }
        }
    }
    if (ok && n_st > 0) drain((n_st - 1) / kBlockStages);
    if (warp == kMmaWarp && lane == 0) {
        tc::mma_commit(&bar->done);   // every MMA is done before the Tensor Memory is released
        if (!tc::mbar_wait(&bar->done, 0u, kTimeoutNs)) atomicExch(err, 25);
    }
    __syncwarp();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    if (warp == kMmaWarp) tc::tmem_dealloc(tbase, kTmemCols);
}

// 2^-36 hi + 2^-68 lo: the sum in units of 2^(ex + ey).  hi is cut in two (its
// upper part exact in FP64), so that only the last addition rounds visibly.
__device__ __forceinline__ double tile_value(int64_t hi, int64_t lo) {
    const int64_t up = hi & ~(int64_t)0xfffff;
    return (double)up * 0x1.0p-36 + fma((double)(hi - up), 0x1.0p-36, (double)lo * 0x1.0p-68);
}

// ---- Gram -----------------------------------------------------------------------
// Tile t -> 128 columns from 128 ta against 64 columns from 64 tb, tb <= 2 ta + 1.
__device__ __forceinline__ void gram_tile(int64_t t, int64_t& ta, int64_t& tb) {
    int64_t i = (int64_t)((sqrt(4.0 * (double)t + 1.0) - 1.0) * 0.5);
    while (i * (i + 1) > t) --i;
    while ((i + 1) * (i + 2) <= t) ++i;
    ta = i;
    tb = t - i * (i + 1);
}

// partial[(split * n_tiles + tile)][n][m] (+)= the tile's sums over the split's rows.
__global__ void __launch_bounds__(kThreads, 1)
gram_f64_tc_kernel(const uint64_t* __restrict__ q, int64_t rows, int64_t k, int64_t ld, int n_tiles,
                   int64_t rows_per, int add, double* __restrict__ partial, int* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Bars* bar = reinterpret_cast<Bars*>(base + 2 * (size_t)kStageBytes);
    const int64_t tix = blockIdx.x % n_tiles, split = blockIdx.x / n_tiles;
    int64_t ta, tb;
    gram_tile(tix, ta, tb);
    const int64_t r0 = min(rows, split * rows_per), r1 = min(rows, r0 + rows_per);
    const Operand A{q, ld, ta * kM, min((int64_t)kM, k - ta * kM)};
    const Operand B{q, ld, tb * kN, min((int64_t)kN, k - tb * kN)};
    int64_t hi[16], lo[16];
    tile_sums<true>(A, B, r0, r1, base, bar, err, hi, lo);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double* out = partial + (int64_t)blockIdx.x * kM * kN + (int64_t)(16 * (warp >> 2)) * kM + 32 * (warp & 3) + lane;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const double v = tile_value(hi[c], lo[c]);
        out[c * kM] = add ? out[c * kM] + v : v;
    }
}

// G (column-major, full) from the partial tiles, lower entries mirrored.
__global__ void gram_f64_reduce_kernel(const double* __restrict__ partial, int n_tiles, int n_split, int64_t k,
                                       const int* __restrict__ e, const unsigned long long* __restrict__ diag8,
                                       double* __restrict__ G) {
    int64_t ta, tb;
    gram_tile(blockIdx.x, ta, tb);
    for (int x = threadIdx.x; x < kM * kN; x += blockDim.x) {
        const int n = x / kM, m = x - n * kM;
        const int64_t ga = ta * kM + m, gb = tb * kN + n;
        if (ga >= k || gb >= k || gb > ga) continue;
        double s = 0.0;
        for (int p = 0; p < n_split; ++p) s += partial[((int64_t)p * n_tiles + blockIdx.x) * kM * kN + x];
        if (ga == gb) s += (double)(int64_t)diag8[ga] * 0x1.0p-76;
        s = ldexp(s, e[ga] + e[gb]);
        G[gb * k + ga] = s;
        G[ga * k + gb] = s;
    }
}

// max_i |s_i F(i, c)| per column, as the bits of a non-negative double.
__global__ void __launch_bounds__(256) colmax_kernel(const double* __restrict__ F, int64_t ldF, int64_t N, int64_t k,
                                                     const double* __restrict__ s, int64_t rows_per,
                                                     unsigned long long* __restrict__ colmax) {
    const int64_t c = (int64_t)blockIdx.x * 256 + threadIdx.x;
    const int64_t r0 = (int64_t)blockIdx.y * rows_per, r1 = min(N, r0 + rows_per);
    if (c >= k) return;
    unsigned long long m = 0;
#pragma unroll 8
    for (int64_t i = r0; i < r1; ++i) {
        const double y = s ? F[i * ldF + c] * s[i] : F[i * ldF + c];
        m = max(m, (unsigned long long)__double_as_longlong(y) & 0x7fffffffffffffffull);
    }
    atomicMax(colmax + c, m);
}

__global__ void colexp_kernel(const unsigned long long* __restrict__ colmax, int64_t k, int* __restrict__ e) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c < k) e[c] = digits_exp(colmax[c]);
}

// Column digits of a panel.  The digit pairs with i + j = 8 that the products
// leave out average out between two columns, but not of a column with itself
// (a_4^2 >= 0): their sum is added up exactly per column, for the diagonal of G.
__global__ void __launch_bounds__(256) digits_cols_kernel(const double* __restrict__ F, int64_t ldF, int64_t rows,
                                                          int64_t k, const double* __restrict__ s,
                                                          const int* __restrict__ e, uint64_t* __restrict__ q,
                                                          int64_t ld, unsigned long long* __restrict__ diag8) {
    const int64_t c = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (c >= k) return;
    const int ec = e[c];
    int64_t sum = 0;
#pragma unroll 4
    for (int64_t i = blockIdx.y; i < rows; i += gridDim.y) {
        const uint64_t w = pack_digits(s ? F[i * ldF + c] * s[i] : F[i * ldF + c], ec);
        q[i * ld + c] = w;
        int a[kSlices];
#pragma unroll
        for (int t = 1; t < kSlices; ++t) a[t] = (int)((w >> (8 * (kSlices - 1 - t))) & 0xff) - 128;
        sum += 2 * (a[1] * a[7] + a[2] * a[6] + a[3] * a[5]) + a[4] * a[4];
    }
    atomicAdd(diag8 + c, (unsigned long long)sum);   // integers: any order gives the same
}

// Columns whose fixed point would lose digits: not finite, or largest entry above
// kSpike times the root mean square (G(c, c) / N).  The pairs left out are worth
// 2e-19 of the product of the largest entries per term, at random: with entries
// up to 512 times the root mean square, 5e-14 / sqrt(N) of a Gram entry's scale
// (and below N = 2^18 no column can be that uneven).
constexpr double kSpike = 512.0;
__global__ void gram_check_kernel(const unsigned long long* __restrict__ colmax, const double* __restrict__ G, int64_t k,
                                  int64_t N, int* __restrict__ bad) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= k) return;
    const double m = __longlong_as_double((long long)colmax[c]);
    if (!(m == 0.0 || (isfinite(m) && m * sqrt((double)N) <= kSpike * sqrt(G[c * k + c])))) atomicOr(bad, 1);
}

// The same from one row of every 16, before the product: part[y][c] the sum of squares of
// column c over the y-th share of those rows, then bad |= 1 where a column is beyond twice
// the limit.  Only above N = kSpike^2 rows can a column be so uneven.  N = 400,000, k =
// 300: the product that is then thrown away takes 3.6 ms beside 43.6 on the FP64 pipe.
constexpr int kSampleParts = 64;
__global__ void __launch_bounds__(256) colsq_sample_kernel(const double* __restrict__ F, int64_t ldF, int64_t N, int64_t k,
                                                           const double* __restrict__ s, double* __restrict__ part) {
    const int64_t c = (int64_t)blockIdx.x * 256 + threadIdx.x;
    if (c >= k) return;
    double v = 0.0;
#pragma unroll 8
    for (int64_t b = blockIdx.y; 16 * b < N; b += kSampleParts) {
        const int64_t i = 16 * b + ((uint32_t)b * 0x9E3779B1u >> 28);
        const double y = i < N ? (s ? F[i * ldF + c] * s[i] : F[i * ldF + c]) : 0.0;
        v = fma(y, y, v);
    }
    part[blockIdx.y * k + c] = v;
}
__global__ void sample_check_kernel(const unsigned long long* __restrict__ colmax, const double* __restrict__ part,
                                    int64_t k, int64_t N, int* __restrict__ bad) {
    const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= k) return;
    double v = 0.0;
    for (int y = 0; y < kSampleParts; ++y) v += part[y * k + c];
    const double m = __longlong_as_double((long long)colmax[c]);
    if (!(m == 0.0 || (isfinite(m) && m * sqrt((double)N) <= 2.0 * kSpike * sqrt(16.0 * v)))) atomicOr(bad, 1);
}

// ---- row products ------------------------------------------------------------------
// One warp per row: the row's exponent, then its digits.
__global__ void __launch_bounds__(256) digits_rows_kernel(const double* __restrict__ A, int64_t rows, int64_t K,
                                                          int64_t sr, int64_t sc, int lower,
                                                          uint64_t* __restrict__ out, int64_t ld,
                                                          int* __restrict__ ea, int* __restrict__ prefix) {
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= rows) return;
    const int64_t kc = lower ? min(K, i + 1) : K, nb = (K + kN - 1) / kN;
    unsigned long long m = 0;
    for (int64_t b = 0; b < nb; ++b) {
#pragma unroll
        for (int u = 0; u < kN; u += 32) {
            const int64_t c = b * kN + u + lane;
            if (c < kc) m = max(m, (unsigned long long)__double_as_longlong(A[i * sr + c * sc]) & 0x7fffffffffffffffull);
        }
        if (prefix || b == nb - 1) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
            if (prefix && lane == 0) prefix[i * nb + b] = m ? digits_exp(m) : -2048;
        }
    }
    const int e = digits_exp(m);
    if (lane == 0) ea[i] = m >= 0x7ff0000000000000ull ? kDigitsNotFinite : e;
    for (int64_t c = lane; c < ld; c += 32)
        out[i * ld + c] = c < kc ? pack_digits(A[i * sr + c * sc], e) : kZeroDigits;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One output of a row product (NaN where an operand row is not finite).
__device__ __forceinline__ double row_value(int64_t hi, int64_t lo, int e, int en) {
    return e == kDigitsNotFinite || en == kDigitsNotFinite ? (double)NAN : ldexp(tile_value(hi, lo), e + en);
}

__global__ void __launch_bounds__(kThreads, 1)
rows_f64_tc_kernel(const uint64_t* __restrict__ Aq, const int* __restrict__ ea, int64_t M,
                   const uint64_t* __restrict__ Bq, const int* __restrict__ eb, int64_t n_cols, int64_t K, int64_t ld,
                   const double* __restrict__ scale, float* __restrict__ C, int64_t ldc, int* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Bars* bar = reinterpret_cast<Bars*>(base + 2 * (size_t)kStageBytes);
    const int64_t i0 = (int64_t)blockIdx.y * kM, n0 = (int64_t)blockIdx.x * kN;
    const Operand A{Aq, ld, i0, min((int64_t)kM, M - i0)};
    const Operand B{Bq, ld, n0, min((int64_t)kN, n_cols - n0)};
    int64_t hi[16], lo[16];
    tile_sums<false>(A, B, 0, K, base, bar, err, hi, lo);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t i = i0 + 32 * (warp & 3) + lane;
    if (i >= M) return;
    const int e = ea[i];
    const double sc = scale[i];
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const int64_t n = n0 + 16 * (warp >> 2) + c;
        if (n < n_cols) C[i * ldc + n] = (float)(row_value(hi[c], lo[c], e, eb[n]) * sc);
    }
}

// The first 64 columns, whose sums are short and may miss the row's largest entry
// altogether, are formed in FP64 (2,080 products a row), and so is a row's part of
// a later tile when the entries of the tiles before lie more than 2^-kPrefixBits
// below that largest entry.
constexpr int kPrefixBits = 4;
__device__ __forceinline__ bool tri_direct(int ek, int prefix) { return ek - prefix > kPrefixBits; }

__global__ void __launch_bounds__(kThreads, 1)
tri_f64_tc_kernel(const double* __restrict__ K, const double* __restrict__ Linv, const uint64_t* __restrict__ Kq,
                  const uint64_t* __restrict__ Lq, const int* __restrict__ ek, const int* __restrict__ el,
                  const int* __restrict__ prefix, int64_t M, int64_t r, int64_t ld, double* __restrict__ Fd,
                  float* __restrict__ Ff, int64_t ldF, const int* __restrict__ skip, int* __restrict__ err) {
    if (*skip) return;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Bars* bar = reinterpret_cast<Bars*>(base + 2 * (size_t)kStageBytes);
    const int64_t i0 = (int64_t)blockIdx.y * kM, n0 = (int64_t)blockIdx.x * kN, nb = (r + kN - 1) / kN;
    int64_t hi[16], lo[16];
    if (blockIdx.x > 0) {
        const Operand A{Kq, ld, i0, min((int64_t)kM, M - i0)};
        const Operand B{Lq, ld, n0, min((int64_t)kN, r - n0)};
        tile_sums<false, kBlockStages, true>(A, B, 0, min(r, n0 + kN), base, bar, err, hi, lo);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t i = i0 + 32 * (warp & 3) + lane;
    if (i >= M) return;
    const int e = ek[i];
    const bool direct = blockIdx.x == 0 || tri_direct(e, prefix[i * nb + blockIdx.x - 1]);
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const int64_t n = n0 + 16 * (warp >> 2) + c;
        if (n >= r) break;
        double v;
        if (direct) {
            v = 0.0;
            for (int64_t k = 0; k <= n; ++k) v = fma(K[i * r + k], Linv[k * r + n], v);
        } else {
            v = row_value(hi[c], lo[c], e, el[n]);
        }
        if (Fd) Fd[i * ldF + n] = v;
        else Ff[i * ldF + n] = (float)v;
    }
}

// |x| 2^-e in FP32, rounded towards 0, for |x| <= 2^e (0 below 2^-126).
__device__ __forceinline__ float scaled_abs(double x, int e) {
    const uint32_t hi = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    const int ex = (int)(hi >> 20) - e - (1023 - 127);
    return ex <= 0 ? 0.f : __uint_as_float(((uint32_t)ex << 23) | ((hi & 0xfffffu) << 3) | ((uint32_t)__double2loint(x) >> 29));
}

// Sum and count over 32 columns of four sample rows of (n + 1) / S^2, S = sum_{k <= n}
// |K(i, k) Linv(n, k)| / 2^(ek + el), for the outputs that the digits form.  Thread (j, c)
// of 8 x 32 takes every eighth k of column c.  One wave of latency-bound CTAs; 1,024
// terms staged at a time for few barriers.
constexpr int kRangeChunk = 1024;
__global__ void __launch_bounds__(256)
tri_range_kernel(const double* __restrict__ K, const double* __restrict__ Linv, const int* __restrict__ ek,
                 const int* __restrict__ el, const int* __restrict__ prefix, int64_t M, int64_t r,
                 double* __restrict__ part) {
    __shared__ __align__(16) float ks[kRangeChunk][4];
    __shared__ float sums[8][32][4];
    __shared__ int64_t row[4];
    const int tid = threadIdx.x, c = tid & 31, j = tid >> 5;
    const int64_t nb = (r + kN - 1) / kN, n0 = (int64_t)blockIdx.x * 32, n = n0 + c;
    if (tid < 4) {
        uint64_t z = ((uint64_t)blockIdx.y * 4 + tid + 1) * 0x9E3779B97F4A7C15ull;   // splitmix64
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        row[tid] = (int64_t)((z >> 32) * (uint64_t)M >> 32);
    }
    __syncthreads();
    const int en = n < r ? el[n] : 0;
    const double* L = Linv + (n < r ? n : 0);
    float s[4] = {0.f, 0.f, 0.f, 0.f};
    const int64_t kend = min(r, n0 + 32);
    for (int64_t k0 = 0; k0 < kend; k0 += kRangeChunk) {
        const int kc = (int)min((int64_t)kRangeChunk, kend - k0);
        __syncthreads();
        {   // a wave along the row: row tid / 64 of the four
            const int64_t i = row[tid >> 6];
            const int e = ek[i];
#pragma unroll 4
            for (int k = tid & 63; k < kc; k += 64) ks[k][tid >> 6] = scaled_abs(K[i * r + k0 + k], e);
        }
        __syncthreads();
        const int kn = n < r ? (int)min((int64_t)kc, n + 1 - k0) : 0;
#pragma unroll 16
        for (int k = j; k < kn; k += 8) {
            const float l = scaled_abs(L[(k0 + k) * r], en);
            const float4 x = *reinterpret_cast<const float4*>(ks[k]);
            s[0] = fmaf(x.x, l, s[0]);
            s[1] = fmaf(x.y, l, s[1]);
            s[2] = fmaf(x.z, l, s[2]);
            s[3] = fmaf(x.w, l, s[3]);
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) sums[j][c][q] = s[q];
    __syncthreads();
    if (j != 0) return;
    double v = 0.0, cnt = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        float t = 0.f;
        for (int u = 0; u < 8; ++u) t += sums[u][c][q];
        const int64_t i = row[q];
        if (n < r && n >= kN && !tri_direct(ek[i], prefix[i * nb + n / kN - 1])) {
            v += (double)(n + 1) / ((double)t * (double)t);
            cnt += 1.0;
        }
    }
    v = warp_sum(v);
    cnt = warp_sum(cnt);
    if (c == 0) {
        double* out = part + 2 * (blockIdx.y * gridDim.x + blockIdx.x);
        out[0] = v;
        out[1] = cnt;
    }
}

// *skip from the parts, in a fixed order.  One warp.
__global__ void tri_suited_kernel(const double* __restrict__ part, int n, double limit, int* __restrict__ skip) {
    double v = 0.0, c = 0.0;
    for (int q = threadIdx.x; q < n; q += 32) {
        v += part[2 * q];
        c += part[2 * q + 1];
    }
    v = warp_sum(v);
    c = warp_sum(c);
    if (threadIdx.x == 0) *skip = c == 0.0 || v <= limit * limit * c ? 0 : 1;   // NaN: skip
}

// ---- kernel blocks -------------------------------------------------------------------
// max |X| as the bits of a non-negative float.
__global__ void __launch_bounds__(256) absmax_kernel(const float* __restrict__ X, int64_t n, unsigned* __restrict__ mx) {
    unsigned m = 0;
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256)
        m = max(m, __float_as_uint(X[i]) & 0x7fffffffu);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(mx, m);
}

// One warp per state: its digits, and its squared norm by the digit pairs that
// the tensor cores form of a product, so that ||x||^2 + ||s||^2 - 2 x s cancels
// exactly (an integer zero for x = s).
__global__ void __launch_bounds__(256) digits_states_kernel(const float* __restrict__ X, int64_t row0,
                                                            const int64_t* __restrict__ idx, int64_t n, int d, int e,
                                                            uint64_t* __restrict__ q, int64_t ld,
                                                            int64_t* __restrict__ norm) {
    const int lane = threadIdx.x & 31;
    const int64_t i = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= n) return;
    const float* x = X + (idx ? idx[i] : row0 + i) * d;
    int S[kDiags];
#pragma unroll
    for (int t = 0; t < kDiags; ++t) S[t] = 0;
    for (int64_t c = lane; c < ld; c += 32) {
        const uint64_t w = c < d ? pack_digits((double)x[c], e) : kZeroDigits;
        q[i * ld + c] = w;
        int a[kSlices];
#pragma unroll
        for (int t = 0; t < kSlices; ++t) a[t] = (int)((w >> (8 * (kSlices - 1 - t))) & 0xff) - 128;
#pragma unroll
        for (int t = 0; t < kDiags; ++t)
#pragma unroll
            for (int u = 0; u <= t; ++u) S[t] += a[u] * a[t - u];   // |S| <= 1024 x 8 x 2^14
    }
#pragma unroll
    for (int t = 0; t < kDiags; ++t)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) S[t] += __shfl_xor_sync(0xffffffffu, S[t], o);
    if (lane < 2) {
        int64_t v = 0;
#pragma unroll
        for (int t = 0; t < 4; ++t) v = v * 256 + (lane == 0 ? S[t] : S[4 + t]);
        norm[2 * i + lane] = v;
    }
}

// K tile: 128 states against 64.  What bounds it is the FP64 exponential (about
// 25 FP64 operations an entry), no longer the 2 d of a distance.
__global__ void __launch_bounds__(kThreads, 1)
kernel_f64_tc_kernel(const uint64_t* __restrict__ xq, const int64_t* __restrict__ xn, int64_t n,
                     const uint64_t* __restrict__ sq, const int64_t* __restrict__ sn, int64_t r, int d, int64_t ldq,
                     double scale_e, double* __restrict__ K, int64_t ld, int* __restrict__ err) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    Bars* bar = reinterpret_cast<Bars*>(base + 2 * (size_t)kStageBytes);
    const int64_t i0 = (int64_t)blockIdx.y * kM, n0 = (int64_t)blockIdx.x * kN;
    const Operand A{xq, ldq, i0, min((int64_t)kM, n - i0)};
    const Operand B{sq, ldq, n0, min((int64_t)kN, r - n0)};
    int64_t hi[16], lo[16];
    tile_sums<false, 4>(A, B, 0, d, base, bar, err, hi, lo);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t i = i0 + 32 * (warp & 3) + lane;
    if (i >= n) return;
    const int64_t xh = xn[2 * i], xl = xn[2 * i + 1];
#pragma unroll
    for (int c = 0; c < 16; ++c) {
        const int64_t col = n0 + 16 * (warp >> 2) + c;
        if (col >= r) break;
        const int64_t dh = xh + sn[2 * col] - 2 * hi[c], dl = xl + sn[2 * col + 1] - 2 * lo[c];
        K[i * ld + col] = exp(-scale_e * fmax(tile_value(dh, dl), 0.0));
    }
}

}  // namespace

// The digits carry a squared distance to about 2^-56 4^e, whatever its size; an
// FP64 sum of d squares carries it to a few 2^-53 of itself.  With 4^e scale up
// to 16 the exponent scale D then moves by at most 2^-52.
int states_exp(kevd_ctx* ctx, const float* X, int64_t N, int d, double scale, int* e, bool* suited, cudaStream_t st) {
    *suited = false;
    int rc = KEVD_OK;
    unsigned* mx = arena_get<unsigned>(ctx, "f64.xmax", 1, &rc);
    if (rc != KEVD_OK) return KEVD_OK;
    KEVD_CUDA(ctx, cudaMemsetAsync(mx, 0, sizeof(unsigned), st));
    absmax_kernel<<<(unsigned)std::min<int64_t>((N * d + 2047) / 2048, (int64_t)ctx->num_sms * 8), 256, 0, st>>>(X, N * d,
                                                                                                              mx);
    KEVD_LAUNCH(ctx);
    unsigned h = 0;
    KEVD_CUDA(ctx, cudaMemcpyAsync(&h, mx, sizeof(h), cudaMemcpyDeviceToHost, st));
    KEVD_CUDA(ctx, cudaStreamSynchronize(st));
    if (h >= 0x7f800000u) return KEVD_OK;
    float m;
    std::memcpy(&m, &h, sizeof(m));
    int ex = 0;
    std::frexp(m, &ex);   // m < 2^ex
    *e = ex;
    *suited = scale >= 0.0 && std::ldexp(scale, 2 * ex) <= 16.0;
    return KEVD_OK;
}

int launch_digits_states(kevd_ctx* ctx, const float* X, int64_t row0, const int64_t* idx, int64_t n, int d, int e,
                         StateDigits out, cudaStream_t st) {
    digits_states_kernel<<<(unsigned)((n + 7) / 8), 256, 0, st>>>(X, row0, idx, n, d, e, out.q, digits_ld(d), out.norm);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

int launch_kernel_f64_tc(kevd_ctx* ctx, StateDigits x, int64_t n, StateDigits s, int64_t r, int d, int e, double scale,
                         double* K, int64_t ld, int* err, cudaStream_t st) {
    KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&kernel_f64_tc_kernel), kSmem));
    const dim3 grid((unsigned)((r + kN - 1) / kN), (unsigned)((n + kM - 1) / kM));
    if (grid.y > 65535) return set_error(ctx, KEVD_ERR_ARG, "kernel_f64_tc: too many rows");
    kernel_f64_tc_kernel<<<grid, kThreads, kSmem, st>>>(x.q, x.norm, n, s.q, s.norm, r, d, digits_ld(d),
                                                        std::ldexp(scale, 2 * e), K, ld, err);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

int launch_digits_rows(kevd_ctx* ctx, const double* A, int64_t rows, int64_t K, int64_t lda, bool lower,
                       bool col_major, uint64_t* out, int* ea, int* prefix, cudaStream_t st) {
    digits_rows_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, st>>>(A, rows, K, col_major ? 1 : lda,
                                                                  col_major ? lda : 1, lower ? 1 : 0, out,
                                                                  digits_ld(K), ea, prefix);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

constexpr int64_t kMaxRowTiles = 65535;   // grid.y

int launch_rows_f64_tc(kevd_ctx* ctx, const uint64_t* A, const int* ea, int64_t M, const uint64_t* B, const int* eb,
                       int64_t n_cols, int64_t K, const double* scale, float* C, int64_t ldc, int* err,
                       cudaStream_t st) {
    KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&rows_f64_tc_kernel), kSmem));
    for (int64_t i = 0; i < M; i += kMaxRowTiles * kM) {
        const int64_t m = std::min(M - i, kMaxRowTiles * kM);
        const dim3 grid((unsigned)((n_cols + kN - 1) / kN), (unsigned)((m + kM - 1) / kM));
        rows_f64_tc_kernel<<<grid, kThreads, kSmem, st>>>(A + i * digits_ld(K), ea + i, m, B, eb, n_cols, K,
                                                          digits_ld(K), scale + i, C + i * ldc, ldc, err);
        KEVD_LAUNCH(ctx);
    }
    return KEVD_OK;
}

int launch_tri_f64_tc(kevd_ctx* ctx, const TriOperands& o, int64_t M, int64_t r, double* Fd, float* Ff, int64_t ldF,
                      const int* skip, int* err, cudaStream_t st) {
    KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&tri_f64_tc_kernel), kSmem));
    const dim3 grid((unsigned)((r + kN - 1) / kN), (unsigned)((M + kM - 1) / kM));
    if (grid.y > kMaxRowTiles) return set_error(ctx, KEVD_ERR_ARG, "tri_f64_tc: too many rows");
    tri_f64_tc_kernel<<<grid, kThreads, kSmem, st>>>(o.K, o.Linv, o.Kq, o.Lq, o.ek, o.el, o.prefix, M, r, digits_ld(r),
                                                     Fd, Ff, ldF, skip, err);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

int launch_tri_range(kevd_ctx* ctx, const TriOperands& o, int64_t M, int64_t r, double limit, double* part, int* skip,
                     cudaStream_t st) {
    const dim3 grid((unsigned)((r + 31) / 32), kRangeRows / 4);
    tri_range_kernel<<<grid, 256, 0, st>>>(o.K, o.Linv, o.ek, o.el, o.prefix, M, r, part);
    KEVD_LAUNCH(ctx);
    tri_suited_kernel<<<1, 32, 0, st>>>(part, (int)(grid.x * grid.y), limit, skip);
    KEVD_LAUNCH(ctx);
    return KEVD_OK;
}

int run_gram_f64_tc(kevd_ctx* ctx, const double* F, int64_t N, int64_t k, int64_t ldF, const double* s, double* G,
                    bool* done, cudaStream_t st) {
    *done = false;
    const int64_t na = (k + kM - 1) / kM;
    const int n_tiles = (int)(na * (na + 1));
    const int64_t ld = k;
    // digits in panels of rows, at most 2 GiB of them and 2^20 rows at a time (the
    // 64-bit sums hold 2^21 terms)
    const int64_t panel = std::min(std::min<int64_t>(N, 1 << 20), std::max<int64_t>(4096, ((int64_t)2 << 30) / (8 * ld)));
    // row splits: the fewest whose CTAs fill their waves to 95 %, at least 1,024 rows each
    int n_split = 1;
    const int max_split = (int)std::max<int64_t>(1, std::min<int64_t>(256, panel / 1024));
    double best = 0.0;
    for (int p = 1; p <= max_split; ++p) {
        const int64_t ctas = (int64_t)n_tiles * p;
        const double fill = (double)ctas / (double)((ctas + ctx->num_sms - 1) / ctx->num_sms * ctx->num_sms);
        if (fill > best + 1e-9) {
            best = fill;
            n_split = p;
        }
        if (fill >= 0.95) break;
    }
    const int64_t rows_per = ((panel + n_split - 1) / n_split + kKs * kBlockStages - 1) / (kKs * kBlockStages) *
                             (kKs * kBlockStages);
    int rc = KEVD_OK;
    uint64_t* q = arena_get<uint64_t>(ctx, "f64.q", (size_t)panel * ld, &rc);
    double* partial = arena_get<double>(ctx, "f64.part", (size_t)n_split * n_tiles * kM * kN, &rc);
    unsigned long long* colmax = arena_get<unsigned long long>(ctx, "f64.max", (size_t)2 * k, &rc);   // and diag8
    int* e = arena_get<int>(ctx, "f64.exp", (size_t)k + 2, &rc);
    // the caller's later buffers come first: these are free for them once the call
    // returns, and with no room for all of them none is kept
    struct Idle {
        kevd_ctx* ctx;
        ~Idle() {
            for (const char* b : {"f64.q", "f64.part", "f64.max", "f64.exp"}) ctx->arena.idle(b);
        }
    } idle{ctx};
    if (rc != KEVD_OK) return KEVD_OK;   // no room for the slices: not done
    int* flags = e + k;                  // error, unsuited column
    KEVD_CUDA(ctx, cudaMemsetAsync(colmax, 0, (size_t)2 * k * sizeof(*colmax), st));
    KEVD_CUDA(ctx, cudaMemsetAsync(flags, 0, 2 * sizeof(int), st));
    KEVD_CUDA(ctx, raise_smem_limit(reinterpret_cast<const void*>(&gram_f64_tc_kernel), kSmem));
    const unsigned cx = (unsigned)((k + 255) / 256);
    {
        const int64_t ny = std::min<int64_t>(std::max<int64_t>(1, N / 64), std::max<int64_t>(1, 16 * ctx->num_sms / cx));
        colmax_kernel<<<dim3(cx, (unsigned)ny), 256, 0, st>>>(F, ldF, N, k, s, (N + ny - 1) / ny, colmax);
        KEVD_LAUNCH(ctx);
    }
    colexp_kernel<<<cx, 256, 0, st>>>(colmax, k, e);
    KEVD_LAUNCH(ctx);
    if ((double)N > kSpike * kSpike) {
        colsq_sample_kernel<<<dim3(cx, kSampleParts), 256, 0, st>>>(F, ldF, N, k, s, partial);
        KEVD_LAUNCH(ctx);
        sample_check_kernel<<<cx, 256, 0, st>>>(colmax, partial, k, N, flags + 1);
        KEVD_LAUNCH(ctx);
        int bad = 0;
        KEVD_CUDA(ctx, cudaMemcpyAsync(&bad, flags + 1, sizeof(int), cudaMemcpyDeviceToHost, st));
        KEVD_CUDA(ctx, cudaStreamSynchronize(st));
        if (bad) return KEVD_OK;
    }
    {
        ProfScope ps(ctx, "gram_f64_tc", st);
        for (int64_t r = 0; r < N; r += panel) {
            const int64_t rows = std::min(panel, N - r);
            const unsigned ny = (unsigned)std::min<int64_t>(rows, std::max<int64_t>(1, 16 * ctx->num_sms / cx));
            digits_cols_kernel<<<dim3(cx, ny), 256, 0, st>>>(F + r * ldF, ldF, rows, k, s ? s + r : nullptr, e, q, ld,
                                                             colmax + k);
            KEVD_LAUNCH(ctx);
            gram_f64_tc_kernel<<<n_tiles * n_split, kThreads, kSmem, st>>>(q, rows, k, ld, n_tiles, rows_per, r > 0,
                                                                           partial, flags);
            KEVD_LAUNCH(ctx);
        }
    }
    gram_f64_reduce_kernel<<<n_tiles, 256, 0, st>>>(partial, n_tiles, n_split, k, e, colmax + k, G);
    KEVD_LAUNCH(ctx);
    gram_check_kernel<<<cx, 256, 0, st>>>(colmax, G, k, N, flags + 1);
    KEVD_LAUNCH(ctx);
    int h[2] = {0, 0};
    KEVD_CUDA(ctx, cudaMemcpyAsync(h, flags, sizeof(h), cudaMemcpyDeviceToHost, st));
    KEVD_CUDA(ctx, cudaStreamSynchronize(st));
    if (h[0] != 0) return set_error(ctx, KEVD_ERR_TIMEOUT, "gram_f64_tc: pipeline wait timed out (code %d)", h[0]);
    *done = h[1] == 0;
    return KEVD_OK;
}

}  // namespace kevd
