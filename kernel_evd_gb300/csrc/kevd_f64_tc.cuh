// FP64 products on the tensor cores in exact slices (kevd_f64_tc.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

struct kevd_ctx;

namespace kevd {

// G (k x k, column-major, full) = F^T diag(s)^2 F of a row-major FP64 factor, an entry
// to a few 2^-53 of sqrt(G_aa G_bb).  *done = false, and G undefined, when the call does
// not suit the slices: the workspace does not fit, or a column's largest entry is so far
// above its root mean square that fixed point would lose digits (the caller then takes
// the FP64 SIMT Gram).  s: device, N doubles.  Synchronises the stream.
int run_gram_f64_tc(kevd_ctx* ctx, const double* F, int64_t N, int64_t k, int64_t ldF, const double* s, double* G,
                    bool* done, cudaStream_t st);

// Digits of the rows of a row-major FP64 matrix A (rows x K, lda): out[i * K4 + c]
// (K4 = K rounded up to 4, words past K are zero digits), ea[i] the exponent.
// lower: entries with column > row count as zero.  col_major: A(i, c) is at
// A[c * lda + i].  prefix (or nullptr): the exponent of row i's columns
// < 64 (b + 1) at prefix[i * ceil(K / 64) + b].
int launch_digits_rows(kevd_ctx* ctx, const double* A, int64_t rows, int64_t K, int64_t lda, bool lower,
                       bool col_major, uint64_t* out, int* ea, int* prefix, cudaStream_t st);

// C(i, n) = scale[i] sum_k A(i, k) B(n, k) from row digits (word stride K4 for both,
// see launch_digits_rows), i < M, n < n_cols, as float (row stride ldc).  err:
// device int, set on a device-side timeout.
int launch_rows_f64_tc(kevd_ctx* ctx, const uint64_t* A, const int* ea, int64_t M, const uint64_t* B, const int* eb,
                       int64_t n_cols, int64_t K, const double* scale, float* C, int64_t ldc, int* err,
                       cudaStream_t st);

// F(i, n) = sum_{k <= n} K(i, k) Linv(n, k), i < M, n < r: K row-major M x r, Linv
// column-major r x r, with the digits and exponents of both.  Outputs whose K(i,
// k <= n) lie far below their row's largest entry, which sets the row's fixed
// point, are formed in FP64.  Written as double to Fd (row stride ldF) or, if Fd ==
// nullptr, as float to Ff.
struct TriOperands {
    const double *K, *Linv;
    const uint64_t *Kq, *Lq;
    const int *ek, *el, *prefix;
};
// *skip != 0: nothing is done.
int launch_tri_f64_tc(kevd_ctx* ctx, const TriOperands& o, int64_t M, int64_t r, double* Fd, float* Ff, int64_t ldF,
                      const int* skip, int* err, cudaStream_t st);

// Whether launch_tri_f64_tc keeps the outputs of this panel to FP64 accuracy, by a sample
// of its rows: *skip = 0 where the root mean square over their outputs of
// sqrt(n + 1) 2^(ek + el) / sum |K| |Linv| is at most limit, else 1; the product's error
// is 2^-67.2 of the sum a unit.  part: device, tri_range_size(r) doubles.
constexpr int kRangeRows = 32;
inline size_t tri_range_size(int64_t r) { return (size_t)(2 * (kRangeRows / 4) * ((r + 31) / 32)); }
int launch_tri_range(kevd_ctx* ctx, const TriOperands& o, int64_t M, int64_t r, double limit, double* part, int* skip,
                     cudaStream_t st);

// Kernel blocks K(i, c) = exp(-scale ||x_i - s_c||^2) in FP64 from exact squared
// distances (integer digits of the FP32 states at one common exponent).
//   states_exp     e with |X| <= 2^e over N x d states; *suited = false when the
//                  states are not finite or 4^e scale is too large for the digits
//                  to stand in for FP64 differences.  Synchronises the stream.
//   launch_digits_states  digits and squared norms of n states, rows row0 + i or
//                  idx[i] of X
//   launch_kernel_f64_tc  the n x r block, row stride ld
struct StateDigits {
    uint64_t* q;      // n x digits_ld(d)
    int64_t* norm;    // 2 n: squared norm of state i as the integer pair (hi, lo) at 2 i
};
int states_exp(kevd_ctx* ctx, const float* X, int64_t N, int d, double scale, int* e, bool* suited, cudaStream_t st);
int launch_digits_states(kevd_ctx* ctx, const float* X, int64_t row0, const int64_t* idx, int64_t n, int d, int e,
                         StateDigits out, cudaStream_t st);
int launch_kernel_f64_tc(kevd_ctx* ctx, StateDigits x, int64_t n, StateDigits s, int64_t r, int d, int e, double scale,
                         double* K, int64_t ld, int* err, cudaStream_t st);

// ea of a row with an infinity or a NaN (products with it are NaN).
constexpr int kDigitsNotFinite = 1 << 20;

inline int64_t digits_ld(int64_t K) { return (K + 3) / 4 * 4; }

}  // namespace kevd
