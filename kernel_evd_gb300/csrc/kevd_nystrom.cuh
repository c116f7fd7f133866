// Out-of-sample model (shared by the C boundary and the query kernel).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

struct kevd_ctx;

namespace kevd {

// Landmark rows, and W = [Z' | p1'] = L^{-T} [Z | c1] (r x (k_out + 1)) as the
// query kernel reads it: row-major, each entry an FP32 pair hi + lo (48 bits)
// of W 2^-ex[c], with 2^(ex[c] + 100) the binade of the column's largest entry.
struct Model {
    int64_t r = 0;
    int d = 0;
    int k_out = 0;
    double scale = 0.0;
    float* xs = nullptr;   // r x d
    float2* w = nullptr;   // r x (k_out + 1)
    int* ex = nullptr;     // k_out + 1
};

// zp: r x (k_out + 1) column-major FP64 -> m.w, m.ex.
int launch_nystrom_pack(kevd_ctx* ctx, const double* zp, const Model& m, cudaStream_t s);
int launch_nystrom_eval(kevd_ctx* ctx, const Model& m, const float* Y, int64_t n, float* Uy, cudaStream_t s);

}  // namespace kevd
