// dense.h -- inverse of a symmetric positive definite matrix (dense.cu).
#pragma once
#include "device.cuh"

namespace cfdxg {

constexpr int kSpdBlock = 64;

// Work arrays, kept with the hierarchy for its refreshes: the matrix padded to
// whole blocks (the LU route's too), two panels and two pivot blocks, and the
// status words.
struct SpdWorkspace {
    DevBuf<double> a, panels;
    DevBuf<int> info;
};

enum class SpdStatus { kInverted, kNotSymmetric, kNotPositive };

// The inverse of the n x n matrix given by its device CSR (unique columns),
// row-major (leading dimension ld_out) into out64, or rounded into out32 when
// out64 is null.  A matrix that is not symmetric to rounding is reported before
// any sweep, one that is not positive definite after them; either leaves the
// output undefined.  Synchronises the stream.
SpdStatus spd_inverse(cfdxg_context* ctx, int n, const int* ro, const int* co, const double* va, SpdWorkspace& w,
                      int ld_out, float* out32, double* out64);

}  // namespace cfdxg
