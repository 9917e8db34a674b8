// cycle_tail.h -- the smallest levels of the FP64 V-cycle in one block (cycle_tail.cu).
#pragma once
#include <cstdint>

#include "device.cuh"

namespace cfdxg {

constexpr int kTailMaxLevels = 16;

struct TailLevel {
    int n = 0;
    const int* ro = nullptr;
    const int* co = nullptr;         // absolute columns, or
    const int16_t* co16 = nullptr;   // offsets from the row
    const double* va = nullptr;
    const double* inv_diag = nullptr;
    // transfer to the next level (none on the coarsest): P by fine rows, P^T by coarse rows
    const int* p_off = nullptr;
    const int* p_col = nullptr;
    const double* p_val = nullptr;
    const int* r_off = nullptr;
    const int* r_row = nullptr;
    const double* r_val = nullptr;
    int at = 0;                       // of the level's r, x and second x in shared memory
    int tpr = 1, tpr_r = 1, tpr_p = 1;   // threads per row of A, P^T (rows of the next level) and P
    int parts = 0;                    // entries of the longest row of A per thread
    int pre = 0, post = 0;
};

struct TailPlan {
    int levels = 0;
    int coarse_lu = 0;       // 1: dense pivoted LU on the coarsest level, else Jacobi sweeps
    int coarse_sweeps = 0;
    double omega = 0.0;
    TailLevel L[kTailMaxLevels];
};

// Threads of the block, the entries of a row that one of them keeps, and the
// rows of all the tail's levels together (three FP64 vectors each in 42 KB of
// shared memory).
constexpr int kTailThreads = 512;
constexpr int kTailRowEntries = 28;
constexpr int64_t kTailRows = 1792;

// z = the cycle from the plan's first level applied to r (device vectors of that level).
void launch_tail(cfdxg_context* ctx, const TailPlan& plan, const double* r, double* z, int* status);
// Threads per row that spread `rows` rows of `entries` entries over the block.
int tail_threads_per_row(int64_t rows, int64_t entries);
// Whether a level's rows then fit the block's threads and their registers.
bool tail_fits(int64_t rows, int64_t longest_row, int tpr);

// Reference dense pivoted solve of the coarsest level (amg_preconditioner.h:2592-2663)
// by the first warp of a block, every value formed in the reference's order:
// the elimination's entries are independent of one another, the sums of the
// back substitution run on one lane.  Under the constant null space (ns = 1)
// the system is bordered by a row and a column of ones and the mean of the
// solution is removed, summed in order.  r and x may be shared or global
// memory; returns false on a pivot below the tolerance or a non-finite value.
constexpr int kDenseDirectLimit = 16;
constexpr int kLuMax = kDenseDirectLimit + 1;
struct LuScratch {
    double m[kLuMax][kLuMax + 1];   // the last column is the right-hand side
    double sol[kLuMax];
};

template <class T, class R, class X>
__device__ __forceinline__ bool dense_lu_warp(LuScratch& S, int n, const int* __restrict__ ro,
                                              const int* __restrict__ co, const T* __restrict__ va, const R* r, X* x,
                                              int ns, int lane) {
    const int sn = n + (ns ? 1 : 0);
    double scale = 0.0;
    if (lane < sn) {
        for (int j = 0; j < sn; ++j) S.m[lane][j] = 0.0;
        S.m[lane][kLuMax] = 0.0;
        if (lane < n) {
            S.m[lane][kLuMax] = static_cast<double>(r[lane]);
            for (int k = ro[lane]; k < ro[lane + 1]; ++k) S.m[lane][co[k]] += static_cast<double>(va[k]);
            if (ns) S.m[lane][n] = 1.0;
        } else {
            for (int j = 0; j < n; ++j) S.m[lane][j] = 1.0;
        }
        for (int j = 0; j < sn; ++j) {
            const double a = fabs(S.m[lane][j]);
            scale = (scale < a) ? a : scale;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const double a = __shfl_xor_sync(0xffffffffu, scale, o);
        scale = (scale < a) ? a : scale;
    }
    const double pivot_tol = 128.0 * 2.220446049250313080847e-16 * (1.0 < scale ? scale : 1.0);
    __syncwarp();
    bool ok = true;
    for (int k = 0; k < sn && ok; ++k) {
        // the largest magnitude of column k from row k on, the first row of equals
        int pivot = k;
        double pivot_abs = fabs(S.m[k][k]);
        for (int i = k + 1; i < sn; ++i) {
            const double c = fabs(S.m[i][k]);
            if (c > pivot_abs) { pivot_abs = c; pivot = i; }
        }
        if (!isfinite(pivot_abs) || pivot_abs <= pivot_tol) { ok = false; break; }
        __syncwarp();
        if (pivot != k && lane <= kLuMax && lane >= k && (lane < sn || lane == kLuMax)) {
            const double t = S.m[k][lane];
            S.m[k][lane] = S.m[pivot][lane];
            S.m[pivot][lane] = t;
        }
        __syncwarp();
        const double diagonal = S.m[k][k];
        bool bad = false;
        if (lane > k && lane < sn) {
            const double factor = S.m[lane][k] / diagonal;
            bad = !isfinite(factor);
            S.m[lane][k] = 0.0;
            for (int j = k + 1; j < sn; ++j) S.m[lane][j] -= factor * S.m[k][j];
            S.m[lane][kLuMax] -= factor * S.m[k][kLuMax];
        }
        if (__any_sync(0xffffffffu, bad)) ok = false;
        __syncwarp();
    }
    if (ok && lane == 0) {
        for (int ii = sn - 1; ii >= 0 && ok; --ii) {
            double sum = S.m[ii][kLuMax];
            for (int j = ii + 1; j < sn; ++j) sum -= S.m[ii][j] * S.sol[j];
            const double diagonal = S.m[ii][ii];
            if (!isfinite(diagonal) || fabs(diagonal) <= pivot_tol) { ok = false; break; }
            S.sol[ii] = sum / diagonal;
            if (!isfinite(S.sol[ii])) ok = false;
        }
        if (ok && ns) {
            double mean = 0.0;
            for (int i = 0; i < n; ++i) mean += S.sol[i];
            mean /= static_cast<double>(n);
            for (int i = 0; i < n; ++i) S.sol[i] -= mean;
        }
    }
    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    __syncwarp();
    if (ok && lane < n) x[lane] = static_cast<X>(S.sol[lane]);
    return ok;
}

}  // namespace cfdxg
