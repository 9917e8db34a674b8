// cycle_tail.cu -- the FP64 V-cycle's smallest levels in one block.
//
// A sweep of a level of a few thousand nonzeros is a fraction of a
// microsecond of work, and as a kernel of its own it costs 1.5-2.5 us
// (launch, row offsets, entries and vectors each waiting for L2): the last
// four levels of a 2,058-cell system (92 rows and fewer) were 90 of its
// cycle's 230 kernels.  Here one block runs them all in one launch, 0.5 us a
// step (a 2,058-cell system's cycle 347 -> 270 us and FP64 solve 2.81 -> 2.26
// ms; a 384-cell one's whole cycle 247 -> 97 us):
//
//  * the vectors of these levels stay in shared memory;
//  * a thread keeps its part of its row -- up to kTailRowEntries entries, with
//    the inverse diagonal and the right-hand side -- in registers over a
//    level's sweeps: a sweep is shared-memory reads, the sum, a store and a
//    barrier.  The next level's entries are requested before the transfer to
//    it.
//
// Bound by the barriers and the serial sum of a thread's entries.  512 threads
// of 28 entries: 1,024 of 14 spilled.
//
// One block, not a cluster: with the rows spread over 16 CTAs (every CTA a
// copy of the vectors, new entries stored into all of them) a step took
// 1.25 us, and larger levels were slower than their kernels.
//
// Row sums are formed by a power of two of threads per row with a fixed
// butterfly (deterministic); the operations per entry are the sweep,
// residual and transfer kernels'.
#include "cycle_tail.h"

#include <cmath>

#include "objects.h"

namespace cfdxg {
namespace {

// one row's product with x over the row's threads; every one of them gets it
__device__ __forceinline__ double row_product(int b, int e, int lane, int tpr, const int* __restrict__ col,
                                              const double* __restrict__ val, const double* x) {
    double s = 0.0;
#pragma unroll 4
    for (int k = b + lane; k < e; k += tpr) s += __ldg(val + k) * x[__ldg(col + k)];
    for (int o = tpr >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// This thread's entries of its row of a level's operator, in registers (at
// most one row per thread: the plan sees to it).
struct RowPart {
    double v[kTailRowEntries];
    uint16_t c[kTailRowEntries];   // columns: a tail level has at most kTailRows rows
    double di, ri;                 // inverse diagonal, right-hand side
    int i, lane;
    bool valid;
};

struct Tail {
    double* vec;       // the vectors, in shared memory
    int* status;

    // calls f(row, valid, lane of the row) for this thread's rows, the whole warp together
    template <class F>
    __device__ __forceinline__ void rows(int n, int tpr, F&& f) const {
        const int t = static_cast<int>(threadIdx.x);
        const int lane = t & (tpr - 1), per_warp = 32 / tpr, step = kTailThreads / tpr;
        for (int base = (t >> 5) * per_warp; base < n; base += step) {
            const int i = base + (t & 31) / tpr;
            f(i, i < n, lane);
        }
    }

    // the row's fixed part (not the right-hand side)
    __device__ __forceinline__ void load_row(RowPart& R, const TailLevel& L) const {
        const int t = static_cast<int>(threadIdx.x);
        R.lane = t & (L.tpr - 1);
        R.i = t / L.tpr;
        R.valid = R.i < L.n;
        const int b = R.valid ? __ldg(L.ro + R.i) : 0, e = R.valid ? __ldg(L.ro + R.i + 1) : 0;
        R.di = R.valid ? __ldg(L.inv_diag + R.i) : 0.0;
#pragma unroll
        for (int q = 0; q < kTailRowEntries; ++q) {
            R.v[q] = 0.0;
            R.c[q] = static_cast<uint16_t>(R.valid ? R.i : 0);   // padding: the row's own x, weight 0
            if (q < L.parts) {
                const int k = b + R.lane + q * L.tpr;
                if (k < e) {
                    R.v[q] = __ldg(L.va + k);
                    R.c[q] = static_cast<uint16_t>(L.co16 ? R.i + __ldg(L.co16 + k) : __ldg(L.co + k));
                }
            }
        }
    }

    // the row's product with x; every thread of the row gets it.  Four entries
    // at a time (the last ones padding), so that their reads overlap: one at a
    // time, each behind its own test, a step took 0.9 us.
    __device__ __forceinline__ double product(const RowPart& R, const TailLevel& L, const double* x) const {
        double s = 0.0, u = 0.0;
#pragma unroll
        for (int q = 0; q < kTailRowEntries; q += 4) {
            if (q >= L.parts) break;
            const double x0 = x[R.c[q]], x1 = x[R.c[q + 1]], x2 = x[R.c[q + 2]], x3 = x[R.c[q + 3]];
            s += R.v[q] * x0;
            u += R.v[q + 1] * x1;
            s += R.v[q + 2] * x2;
            u += R.v[q + 3] * x3;
        }
        s += u;
        for (int o = L.tpr >> 1; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    }

    // x_out = x + omega (inv_diag (r - A x))
    __device__ __forceinline__ void sweep(const RowPart& R, const TailLevel& L, double omega, int x, int out) const {
        const double s = product(R, L, vec + x);
        if (R.valid && R.lane == 0) {
            const double xn = vec[x + R.i] + omega * (R.di * (R.ri - s));
            vec[out + R.i] = xn;
            if (!isfinite(xn)) atomicOr(status, kStatusNonFinite);
        }
        __syncthreads();
    }

    // `sweeps` sweeps from x = 0 with the row in R; returns where x ends up (x, or the other buffer)
    __device__ __forceinline__ int sweeps_from_zero(const RowPart& R, const TailLevel& L, double omega, int sweeps,
                                                    int r, int x, int x2) const {
        for (int i = threadIdx.x; i < L.n; i += kTailThreads) {
            double xi = 0.0;
            if (sweeps > 0) {
                xi = 0.0 + omega * (__ldg(L.inv_diag + i) * (vec[r + i] - 0.0));
                if (!isfinite(xi)) atomicOr(status, kStatusNonFinite);
            }
            vec[x + i] = xi;
        }
        __syncthreads();
        for (int k = 1; k < sweeps; ++k) {
            sweep(R, L, omega, x, x2);
            const int t = x;
            x = x2;
            x2 = t;
        }
        return x;
    }
};

__global__ void __launch_bounds__(kTailThreads, 1) k_cycle_tail(const __grid_constant__ TailPlan plan,
                                                                const double* r_in, double* z_out, int* status) {
    extern __shared__ __align__(16) double vec[];
    __shared__ LuScratch lu;
    __shared__ int where[kTailMaxLevels];   // of each level's x on the way down
    const Tail T{vec, status};
    const int last = plan.levels - 1;
    RowPart R;
    T.load_row(R, plan.L[0]);
    pdl_entry();
    for (int i = threadIdx.x; i < plan.L[0].n; i += kTailThreads) vec[plan.L[0].at + i] = r_in[i];
    __syncthreads();
    for (int l = 0; l < last; ++l) {
        const TailLevel& L = plan.L[l];
        const TailLevel& C = plan.L[l + 1];
        const int r = L.at, x0 = L.at + L.n, x1 = L.at + 2 * L.n;
        int x = x0, res = r;
        if (L.pre > 0) {
            R.ri = R.valid ? vec[r + R.i] : 0.0;
            x = T.sweeps_from_zero(R, L, plan.omega, L.pre, r, x0, x1);
            res = x == x0 ? x1 : x0;
            const double s = T.product(R, L, vec + x);
            if (R.valid && R.lane == 0) vec[res + R.i] = R.ri - s;
            __syncthreads();
        }
        if (threadIdx.x == 0) where[l] = x;
        T.load_row(R, C);
        T.rows(C.n, L.tpr_r, [&](int c, bool valid, int lane) {
            const int b = valid ? __ldg(L.r_off + c) : 0, e = valid ? __ldg(L.r_off + c + 1) : 0;
            const double s = row_product(b, e, lane, L.tpr_r, L.r_row, L.r_val, vec + res);
            if (valid && lane == 0) vec[C.at + c] = s;
        });
        __syncthreads();
    }
    int x;
    {
        const TailLevel& L = plan.L[last];
        const int r = L.at, x0 = L.at + L.n, x1 = L.at + 2 * L.n;
        if (plan.coarse_lu) {
            if (threadIdx.x < 32 &&
                !dense_lu_warp(lu, L.n, L.ro, L.co, L.va, vec + r, vec + x0, 0, static_cast<int>(threadIdx.x)) &&
                threadIdx.x == 0)
                atomicOr(status, kStatusNonFinite);
            __syncthreads();
            x = x0;
        } else {
            R.ri = R.valid ? vec[r + R.i] : 0.0;
            x = T.sweeps_from_zero(R, L, plan.omega, plan.coarse_sweeps, r, x0, x1);
        }
    }
    for (int l = last - 1; l >= 0; --l) {
        const TailLevel& L = plan.L[l];
        const int xc = x, r = L.at, x0 = L.at + L.n, x1 = L.at + 2 * L.n;
        x = where[l];
        const bool assign = L.pre == 0;   // x = 0 before the correction
        if (L.post > 0) {
            T.load_row(R, L);
            R.ri = R.valid ? vec[r + R.i] : 0.0;
        }
        T.rows(L.n, L.tpr_p, [&](int i, bool valid, int lane) {
            const int b = valid ? __ldg(L.p_off + i) : 0, e = valid ? __ldg(L.p_off + i + 1) : 0;
            const double s = row_product(b, e, lane, L.tpr_p, L.p_col, L.p_val, vec + xc);
            if (!valid || lane != 0) return;
            const double v = (assign ? 0.0 : vec[x + i]) + s;
            vec[x + i] = v;
            if (!isfinite(v)) atomicOr(status, kStatusNonFinite);
        });
        __syncthreads();
        int other = x == x0 ? x1 : x0;
        for (int k = 0; k < L.post; ++k) {
            T.sweep(R, L, plan.omega, x, other);
            const int t = x;
            x = other;
            other = t;
        }
    }
    for (int i = threadIdx.x; i < plan.L[0].n; i += kTailThreads) z_out[i] = vec[x + i];
}

}  // namespace

int tail_threads_per_row(int64_t rows, int64_t entries) {
    int tpr = 1;
    while (tpr < 32 && rows * tpr * 2 <= kTailThreads && entries >= rows * tpr * 2) tpr *= 2;
    return tpr;
}

bool tail_fits(int64_t rows, int64_t longest_row, int tpr) {
    return rows * tpr <= kTailThreads && longest_row <= static_cast<int64_t>(kTailRowEntries) * tpr;
}

void launch_tail(cfdxg_context* ctx, const TailPlan& plan, const double* r, double* z, int* status) {
    std::size_t rows = 0;
    for (int l = 0; l < plan.levels; ++l) rows += static_cast<std::size_t>(plan.L[l].n);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(1);
    cfg.blockDim = dim3(kTailThreads);
    cfg.dynamicSmemBytes = 3 * sizeof(double) * rows;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    CFDXG_CUDA(cudaLaunchKernelEx(&cfg, k_cycle_tail, plan, r, z, status));
    check_launch(ctx);
}

}  // namespace cfdxg
