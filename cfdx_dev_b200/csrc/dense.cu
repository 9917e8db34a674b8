// dense.cu -- inverse of a symmetric positive definite matrix in FP64, by
// blocked symmetric sweeps (Gauss-Jordan elimination in place).
//
// Sweeping the block column k of a symmetric matrix with pivot block D^-1 =
// A_kk replaces A_kk by -D, A_ik by A_ik D and A_ij by A_ij - A_ik D A_kj; all
// blocks swept once leave -A^-1 (the sweep operator: J. H. Goodnight, "A
// tutorial on the SWEEP operator", The American Statistician 33, 1979).  The
// pivot blocks are the Schur complements, so no pivoting is needed exactly
// when the matrix is positive definite, and a pivot that is not positive says
// that it is not.  The matrix stays symmetric throughout: only the tiles on and
// below the diagonal are kept.
//
// (Pointers that the preceding kernel writes carry no __restrict__: these
// kernels start before it ends, and an invariant load could be moved above
// their wait.)
//
// Two launches per 64-wide block column: the panel (P = A_:k, W = P D, both
// left transposed for the next kernel) and the rank-64 update of the lower
// tiles, whose first block also inverts the next pivot block, so that the
// serial part hides behind the update: n^3 / 2 multiply-adds in the updates, 64
// n^2 in the panels.  An update takes 20 us at 500 rows, where the serial pivots
// (19 alone) are all of it, 27 at 2,000, 43 at 3,429 (FP64 tensor cores 52%
// busy) and 95 at 5,287, where the products bound it; a panel 11 to 17.  3,429
// rows: 3.2 ms, against 10.5 ms by cuSOLVER's potrf and potri, whose triangular
// inverse and product run in many small kernels.
#include "dense.h"

#include <cmath>

namespace cfdxg {
namespace {

constexpr int kB = kSpdBlock;      // 64
constexpr int kThreads = 256;      // 16 x 16, a 4 x 4 part of a tile each

// rows (or columns) of a thread's 4 x 4 part: 2 q, 2 q + 1, 32 + 2 q, 33 + 2 q,
// so that 16 threads' 16-byte shared loads are contiguous
__device__ __forceinline__ int part(int q, int u) { return (u & 2) * 16 + 2 * q + (u & 1); }

__device__ __forceinline__ void load4(const double* row, int q, double (&v)[4]) {
    const double2 a = *reinterpret_cast<const double2*>(row + 2 * q);
    const double2 b = *reinterpret_cast<const double2*>(row + 32 + 2 * q);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}

// acc += sum_k a[k][rows]^T b[k][cols] over 64 k (leading dimensions lda, ldb)
__device__ __forceinline__ void tile_product(const double* a, int lda, const double* b, int ldb, int ty, int tx,
                                             double (&acc)[4][4]) {
#pragma unroll 4
    for (int k = 0; k < kB; ++k) {
        double x[4], y[4];
        load4(a + k * lda, ty, x);
        load4(b + k * ldb, tx, y);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] += x[i] * y[j];
    }
}

// Inverts the 64 x 64 symmetric block held 4 x 4 per thread (rows part(ty, .),
// columns part(tx, .)) by 64 scalar sweeps; *info = 1 when a pivot is not
// positive and finite.  The pivots are taken by their place in the threads'
// parts (any order of a positive definite block will do), so that the pivot
// row and column sit in fixed registers of the threads that hold them: with
// the place known only at run time, selecting it cost more instructions than
// the sweep and the block took 47 us.  rowbuf, colbuf: 2 x 64 doubles of shared
// memory.
__device__ void invert_block(double (&v)[4][4], int ty, int tx, double* rowbuf, double* colbuf, int* info) {
#pragma unroll
    for (int pu = 0; pu < 4; ++pu) {
#pragma unroll 1
        for (int pq = 0; pq < 16; ++pq) {
            const int p = part(pq, pu);
            double* rb = rowbuf + (pq & 1) * kB;
            double* cb = colbuf + (pq & 1) * kB;
            if (ty == pq) {
                *reinterpret_cast<double2*>(rb + 2 * tx) = make_double2(v[pu][0], v[pu][1]);
                *reinterpret_cast<double2*>(rb + 32 + 2 * tx) = make_double2(v[pu][2], v[pu][3]);
            }
            if (tx == pq) {
                *reinterpret_cast<double2*>(cb + 2 * ty) = make_double2(v[0][pu], v[1][pu]);
                *reinterpret_cast<double2*>(cb + 32 + 2 * ty) = make_double2(v[2][pu], v[3][pu]);
            }
            __syncthreads();
            const double pivot = rb[p];
            if (!(pivot > 0.0) || !isfinite(pivot)) *info = 1;
            const double inv = 1.0 / pivot;
            double r[4], c[4];
            load4(rb, tx, r);
            load4(cb, ty, c);
#pragma unroll
            for (int j = 0; j < 4; ++j) r[j] *= inv;
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) v[i][j] -= c[i] * r[j];
            if (ty == pq) {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[pu][j] = r[j];
            }
            if (tx == pq) {
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i][pu] = -c[i] * inv;
                if (ty == pq) v[pu][pu] = inv;
            }
        }
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kThreads) k_spd_first_pivot(const double* __restrict__ a, int ld,
                                                              double* __restrict__ d, int* info) {
    __shared__ __align__(16) double rowbuf[2 * kB], colbuf[2 * kB];
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    double v[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = a[static_cast<size_t>(part(ty, i)) * ld + part(tx, j)];
    invert_block(v, ty, tx, rowbuf, colbuf, info);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) d[part(ty, i) * kB + part(tx, j)] = v[i][j];
}

constexpr int kPanelLd = kB + 2;   // keeps 16-byte rows, spreads the transposing stores over the banks

// Block I of the panel: P_I = A_Ik (A_kI^T above the diagonal) and W_I = P_I D,
// transposed into pt and wt ([column][row], leading dimension ld); A_Ik is
// replaced by W_I, the pivot tile by -D.
__global__ void __launch_bounds__(kThreads) k_spd_panel(double* a, int ld, int k, const double* d, double* pt,
                                                        double* wt) {
    pdl_entry();
    extern __shared__ __align__(16) double smem[];
    double* sp = smem;                    // [k][row]
    double* sd = smem + kB * kPanelLd;    // [k][column]
    const int I = blockIdx.x;
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    if (I == k) {
        for (int q = threadIdx.x; q < kB * kB; q += kThreads)
            a[static_cast<size_t>(k * kB + q / kB) * ld + k * kB + q % kB] = -d[q];
        return;
    }
    for (int q = threadIdx.x; q < kB * kB; q += kThreads) {
        const int r = q / kB, c = q % kB;
        sd[r * kB + c] = d[q];
        if (I > k) sp[c * kPanelLd + r] = a[static_cast<size_t>(I * kB + r) * ld + k * kB + c];
        else sp[r * kPanelLd + c] = a[static_cast<size_t>(k * kB + r) * ld + I * kB + c];
    }
    __syncthreads();
    for (int q = threadIdx.x; q < kB * kB; q += kThreads)
        pt[static_cast<size_t>(q / kB) * ld + I * kB + q % kB] = sp[(q / kB) * kPanelLd + q % kB];
    double acc[4][4] = {};
    tile_product(sp, kPanelLd, sd, kB, ty, tx, acc);
    __syncthreads();
    // W into shared memory as [column][row], then out in whole rows either way
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) sp[part(tx, j) * kPanelLd + part(ty, i)] = acc[i][j];
    __syncthreads();
    for (int q = threadIdx.x; q < kB * kB; q += kThreads) {
        const int r = q / kB, c = q % kB;
        wt[static_cast<size_t>(r) * ld + I * kB + c] = sp[r * kPanelLd + c];
        if (I > k) a[static_cast<size_t>(I * kB + r) * ld + k * kB + c] = sp[c * kPanelLd + r];
        else a[static_cast<size_t>(k * kB + r) * ld + I * kB + c] = sp[r * kPanelLd + c];
    }
}

// d += a b on the FP64 tensor cores: a 8 x 4 (lane: row lane / 4, column lane
// % 4), b 4 x 8 (row lane % 4, column lane / 4), d 8 x 8 (row lane / 4, columns
// 2 (lane % 4) and the next).  FP64 multiply-adds throughout.
__device__ __forceinline__ void mma_f64(double (&d)[2], double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d[0]), "+d"(d[1])
        : "d"(a), "d"(b));
}

// A_IJ -= W_I P_J^T for the lower tiles outside row and column k.  Block 0 takes
// the next pivot tile and inverts it into d.
//
// A warp takes 32 x 16 of the tile as 4 x 2 tensor products over 16 steps of
// four k: six shared reads (two wavefronts each, kUpdateLd spreading the four k
// over the banks) for 2,048 multiply-adds.  With 4 x 4 register tiles a thread's
// shared reads took as long as its multiply-adds: 63 us a launch at 3,429 rows
// against 43.
constexpr int kUpdateLd = kB + 4;
__global__ void __launch_bounds__(kThreads, 3) k_spd_update(double* a, int ld, int tiles, int k,
                                                            const double* pt, const double* wt, double* d, int* info) {
    pdl_entry();
    extern __shared__ __align__(16) double smem[];
    double* sw = smem;                     // [k][row]
    double* sp = smem + kB * kUpdateLd;    // [k][column]
    const int count = (tiles - 1) * tiles / 2;   // lower tiles of the other tiles - 1 block rows
    // the next pivot tile (k + 1, k + 1) is lower tile (k, k) once row k is left out
    const int next = k + 1 < tiles ? k * (k + 1) / 2 + k : -1;
    const int t = next < 0 ? blockIdx.x : (blockIdx.x == 0 ? next : (static_cast<int>(blockIdx.x) <= next ? blockIdx.x - 1 : blockIdx.x));
    if (t >= count) return;
    int I = static_cast<int>((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
    while ((I + 1) * (I + 2) / 2 <= t) ++I;
    while (I * (I + 1) / 2 > t) --I;
    int J = t - I * (I + 1) / 2;
    if (I >= k) ++I;
    if (J >= k) ++J;
    for (int q = threadIdx.x; q < kB * kB / 2; q += kThreads) {
        const int r = q / (kB / 2), c = 2 * (q % (kB / 2));
        *reinterpret_cast<double2*>(sw + r * kUpdateLd + c) =
            *reinterpret_cast<const double2*>(wt + static_cast<size_t>(r) * ld + I * kB + c);
        *reinterpret_cast<double2*>(sp + r * kUpdateLd + c) =
            *reinterpret_cast<const double2*>(pt + static_cast<size_t>(r) * ld + J * kB + c);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, m = lane & 3;
    const int row0 = (warp & 1) * 32, col0 = (warp >> 1) * 16;
    double* tile = a + static_cast<size_t>(I * kB + row0 + g) * ld + J * kB + col0 + 2 * m;
    double2 v[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
            v[i][j] = *reinterpret_cast<const double2*>(tile + static_cast<size_t>(8 * i) * ld + 8 * j);
    __syncthreads();
    double acc[4][2][2] = {};
#pragma unroll 4
    for (int q = 0; q < kB; q += 4) {
        const double* wr = sw + (q + m) * kUpdateLd + row0 + g;
        const double* pr = sp + (q + m) * kUpdateLd + col0 + g;
        double x[4], y[2];
#pragma unroll
        for (int i = 0; i < 4; ++i) x[i] = wr[8 * i];
#pragma unroll
        for (int j = 0; j < 2; ++j) y[j] = pr[8 * j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) mma_f64(acc[i][j], x[i], y[j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
            *reinterpret_cast<double2*>(tile + static_cast<size_t>(8 * i) * ld + 8 * j) =
                make_double2(v[i][j].x - acc[i][j][0], v[i][j].y - acc[i][j][1]);
    if (I == J && I == k + 1) {
        __syncthreads();   // the tile is written; smem becomes the pivot buffers
        const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
        double p[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) load4(a + static_cast<size_t>(I * kB + part(ty, i)) * ld + J * kB, tx, p[i]);
        invert_block(p, ty, tx, smem, smem + 2 * kB, info);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) d[part(ty, i) * kB + part(tx, j)] = p[i][j];
    }
}

// A row per warp: the CSR rows of a (n x n) into the zeroed dense array, ones on the padding's diagonal.
__global__ void k_dense_rows(int n, int np, const int* __restrict__ ro, const int* __restrict__ co,
                             const double* __restrict__ va, double* __restrict__ a) {
    const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (i >= np) return;
    double* row = a + static_cast<size_t>(i) * np;
    if (i >= n) {
        if (lane == 0) row[i] = 1.0;
        return;
    }
    for (int k = ro[i] + lane; k < ro[i + 1]; k += 32) row[co[k]] = va[k];
}

// flag = 1 when the n x n matrix a is not symmetric: |a_ij - a_ji| above
// 1e-12 of the pair's magnitude plus 1e-14 of sqrt(|a_ii a_jj|) (the coarse
// Galerkin operators of a symmetric system differ from symmetry only by the
// rounding of their sums, which leaves entries cancelled to near zero with
// differences far above their own size but far below the diagonal's).  One
// 32 x 32 tile and its mirror per block.
__global__ void k_symmetry_check(int n, int ld, const double* __restrict__ a, int* flag) {
    __shared__ double mirror[32][33];
    const int I = blockIdx.y, J = blockIdx.x;
    if (J > I) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < 32; r += 8) {
        const int i = J * 32 + r, j = I * 32 + tx;
        mirror[r][tx] = i < n && j < n ? a[static_cast<size_t>(i) * ld + j] : 0.0;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int i = I * 32 + r, j = J * 32 + tx;
        if (i >= n || j >= i) continue;
        const double x = a[static_cast<size_t>(i) * ld + j], y = mirror[tx][r];
        const double scale = sqrt(fabs(a[static_cast<size_t>(i) * ld + i]) * fabs(a[static_cast<size_t>(j) * ld + j]));
        if (!(fabs(x - y) <= 1e-12 * (fabs(x) + fabs(y)) + 1e-14 * scale)) atomicOr(flag, 1);
    }
}

// b (n x n, row-major with leading dimension ldb, both triangles) = the negated lower triangle of a
template <class S>
__global__ void k_negated_symmetric(int n, int ld, int ldb, const double* __restrict__ a, S* __restrict__ b) {
    __shared__ double tile[32][33];
    const int I = blockIdx.y, J = blockIdx.x;
    if (J > I) return;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    for (int r = ty; r < 32; r += 8) {
        const int i = I * 32 + r, j = J * 32 + tx;
        tile[r][tx] = i < n && j < n ? -a[static_cast<size_t>(i) * ld + j] : 0.0;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int i = I * 32 + r, j = J * 32 + tx;
        if (i < n && j <= i) b[static_cast<size_t>(i) * ldb + j] = static_cast<S>(tile[r][tx]);
        const int mi = J * 32 + r, mj = I * 32 + tx;   // the mirrored entry (mi, mj), mj > mi
        if (mi < n && mj < n && mj > mi) b[static_cast<size_t>(mi) * ldb + mj] = static_cast<S>(tile[tx][r]);
    }
}

void launch_shared(cfdxg_context* ctx, void (*kern)(double*, int, int, const double*, double*, double*), int grid,
                   std::size_t smem, double* a, int ld, int k, const double* d, double* pt, double* wt) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    CFDXG_CUDA(cudaLaunchKernelEx(&cfg, kern, a, ld, k, d, pt, wt));
    check_launch(ctx);
}

}  // namespace

SpdStatus spd_inverse(cfdxg_context* ctx, int n, const int* ro, const int* co, const double* va, SpdWorkspace& w,
                      int ld_out, float* out32, double* out64) {
    cudaStream_t s = ctx->stream;
    const int tiles = (n + kB - 1) / kB, np = tiles * kB;
    const std::size_t nn = static_cast<std::size_t>(np) * np;
    if (w.a.size() < nn) w.a.resize(nn);
    const std::size_t panel = static_cast<std::size_t>(kB) * np;
    if (w.panels.size() < 2 * panel + 2 * kB * kB) w.panels.resize(2 * panel + 2 * kB * kB);
    if (w.info.size() < 2) w.info.resize(2);
    double* a = w.a.get();
    double* pt = w.panels.get();
    double* wt = pt + panel;
    double* d[2] = {wt + panel, wt + panel + kB * kB};
    CFDXG_CUDA(cudaMemsetAsync(a, 0, sizeof(double) * nn, s));
    CFDXG_CUDA(cudaMemsetAsync(w.info.get(), 0, 2 * sizeof(int), s));
    k_dense_rows<<<blocks_for(static_cast<int64_t>(np) * 32, kThreads), kThreads, 0, s>>>(n, np, ro, co, va, a);
    check_launch(ctx);
    const int t32 = (n + 31) / 32;
    k_symmetry_check<<<dim3(t32, t32), 256, 0, s>>>(n, np, a, w.info.get());
    check_launch(ctx);
    // one wait here, for the caller's other route not to pay the sweeps as well
    int info[2] = {0, 0};
    CFDXG_CUDA(cudaMemcpyAsync(info, w.info.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
    CFDXG_CUDA(cudaStreamSynchronize(s));
    if (info[0]) return SpdStatus::kNotSymmetric;
    k_spd_first_pivot<<<1, kThreads, 0, s>>>(a, np, d[0], w.info.get() + 1);
    check_launch(ctx);
    constexpr std::size_t kPanelSmem = sizeof(double) * (kB * kPanelLd + kB * kB);
    constexpr std::size_t kUpdateSmem = sizeof(double) * 2 * kB * kUpdateLd;
    CFDXG_CUDA(cudaFuncSetAttribute(k_spd_panel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(kPanelSmem)));
    CFDXG_CUDA(cudaFuncSetAttribute(k_spd_update, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(kUpdateSmem)));
    const int lower = (tiles - 1) * tiles / 2;
    for (int k = 0; k < tiles; ++k) {
        launch_shared(ctx, k_spd_panel, tiles, kPanelSmem, a, np, k, d[k & 1], pt, wt);
        if (lower > 0) {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(lower);
            cfg.blockDim = dim3(kThreads);
            cfg.dynamicSmemBytes = kUpdateSmem;
            cfg.stream = s;
            cudaLaunchAttribute attr{};
            attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr.val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            CFDXG_CUDA(cudaLaunchKernelEx(&cfg, k_spd_update, a, np, tiles, k, static_cast<const double*>(pt),
                                          static_cast<const double*>(wt), d[(k + 1) & 1], w.info.get() + 1));
            check_launch(ctx);
        }
    }
    if (out64) k_negated_symmetric<double><<<dim3(t32, t32), 256, 0, s>>>(n, np, ld_out, a, out64);
    else k_negated_symmetric<float><<<dim3(t32, t32), 256, 0, s>>>(n, np, ld_out, a, out32);
    check_launch(ctx);
    CFDXG_CUDA(cudaMemcpyAsync(info, w.info.get(), 2 * sizeof(int), cudaMemcpyDeviceToHost, s));
    CFDXG_CUDA(cudaStreamSynchronize(s));
    return info[1] ? SpdStatus::kNotPositive : SpdStatus::kInverted;
}

}  // namespace cfdxg
