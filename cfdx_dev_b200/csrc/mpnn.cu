// mpnn.cu -- learned message-passing preconditioner on the matrix graph.
//
// Network (no counterpart in the reference; the FP64 oracle is
// oracle/mpnn_oracle.py, whose parameter layout this file shares):
//   s = rms(r);  x_i = [r_i/s, f_V, f_P, f_D]   (standardised log volume, log a_P, log a_ii)
//   h = relu(W_in x + b_in)
//   4 rounds:  a_i = sum_j w_ij h_j  (w_ij = -a_ij / sqrt(a_ii a_jj));
//              h_i += W2 relu(W1 [h_i, a_i] + b1) + b2
//   N(r)_i = s (w_out . h_i + b_out) / a_ii
//
// Training kernels run in FP32 (forward, backward, Adam), several pairs of a
// batch at a time, as register-tiled products over 64-cell tiles in shared
// memory, with deterministic weight-gradient reductions: each thread of a
// block owns its gradient entries over a fixed set of tiles, and the blocks
// are combined in a fixed order at the end.
// Inference runs each round as one fused kernel: the neighbour gather leaves
// [h, a] in the MMA's operand registers and both MLP layers run on the tensor cores
// (mma.sync m16n8k16, BF16 operands, FP32 accumulation); the state h is
// stored as BF16 between rounds and carried in FP32 within one.
// The encoder is folded into the first round (h0 formed from r where it is
// read) and the readout into the last, so inference is four kernels.
#include <cuda_bf16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <thread>

#include "io.h"
#include "krylov.h"
#include "mpnn.h"

namespace cfdxg {
namespace mp {

constexpr int F = 32;
constexpr int R = 4;
constexpr int OFF_WIN = 0, OFF_BIN = 128;
constexpr int ROUND0 = 160, ROUND_SIZE = 3136;   // W1 2048, b1 32, W2 1024, b2 32
constexpr int OFF_W1 = 0, OFF_B1 = 2048, OFF_W2 = 2080, OFF_B2 = 3104;
constexpr int OFF_WOUT = ROUND0 + R * ROUND_SIZE;   // 12704
constexpr int OFF_BOUT = OFF_WOUT + F;              // 12736
constexpr int NP = OFF_BOUT + 1;                    // 12737
constexpr int kGridBlocks = 592;                    // fixed partition of cells for reductions (4 blocks per SM)
constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kTrainTile = 64;                      // cells per tile of the training kernels
// Pairs of a batch that go through the kernels together: as many as keep the
// cells in flight at or below this (at least one pair) -- enough to fill the
// GPU several times over, and a bounded workspace (2.1 KB per cell, 540 MB).
constexpr int64_t kTrainCells = 262144;

}  // namespace mp
}  // namespace cfdxg

struct cfdxg_mpnn {
    std::vector<float> host;   // FP32 master parameters (host mirror)
    cfdxg::DevBuf<float> params, grad, adam_m, adam_v, partial;
    cfdxg::DevBuf<__nv_bfloat16> wbf;   // per round: W1 (32x64) then W2 (32x32), BF16
    int64_t steps = 0;
    // binding
    const cfdxg_matrix* A = nullptr;
    int n = 0;
    cfdxg::DevBuf<float> feats;
    cfdxg::DevBuf<int> gro, gco;   // off-diagonal couplings only (inference gather)
    cfdxg::DevBuf<float> gew;
    cfdxg::DevBuf<double> diag;
    // work
    cfdxg::DevBuf<float> hA, hB;
    cfdxg::DevBuf<double> y, t;
    // training workspace, grown by the training calls: states and gradients
    // of the pairs in flight, per-pair sums and their partials
    cfdxg::DevBuf<float> H, AG, Z, dh, da, da2, dyf;
    cfdxg::DevBuf<double> Ad, Ae, outb, w1, w2, q, terms, sums;
    cfdxg::DevBuf<unsigned> tickets;
    cfdxg_amg* vcycle = nullptr;   // V-cycle the network is trained in front of
};

namespace cfdxg {
namespace {

using namespace mp;

// x = [r/s, feats]; h0 = relu(W_in x + b_in) of the pairs' cells (pair s holds
// cells [s n, (s+1) n)).  Eight lanes per cell, each lane four features (one
// 16-byte store); the group's first lane forms r/s.
__global__ void k_encode(int n, int cells, const double* __restrict__ r, const double* __restrict__ rr,
                         const float* __restrict__ feats, const float* __restrict__ P, float* __restrict__ h) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = t >> 3;
    const int quarter = static_cast<int>(t & 7);
    const unsigned grp_mask = 0xffu << (threadIdx.x & 24);
    const int pair = c < cells ? c / n : 0;
    const int i = c < cells ? c - pair * n : 0;
    float x0 = 0.0f;
    if (c < cells && quarter == 0) {
        const double s = sqrt(rr[pair] / n);
        x0 = s > 0.0 ? static_cast<float>(r[c] / s) : 0.0f;
    }
    x0 = __shfl_sync(grp_mask, x0, 0, 8);
    if (c >= cells) return;
    const float fv = feats[i], fp = feats[n + i], fd = feats[2 * n + i];
    const float* W = P + OFF_WIN;
    float o[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int f = 4 * quarter + q;
        const float pre = P[OFF_BIN + f] + W[f * 4 + 0] * x0 + W[f * 4 + 1] * fv + W[f * 4 + 2] * fp +
                          W[f * 4 + 3] * fd;
        o[q] = fmaxf(pre, 0.0f);
    }
    reinterpret_cast<float4*>(h)[c * (F / 4) + quarter] = make_float4(o[0], o[1], o[2], o[3]);
}

// ---- training tiles
//
// A block of 128 threads takes 64 cells at a time, their features transposed
// in shared memory ([feature][cell]), and forms every layer's products as
// register tiles (4 cells x 4 outputs per thread: two 16-byte shared loads
// per 16 multiply-adds), so the kernels run on the FMA pipe.  The earlier
// form, a warp per cell with a shuffle per multiply-add and one pair at a
// time, spent 23 us per forward and 80 us per backward round on 24,576 cells
// (16^3 lattice); the tiles take the eight pairs of such a batch together in
// 70 and 127 us (a batch's gradient 4.67 -> 1.00 ms; the multiply-adds alone
// are 17 and 34 us at the FP32 rate: the rest is the gather's L2 latency
// between the tile's barriers).
// Cells are stored in groups of four, group g of row m at g ^ (m / 4 mod 8):
// the transposing stores (8 lanes per cell, 4 features each) and the 16-byte
// loads are then free of bank conflicts.
__device__ __forceinline__ int tile_at(int row, int cell) {
    return row * kTrainTile + ((((cell >> 2) ^ ((row >> 2) & 7)) << 2) | (cell & 3));
}
__device__ __forceinline__ float4 tile_ld4(const float* t, int row, int group) {
    return *reinterpret_cast<const float4*>(t + row * kTrainTile + ((group ^ ((row >> 2) & 7)) << 2));
}
__device__ __forceinline__ void tile_st4(float* t, int row, int group, float4 v) {
    *reinterpret_cast<float4*>(t + row * kTrainTile + ((group ^ ((row >> 2) & 7)) << 2)) = v;
}
// features 4q..4q+3 of one cell into rows row0 + 4q..
__device__ __forceinline__ void tile_put(float* t, int row0, int quarter, int cell, float4 v) {
    t[tile_at(row0 + 4 * quarter + 0, cell)] = v.x;
    t[tile_at(row0 + 4 * quarter + 1, cell)] = v.y;
    t[tile_at(row0 + 4 * quarter + 2, cell)] = v.z;
    t[tile_at(row0 + 4 * quarter + 3, cell)] = v.w;
}

// sum over the couplings of cell i of w_ij v_j (one lane's four features; base
// = first cell of the pair), four neighbour rows in flight
__device__ __forceinline__ float4 gather_couplings(const int* __restrict__ gro, const int* __restrict__ gco,
                                                   const float* __restrict__ gew, const float* __restrict__ v,
                                                   int i, int base, int quarter) {
    const float4* rows = reinterpret_cast<const float4*>(v) + base * (F / 4) + quarter;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
    const int b = gro[i], e = gro[i + 1];
    for (int k0 = b; k0 < e; k0 += 4) {
        float4 x[4];
        float w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool ok = k0 + u < e;
            w[u] = ok ? gew[k0 + u] : 0.0f;
            const int j = ok ? gco[k0 + u] : i;
            x[u] = rows[j * (F / 4)];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (k0 + u < e) {
                a.x += w[u] * x[u].x; a.y += w[u] * x[u].y; a.z += w[u] * x[u].z; a.w += w[u] * x[u].w;
            }
    }
    return a;
}

__device__ __forceinline__ void fma4x4(float (&acc)[4][4], float4 u, float4 w) {
    const float uu[4] = {u.x, u.y, u.z, u.w}, ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int o = 0; o < 4; ++o) acc[c][o] += uu[c] * ww[o];
}

// One round forward: a_i = sum_j w_ij h_j; z = W1 [h, a] + b1;
// h_next = h + W2 relu(z) + b2.  Keeps a and z for the backward pass.
__global__ void __launch_bounds__(kThreads) k_round_fwd(int n, int cells, const int* __restrict__ gro,
                                                        const int* __restrict__ gco, const float* __restrict__ gew,
                                                        const float* __restrict__ h, const float* __restrict__ Pr,
                                                        float* __restrict__ ag, float* __restrict__ z,
                                                        float* __restrict__ hn) {
    __shared__ __align__(16) float sU[2 * F * kTrainTile];
    __shared__ __align__(16) float sG[F * kTrainTile];
    __shared__ __align__(16) float sW1[2 * F * F];   // [input][output]
    __shared__ __align__(16) float sW2[F * F];       // [input][output]
    for (int q = threadIdx.x; q < 2 * F * F; q += kThreads) sW1[q] = Pr[OFF_W1 + (q % F) * (2 * F) + q / F];
    for (int q = threadIdx.x; q < F * F; q += kThreads) sW2[q] = Pr[OFF_W2 + (q % F) * F + q / F];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int quarter = lane & 7;
    const int cg = (lane & 7) + 8 * (warp & 1), og = (lane >> 3) + 4 * (warp >> 1);
    float b1[4], b2[4];
#pragma unroll
    for (int o = 0; o < 4; ++o) {
        b1[o] = Pr[OFF_B1 + 4 * og + o];
        b2[o] = Pr[OFF_B2 + 4 * og + o];
    }
    const int tiles = (cells + kTrainTile - 1) / kTrainTile;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int c0 = tile * kTrainTile;
        __syncthreads();   // the previous tile's reads (and the weights) are done
#pragma unroll
        for (int pass = 0; pass < kTrainTile / 16; ++pass) {
            const int c = warp * (kTrainTile / kWarps) + pass * 4 + (lane >> 3);
            const int g = c0 + c;
            float4 hv = make_float4(0.f, 0.f, 0.f, 0.f), av = hv;
            if (g < cells) {
                const int base = g / n * n;
                hv = reinterpret_cast<const float4*>(h)[g * (F / 4) + quarter];
                av = gather_couplings(gro, gco, gew, h, g - base, base, quarter);
                reinterpret_cast<float4*>(ag)[g * (F / 4) + quarter] = av;
            }
            tile_put(sU, 0, quarter, c, hv);
            tile_put(sU, F, quarter, c, av);
        }
        __syncthreads();
        float acc[4][4];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int o = 0; o < 4; ++o) acc[c][o] = b1[o];
#pragma unroll 8
        for (int m = 0; m < 2 * F; ++m)
            fma4x4(acc, tile_ld4(sU, m, cg), *reinterpret_cast<const float4*>(sW1 + m * F + 4 * og));
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int g = c0 + 4 * cg + c;
            if (g < cells)
                reinterpret_cast<float4*>(z)[g * (F / 4) + og] =
                    make_float4(acc[c][0], acc[c][1], acc[c][2], acc[c][3]);
        }
#pragma unroll
        for (int o = 0; o < 4; ++o)
            tile_st4(sG, 4 * og + o, cg, make_float4(fmaxf(acc[0][o], 0.f), fmaxf(acc[1][o], 0.f),
                                                     fmaxf(acc[2][o], 0.f), fmaxf(acc[3][o], 0.f)));
        __syncthreads();
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int o = 0; o < 4; ++o) acc[c][o] = b2[o];
#pragma unroll 8
        for (int q = 0; q < F; ++q)
            fma4x4(acc, tile_ld4(sG, q, cg), *reinterpret_cast<const float4*>(sW2 + q * F + 4 * og));
        float hrow[4][4];
#pragma unroll
        for (int o = 0; o < 4; ++o) {
            const float4 v = tile_ld4(sU, 4 * og + o, cg);
            hrow[0][o] = v.x; hrow[1][o] = v.y; hrow[2][o] = v.z; hrow[3][o] = v.w;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int g = c0 + 4 * cg + c;
            if (g < cells)
                reinterpret_cast<float4*>(hn)[g * (F / 4) + og] =
                    make_float4(hrow[c][0] + acc[c][0], hrow[c][1] + acc[c][1], hrow[c][2] + acc[c][2],
                                hrow[c][3] + acc[c][3]);
        }
    }
}

// out_i = s (w_out . h_i + b_out) / a_ii.  Eight lanes per cell (16-byte loads),
// combined with a fixed butterfly.
__global__ void k_readout(int n, int cells, const float* __restrict__ h, const float* __restrict__ P,
                          const double* __restrict__ rr, const double* __restrict__ diag, double* __restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = t >> 3;
    const int quarter = static_cast<int>(t & 7);
    const unsigned grp_mask = 0xffu << (threadIdx.x & 24);
    float y = 0.0f;
    if (c < cells) {
        const float4 v = reinterpret_cast<const float4*>(h)[c * (F / 4) + quarter];
        const float* w = P + OFF_WOUT + 4 * quarter;
        y = w[0] * v.x + w[1] * v.y + w[2] * v.z + w[3] * v.w;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) y += __shfl_xor_sync(grp_mask, y, o, 8);
    if (c < cells && quarter == 0) {
        const int pair = c / n;
        const double s = sqrt(rr[pair] / n);
        out[c] = s * static_cast<double>(y + P[OFF_BOUT]) / diag[c - pair * n];
    }
}

// ---------------- fused tensor-core round (inference) ----------------
__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

__device__ __forceinline__ uint32_t ld32(const __nv_bfloat16* p) { return *reinterpret_cast<const uint32_t*>(p); }

// Inference rounds.  A warp owns 16 consecutive cells, rows g and g + 8 (g =
// lane / 4) of the MMA tile, and the four lanes of a row (t = lane % 4) gather
// its neighbours' states 16 bytes each.  The state between rounds is stored in
// the order in which the MMA's registers hold it: a lane's 16 bytes are
// features 8 p + 2 t and 8 p + 2 t + 1, p = 0 .. 3 (lane_feature), its pairs of
// k slots in the A operand and its columns of the result.  So [h, a] is the A
// operand straight from registers, with feature f in k slot f; the new state
// leaves in 16-byte stores, and nothing passes through shared memory.  (The k
// slots matter: another assignment adds the FP32 products in another order,
// which turned some BF16 roundings of the state over the rounds and moved the
// result by 1.7e-4.)  The
// weights stay in registers (48) over the warp's tiles, and a tile's couplings
// are loaded one tile ahead.  Bound by the latency of the L2 gathers (some 400
// bytes a cell and round): four rounds at 663,552 cells take 250 us; with 8
// lanes of 8 bytes per row and the operands staged in shared memory 330.
constexpr int kTileCells = 16;
constexpr int kRoundThreads = 128;

// feature q (0 .. 7) of lane t of a row
__device__ __forceinline__ constexpr int lane_feature(int t, int q) { return 8 * (q >> 1) + 2 * t + (q & 1); }

// x_i = [r_i / s, f_V, f_P, f_D] packed as one float4 per cell (k_encode's
// input, 16 bytes), so the first round reads it instead of a 128-byte h0 row.
__global__ void k_pack_input(int n, const double* __restrict__ r, const double* __restrict__ rr,
                             const float* __restrict__ feats, float4* __restrict__ xin) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double s = sqrt(*rr / n);
    const float x0 = s > 0.0 ? static_cast<float>(r[i] / s) : 0.0f;
    xin[i] = make_float4(x0, feats[i], feats[n + i], feats[2 * n + i]);
}

// One row's state of the lane's eight features as FP32.  BF16 -> FP32 is
// exact: the BF16 bits are the upper half of the FP32 word.
__device__ __forceinline__ void unpack8(uint4 u, float (&f)[8]) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        f[2 * q] = __uint_as_float(w[q] << 16);
        f[2 * q + 1] = __uint_as_float(w[q] & 0xffff0000u);
    }
}

// The first round's state h0 = relu(W_in x + b_in), formed where the round
// reads it (k_encode's arithmetic) instead of being written by a separate
// kernel and read back: the lane's eight features.
struct Encoder {
    float w[8][4], b[8];
    __device__ __forceinline__ void load(const float* P, int t) {
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int f = lane_feature(t, q);
            b[q] = P[OFF_BIN + f];
#pragma unroll
            for (int c = 0; c < 4; ++c) w[q][c] = P[OFF_WIN + f * 4 + c];
        }
    }
    __device__ __forceinline__ void h0(float4 x, float (&f)[8]) const {
#pragma unroll
        for (int q = 0; q < 8; ++q)
            f[q] = fmaxf(b[q] + w[q][0] * x.x + w[q][1] * x.y + w[q][2] * x.z + w[q][3] * x.w, 0.0f);
    }
};

// The couplings of one tile row: its range, and this lane's entry of the first four.
struct RowCouplings {
    int b, e, j;
    float w;
};

__device__ __forceinline__ RowCouplings load_couplings(int cell, int n, int t, const int* __restrict__ gro,
                                                       const int* __restrict__ gco, const float* __restrict__ gew) {
    RowCouplings c{0, 0, cell < n ? cell : 0, 0.0f};
    if (cell < n) {
        c.b = gro[cell];
        c.e = gro[cell + 1];
        if (c.b + t < c.e) {
            c.j = gco[c.b + t];
            c.w = gew[c.b + t];
        }
    }
    return c;
}

// One round.  FIRST: the input state is formed from r by the encoder (no h0
// in memory).  LAST: the new state goes straight to the readout,
// out_i = s (w_out . h_i + b_out) / a_ii, instead of to h_out.
template <bool FIRST, bool LAST>
__global__ void __launch_bounds__(kRoundThreads, FIRST ? 2 : 4) k_round_gather_tc(
    int n, const int* __restrict__ gro, const int* __restrict__ gco, const float* __restrict__ gew,
    const float4* __restrict__ xin, const __nv_bfloat16* __restrict__ h_in, __nv_bfloat16* __restrict__ h_out,
    const __nv_bfloat16* __restrict__ W1g, const __nv_bfloat16* __restrict__ W2g, const float* __restrict__ Pr,
    const float* __restrict__ P, const double* __restrict__ rr, const double* __restrict__ diag,
    double* __restrict__ yout) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // B operands (W1's k blocks 0, 1: h; 2, 3: a)
    uint32_t w1[4][4][2], w2[2][4][2];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __nv_bfloat16* row = W1g + (8 * j + g) * (2 * F) + 16 * k + 2 * t;
            w1[k][j][0] = ld32(row);
            w1[k][j][1] = ld32(row + 8);
        }
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __nv_bfloat16* row = W2g + (8 * j + g) * F + 16 * k + 2 * t;
            w2[k][j][0] = ld32(row);
            w2[k][j][1] = ld32(row + 8);
        }
    Encoder enc;
    if constexpr (FIRST) enc.load(P, t);
    const double scale = LAST ? sqrt(*rr / n) : 0.0;
    const uint4* h16 = reinterpret_cast<const uint4*>(h_in);
    const int warps = gridDim.x * (kRoundThreads / 32);
    int tile = blockIdx.x * (kRoundThreads / 32) + (threadIdx.x >> 5);
    if (tile * kTileCells >= n) return;
    RowCouplings cur[2];
#pragma unroll
    for (int p = 0; p < 2; ++p) cur[p] = load_couplings(tile * kTileCells + g + 8 * p, n, t, gro, gco, gew);
    for (; tile * kTileCells < n; tile += warps) {
        const int c0 = tile * kTileCells;
        float hv[2][8], av[2][8];
        uint32_t ah[2][4];
        // the first four neighbours of both rows, all loads in flight together
        if constexpr (FIRST) {
            float4 xo[2], xn[2][4];
            float w[2][4];
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const int cell = min(c0 + g + 8 * p, n - 1);
                xo[p] = xin[cell];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    xn[p][u] = xin[__shfl_sync(0xffffffffu, cur[p].j, u, 4)];
                    w[p][u] = __shfl_sync(0xffffffffu, cur[p].w, u, 4);
                }
            }
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                enc.h0(xo[p], hv[p]);
#pragma unroll
                for (int q = 0; q < 8; ++q) av[p][q] = 0.0f;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float v[8];
                    enc.h0(xn[p][u], v);
#pragma unroll
                    for (int q = 0; q < 8; ++q) av[p][q] += w[p][u] * v[q];
                }
#pragma unroll
                for (int q = 0; q < 4; ++q) ah[p][q] = pack_bf16(hv[p][2 * q], hv[p][2 * q + 1]);
            }
        } else {
            uint4 own[2], nb[2][4];
            float w[2][4];
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const int cell = min(c0 + g + 8 * p, n - 1);
                own[p] = h16[cell * (F / 8) + t];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    nb[p][u] = h16[__shfl_sync(0xffffffffu, cur[p].j, u, 4) * (F / 8) + t];
                    w[p][u] = __shfl_sync(0xffffffffu, cur[p].w, u, 4);
                }
            }
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                unpack8(own[p], hv[p]);
                ah[p][0] = own[p].x; ah[p][1] = own[p].y; ah[p][2] = own[p].z; ah[p][3] = own[p].w;
#pragma unroll
                for (int q = 0; q < 8; ++q) av[p][q] = 0.0f;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    float v[8];
                    unpack8(nb[p][u], v);
#pragma unroll
                    for (int q = 0; q < 8; ++q) av[p][q] += w[p][u] * v[q];
                }
            }
        }
        // rows of more than four neighbours
#pragma unroll
        for (int p = 0; p < 2; ++p)
            for (int k0 = cur[p].b + 4; __any_sync(0xffffffffu, k0 < cur[p].e); k0 += 4) {
                const int self = min(c0 + g + 8 * p, n - 1);
                const int j = k0 + t < cur[p].e ? gco[k0 + t] : self;
                const float wj = k0 + t < cur[p].e ? gew[k0 + t] : 0.0f;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int ju = __shfl_sync(0xffffffffu, j, u, 4);
                    const float wu = __shfl_sync(0xffffffffu, wj, u, 4);
                    float v[8];
                    if constexpr (FIRST) enc.h0(xin[ju], v);
                    else unpack8(h16[ju * (F / 8) + t], v);
#pragma unroll
                    for (int q = 0; q < 8; ++q) av[p][q] += wu * v[q];
                }
            }
        // the next tile's couplings, in flight during the products
        if ((tile + warps) * kTileCells < n) {
#pragma unroll
            for (int p = 0; p < 2; ++p)
                cur[p] = load_couplings((tile + warps) * kTileCells + g + 8 * p, n, t, gro, gco, gew);
        }
        float acc[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 b1 = *reinterpret_cast<const float2*>(Pr + OFF_B1 + 8 * j + 2 * t);
            acc[j][0] = acc[j][2] = b1.x;
            acc[j][1] = acc[j][3] = b1.y;
        }
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                mma_bf16(acc[j], ah[0][2 * k], ah[1][2 * k], ah[0][2 * k + 1], ah[1][2 * k + 1], w1[k][j][0],
                         w1[k][j][1]);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t a0 = pack_bf16(av[0][4 * k], av[0][4 * k + 1]);
            const uint32_t a1 = pack_bf16(av[1][4 * k], av[1][4 * k + 1]);
            const uint32_t a2 = pack_bf16(av[0][4 * k + 2], av[0][4 * k + 3]);
            const uint32_t a3 = pack_bf16(av[1][4 * k + 2], av[1][4 * k + 3]);
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_bf16(acc[j], a0, a1, a2, a3, w1[2 + k][j][0], w1[2 + k][j][1]);
        }
        float out[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 b2 = *reinterpret_cast<const float2*>(Pr + OFF_B2 + 8 * j + 2 * t);
            out[j][0] = b2.x + hv[0][2 * j];
            out[j][1] = b2.y + hv[0][2 * j + 1];
            out[j][2] = b2.x + hv[1][2 * j];
            out[j][3] = b2.y + hv[1][2 * j + 1];
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t a0 = pack_bf16(fmaxf(acc[2 * k][0], 0.f), fmaxf(acc[2 * k][1], 0.f));
            const uint32_t a1 = pack_bf16(fmaxf(acc[2 * k][2], 0.f), fmaxf(acc[2 * k][3], 0.f));
            const uint32_t a2 = pack_bf16(fmaxf(acc[2 * k + 1][0], 0.f), fmaxf(acc[2 * k + 1][1], 0.f));
            const uint32_t a3 = pack_bf16(fmaxf(acc[2 * k + 1][2], 0.f), fmaxf(acc[2 * k + 1][3], 0.f));
#pragma unroll
            for (int j = 0; j < 4; ++j) mma_bf16(out[j], a0, a1, a2, a3, w2[k][j][0], w2[k][j][1]);
        }
        if constexpr (LAST) {
            // readout: row sums over this lane's features, then across the 4 lanes of the row
            float ya = 0.0f, yb = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float wo0 = P[OFF_WOUT + 8 * j + 2 * t], wo1 = P[OFF_WOUT + 8 * j + 2 * t + 1];
                ya += wo0 * out[j][0] + wo1 * out[j][1];
                yb += wo0 * out[j][2] + wo1 * out[j][3];
            }
            ya += __shfl_xor_sync(0xffffffffu, ya, 1);
            ya += __shfl_xor_sync(0xffffffffu, ya, 2);
            yb += __shfl_xor_sync(0xffffffffu, yb, 1);
            yb += __shfl_xor_sync(0xffffffffu, yb, 2);
            if (t == 0) {
                const float bo = P[OFF_BOUT];
                const int ra = c0 + g, rb = c0 + g + 8;
                if (ra < n) yout[ra] = scale * static_cast<double>(ya + bo) / diag[ra];
                if (rb < n) yout[rb] = scale * static_cast<double>(yb + bo) / diag[rb];
            }
        } else {
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                const int row = c0 + g + 8 * p;
                if (row < n)
                    reinterpret_cast<uint4*>(h_out)[row * (F / 8) + t] =
                        make_uint4(pack_bf16(out[0][2 * p], out[0][2 * p + 1]),
                                   pack_bf16(out[1][2 * p], out[1][2 * p + 1]),
                                   pack_bf16(out[2][2 * p], out[2][2 * p + 1]),
                                   pack_bf16(out[3][2 * p], out[3][2 * p + 1]));
            }
        }
    }
}

// ---------------- backward (FP32) ----------------
// loss pieces: d = e - out
__global__ void k_sub(int n, const double* __restrict__ e, const double* __restrict__ out, double* __restrict__ d) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) d[i] = e[i] - out[i];
}

// out[pair] = r . r of each pair: blockIdx.y is the pair, its blocks' partials
// added in block order by the last of them (as k_dot)
__global__ void k_pair_norms(int n, const double* __restrict__ r, double* sums, unsigned* tickets, double* out) {
    __shared__ double sm[32];
    const double* v = r + static_cast<int64_t>(blockIdx.y) * n;
    double s = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) s += v[i] * v[i];
    s = block_sum(s, sm);
    double* part = sums + static_cast<int64_t>(blockIdx.y) * gridDim.x;
    if (threadIdx.x == 0) part[blockIdx.x] = s;
    if (last_block(tickets + blockIdx.y)) {
        double t = 0.0;
        for (int q = threadIdx.x; q < static_cast<int>(gridDim.x); q += blockDim.x) t += part[q];
        t = block_sum(t, sm);
        if (threadIdx.x == 0) {
            out[blockIdx.y] = t;
            tickets[blockIdx.y] = 0;
        }
    }
}

// The loss products of each pair (blockIdx.y) in one pass over the operator:
// Ad = A (e - out), eAe = e . A e and dAd = (e - out) . A (e - out).
__global__ void k_pair_energies(int n, const int* __restrict__ ro, const int* __restrict__ co,
                                const double* __restrict__ va, const double* __restrict__ e_all,
                                const double* __restrict__ out_all, double* __restrict__ Ad_all, double* sums,
                                unsigned* tickets, double* eAe, double* dAd) {
    __shared__ double sm[32];
    const int64_t base = static_cast<int64_t>(blockIdx.y) * n;
    const double *e = e_all + base, *out = out_all + base;
    double se = 0.0, sd = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double ae = 0.0, ad = 0.0;
        const int end = ro[i + 1];
#pragma unroll 4
        for (int k = ro[i]; k < end; ++k) {
            const int j = co[k];
            const double v = va[k], ej = e[j], dj = ej - out[j];
            ae += v * ej;
            ad += v * dj;
        }
        Ad_all[base + i] = ad;
        const double ei = e[i];
        se += ei * ae;
        sd += (ei - out[i]) * ad;
    }
    se = block_sum(se, sm);
    sd = block_sum(sd, sm);
    double* part = sums + 2 * static_cast<int64_t>(blockIdx.y) * gridDim.x;
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = se;
        part[2 * blockIdx.x + 1] = sd;
    }
    if (last_block(tickets + blockIdx.y)) {
        double te = 0.0, td = 0.0;
        for (int q = threadIdx.x; q < static_cast<int>(gridDim.x); q += blockDim.x) {
            te += part[2 * q];
            td += part[2 * q + 1];
        }
        te = block_sum(te, sm);
        td = block_sum(td, sm);
        if (threadIdx.x == 0) {
            eAe[blockIdx.y] = te;
            dAd[blockIdx.y] = td;
            tickets[blockIdx.y] = 0;
        }
    }
}

// dy = s * (-2 Ad / eAe) / a_ii
__global__ void k_dy(int n, int cells, const double* __restrict__ Ad, const double* __restrict__ eAe,
                     const double* __restrict__ rr, const double* __restrict__ diag, float* __restrict__ dy) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cells) return;
    const int pair = c / n;
    const double s = sqrt(rr[pair] / n);
    dy[c] = static_cast<float>(s * (-2.0 * Ad[c] / eAe[pair]) / diag[c - pair * n]);
}

// Adds a lane's accumulators (features 4 quarter .. 4 quarter + 3, V values
// each, at base + feature V + q) over the warp's four cell groups, then over
// the warps in order, into the block's partial.
template <int V>
__device__ __forceinline__ void block_accumulate(float (*acc_smem)[F * V], const float (&lane_vals)[4][V],
                                                 int base, float* partial_block) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int f = 0; f < 4; ++f)
#pragma unroll
        for (int q = 0; q < V; ++q) {
            float v = lane_vals[f][q];
            v += __shfl_xor_sync(0xffffffffu, v, 8);
            v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (lane < 8) acc_smem[warp][(4 * lane + f) * V + q] = v;
        }
    __syncthreads();
    for (int q = threadIdx.x; q < F * V; q += kThreads) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) t += acc_smem[w][q];
        partial_block[base + q] += t;
    }
    __syncthreads();
}

// dL/dh_R = w_out dy, and the readout's gradients.  Eight lanes per cell.
__global__ void __launch_bounds__(kThreads) k_readout_bwd(int cells, const float* __restrict__ h,
                                                          const float* __restrict__ dy, const float* __restrict__ P,
                                                          float* __restrict__ dh, float* __restrict__ partial) {
    __shared__ float acc[kWarps][F];
    __shared__ float accb[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quarter = lane & 7;
    float w[4], aw[4][1] = {{0.f}, {0.f}, {0.f}, {0.f}}, ab = 0.0f;
#pragma unroll
    for (int f = 0; f < 4; ++f) w[f] = P[OFF_WOUT + 4 * quarter + f];
    const int stride = gridDim.x * kWarps * 4;
#pragma unroll 2
    for (int c = (blockIdx.x * kWarps + warp) * 4 + (lane >> 3); c < cells; c += stride) {
        const float d = dy[c];
        const float4 v = reinterpret_cast<const float4*>(h)[c * (F / 4) + quarter];
        reinterpret_cast<float4*>(dh)[c * (F / 4) + quarter] = make_float4(w[0] * d, w[1] * d, w[2] * d, w[3] * d);
        aw[0][0] += d * v.x; aw[1][0] += d * v.y; aw[2][0] += d * v.z; aw[3][0] += d * v.w;
        ab += d;
    }
    float* pb = partial + static_cast<size_t>(blockIdx.x) * NP;
    block_accumulate<1>(acc, aw, OFF_WOUT, pb);
    ab += __shfl_xor_sync(0xffffffffu, ab, 8);
    ab += __shfl_xor_sync(0xffffffffu, ab, 16);
    if (lane == 0) accb[warp] = ab;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
        for (int q = 0; q < kWarps; ++q) t += accb[q];
        pb[OFF_BOUT] += t;
    }
}

// One round backward over the same tiles as k_round_fwd.  The gradient of the
// round's output state is dL/dh_{k+1} = dh + sum_i w_ji da_i (symmetric
// couplings: a gather over da_in, absent in the last round); the kernel leaves
// the part of dL/dh_k known without the couplings in dh (own cells only, so
// in place) and dL/da_k in da_out for the next gather, and adds the weight
// gradients to this block's partial: every thread keeps its gradient entries
// (4 x 4 of dW1, 4 x 2 of dW2) in registers over its block's tiles.
__global__ void __launch_bounds__(kThreads) k_round_bwd(int n, int cells, const int* __restrict__ gro,
                                                        const int* __restrict__ gco, const float* __restrict__ gew,
                                                        const float* __restrict__ h, const float* __restrict__ ag,
                                                        const float* __restrict__ z, const float* __restrict__ Pr,
                                                        const float* __restrict__ da_in, float* __restrict__ dh,
                                                        float* __restrict__ da_out, float* __restrict__ partial,
                                                        int round_base) {
    // exactly 48 KB; W2 is read through the L1 cache (4 KB)
    __shared__ __align__(16) float sU[2 * F * kTrainTile];   // [h, a]
    __shared__ __align__(16) float sD[F * kTrainTile];       // dL/dh_{k+1}
    __shared__ __align__(16) float sG[F * kTrainTile];       // z, then relu(z)
    __shared__ __align__(16) float sE[F * kTrainTile];       // dL/dz
    __shared__ __align__(16) float sW1[F * 2 * F];           // [output][input]
    for (int q = threadIdx.x; q < 2 * F * F; q += kThreads) sW1[q] = Pr[OFF_W1 + q];
    const float4* W2 = reinterpret_cast<const float4*>(Pr + OFF_W2);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quarter = lane & 7;
    const int cg = (lane & 7) + 8 * (warp & 1), og = (lane >> 3) + 4 * (warp >> 1);
    // gradient entries of this thread: dW1 rows 4 q1 .., columns 4 m1 ..;
    // dW2 rows 4 o2 .., columns 2 q2 ..
    const int q1 = (lane & 3) + 4 * (warp & 1), m1 = (lane >> 2) + 8 * (warp >> 1);
    const int o2 = (lane & 3) + 4 * (warp & 1), q2 = (lane >> 2) + 8 * (warp >> 1);
    float gW1[4][4], gW2[4][2], gb1[4], gb2[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        gb1[a] = gb2[a] = 0.0f;
#pragma unroll
        for (int b = 0; b < 4; ++b) gW1[a][b] = 0.0f;
        gW2[a][0] = gW2[a][1] = 0.0f;
    }
    const int tiles = (cells + kTrainTile - 1) / kTrainTile;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int c0 = tile * kTrainTile;
        __syncthreads();
#pragma unroll
        for (int pass = 0; pass < kTrainTile / 16; ++pass) {
            const int c = warp * (kTrainTile / kWarps) + pass * 4 + (lane >> 3);
            const int g = c0 + c;
            float4 hv = make_float4(0.f, 0.f, 0.f, 0.f), av = hv, zv = hv, dv = hv;
            if (g < cells) {
                hv = reinterpret_cast<const float4*>(h)[g * (F / 4) + quarter];
                av = reinterpret_cast<const float4*>(ag)[g * (F / 4) + quarter];
                zv = reinterpret_cast<const float4*>(z)[g * (F / 4) + quarter];
                dv = reinterpret_cast<const float4*>(dh)[g * (F / 4) + quarter];
                if (da_in) {
                    const int base = g / n * n;
                    const float4 s = gather_couplings(gro, gco, gew, da_in, g - base, base, quarter);
                    dv.x += s.x; dv.y += s.y; dv.z += s.z; dv.w += s.w;
                }
            }
            tile_put(sU, 0, quarter, c, hv);
            tile_put(sU, F, quarter, c, av);
            tile_put(sG, 0, quarter, c, zv);
            tile_put(sD, 0, quarter, c, dv);
        }
        __syncthreads();
        {
            // dL/dz[q] = (z[q] > 0) sum_o W2[o][q] dL/dh[o]
            float acc[4][4] = {};
#pragma unroll 8
            for (int o = 0; o < F; ++o) fma4x4(acc, tile_ld4(sD, o, cg), __ldg(W2 + o * (F / 4) + og));
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 v = tile_ld4(sG, 4 * og + q, cg);
                tile_st4(sE, 4 * og + q, cg,
                         make_float4(v.x > 0.f ? acc[0][q] : 0.f, v.y > 0.f ? acc[1][q] : 0.f,
                                     v.z > 0.f ? acc[2][q] : 0.f, v.w > 0.f ? acc[3][q] : 0.f));
                tile_st4(sG, 4 * og + q, cg,
                         make_float4(fmaxf(v.x, 0.f), fmaxf(v.y, 0.f), fmaxf(v.z, 0.f), fmaxf(v.w, 0.f)));
            }
        }
        __syncthreads();
        // weight gradients: sums over the tile's cells, four at a time
#pragma unroll 4
        for (int g = 0; g < kTrainTile / 4; ++g) {
            float4 dq[4], um[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                dq[a] = tile_ld4(sE, 4 * q1 + a, g);
                um[a] = tile_ld4(sU, 4 * m1 + a, g);
            }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b)
                    gW1[a][b] += dq[a].x * um[b].x + dq[a].y * um[b].y + dq[a].z * um[b].z + dq[a].w * um[b].w;
            if (m1 == 0) {
#pragma unroll
                for (int a = 0; a < 4; ++a) gb1[a] += (dq[a].x + dq[a].y) + (dq[a].z + dq[a].w);
            }
        }
#pragma unroll 4
        for (int g = 0; g < kTrainTile / 4; ++g) {
            float4 d[4], v[2];
#pragma unroll
            for (int a = 0; a < 4; ++a) d[a] = tile_ld4(sD, 4 * o2 + a, g);
            v[0] = tile_ld4(sG, 2 * q2, g);
            v[1] = tile_ld4(sG, 2 * q2 + 1, g);
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b)
                    gW2[a][b] += d[a].x * v[b].x + d[a].y * v[b].y + d[a].z * v[b].z + d[a].w * v[b].w;
            if (q2 == 0) {
#pragma unroll
                for (int a = 0; a < 4; ++a) gb2[a] += (d[a].x + d[a].y) + (d[a].z + d[a].w);
            }
        }
        // d[h, a][m] = sum_q W1[q][m] dL/dz[q]: the h half (+ dL/dh_{k+1}) to dh, the a half to da
        {
            float lo[4][4] = {}, hi[4][4] = {};
#pragma unroll 4
            for (int q = 0; q < F; ++q) {
                const float4 d = tile_ld4(sE, q, cg);
                fma4x4(lo, d, *reinterpret_cast<const float4*>(sW1 + q * 2 * F + 4 * og));
                fma4x4(hi, d, *reinterpret_cast<const float4*>(sW1 + q * 2 * F + F + 4 * og));
            }
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const float4 v = tile_ld4(sD, 4 * og + m, cg);
                lo[0][m] = v.x + lo[0][m]; lo[1][m] = v.y + lo[1][m];
                lo[2][m] = v.z + lo[2][m]; lo[3][m] = v.w + lo[3][m];
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int g = c0 + 4 * cg + c;
                if (g >= cells) continue;
                reinterpret_cast<float4*>(dh)[g * (F / 4) + og] = make_float4(lo[c][0], lo[c][1], lo[c][2], lo[c][3]);
                reinterpret_cast<float4*>(da_out)[g * (F / 4) + og] =
                    make_float4(hi[c][0], hi[c][1], hi[c][2], hi[c][3]);
            }
        }
    }
    float* pb = partial + static_cast<size_t>(blockIdx.x) * NP + round_base;
#pragma unroll
    for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int b = 0; b < 4; ++b) pb[OFF_W1 + (4 * q1 + a) * (2 * F) + 4 * m1 + b] += gW1[a][b];
#pragma unroll
        for (int b = 0; b < 2; ++b) pb[OFF_W2 + (4 * o2 + a) * F + 2 * q2 + b] += gW2[a][b];
        if (m1 == 0) pb[OFF_B1 + 4 * q1 + a] += gb1[a];
        if (q2 == 0) pb[OFF_B2 + 4 * o2 + a] += gb2[a];
    }
}

// The encoder's gradients, dL/dh_0 formed as in k_round_bwd.  Eight lanes per cell.
__global__ void __launch_bounds__(kThreads) k_encode_bwd(int n, int cells, const int* __restrict__ gro,
                                                         const int* __restrict__ gco, const float* __restrict__ gew,
                                                         const double* __restrict__ r, const double* __restrict__ rr,
                                                         const float* __restrict__ feats, const float* __restrict__ h0,
                                                         const float* __restrict__ dh, const float* __restrict__ da,
                                                         float* __restrict__ partial) {
    __shared__ float acc[kWarps][F * 4];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, quarter = lane & 7;
    float gw[4][4], gb[4][1];
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        gb[f][0] = 0.0f;
#pragma unroll
        for (int q = 0; q < 4; ++q) gw[f][q] = 0.0f;
    }
    const int stride = gridDim.x * kWarps * 4;
    for (int c = (blockIdx.x * kWarps + warp) * 4 + (lane >> 3); c < cells; c += stride) {
        const int pair = c / n, base = pair * n, i = c - base;
        const float4 hv = reinterpret_cast<const float4*>(h0)[c * (F / 4) + quarter];
        const float4 dv = reinterpret_cast<const float4*>(dh)[c * (F / 4) + quarter];
        const float4 s4 = gather_couplings(gro, gco, gew, da, i, base, quarter);
        const float d[4] = {hv.x > 0.f ? dv.x + s4.x : 0.f, hv.y > 0.f ? dv.y + s4.y : 0.f,
                            hv.z > 0.f ? dv.z + s4.z : 0.f, hv.w > 0.f ? dv.w + s4.w : 0.f};
        const double s = sqrt(rr[pair] / n);
        const float x[4] = {s > 0.0 ? static_cast<float>(r[c] / s) : 0.0f, feats[i], feats[n + i], feats[2 * n + i]};
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            gb[f][0] += d[f];
#pragma unroll
            for (int q = 0; q < 4; ++q) gw[f][q] += d[f] * x[q];
        }
    }
    float* pb = partial + static_cast<size_t>(blockIdx.x) * NP;
    block_accumulate<4>(acc, gw, OFF_WIN, pb);
    block_accumulate<1>(reinterpret_cast<float(*)[F]>(acc), gb, OFF_BIN, pb);
}

// grad = scale * the blocks' partials: each parameter by eight threads that
// take the blocks in turn, combined in thread order
__global__ void k_reduce_partials(const float* __restrict__ partial, int blocks, float scale, float* __restrict__ grad) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    // 32 parameters per eight warps: lane = parameter, warp = slice of the blocks
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const int p = (t >> 8) * 32 + lane;
    __shared__ float sm[8][32];
    float s = 0.0f;
    if (p < NP)
#pragma unroll 8
        for (int b = slice; b < blocks; b += 8) s += partial[static_cast<size_t>(b) * NP + p];
    sm[slice][lane] = s;
    __syncthreads();
    if (slice == 0 && p < NP) {
        float v = 0.0f;
#pragma unroll
        for (int q = 0; q < 8; ++q) v += sm[q][lane];
        grad[p] = v * scale;
    }
}

__global__ void k_adam(float* __restrict__ P, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                       float lr, float bc1, float bc2) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= NP) return;
    const float gi = g[p];
    m[p] = 0.9f * m[p] + 0.1f * gi;
    v[p] = 0.999f * v[p] + 0.001f * gi * gi;
    P[p] -= lr * (m[p] / bc1) / (sqrtf(v[p] / bc2) + 1e-8f);
}

__global__ void k_to_bf16(const float* __restrict__ P, __nv_bfloat16* __restrict__ wbf) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= R * 3 * F * F) return;
    const int r = q / (3 * F * F), k = q % (3 * F * F);
    const float* base = P + ROUND0 + r * ROUND_SIZE;
    wbf[q] = __float2bfloat16_rn(k < 2 * F * F ? base[OFF_W1 + k] : base[OFF_W2 + (k - 2 * F * F)]);
}

// learned composition helpers
__global__ void k_residual64(int n, const int* __restrict__ ro, const int* __restrict__ co,
                             const double* __restrict__ va, const double* __restrict__ v,
                             const double* __restrict__ y, double* __restrict__ t) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = 0.0;
    for (int k = ro[i]; k < ro[i + 1]; ++k) s += va[k] * y[co[k]];
    t[i] = v[i] - s;
}

__global__ void k_add_inplace(int n, double* __restrict__ z, const double* __restrict__ y) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) z[i] += y[i];
}

// ---------------- host helpers ----------------
void require_bound(const cfdxg_mpnn* net) {
    if (!net->A || net->n <= 0) throw Error(CFDXG_ERR_NOT_READY, "network is not bound to a matrix (cfdxg_mpnn_bind)");
}

void upload_params(cfdxg_context* ctx, cfdxg_mpnn* net) {
    net->params.upload(net->host, ctx->stream);
    net->wbf.resize(static_cast<size_t>(R) * 3 * F * F);
    k_to_bf16<<<blocks_for(R * 3 * F * F, 256), 256, 0, ctx->stream>>>(net->params.get(), net->wbf.get());
    check_launch(ctx);
    CFDXG_CUDA(cudaStreamSynchronize(ctx->stream));
}

// Blocks per pair of the pairs' reductions, and the most pairs in flight.
constexpr int kPairBlocks = 256;
constexpr int kMaxPairs = 64;

double* scalar(cfdxg_context* ctx, int k) { return ctx->scratch.scalars + 3000 + k; }

// Inference: out = N(r) (tensor-core rounds).
void infer(cfdxg_context* ctx, cfdxg_mpnn* net, const double* r, double* out) {
    const int n = net->n;
    cudaStream_t s = ctx->stream;
    double* rr = scalar(ctx, 0);
    enqueue_dot(ctx, n, r, r, rr);
    // the packed first-round input x (16 bytes per cell) in the first quarter
    // of hA: the first round reads it and writes hB, and hA is next written by
    // the second round
    float4* xin = reinterpret_cast<float4*>(net->hA.get());
    {
        ProfScope ps(ctx, "mpnn_pack_input", (8.0 + 12.0 + 16.0) * n);
        k_pack_input<<<blocks_for(n, 256), 256, 0, s>>>(n, r, rr, net->feats.get(), xin);
        check_launch(ctx);
    }
    // the state between rounds is BF16 (64 bytes per cell: the 1.57 M-cell
    // state fits in L2, so the neighbour gathers hit it there)
    __nv_bfloat16* hin = reinterpret_cast<__nv_bfloat16*>(net->hA.get());
    __nv_bfloat16* hout = reinterpret_cast<__nv_bfloat16*>(net->hB.get());
    const int tiles = (n + kTileCells - 1) / kTileCells;
    for (int k = 0; k < R; ++k) {
        const __nv_bfloat16* w = net->wbf.get() + static_cast<size_t>(k) * 3 * F * F;
        const bool first = k == 0, last = k == R - 1;
        // compulsory bytes: the state read (r and the cell features in the
        // first round) and written (the output and diagonal in the last), the
        // coupling list once
        const double in_bytes = first ? 16.0 * n : 2.0 * F * n;
        const double out_bytes = last ? 16.0 * n : 2.0 * F * n;
        ProfScope ps(ctx, first ? "mpnn_round_first_tc" : (last ? "mpnn_round_last_tc" : "mpnn_round_gather_tc"),
                     in_bytes + out_bytes + 4.0 * (n + 1) + 8.0 * static_cast<double>(net->gco.size()));
        auto kern = first ? k_round_gather_tc<true, false>
                          : (last ? k_round_gather_tc<false, true> : k_round_gather_tc<false, false>);
        // one resident wave (two blocks per SM in the first round, whose lanes
        // hold the encoder's weights too, four of 128 registers in the others)
        const int all = (tiles + kRoundThreads / 32 - 1) / (kRoundThreads / 32);
        const int grid = std::min(all, (first ? 2 : 4) * ctx->sm_count);
        kern<<<grid, kRoundThreads, 0, s>>>(n, net->gro.get(), net->gco.get(), net->gew.get(), xin, hin, hout, w,
                                            w + 2 * F * F, net->params.get() + ROUND0 + k * ROUND_SIZE,
                                            net->params.get(), rr, net->diag.get(), out);
        check_launch(ctx);
        std::swap(hin, hout);
    }
}

template <class T>
void grow(DevBuf<T>& b, size_t count) {
    if (b.size() < count) b.resize(count);
}

// Loss terms and gradient (accumulated into net->partial) of `pairs` pairs of
// the batch, the first of them pair `first`: their cells go through every
// kernel together.
void loss_grad_pairs(cfdxg_context* ctx, cfdxg_mpnn* net, const double* r, const double* e, int first, int pairs,
                     int batch) {
    const int n = net->n;
    cudaStream_t s = ctx->stream;
    const int cells = pairs * n;   // below 2^31 / F (the binding's limit, kTrainCells)
    const size_t st = static_cast<size_t>(cells) * F;
    double* rr = net->terms.get() + first;
    double* eAe = net->terms.get() + batch + first;
    double* dAd = net->terms.get() + 2 * batch + first;
    const int* gro = net->gro.get();
    const int* gco = net->gco.get();
    const float* gew = net->gew.get();
    const float* P = net->params.get();
    const int sum_blocks = std::min(reduce_blocks(n), kPairBlocks);
    const dim3 pair_grid(static_cast<unsigned>(sum_blocks), static_cast<unsigned>(pairs));
    k_pair_norms<<<pair_grid, kReduceThreads, 0, s>>>(n, r, net->sums.get(), net->tickets.get(), rr);
    check_launch(ctx);
    k_encode<<<blocks_for(8 * static_cast<int64_t>(cells), 256), 256, 0, s>>>(n, cells, r, rr, net->feats.get(), P,
                                                                              net->H.get());
    check_launch(ctx);
    const int tiles = (cells + kTrainTile - 1) / kTrainTile;
    const int fwd_blocks = std::min(tiles, 6 * ctx->sm_count);   // six blocks of 36 KB per SM
    for (int k = 0; k < R; ++k) {
        k_round_fwd<<<fwd_blocks, kThreads, 0, s>>>(n, cells, gro, gco, gew, net->H.get() + k * st,
                                                    P + ROUND0 + k * ROUND_SIZE, net->AG.get() + k * st,
                                                    net->Z.get() + k * st, net->H.get() + (k + 1) * st);
        check_launch(ctx);
    }
    k_readout<<<blocks_for(8 * static_cast<int64_t>(cells), 256), 256, 0, s>>>(n, cells, net->H.get() + R * st, P, rr,
                                                                               net->diag.get(), net->outb.get());
    check_launch(ctx);
    if (!net->vcycle) {
        k_pair_energies<<<pair_grid, kReduceThreads, 0, s>>>(n, net->A->ro.get(), net->A->co.get(), net->A->va.get(),
                                                             e, net->outb.get(), net->Ad.get(), net->sums.get(),
                                                             net->tickets.get(), eAe, dAd);
        check_launch(ctx);
    } else {
        for (int p = 0; p < pairs; ++p) {
            const double* ep = e + static_cast<size_t>(p) * n;
            double* Ad = net->Ad.get() + static_cast<size_t>(p) * n;
            k_sub<<<blocks_for(n, 256), 256, 0, s>>>(n, ep, net->outb.get() + static_cast<size_t>(p) * n,
                                                     net->t.get());
            check_launch(ctx);
            spmv_fp64(ctx, net->A, net->t.get(), Ad);
            spmv_fp64(ctx, net->A, ep, net->Ae.get());
            // w1 = E d, w2 = E w1 (E = I - M A); gradient direction A w2; scale by ||E e||_A^2
            amg_apply_device(ctx, net->vcycle, Ad, net->q.get());
            k_sub<<<blocks_for(n, 256), 256, 0, s>>>(n, net->t.get(), net->q.get(), net->w1.get());
            check_launch(ctx);
            spmv_fp64(ctx, net->A, net->w1.get(), Ad);            // A w1
            enqueue_dot(ctx, n, net->w1.get(), Ad, dAd + p);
            amg_apply_device(ctx, net->vcycle, Ad, net->q.get());
            k_sub<<<blocks_for(n, 256), 256, 0, s>>>(n, net->w1.get(), net->q.get(), net->w2.get());
            check_launch(ctx);
            spmv_fp64(ctx, net->A, net->w2.get(), Ad);            // A w2
            amg_apply_device(ctx, net->vcycle, net->Ae.get(), net->q.get());  // M A e
            k_sub<<<blocks_for(n, 256), 256, 0, s>>>(n, ep, net->q.get(), net->w1.get());   // E e
            check_launch(ctx);
            spmv_fp64(ctx, net->A, net->w1.get(), net->Ae.get());
            enqueue_dot(ctx, n, net->w1.get(), net->Ae.get(), eAe + p);
        }
    }
    k_dy<<<blocks_for(cells, 256), 256, 0, s>>>(n, cells, net->Ad.get(), eAe, rr, net->diag.get(), net->dyf.get());
    check_launch(ctx);
    k_readout_bwd<<<kGridBlocks, kThreads, 0, s>>>(cells, net->H.get() + R * st, net->dyf.get(), P, net->dh.get(),
                                                   net->partial.get());
    check_launch(ctx);
    const int bwd_blocks = std::min(tiles, kGridBlocks);
    const float* da_in = nullptr;
    float* da = net->da.get();
    float* da_next = net->da2.get();
    for (int k = R - 1; k >= 0; --k) {
        k_round_bwd<<<bwd_blocks, kThreads, 0, s>>>(n, cells, gro, gco, gew, net->H.get() + k * st,
                                                    net->AG.get() + k * st, net->Z.get() + k * st,
                                                    P + ROUND0 + k * ROUND_SIZE, da_in, net->dh.get(), da,
                                                    net->partial.get(), ROUND0 + k * ROUND_SIZE);
        check_launch(ctx);
        da_in = da;
        std::swap(da, da_next);
    }
    k_encode_bwd<<<kGridBlocks, kThreads, 0, s>>>(n, cells, gro, gco, gew, r, rr, net->feats.get(), net->H.get(),
                                                  net->dh.get(), da_in, net->partial.get());
    check_launch(ctx);
}

double loss_grad_batch(cfdxg_context* ctx, cfdxg_mpnn* net, const double* r, const double* e, int batch) {
    require_bound(net);
    if (net->vcycle && net->vcycle->host.levels.front().A.n != net->n)
        throw Error(CFDXG_ERR_INVALID_ARGUMENT, "training V-cycle and bound matrix differ in size");
    const int n = net->n;
    const int together = static_cast<int>(std::min<int64_t>({batch, kMaxPairs, std::max<int64_t>(1, kTrainCells / n)}));
    const size_t cells = static_cast<size_t>(together) * n, st = cells * F;
    grow(net->H, st * (R + 1));
    grow(net->AG, st * R);
    grow(net->Z, st * R);
    grow(net->dh, st);
    grow(net->da, st);
    grow(net->da2, st);
    grow(net->dyf, cells);
    grow(net->outb, cells);
    grow(net->Ad, cells);
    if (net->vcycle) {
        grow(net->Ae, static_cast<size_t>(n));
        grow(net->w1, static_cast<size_t>(n));
        grow(net->w2, static_cast<size_t>(n));
        grow(net->q, static_cast<size_t>(n));
    }
    grow(net->terms, 3 * static_cast<size_t>(batch));
    grow(net->sums, static_cast<size_t>(2 * kPairBlocks) * kMaxPairs);
    if (net->tickets.size() == 0) {
        net->tickets.resize(kMaxPairs);
        net->tickets.zero(ctx->stream);
    }
    net->partial.resize(static_cast<size_t>(kGridBlocks) * NP);
    net->partial.zero(ctx->stream);
    net->grad.resize(NP);
    for (int b = 0; b < batch; b += together)
        loss_grad_pairs(ctx, net, r + static_cast<size_t>(b) * n, e + static_cast<size_t>(b) * n, b,
                        std::min(together, batch - b), batch);
    k_reduce_partials<<<blocks_for(NP, 32), 256, 0, ctx->stream>>>(net->partial.get(), kGridBlocks,
                                                                   1.0f / static_cast<float>(batch), net->grad.get());
    check_launch(ctx);
    std::vector<double> h(2 * static_cast<size_t>(batch));
    CFDXG_CUDA(cudaMemcpyAsync(h.data(), net->terms.get() + batch, sizeof(double) * h.size(), cudaMemcpyDeviceToHost,
                               ctx->stream));
    CFDXG_CUDA(cudaStreamSynchronize(ctx->stream));
    double total = 0.0;
    for (int b = 0; b < batch; ++b) total += h[static_cast<size_t>(batch) + b] / h[b];
    return total / batch;
}

uint64_t fnv1a(const void* data, size_t bytes) {
    const auto* p = static_cast<const unsigned char*>(data);
    uint64_t h = 1469598103934665603ull;
    for (size_t i = 0; i < bytes; ++i) {
        h ^= p[i];
        h *= 1099511628211ull;
    }
    return h;
}

}  // namespace

void bind_learned_to_matrix(cfdxg_context*, cfdxg_mpnn* net, const cfdxg_matrix* A) {
    if (!net->A || net->A != A)
        throw Error(CFDXG_ERR_NOT_READY, "the learned network is not bound to this matrix (cfdxg_mpnn_bind)");
}

bool learned_then_amg(cfdxg_context* ctx, cfdxg_mpnn* net, const cfdxg_matrix* A, const double* v, double* z,
                      const std::function<void(const double*, double*)>& amg, int64_t*) {
    const int n = net->n;
    cudaStream_t s = ctx->stream;
    infer(ctx, net, v, net->y.get());
    k_residual64<<<blocks_for(n, 256), 256, 0, s>>>(n, A->ro.get(), A->co.get(), A->va.get(), v, net->y.get(),
                                                     net->t.get());
    check_launch(ctx);
    amg(net->t.get(), z);
    k_add_inplace<<<blocks_for(n, 256), 256, 0, s>>>(n, z, net->y.get());
    check_launch(ctx);
    return true;
}

}  // namespace cfdxg

using namespace cfdxg;

extern "C" int cfdxg_mpnn_create(cfdxg_context* ctx, uint64_t seed, cfdxg_mpnn** out) {
    if (!ctx || !out) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    auto net = std::make_unique<cfdxg_mpnn>();
    net->host.assign(mp::NP, 0.0f);
    std::mt19937_64 g(seed);
    std::normal_distribution<double> nd(0.0, 1.0);
    auto fill = [&](int off, int rows, int cols) {
        const double sc = std::sqrt(1.0 / cols);
        for (int q = 0; q < rows * cols; ++q) net->host[off + q] = static_cast<float>(nd(g) * sc);
    };
    fill(mp::OFF_WIN, mp::F, 4);
    for (int k = 0; k < mp::R; ++k) {
        fill(mp::ROUND0 + k * mp::ROUND_SIZE + mp::OFF_W1, mp::F, 2 * mp::F);
        fill(mp::ROUND0 + k * mp::ROUND_SIZE + mp::OFF_W2, mp::F, mp::F);
    }
    for (int q = 0; q < mp::F; ++q) net->host[mp::OFF_WOUT + q] = static_cast<float>(0.1 * nd(g));
    net->adam_m.resize(mp::NP);
    net->adam_v.resize(mp::NP);
    net->adam_m.zero(ctx->stream);
    net->adam_v.zero(ctx->stream);
    upload_params(ctx, net.get());
    *out = net.release();
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}

extern "C" int cfdxg_mpnn_destroy(cfdxg_mpnn* net) {
    delete net;
    return CFDXG_OK;
}

extern "C" int cfdxg_mpnn_num_parameters(const cfdxg_mpnn* net, int64_t* count) {
    if (!net || !count) return CFDXG_ERR_INVALID_ARGUMENT;
    *count = mp::NP;
    return CFDXG_OK;
}

extern "C" int cfdxg_mpnn_get_parameters(cfdxg_context* ctx, const cfdxg_mpnn* net, float* params) {
    if (!ctx || !net || !params) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    net->params.download(params, ctx->stream);
    CFDXG_CUDA(cudaStreamSynchronize(ctx->stream));
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}

extern "C" int cfdxg_mpnn_set_parameters(cfdxg_context* ctx, cfdxg_mpnn* net, const float* params) {
    if (!ctx || !net || !params) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    net->host.assign(params, params + mp::NP);
    upload_params(ctx, net);
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}

extern "C" int cfdxg_mpnn_save(cfdxg_context* ctx, const cfdxg_mpnn* net, const char* path) {
    if (!ctx || !net || !path) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    std::vector<float> p(mp::NP);
    net->params.download(p.data(), ctx->stream);
    CFDXG_CUDA(cudaStreamSynchronize(ctx->stream));
    FILE* f = std::fopen(path, "wb");
    if (!f) throw Error(CFDXG_ERR_IO, std::string("cannot open ") + path);
    const char magic[8] = {'C', 'F', 'D', 'X', 'M', 'P', 'N', 'N'};
    const uint32_t version = 1, count = mp::NP;
    const uint64_t sum = fnv1a(p.data(), p.size() * sizeof(float));
    bool ok = std::fwrite(magic, 1, 8, f) == 8 && std::fwrite(&version, 4, 1, f) == 1 &&
              std::fwrite(&count, 4, 1, f) == 1 && std::fwrite(p.data(), sizeof(float), p.size(), f) == p.size() &&
              std::fwrite(&sum, 8, 1, f) == 1;
    ok = (std::fclose(f) == 0) && ok;
    if (!ok) throw Error(CFDXG_ERR_IO, std::string("cannot write ") + path);
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}

extern "C" int cfdxg_mpnn_load(cfdxg_context* ctx, cfdxg_mpnn* net, const char* path) {
    if (!ctx || !net || !path) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    FILE* f = std::fopen(path, "rb");
    if (!f) throw Error(CFDXG_ERR_IO, std::string("cannot open ") + path);
    char magic[8];
    uint32_t version = 0, count = 0;
    uint64_t sum = 0;
    std::vector<float> p(mp::NP);
    const bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, "CFDXMPNN", 8) == 0 &&
                    std::fread(&version, 4, 1, f) == 1 && version == 1 && std::fread(&count, 4, 1, f) == 1 &&
                    count == static_cast<uint32_t>(mp::NP) &&
                    std::fread(p.data(), sizeof(float), p.size(), f) == p.size() && std::fread(&sum, 8, 1, f) == 1;
    std::fclose(f);
    if (!ok) throw Error(CFDXG_ERR_IO, std::string("not a network weight file: ") + path);
    if (sum != fnv1a(p.data(), p.size() * sizeof(float))) throw Error(CFDXG_ERR_IO, "weight file checksum mismatch");
    net->host = p;
    upload_params(ctx, net);
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}

extern "C" int cfdxg_mpnn_bind(cfdxg_context* ctx, cfdxg_mpnn* net, cfdxg_mesh* mesh, const cfdxg_matrix* A,
                               const double* a_P, int32_t mem) {
    if (!ctx || !net || !mesh || !A || !a_P) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    check_mem_flag(mem);
    if (!mesh->geometry_ready) throw Error(CFDXG_ERR_NOT_READY, "geometry not built");
    if (A->n != mesh->n_cells) throw Error(CFDXG_ERR_INVALID_ARGUMENT, "matrix and mesh sizes differ");
    // inference addresses the state with 32-bit row offsets (n * F / 4 quarter-rows)
    if (A->n > std::numeric_limits<int>::max() / mp::F)
        throw Error(CFDXG_ERR_INVALID_ARGUMENT, "mesh too large for the learned stage");
    auto* M = const_cast<cfdxg_matrix*>(A);
    matrix_sync_host_values(ctx, M);
    const int64_t n = A->n;
    const HostCsr& H = M->host;
    // per-row work on the host threads (every value is formed as before; only
    // the sums of the feature standardisation stay sequential, in row order)
    const auto rows = [n](auto&& fn) {
        const int workers = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(host_threads(), n / 65536)));
        if (workers <= 1) { fn(int64_t(0), n); return; }
        std::vector<std::thread> pool;
        for (int w = 0; w < workers; ++w) pool.emplace_back([&fn, n, w, workers] { fn(n * w / workers, n * (w + 1) / workers); });
        for (auto& t : pool) t.join();
    };
    std::vector<double> diag(n, 0.0), vol(n), ap(n);
    std::atomic<bool> bad_diag{false}, asymmetric{false}, bad_cell{false};
    rows([&](int64_t b, int64_t e) {
        for (int64_t i = b; i < e; ++i) {
            for (uint32_t k = H.ro[i]; k < H.ro[i + 1]; ++k)
                if (H.co[k] == i) diag[i] = H.va[k];
            if (!(diag[i] > 0.0)) bad_diag = true;
        }
    });
    if (bad_diag) throw Error(CFDXG_ERR_INVALID_ARGUMENT, "the learned preconditioner needs a positive diagonal");
    // symmetric couplings are required (the backward pass gathers over the same graph)
    std::vector<float> ew(H.co.size(), 0.0f);
    std::vector<int> gro(n + 1, 0);
    rows([&](int64_t b, int64_t e) {
        for (int64_t i = b; i < e; ++i) {
            int off = 0;
            for (uint32_t k = H.ro[i]; k < H.ro[i + 1]; ++k) {
                const uint32_t j = H.co[k];
                if (j == i) continue;
                ++off;
                const uint32_t* lo = H.co.data() + H.ro[j];
                const uint32_t* hi = H.co.data() + H.ro[j + 1];
                const uint32_t* it = std::lower_bound(lo, hi, static_cast<uint32_t>(i));
                if (it == hi || *it != i || H.va[it - H.co.data()] != H.va[k]) {
                    asymmetric = true;
                    return;
                }
                ew[k] = static_cast<float>(-H.va[k] / std::sqrt(diag[i] * diag[j]));
            }
            gro[i + 1] = off;
        }
    });
    if (asymmetric) throw Error(CFDXG_ERR_INVALID_ARGUMENT, "the learned preconditioner needs a symmetric matrix");
    mesh->cell_volume.download(vol.data(), ctx->stream);
    if (mem == CFDXG_MEM_DEVICE) CFDXG_CUDA(cudaMemcpyAsync(ap.data(), a_P, n * sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    else std::memcpy(ap.data(), a_P, n * sizeof(double));
    CFDXG_CUDA(cudaStreamSynchronize(ctx->stream));
    std::vector<float> feats(3 * n);
    std::vector<double> logs(n);
    const auto standardise = [&](const std::vector<double>& v, int slot) {
        rows([&](int64_t b, int64_t e) { for (int64_t i = b; i < e; ++i) logs[i] = std::log(v[i]); });
        double mean = 0.0, sq = 0.0;
        for (int64_t i = 0; i < n; ++i) mean += logs[i];
        mean /= n;
        for (int64_t i = 0; i < n; ++i) sq += (logs[i] - mean) * (logs[i] - mean);
        // On a uniform mesh the logarithms differ by rounding alone (some 1e-15,
        // more on finer lattices), which a division by its own deviation would
        // turn into inputs of size one: a constant is left at its distance from
        // the mean, next to zero.
        const double deviation = std::sqrt(sq / n);
        const double sd = deviation > 1e-12 * std::max(1.0, std::abs(mean)) ? deviation : 1.0;
        rows([&](int64_t b, int64_t e) {
            for (int64_t i = b; i < e; ++i)
                feats[slot * n + i] = static_cast<float>((logs[i] - mean) / sd);
        });
    };
    rows([&](int64_t b, int64_t e) {
        for (int64_t i = b; i < e; ++i)
            if (!(vol[i] > 0.0) || !(ap[i] > 0.0)) bad_cell = true;
    });
    if (bad_cell) throw Error(CFDXG_ERR_INVALID_ARGUMENT, "volumes and a_P must be positive");
    standardise(vol, 0);
    standardise(ap, 1);
    standardise(diag, 2);
    // the coupling list without the diagonal: row offsets by a prefix sum, then rows in parallel
    for (int64_t i = 0; i < n; ++i) gro[i + 1] += gro[i];
    std::vector<int> gco(static_cast<std::size_t>(gro[n]));
    std::vector<float> gew(static_cast<std::size_t>(gro[n]));
    rows([&](int64_t b, int64_t e) {
        for (int64_t i = b; i < e; ++i) {
            int o = gro[i];
            for (uint32_t k = H.ro[i]; k < H.ro[i + 1]; ++k)
                if (H.co[k] != i) {
                    gco[o] = static_cast<int>(H.co[k]);
                    gew[o] = ew[k];
                    ++o;
                }
        }
    });
    net->gro.upload(gro, ctx->stream);
    net->gco.upload(gco, ctx->stream);
    net->gew.upload(gew, ctx->stream);
    net->feats.upload(feats, ctx->stream);
    net->diag.upload(diag, ctx->stream);
    const size_t st = static_cast<size_t>(n) * mp::F;
    net->hA.resize(st); net->hB.resize(st);
    net->y.resize(n); net->t.resize(n);
    CFDXG_CUDA(cudaStreamSynchronize(ctx->stream));
    net->A = A;
    net->n = static_cast<int>(n);
    ctx->error.clear();
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}

extern "C" int cfdxg_mpnn_set_vcycle(cfdxg_context* ctx, cfdxg_mpnn* net, cfdxg_amg* amg) {
    if (!ctx || !net) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    if (amg && (!amg->ready || (!amg->d64 && !amg->d32)))
        throw Error(CFDXG_ERR_NOT_READY, "the V-cycle is not set up on the device");
    net->vcycle = amg;
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}

extern "C" int cfdxg_mpnn_apply(cfdxg_context* ctx, cfdxg_mpnn* net, const double* r, double* y, int32_t mem) {
    if (!ctx || !net || !r || !y) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    NvtxRange nvtx_range("cfdxg.mpnn_apply");
    check_mem_flag(mem);
    require_bound(net);
    In<double> rin(ctx, r, net->n, mem);
    Out<double> yo(ctx, y, net->n, mem);
    infer(ctx, net, rin.get(), yo.get());
    yo.finish();
    CFDXG_CUDA(cudaStreamSynchronize(ctx->stream));
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}

extern "C" int cfdxg_mpnn_loss_grad(cfdxg_context* ctx, cfdxg_mpnn* net, const double* r, const double* e,
                                    int32_t batch, int32_t mem, double* loss, float* grad) {
    if (!ctx || !net || !r || !e || batch <= 0) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    check_mem_flag(mem);
    require_bound(net);
    const int64_t total = static_cast<int64_t>(batch) * net->n;
    In<double> rin(ctx, r, total, mem), ein(ctx, e, total, mem);
    const double L = loss_grad_batch(ctx, net, rin.get(), ein.get(), batch);
    if (loss) *loss = L;
    if (grad) net->grad.download(grad, ctx->stream);
    CFDXG_CUDA(cudaStreamSynchronize(ctx->stream));
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}

extern "C" int cfdxg_mpnn_train_step(cfdxg_context* ctx, cfdxg_mpnn* net, const double* r, const double* e,
                                     int32_t batch, float lr, int32_t mem, double* loss) {
    if (!ctx || !net || !r || !e || batch <= 0 || !(lr > 0.0f)) return CFDXG_ERR_INVALID_ARGUMENT;
    CFDXG_GUARD_BEGIN
    check_mem_flag(mem);
    require_bound(net);
    const int64_t total = static_cast<int64_t>(batch) * net->n;
    In<double> rin(ctx, r, total, mem), ein(ctx, e, total, mem);
    const double L = loss_grad_batch(ctx, net, rin.get(), ein.get(), batch);
    ++net->steps;
    const float bc1 = 1.0f - std::pow(0.9f, static_cast<float>(net->steps));
    const float bc2 = 1.0f - std::pow(0.999f, static_cast<float>(net->steps));
    k_adam<<<blocks_for(mp::NP, 256), 256, 0, ctx->stream>>>(net->params.get(), net->grad.get(), net->adam_m.get(),
                                                             net->adam_v.get(), lr, bc1, bc2);
    check_launch(ctx);
    k_to_bf16<<<blocks_for(mp::R * 3 * mp::F * mp::F, 256), 256, 0, ctx->stream>>>(net->params.get(), net->wbf.get());
    check_launch(ctx);
    CFDXG_CUDA(cudaStreamSynchronize(ctx->stream));
    if (loss) *loss = L;
    return CFDXG_OK;
    CFDXG_GUARD_END(ctx)
}
