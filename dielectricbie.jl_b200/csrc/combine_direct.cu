// K4 for panels of 4 x 4 and 6 x 6 nodes: the block-row correction apply with its operands loaded
// straight into the fragments of mma.sync.m8n8k4.f64.
//
//   Y[i][c] = (1/4pi) sum_s part[s][i][c] + sum_b (C_b (p X)[col_b])[i][c] + t_i p_i X[i][c]
//
// (the CSC SpMV / sparse mat-mat of laplace3d_DT_fmm3d_corrected and
// BatchedDielectricOperator, src/kernel/laplace3d_near.jl:395-419,
// src/solver/multi_rhs.jl:103-136, fused with the reduction of the direct-sum split
// partials and the diagonal term).
//
// One CTA per (target panel, 8 NT columns); its W warps take the row's blocks in turn. A fragment is 8
// rows of 4 block columns (64-byte pieces of the column-major block), B 4 source nodes by 8 columns: every
// byte of a block is used once by the warp that loads it, so staging it in shared memory gains
// nothing, and a warp has all loads of a block (45 + 9 NT a lane at 36 nodes) in flight at once. The warps'
// sums meet in shared memory; the split partials are loaded ahead of the blocks.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "solver.h"

namespace bie {
namespace {

__device__ __forceinline__ void dmma_cd(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// Warps of a CTA: a row of 16-node panels has about 50 blocks, one of 36-node panels about 7.
template <int NB, int NT> __host__ __device__ constexpr int cd_warps() { return NB == 16 ? (NT <= 2 ? 16 : 8) : (NT <= 2 ? 8 : 4); }
template <int NB, int NT> constexpr size_t cd_smem() {
    return sizeof(double) * cd_warps<NB, NT>() * ((NB + 7) / 8) * NT * 2 * 32;
}

template <int NB, int NT, typename TP>
__global__ void __launch_bounds__(32 * cd_warps<NB, NT>())
    k_combine_direct(int64_t n, int k, const TP* __restrict__ part, int nsplit, const double* __restrict__ X,
                     const double* __restrict__ pre, const double* __restrict__ diag,
                     const int32_t* __restrict__ rowptr, const int32_t* __restrict__ col,
                     const double* __restrict__ val, double* __restrict__ Y) {
    constexpr int W = cd_warps<NB, NT>(), MT = (NB + 7) / 8, KS = NB / 4;
    constexpr int OUT = (NB * 8 * NT + 32 * W - 1) / (32 * W);  // outputs a thread
    extern __shared__ double red[];                             // [W][MT][NT][2][32]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    const int c0 = blockIdx.y * 8 * NT, kt = min(8 * NT, k - c0);
    const int64_t row0 = (int64_t)blockIdx.x * NB, tot = n * (int64_t)k;
    const int b0 = val ? rowptr[blockIdx.x] : 0, b1 = val ? rowptr[blockIdx.x + 1] : 0;
    // output o of the thread: row e / kt, column c0 + e % kt of the panel, e = tid + o 32 W
    double sp[OUT];
#pragma unroll
    for (int o = 0; o < OUT; ++o) {
        const int e = threadIdx.x + o * 32 * W;
        sp[o] = 0.0;
        if (e < NB * kt) {
            const TP* p = part + (row0 + e / kt) * k + c0 + e % kt;
#pragma unroll 4
            for (int s = 0; s < nsplit; ++s) sp[o] += (double)p[(int64_t)s * tot];
        }
    }
    double acc[MT][NT][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) acc[m][t][0] = acc[m][t][1] = 0.0;
    for (int b = b0 + warp; b < b1; b += W) {
        const double* vb = val + (int64_t)b * NB * NB + q * NB + r;
        const int64_t src = (int64_t)col[b] * NB + q;
        const double* xb = X + src * k + c0 + r;
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
            double a[MT], x[NT];
#pragma unroll
            for (int m = 0; m < MT; ++m) a[m] = 8 * m + r < NB ? vb[4 * ks * NB + 8 * m] : 0.0;
#pragma unroll
            for (int t = 0; t < NT; ++t) x[t] = 8 * t + r < kt ? xb[(int64_t)(4 * ks) * k + 8 * t] : 0.0;
            if (pre) {
                const double p = pre[src + 4 * ks];
#pragma unroll
                for (int t = 0; t < NT; ++t) x[t] *= p;
            }
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int t = 0; t < NT; ++t) dmma_cd(acc[m][t][0], acc[m][t][1], a[m], x[t]);
        }
    }
    double* mine = red + (size_t)warp * MT * NT * 64 + lane;
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            mine[((m * NT + t) * 2 + 0) * 32] = acc[m][t][0];
            mine[((m * NT + t) * 2 + 1) * 32] = acc[m][t][1];
        }
    __syncthreads();
#pragma unroll
    for (int o = 0; o < OUT; ++o) {
        const int e = threadIdx.x + o * 32 * W;
        if (e < NB * kt) {
            const int rr = e / kt, cc = e % kt;
            // D fragment: lane 4 (row % 8) + (column % 8) / 2, register column % 2
            const double* f = red + (((rr >> 3) * NT + (cc >> 3)) * 2 + (cc & 1)) * 32 + (rr & 7) * 4 + ((cc & 7) >> 1);
            double y = 0.0;
#pragma unroll
            for (int w = 0; w < W; ++w) y += f[(size_t)w * MT * NT * 64];
            const int64_t i = row0 + rr, idx = i * k + c0 + cc;
            y += sp[o] * kInv4Pi;
            if (diag) y += diag[i] * (pre ? pre[i] : 1.0) * X[idx];
            Y[idx] = y;
        }
    }
}

template <int NB, int NT, typename TP>
void launch_cd(int64_t n, int k, int npanels, const TP* part, int nsplit, const double* X, const double* pre,
               const double* diag, const int32_t* rowptr, const int32_t* col, const double* val, double* Y,
               cudaStream_t s) {
    const auto f = k_combine_direct<NB, NT, TP>;
    ensure_smem_limit((const void*)f, cd_smem<NB, NT>());
    const dim3 grid((unsigned)npanels, (unsigned)((k + 8 * NT - 1) / (8 * NT)));
    f<<<grid, 32 * cd_warps<NB, NT>(), cd_smem<NB, NT>(), s>>>(n, k, part, nsplit, X, pre, diag, rowptr, col, val, Y);
}

template <int NB, typename TP>
void launch_nb(int64_t n, int k, int npanels, const TP* part, int nsplit, const double* X, const double* pre,
               const double* diag, const int32_t* rowptr, const int32_t* col, const double* val, double* Y,
               cudaStream_t s) {
    if (k <= 8)
        launch_cd<NB, 1, TP>(n, k, npanels, part, nsplit, X, pre, diag, rowptr, col, val, Y, s);
    else if (k <= 16)
        launch_cd<NB, 2, TP>(n, k, npanels, part, nsplit, X, pre, diag, rowptr, col, val, Y, s);
    else if (k <= 24)
        launch_cd<NB, 3, TP>(n, k, npanels, part, nsplit, X, pre, diag, rowptr, col, val, Y, s);
    else if constexpr (NB == 16)
        launch_cd<NB, 4, TP>(n, k, npanels, part, nsplit, X, pre, diag, rowptr, col, val, Y, s);
}

}  // namespace

template <typename TP>
bool launch_combine_direct(int64_t n, int k, int nb, int npanels, const TP* part, int nsplit, const double* X,
                           const double* pre, const double* diag, const int32_t* rowptr, const int32_t* col,
                           const double* val, double* Y, cudaStream_t s) {
    if (nb != 16 && (nb != 36 || k > 24)) return false;
    if (nb == 16)
        launch_nb<16, TP>(n, k, npanels, part, nsplit, X, pre, diag, rowptr, col, val, Y, s);
    else
        launch_nb<36, TP>(n, k, npanels, part, nsplit, X, pre, diag, rowptr, col, val, Y, s);
    BIE_CK(cudaGetLastError());
    return true;
}

template bool launch_combine_direct<float>(int64_t, int, int, int, const float*, int, const double*, const double*,
                                           const double*, const int32_t*, const int32_t*, const double*, double*,
                                           cudaStream_t);
template bool launch_combine_direct<double>(int64_t, int, int, int, const double*, int, const double*, const double*,
                                            const double*, const int32_t*, const int32_t*, const double*, double*,
                                            cudaStream_t);

}  // namespace bie
