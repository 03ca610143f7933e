// Orthogonalisation step of the per-column GMRES (FP64) for small vectors, one launch: the new
// direction W against the basis V_0 .. V_j of each column's own Krylov space by classical Gram-Schmidt
// (once or twice), its norm, the next basis vector and the Givens update of the least-squares
// problem. Multi-column vectors are node-major (n x k). A step on small vectors costs its launches and
// their tails, not its bytes, so one cluster of 8 CTAs does all of it: W stays in shared memory, the
// CTAs' partial dot products are summed through distributed shared memory.
#pragma once
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace bie {

// Per-column least-squares state of a GMRES cycle. R: [(m+1) x (m+1) x k], column j holds the rotated
// Hessenberg column; cs/sn: [m x k]; gv: [(m+1) x k].
struct Givens {
    double *R, *cs, *sn, *gv;
    int *active, *jlast;
    const double* eps;
    double* resid;
    int m1, k;
};

// Givens step j of column c: Hessenberg column h + h2 (h2 may be null; stride ldh between entries),
// norm of the new direction hn. Retires the column when its residual reaches its tolerance.
__device__ __forceinline__ void givens_column(const Givens& G, int c, const double* h, const double* h2, int ldh,
                                              double hn, int j) {
    if (!G.active[c]) return;
    const int k = G.k;
    double* Rj = G.R + (int64_t)j * G.m1 * k + c;
    double t = h[0] + (h2 ? h2[0] : 0.0);
    for (int i0 = 0; i0 < j; i0 += 8) {
        double b[8], ci[8], si[8];  // loaded ahead of the chain of rotations
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int i = min(i0 + u, j - 1);
            b[u] = h[(i + 1) * ldh] + (h2 ? h2[(i + 1) * ldh] : 0.0);
            ci[u] = G.cs[i * k + c];
            si[u] = G.sn[i * k + c];
        }
#pragma unroll
        for (int u = 0; u < 8; ++u)
            if (i0 + u < j) {
                Rj[(int64_t)(i0 + u) * k] = ci[u] * t + si[u] * b[u];
                t = -si[u] * t + ci[u] * b[u];
            }
    }
    const double r = hypot(t, hn);
    const double cj = r > 0 ? t / r : 1.0, sj = r > 0 ? hn / r : 0.0;
    G.cs[j * k + c] = cj;
    G.sn[j * k + c] = sj;
    Rj[(int64_t)j * k] = r;
    Rj[(int64_t)(j + 1) * k] = 0.0;
    const double gj = G.gv[j * k + c];
    G.gv[(j + 1) * k + c] = -sj * gj;
    G.gv[j * k + c] = cj * gj;
    const double res = fabs(sj * gj);
    G.resid[c] = res;
    G.jlast[c] = j + 1;
    if (res <= G.eps[c] || hn == 0.0) G.active[c] = 0;
}

// ---------------------------------------------------------------------------
// CTA r owns rows [r rpc, (r + 1) rpc); warps take (vector, column, row part) items of the dot
// products, threads take elements of the updates.
// ---------------------------------------------------------------------------
constexpr int kArnCtas = 8, kArnThreads = 1024;
// Largest n k and k. Whole solves, one launch a pass against the cluster: 2,560 nodes, 1 column, FP64
// 1.35 and 1.14 ms; 23,040 nodes, 1 column, FP32 4.38 and 4.38 ms; 2,048 nodes, 16 columns 1.63 and 1.93.
constexpr int64_t kArnElems = 8192;
constexpr int kArnCols = 8;

// Row parts of each dot product, so that all 32 warps have one.
__host__ __device__ inline int arn_parts(int pairs) { return pairs >= 32 ? 1 : 32 / pairs; }
// Shared memory: own rows of W, coefficients of both passes, the CTA's sums of both passes and the norm,
// the warps' sums.
inline size_t arn_smem(int64_t n, int k, int nv) {
    const int64_t rpc = (n + kArnCtas - 1) / kArnCtas, pairs = (int64_t)nv * k;
    return sizeof(double) * (size_t)(rpc * k + 4 * pairs + 2 * k + pairs + 32);
}

__global__ void __cluster_dims__(kArnCtas, 1, 1) __launch_bounds__(kArnThreads)
    k_arnoldi_cluster(const double* __restrict__ W, double* __restrict__ V, int64_t strideV, int j, int64_t n, int passes,
                      Givens G) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ double arn[];
    const int k = G.k, nv = j + 1, pairs = nv * k;
    const int rank = (int)cl.block_rank();
    const int64_t rpc = (n + kArnCtas - 1) / kArnCtas;
    const int64_t r0 = min(n, rank * rpc);
    const int rows = (int)(min(n, r0 + rpc) - r0), elems = rows * k;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = kArnThreads / 32;
    double* w = arn;               // [rows][k]
    double* hs = w + rpc * k;      // [2][pairs]
    double* own = hs + 2 * pairs;  // [2][pairs] and [k], read by the other CTAs
    double* hn = own + 2 * pairs + k;  // [k]
    double* part = hn + k;         // warps' sums: [pairs][parts]
    const double* Vr = V + r0 * k;
    for (int e = threadIdx.x; e < elems; e += kArnThreads) w[e] = W[r0 * k + e];
    __syncthreads();
    // to[q], q < m: this CTA's sums of A_v[i][c] w[i][c], q = v k + c (A null: w itself), m = items
    auto own_sums = [&](const double* A, int m, double* to) {
        const int parts = arn_parts(m);
        for (int it = warp; it < m * parts; it += nwarp) {
            const int q = it / parts, s = it - q * parts, v = q / k, c = q - v * k;
            const double* a = A ? A + (int64_t)v * strideV + c : w + c;
            double acc = 0.0;
#pragma unroll 8
            for (int r = s * 32 + lane; r < rows; r += 32 * parts) acc = fma(a[(int64_t)r * k], w[r * k + c], acc);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, o);
            if (lane == 0) part[it] = acc;
        }
        __syncthreads();
        for (int q = threadIdx.x; q < m; q += kArnThreads) {
            double acc = 0.0;
            for (int s = 0; s < parts; ++s) acc += part[q * parts + s];
            to[q] = acc;
        }
    };
    // sum of entry q of every CTA's `from`
    auto all_sum = [&](double* from, int q) {
        double a[kArnCtas];
#pragma unroll
        for (int r = 0; r < kArnCtas; ++r) a[r] = cl.map_shared_rank(from, r)[q];
        double acc = 0.0;
#pragma unroll
        for (int r = 0; r < kArnCtas; ++r) acc += a[r];
        return acc;
    };
    for (int p = 0; p < passes; ++p) {
        double* hp = hs + p * pairs;
        own_sums(Vr, pairs, own + p * pairs);
        cl.sync();
        for (int q = threadIdx.x; q < pairs; q += kArnThreads) hp[q] = all_sum(own + p * pairs, q);
        __syncthreads();
        for (int e = threadIdx.x; e < elems; e += kArnThreads) {
            const int c = e % k;
            double x = w[e];
#pragma unroll 8
            for (int v = 0; v < nv; ++v) x = fma(-Vr[(int64_t)v * strideV + e], hp[v * k + c], x);
            w[e] = x;
        }
        __syncthreads();
    }
    own_sums(nullptr, k, own + 2 * pairs);
    cl.sync();
    if (threadIdx.x < (unsigned)k) hn[threadIdx.x] = sqrt(all_sum(own + 2 * pairs, threadIdx.x));
    __syncthreads();
    double* Vn = V + (int64_t)nv * strideV + r0 * k;
    for (int e = threadIdx.x; e < elems; e += kArnThreads) {
        const double d = hn[e % k];
        Vn[e] = d > 0.0 ? w[e] / d : 0.0;
    }
    if (rank == 0 && threadIdx.x < (unsigned)k)
        givens_column(G, threadIdx.x, hs + threadIdx.x, passes > 1 ? hs + pairs + threadIdx.x : nullptr, k,
                      hn[threadIdx.x], j);
    cl.sync();  // no CTA leaves while another may still read its partial sums
}

}  // namespace bie
