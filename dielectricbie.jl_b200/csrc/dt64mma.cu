// K1 for k >= 8 right-hand sides: FP64 direct D^T sum whose RHS contraction runs
// on the FP64 tensor-core path (mma.sync m8n8k4 f64), the plain path of the
// solver (FP64 end to end).
//
//   part[s][i][c0 + c] = sum_{j in split s, j != i} n_i.(x_i - y_j)/|x_i - y_j|^3 w_j p_j X[j][c0 + c]
//
// Same operator as laplace3d_DT (src/kernel/laplace3d.jl:30-40) / lfmm3d pg=2
// (src/kernel/laplace3d.jl:100-107); the 1/(4 pi) is applied by the combine.
//
// Bound by the FP64 pipes: FP64 MMA and FP64 FMA share one throughput budget, so a pair costs
// NC + (kernel value) operations. CTA = 4 warps; a warp owns MTW 8-row m-tiles and NC columns
// (NC / 8 n-tiles). Per k-step of 4 sources each thread generates the MTW FP64 kernel values of
// its A fragments (target = m-tile row l/4, source = l%4), with the source's weight multiplied
// in, and loads its B fragments (source l%4, column l/4 of each n-tile) from shared memory.
// In a planar tile (TileInfo) the difference along the normal axis and its square belong to the
// source and are formed once for the warp's MTW rows: 11 + 3 / MTW operations a value; other
// tiles take 17. Sources of the tile's own plane are left out. Source tiles of TSRC sources
// (coordinates, weights and rows of X, gathered through the sorted order) arrive by cp.async in
// a ring of NST stages, one barrier a tile, so that the loads of the next tiles run beside the
// sums of this one.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "solver.h"

namespace bie {
namespace d64 {

constexpr int NTHR = 128;  // threads per CTA
constexpr int TSRC = 32;   // sources per shared-memory tile
constexpr int NST = 3;     // stages of the source ring

// m-tiles per warp and resident CTAs per SM: the accumulators take MTW * NC / 4 doubles a thread. Four
// m-tiles share the source's part of a value (8 columns, 42,048 nodes: 2.02 ms, two m-tiles 2.22); the
// 8-column instance needs more than 128 registers to overlap its chains (three CTAs 2.02 ms, four 2.08).
template <int NC> constexpr int mtw() { return NC <= 16 ? 4 : 2; }
template <int NC> constexpr int occ() { return NC > 8 && NC <= 32 ? 4 : 3; }
// Row stride of a staged X tile (= 4 or 12 mod 16 doubles): the four k-rows a half-warp's
// B-fragment load touches fall on distinct banks; rows stay 16-byte aligned.
template <int NC> constexpr int ldq() { return NC + 4; }
// A stage: a, b, c coordinates, weights, preconditioner (TSRC each) and the X rows.
template <int NC> constexpr int stage_doubles() { return 5 * TSRC + TSRC * ldq<NC>(); }

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}
// Asynchronous copies to shared memory; `live` false writes zeros and reads nothing.
__device__ __forceinline__ void copy8(double* dst, const double* src, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(live ? 8 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy16(double* dst, const double* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src), "r"(live ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Kernel values: the adjoint double layer in a planar or another tile, the single layer 1 / r.
enum Value { kPlanar, kGeneral, kSingle };

// One source tile into the warp's accumulators. stg: the stage; cnt: its live sources; self:
// the tile's first slot when it may hold one of the warp's own targets, else negative.
template <int NC, Value V>
__device__ __forceinline__ void tile_step(const double* __restrict__ stg, int cnt, double plane,
                                          const double (&ta)[mtw<NC>()], const double (&tb)[mtw<NC>()],
                                          const double (&tc)[mtw<NC>()], const double (&tn)[mtw<NC>()][3],
                                          double (&acc)[mtw<NC>()][NC / 8][2], int lane, bool has_pre, int64_t self,
                                          int64_t slot0) {
    constexpr int MTW = mtw<NC>(), LDQ = ldq<NC>();
    const int kq = lane & 3, grp = lane >> 2;
    const double* sq = stg + 5 * TSRC;
#pragma unroll 2
    for (int k0 = 0; k0 < TSRC; k0 += 4) {
        const int j = k0 + kq;
        const double sa = stg[j], sb = stg[TSRC + j], sc = stg[2 * TSRC + j];
        double wj = stg[3 * TSRC + j];
        if (has_pre) wj *= stg[4 * TSRC + j];
        double a[MTW];
        if (V == kPlanar) {
            const double da = plane - sa, da2 = da * da;
            wj *= da;
#pragma unroll
            for (int mt = 0; mt < MTW; ++mt) {
                const double db = tb[mt] - sb, dc = tc[mt] - sc;
                a[mt] = over_r3(fma(db, db, fma(dc, dc, da2))) * wj;
            }
        } else {
#pragma unroll
            for (int mt = 0; mt < MTW; ++mt) {
                const double dx = ta[mt] - sa, dy = tb[mt] - sb, dz = tc[mt] - sc;
                const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
                if (V == kSingle)
                    a[mt] = rsqrt(r2) * wj;
                else
                    a[mt] = over_r3(r2) * (fma(tn[mt][0], dx, fma(tn[mt][1], dy, tn[mt][2] * dz)) * wj);
                if (j >= cnt || (self >= 0 && self + j == slot0 + mt * 8)) a[mt] = 0.0;
            }
        }
        double b[NC / 8];
#pragma unroll
        for (int nt = 0; nt < NC / 8; ++nt) b[nt] = sq[j * LDQ + nt * 8 + grp];
#pragma unroll
        for (int mt = 0; mt < MTW; ++mt)
#pragma unroll
            for (int nt = 0; nt < NC / 8; ++nt) dmma(acc[mt][nt][0], acc[mt][nt][1], a[mt], b[nt]);
    }
}

// POT: the single-layer potential at M targets T (3 x M) instead of the adjoint double
// layer at the nodes.
template <int NC, bool POT>
__global__ void __launch_bounds__(NTHR, occ<NC>()) k_dt_f64_mma(GeomDev g, const double* __restrict__ T, int64_t M,
                                                               const double* __restrict__ X, int ldx, int c0, int kc,
                                                               const double* __restrict__ pre,
                                                               double* __restrict__ part, int ldp) {
    constexpr int MTW = mtw<NC>(), LDQ = ldq<NC>(), TB = 32 * MTW;
    extern __shared__ __align__(16) double ring[];  // [NST][stage_doubles]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = lane >> 2, kq = lane & 3;
    const int64_t t0 = (int64_t)blockIdx.x * TB;
    const TileInfo ti = !POT && g.tiles ? g.tiles[t0 / kTB] : TileInfo{3, 0, 0, {}, {}};
    // coordinate arrays, the tile's axis first
    const double* pa = ti.axis == 1 ? g.sy : (ti.axis == 2 ? g.sz : g.sx);
    const double* pb = ti.axis == 1 ? g.sz : (ti.axis == 2 ? g.sx : g.sy);
    const double* pc = ti.axis == 1 ? g.sx : (ti.axis == 2 ? g.sy : g.sz);
    // the thread's targets: m-tile mt, row grp -> slot slot0 + 8 mt
    const int64_t slot0 = t0 + warp * 8 * MTW + grp;
    double ta[MTW], tb[MTW], tc[MTW], tn[MTW][3];
#pragma unroll
    for (int mt = 0; mt < MTW; ++mt) {
        const int64_t slot = slot0 + 8 * mt;
        ta[mt] = tb[mt] = tc[mt] = -kFar;  // no target: not stored
        tn[mt][0] = tn[mt][1] = tn[mt][2] = 0.0;
        if (POT) {
            if (slot < M) {
                ta[mt] = T[3 * slot]; tb[mt] = T[3 * slot + 1]; tc[mt] = T[3 * slot + 2];
            }
            continue;
        }
        const int64_t i = slot < g.ns ? (g.perm ? (int64_t)g.perm[slot] : slot) : -1;
        if (i >= 0) {
            ta[mt] = pa[slot]; tb[mt] = pb[slot]; tc[mt] = pc[slot];
            tn[mt][0] = g.nx[i]; tn[mt][1] = g.ny[i]; tn[mt][2] = g.nz[i];
        }
    }
    const double plane = POT ? 0.0 : pa[t0];
    double acc[MTW][NC / 8][2];
#pragma unroll
    for (int mt = 0; mt < MTW; ++mt)
#pragma unroll
        for (int nt = 0; nt < NC / 8; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = 0.0;

    const int64_t live = live_slots(g, ti), chunk = live_chunk(live, gridDim.y);
    const int64_t l0 = (int64_t)blockIdx.y * chunk, l1 = min(live, l0 + chunk);
    const int ntile = l1 > l0 ? (int)((l1 - l0 + TSRC - 1) / TSRC) : 0;
    // 16-byte copies of X rows: c0 is a multiple of 64
    const bool x16 = (ldx & 1) == 0 && (reinterpret_cast<uintptr_t>(X) & 15) == 0;
    // node of the source tile's row 8 warp + lane % 8 (-1: none); the warp copies those 8 rows
    auto row_node = [&](int t) -> int {
        if (t >= ntile) return -1;
        const int64_t j = live_slot(ti, l0 + (int64_t)t * TSRC) + 8 * warp + (lane & 7);
        return j < g.ns ? (g.perm ? g.perm[j] : (int)j) : -1;
    };
    auto issue = [&](int t, int node) {
        double* stg = ring + (t % NST) * stage_doubles<NC>();
        const int64_t j = live_slot(ti, l0 + (int64_t)t * TSRC) + lane;
        const double* arr = warp == 0 ? pa : (warp == 1 ? pb : (warp == 2 ? pc : g.sw));
        copy8(stg + warp * TSRC + lane, arr + (j < g.ns ? j : 0), j < g.ns);
        if (pre && lane < 8) copy8(stg + 4 * TSRC + 8 * warp + lane, pre + (node < 0 ? 0 : node), node >= 0);
        double* sq = stg + 5 * TSRC + 8 * warp * LDQ;
        if (x16) {
#pragma unroll
            for (int e0 = 0; e0 < 4 * NC; e0 += 32) {
                const int e = e0 + lane, u = e / (NC / 2), cc = 2 * (e % (NC / 2));
                const int p = __shfl_sync(0xFFFFFFFFu, node, u);
                if (cc < kc) copy16(sq + u * LDQ + cc, X + (int64_t)(p < 0 ? 0 : p) * ldx + c0 + cc, p >= 0);
            }
        } else {
#pragma unroll
            for (int e0 = 0; e0 < 8 * NC; e0 += 32) {
                const int e = e0 + lane, u = e / NC, cc = e % NC;
                const int p = __shfl_sync(0xFFFFFFFFu, node, u);
                if (cc < kc) copy8(sq + u * LDQ + cc, X + (int64_t)(p < 0 ? 0 : p) * ldx + c0 + cc, p >= 0);
            }
        }
    };
    // columns kc .. NC - 1 of the staged rows are never copied: zero, not what the memory held
    if (kc < NC) {
        for (int e = threadIdx.x; e < NST * stage_doubles<NC>(); e += NTHR) ring[e] = 0.0;
        __syncthreads();
    }
#pragma unroll
    for (int t = 0; t < NST - 1; ++t) {
        if (t < ntile) issue(t, row_node(t));
        copy_commit();
    }
    int next = row_node(NST - 1);
    for (int t = 0; t < ntile; ++t) {
        copy_wait<NST - 2>();
        __syncthreads();  // tile t landed for all warps; stage (t - 1) % NST is free
        if (t + NST - 1 < ntile) issue(t + NST - 1, next);
        copy_commit();
        next = row_node(t + NST);
        const double* stg = ring + (t % NST) * stage_doubles<NC>();
        const int cnt = (int)min((int64_t)TSRC, l1 - l0 - (int64_t)t * TSRC);
        if (POT) {
            tile_step<NC, kSingle>(stg, cnt, plane, ta, tb, tc, tn, acc, lane, false, -1, slot0);
        } else if (ti.axis < 3) {
            tile_step<NC, kPlanar>(stg, cnt, plane, ta, tb, tc, tn, acc, lane, pre != nullptr, -1, slot0);
        } else {
            const int64_t jt = live_slot(ti, l0 + (int64_t)t * TSRC);
            const bool self = jt < t0 + TB && jt + TSRC > t0;
            tile_step<NC, kGeneral>(stg, cnt, plane, ta, tb, tc, tn, acc, lane, pre != nullptr, self ? jt : -1, slot0);
        }
    }
    // D fragment: (row grp, columns 2 kq, 2 kq + 1) of each (m-tile, n-tile)
#pragma unroll
    for (int mt = 0; mt < MTW; ++mt) {
        const int64_t slot = slot0 + 8 * mt;
        const int64_t i = POT ? (slot < M ? slot : -1)
                              : (slot < g.ns ? (g.perm ? (int64_t)g.perm[slot] : slot) : -1);
        if (i < 0) continue;
        const double sgn = ti.axis == 0 ? g.nx[i] : (ti.axis == 1 ? g.ny[i] : (ti.axis == 2 ? g.nz[i] : 1.0));
        double* o = part + ((int64_t)blockIdx.y * (POT ? M : g.n) + i) * ldp + c0;
#pragma unroll
        for (int nt = 0; nt < NC / 8; ++nt) {
            const int c = nt * 8 + 2 * kq;
            if (c < kc) o[c] = sgn * acc[mt][nt][0];
            if (c + 1 < kc) o[c + 1] = sgn * acc[mt][nt][1];
        }
    }
}

template <int NC> constexpr size_t smem() { return sizeof(double) * NST * stage_doubles<NC>(); }

template <int NC, bool POT>
void launch(const GeomDev& g, const double* T, int64_t M, const double* X, int ldx, int c0, int kc, const double* pre,
            int nsplit, double* part, int ldp, cudaStream_t s) {
    constexpr int TB = 32 * mtw<NC>();
    const auto k = k_dt_f64_mma<NC, POT>;
    ensure_smem_limit((const void*)k, smem<NC>());
    const dim3 grid((unsigned)(((POT ? M : g.ns) + TB - 1) / TB), (unsigned)nsplit);
    k<<<grid, NTHR, smem<NC>(), s>>>(g, T, M, X, ldx, c0, kc, pre, part, ldp);
}

// Runs f(NC as an integral constant) for the instance of a pass of kc columns.
template <class F>
auto with_width(int kc, F&& f) {
    using std::integral_constant;
    if (kc > 32) return f(integral_constant<int, 64>());
    if (kc > 16) return f(integral_constant<int, 32>());
    if (kc > 8) return f(integral_constant<int, 16>());
    return f(integral_constant<int, 8>());
}

template <bool POT>
void launch_width(const GeomDev& g, const double* T, int64_t M, const double* X, int ldx, int c0, int kc,
                  const double* pre, int nsplit, double* part, int ldp, cudaStream_t s) {
    with_width(kc, [&](auto nc) { launch<nc.value, POT>(g, T, M, X, ldx, c0, kc, pre, nsplit, part, ldp, s); });
    BIE_CK(cudaGetLastError());
}

// Targets per CTA and resident CTAs per SM of the instance of a pass of kc columns.
struct Instance {
    int tb, per_sm;
};
template <bool POT>
Instance instance_of(int kc) {
    return with_width(kc, [](auto nc) {
        constexpr int NC = nc.value;
        return Instance{32 * mtw<NC>(), occupancy((const void*)k_dt_f64_mma<NC, POT>, NTHR, smem<NC>())};
    });
}

}  // namespace d64

// Columns [c0, c0 + kc) with kc <= 64 (NC = 8, 16, 32 or 64 columns per launch), c0 a multiple
// of 64. The sources are split evenly into nsplit parts, each writing its own partial.
void launch_dt_f64_mma(const GeomDev& g, const double* X, int ldx, int c0, int kc, const double* pre, int nsplit,
                       double* part, int ldp, cudaStream_t s) {
    d64::launch_width<false>(g, nullptr, 0, X, ldx, c0, kc, pre, nsplit, part, ldp, s);
}

int dt_f64_mma_ctas_per_sm(int kc) { return d64::instance_of<false>(kc).per_sm; }

// Source splits of the potential at M targets, for the instance of the first pass. 20,000 targets, 42,048
// nodes, at most one wave and now: 8 columns 1.78 and 1.41 ms, 17 columns 4.16 and 2.78, 64 columns
// 6.27 and 4.50; 1,000 targets as before.
int pot_f64_mma_splits(int64_t n, int64_t M, int k, int sms) {
    const d64::Instance in = d64::instance_of<true>(std::min(k, 64));
    return wave_splits(n, (M + in.tb - 1) / in.tb, (int64_t)sms * in.per_sm);
}

// Single-layer potential partials (laplace3d_pottrg, src/kernel/laplace3d.jl:69-82, without the
// 1/(4 pi)) of columns [c0, c0 + kc), kc <= 64 and c0 a multiple of 64, at M targets T (3 x M):
//   part[s][m][c0 + c] = sum_{j in split s} w_j X[j][c0 + c] / |x_m - y_j|
// The same kernel with 1 / r for its value: 42,048 nodes, 1,000 targets, 64 columns 0.55 -> 0.27 ms with
// the split reduction, where the sum on FP64 FMAs alone is limited by its shared-memory loads.
void launch_pot_f64_mma(const GeomDev& g, const double* T, int64_t M, const double* X, int ldx, int c0, int kc,
                        int nsplit, double* part, int ldp, cudaStream_t s) {
    GeomDev r = g;  // the nodes in the caller's order and unit: the targets are not scaled
    r.sx = g.x; r.sy = g.y; r.sz = g.z; r.sw = g.w;
    r.perm = nullptr;
    r.tiles = nullptr;
    r.ns = g.n;
    d64::launch_width<true>(r, T, M, X, ldx, c0, kc, nullptr, nsplit, part, ldp, s);
}

}  // namespace bie
