// Device-side types shared by the kernel translation units.
#pragma once
#include <vector>
#include <cuda_runtime.h>
#include <stdint.h>

#include "sorted_nodes.h"
#include "splits.h"

namespace bie {

// Packed FP32 pairs (sm_100 f32x2 arithmetic): one instruction applies the same
// round-to-nearest operation to two lanes of data.
__device__ __forceinline__ uint64_t pk2(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 upk2(uint64_t r) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(r));
    return v;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}


constexpr double kInv4Pi = 0.079577471545947667884;  // 1 / (4 pi)

// MUFU reciprocal square root (approximate, flush-to-zero): a single instruction.
__device__ __forceinline__ float rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Device-resident geometry: SoA FP64 arrays of length n in the caller's node order, and the
// sorted order of the direct sums. Sorted order: the nodes of each coordinate plane with at
// least kPlaneMin nodes on it (axis-aligned normals) together, the others after them, each
// group bisected into compact tiles (coordinates rounded to FP32 relative to a tile's middle stay
// accurate for near pairs) and padded to a multiple of kTB slots. Sorted coordinates are scaled by a power of two to an extent in [0.5, 1), the
// weights by its square, which leaves the sums unchanged bit for bit and keeps 1 / r^3 in range
// in FP32 whatever the unit of length. Padding slots: perm -1, far away (kFar), weight 0.
struct GeomDev {
    const double *x, *y, *z;     // node positions
    const double *nx, *ny, *nz;  // node normals
    const double* w;             // quadrature weights
    int64_t n;
    const double *sx, *sy, *sz, *sw;  // sorted positions and weights (ns slots)
    const int32_t* perm;              // node of each slot; null: slots are the nodes in order
    const TileInfo* tiles;            // one per kTB slots; null: no planar tile
    int64_t ns;                       // slots
};
// Slots a tile sums over (all but its own plane's) and the l-th of them (s0, s1 and l are
// multiples of every source tile, so a source tile never straddles the gap).
__device__ __forceinline__ int64_t live_slots(const GeomDev& g, const TileInfo& t) { return g.ns - (t.s1 - t.s0); }
__device__ __forceinline__ int64_t live_slot(const TileInfo& t, int64_t l) { return l < t.s0 ? l : l + (t.s1 - t.s0); }
// First live slot of source split y of nsplit (splits rounded up to kTS slots).
__device__ __forceinline__ int64_t live_chunk(int64_t live, int nsplit) {
    const int64_t c = (live + nsplit - 1) / nsplit;
    return (c + kTS - 1) / kTS * kTS;
}

// Near tiles of the FP32 sum (K2). A coordinate relative to the target tile's origin, rounded to FP32,
// is off by up to 2^-25 of the tile's half side h, which at a distance r puts an error of a few
// 2^-25 h / r into a kernel value: below that of the FP32 operations unless the tiles (nearly) touch.
// For source tiles closer than h / 4 the differences are therefore formed from two FP32 numbers a
// coordinate (the rounded one and what it leaves), which makes them good to an FP32 rounding.
// 23,040 nodes, random values: 1.2 % of the tile pairs, error of the FP32 sum 1.3e-6 -> 1.9e-7.
struct NearBox {
    double o[3], reach[3];
    __device__ __forceinline__ explicit NearBox(const TileInfo& t) {
        const double gap = 0.25 * fmax(t.h[0], fmax(t.h[1], t.h[2]));
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            o[c] = t.o[c];
            reach[c] = t.h[c] + gap;
        }
    }
    __device__ __forceinline__ bool holds(const TileInfo& s) const {
        return fabs(s.o[0] - o[0]) - s.h[0] < reach[0] && fabs(s.o[1] - o[1]) - s.h[1] < reach[1] &&
               fabs(s.o[2] - o[2]) - s.h[2] < reach[2];
    }
};
// What the FP32 rounding f of x leaves.
__device__ __forceinline__ float rest32(double x, float f) { return (float)(x - (double)f); }

// FP64 seed of 1 / sqrt(x), relative error about 2^-20: one MUFU instruction (PTX
// rsqrt.approx.ftz.f64).
__device__ __forceinline__ double rsqrt_seed(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    return y;
}
// 1 / r^3 from r2 = r^2. With the seed y and e = 1 - r2 y^2, 1 / r^3 = y^3 (1 - e)^(-3/2), the
// binomial series cut after e^2: the next term, 35/16 e^3, is below 2^-55 for |e| < 2^-19.
// 6 FP64 operations, where 1 / sqrt to full precision and its cube take about 11.
__device__ __forceinline__ double over_r3(double r2) {
    const double y = rsqrt_seed(r2);
    const double q = y * y;
    const double e = fma(-r2, q, 1.0);
    const double s = e * fma(e, 1.875, 1.5);
    const double w = y * q;
    return fma(w, s, w);
}

// K3 (blocktc.cu): tensor-core block direct sum for columns [c0, c0 + kc), kc <= 128,
// kernel and right-hand sides split into `pieces` bf16 pieces (2 or 3).
void launch_block_tc(const GeomDev& g, const double* X, int ldx, int c0, int kc, const double* pre, int nsplit,
                     float* part, int ldp, uint8_t* bpack, int* err, int pieces, cudaStream_t s);
size_t block_tc_pack_bytes(int64_t slots, int kc, int pieces);
// One geometry's share of a K3 work-list launch: columns [c0, c0 + kc) (kc <= 128) of X,
// nsplit source splits, partials into part (ldp), Q images into bpack.
struct TcMember {
    GeomDev g;
    const double* X;
    int ldx, c0, kc;
    const double* pre;
    int nsplit;
    float* part;
    int ldp;
    uint8_t* bpack;
};
// K3 over the (target tile, source split) work items of several geometries in one launch
// (members in the given order, each member's Q packed first); the work list and the
// members' parameters go to dscratch (block_tc_list_bytes of it).
void launch_block_tc_list(const std::vector<TcMember>& ms, int pieces, int* err, void* dscratch, size_t scratch_bytes,
                          cudaStream_t s);
size_t block_tc_list_bytes(int nmembers, int64_t nitems);
int block_tc_ctas_per_sm(int kc, int pieces);
int tc_npad(int kc);
// K1 with the FP64 tensor-core contraction (dt64mma.cu), columns [c0, c0 + kc), kc <= 64.
void launch_dt_f64_mma(const GeomDev& g, const double* X, int ldx, int c0, int kc, const double* pre, int nsplit,
                       double* part, int ldp, cudaStream_t s);
int dt_f64_mma_ctas_per_sm(int kc);  // of the instance for kc columns
// Single-layer potential at M targets with the same contraction (dt64mma.cu).
int pot_f64_mma_splits(int64_t n, int64_t M, int k, int sms);
void launch_pot_f64_mma(const GeomDev& g, const double* T, int64_t M, const double* X, int ldx, int c0, int kc,
                        int nsplit, double* part, int ldp, cudaStream_t s);
constexpr int kTcTileM = 128;   // targets per tensor-core tile
constexpr int kTcChunk = 64;    // sources per tensor-core chunk

}  // namespace bie
