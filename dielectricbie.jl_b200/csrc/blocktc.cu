// K3: block direct sum of the reduced-precision operators on the 5th-generation tensor cores
// (tcgen05, sm_100a).
//
//   part[s][i][c0 + c] = sum_{j in split s, j != i} G(i, j) Q(j, c)
//   G(i, j) = n_i . (x_i - y_j) / |x_i - y_j|^3        (generated in FP32 registers)
//   Q(j, c) = w_j p_j X[j][c0 + c]                     (packed per call, in the sorted order)
//
// G is the adjoint double-layer kernel of laplace3d_DT (src/kernel/laplace3d.jl:30-40);
// the contraction replaces the batched lfmm3d(nd = K) of
// mul!(Y, ::BatchedDielectricOperator, X) (src/solver/multi_rhs.jl:103-130).
//
// Split-BF16 products: G = Gh + Gl and Q = Qh + Ql (bf16 hi/lo), all four products; with three
// pieces the six whose orders sum to at most 2. The tensor cores accumulate FP32 in tensor memory
// over kPeriod = 256 sources into one of two alternating accumulators; the generator threads add
// each finished period into FP32 running sums in registers. The tensor-core accumulation error
// grows with the number of accumulation steps; restarting it every period bounds it by that of
// 256 sources, and the running sum of the periods (round-to-nearest additions) adds a random-walk
// error of a few units in the last place. Each source split writes the sum as an FP32 partial.
//
// CTA = 128 NQ + 64 threads: warps 0 .. 4 NQ - 1 generate the kernel tile of a stage of KS = NQ SPT
// sources (NQ threads per target row, SPT sources each), fold the accumulators and run the epilogue;
// the next warp issues the MMAs (one thread); the last warp streams the pre-swizzled Q tiles with
// bulk copies into a ring and stages the source coordinates.
//
// The kernel tile is the MMA's A operand in tensor memory: a generator thread owns a row, which is
// a tensor-memory lane, and stores its packed pieces there (two stages). Kept in shared memory, as
// the tile was, every product of a 16-source step reads the 4 KB of A again beside 2 KB of Q: 16
// bytes of shared-memory traffic a pair at 64 columns, half of the bandwidth at the old rate and
// all of it at this one. Bound by the generators' instruction stream (FP32 and MUFU pipes): a
// planar tile (TileInfo) takes the difference along its axis and the square of it from the staged
// source, 7 packed operations for two pairs, other tiles 12; sources of the tile's own plane are
// left out. Barriers are arrived at once a warp, ring positions are counted, not divided.
//
// Two CTAs per SM (NQ = 2, 256 tensor-memory columns each) where the accumulators and the two A
// stages fit, so that one CTA's prologue, folds and epilogue are filled by the other; wider tiles
// run one CTA per SM (NQ = 4, 512 columns).
//
// Measured, 42,048 nodes in two pieces, before and after: 8 columns 1.33 and 0.74 ms, 64 columns 1.50
// and 0.82, 128 columns 2.19 and 1.16. 12.1 warp instructions per 32 pairs, where the arithmetic takes
// 9 and the generator alone, without MMAs, runs 30 % faster.
// Every mbarrier wait is bounded: on expiry the CTA records an error code and
// returns after releasing its tensor memory.
#include <cuda_bf16.h>
#include <algorithm>
#include <cstdlib>
#include <vector>
#include <cuda_runtime.h>
#include <stdint.h>

#include "common.cuh"
#include "mbar.cuh"
#include "solver.h"

namespace bie {
namespace tc {

constexpr int M = 128;      // targets per tile (MMA M)
constexpr int KC = 64;      // sources per chunk = one 128-byte bf16 row of a Q tile
constexpr int SA = 2;       // A (kernel tile) stages in tensor memory
constexpr int SBMAX = 4;    // B (Q tile) ring stages at most (Params::sb)
constexpr int kPeriod = 256;  // sources accumulated in tensor memory before a fold
constexpr int SC = 2;       // source-coordinate slots, one period of sources each
// NQ = generator threads per tile row: 2 for the two-CTAs-per-SM shape (320 threads, <= 96
// registers), 4 for the one-CTA shape (576 threads, <= 112 registers).
template <int NQ> __host__ __device__ constexpr int ngen() { return M * NQ; }
template <int NQ> __host__ __device__ constexpr int nthreads() { return M * NQ + 64; }
// Columns each generator thread folds: CPQ (8, 16 or 32), so a tile has up to NQ CPQ columns.
// Sources per generator thread and stage: 32, or 16 where three pieces of that many and the
// accumulators of up to 128 columns would not fit the tensor memory.
template <int NP, int CPQ> __host__ __device__ constexpr int spt() { return NP == 3 && CPQ == 32 ? 16 : 32; }
template <int NP, int NQ, int CPQ> __host__ __device__ constexpr int ks() { return NQ * spt<NP, CPQ>(); }
constexpr uint32_t kWaitLimit = 1u << 26;  // default wait attempts before a CTA gives up (seconds)
constexpr int kErrTimeout = 1;

struct Params {
    GeomDev g;
    const uint8_t* bpack;  // [chunks][NP][npad][128 B] pre-swizzled bf16 images
    int npad;              // MMA N (multiple of 16, <= 128)
    int keff;              // columns stored (<= npad)
    int nsplit;            // source splits
    int sb;                // B ring stages (2 .. SBMAX)
    uint32_t wait_limit;   // mbarrier wait attempts before the CTA gives up
    int stall_test;        // nonzero: withhold the first Q tile (exercises the timeout path)
    float* part;           // [nsplit][n][ldp] FP32 split partials
    int ldp, c0;
    int* err;
};

// Shared-memory head holding a CTA's copy of its Params and work item.
constexpr uint32_t kParamHead = ((uint32_t)sizeof(Params) + 2 * sizeof(int) + 15u) & ~15u;

// A ring position and the parity of its current pass.
struct Ring {
    int s = 0;
    uint32_t ph = 0;
    __device__ __forceinline__ void next(int n) {
        if (++s == n) {
            s = 0;
            ph ^= 1u;
        }
    }
};

// OR-reduction of a predicate over the NG generator threads (named barrier 1):
// also orders their shared-memory accesses like bar.sync.
template <int NG>
__device__ __forceinline__ bool gen_any(bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.or.pred p, 1, %2, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)v), "n"(NG)
        : "memory");
    return r != 0;
}

__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    // K-major, 128-byte swizzle: rows of 128 B, 8-row atoms 1024 B apart (SBO),
    // LBO unused (1), descriptor version 1, layout type 2 (SWIZZLE_128B).
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1u << 16;
    d |= (uint64_t)(1024u >> 4) << 32;
    d |= (uint64_t)1u << 46;
    d |= (uint64_t)2u << 61;
    return d;
}

__device__ __forceinline__ uint32_t idesc_bf16(int n) {
    // c_format F32 (1) @4, a/b format BF16 (1) @7/@10, K-major A/B, N>>3 @17, M>>4 @24
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D (tensor memory) += A (tensor memory, K-major rows in lanes) B (shared memory).
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint32_t tmem_a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

// One lane of a converged warp. A branch on elect.sync lets the compiler keep the MMA operands in
// uniform registers: a thread picked by its lane index issues at most one MMA in 45 cycles (136 with
// addresses computed at run time), the elected one in 10 (N = 16) to 64 (N = 128, the tensor cores' rate).
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xFFFFFFFF;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 32 lanes x C columns of tensor memory (C = 8 or 16) to registers, valid after tmem_wait_ld().
template <int C>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, uint32_t* r) {
    if constexpr (C == 8)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr));
    else
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 8 registers a lane to 8 columns of tensor memory.
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

__device__ __forceinline__ uint32_t pack_bf16(float lo_elem, float hi_elem) {
    __nv_bfloat162 h = __floats2bfloat162_rn(lo_elem, hi_elem);  // .x (low 16 bits) = lo_elem
    return *reinterpret_cast<uint32_t*>(&h);
}

// Split two FP32 values into NP packed bf16 pieces (hi, lo or hi, mid, lo): each
// piece is the bf16 rounding of what the previous pieces leave.
template <int NP>
__device__ __forceinline__ void split_pieces(float a, float b, uint32_t* out) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const uint32_t w = pack_bf16(a, b);
        out[p] = w;
        if (p + 1 < NP) {
            a -= __uint_as_float(w << 16);
            b -= __uint_as_float(w & 0xFFFF0000u);
        }
    }
}

// split_pieces on a packed pair (the remainders are formed with one packed operation).
template <int NP>
__device__ __forceinline__ void split_pieces2(uint64_t x, uint32_t* out) {
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const float2 xu = upk2(x);
        const uint32_t w = pack_bf16(xu.x, xu.y);
        out[p] = w;
        if (p + 1 < NP)
            x = fma2(pk2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u)), pk2(-1.f, -1.f), x);
    }
}

// One thread's share of a stage's kernel tile: SPT sources, 16 at a time as 8 packed pairs, to the
// tensor-memory columns ta (piece p at ta + p * pstride, 8 columns per 16 sources). Four coordinate
// arrays of kPeriod from a0. PLANAR: the source's difference along the tile's axis, its square, and
// minus its other two coordinates; t1 and t2: the target's (duplicated into both halves of a pair).
// !PLANAR: minus x, y, z; the target's own source gives n . 0 = 0 with r^2 = kTiny.
constexpr float kTiny = 1.2e-38f;
template <bool PLANAR, int NP, int SPT>
__device__ __forceinline__ void gen_row_part(const float* __restrict__ a0, uint64_t t0, uint64_t t1, uint64_t t2,
                                             uint64_t n0, uint64_t n1, uint64_t n2, uint32_t ta, uint32_t pstride) {
    const float *a1 = a0 + kPeriod, *a2 = a1 + kPeriod, *a3 = a2 + kPeriod;
#pragma unroll
    for (int g = 0; g < SPT; g += 16) {
        uint64_t v[8];  // kernel values of sources g + 2 m, + 1
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const ulonglong2 A = *reinterpret_cast<const ulonglong2*>(a0 + g + 4 * e);
            const ulonglong2 B = *reinterpret_cast<const ulonglong2*>(a1 + g + 4 * e);
            const ulonglong2 C = *reinterpret_cast<const ulonglong2*>(a2 + g + 4 * e);
            if (PLANAR) {
                const ulonglong2 D = *reinterpret_cast<const ulonglong2*>(a3 + g + 4 * e);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint64_t db = add2(t1, h ? C.y : C.x), dc = add2(t2, h ? D.y : D.x);
                    const float2 r2 = upk2(fma2(db, db, fma2(dc, dc, h ? B.y : B.x)));
                    const uint64_t ri = pk2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
                    v[e * 2 + h] = mul2(mul2(h ? A.y : A.x, ri), mul2(ri, ri));
                }
            } else {
                const uint64_t tiny = pk2(kTiny, kTiny);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint64_t dx = add2(t0, h ? A.y : A.x), dy = add2(t1, h ? B.y : B.x),
                                   dz = add2(t2, h ? C.y : C.x);
                    const float2 r2 = upk2(fma2(dx, dx, fma2(dy, dy, fma2(dz, dz, tiny))));
                    const uint64_t ri = pk2(rsqrt_approx(r2.x), rsqrt_approx(r2.y));
                    const uint64_t dn = fma2(n0, dx, fma2(n1, dy, mul2(n2, dz)));
                    v[e * 2 + h] = mul2(mul2(dn, ri), mul2(ri, ri));
                }
            }
        }
        uint32_t w[NP][8];
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            uint32_t o[NP];
            split_pieces2<NP>(v[m], o);
#pragma unroll
            for (int p = 0; p < NP; ++p) w[p][m] = o[p];
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) tmem_st8(ta + (uint32_t)p * pstride + (uint32_t)(g / 2), w[p]);
    }
}

// The CTA body: target tile `tile`, source split `split` of the geometry in P. The plain
// launch (k_dt_tc, grid = tiles x splits) reads P from the kernel parameters; the
// work-list launch (k_dt_tc_list) runs one item of several geometries' tiles per CTA and
// reads its P from a copy at the head of the CTA's shared memory.
template <int NP, int NQ, int CPQ>
__device__ __forceinline__ void tc_body(const Params& P, const int tile, const int split, uint8_t* smem_raw) {
    constexpr int NGEN = ngen<NQ>(), NGW = NGEN / 32;
    constexpr int SPT = spt<NP, CPQ>(), KS = ks<NP, NQ, CPQ>(), CPS = KS / KC;  // CPS: chunks per stage
    constexpr int SPP = kPeriod / KS;                                           // stages per period
    constexpr uint32_t TCOLS = NQ == 2 ? 256 : 512;
    constexpr uint32_t A_COLS = KS / 2;  // tensor-memory columns of one piece of a stage
    // carve-up aligned to 1024 bytes in the shared window (128-byte swizzle atoms), after
    // the parameter head
    uint8_t* const head_end = smem_raw + kParamHead;
    uint8_t* base = head_end + ((1024u - (smem_u32(head_end) & 1023u)) & 1023u);
    const int npad = P.npad;
    const uint32_t b_bytes = (uint32_t)npad * 128;  // one piece of a chunk's Q tile
    const uint32_t ch_bytes = NP * b_bytes;         // a chunk's Q tile
    const int SB = P.sb;
    uint8_t* B = base;                                    // [SB][CPS][NP][b_bytes]
    float* crd = (float*)(B + (size_t)SB * CPS * ch_bytes);  // [SC][4][kPeriod] source coordinates (see gen_row_part)
    uint64_t* full_a = (uint64_t*)(crd + SC * 4 * kPeriod);  // [SA] kernel tile stored (generator warps)
    uint64_t* empty_a = full_a + SA;       // [SA] A stage consumed (MMA commit)
    uint64_t* full_b = empty_a + SA;       // [SBMAX] Q tile landed (bulk copy)
    uint64_t* empty_b = full_b + SBMAX;    // [SBMAX] Q tile consumed (MMA commit)
    uint64_t* crd_full = empty_b + SBMAX;  // [SC] coordinates staged (producer warp)
    uint64_t* crd_empty = crd_full + SC;   // [SC] coordinates consumed (generator warps)
    uint64_t* acc_full = crd_empty + SC;   // [2] accumulation period finished (MMA commit)
    uint64_t* acc_empty = acc_full + 2;    // [2] accumulator folded (generator warps)
    uint64_t* acc_done = acc_empty + 2;
    uint32_t* tmem_slot = (uint32_t*)(acc_done + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t n = P.g.n;
    const int64_t i0 = (int64_t)tile * M;
    const TileInfo& ti = P.g.tiles[tile];
    const int axis = ti.axis;
    // this split's share of the tile's live chunks (whole stages)
    const int nlive = (int)(live_slots(P.g, ti) / KC);
    const int share = ((nlive + P.nsplit - 1) / P.nsplit + CPS - 1) / CPS * CPS;
    const int ch0 = split * share;
    const int nch = max(0, min(nlive - ch0, share));
    const int nst = (nch + CPS - 1) / CPS;
    const int nper = (nst + SPP - 1) / SPP;

    if (threadIdx.x == 0) {
        for (int s = 0; s < SA; ++s) {
            mbar_init(&full_a[s], NGW);
            mbar_init(&empty_a[s], 1);
        }
        for (int s = 0; s < SBMAX; ++s) {
            mbar_init(&full_b[s], 1);
            mbar_init(&empty_b[s], 1);
        }
        for (int s = 0; s < SC; ++s) {
            mbar_init(&crd_full[s], 1);
            mbar_init(&crd_empty[s], NGW);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], NGW);
        }
        mbar_init(acc_done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(TCOLS)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;              // two accumulators, npad columns each
    const uint32_t t_a = tmem + 2u * (uint32_t)npad;  // [SA][NP][A_COLS]

    // tile origin and coordinate order (a planar tile's axis first)
    const int x0 = axis < 3 ? axis : 0, x1 = x0 == 2 ? 0 : x0 + 1, x2 = x1 == 2 ? 0 : x1 + 1;
    const double* const p0 = x0 == 0 ? P.g.sx : (x0 == 1 ? P.g.sy : P.g.sz);
    const double* const p1 = x1 == 0 ? P.g.sx : (x1 == 1 ? P.g.sy : P.g.sz);
    const double* const p2 = x2 == 0 ? P.g.sx : (x2 == 1 ? P.g.sy : P.g.sz);
    const double o0 = ti.o[x0], o1 = ti.o[x1], o2 = ti.o[x2];

    if (warp < NGW) {
        // ------------------------- generators -------------------------------
        const int r = threadIdx.x & (M - 1);  // tile row
        const int qt = threadIdx.x / M;       // which SPT sources of each stage (warp-uniform)
        const int64_t i = P.g.perm[i0 + r];   // the target's node, -1 in a padding slot
        const bool valid = i >= 0;
        float f0 = -1.0e18f, f1 = -1.0e18f, f2 = -1.0e18f;  // no target: not stored
        float m0 = 0.f, m1 = 0.f, m2 = 0.f;
        if (valid) {
            f0 = (float)(p0[i0 + r] - o0); f1 = (float)(p1[i0 + r] - o1); f2 = (float)(p2[i0 + r] - o2);
            m0 = (float)P.g.nx[i]; m1 = (float)P.g.ny[i]; m2 = (float)P.g.nz[i];
        }
        const float sgn = axis == 0 ? m0 : (axis == 1 ? m1 : (axis == 2 ? m2 : 1.f));
        const uint64_t t0 = pk2(f0, f0), t1 = pk2(f1, f1), t2 = pk2(f2, f2);
        const uint64_t n0 = pk2(m0, m0), n1 = pk2(m1, m1), n2 = pk2(m2, m2);
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        uint64_t sum[CPQ / 2];  // packed pairs
#pragma unroll
        for (int c = 0; c < CPQ / 2; ++c) sum[c] = 0ull;

        // Adds the FP32 accumulator of the next period into the running sums.
        Ring fr;
        auto fold = [&]() -> bool {
            const bool ok = mbar_wait(&acc_full[fr.s], fr.ph, abort_flag, P.wait_limit);
            if (!__all_sync(0xFFFFFFFFu, ok)) return false;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            constexpr int C = CPQ < 16 ? CPQ : 16;
#pragma unroll
            for (int c = 0; c < CPQ; c += C) {
                if (qt * CPQ + c < npad) {
                    uint32_t a[C];
                    tmem_ld<C>(tmem + lane_base + (uint32_t)(fr.s * npad + qt * CPQ + c), a);
                    tmem_wait_ld();
#pragma unroll
                    for (int q = 0; q < C; q += 2)
                        sum[(c + q) / 2] = add2(sum[(c + q) / 2], pk2(__uint_as_float(a[q]), __uint_as_float(a[q + 1])));
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[fr.s]);
            fr.next(2);
            return true;
        };

        bool ok = true;
        int use = 0;  // stages so far; stage use & 1 of the A ring (SPP is even)
        for (int p = 0; p < nper && ok; ++p) {
            const float* cs = crd + (p & 1) * 4 * kPeriod + qt * SPT;
            ok = mbar_wait(&crd_full[p & 1], (uint32_t)(p >> 1) & 1u, abort_flag, P.wait_limit);
            const int stages = min(SPP, nst - p * SPP);
#pragma unroll 1
            for (int q = 0; q < stages; ++q, ++use) {
                // the stage was released by the MMAs of two stages ago
                const int sa = use & 1;
                ok = ok && mbar_wait(&empty_a[sa], ((uint32_t)(use >> 1) & 1u) ^ 1u, abort_flag, P.wait_limit);
                if (!__all_sync(0xFFFFFFFFu, ok)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const float* c = cs + q * KS;
                const uint32_t ta = t_a + lane_base + (uint32_t)(sa * NP) * A_COLS + (uint32_t)(qt * SPT / 2);
                if (axis < 3)
                    gen_row_part<true, NP, SPT>(c, t0, t1, t2, n0, n1, n2, ta, A_COLS);
                else
                    gen_row_part<false, NP, SPT>(c, t0, t1, t2, n0, n1, n2, ta, A_COLS);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_a[sa]);
            }
            if (lane == 0) mbar_arrive(&crd_empty[p & 1]);
            // fold the period before this one (its MMAs finished while this one was generated)
            if (ok && p >= 1) ok = fold();
        }
        // ------------------------- epilogue ---------------------------------
        ok = ok && !*abort_flag;
        if (nst > 0 && ok) ok = fold();
        ok = !gen_any<NGEN>(!ok);  // every generator warp takes the same branch
        if (ok && valid) {
            float* out = P.part + ((int64_t)split * n + i) * P.ldp + P.c0;
            const bool v4 = ((P.ldp | P.c0) & 3) == 0;  // rows start on 16 bytes
#pragma unroll
            for (int c = 0; c < CPQ; c += 4) {
                const int cc = qt * CPQ + c;
                const float2 u = upk2(sum[c / 2]), w = upk2(sum[c / 2 + 1]);
                const float v[4] = {sgn * u.x, sgn * u.y, sgn * w.x, sgn * w.y};
                if (v4 && cc + 4 <= P.keff)
                    *reinterpret_cast<float4*>(out + cc) = make_float4(v[0], v[1], v[2], v[3]);
                else
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (cc + q < P.keff) out[cc + q] = v[q];
            }
        }
    } else if (warp == NGW) {
        // ------------------------- MMA issuer --------------------------------
        if (elect_one()) {
            const uint32_t idesc = idesc_bf16(npad);
            Ring ra, rb, rp;
            int in_period = 0;
            for (int st = 0; st < nst; ++st) {
                if (!mbar_wait(&full_a[ra.s], ra.ph, abort_flag, P.wait_limit)) break;
                if (!mbar_wait(&full_b[rb.s], rb.ph, abort_flag, P.wait_limit)) break;
                // the accumulator is reused once the generators folded its last period
                const bool pfirst = in_period == 0;
                if (pfirst && !mbar_wait(&acc_empty[rp.s], rp.ph ^ 1u, abort_flag, P.wait_limit)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t dacc = tmem + (uint32_t)(rp.s * npad);
                const uint32_t ta = t_a + (uint32_t)(ra.s * NP) * A_COLS;
                const int present = min(CPS, nch - st * CPS);  // chunks of this stage
#pragma unroll 1
                for (int h = 0; h < present; ++h) {
                    // the start-address field (bits 0-13, address >> 4) is advanced in place: every
                    // address stays below 256 KB
                    const uint64_t db = sw128_desc(smem_u32(B + (size_t)(rb.s * CPS + h) * ch_bytes));
                    // all four products of two pieces, or the six of three whose orders sum to at most 2
#pragma unroll
                    for (int kk = 0; kk < KC / 16; ++kk)
#pragma unroll
                        for (int pa = 0; pa < NP; ++pa)
#pragma unroll
                            for (int pb = 0; pb < (NP == 2 ? 2 : NP - pa); ++pb)
                                mma_bf16(dacc, ta + (uint32_t)pa * A_COLS + (uint32_t)(h * (KC / 2) + kk * 8),
                                         db + (uint64_t)((pb * b_bytes + kk * 32) >> 4), idesc,
                                         pfirst && h == 0 && kk == 0 && pa == 0 && pb == 0 ? 0u : 1u);
                }
                mma_commit(&empty_a[ra.s]);
                mma_commit(&empty_b[rb.s]);
                if (++in_period == SPP || st == nst - 1) {
                    mma_commit(&acc_full[rp.s]);
                    in_period = 0;
                    rp.next(2);
                }
                ra.next(SA);
                rb.next(SB);
            }
            mma_commit(acc_done);
            // on abort, drain this thread's MMAs before the CTA releases tensor memory
            if (*abort_flag) mbar_wait_raw(acc_done, 0, P.wait_limit);
        }
        __syncwarp();
    } else {
        // ------------- Q-tile and source-coordinate producer -----------------
        // Runs SB - 1 stages ahead on the Q tiles and a period ahead on the coordinates; each slot is
        // refilled once its last consumer has finished.
        auto slot_of = [&](int ch) -> int64_t { return live_slot(ti, (int64_t)(ch0 + ch) * KC); };
        int issued = 0;
        Ring rb;
        auto stage_b = [&](int st) -> bool {
            if (!mbar_wait(&empty_b[rb.s], rb.ph ^ 1u, abort_flag, P.wait_limit)) return false;
            if (lane == 0) {
                const int present = min(CPS, nch - st * CPS);
                mbar_arrive_tx(&full_b[rb.s], (uint32_t)present * ch_bytes);
                // test of the timeout path: the first Q tile is announced but never copied
                if (!(P.stall_test && st == 0))
                    for (int h = 0; h < present; ++h)
                        bulk_g2s(B + (size_t)(rb.s * CPS + h) * ch_bytes,
                                 P.bpack + (size_t)(slot_of(st * CPS + h) / KC) * ch_bytes, ch_bytes, &full_b[rb.s]);
                issued = st + 1;
            }
            rb.next(SB);
            return true;
        };
        // coordinates of period p, FP32 relative to the tile origin; the global loads are issued
        // before the wait for the slot. Chunks past the last repeat it (they are not multiplied).
        auto stage_crd = [&](int p) -> bool {
            double d[kPeriod / 32][3];
#pragma unroll
            for (int h = 0; h < kPeriod / 32; ++h) {
                const int ch = p * (kPeriod / KC) + h / (KC / 32);
                const int64_t j = slot_of(min(ch, nch - 1)) + lane + 32 * (h % (KC / 32));
                d[h][0] = p0[j];
                d[h][1] = p1[j];
                d[h][2] = p2[j];
            }
            if (!mbar_wait(&crd_empty[p & 1], ((uint32_t)(p >> 1) & 1u) ^ 1u, abort_flag, P.wait_limit)) return false;
            float* cs = crd + (p & 1) * 4 * kPeriod + lane;
#pragma unroll
            for (int h = 0; h < kPeriod / 32; ++h) {
                const float a = (float)(o0 - d[h][0]), b = (float)(o1 - d[h][1]), c = (float)(o2 - d[h][2]);
                cs[32 * h] = a;
                cs[kPeriod + 32 * h] = axis < 3 ? a * a : b;
                cs[2 * kPeriod + 32 * h] = axis < 3 ? b : c;
                if (axis < 3) cs[3 * kPeriod + 32 * h] = c;
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&crd_full[p & 1]);
            return true;
        };
        bool ok = true;
        if (nper > 0) ok = stage_crd(0);
        for (int c = 0; c < SB - 1 && c < nst && ok; ++c) ok = stage_b(c);
        for (int p = 0; p < nper && ok; ++p) {
            if (p + 1 < nper) ok = stage_crd(p + 1);
            for (int st = p * SPP; st < min(nst, (p + 1) * SPP) && ok; ++st)
                if (st + SB - 1 < nst) ok = stage_b(st + SB - 1);
        }
        // on abort, wait for the copies still in flight (at most one per slot)
        if (lane == 0 && *abort_flag)
            for (int c = issued > SB ? issued - SB : 0; c < issued; ++c)
                if (!(P.stall_test && c == 0)) mbar_wait_raw(&full_b[c % SB], (c / SB) & 1, P.wait_limit);
        __syncwarp();
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) atomicOr(P.err, kErrTimeout);
    if (warp == 0) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TCOLS) : "memory");
    }
}

template <int NP, int NQ, int CPQ>
__global__ void __launch_bounds__(nthreads<NQ>(), 4 / NQ) k_dt_tc(Params P) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    tc_body<NP, NQ, CPQ>(P, (int)blockIdx.x, (int)blockIdx.y, smem_raw);
}

// Work-list launch: CTA b runs items[b] = (member, target tile, source split, unused) with
// the member's parameters plist[member]; one launch covers the tiles of several geometries,
// each with its own nodes, right-hand-side block, width and partials.
template <int NP, int NQ, int CPQ>
__global__ void __launch_bounds__(nthreads<NQ>(), 4 / NQ)
    k_dt_tc_list(const Params* __restrict__ plist, const int4* __restrict__ items) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    Params* sP = reinterpret_cast<Params*>(smem_raw);
    int* s_item = reinterpret_cast<int*>(smem_raw + sizeof(Params));
    if (threadIdx.x == 0) {
        const int4 it = items[blockIdx.x];
        *sP = plist[it.x];
        s_item[0] = it.y;
        s_item[1] = it.z;
    }
    __syncthreads();
    tc_body<NP, NQ, CPQ>(*sP, s_item[0], s_item[1], smem_raw);
}

// Packs Q(j, c) = w_j p_j X[j][c0 + c] as NP bf16 pieces, in the swizzled K-major
// smem image of each 64-source chunk: [chunk][piece][row c][128 B]. Rows c >= keff
// and padding slots are zero.
template <int NP>
__global__ void k_pack_q(GeomDev g, const double* __restrict__ X, int ldx, int c0, int keff,
                         const double* __restrict__ pre, int npad, int64_t nchunks, uint8_t* __restrict__ out) {
    // one thread per (chunk, row c, 8-source group)
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t total = nchunks * npad * 8;
    if (e >= total) return;
    const int gq = (int)(e & 7);
    const int c = (int)((e >> 3) % npad);
    const int64_t ch = (e >> 3) / npad;
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int64_t j = ch * KC + gq * 8 + q;
        double val = 0.0;
        const int64_t p = g.perm[j];
        if (p >= 0 && c < keff) val = g.sw[j] * (pre ? pre[p] : 1.0) * X[p * ldx + c0 + c];
        v[q] = (float)val;
    }
    uint32_t w[4][NP];
#pragma unroll
    for (int q = 0; q < 4; ++q) split_pieces<NP>(v[2 * q], v[2 * q + 1], w[q]);
    const size_t tile = (size_t)npad * 128;
    uint8_t* base = out + (size_t)ch * NP * tile;
    const uint32_t off = (uint32_t)c * 128u + ((((uint32_t)gq) ^ (uint32_t)(c & 7)) << 4);
#pragma unroll
    for (int p = 0; p < NP; ++p)
        *reinterpret_cast<uint4*>(base + p * tile + off) = make_uint4(w[0][p], w[1][p], w[2][p], w[3][p]);
}

// The kernel instance for npad columns in np pieces: generator threads a row (2: two CTAs per SM),
// columns a generator thread folds, Q-ring stages, shared memory.
struct Shape {
    int ctas, nq, cpq, sb;
    size_t smem;
};

size_t smem_bytes(int npad, int np, int stage, int sb) {
    const size_t b = (size_t)sb * np * npad * 2 * stage, c = (size_t)SC * 4 * kPeriod * sizeof(float);
    const size_t bars = (2 * SA + 2 * SBMAX + 2 * SC + 5) * sizeof(uint64_t) + 16;
    return kParamHead + 1024 + b + c + bars;
}

// Two CTAs per SM wherever their tensor memory (2 npad columns of accumulators and two stages of
// 64 sources in np pieces, 256 columns) holds them: up to 64 columns in two pieces, 32 in three.
// One CTA per SM, with the same number of generator warps but a common pace, takes 12 % longer
// there (42,048 nodes: 0.83 against 0.74 ms at 8 columns, 0.92 against 0.82 at 64).
Shape shape(int npad, int np) {
    const size_t half_sm = 113 * 1024, whole = 227 * 1024;  // 228 KB per SM, 1 KB reserved per CTA
    Shape sh;
    const bool two = 2 * npad + 2 * np * 32 <= 256;
    sh.ctas = two ? 2 : 1;
    sh.nq = two ? 2 : 4;
    sh.cpq = two ? (npad <= 16 ? 8 : (npad <= 32 ? 16 : 32)) : (npad <= 64 ? 16 : 32);
    const int stage = sh.nq * (np == 3 && sh.cpq == 32 ? 16 : 32);
    sh.sb = SBMAX;
    while (sh.sb > 2 && smem_bytes(npad, np, stage, sh.sb) > (two ? half_sm : whole)) --sh.sb;
    sh.smem = smem_bytes(npad, np, stage, sh.sb);
    return sh;
}

// Runs f(NQ, CPQ as integral constants) for the shape's kernel instance.
template <int NP, class F>
void with_instance(const Shape& sh, F&& f) {
    using std::integral_constant;
    if (sh.nq == 4 && sh.cpq == 32) return f(integral_constant<int, 4>(), integral_constant<int, 32>());
    if constexpr (NP == 3)
        if (sh.nq == 4) return f(integral_constant<int, 4>(), integral_constant<int, 16>());
    if (sh.cpq == 8) return f(integral_constant<int, 2>(), integral_constant<int, 8>());
    if (sh.cpq == 16) return f(integral_constant<int, 2>(), integral_constant<int, 16>());
    if constexpr (NP == 2) return f(integral_constant<int, 2>(), integral_constant<int, 32>());
}

template <int NP>
void pack_q(const GeomDev& g, const double* X, int ldx, int c0, int kc, const double* pre, uint8_t* bpack,
            cudaStream_t s) {
    const int npad = ((kc + 15) / 16) * 16;
    const int64_t nchunks = g.ns / KC;
    const int64_t pk = nchunks * npad * 8;
    k_pack_q<NP><<<(unsigned)((pk + 255) / 256), 256, 0, s>>>(g, X, ldx, c0, kc, pre, npad, nchunks, bpack);
    BIE_CK(cudaGetLastError());
}

template <int NP>
void launch_tc(const GeomDev& g, const double* X, int ldx, int c0, int kc, const double* pre, int nsplit, float* part,
               int ldp, uint8_t* bpack, int* err, cudaStream_t s) {
    const int npad = ((kc + 15) / 16) * 16;
    pack_q<NP>(g, X, ldx, c0, kc, pre, bpack, s);
    const Shape sh = shape(npad, NP);
    Params P;
    P.g = g;
    P.bpack = bpack;
    P.npad = npad;
    P.keff = kc;
    P.nsplit = nsplit;
    // BIE_TEST_TC_STALL (tests only): every CTA's first Q tile never arrives, so the
    // bounded waits expire quickly and the launch reports a timeout
    P.stall_test = std::getenv("BIE_TEST_TC_STALL") != nullptr;
    P.wait_limit = P.stall_test ? (1u << 14) : kWaitLimit;
    P.sb = sh.sb;
    P.part = part;
    P.ldp = ldp;
    P.c0 = c0;
    P.err = err;
    const dim3 grid((unsigned)(g.ns / M), (unsigned)nsplit);
    with_instance<NP>(sh, [&](auto nq, auto cpq) {
        const auto k = k_dt_tc<NP, nq.value, cpq.value>;
        ensure_smem_limit((const void*)k, sh.smem);
        k<<<grid, nthreads<nq.value>(), sh.smem, s>>>(P);
    });
    BIE_CK(cudaGetLastError());
}

// Work-list launch over the members' (tile, split) items; the shape (CTAs per SM, rings)
// is that of the widest member, the others run inside it.
template <int NP>
void launch_tc_list(const std::vector<TcMember>& ms, int* err, void* dscratch, size_t scratch_bytes, cudaStream_t s) {
    int npad_max = 16;
    for (const auto& m : ms) npad_max = std::max(npad_max, ((m.kc + 15) / 16) * 16);
    const Shape sh = shape(npad_max, NP);
    std::vector<Params> ps(ms.size());
    std::vector<int4> items;
    // members in the caller's order (largest first), each member's tiles x splits
    for (size_t m = 0; m < ms.size(); ++m) {
        const TcMember& t = ms[m];
        pack_q<NP>(t.g, t.X, t.ldx, t.c0, t.kc, t.pre, t.bpack, s);
        Params& P = ps[m];
        P.g = t.g;
        P.bpack = t.bpack;
        P.npad = ((t.kc + 15) / 16) * 16;
        P.keff = t.kc;
        P.nsplit = t.nsplit;
        P.stall_test = 0;
        P.wait_limit = kWaitLimit;
        P.sb = sh.sb;
        P.part = t.part;
        P.ldp = t.ldp;
        P.c0 = t.c0;
        P.err = err;
        const int tiles = (int)(t.g.ns / M);
        for (int sp = 0; sp < t.nsplit; ++sp)
            for (int ti = 0; ti < tiles; ++ti) items.push_back(make_int4((int)m, ti, sp, 0));
    }
    const size_t need = block_tc_list_bytes((int)ms.size(), (int64_t)items.size());
    if (need > scratch_bytes) throw Error(BIE_EINVAL, "launch_block_tc_list: work-list buffer too small");
    uint8_t* d = static_cast<uint8_t*>(dscratch);
    const size_t poff = 0, ioff = ((sizeof(Params) * ms.size() + 255) / 256) * 256;
    BIE_CK(cudaMemcpyAsync(d + poff, ps.data(), sizeof(Params) * ps.size(), cudaMemcpyHostToDevice, s));
    BIE_CK(cudaMemcpyAsync(d + ioff, items.data(), sizeof(int4) * items.size(), cudaMemcpyHostToDevice, s));
    // the host vectors are pageable: the copies are staged before cudaMemcpyAsync returns
    const Params* dp = reinterpret_cast<const Params*>(d + poff);
    const int4* di = reinterpret_cast<const int4*>(d + ioff);
    const dim3 grid((unsigned)items.size());
    with_instance<NP>(sh, [&](auto nq, auto cpq) {
        const auto k = k_dt_tc_list<NP, nq.value, cpq.value>;
        ensure_smem_limit((const void*)k, sh.smem);
        k<<<grid, nthreads<nq.value>(), sh.smem, s>>>(dp, di);
    });
    BIE_CK(cudaGetLastError());
}

}  // namespace tc

size_t block_tc_list_bytes(int nmembers, int64_t nitems) {
    return ((sizeof(tc::Params) * (size_t)nmembers + 255) / 256) * 256 + sizeof(int4) * (size_t)nitems;
}

void launch_block_tc_list(const std::vector<TcMember>& ms, int pieces, int* err, void* dscratch, size_t scratch_bytes,
                          cudaStream_t s) {
    if (ms.empty()) return;
    if (pieces == 3)
        tc::launch_tc_list<3>(ms, err, dscratch, scratch_bytes, s);
    else
        tc::launch_tc_list<2>(ms, err, dscratch, scratch_bytes, s);
}

int tc_npad(int kc) { return ((kc + 15) / 16) * 16; }

// Runs K3 for columns [c0, c0 + kc) (kc <= 128) of X into part[s][i][c0 + c],
// with the kernel and right-hand sides split into `pieces` (2: four products,
// 3: six products) bf16 pieces.
void launch_block_tc(const GeomDev& g, const double* X, int ldx, int c0, int kc, const double* pre, int nsplit,
                     float* part, int ldp, uint8_t* bpack, int* err, int pieces, cudaStream_t s) {
    if (pieces == 3)
        tc::launch_tc<3>(g, X, ldx, c0, kc, pre, nsplit, part, ldp, bpack, err, s);
    else
        tc::launch_tc<2>(g, X, ldx, c0, kc, pre, nsplit, part, ldp, bpack, err, s);
}

size_t block_tc_pack_bytes(int64_t slots, int kc, int pieces) {
    return (size_t)(slots / tc::KC) * pieces * tc_npad(kc) * 128;
}

int block_tc_ctas_per_sm(int kc, int pieces) {
    return tc::shape(tc_npad(kc), pieces).ctas;
}

}  // namespace bie
