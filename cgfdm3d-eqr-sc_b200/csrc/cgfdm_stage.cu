// Fused CGFDM Runge-Kutta stage for sm_100a.
//
// One launch does, for every interior point, what the reference does in up
// to fifteen launches per stage (src/propagate.cpp:212-251): the one-sided
// MacCormack derivatives with PML stretching (wave_deriv,
// src/wave_deriv.cpp:76-284), the traction-image free surface that
// overwrites the top three layers (free_surface_deriv,
// src/freeSurface.cpp:242-494), the CFS-PML auxiliary update and its
// correction of the RHS (pml_deriv_x/y/z, src/pml_deriv.cpp:125-584), the
// free-surface term of the PML auxiliaries (src/pml_freeSurface.cpp:16-242),
// and the RK4 update of both wavefield and auxiliaries (src/wave_rk.cpp:17-104,
// src/pml_rk.cpp:18-73).  In stage 3 it also updates the peak ground
// velocity (src/PGV.cpp:61-175) and, if enabled, the displacement
// (src/solve_displacement.cpp:27-63).
//
// Tiling: a CTA owns a 32 x 4 column tile and marches up a chunk of z.  Only
// the current plane needs its x/y halo: it arrives as one TMA box (40 x 8 x 1 x
// 9 floats, cp.async.bulk.tensor.4d) in a two-slot ring, and every plane of
// the one-sided z window as an interior column box (32 x 4 x 1 x 9) in a
// six-slot ring, completion tracked by one mbarrier per slot; one elected
// thread issues the copies one plane ahead of use.  (The ring pipeline of
// batches and linked parts brings every plane as a halo box in one six-slot
// ring.)  The FB signs are template parameters, so every stencil tap is a
// fixed shared-memory offset.  Metric, medium and RK inputs are plain
// coalesced loads issued before the ring wait.
//
// What bounds it: 400 x 400 x 200, the default build, moves 21.8 GB a step in
// 6.4 ms (3.4 TB/s of algorithmic bytes; DRAM at 37-56 % of its peak, issue
// slots 45-48 % full, the rest waits for memory with twelve warps an SM).
// Before the zero metric terms, the factored sums and the running sum's going
// it was 8.2 ms, 1174-1304 instructions a warp of points against 720-970 now.
//
// Every wait on an mbarrier is bounded: on timeout the CTA records the fact
// in a device error word, waits (bounded) for its copies in flight and exits.
//
// The exact build (CGFDM_EXACT, --fmad=false) follows the reference's
// expression order term by term and reproduces its FP32 results bit for bit;
// the default build factors the sums and ends the RK step without a running
// sum, and is no further from FP64.
#include <type_traits>

#include "cg_ops.cuh"
#include "device.cuh"
#include "kernels.cuh"
#include "tma.cuh"

// L2 promotion of the plane-ring (halo) and point-operand tensor maps, and
// which point operands are prefetched into L2 ahead of their loads.
#ifndef CG_PROMO_HALO
#define CG_PROMO_HALO CU_TENSOR_MAP_L2_PROMOTION_L2_256B
#endif
#ifndef CG_PROMO_POINT
#define CG_PROMO_POINT CU_TENSOR_MAP_L2_PROMOTION_L2_256B
#endif
#ifndef CG_PREFETCH_C
#define CG_PREFETCH_C 1
#endif
#ifndef CG_PREFETCH_MT
#define CG_PREFETCH_MT 1
#endif
// how many planes ahead the point operands are prefetched
#ifndef CG_PREFETCH_DIST
#define CG_PREFETCH_DIST 1
#endif
// RK4 without the running sum: the step ends from the step start and the
// three stage values, m + ((B - m) + 2 (C - m) + (D - m)) / 3 + h3 / 6, each in
// a buffer of its own.  A step then moves 149 floats a point instead of 176,
// and rounds less (the differences are exact where the stages are close).  The
// absorbing layers' auxiliaries, which no other point reads, need three
// buffers: stage 1 stores C over T and (B - m) + 2 (C - m) over B, stage 2 D
// over C, 117 floats a point instead of 144 (18 + 36 + 27 + 36).  The exact
// build keeps the reference's running sum T.
#ifdef CGFDM_EXACT
#define CG_RK_SUM 1
#else
#define CG_RK_SUM 0
#endif
// Cache policy of the point streams (used once per stage): 1 marks the
// stage-output and RK-sum stores evict-first, 2 also the metric, step-start
// and RK-sum loads, so L2 keeps the plane ring the neighbouring tiles share.
#ifndef CG_STREAM_HINTS
#define CG_STREAM_HINTS 1
#endif
#if CG_STREAM_HINTS >= 1
#define CG_ST(p, v) __stcs(&(p), (v))
#else
#define CG_ST(p, v) ((p) = (v))
#endif
// PML auxiliary stores: 1 evict-first like the stage outputs, 0 plain
// (400x400x200: 7.57 ms per step with 1, 7.51-7.57 with 0; evict-first
// loads as well, CG_STREAM_HINTS 2, took 8.32)
#ifndef CG_PML_STORE_HINT
#define CG_PML_STORE_HINT 0
#endif
#if CG_PML_STORE_HINT
#define CG_PST(p, v) __stcs(&(p), (v))
#else
#define CG_PST(p, v) ((p) = (v))
#endif
#if CG_STREAM_HINTS >= 2
#define CG_LD(p) __ldcs(&(p))
#else
#define CG_LD(p) (p)
#endif

// The file is compiled once per tile height -- CG_TILE_Y 4 (an inline
// namespace, so callers name its functions plainly) and 8 (namespace
// cgfdm::ty8); a session picks one -- and, the instantiations being many, in
// several objects: CG_STAGE_SET 0 batches and the tensor maps, 1 the split
// pipeline, 2 mixed storage, 3 halo-linked parts (1 to 3 with 4-row tiles
// only), 4 the ring pipeline of single sessions.
#ifndef CG_STAGE_SET
#define CG_STAGE_SET 0
#endif
#ifndef CG_TILE_NS
#define CG_TILE_NS ty4
#define CG_TILE_NS_INLINE inline
#else
#define CG_TILE_NS_INLINE
#endif

namespace cgfdm {
CG_TILE_NS_INLINE namespace CG_TILE_NS {

// 32 x 4 tiles, three CTAs per SM (12 warps, 168 registers): on 400 x 400 x
// 200 6.95 ms per step against 7.43 for 32 x 8 tiles at two CTAs of 128
// registers, which spill, and 7.07 for 128 threads of two points each in
// packed arithmetic (8 warps).
#ifndef CG_TILE_Y
#define CG_TILE_Y 4      // rows per tile (threads per CTA = 32 x CG_TILE_Y)
#endif
#ifndef CG_CTAS_PER_SM
#define CG_CTAS_PER_SM 3
#endif
#ifndef CG_SPLIT_CTAS_PER_SM
#define CG_SPLIT_CTAS_PER_SM CG_CTAS_PER_SM
#endif
#define TX 32
#define TY CG_TILE_Y
#define BXW 40           // box width: columns i0-4 .. i0+35 (start 16-byte aligned)
#define BYW (TY + 4)     // box height: one-sided y halo (1 behind, 3 ahead)
#define PF (BXW * BYW)   // floats per field in a slot
#define SLOT_F (9 * PF)  // floats per slot
#define SLOT_BYTES (SLOT_F * 4)
#define NSLOT 6
// split pipeline: the current plane's halo box in a 2-slot ring, the
// z-window's interior column boxes (32 x TY x 9) in a 6-slot ring (three and
// seven slots, a plane more ahead: 5 % slower)
#define CW (TX * TY)
#define CSLOT_F (9 * CW)
#define CSLOT_BYTES (CSLOT_F * 4)
#ifndef CG_SPLIT_HSLOTS
#define CG_SPLIT_HSLOTS 2   // halo ring: the current plane and CG_SPLIT_HSLOTS - 1 ahead
#endif
#ifndef CG_SPLIT_CSLOTS
#define CG_SPLIT_CSLOTS 6   // column ring: the 5-plane window and CG_SPLIT_CSLOTS - 5 ahead
#endif
#define NHSLOT CG_SPLIT_HSLOTS
#define NCSLOT CG_SPLIT_CSLOTS
#define SLOT_HB (9 * PF * 2)  // mixed storage: bytes of a slot's FP16 delta box
// Mixed storage: the ring also holds each plane's FP16 delta box, so a CTA
// needs 104 KB and two fit on an SM.
#ifndef CG_MIX_CTAS_PER_SM
#define CG_MIX_CTAS_PER_SM 2
#endif

// Slot strides: a TMA copy's shared-memory destination must be 128-byte
// aligned, so each slot starts on a 128-byte boundary whatever the box size
// (a 40 x 6 x 9 float box, the 2-row tile's, is 8640 bytes).
#define SLOT_SF ((SLOT_F + 31) / 32 * 32)          // floats between halo-box slots
#define CSLOT_SF ((CSLOT_F + 31) / 32 * 32)        // floats between column-box slots
#define SLOT_HSF ((9 * PF + 63) / 64 * 64)         // halves between FP16 delta-box slots
static_assert(SLOT_SF % 32 == 0 && CSLOT_SF % 32 == 0 && SLOT_HSF % 64 == 0 && CW % 32 == 0,
              "TMA destinations on 128-byte boundaries");

static size_t stage_smem(bool mix)
{
    return (size_t)NSLOT * (SLOT_SF * 4 + (mix ? SLOT_HSF * 2 : 0)) + NSLOT * 8;
}
static size_t stage2_smem()
{
    return (size_t)(NHSLOT * SLOT_SF + NCSLOT * CSLOT_SF) * 4 + (NHSLOT + NCSLOT) * 8;
}

// Stencil taps: hc points at this thread's cell of the current plane's halo
// box (x and y derivatives), zp[m] at its cell of plane k + FB3*(m-1) for the
// z derivative, ZS floats a field apart (the halo box itself in the ring
// pipeline, the interior column boxes in the split one).
template <int FB1, int FB2, int FB3, int ZS = PF>
struct Taps {
    const float *hc;
    const float *zp[5];
    __device__ __forceinline__ float rx(int f, float rDH) const
    {
        const float *c = hc + f * PF;
        return lop(c[-FB1], c[0], c[FB1], c[2 * FB1], c[3 * FB1], FB1, rDH);
    }
    __device__ __forceinline__ float ry(int f, float rDH) const
    {
        const float *c = hc + f * PF;
        return lop(c[-FB2 * BXW], c[0], c[FB2 * BXW], c[2 * FB2 * BXW], c[3 * FB2 * BXW], FB2, rDH);
    }
    __device__ __forceinline__ float rz(int f, float rDH) const
    {
        return lop(zp[0][f * ZS], zp[1][f * ZS], zp[2][f * ZS], zp[3][f * ZS], zp[4][f * ZS], FB3, rDH);
    }
    // unscaled sums: (FB * rDH) times these are the derivatives
    template <int DIR>
    __device__ __forceinline__ float sum(int f) const
    {
        const float *c = hc + f * PF;
        if constexpr (DIR == 0) return lsum(c[-FB1], c[0], c[FB1], c[2 * FB1], c[3 * FB1]);
        else if constexpr (DIR == 1)
            return lsum(c[-FB2 * BXW], c[0], c[FB2 * BXW], c[2 * FB2 * BXW], c[3 * FB2 * BXW]);
        else return lsum(zp[0][f * ZS], zp[1][f * ZS], zp[2][f * ZS], zp[3][f * ZS], zp[4][f * ZS]);
    }
    template <int DIR>
    __device__ __forceinline__ float rdir(int f, float rDH) const
    {
        return DIR == 0 ? rx(f, rDH) : DIR == 1 ? ry(f, rDH) : rz(f, rDH);
    }
    __device__ __forceinline__ float c(int f) const { return hc[f * PF]; }
    __device__ __forceinline__ float z(int m, int f) const { return zp[m][f * ZS]; }
};

// J * (metric row . stress) of a point, only the metric terms that are not
// zero on a grid of vertical columns (see xi_rhs)
template <class FW, class FC>
__device__ __forceinline__ void jt_point(int mdir, FW W, FC C, float jac, float out[3])
{
    if (mdir == 0) {
        const float m = C(C_XI_X);
        out[0] = (m * W(3)) * jac, out[1] = (m * W(6)) * jac, out[2] = (m * W(7)) * jac;
    } else if (mdir == 1) {
        const float m = C(C_ET_Y);
        out[0] = (m * W(6)) * jac, out[1] = (m * W(4)) * jac, out[2] = (m * W(8)) * jac;
    } else {
        const float m0 = C(C_ZT_X), m1 = C(C_ZT_Y), m2 = C(C_ZT_Z);
        const float Txy = W(6), Txz = W(7), Tyz = W(8);
        out[0] = ((m0 * W(3) + m1 * Txy) + m2 * Txz) * jac;
        out[1] = ((m0 * Txy + m1 * W(4)) + m2 * Tyz) * jac;
        out[2] = ((m0 * Txz + m1 * Tyz) + m2 * W(5)) * jac;
    }
}
// J * (metric . traction) at a point, for the traction image
// (src/freeSurface.cpp:358-395).  mdir: 0 xi, 1 eta, 2 zeta.
__device__ __forceinline__ void jt_at(const float *__restrict__ W, const float *__restrict__ cjm, long long F,
                                      long long q, int mdir, float out[3])
{
    const float jac = cjm[C_JAC * F + q];
    jt_point(
        mdir, [&](int f) { return W[f * F + q]; }, [&](int c) { return cjm[c * F + q]; }, jac, out);
}

// L_J_T along x or y (src/axis.h:264): taps at offsets FB*(-1..3).
__device__ __forceinline__ void ljt_xy(const float *__restrict__ W, const float *__restrict__ cjm, const DevGrid &g,
                                       int i, int j, int k, int dir, int FB, float rDH, float out[3])
{
    float J[5][3];
    for (int m = 0; m < 5; m++) {
        int o = (m - 1) * FB;
        long long q = dir == 0 ? g.at(i + o, j, k) : g.at(i, j + o, k);
        jt_at(W, cjm, g.fstride, q, dir, J[m]);
    }
    for (int c = 0; c < 3; c++) out[c] = lop(J[0][c], J[1][c], J[2][c], J[3][c], J[4][c], FB, rDH);
}

// L_J_T along zeta with the antisymmetric image about the surface
// (src/freeSurface.cpp:384-405): J[l] for l < k_s from the field,
// J[k_s] = 0, J[l] = -J[2 k_s - l] above.
__device__ __forceinline__ void ljt_z(const float *__restrict__ W, const float *__restrict__ cjm, const DevGrid &g,
                                      int i, int j, int k, int ks_rel, int FB, float rDH, float out[3])
{
    float J[5][3];
    for (int m = 0; m < 5; m++) {
        int l = 3 + (m - 1) * FB;
        int src = l, sign = 1;
        if (l > ks_rel) src = 2 * ks_rel - l, sign = -1;
        if (src == ks_rel) {
            J[m][0] = J[m][1] = J[m][2] = 0.0f;
        } else {
            jt_at(W, cjm, g.fstride, g.at(i, j, k + src - 3), 2, J[m]);
            if (sign < 0) J[m][0] = -J[m][0], J[m][1] = -J[m][1], J[m][2] = -J[m][2];
        }
    }
    for (int c = 0; c < 3; c++) out[c] = lop(J[0][c], J[1][c], J[2][c], J[3][c], J[4][c], FB, rDH);
}

// Mixed storage: the stage's stencil input at a point, the FP32 step-start
// state plus the FP16 delta times its inverse scale (stage 0: no delta).
struct MixIn {
    const float *W;
    const __half *S;
    const float *inv;
    DevGrid g, gh;
    __device__ __forceinline__ float operator()(int f, int i, int j, int k) const
    {
        const float v = W[f * g.fstride + g.at(i, j, k)];
        return S ? v + __half2float(S[f * gh.fstride + gh.at(i, j, k)]) * inv[f] : v;
    }
};

// jt_at, ljt_xy and ljt_z of the traction image on the mixed-storage input
__device__ __forceinline__ void jt_at_m(const MixIn &w, const float *__restrict__ cjm, int i, int j, int k, int mdir,
                                        float out[3])
{
    const long long F = w.g.fstride, q = w.g.at(i, j, k);
    jt_point(
        mdir, [&](int f) { return w(f, i, j, k); }, [&](int c) { return cjm[c * F + q]; }, cjm[C_JAC * F + q], out);
}

__device__ __forceinline__ void ljt_xy_m(const MixIn &w, const float *__restrict__ cjm, int i, int j, int k, int dir,
                                         int FB, float rDH, float out[3])
{
    float J[5][3];
    for (int m = 0; m < 5; m++) {
        const int o = (m - 1) * FB;
        jt_at_m(w, cjm, dir == 0 ? i + o : i, dir == 1 ? j + o : j, k, dir, J[m]);
    }
    for (int c = 0; c < 3; c++) out[c] = lop(J[0][c], J[1][c], J[2][c], J[3][c], J[4][c], FB, rDH);
}

__device__ __forceinline__ void ljt_z_m(const MixIn &w, const float *__restrict__ cjm, int i, int j, int k, int ks_rel,
                                        int FB, float rDH, float out[3])
{
    float J[5][3];
    for (int m = 0; m < 5; m++) {
        const int l = 3 + (m - 1) * FB;
        int src = l, sign = 1;
        if (l > ks_rel) src = 2 * ks_rel - l, sign = -1;
        if (src == ks_rel) {
            J[m][0] = J[m][1] = J[m][2] = 0.0f;
        } else {
            jt_at_m(w, cjm, i, j, k + src - 3, 2, J[m]);
            if (sign < 0) J[m][0] = -J[m][0], J[m][1] = -J[m][1], J[m][2] = -J[m][2];
        }
    }
    for (int c = 0; c < 3; c++) out[c] = lop(J[0][c], J[1][c], J[2][c], J[3][c], J[4][c], FB, rDH);
}

// RK4 without the running sum: stage irk's value (irk 0..2), the sum of the
// first two stages' differences and the step's end from the step start m, that
// sum bc and the last stage value d.  Every rounding is explicit, so the
// pipelines agree bit for bit.
__device__ __forceinline__ float rk_stage(int irk, float m, float h)
{
    return irk == 2 ? __fadd_rn(m, h) : __fmaf_rn(RK_ALPHA2, h, m);
}
__device__ __forceinline__ float rk_bc(float m, float b, float c)
{
    return __fmaf_rn(2.0f, __fsub_rn(c, m), __fsub_rn(b, m));
}
__device__ __forceinline__ float rk_end(float m, float bc, float d, float h)
{
    const float s = __fadd_rn(bc, __fsub_rn(d, m));
    return __fadd_rn(m, __fmaf_rn(RK_BETA4, h, __fmul_rn(RK_BETA2, s)));
}

// a delta to its stored FP16 value (scaled, saturated)
__device__ __forceinline__ __half to_h16(float x, float sc)
{
    return __float2half_rn(fminf(fmaxf(x * sc, -65504.0f), 65504.0f));
}

// ------------------------------------------------------------- the stage
// Persistent CTAs (three per SM) take work items -- one 32 x 4 column tile
// over one z-chunk -- from an atomic counter, chunks of a tile adjacent in
// the order, so concurrently running items share their halo and chunk-edge
// planes through L2 and no launch ends on a partial wave.
//
// BATCH = false: one session, its descriptor a kernel parameter (arguments
// and tensor maps in parameter space).  BATCH = true: the work items of
// nsess sessions, their descriptors in global memory; a CTA copies the
// arguments of the session its current item belongs to into shared memory.
//
// MIX = true: mixed-precision storage (see CgStageArgs).  Each slot also
// receives the plane's FP16 delta box; when a plane arrives, the CTA adds the
// delta into the FP32 box in place, so the taps read the stage's input as in
// the FP32 kernel.
//
// V2 = true: the split pipeline (see CSLOT_F above).
//
// IRK >= 0: the RK stage at compile time (a runtime stage spilled 200-300
// bytes a thread), -1: a.irk (batches with FP16 storage).
template <int FB1, int FB2, int FB3, bool BATCH, bool HOUT, bool MIX = false, bool V2 = false, int IRK = -1>
__global__ void __launch_bounds__(TX *TY, MIX  ? CG_MIX_CTAS_PER_SM
                                            : V2 ? CG_SPLIT_CTAS_PER_SM
                                                 : CG_CTAS_PER_SM)
    k_cg_stage(const __grid_constant__ CgStageDesc d1, const CgStageDesc *__restrict__ descs,
               const int *__restrict__ item_start, int nsess, int *work)
{
    static_assert(!(V2 && (BATCH || HOUT || MIX)), "the split pipeline is a single-session FP32 variant");
    extern __shared__ __align__(128) unsigned char smem_raw[];
    float *ring = reinterpret_cast<float *>(smem_raw);   // V2: the halo ring (2 slots)
    __half *ring16 = reinterpret_cast<__half *>(smem_raw + NSLOT * SLOT_SF * 4);
    float *col = ring + NHSLOT * SLOT_SF;                 // V2: column ring
    constexpr int NCS = V2 ? NCSLOT : NSLOT;              // column (V2) or ring slots
    unsigned long long *bars = reinterpret_cast<unsigned long long *>(
        V2 ? smem_raw + (NHSLOT * SLOT_SF + NCSLOT * CSLOT_SF) * 4
           : smem_raw + NSLOT * (SLOT_SF * 4 + (MIX ? SLOT_HSF * 2 : 0)));
    // barrier of column (V2) or ring slot s
    auto cbar = [&](int s) -> unsigned long long * { return V2 ? &bars[NHSLOT + s] : &bars[s]; };
    __shared__ int s_abort, s_item;
    __shared__ float s_sc[MIX ? 9 : 1], s_inv[MIX ? 9 : 1];
    __shared__ int s_par;
    __shared__ __align__(16) CgStageArgs s_args;
    const CgStageArgs &a = BATCH ? s_args : d1.a;
    const int tx = threadIdx.x, ty = threadIdx.y, tid = ty * TX + tx;
    constexpr int hyL = FB2 > 0 ? 1 : 3;
    constexpr int za = FB3 > 0 ? 1 : 3;
    const int cell = (ty + hyL) * BXW + tx + 4;
    const int total = BATCH ? item_start[nsess] : d1.a.ntiles_x * d1.a.ntiles_y * d1.a.nchunk * (V2 ? d1.a.sweeps : 1);
    int sess = -1;
    // mixed storage (one thread): per-field scales of this step from the
    // bounds of the session's step-start state -- the bound of field f
    // maps below 2^13
    auto mix_scales = [&](const CgStageArgs &A0) {
        const int p = *A0.it_dev & 1;
        s_par = p;
        float M[9], Mv = 0.0f, Ms = 0.0f;
        for (int f = 0; f < 9; f++) {
            M[f] = __uint_as_float(A0.mx[p * 9 + f]);
            if (f < 3 && M[f] > Mv) Mv = M[f];
            if (f >= 3 && M[f] > Ms) Ms = M[f];
        }
        for (int f = 0; f < 9; f++) {
            const float c = f < 3 ? Ms / A0.zs_min : Mv * A0.zp_max;
            const float b = M[f] > c ? M[f] : c;
            int e = 0;
            if (b > 0.0f) frexpf(b, &e);
            s_sc[f] = b > 0.0f ? ldexpf(1.0f, 13 - e) : 1.0f;
            s_inv[f] = b > 0.0f ? ldexpf(1.0f, e - 13) : 1.0f;
        }
    };
    // mixed storage, stage 3 (all threads): this CTA's maxima of the new
    // state raise the bounds of the session's next step
    auto mix_flush = [&](const CgStageArgs &A0, float *r) {
        if (A0.irk != 3) return;
#pragma unroll 1
        for (int f = 0; f < 9; f++) {
            float v = r[f];
            for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
            if ((tid & 31) == 0 && v > 0.0f) atomicMax(&A0.mx[(s_par ^ 1) * 9 + f], __float_as_uint(v));
            r[f] = 0.0f;
        }
    };

    if (tid == 0) {
        s_abort = 0;
        for (int s = 0; s < (V2 ? NHSLOT + NCSLOT : NSLOT); s++) mbar_init(smem_u32(&bars[s]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        if constexpr (MIX && !BATCH) {
            mix_scales(d1.a);
            // the next step's bounds start from zero; stage 3 raises them
            if (d1.a.irk == 0 && blockIdx.x == 0)
                for (int f = 0; f < 9; f++) d1.a.mx[((s_par) ^ 1) * 9 + f] = 0u;
        }
    }
    unsigned seq0 = 0;  // fills issued by this CTA before the current item
    unsigned hseq0 = 0;   // V2: halo-ring fills before the current item
    float rm[MIX ? 9 : 1];   // mixed storage, stage 3: running max |new state| per field
#pragma unroll
    for (int f = 0; f < (MIX ? 9 : 1); f++) rm[f] = 0.0f;

    // The split pipeline's items may be `sweeps` tiles high; their sweeps are
    // handed out one by one, so the sweeps of an item run side by side.
    const int sweeps = V2 ? d1.a.sweeps : 1;
    for (;;) {
    __syncthreads();
    if (tid == 0) s_item = atomicAdd(&work[0], 1);
    __syncthreads();
    const int gitem = s_item;
    if (gitem >= total || s_abort) break;
    if (BATCH) {
        // items of one session are consecutive; find this one's session
        int ns = 0;
        while (ns + 1 < nsess && gitem >= item_start[ns + 1]) ns++;
        if (ns != sess) {
            if constexpr (MIX) {
                // the previous session's maxima go to its bounds first
                if (sess >= 0) mix_flush(s_args, rm);
                __syncthreads();
            }
            sess = ns;
            const int *src = reinterpret_cast<const int *>(&descs[sess].a);
            int *dst = reinterpret_cast<int *>(&s_args);
            for (int w = tid; w < (int)(sizeof(CgStageArgs) / 4); w += TX * TY) dst[w] = src[w];
            __syncthreads();
            if constexpr (MIX) {
                if (tid == 0) {
                    mix_scales(s_args);
                    // the CTA with the session's first item resets its next
                    // step's bounds (stage 3, a later launch, raises them)
                    if (s_args.irk == 0 && gitem == item_start[sess])
                        for (int f = 0; f < 9; f++) s_args.mx[(s_par ^ 1) * 9 + f] = 0u;
                }
                __syncthreads();
            }
        }
    } else {
        sess = 0;
    }
    const CgStageDesc &D = BATCH ? descs[sess] : d1;
    const CUtensorMap *tmW = reinterpret_cast<const CUtensorMap *>(D.tmW);
    const CUtensorMap *tmC = reinterpret_cast<const CUtensorMap *>(D.tmC);
    const CUtensorMap *tmC1 = reinterpret_cast<const CUtensorMap *>(D.tmC1);
    const CUtensorMap *tmM = reinterpret_cast<const CUtensorMap *>(D.tmM);
    const CUtensorMap *tmT = reinterpret_cast<const CUtensorMap *>(D.tmT);
    const CUtensorMap *tmS = reinterpret_cast<const CUtensorMap *>(D.tmS);
    const CUtensorMap *tmWc = reinterpret_cast<const CUtensorMap *>(D.tmWc);
    const DevGrid g = a.g;
    const int irk = IRK >= 0 ? IRK : a.irk;
    const long long F = g.fstride;
    const int _nx = g.nxp - CGFDM_HALO, _ny = g.nyp - CGFDM_HALO, _nz = g.nzp - CGFDM_HALO;
    const float rDH = a.rDH, DT = a.DT;
    const int nPML = a.nPML;
    // position of point (ii, jj, kk) in the auxiliary arrays of PML face fc
    // (x faces: [z][y][x of the layer]; y faces: [z][y of the layer][x];
    // the z face: [z of the layer][y][x])
    auto pml_pos = [&](int fc, int ii, int jj, int kk) -> long long {
        const int ip = ii - CGFDM_HALO, jp = jj - CGFDM_HALO, kp = kk - CGFDM_HALO;
        if (fc == 0 || fc == 3)
            return (long long)(ip - (fc == 3 ? g.nx - nPML : 0)) + (long long)jp * nPML + (long long)kp * nPML * g.ny;
        if (fc == 1 || fc == 4)
            return (long long)ip + (long long)(jp - (fc == 4 ? g.ny - nPML : 0)) * g.nx +
                   (long long)kp * g.nx * nPML;
        return (long long)ip + (long long)jp * g.nx + (long long)kp * g.nx * g.ny;
    };
    // a face's auxiliaries at the stage's input: A, then B B B with a running
    // sum in T, or B T T without
    auto pml_in = [&](const PmlFace &P) -> const float * {
        if (CG_RK_SUM) return irk == 0 ? P.A : P.B;
        return irk == 0 ? P.A : irk == 1 ? P.B : P.T;
    };
    const int item = BATCH ? gitem - item_start[sess] : V2 ? gitem / sweeps : gitem;
    const int sweep = V2 ? gitem - item * sweeps : 0;
    const int tile = item / a.nchunk, chunk = item - tile * a.nchunk;
    const int by_ = tile / a.ntiles_x, bx_ = tile - by_ * a.ntiles_x;
    const int i0 = CGFDM_HALO + bx_ * TX, j0 = CGFDM_HALO + (by_ * sweeps + sweep) * TY;
    const int i = i0 + tx, j = j0 + ty;
    const bool active = i < _nx && j < _ny;
    const int kb = CGFDM_HALO + chunk * a.kchunk;
    const int ke = min(kb + a.kchunk, _nz);
    if (kb >= ke || j0 >= _ny) continue;
    const int kf = kb - za;                 // first plane this item loads
    const int tx0 = g.xoff + i0 - 4;        // halo box origin column: a multiple of 4 (16 bytes)
    const int ty0 = j0 - hyL;
    const int px0 = g.xoff + i0;            // point box origin column: a multiple of 4
    const int tx0h = MIX ? a.gh.xoff + i0 - 4 : 0;   // FP16 halo box origin: a multiple of 8 (16 bytes)

    // plane kk of this item is fill number seq0 + (kk - kf) of the CTA
    auto slot_of = [&](int kk) { return (int)((seq0 + (unsigned)(kk - kf)) % NCS); };
    auto parity_of = [&](int kk) { return ((seq0 + (unsigned)(kk - kf)) / NCS) & 1u; };
    // V2: halo box of plane kk (kb <= kk < ke)
    auto hslot_of = [&](int kk) { return (int)((hseq0 + (unsigned)(kk - kb)) % NHSLOT); };
    auto hparity_of = [&](int kk) { return ((hseq0 + (unsigned)(kk - kb)) / NHSLOT) & 1u; };
    auto issue_halo = [&](int kk) {
        const int hs = hslot_of(kk);
        const unsigned bar = smem_u32(&bars[hs]);
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        mbar_expect_tx(bar, SLOT_BYTES);
        tma_load_4d(smem_u32(ring + hs * SLOT_SF), tmW, tx0, ty0, kk, 0, bar);
    };
    auto issue = [&](int kk) {
        int s = slot_of(kk);
        unsigned bar = smem_u32(cbar(s));
        // test hook: leave this plane's slot without a copy (and without the
        // arrival that would complete its barrier phase), once
        if (a.stall && (BATCH ? gitem : item) == a.stall_item && sweep == 0 && kk - kf == a.stall_fill && atomicExch(a.stall, 0) == 1) return;
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        if constexpr (MIX) {
            const bool hs = irk != 0;
            mbar_expect_tx(bar, SLOT_BYTES + (hs ? SLOT_HB : 0));
            tma_load_4d(smem_u32(ring + s * SLOT_SF), tmW, tx0, ty0, kk, 0, bar);
            if (hs) tma_load_4d(smem_u32(ring16 + s * SLOT_HSF), tmS, tx0h, ty0, kk, 0, bar);
            return;
        }
        if constexpr (V2) {
            mbar_expect_tx(bar, CSLOT_BYTES);
            tma_load_4d(smem_u32(col + s * CSLOT_SF), tmWc, px0, j0, kk, 0, bar);
            return;
        }
        mbar_expect_tx(bar, SLOT_BYTES);
        tma_load_4d(smem_u32(ring + s * SLOT_SF), tmW, tx0, ty0, kk, 0, bar);
    };
    // point operands of plane kk into L2 ahead of their plain loads
    auto prefetch_points = [&](int kk) {
        if (CG_PREFETCH_C) {
            // the eight fields in use: xi_x, et_y, zt_x..z, mu, lambda, buoyancy
            tma_prefetch_4d(tmC1, px0, j0, kk, C_XI_X);
            tma_prefetch_4d(tmC1, px0, j0, kk, C_ET_Y);
            tma_prefetch_4d(tmC, px0, j0, kk, C_ZT_X);
            tma_prefetch_4d(tmC, px0, j0, kk, C_MU);
        }
        if constexpr (MIX) {
            // the step-start state in stages 1-3, the FP16 accumulator (halo map) in 2-3
            if (CG_PREFETCH_MT && irk != 0) tma_prefetch_4d(tmM, px0, j0, kk, 0);
            if (CG_PREFETCH_MT && irk >= 2) tma_prefetch_4d(tmT, tx0h, ty0, kk, 0);
            return;
        }
        // the step start; the running sum or, in the last stage, the other two
        // stage values
        if (CG_PREFETCH_MT && (irk == 1 || irk == 2 || (irk == 3 && !CG_RK_SUM))) tma_prefetch_4d(tmM, px0, j0, kk, 0);
        if (CG_PREFETCH_MT && (CG_RK_SUM ? irk != 0 : irk == 3)) tma_prefetch_4d(tmT, px0, j0, kk, 0);
        if (CG_PREFETCH_MT && !CG_RK_SUM && irk == 3) tma_prefetch_4d(tmS, px0, j0, kk, 0);
    };
    // mixed storage: the delta box of plane kk into its FP32 box, in place,
    // two values at a time (both boxes are [field][row][column], PF values a
    // field, so pair e of one is pair e of the other)
    auto convert = [&](int kk) {
        float2 *r32 = reinterpret_cast<float2 *>(ring + slot_of(kk) * SLOT_SF);
        const __half2 *r16 = reinterpret_cast<const __half2 *>(ring16 + slot_of(kk) * SLOT_HSF);
        for (int e = tid; e < 9 * PF / 2; e += TX * TY) {
            const float inv = s_inv[e / (PF / 2)];
            const float2 d = __half22float2(r16[e]);
            float2 w = r32[e];
            w.x = w.x + d.x * inv;
            w.y = w.y + d.y * inv;
            r32[e] = w;
        }
    };

    const long long wlim = a.wait_limit > 0 ? a.wait_limit : (1LL << 31);
    const int klast = ke - za + 3;          // last plane of the last window
    if (tid == 0) {
        for (int kk = kf; kk <= min(kf + NCS - 1, klast); kk++) issue(kk);
        if constexpr (V2) {
            for (int kk = kb; kk < min(kb + NHSLOT, ke); kk++) issue_halo(kk);
        }
        for (int kk = kb; kk < min(kb + CG_PREFETCH_DIST, ke); kk++) prefetch_points(kk);
    }
    int issued = min(kf + NCS - 1, klast);  // same value in every thread
    int hissued = min(kb + NHSLOT - 1, ke - 1);  // V2
    // the first window: planes kf .. kf+3 (kf+4 is waited for in the loop)
    bool ok = true;
    for (int kk = kf; kk < kf + 4; kk++) ok = ok && mbar_wait_bounded(smem_u32(cbar(slot_of(kk))), parity_of(kk), wlim);
    if (!ok) {
        s_abort = 1;
        atomicOr(a.err, 1);
    }
    if constexpr (MIX) {
        // (after a failed wait the values are unused: the loop head leaves)
        if (irk != 0)
            for (int kk = kf; kk < kf + 4; kk++) convert(kk);
    }

    const float bx = active ? a.pml_beta_x[i] : 1.0f, by = active ? a.pml_beta_y[j] : 1.0f;
    // pml_on: one bit per absorbing face, x1 y1 z1 x2 y2 (bits 0..4)
    const bool inx1 = (a.pml_on & 1) && i < CGFDM_HALO + nPML, inx2 = (a.pml_on & 8) && i >= _nx - nPML;
    const bool iny1 = (a.pml_on & 2) && j < CGFDM_HALO + nPML, iny2 = (a.pml_on & 16) && j >= _ny - nPML;

    for (int k = kb; k < ke; k++) {
        __syncthreads();                    // every thread is done with plane k - za - 1's slot
        if (s_abort) break;
        // issue plane k - za - 1 + NCS into the slot plane k - za - 1 has left
        const int want = k - za - 1 + NCS;
        if (want > issued && want <= klast) {
            if (tid == 0) issue(want);
            issued = want;
        }
        if constexpr (V2) {
            // the halo slot plane k - 1 has left takes plane k - 1 + NHSLOT
            if (k > kb && k - 1 + NHSLOT < ke) {
                if (tid == 0) issue_halo(k - 1 + NHSLOT);
                hissued = k - 1 + NHSLOT;
            }
        }
        if (tid == 0 && k + CG_PREFETCH_DIST < ke) prefetch_points(k + CG_PREFETCH_DIST);
        const long long q = g.at(i, j, k);
        // point-wise operands, loaded before the ring wait
        float xi_x = 0, et_y = 0, zt_x = 0, zt_y = 0, zt_z = 0;
        float mu = 0, lam = 0, buo = 0, bz = 1;
        float mv[9], tv[9], cv[9];   // step start; running sum, or B and C
        if (active) {
            xi_x = CG_LD(a.cjm[C_XI_X * F + q]), et_y = CG_LD(a.cjm[C_ET_Y * F + q]);
            zt_x = CG_LD(a.cjm[C_ZT_X * F + q]), zt_y = CG_LD(a.cjm[C_ZT_Y * F + q]);
            zt_z = CG_LD(a.cjm[C_ZT_Z * F + q]);
            mu = CG_LD(a.cjm[C_MU * F + q]), lam = CG_LD(a.cjm[C_LAMBDA * F + q]);
            buo = CG_LD(a.cjm[C_BUOY * F + q]) * 1.0f;  // buoyancy *= Crho (= 1)
            bz = a.pml_beta_z[k];
            if constexpr (MIX) {
                if (irk != 0)
                    for (int f = 0; f < 9; f++) mv[f] = a.Wm[f * F + q];
                if (irk >= 2) {
                    const long long qh = a.gh.at(i, j, k);
                    for (int f = 0; f < 9; f++) tv[f] = __half2float(a.T16[f * a.gh.fstride + qh]) * s_inv[f];
                }
            } else {
                if (irk == 1 || irk == 2 || (irk == 3 && !CG_RK_SUM))
                    for (int f = 0; f < 9; f++) mv[f] = CG_LD(a.Wm[f * F + q]);
                if (CG_RK_SUM && irk != 0)
                    for (int f = 0; f < 9; f++) tv[f] = CG_LD(a.T[f * F + q]);
                if (!CG_RK_SUM && irk == 3)
                    for (int f = 0; f < 9; f++) tv[f] = CG_LD(a.Wb[f * F + q]), cv[f] = CG_LD(a.Wc[f * F + q]);
            }
        }
        const int kk_new = k - za + 4;
        bool okw = mbar_wait_bounded(smem_u32(cbar(slot_of(kk_new))), parity_of(kk_new), wlim);
        if constexpr (V2) {
            okw = okw && mbar_wait_bounded(smem_u32(&bars[hslot_of(k)]), hparity_of(k), wlim);
        }
        if (!okw) {
            s_abort = 1;
            atomicOr(a.err, 1);
        }
        if constexpr (MIX) {
            if (irk != 0) {
                convert(kk_new);   // unused if a wait failed: the loop head then leaves
                __syncthreads();
                if (s_abort) continue;
            }
        }
        if (!okw) continue;
        if (!active) continue;

        Taps<FB1, FB2, FB3, V2 ? CW : PF> T;
        for (int m = 0; m < 5; m++) {
            int kk = k + FB3 * (m - 1);
            T.zp[m] = V2 ? col + slot_of(kk) * CSLOT_SF + ty * TX + tx : ring + slot_of(kk) * SLOT_SF + cell;
        }
        T.hc = V2 ? ring + hslot_of(k) * SLOT_SF + cell : T.zp[1];
        if (irk == 0)
            for (int f = 0; f < 9; f++) mv[f] = T.c(f);

        float h[9];
        const bool fs = a.fs_on && k >= _nz - 3;
        if (!fs) {
            // src/wave_deriv.cpp:214-282
#ifdef CGFDM_EXACT
            float d[9], c[9];
#pragma unroll
            for (int f = 0; f < 9; f++)
                if (CG_XI_NEEDS(f)) d[f] = T.rx(f, rDH) * bx;
            xi_rhs(xi_x, d, mu, lam, buo, c);
#pragma unroll
            for (int f = 0; f < 9; f++) h[f] = c[f];
#pragma unroll
            for (int f = 0; f < 9; f++)
                if (CG_ET_NEEDS(f)) d[f] = T.ry(f, rDH) * by;
            et_rhs(et_y, d, mu, lam, buo, c);
#pragma unroll
            for (int f = 0; f < 9; f++) h[f] = h[f] + c[f];
#pragma unroll
            for (int f = 0; f < 9; f++) d[f] = T.rz(f, rDH) * bz;
            dir_rhs(zt_x, zt_y, zt_z, d, mu, lam, buo, c);
#pragma unroll
            for (int f = 0; f < 9; f++) h[f] = (h[f] + c[f]) * DT;
#else
            // the scale of each direction's differences goes into its metric
            // row, the medium and DT onto the sums over the directions: about
            // 160 operations a point where the reference's order takes 330
            // (400x400x200, with the zero metric terms: 8.2 -> 7.4 ms per step)
            const float mx = xi_x * (FB1 * rDH * bx), my = et_y * (FB2 * rDH * by), sz = FB3 * rDH * bz;
            const float m0 = zt_x * sz, m1 = zt_y * sz, m2 = zt_z * sz;
            float e0, e1, e2;
            {
                const float s0 = T.template sum<0>(0), s1 = T.template sum<0>(1), s2 = T.template sum<0>(2);
                e0 = mx * s0, h[6] = mx * s1, h[7] = mx * s2;
                h[0] = mx * T.template sum<0>(3), h[1] = mx * T.template sum<0>(6), h[2] = mx * T.template sum<0>(7);
            }
            {
                const float s0 = T.template sum<1>(0), s1 = T.template sum<1>(1), s2 = T.template sum<1>(2);
                e1 = my * s1, h[6] += my * s0, h[8] = my * s2;
                h[0] += my * T.template sum<1>(6), h[1] += my * T.template sum<1>(4), h[2] += my * T.template sum<1>(8);
            }
            {
                const float s0 = T.template sum<2>(0), s1 = T.template sum<2>(1), s2 = T.template sum<2>(2);
                e0 += m0 * s0, e1 += m1 * s1, e2 = m2 * s2;
                h[6] += m1 * s0 + m0 * s1, h[7] += m2 * s0 + m0 * s2, h[8] += m2 * s1 + m1 * s2;
                const float t0 = T.template sum<2>(6), t1 = T.template sum<2>(7), t2 = T.template sum<2>(8);
                h[0] += m0 * T.template sum<2>(3) + m1 * t0 + m2 * t1;
                h[1] += m0 * t0 + m1 * T.template sum<2>(4) + m2 * t2;
                h[2] += m0 * t1 + m1 * t2 + m2 * T.template sum<2>(5);
            }
            const float bd = buo * DT, md = mu * DT, tr = (lam * DT) * (e0 + e1 + e2);
            h[0] *= bd, h[1] *= bd, h[2] *= bd;
            h[3] = tr + 2.0f * md * e0, h[4] = tr + 2.0f * md * e1, h[5] = tr + 2.0f * md * e2;
            h[6] *= md, h[7] *= md, h[8] *= md;
#endif
        } else {
            // src/freeSurface.cpp:345-492
            const int ks_rel = (_nz - 1) - k + CGFDM_HALO;
            float jx[3], jy[3], jz[3];
            if constexpr (MIX) {
                const MixIn w{a.Win, irk != 0 ? a.Sin : nullptr, s_inv, g, a.gh};
                ljt_xy_m(w, a.cjm, i, j, k, 0, FB1, rDH, jx);
                ljt_xy_m(w, a.cjm, i, j, k, 1, FB2, rDH, jy);
                ljt_z_m(w, a.cjm, i, j, k, ks_rel, FB3, rDH, jz);
            } else {
                ljt_xy(a.Win, a.cjm, g, i, j, k, 0, FB1, rDH, jx);
                ljt_xy(a.Win, a.cjm, g, i, j, k, 1, FB2, rDH, jy);
                ljt_z(a.Win, a.cjm, g, i, j, k, ks_rel, FB3, rDH, jz);
            }
            const float jinv = 1.0f / a.cjm[C_JAC * F + q];
            const float bj = buo * jinv;
            for (int c = 0; c < 3; c++) h[c] = (bj * ((jx[c] * bx + jy[c] * by) + jz[c])) * DT;
            float vxi[3], vet[3], vzt[3];
            for (int c = 0; c < 3; c++) vxi[c] = T.rx(c, rDH) * bx;
            for (int c = 0; c < 3; c++) vet[c] = T.ry(c, rDH) * by;
            if (k == _nz - 1) {
                const long long s = g.at2(i, j);
                if (a.vdstore)
                    for (int c = 0; c < 3; c++) {
                        a.vdstore[c * g.plane + s] = vxi[c];
                        a.vdstore[(3 + c) * g.plane + s] = vet[c];
                    }
                for (int r = 0; r < 3; r++) {
                    const float *dx = a.rdz + (long long)(r * 3) * g.plane + s;
                    const float *dy = a.rdz + (long long)(9 + r * 3) * g.plane + s;
                    vzt[r] = ((dx[0] * vxi[0] + dx[g.plane] * vxi[1]) + dx[2 * g.plane] * vxi[2]) +
                             ((dy[0] * vet[0] + dy[g.plane] * vet[1]) + dy[2 * g.plane] * vet[2]);
                }
            } else if (k == _nz - 2) {
                // L2: plane k + FB3 is tap m = 2
                for (int c = 0; c < 3; c++) vzt[c] = ((float)FB3 * (T.z(2, c) - T.z(1, c))) * rDH;
            } else {
                // L3: planes k, k + FB3, k + 2 FB3 are taps 1, 2, 3
                for (int c = 0; c < 3; c++)
                    vzt[c] = ((float)FB3 * ((CG_CF1 * T.z(1, c) + CG_CF2 * T.z(2, c)) +
                                            CG_CF3 * T.z(3, c))) *
                             rDH;
            }
            float s1[9], s2[9], s3[9];
            xi_stress(xi_x, vxi, mu, lam, s1);
            et_stress(et_y, vet, mu, lam, s2);
            dir_stress(zt_x, zt_y, zt_z, vzt, mu, lam, s3);
            for (int f = 3; f < 9; f++) h[f] = ((s1[f] + s2[f]) + s3[f]) * DT;
        }

        // ---- PML auxiliaries, faces in the reference's launch order x1 y1 z1 x2 y2
        // A point rarely lies in more than one: the loop over its faces stays
        // rolled, with one body per direction.
        const bool inz1 = (a.pml_on & 4) && k < CGFDM_HALO + nPML;
        auto face = [&](auto dirc, int fc) {
            constexpr int DIR = decltype(dirc)::value;
            // rhs is zero for Tyz in the x faces and for Txz in the y faces,
            // whose auxiliaries therefore stay zero but in the surface
            // layer: neither read nor written elsewhere
            const bool surf = a.fs_on && k == _nz - 1;
            auto on = [&](int f) { return DIR == 2 || f != (DIR == 0 ? 8 : 7) || surf; };
            const PmlFace &P = a.face[fc];
            const long long pos = pml_pos(fc, i, j, k);
            const float *al = DIR == 0 ? a.pml_alpha_x : DIR == 1 ? a.pml_alpha_y : a.pml_alpha_z;
            const float *dd = DIR == 0 ? a.pml_d_x : DIR == 1 ? a.pml_d_y : a.pml_d_z;
            const int ix = DIR == 0 ? i : DIR == 1 ? j : k;
            const float dval = dd[ix], beta = DIR == 0 ? bx : DIR == 1 ? by : bz, alpha_d = dval + al[ix];
            float d[9], rhs[9], aux[9], hA[9];
#ifdef CGFDM_EXACT
#pragma unroll
            for (int f = 0; f < 9; f++)
                if (DIR == 2 || (DIR == 0 ? CG_XI_NEEDS(f) : CG_ET_NEEDS(f))) d[f] = T.template rdir<DIR>(f, rDH) * dval;
#else
            const float sc = (DIR == 0 ? FB1 : DIR == 1 ? FB2 : FB3) * rDH * dval;
#pragma unroll
            for (int f = 0; f < 9; f++)
                if (DIR == 2 || (DIR == 0 ? CG_XI_NEEDS(f) : CG_ET_NEEDS(f))) d[f] = T.template sum<DIR>(f) * sc;
#endif
            if constexpr (DIR == 0) xi_rhs(xi_x, d, mu, lam, buo, rhs);
            else if constexpr (DIR == 1) et_rhs(et_y, d, mu, lam, buo, rhs);
            else dir_rhs(zt_x, zt_y, zt_z, d, mu, lam, buo, rhs);
            const float *cur = pml_in(P);
            constexpr bool SUM = CG_RK_SUM;
            const bool need_a = SUM ? irk == 1 || irk == 2 : irk != 0;   // the step start
            const bool need_t = SUM ? irk != 0 : irk == 3;               // the running sum, or that of stages 0, 1
            const float *pt = SUM ? P.T : P.B;
            // every operand of this face loaded before the first store: the
            // stores go through pointers the compiler cannot tell apart from
            // the loads, which would otherwise wait for them (8.24 ms per
            // step on 400x400x200 against 8.02 with them first).  Copying them
            // to shared memory during the stencil took more L1 from the point
            // loads than it hid: 64x60x48 0.127 ms per step with 27 floats a
            // thread, 0.108 without, 213x151x117 0.947 and 0.893.
            float xa[9], xt[9];
#pragma unroll
            for (int f = 0; f < 9; f++) aux[f] = on(f) ? cur[f * P.count + pos] : 0.0f;
            if (need_t)
#pragma unroll
                for (int f = 0; f < 9; f++) xt[f] = on(f) ? pt[f * P.count + pos] : 0.0f;
            if (need_a)
#pragma unroll
                for (int f = 0; f < 9; f++) xa[f] = on(f) ? P.A[f * P.count + pos] : 0.0f;
#pragma unroll
            for (int f = 0; f < 9; f++) hA[f] = (rhs[f] - alpha_d * aux[f]) * DT;
            if (DIR < 2 && surf) {
                // src/pml_freeSurface.cpp:90-125
                const long long s = g.at2(i, j);
                float vz[3], t3[9];
                for (int r = 0; r < 3; r++) {
                    const float *mr = a.rdz + (long long)(DIR * 9 + r * 3) * g.plane + s;
                    vz[r] = (mr[0] * d[0] + mr[g.plane] * d[1]) + mr[2 * g.plane] * d[2];
                }
                dir_stress(zt_x, zt_y, zt_z, vz, mu, lam, t3);
                for (int f = 3; f < 9; f++) hA[f] = hA[f] + t3[f] * DT;
            }
#pragma unroll
            for (int f = 0; f < 9; f++) h[f] = h[f] + (-beta * aux[f]) * DT;
            // src/pml_rk.cpp:18-73
#if CG_RK_SUM
            if (irk == 0) {
#pragma unroll
                for (int f = 0; f < 9; f++)
                    if (on(f)) {
                        CG_PST(P.T[f * P.count + pos], aux[f] + RK_BETA1 * hA[f]);
                        CG_PST(P.B[f * P.count + pos], aux[f] + RK_ALPHA2 * hA[f]);
                    }
            } else if (irk == 1 || irk == 2) {
#pragma unroll
                for (int f = 0; f < 9; f++)
                    if (on(f)) {
                        CG_PST(P.T[f * P.count + pos], xt[f] + (irk == 1 ? RK_BETA2 : RK_BETA3) * hA[f]);
                        CG_PST(P.B[f * P.count + pos], irk == 1 ? xa[f] + RK_ALPHA3 * hA[f] : xa[f] + hA[f]);
                    }
            } else {
#pragma unroll
                for (int f = 0; f < 9; f++)
                    if (on(f)) CG_PST(P.A[f * P.count + pos], xt[f] + RK_BETA4 * hA[f]);
            }
#else
            float *out = irk == 0 ? P.B : irk == 3 ? P.A : P.T;
#pragma unroll
            for (int f = 0; f < 9; f++) {
                if (!on(f)) continue;
                const float v = irk == 0   ? rk_stage(0, aux[f], hA[f])
                                : irk == 3 ? rk_end(xa[f], xt[f], aux[f], hA[f])
                                           : rk_stage(irk, xa[f], hA[f]);
                CG_PST(out[f * P.count + pos], v);
                if (irk == 1) CG_PST(P.B[f * P.count + pos], rk_bc(xa[f], aux[f], v));
            }
#endif
        };
        unsigned left = (inx1 ? 1u : 0u) | (iny1 ? 2u : 0u) | (inz1 ? 4u : 0u) | (inx2 ? 8u : 0u) | (iny2 ? 16u : 0u);
#pragma unroll 1
        while (left) {
            const int fc = __ffs(left) - 1;
            left &= left - 1;
            if (fc == 2) face(std::integral_constant<int, 2>{}, fc);
            else if (fc == 0 || fc == 3) face(std::integral_constant<int, 0>{}, fc);
            else face(std::integral_constant<int, 1>{}, fc);
        }

        // the adjoint's gradient reads h outside the PML layers only
        if (a.hstore && a.hbox.contains(i, j, k)) {
            const long long hq = a.hbox.at(i, j, k);
#pragma unroll
            for (int f = 0; f < 9; f++) a.hstore[f * a.hbox.fstride + hq] = h[f];
        }

        // ---- RK4 update of the wavefield (src/wave_rk.cpp:17-104)
        float wout[9];
        if constexpr (MIX) {
            // stage deltas d1 = h0 / 2, d2 = h1 / 2, d3 = h2 and the
            // accumulator delta t - m (b1 h0 = d1 / 3, formed in stage 1)
            const long long qh = a.gh.at(i, j, k), Fh = a.gh.fstride;
            if (irk == 0) {
#pragma unroll
                for (int f = 0; f < 9; f++) a.Sout[f * Fh + qh] = to_h16(RK_ALPHA2 * h[f], s_sc[f]);
            } else if (irk == 1) {
                const __half *cur16 = ring16 + slot_of(k) * SLOT_HSF + cell;
#pragma unroll
                for (int f = 0; f < 9; f++) {
                    const float d1 = __half2float(cur16[f * PF]) * s_inv[f];
                    a.T16[f * Fh + qh] = to_h16(d1 * 0.33333334f + RK_BETA2 * h[f], s_sc[f]);
                    a.Sout[f * Fh + qh] = to_h16(RK_ALPHA3 * h[f], s_sc[f]);
                }
            } else if (irk == 2) {
#pragma unroll
                for (int f = 0; f < 9; f++) {
                    a.T16[f * Fh + qh] = to_h16(tv[f] + RK_BETA3 * h[f], s_sc[f]);
                    a.Sout[f * Fh + qh] = to_h16(h[f], s_sc[f]);
                }
            } else {
#pragma unroll
                for (int f = 0; f < 9; f++) {
                    wout[f] = mv[f] + (tv[f] + RK_BETA4 * h[f]);
                    CG_ST(a.Wout[f * F + q], wout[f]);
                    rm[f] = fmaxf(rm[f], fabsf(wout[f]));
                }
            }
        } else {
#if CG_RK_SUM
        if (irk == 0) {
#pragma unroll
            for (int f = 0; f < 9; f++) {
                CG_ST(a.T[f * F + q], mv[f] + RK_BETA1 * h[f]);
                wout[f] = mv[f] + RK_ALPHA2 * h[f];
            }
        } else if (irk == 1) {
#pragma unroll
            for (int f = 0; f < 9; f++) {
                CG_ST(a.T[f * F + q], tv[f] + RK_BETA2 * h[f]);
                wout[f] = mv[f] + RK_ALPHA3 * h[f];
            }
        } else if (irk == 2) {
#pragma unroll
            for (int f = 0; f < 9; f++) {
                CG_ST(a.T[f * F + q], tv[f] + RK_BETA3 * h[f]);
                wout[f] = mv[f] + h[f];
            }
        } else {
#pragma unroll
            for (int f = 0; f < 9; f++) wout[f] = tv[f] + RK_BETA4 * h[f];
        }
#else
#pragma unroll
        for (int f = 0; f < 9; f++)
            wout[f] = irk == 3 ? rk_end(mv[f], rk_bc(mv[f], tv[f], cv[f]), T.c(f), h[f]) : rk_stage(irk, mv[f], h[f]);
#endif
#pragma unroll
        for (int f = 0; f < 9; f++) CG_ST(a.Wout[f * F + q], wout[f]);
        }
        if (HOUT) {
            // a part of a decomposed grid: the interior layers next to a face
            // shared with a neighbour go straight into the neighbour's halo
#pragma unroll 1
            for (int fc = 0; fc < 6; fc++) {
                const HaloOut &h = a.ho[fc];
                if (!h.base) continue;
                const int axis = fc >> 1;
                const int c = axis == 0 ? i : axis == 1 ? j : k;
                const int n = axis == 0 ? g.nx : axis == 1 ? g.ny : g.nz;
                if ((fc & 1) ? c < n : c >= 2 * CGFDM_HALO) continue;
                const long long d = (long long)(k + (axis == 2 ? h.shift : 0)) * h.plane +
                                    (long long)(j + (axis == 1 ? h.shift : 0)) * h.pitch + h.xoff +
                                    (i + (axis == 0 ? h.shift : 0));
#pragma unroll
                for (int f = 0; f < 9; f++) h.base[f * h.fstride + d] = wout[f];
            }
        }

        if (irk == 3) {
            // displacement: only the surface layer is ever read (the FreeSurfU
            // files, src/data_io.cpp:619-633), so only it is integrated
            if (a.dis && k == _nz - 1)
                for (int c = 0; c < 3; c++) a.dis[c * F + q] = a.dis[c * F + q] + wout[c] * DT;
            if (a.pgv && k == _nz - 1) {
                long long pp = (long long)(i - CGFDM_HALO) + (long long)(j - CGFDM_HALO) * g.nx;
                float Vx = wout[0], Vy = wout[1], Vz = wout[2];
                float Vh = sqrtf(Vx * Vx + Vy * Vy);
                float V = sqrtf(Vx * Vx + Vy * Vy + Vz * Vz);
                if (a.pgv[pp * 2 + 0] < Vh) a.pgv[pp * 2 + 0] = Vh;
                if (a.pgv[pp * 2 + 1] < V) a.pgv[pp * 2 + 1] = V;
            }
        }
    }
    __syncthreads();
    if (s_abort) {
        // no copy may still be landing in shared memory when the CTA exits
        if (tid == 0) {
            for (int kk = max(kf, issued - NCS + 1); kk <= issued; kk++)
                if (!mbar_wait_bounded(smem_u32(cbar(slot_of(kk))), parity_of(kk), wlim)) atomicOr(a.err, 2);
            if constexpr (V2) {
                for (int kk = max(kb, hissued - NHSLOT + 1); kk <= hissued; kk++)
                    if (!mbar_wait_bounded(smem_u32(&bars[hslot_of(kk)]), hparity_of(kk), wlim)) atomicOr(a.err, 2);
            }
        }
        break;
    }
    seq0 += (unsigned)(issued - kf + 1);
    hseq0 += (unsigned)(ke - kb);
    }  // work items

    if constexpr (MIX) {
        // stage 3: raise the bounds of the next step with this CTA's maxima
        if (!BATCH) mix_flush(d1.a, rm);
        else if (sess >= 0) mix_flush(s_args, rm);
    }
    // the last CTA out resets the work counter for the next launch
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        int done = atomicAdd(&work[1], 1);
        if (done == (int)(gridDim.x * gridDim.y * gridDim.z) - 1) {
            atomicExch(&work[0], 0);
            atomicExch(&work[1], 0);
            __threadfence();
        }
    }
}

// ------------------------------------------------------------ host side
template <int FB1, int FB2, int FB3, bool BATCH, bool HOUT, bool MIX, bool V2, int IRK>
static cudaError_t launch_t(const CgStageDesc &d1, const CgStageDesc *descs, const int *item_start, int nsess,
                            int *work, int ctas, cudaStream_t st)
{
    // The shared-memory limit is an attribute of the kernel on the current
    // device (and is lost with a device reset), so it is set on every launch:
    // a host-side call of about a microsecond, legal during stream capture.
    const size_t smem = V2 ? stage2_smem() : stage_smem(MIX);
    CUDA_TRY(cudaFuncSetAttribute(k_cg_stage<FB1, FB2, FB3, BATCH, HOUT, MIX, V2, IRK>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_cg_stage<FB1, FB2, FB3, BATCH, HOUT, MIX, V2, IRK>
        <<<ctas, dim3(TX, TY, 1), smem, st>>>(d1, descs, item_start, nsess, work);
    return cudaGetLastError();
}

// The instantiation for the FB signs (and the RK stage irk, -1: the kernel
// reads it from its arguments).
template <bool BATCH, bool HOUT, bool MIX, bool V2, int IRK>
static cudaError_t launch_fb(int FB1, int FB2, int FB3, const CgStageDesc &d1, const CgStageDesc *descs,
                             const int *item_start, int nsess, int *work, int ctas, cudaStream_t st)
{
    const int key = (FB1 > 0) * 4 + (FB2 > 0) * 2 + (FB3 > 0);
    switch (key) {
    case 0: return launch_t<-1, -1, -1, BATCH, HOUT, MIX, V2, IRK>(d1, descs, item_start, nsess, work, ctas, st);
    case 1: return launch_t<-1, -1, 1, BATCH, HOUT, MIX, V2, IRK>(d1, descs, item_start, nsess, work, ctas, st);
    case 2: return launch_t<-1, 1, -1, BATCH, HOUT, MIX, V2, IRK>(d1, descs, item_start, nsess, work, ctas, st);
    case 3: return launch_t<-1, 1, 1, BATCH, HOUT, MIX, V2, IRK>(d1, descs, item_start, nsess, work, ctas, st);
    case 4: return launch_t<1, -1, -1, BATCH, HOUT, MIX, V2, IRK>(d1, descs, item_start, nsess, work, ctas, st);
    case 5: return launch_t<1, -1, 1, BATCH, HOUT, MIX, V2, IRK>(d1, descs, item_start, nsess, work, ctas, st);
    case 6: return launch_t<1, 1, -1, BATCH, HOUT, MIX, V2, IRK>(d1, descs, item_start, nsess, work, ctas, st);
    default: return launch_t<1, 1, 1, BATCH, HOUT, MIX, V2, IRK>(d1, descs, item_start, nsess, work, ctas, st);
    }
}
template <bool BATCH, bool HOUT, bool MIX = false, bool V2 = false>
static cudaError_t launch_b(int FB1, int FB2, int FB3, const CgStageDesc &d1, const CgStageDesc *descs,
                            const int *item_start, int nsess, int *work, int ctas, cudaStream_t st, int irk)
{
    switch (irk) {
    case 0: return launch_fb<BATCH, HOUT, MIX, V2, 0>(FB1, FB2, FB3, d1, descs, item_start, nsess, work, ctas, st);
    case 1: return launch_fb<BATCH, HOUT, MIX, V2, 1>(FB1, FB2, FB3, d1, descs, item_start, nsess, work, ctas, st);
    case 2: return launch_fb<BATCH, HOUT, MIX, V2, 2>(FB1, FB2, FB3, d1, descs, item_start, nsess, work, ctas, st);
    default: return launch_fb<BATCH, HOUT, MIX, V2, 3>(FB1, FB2, FB3, d1, descs, item_start, nsess, work, ctas, st);
    }
}

#if CG_STAGE_SET == 1
int cg_stage_split_ctas_per_sm() { return CG_SPLIT_CTAS_PER_SM; }
cudaError_t launch_cg_stage_split(int FB1, int FB2, int FB3, const CgStageDesc &d, int *work, int ctas,
                                  cudaStream_t st)
{
    return launch_b<false, false, false, true>(FB1, FB2, FB3, d, nullptr, nullptr, 1, work, ctas, st, d.a.irk);
}
#elif CG_STAGE_SET == 3
cudaError_t launch_cg_stage_part(int FB1, int FB2, int FB3, const CgStageDesc &d, int *work, int ctas, cudaStream_t st)
{
    return launch_b<false, true, false, false>(FB1, FB2, FB3, d, nullptr, nullptr, 1, work, ctas, st, d.a.irk);
}
#elif CG_STAGE_SET == 4
cudaError_t launch_cg_stage(int FB1, int FB2, int FB3, const CgStageDesc &d, int *work, int ctas, cudaStream_t st)
{
    return launch_b<false, false, false, false>(FB1, FB2, FB3, d, nullptr, nullptr, 1, work, ctas, st, d.a.irk);
}
#elif CG_STAGE_SET == 2
cudaError_t launch_cg_stage_mix(int FB1, int FB2, int FB3, const CgStageDesc &d, int *work, int ctas, cudaStream_t st)
{
    return launch_b<false, false, true, false>(FB1, FB2, FB3, d, nullptr, nullptr, 1, work, ctas, st, d.a.irk);
}

cudaError_t launch_cg_stage_batch_mix(int FB1, int FB2, int FB3, const CgStageDesc *descs, const int *item_start,
                                      int nsess, int *work, int ctas, cudaStream_t st)
{
    static const CgStageDesc unused{};
    return launch_fb<true, false, true, false, -1>(FB1, FB2, FB3, unused, descs, item_start, nsess, work, ctas, st);
}
#else
int cg_stage_ctas_per_sm() { return CG_CTAS_PER_SM; }

#if CG_TILE_Y == 4
int cg_stage_mix_ctas_per_sm() { return CG_MIX_CTAS_PER_SM; }

cudaError_t make_field_tmap16(void *out, const __half *base, const DevGrid &gh, int nf)
{
    const auto encode = tmap_encoder();
    if (!encode) return cudaErrorNotSupported;
    cuuint64_t dims[4] = {(cuuint64_t)gh.pitch, (cuuint64_t)gh.nyp, (cuuint64_t)gh.nzp, (cuuint64_t)nf};
    cuuint64_t strides[3] = {(cuuint64_t)gh.pitch * 2, (cuuint64_t)gh.plane * 2, (cuuint64_t)gh.fstride * 2};
    cuuint32_t box[4] = {(cuuint32_t)BXW, (cuuint32_t)BYW, 1, (cuuint32_t)nf};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = encode(reinterpret_cast<CUtensorMap *>(out), CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 4, (void *)base, dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CG_PROMO_HALO,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Impedance bounds of the medium over the interior (float bits; the atomics
// order non-negative floats as their bit patterns): min sqrt(mu / b) into
// out[0], max sqrt((lambda + 2 mu) / b) into out[1].
__global__ void k_impedance_bounds(const float *__restrict__ cjm, DevGrid g, unsigned *out)
{
    const int i = blockIdx.x * 32 + threadIdx.x + CGFDM_HALO, j = blockIdx.y * 4 + threadIdx.y + CGFDM_HALO;
    const int k = blockIdx.z + CGFDM_HALO;
    float zs = 3.4e38f, zp = 0.0f;
    if (i < g.nxp - CGFDM_HALO && j < g.nyp - CGFDM_HALO) {
        const long long F = g.fstride, q = g.at(i, j, k);
        const float mu = cjm[C_MU * F + q], lam = cjm[C_LAMBDA * F + q], b = cjm[C_BUOY * F + q];
        zs = __fsqrt_rn(__fdiv_rn(mu, b));
        zp = __fsqrt_rn(__fdiv_rn(__fadd_rn(lam, __fmul_rn(2.0f, mu)), b));
    }
    for (int o = 16; o > 0; o >>= 1) {
        zs = fminf(zs, __shfl_xor_sync(0xffffffffu, zs, o));
        zp = fmaxf(zp, __shfl_xor_sync(0xffffffffu, zp, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&out[0], __float_as_uint(zs));
        atomicMax(&out[1], __float_as_uint(zp));
    }
}

cudaError_t launch_impedance_bounds(const float *cjm, DevGrid g, unsigned *out, cudaStream_t st)
{
    k_impedance_bounds<<<dim3((g.nx + 31) / 32, (g.ny + 3) / 4, g.nz), dim3(32, 4), 0, st>>>(cjm, g, out);
    return cudaGetLastError();
}

#endif

cudaError_t launch_cg_stage_batch(int FB1, int FB2, int FB3, int irk, const CgStageDesc *descs, const int *item_start,
                                  int nsess, int *work, int ctas, cudaStream_t st)
{
    static const CgStageDesc unused{};
    return launch_b<true, false, false, false>(FB1, FB2, FB3, unused, descs, item_start, nsess, work, ctas, st, irk);
}

cudaError_t make_field_tmap(void *out, const float *base, const DevGrid &g, int nf, bool halo_box, int box_nf)
{
    const auto encode = tmap_encoder();
    if (!encode) return cudaErrorNotSupported;
    cuuint64_t dims[4] = {(cuuint64_t)g.pitch, (cuuint64_t)g.nyp, (cuuint64_t)g.nzp, (cuuint64_t)nf};
    cuuint64_t strides[3] = {(cuuint64_t)g.pitch * 4, (cuuint64_t)g.plane * 4, (cuuint64_t)g.fstride * 4};
    cuuint32_t box[4] = {halo_box ? (cuuint32_t)BXW : (cuuint32_t)TX, halo_box ? (cuuint32_t)BYW : (cuuint32_t)TY, 1,
                         (cuuint32_t)(box_nf ? box_nf : nf)};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    CUresult r = encode(reinterpret_cast<CUtensorMap *>(out), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void *)base, dims,
                        strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                        halo_box ? CG_PROMO_HALO : CG_PROMO_POINT, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
#endif  // CG_STAGE_SET

}  // namespace CG_TILE_NS
}  // namespace cgfdm
