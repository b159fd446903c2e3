// ME-AWENO (SCFDM) time stepping for sm_100a: alternative-flux WENO5
// finite differences, TVD-RK3, characteristic free surface and
// exponential-decay sponge.
//
// A TVD stage is three pencil kernels, one per grid direction.  Each CTA
// owns a tile of NPOS consecutive positions along its direction (the tile's
// points plus the 3 + 3 neighbours their flux differences reach) times NL
// lanes across it, and runs three phases through shared memory:
//
//   A  every position m computes, per variable, both WENO5-JS states that
//      are upwinded from the cell centred at m: the left state of face m+1/2
//      and the right state of face m-1/2 (src/alternative_flux_FD.cpp:42-59
//      called at 137-141).  The two states share their three smoothness
//      indicators, so they are computed once per position.
//   B  every face m+1/2 combines the left state of position m with the
//      right state of position m+1 into the Lax-Friedrichs flux, with the
//      metric and medium of point m (src/alternative_flux_FD.cpp:144-169).
//   C  every point takes the flux difference with the fourth- and
//      sixth-order corrections (cal_du_x/y/z, src/alternative_flux_FD.cpp:
//      1215-1435), or in the top three layers the variant built from point
//      fluxes (1257-1277).
//
// The x pass stores the RHS, the y pass adds to it and the z pass adds its
// part and applies the TVD-RK3 update (src/wave_rk_tvd.cpp:17-78), so the
// RHS accumulates in the reference's order.  After the third stage one
// kernel per surface column applies the characteristic free surface and
// extrapolates into the halo above it (src/freeSurface.cpp:40-194), the
// sponge factor of the top layers (src/exp_decay_absorb.cpp:19-106; the z
// pass of the last stage applies it below them) and the peak ground velocity
// (src/PGV.cpp:61-175).
//
// Faces the reference never writes -- along each direction those before
// index 2 and from _n on -- have zero flux, exactly as its zero-initialised
// flux buffer gives.  Halo points keep their values through a TVD stage, so
// stage buffers only need the top halo planes copied across.
//
// Built with CGFDM_EXACT (and --fmad=false) every float and double operation
// of phases A-C and of the RK update follows the reference's expression
// order, so the result is bit-identical.  The default build shares the
// smoothness indicators between the two states of a position, combines the
// two fluxes of a face before applying the (linear) flux function, and folds
// the flux-difference corrections into one six-tap filter.
#include <algorithm>
#include <cstring>

#include "device.cuh"
#include "kernels.cuh"
#include "pair.cuh"
#include "sc_ops.cuh"
#include "tma.cuh"

// 1: the passes' RHS and stage-output stores evict-first (each is read back
// by a later pass or stage, long after L2 has turned over)
#ifndef SC_STREAM_HINTS
#define SC_STREAM_HINTS 1
#endif
#if SC_STREAM_HINTS
#define SC_ST(p, v) __stcs(&(p), (v))
#else
#define SC_ST(p, v) ((p) = (v))
#endif
// 2: also the single-use loads of the RHS, the step-start state and DT rDH / J
#if SC_STREAM_HINTS >= 2
#define SC_LD(p) __ldcs(&(p))
#else
#define SC_LD(p) (p)
#endif

namespace cgfdm {

namespace {

constexpr int SC_THREADS = 256;

// ------------------------------------------------- two points at a time
#ifndef CGFDM_EXACT
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return vadd(a, b); }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return vsub(a, b); }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return vmul(a, b); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { return vfma(a, b, c); }
// (ftz: one instruction where the subnormal-safe form takes a compare, a
// select and two multiplications; weno_pair scales the arguments, so that no
// finite square of an indicator leads to a subnormal one)
__device__ __forceinline__ F2 rcp2(F2 x)
{
    float a, b;
    unpk(x, a, b);
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(a));
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(b));
    return pk(a, b);
}

// -1 / x
__device__ __forceinline__ F2 rcp2_neg(F2 x)
{
    float a, b;
    unpk(x, a, b);
    return rcp2(pk(-a, -b));
}

// ------------------------------------------------------------ WENO5-JS
// Both states upwinded from the cell centred at c, window a b c d e: uL at
// the face c+1/2, uR at the face c-1/2.  They share the Jiang-Shu indicators
// of the sub-stencils (a,b,c), (b,c,d), (c,d,e), 13/12 s^2 + 1/4 t^2 + 1e-6
// with s the second difference and t the slope, here times 12/13 (a common
// factor of the indicators cancels in the weights).  Everything is written in
// the cell differences d0..d3: the sub-stencils' states are c + q / 8 (uL)
// and c - q / 8 (uR), their weights 5/16, 10/16, 1/16 taken times 16/5.
__device__ __forceinline__ void weno_pair(F2 a, F2 b, F2 c, F2 d, F2 e, F2 &uL, F2 &uR)
{
    const F2 two = pk(2.0f), three = pk(3.0f), four = pk(4.0f), eight = pk(8.0f), fifth = pk(0.2f);
    const F2 k = pk(3.0f / 13.0f), eps = pk(1e-6f * 12.0f / 13.0f);
    const F2 d0 = b - a, d1 = c - b, d2 = d - c, d3 = e - d;
    const F2 s0 = d1 - d0, s1 = d2 - d1, n2 = d2 - d3;   // n2: minus the third second difference
    const F2 t0 = fma2(two, d1, s0), t1 = fma2(two, d1, s1), t2 = fma2(two, d2, n2);
    const F2 B0 = fma2(s0, s0, fma2(k * t0, t0, eps));
    const F2 B1 = fma2(s1, s1, fma2(k * t1, t1, eps));
    const F2 B2 = fma2(n2, n2, fma2(k * t2, t2, eps));
    // the squares scaled by 2^-60 (which cancels in the weights): between
    // 7e-31 and the 8e37 past which the reciprocal would be flushed to zero
    // and the weights 0/0 lie indicators up to 1e28.  Unscaled, indicators of
    // 9e18 were flushed (differences of 3e9 between neighbouring cells) where
    // squares in FP32 hold to 1.8e19.
    const F2 sc = pk(0x1p-60f);
    const F2 r0 = rcp2((sc * B0) * B0), r1 = rcp2((sc * B1) * B1), r2 = rcp2((sc * B2) * B2);
    const F2 wm = two * r1, far0 = fifth * r0, far2 = fifth * r2;
    // q of the face-side, centred and far sub-stencils
    const F2 nL = fma2(r2, fma2(four, d2, n2), fma2(wm, fma2(three, d2, d1), far0 * fma2(two, t0, s0)));
    const F2 nR = fma2(r0, fma2(four, d1, s0), fma2(wm, fma2(three, d1, d2), far2 * fma2(two, t2, n2)));
    const F2 m = eight * wm;
    uL = fma2(nL, rcp2(fma2(eight, r2, fma2(eight, far0, m))), c);
    uR = fma2(nR, rcp2_neg(fma2(eight, r0, fma2(eight, far2, m))), c);
}

// Lax-Friedrichs flux of a face from its left (uL) and right (uR) states,
// n the metric row's terms that are not zero on a grid of vertical columns
// (n[0]: y_eta z_zeta for xi, x_xi z_zeta for eta; all three for zeta).  The
// flux is linear in the state: f(uL) + f(uR) = f(uL + uR).
template <int DIR>
__device__ __forceinline__ void lf_flux(const F2 n[3], F2 lam, F2 mu, F2 buo, F2 ha, const F2 uL[9], const F2 uR[9],
                                        F2 F[9])
{
    F2 s[9];
    const F2 half = pk(-0.5f);
#pragma unroll
    for (int v = 0; v < 9; v++) {
        s[v] = uL[v] + uR[v];
        F[v] = ha * (uL[v] - uR[v]);
    }
    const F2 ltr = lam * ((s[3] + s[4]) + s[5]), m2 = mu + mu;
    const F2 n0 = half * n[0];
    if constexpr (DIR == 0) {
        const F2 nm = n0 * mu, nb = n0 * buo;
        F[0] = fma2(n0, fma2(m2, s[3], ltr), F[0]);
        F[1] = fma2(nm, s[8], F[1]), F[2] = fma2(nm, s[7], F[2]);
        F[3] = fma2(nb, s[0], F[3]), F[7] = fma2(nb, s[2], F[7]), F[8] = fma2(nb, s[1], F[8]);
    } else if constexpr (DIR == 1) {
        const F2 nm = n0 * mu, nb = n0 * buo;
        F[1] = fma2(n0, fma2(m2, s[4], ltr), F[1]);
        F[0] = fma2(nm, s[8], F[0]), F[2] = fma2(nm, s[6], F[2]);
        F[4] = fma2(nb, s[1], F[4]), F[6] = fma2(nb, s[2], F[6]), F[8] = fma2(nb, s[0], F[8]);
    } else {
        const F2 n1 = half * n[1], n2 = half * n[2];
        const F2 m0 = n0 * mu, m1 = n1 * mu, mm2 = n2 * mu, b0 = n0 * buo, b1 = n1 * buo, b2 = n2 * buo;
        F[0] = fma2(n0, fma2(m2, s[3], ltr), fma2(m1, s[8], fma2(mm2, s[7], F[0])));
        F[1] = fma2(n1, fma2(m2, s[4], ltr), fma2(m0, s[8], fma2(mm2, s[6], F[1])));
        F[2] = fma2(n2, fma2(m2, s[5], ltr), fma2(m0, s[7], fma2(m1, s[6], F[2])));
        F[3] = fma2(b0, s[0], F[3]), F[4] = fma2(b1, s[1], F[4]), F[5] = fma2(b2, s[2], F[5]);
        F[6] = fma2(b1, s[2], fma2(b2, s[1], F[6]));
        F[7] = fma2(b0, s[2], fma2(b2, s[0], F[7]));
        F[8] = fma2(b0, s[1], fma2(b1, s[0], F[8]));
    }
}
#else
// The reference's states and flux, term by term.
__device__ __forceinline__ void weno_pair(float a, float b, float c, float d, float e, float &uL, float &uR)
{
    uL = weno5_ref(a, b, c, d, e);
    uR = weno5_ref(e, d, c, b, a);
}
#endif

// Exponential-decay factor product of an interior point, in the
// reference's order x-low, x-high, y-low, y-high, z-low
// (src/exp_decay_absorb.cpp:36-92; free surface on, so no z-high layer).
__device__ __forceinline__ float decay_apply(float w, int i, int j, int k, const DevGrid &g, const float *G, int nl)
{
    const int X = i - CGFDM_HALO, Y = j - CGFDM_HALO, Z = k - CGFDM_HALO;
    if (X <= nl) w = w * G[nl - X];
    if (X >= g.nx - nl) w = w * G[nl - (g.nx - X)];
    if (Y <= nl) w = w * G[nl - Y];
    if (Y >= g.ny - nl) w = w * G[nl - (g.ny - Y)];
    if (Z <= nl) w = w * G[nl - Z];
    return w;
}

}  // namespace

#ifdef CGFDM_EXACT
// Flux difference of one point in the top three layers: the corrections
// come from point fluxes at p-3 .. p+3 along the direction
// (src/alternative_flux_FD.cpp:1253-1279).  Fp, Fm: fluxes of the faces
// p+1/2 and p-1/2.  Only three layers take this path, so it reads its
// operands from global memory.
__device__ __noinline__ void surface_diff(const ScDirArgs &a, long long q, long long stride, int mc0, float coef,
                                          const float *Fp, const float *Fm, float *val)
{
    const long long F = a.g.fstride;
    const float c24 = 1.0f / 24, c7 = 7.0f / 5760;
    float o2A[9], o4A[9], o2B[9], o4B[9];
    const float c2[6] = {-5.0f, 39.0f, -34.0f, -34.0f, 39.0f, -5.0f};
    const float c4[6] = {1.0f, -3.0f, 2.0f, 2.0f, -3.0f, 1.0f};
    for (int n = 0; n < 7; n++) {
        const long long qn = q + (n - 3) * stride;
        float u[9], hu[9];
#pragma unroll
        for (int v = 0; v < 9; v++) u[v] = a.W[v * F + qn];
        point_flux(a.cjm[(mc0 + 0) * F + qn], a.cjm[(mc0 + 1) * F + qn], a.cjm[(mc0 + 2) * F + qn],
                   a.cjm[C_LAMBDA * F + qn], a.cjm[C_MU * F + qn], a.cjm[C_BUOY * F + qn], u, hu);
#pragma unroll
        for (int v = 0; v < 9; v++) {
            // o2 = -5 u1 + 39 u2 - 34 u3 - 34 u4 + 39 u5 - 5 u6, o4 = u1 - 3 u2 + 2 u3 + 2 u4 - 3 u5 + u6,
            // accumulated left to right: B over hu[0..5], A over hu[1..6]
            if (n <= 5) {
                if (n == 0) o2B[v] = c2[0] * hu[v], o4B[v] = hu[v];
                else {
                    o2B[v] = c2[n] < 0.0f ? o2B[v] - (-c2[n]) * hu[v] : o2B[v] + c2[n] * hu[v];
                    o4B[v] = c4[n] < 0.0f ? o4B[v] - (-c4[n]) * hu[v] : (n == 5 ? o4B[v] + hu[v] : o4B[v] + c4[n] * hu[v]);
                }
            }
            if (n >= 1) {
                const int t = n - 1;
                if (t == 0) o2A[v] = c2[0] * hu[v], o4A[v] = hu[v];
                else {
                    o2A[v] = c2[t] < 0.0f ? o2A[v] - (-c2[t]) * hu[v] : o2A[v] + c2[t] * hu[v];
                    o4A[v] = c4[t] < 0.0f ? o4A[v] - (-c4[t]) * hu[v] : (t == 5 ? o4A[v] + hu[v] : o4A[v] + c4[t] * hu[v]);
                }
            }
        }
    }
#pragma unroll
    for (int v = 0; v < 9; v++) {
        const float A = Fp[v] - c24 * ((1.0f / 48) * o2A[v]) + c7 * ((1.0f / 2) * o4A[v]);
        const float B = Fm[v] - c24 * ((1.0f / 48) * o2B[v]) + c7 * ((1.0f / 2) * o4B[v]);
        val[v] = coef * (-(A - B));
    }
}
#endif

// The pass's use of the flux difference val of point q = (i, j, k): the x
// pass stores the RHS, the y pass adds to it, the z pass adds its part and
// applies the TVD-RK3 update (src/wave_rk_tvd.cpp:17-78), the sponge below
// the top four layers in the last stage, and carries the halo above the
// surface into the stage buffer in stages 0 and 1 (the reference's update
// runs over every point; halo points have a zero RHS and keep their value).
#ifdef CGFDM_EXACT
template <int DIR>
__device__ __forceinline__ void epilogue(const ScDirArgs &a, long long q, int i, int j, int k, const float val[9])
{
    const long long F = a.g.fstride;
    if (DIR == 0) {
#pragma unroll
        for (int v = 0; v < 9; v++) SC_ST(a.H[v * F + q], val[v]);
    } else if (DIR == 1) {
#pragma unroll
        for (int v = 0; v < 9; v++) SC_ST(a.H[v * F + q], SC_LD(a.H[v * F + q]) + val[v]);
    } else {
        const int _nz = a.g.nzp - CGFDM_HALO;
        const bool decay = a.decay != nullptr && k < _nz - 4;
#pragma unroll
        for (int v = 0; v < 9; v++) {
            const float h = SC_LD(a.H[v * F + q]) + val[v];
            const float w = a.W[v * F + q];
            float o;
            if (a.irk == 0) {
                o = w + h;
            } else if (a.irk == 1) {
                const double m = SC_LD(a.Wm[v * F + q]);
                o = __double2float_rn(__dadd_rn(__dadd_rn(__dmul_rn(0.75, m), __dmul_rn(0.25, (double)w)),
                                                __dmul_rn(0.25, (double)h)));
            } else {
                const double m = SC_LD(a.Wm[v * F + q]);
                o = __double2float_rn(__dadd_rn(__dadd_rn(__dmul_rn(1.0 / 3.0, m), __dmul_rn(2.0 / 3.0, (double)w)),
                                                __dmul_rn(2.0 / 3.0, (double)h)));
            }
            if (decay) o = decay_apply(o, i, j, k, a.g, a.decay, a.ndecay);
            SC_ST(a.Wout[v * F + q], o);
        }
        if (a.copy_halo && k == _nz - 1)
            for (int h = 1; h <= CGFDM_HALO; h++)
                for (int v = 0; v < 9; v++) a.Wout[v * F + q + h * a.g.plane] = a.W[v * F + q + h * a.g.plane];
    }
}
#else
// Two neighbouring points at once (rows j, j+1 of the x pass, columns i, i+1
// of the others); two: the second one is inside the grid.  val is the
// RHS so far with this pass's part, w0 the stage input.
template <int DIR>
__device__ __forceinline__ void epilogue2(const ScDirArgs &a, long long q, int i, int j, int k, bool two,
                                          const F2 val[9], const F2 w0[9])
{
    const long long F = a.g.fstride;
    auto st = [&](float *p, F2 v) {
        float x, y;
        unpk(v, x, y);
        if (DIR == 0) {
            SC_ST(*p, x);
            if (two) SC_ST(p[a.g.pitch], y);
        } else if (two) SC_ST(*reinterpret_cast<float2 *>(p), make_float2(x, y));
        else SC_ST(*p, x);
    };
    if (DIR < 2) {
#pragma unroll
        for (int v = 0; v < 9; v++) st(a.H + v * F + q, val[v]);
        return;
    }
    const int _nz = a.g.nzp - CGFDM_HALO;
    const bool decay = a.decay != nullptr && k < _nz - 4;
    auto rk = [&](float m, float w, float h) -> float {
        if (a.irk == 1)
            return __double2float_rn(__dadd_rn(__dadd_rn(__dmul_rn(0.75, (double)m), __dmul_rn(0.25, (double)w)),
                                               __dmul_rn(0.25, (double)h)));
        return __double2float_rn(__dadd_rn(__dadd_rn(__dmul_rn(1.0 / 3.0, (double)m), __dmul_rn(2.0 / 3.0, (double)w)),
                                           __dmul_rn(2.0 / 3.0, (double)h)));
    };
    float2 m[9];
    if (a.irk != 0)
#pragma unroll
        for (int v = 0; v < 9; v++) m[v] = SC_LD(*reinterpret_cast<const float2 *>(a.Wm + v * F + q));
#pragma unroll
    for (int v = 0; v < 9; v++) {
        F2 o;
        if (a.irk == 0) o = w0[v] + val[v];
        else {
            float wx, wy, hx, hy;
            unpk(w0[v], wx, wy);
            unpk(val[v], hx, hy);
            o = pk(rk(m[v].x, wx, hx), rk(m[v].y, wy, hy));
        }
        if (decay) {
            float x, y;
            unpk(o, x, y);
            o = pk(decay_apply(x, i, j, k, a.g, a.decay, a.ndecay), decay_apply(y, i + 1, j, k, a.g, a.decay, a.ndecay));
        }
        st(a.Wout + v * F + q, o);
    }
    if (a.copy_halo && k == _nz - 1)
#pragma unroll 1
        for (int h = 1; h <= CGFDM_HALO; h++)
#pragma unroll
            for (int v = 0; v < 9; v++) {
                const long long e = v * F + q + h * a.g.plane;
                const float2 w = *reinterpret_cast<const float2 *>(a.W + e);
                st(a.Wout + e, pk(w.x, w.y));
            }
}

// Flux difference val of two points in the top three layers, where the
// corrections come from point fluxes hu at p-3 .. p+3 along the direction
// (src/alternative_flux_FD.cpp:1253-1279).  With both faces' second and
// fourth differences collected,
//   val = -coef (Fp - Fm + (57 (hu[3] - hu[-3]) - 468 (hu[2] - hu[-2]) + 765 (hu[1] - hu[-1])) / 11520),
// Fp, Fm the fluxes of the faces p+1/2 and p-1/2: six linear fluxes summed
// into nine registers.  (Point by point with the reference's four sums of
// nine, the one warp of a z tile that holds the top layers kept the other
// seven waiting: 5.7 of 18.5 cycles an instruction at the barrier.)
template <int DIR, class LD>
__device__ __forceinline__ void surface_diff(const ScDirArgs &a, long long q, long long stride, F2 coef, const F2 *Fp,
                                             const F2 *Fm, LD ld, F2 val[9])
{
    const long long F = a.g.fstride;
    constexpr float w[6] = {-57.0f / 11520, 468.0f / 11520, -765.0f / 11520, 765.0f / 11520, -468.0f / 11520,
                            57.0f / 11520};
#pragma unroll
    for (int v = 0; v < 9; v++) val[v] = Fm[v * SC_THREADS] - Fp[v * SC_THREADS];
#pragma unroll 1
    for (int t = 0; t < 6; t++) {
        const long long qn = q + (t < 3 ? t - 3 : t - 2) * stride;
        const float *c = a.cjm + qn, *u = a.W + qn;
        const F2 lam = ld(c + C_LAMBDA * F), mu = ld(c + C_MU * F), buo = ld(c + C_BUOY * F), s = pk(w[t]);
        const F2 u0 = ld(u), u1 = ld(u + F), u2 = ld(u + 2 * F), u3 = ld(u + 3 * F), u4 = ld(u + 4 * F),
                 u5 = ld(u + 5 * F), u6 = ld(u + 6 * F), u7 = ld(u + 7 * F), u8 = ld(u + 8 * F);
        const F2 ltr = lam * ((u3 + u4) + u5), m2 = mu + mu;
        // -hu, the flux without its sign, times s
        if constexpr (DIR == 0) {
            const F2 n = s * ld(c + C_XI_X * F), nm = n * mu, nb = n * buo;
            val[0] = fma2(n, fma2(m2, u3, ltr), val[0]);
            val[1] = fma2(nm, u8, val[1]), val[2] = fma2(nm, u7, val[2]);
            val[3] = fma2(nb, u0, val[3]), val[7] = fma2(nb, u2, val[7]), val[8] = fma2(nb, u1, val[8]);
        } else if constexpr (DIR == 1) {
            const F2 n = s * ld(c + C_ET_Y * F), nm = n * mu, nb = n * buo;
            val[1] = fma2(n, fma2(m2, u4, ltr), val[1]);
            val[0] = fma2(nm, u8, val[0]), val[2] = fma2(nm, u6, val[2]);
            val[4] = fma2(nb, u1, val[4]), val[6] = fma2(nb, u2, val[6]), val[8] = fma2(nb, u0, val[8]);
        } else {
            const F2 n0 = s * ld(c + C_ZT_X * F), n1 = s * ld(c + C_ZT_Y * F), n2 = s * ld(c + C_ZT_Z * F);
            const F2 m0 = n0 * mu, m1 = n1 * mu, mm = n2 * mu, b0 = n0 * buo, b1 = n1 * buo, b2 = n2 * buo;
            val[0] = fma2(n0, fma2(m2, u3, ltr), fma2(m1, u8, fma2(mm, u7, val[0])));
            val[1] = fma2(n1, fma2(m2, u4, ltr), fma2(m0, u8, fma2(mm, u6, val[1])));
            val[2] = fma2(n2, fma2(m2, u5, ltr), fma2(m0, u7, fma2(m1, u6, val[2])));
            val[3] = fma2(b0, u0, val[3]), val[4] = fma2(b1, u1, val[4]), val[5] = fma2(b2, u2, val[5]);
            val[6] = fma2(b1, u2, fma2(b2, u1, val[6]));
            val[7] = fma2(b0, u2, fma2(b2, u0, val[7]));
            val[8] = fma2(b0, u1, fma2(b1, u0, val[8]));
        }
    }
#pragma unroll
    for (int v = 0; v < 9; v++) val[v] = coef * val[v];
}
#endif

// ------------------------------------------------------------ tiled pass
// Tiles of NPOS positions along the pass direction (the tile's NPOS - 6
// points and the neighbours their differences reach) times NL lanes across
// it: rows j for the x pass (grid: x tiles, row groups, k), columns i for
// the y and z passes (grid: column groups, y tiles, k / column groups, j,
// z tiles).  Three phases through shared memory:
//   A  both WENO states upwinded from every position,
//   B  the Lax-Friedrichs flux of every face, written over the left states,
//   C  the flux difference of every point and the pass's epilogue.
//
// The default build gives each of the 256 threads one position of two
// neighbouring lanes, packed (F2): 64 positions x 8 rows, 32 positions x 16
// columns.  The build that rounds every operation takes a lane at a time, in
// the reference's order.
#ifndef CGFDM_EXACT
constexpr int SCX_NPOS = 64, SCX_NL = 8;
#else
constexpr int SCX_NPOS = 64, SCX_NL = 4;
#endif
constexpr int SCY_NPOS = 32, SCY_NL = 16;
// two CTAs an SM: the 128 registers hold the epilogue's operands over a
// barrier (three at 80 registers, loading them after it: 17.1 against 14.9 ms
// per step on 384 x 384 x 192)
#ifndef SC_TILE_MIN_CTAS
#define SC_TILE_MIN_CTAS 2
#endif
// shared memory of a tile: left and right states, 9 + 9 fields per position
constexpr size_t sc_tile_smem(int npos, int nl) { return sizeof(float) * 18 * npos * nl; }

#ifndef CGFDM_EXACT
// The box of W a tile's states need, two more positions on either side: 72 x
// 8 rows (from a 16-byte boundary, so up to three columns early) for the x
// pass, 16 x 36 for the others; both 20736 bytes for the nine fields.
constexpr int SC_BOX_F = 36 * 16 * 9;
static_assert(SC_BOX_F == 72 * 8 * 9 && SC_BOX_F * 4 % 128 == 0, "one box size for the three passes");
constexpr size_t SC_PASS_SMEM = sizeof(float) * (SC_BOX_F + 2 * 18 * SC_THREADS) + 8;

// Persistent CTAs, two on an SM, walk the tiles in order.  A tile's box of
// W arrives by TMA while the tile before it is in phases B and C, and the
// values its epilogue adds to are loaded before the barrier that ends phase
// B, so the passes no longer wait for memory in every phase (with plain loads
// the z pass spent 7 of 12 cycles an instruction on them).
template <int DIR, int NPOS, int NL>
__global__ void __launch_bounds__(SC_THREADS, SC_TILE_MIN_CTAS) k_sc_tile(const __grid_constant__ ScPass p)
{
    constexpr int PR = NL / 2;                     // lane pairs
    constexpr int STEP = DIR == 0 ? 1 : PR;        // threads from one position to the next
    static_assert(NPOS * PR == SC_THREADS, "one position of one lane pair a thread");
    extern __shared__ __align__(128) unsigned char sm_raw[];
    float *sW = reinterpret_cast<float *>(sm_raw);
    F2 *sL = reinterpret_cast<F2 *>(sm_raw + SC_BOX_F * 4), *sR = sL + 9 * SC_THREADS;
    const unsigned bar = smem_u32(sR + 9 * SC_THREADS);
    const ScDirArgs &a = p.a;
    const DevGrid &g = a.g;
    const long long F = g.fstride;
    const int _nx = g.nxp - CGFDM_HALO, _ny = g.nyp - CGFDM_HALO, _nz = g.nzp - CGFDM_HALO;
    const int nd = DIR == 0 ? _nx : DIR == 1 ? _ny : _nz;  // points along the pass end before nd
    const long long stride = DIR == 0 ? 1 : DIR == 1 ? (long long)g.pitch : g.plane;
    const int lane_end = DIR == 0 ? _ny : _nx;
    const int t = threadIdx.x;
    const int mi = DIR == 0 ? t % NPOS : t / PR, pr = DIR == 0 ? t / NPOS : t % PR;
    // tile u: its number along the pass, lane group and plane (row for the z pass)
    auto split = [&](int u, int &tile, int &group, int &rest) {
        const int x = u % p.n0, y = u / p.n0 % p.n1, z = u / p.n0 / p.n1;
        if (DIR == 0) tile = x, group = y, rest = z;
        else if (DIR == 1) group = x, tile = y, rest = z;
        else group = x, rest = y, tile = z;
    };
    auto issue = [&](int u) {
        int tile, group, rest;
        if (p.stall && u == p.stall_tile && atomicExch(p.stall, 0) == 1) return;   // test hook
        split(u, tile, group, rest);
        const int m0 = tile * (NPOS - 6) - 2, l0 = CGFDM_HALO + group * NL, r = CGFDM_HALO + rest;
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        mbar_expect_tx(bar, SC_BOX_F * 4);
        if (DIR == 0) tma_load_4d(smem_u32(sW), p.tm, (g.xoff + m0) & ~3, l0, r, 0, bar);
        else if (DIR == 1) tma_load_4d(smem_u32(sW), p.tm, g.xoff + l0, m0, r, 0, bar);
        else tma_load_4d(smem_u32(sW), p.tm, g.xoff + l0, r, m0, 0, bar);
    };
    if (t == 0) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        issue(blockIdx.x);                         // the grid has no more CTAs than tiles
    }
    __syncthreads();
    const long long wlim = p.wait_limit > 0 ? p.wait_limit : (1LL << 31);
    unsigned phase = 0;
#pragma unroll 1
    for (int u = blockIdx.x; u < p.total; u += gridDim.x, phase ^= 1) {
        int tile, group, rest;
        split(u, tile, group, rest);
        const int m = tile * (NPOS - 6) + mi;                                       // padded index along the pass
        const int lane = CGFDM_HALO + group * NL + 2 * pr;
        const int i = DIR == 0 ? m : lane, j = DIR == 0 ? lane : DIR == 1 ? m : CGFDM_HALO + rest,
                  k = DIR == 2 ? m : CGFDM_HALO + rest;
        // the pair's second lane may be the first halo lane of a row (read, never
        // written); columns lie on 8-byte boundaries (xoff 1, tiles of 16)
        const bool have = lane < lane_end, two = lane + 1 < lane_end;
        const long long q = g.at(i, j, k);
        auto ld = [&](const float *x) -> F2 {
            if constexpr (DIR == 0) return pk(__ldg(x), __ldg(x + g.pitch));
            else {
                const float2 w = __ldg(reinterpret_cast<const float2 *>(x));
                return pk(w.x, w.y);
            }
        };
        const bool face = have && mi < NPOS - 1 && m >= 2 && m < nd;
        const bool point = have && mi >= 3 && mi <= NPOS - 4 && m < nd;
        // ---- phase A: both WENO states of every position
        const bool ok = mbar_wait_bounded(bar, phase, wlim);
        if (ok && have && m >= 2 && m <= nd) {
            // this position's value in the box, the next field SF and the next position SP floats on
            constexpr int SF = DIR == 0 ? 72 * NL : 36 * NL, SP = DIR == 0 ? 1 : NL;
            const float *w = DIR == 0 ? sW + 2 * pr * 72 + ((g.xoff + tile * (NPOS - 6) - 2) & 3) + mi + 2
                                      : sW + (mi + 2) * NL + 2 * pr;
            auto at = [&](int v, int o) -> F2 {
                const float *x = w + v * SF + o * SP;
                if constexpr (DIR == 0) return pk(x[0], x[72]);
                else {
                    const float2 y = *reinterpret_cast<const float2 *>(x);
                    return pk(y.x, y.y);
                }
            };
#pragma unroll 3
            for (int v = 0; v < 9; v++)
                weno_pair(at(v, -2), at(v, -1), at(v, 0), at(v, 1), at(v, 2), sL[v * SC_THREADS + t],
                          sR[v * SC_THREADS + t]);
        }
        // (in flight over the barrier)
        F2 n[3], lam, mu, buo;
        if (face) {
            if constexpr (DIR < 2) n[0] = ld(a.cjm + (DIR == 0 ? C_XI_X : C_ET_Y) * F + q);
            else n[0] = ld(a.cjm + C_ZT_X * F + q), n[1] = ld(a.cjm + C_ZT_Y * F + q), n[2] = ld(a.cjm + C_ZT_Z * F + q);
            lam = ld(a.cjm + C_LAMBDA * F + q), mu = ld(a.cjm + C_MU * F + q), buo = ld(a.cjm + C_BUOY * F + q);
        }
        if (__syncthreads_or(!ok)) {
            // a copy that did not arrive: nothing more is computed, and no copy
            // may still be landing in shared memory when the CTA exits
            if (t == 0) {
                atomicOr(p.err, 1);
                if (!mbar_wait_bounded(bar, phase, wlim)) atomicOr(p.err, 2);
            }
            __syncthreads();
            return;
        }
        if (t == 0 && u + (int)gridDim.x < p.total) issue(u + gridDim.x);

        // ---- phase B: Lax-Friedrichs flux of face m+1/2, stored over the left state
        {
            F2 Fv[9];
            if (face) {
                F2 uL[9], uR[9];
#pragma unroll
                for (int v = 0; v < 9; v++) uL[v] = sL[v * SC_THREADS + t], uR[v] = sR[v * SC_THREADS + t + STEP];
                lf_flux<DIR>(n, lam, mu, buo, pk(0.5f * a.alpha), uL, uR, Fv);
            } else {
#pragma unroll
                for (int v = 0; v < 9; v++) Fv[v] = pk(0.0f);
            }
#pragma unroll
            for (int v = 0; v < 9; v++) sL[v * SC_THREADS + t] = Fv[v];
        }
        F2 h[9], w0[9], coef;
        if (point) {
            coef = ld(a.sjac + q);   // DT * rDH / J
#pragma unroll
            for (int v = 0; v < 9; v++) {
                if (DIR > 0) {
                    const float2 x = SC_LD(*reinterpret_cast<const float2 *>(a.H + v * F + q));
                    h[v] = pk(x.x, x.y);
                }
                if (DIR == 2) {
                    const float2 x = *reinterpret_cast<const float2 *>(a.W + v * F + q);
                    w0[v] = pk(x.x, x.y);
                }
            }
        }
        __syncthreads();

        // ---- phase C: flux difference at the tile's points
        if (point) {
            F2 val[9];
            if (k >= _nz - 3) {
                surface_diff<DIR>(a, q, stride, coef, sL + t, sL + t - STEP, ld, val);
            } else {
                // faces p-5/2 .. p+5/2: the fourth- and sixth-order corrected flux is
                // Fh = c2 F-2 + c1 F-1 + c0 F0 + c1 F+1 + c2 F+2 with c0 = 6402/5760,
                // c1 = -348/5760, c2 = 27/5760; val = -coef (Fh[p] - Fh[p-1])
                const F2 e0 = pk(27.0f / 5760) * coef, e1 = pk((-348.0f - 27.0f) / 5760) * coef,
                         e2 = pk((6402.0f + 348.0f) / 5760) * coef;
#pragma unroll
                for (int v = 0; v < 9; v++) {
                    const F2 *f = sL + v * SC_THREADS + t;
                    val[v] = fma2(e2, f[-STEP] - f[0],
                                  fma2(e1, f[-2 * STEP] - f[STEP], e0 * (f[-3 * STEP] - f[2 * STEP])));
                }
            }
            if (DIR > 0)
#pragma unroll
                for (int v = 0; v < 9; v++) val[v] = h[v] + val[v];
            epilogue2<DIR>(a, q, i, j, k, two, val, w0);
        }
        __syncthreads();                           // the fluxes are read: the next tile's states may overwrite them
    }
}
#else
template <int DIR, int NPOS, int NL>
__global__ void __launch_bounds__(SC_THREADS, SC_TILE_MIN_CTAS) k_sc_tile(const ScDirArgs a)
{
    constexpr int P = NPOS - 6;
    extern __shared__ __align__(16) float sm[];
    float *sL = sm, *sR = sm + 9 * NPOS * NL;
    const DevGrid g = a.g;
    const long long F = g.fstride;
    const int _nx = g.nxp - CGFDM_HALO, _ny = g.nyp - CGFDM_HALO, _nz = g.nzp - CGFDM_HALO;
    const int nd = DIR == 0 ? _nx : DIR == 1 ? _ny : _nz;  // points along the pass end before nd
    const long long stride = DIR == 0 ? 1 : DIR == 1 ? (long long)g.pitch : g.plane;
    const int tile = DIR == 0 ? blockIdx.x : DIR == 1 ? blockIdx.y : blockIdx.z;
    const int p0 = CGFDM_HALO + tile * P;
    const int lane0 = CGFDM_HALO + (DIR == 0 ? blockIdx.y : blockIdx.x) * NL;
    const int lane_end = DIR == 0 ? _ny : _nx;
    const int jfix = DIR == 2 ? CGFDM_HALO + (int)blockIdx.y : 0;
    const int kfix = DIR == 2 ? 0 : CGFDM_HALO + (int)blockIdx.z;
    constexpr int mc0 = DIR == 0 ? C_XI_X : DIR == 1 ? C_ET_X : C_ZT_X;  // metric row of this direction

    auto coords = [&](int m, int lane, int &i, int &j, int &k) {
        if (DIR == 0) i = m, j = lane0 + lane, k = kfix;
        else if (DIR == 1) i = lane0 + lane, j = m, k = kfix;
        else i = lane0 + lane, j = jfix, k = m;
    };
    // consecutive threads take consecutive x: positions for the x pass, lanes otherwise
    auto sidx = [](int v, int mi, int lane) {
        return DIR == 0 ? (v * NL + lane) * NPOS + mi : (v * NPOS + mi) * NL + lane;
    };
    auto split = [](int it, int n_along, int &mi, int &lane) {
        if (DIR == 0) mi = it % n_along, lane = it / n_along;
        else lane = it % NL, mi = it / NL;
    };

    // ---- phase A: both WENO states of every position
    for (int it = threadIdx.x; it < NPOS * NL; it += SC_THREADS) {
        int mi, lane;
        split(it, NPOS, mi, lane);
        const int m = p0 - CGFDM_HALO + mi;
        if (lane0 + lane >= lane_end || m < 2 || m > nd) continue;
        int i, j, k;
        coords(m, lane, i, j, k);
        const float *w = a.W + g.at(i, j, k);
#pragma unroll 3
        for (int v = 0; v < 9; v++) {
            const float *wv = w + v * F;
            float uL, uR;
            weno_pair(__ldg(wv - 2 * stride), __ldg(wv - stride), __ldg(wv), __ldg(wv + stride), __ldg(wv + 2 * stride),
                      uL, uR);
            sL[sidx(v, mi, lane)] = uL;
            sR[sidx(v, mi, lane)] = uR;
        }
    }
    __syncthreads();

    // ---- phase B: Lax-Friedrichs flux of face m+1/2, stored over the left state
    for (int it = threadIdx.x; it < NPOS * NL; it += SC_THREADS) {
        int mi, lane;
        split(it, NPOS, mi, lane);
        const int m = p0 - CGFDM_HALO + mi;
        if (lane0 + lane >= lane_end || mi == NPOS - 1) continue;
        float Fv[9];
        if (m >= 2 && m < nd) {
            int i, j, k;
            coords(m, lane, i, j, k);
            const long long q = g.at(i, j, k);
            const float n0 = a.cjm[(mc0 + 0) * F + q], n1 = a.cjm[(mc0 + 1) * F + q], n2 = a.cjm[(mc0 + 2) * F + q];
            const float mu = a.cjm[C_MU * F + q], lam = a.cjm[C_LAMBDA * F + q], buo = a.cjm[C_BUOY * F + q];
            float uL[9], uR[9];
#pragma unroll
            for (int v = 0; v < 9; v++) uL[v] = sL[sidx(v, mi, lane)], uR[v] = sR[sidx(v, mi + 1, lane)];
            lf_flux_ref(n0, n1, n2, lam, mu, buo, a.alpha, uL, uR, Fv);
        } else {
#pragma unroll
            for (int v = 0; v < 9; v++) Fv[v] = 0.0f;
        }
#pragma unroll
        for (int v = 0; v < 9; v++) sL[sidx(v, mi, lane)] = Fv[v];
    }
    __syncthreads();

    // ---- phase C: flux difference at the tile's points
    for (int it = threadIdx.x; it < P * NL; it += SC_THREADS) {
        int pi, lane;
        split(it, P, pi, lane);
        const int p = p0 + pi;
        if (lane0 + lane >= lane_end || p >= nd) continue;
        int i, j, k;
        coords(p, lane, i, j, k);
        const long long q = g.at(i, j, k);
        const float coef = SC_LD(a.sjac[q]);  // DT * rDH / J
        float val[9];
        if (k >= _nz - 3) {
            float Fp[9], Fm[9];
#pragma unroll
            for (int v = 0; v < 9; v++) Fp[v] = sL[sidx(v, pi + 3, lane)], Fm[v] = sL[sidx(v, pi + 2, lane)];
            surface_diff(a, q, stride, mc0, coef, Fp, Fm, val);
        } else {
#pragma unroll
            for (int v = 0; v < 9; v++) {
                float f[6];
#pragma unroll
                for (int t = 0; t < 6; t++) f[t] = sL[sidx(v, pi + t, lane)];  // faces p-5/2 .. p+5/2
                val[v] = interior_diff_ref(f, coef);
            }
        }
        epilogue<DIR>(a, q, i, j, k, val);
    }
}
#endif

// --------------------------------------------------------- free surface
// One thread per surface column (src/freeSurface.cpp:40-194).  The
// characteristic condition is restated with the inverse of the basis
// B = [n s t]: T = B^-1 sigma B^-T and v' = B^-1 v are the stress and
// velocity in that basis; after the condition, sigma = B T B^T, v = B v'.
// Evaluated in double from the float fields and rounded once.
__global__ void k_sc_surface(float *W, const float *__restrict__ cjm, DevGrid g, const float *__restrict__ decayG,
                             int ndecay, float *pgv, float *dis, float DT)
{
    const int i = CGFDM_HALO + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = CGFDM_HALO + blockIdx.y * blockDim.y + threadIdx.y;
    const int _nx = g.nxp - CGFDM_HALO, _ny = g.nyp - CGFDM_HALO, _nz = g.nzp - CGFDM_HALO;
    if (i >= _nx || j >= _ny) return;
    const long long F = g.fstride;
    const long long q = g.at(i, j, _nz - 1);
    const float mu = cjm[C_MU * F + q], lam = cjm[C_LAMBDA * F + q], buo = cjm[C_BUOY * F + q];
    float u[9], o[9];
    for (int v = 0; v < 9; v++) u[v] = W[v * F + q];
    const float nrm[3] = {cjm[C_ZT_X * F + q], cjm[C_ZT_Y * F + q], cjm[C_ZT_Z * F + q]};
    const float tan1[3] = {cjm[C_X_XI * F + q], cjm[C_Y_XI * F + q], cjm[C_Z_XI * F + q]};
    const float tan2[3] = {cjm[C_X_ET * F + q], cjm[C_Y_ET * F + q], cjm[C_Z_ET * F + q]};
    char_surface_point(u, mu, lam, buo, cjm[C_JAC * F + q], nrm, tan1, tan2, o);
    for (int v = 0; v < 9; v++) W[v * F + q] = o[v];

    // cubic extrapolation into the three halo layers above
    // (src/freeSurface.cpp:180-190: extrap3 = 4 k1 - 6 k2 + 4 k3 - k4)
    for (int v = 0; v < 9; v++) {
        float *c = W + v * F + q;
        for (int h = 1; h <= CGFDM_HALO; h++) {
            const long long P = g.plane;
            c[h * P] = 4.0f * c[(h - 1) * P] - 6.0f * c[(h - 2) * P] + 4.0f * c[(h - 3) * P] - c[(h - 4) * P];
        }
    }

    // sponge factors of the top four layers (the z pass of the last stage
    // did the layers below; the extrapolation above used values before it)
    if (decayG)
        for (int k = max(CGFDM_HALO, _nz - 4); k < _nz; k++) {
            const long long qk = g.at(i, j, k);
            for (int v = 0; v < 9; v++) W[v * F + qk] = decay_apply(W[v * F + qk], i, j, k, g, decayG, ndecay);
        }

    // displacement, Dis += (momentum * buoyancy) * DT after the sponge
    // (src/solve_displacement.cpp:45-62, called at src/propagate.cpp:264-266).
    // Only the surface layer of Dis is ever read (the FreeSurfU files,
    // src/data_io.cpp:619-633), so only that layer is integrated.
    if (dis)
        for (int c = 0; c < 3; c++)
            dis[c * F + q] = __fadd_rn(dis[c * F + q], __fmul_rn(__fmul_rn(W[c * F + q], buo), DT));

    // peak ground velocity of the surface layer (src/PGV.cpp:115-137)
    if (pgv) {
        const float Vx = __fmul_rn(W[0 * F + q], buo), Vy = __fmul_rn(W[1 * F + q], buo),
                    Vz = __fmul_rn(W[2 * F + q], buo);
        const float Vh = __fsqrt_rn(__fadd_rn(__fmul_rn(Vx, Vx), __fmul_rn(Vy, Vy)));
        const float V = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(Vx, Vx), __fmul_rn(Vy, Vy)), __fmul_rn(Vz, Vz)));
        const long long pp = (long long)(i - CGFDM_HALO) + (long long)(j - CGFDM_HALO) * g.nx;
        if (pgv[pp * 2 + 0] < Vh) pgv[pp * 2 + 0] = Vh;
        if (pgv[pp * 2 + 1] < V) pgv[pp * 2 + 1] = V;
    }
}

// DT * rDH / J per interior point, as cal_du forms it (jac = 1.0 / CJM[9]
// in double, stored float; src/alternative_flux_FD.cpp:1251, 1283).
__global__ void k_sc_sjac(const float *__restrict__ cjm, DevGrid g, float DT, float rDH, float *sjac)
{
    const int i = CGFDM_HALO + blockIdx.x * blockDim.x + threadIdx.x;
    const int j = CGFDM_HALO + blockIdx.y * blockDim.y + threadIdx.y;
    const int k = CGFDM_HALO + blockIdx.z;
    if (i >= g.nxp - CGFDM_HALO || j >= g.nyp - CGFDM_HALO) return;
    const long long q = g.at(i, j, k);
    const float jac = __double2float_rn(__ddiv_rn(1.0, (double)cjm[C_JAC * g.fstride + q]));
    sjac[q] = __fmul_rn(__fmul_rn(DT, rDH), jac);
}

// ------------------------------------------------------------ launchers
ScTiling sc_tiling(const DevGrid &g)
{
    ScTiling t;
    t.npos[0] = SCX_NPOS, t.nl[0] = SCX_NL;
    t.ntiles[0] = (g.nx + SCX_NPOS - 7) / (SCX_NPOS - 6);
    t.npos[1] = t.npos[2] = SCY_NPOS, t.nl[1] = t.nl[2] = SCY_NL;
    t.ntiles[1] = (g.ny + SCY_NPOS - 7) / (SCY_NPOS - 6);
    t.ntiles[2] = (g.nz + SCY_NPOS - 7) / (SCY_NPOS - 6);
    return t;
}

#ifndef CGFDM_EXACT
// The tensor map of a nine-field buffer with the box of pass dir.
cudaError_t sc_tmap(void *out, const float *base, const DevGrid &g, int dir)
{
    const auto encode = tmap_encoder();
    if (!encode) return cudaErrorNotSupported;
    cuuint64_t dims[4] = {(cuuint64_t)g.pitch, (cuuint64_t)g.nyp, (cuuint64_t)g.nzp, 9};
    cuuint64_t strides[3] = {(cuuint64_t)g.pitch * 4, (cuuint64_t)g.plane * 4, (cuuint64_t)g.fstride * 4};
    cuuint32_t box[4] = {dir == 0 ? 72u : (cuuint32_t)SCY_NL, dir == 0 ? (cuuint32_t)SCX_NL : dir == 1 ? 36u : 1u,
                         dir == 2 ? 36u : 1u, 9};
    cuuint32_t estr[4] = {1, 1, 1, 1};
    const CUresult r = encode(reinterpret_cast<CUtensorMap *>(out), CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (void *)base,
                              dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int DIR, int NPOS, int NL>
static cudaError_t launch_pass(ScPass &p, int sms, cudaStream_t st)
{
    CUDA_TRY(cudaFuncSetAttribute(k_sc_tile<DIR, NPOS, NL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)SC_PASS_SMEM));
    const int grid = std::min(p.total, sms * SC_TILE_MIN_CTAS);
    k_sc_tile<DIR, NPOS, NL><<<grid, SC_THREADS, SC_PASS_SMEM, st>>>(p);
    return cudaGetLastError();
}

static int lane_groups(int dir, const DevGrid &g, const ScTiling &t)
{
    return ((dir == 0 ? g.ny : g.nx) + t.nl[dir] - 1) / t.nl[dir];
}

int sc_dir_tiles(int dir, const DevGrid &g, const ScTiling &t)
{
    return t.ntiles[dir] * lane_groups(dir, g, t) * (dir == 2 ? g.ny : g.nz);
}

cudaError_t launch_sc_dir(int dir, const ScDirArgs &a, const ScTiling &t, const unsigned char *tmap, int *err, int sms,
                          const ScStall &stall, cudaStream_t st)
{
    const DevGrid &g = a.g;
    ScPass p{};
    std::memcpy(p.tm, tmap, sizeof p.tm);
    p.a = a;
    p.err = err;
    p.stall = stall.dir == dir ? stall.stall : nullptr;
    p.stall_tile = stall.tile;
    p.wait_limit = stall.wait_limit;
    p.total = sc_dir_tiles(dir, g, t);
    const int along = t.ntiles[dir], groups = lane_groups(dir, g, t);
    if (dir == 0) {
        p.n0 = along, p.n1 = groups, p.n2 = g.nz;
        return launch_pass<0, SCX_NPOS, SCX_NL>(p, sms, st);
    }
    p.n0 = groups, p.n1 = dir == 1 ? along : g.ny, p.n2 = dir == 1 ? g.nz : along;
    return dir == 1 ? launch_pass<1, SCY_NPOS, SCY_NL>(p, sms, st) : launch_pass<2, SCY_NPOS, SCY_NL>(p, sms, st);
}
#else
cudaError_t sc_tmap(void *, const float *, const DevGrid &, int) { return cudaSuccess; }   // plain loads

int sc_dir_tiles(int, const DevGrid &, const ScTiling &) { return 0; }

cudaError_t launch_sc_dir(int dir, const ScDirArgs &a, const ScTiling &t, const unsigned char *, int *, int,
                          const ScStall &, cudaStream_t st)
{
    const DevGrid &g = a.g;
    if (dir == 0) {
        dim3 gr(t.ntiles[0], (g.ny + SCX_NL - 1) / SCX_NL, g.nz);
        k_sc_tile<0, SCX_NPOS, SCX_NL><<<gr, SC_THREADS, sc_tile_smem(SCX_NPOS, SCX_NL), st>>>(a);
    } else {
        const size_t smem = sc_tile_smem(SCY_NPOS, SCY_NL);
        if (dir == 1) {
            dim3 gr((g.nx + SCY_NL - 1) / SCY_NL, t.ntiles[1], g.nz);
            k_sc_tile<1, SCY_NPOS, SCY_NL><<<gr, SC_THREADS, smem, st>>>(a);
        } else {
            dim3 gr((g.nx + SCY_NL - 1) / SCY_NL, g.ny, t.ntiles[2]);
            k_sc_tile<2, SCY_NPOS, SCY_NL><<<gr, SC_THREADS, smem, st>>>(a);
        }
    }
    return cudaGetLastError();
}
#endif

cudaError_t launch_sc_surface(float *W, const float *cjm, DevGrid g, const float *decayG, int ndecay, float *pgv,
                              float *dis, float DT, cudaStream_t st)
{
    dim3 b(32, 4), gr((g.nx + 31) / 32, (g.ny + 3) / 4);
    k_sc_surface<<<gr, b, 0, st>>>(W, cjm, g, decayG, ndecay, pgv, dis, DT);
    return cudaGetLastError();
}

cudaError_t launch_sc_sjac(const float *cjm, DevGrid g, float DT, float rDH, float *sjac, cudaStream_t st)
{
    dim3 b(32, 8), gr((g.nx + 31) / 32, (g.ny + 7) / 8, g.nz);
    k_sc_sjac<<<gr, b, 0, st>>>(cjm, g, DT, rDH, sjac);
    return cudaGetLastError();
}

}  // namespace cgfdm
