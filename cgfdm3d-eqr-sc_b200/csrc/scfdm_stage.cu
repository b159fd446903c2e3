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
#include "device.cuh"
#include "kernels.cuh"
#include "pair.cuh"
#include "sc_ops.cuh"

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
__device__ __forceinline__ F2 rcp2(F2 x)
{
    float a, b;
    unpk(x, a, b);
    asm("rcp.approx.f32 %0, %0;" : "+f"(a));
    asm("rcp.approx.f32 %0, %0;" : "+f"(b));
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
    const F2 r0 = rcp2(B0 * B0), r1 = rcp2(B1 * B1), r2 = rcp2(B2 * B2);
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

// The pass's use of the flux difference val of point q = (i, j, k): the x
// pass stores the RHS, the y pass adds to it, the z pass adds its part and
// applies the TVD-RK3 update (src/wave_rk_tvd.cpp:17-78), the sponge below
// the top four layers in the last stage, and carries the halo above the
// surface into the stage buffer in stages 0 and 1 (the reference's update
// runs over every point; halo points have a zero RHS and keep their value).
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

#ifndef CGFDM_EXACT
// The same for two neighbouring points (rows j, j+1 of the x pass, columns
// i, i+1 of the others); two: the second one is inside the grid.
template <int DIR>
__device__ __forceinline__ void epilogue2(const ScDirArgs &a, long long q, int i, int j, int k, bool two,
                                          const F2 val[9])
{
    const long long F = a.g.fstride;
    auto ld = [&](const float *p) { return SC_LD(*reinterpret_cast<const float2 *>(p)); };
    auto st = [&](float *p, float x, float y) {
        if (two) SC_ST(*reinterpret_cast<float2 *>(p), make_float2(x, y));
        else SC_ST(*p, x);
    };
    if (DIR == 0) {
#pragma unroll
        for (int v = 0; v < 9; v++) {
            float x, y;
            unpk(val[v], x, y);
            SC_ST(a.H[v * F + q], x);
            if (two) SC_ST(a.H[v * F + q + a.g.pitch], y);
        }
    } else if (DIR == 1) {
        F2 h[9];
#pragma unroll
        for (int v = 0; v < 9; v++) {
            const float2 w = ld(a.H + v * F + q);
            h[v] = pk(w.x, w.y) + val[v];
        }
#pragma unroll
        for (int v = 0; v < 9; v++) {
            float x, y;
            unpk(h[v], x, y);
            st(a.H + v * F + q, x, y);
        }
    } else {
        const int _nz = a.g.nzp - CGFDM_HALO;
        const bool decay = a.decay != nullptr && k < _nz - 4;
        auto rk = [&](float m, float w, float h) -> float {
            if (a.irk == 1)
                return __double2float_rn(__dadd_rn(__dadd_rn(__dmul_rn(0.75, (double)m), __dmul_rn(0.25, (double)w)),
                                                   __dmul_rn(0.25, (double)h)));
            return __double2float_rn(__dadd_rn(__dadd_rn(__dmul_rn(1.0 / 3.0, (double)m),
                                                         __dmul_rn(2.0 / 3.0, (double)w)),
                                               __dmul_rn(2.0 / 3.0, (double)h)));
        };
#pragma unroll 3
        for (int v = 0; v < 9; v++) {
            const float2 h0 = ld(a.H + v * F + q), w = *reinterpret_cast<const float2 *>(a.W + v * F + q);
            float2 m = make_float2(0.0f, 0.0f), o;
            if (a.irk != 0) m = ld(a.Wm + v * F + q);
            float hx, hy;
            unpk(pk(h0.x, h0.y) + val[v], hx, hy);
            if (a.irk == 0) o.x = w.x + hx, o.y = w.y + hy;
            else o.x = rk(m.x, w.x, hx), o.y = rk(m.y, w.y, hy);
            if (decay) {
                o.x = decay_apply(o.x, i, j, k, a.g, a.decay, a.ndecay);
                o.y = decay_apply(o.y, i + 1, j, k, a.g, a.decay, a.ndecay);
            }
            st(a.Wout + v * F + q, o.x, o.y);
        }
    }
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
#ifndef SC_TILE_MIN_CTAS
#define SC_TILE_MIN_CTAS 3
#endif
// shared memory of a tile: left and right states, 9 + 9 fields per position
constexpr size_t sc_tile_smem(int npos, int nl) { return sizeof(float) * 18 * npos * nl; }

#ifndef CGFDM_EXACT
template <int DIR, int NPOS, int NL>
__global__ void __launch_bounds__(SC_THREADS, SC_TILE_MIN_CTAS) k_sc_tile(const ScDirArgs a)
{
    constexpr int PR = NL / 2;                     // lane pairs
    constexpr int STEP = DIR == 0 ? 1 : PR;        // threads from one position to the next
    static_assert(NPOS * PR == SC_THREADS, "one position of one lane pair a thread");
    extern __shared__ __align__(16) unsigned char sm_raw[];
    F2 *sL = reinterpret_cast<F2 *>(sm_raw), *sR = sL + 9 * SC_THREADS;
    const DevGrid &g = a.g;
    const long long F = g.fstride;
    const int _nx = g.nxp - CGFDM_HALO, _ny = g.nyp - CGFDM_HALO, _nz = g.nzp - CGFDM_HALO;
    const int nd = DIR == 0 ? _nx : DIR == 1 ? _ny : _nz;  // points along the pass end before nd
    const long long stride = DIR == 0 ? 1 : DIR == 1 ? (long long)g.pitch : g.plane;
    const int tile = DIR == 0 ? blockIdx.x : DIR == 1 ? blockIdx.y : blockIdx.z;
    const int lane_end = DIR == 0 ? _ny : _nx;
    const int t = threadIdx.x;
    const int mi = DIR == 0 ? t % NPOS : t / PR, pr = DIR == 0 ? t / NPOS : t % PR;
    const int m = tile * (NPOS - 6) + mi;                                           // padded index along the pass
    const int lane = CGFDM_HALO + (DIR == 0 ? blockIdx.y : blockIdx.x) * NL + 2 * pr;
    const int i = DIR == 0 ? m : lane, j = DIR == 0 ? lane : DIR == 1 ? m : CGFDM_HALO + (int)blockIdx.y,
              k = DIR == 2 ? m : CGFDM_HALO + (int)blockIdx.z;
    // the pair's second lane may be the first halo lane of a row (read, never
    // written); columns lie on 8-byte boundaries (xoff 1, tiles of 16)
    const bool have = lane < lane_end, two = lane + 1 < lane_end;
    const long long q = g.at(i, j, k);
    auto ld = [&](const float *p) -> F2 {
        if constexpr (DIR == 0) return pk(__ldg(p), __ldg(p + g.pitch));
        else {
            const float2 w = __ldg(reinterpret_cast<const float2 *>(p));
            return pk(w.x, w.y);
        }
    };
    // ---- phase A: both WENO states of every position
    const bool face = have && mi < NPOS - 1 && m >= 2 && m < nd;
    F2 n[3], lam, mu, buo;
    if (face) {
        if constexpr (DIR < 2) n[0] = ld(a.cjm + (DIR == 0 ? C_XI_X : C_ET_Y) * F + q);
        else n[0] = ld(a.cjm + C_ZT_X * F + q), n[1] = ld(a.cjm + C_ZT_Y * F + q), n[2] = ld(a.cjm + C_ZT_Z * F + q);
        lam = ld(a.cjm + C_LAMBDA * F + q), mu = ld(a.cjm + C_MU * F + q), buo = ld(a.cjm + C_BUOY * F + q);
    }
    if (have && m >= 2 && m <= nd) {
        const float *w = a.W + q;
#pragma unroll 3
        for (int v = 0; v < 9; v++) {
            const float *wv = w + v * F;
            weno_pair(ld(wv - 2 * stride), ld(wv - stride), ld(wv), ld(wv + stride), ld(wv + 2 * stride),
                      sL[v * SC_THREADS + t], sR[v * SC_THREADS + t]);
        }
    }
    __syncthreads();

    // ---- phase B: Lax-Friedrichs flux of face m+1/2, stored over the left state
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
    __syncthreads();

    // ---- phase C: flux difference at the tile's points
    if (!have || mi < 3 || mi > NPOS - 4 || m >= nd) return;
    F2 val[9];
    const F2 coef = ld(a.sjac + q);   // DT * rDH / J
    if (k >= _nz - 3) {
        for (int l = 0; l < (two ? 2 : 1); l++) {
            float Fp[9], Fm[9], r[9], c[2];
            unpk(coef, c[0], c[1]);
            for (int v = 0; v < 9; v++) {
                float x[2];
                unpk(sL[v * SC_THREADS + t], x[0], x[1]);
                Fp[v] = l ? x[1] : x[0];
                unpk(sL[v * SC_THREADS + t - STEP], x[0], x[1]);
                Fm[v] = l ? x[1] : x[0];
            }
            const long long ql = q + l * (DIR == 0 ? g.pitch : 1);
            const int mc0 = DIR == 0 ? C_XI_X : DIR == 1 ? C_ET_X : C_ZT_X;
            surface_diff(a, ql, stride, mc0, l ? c[1] : c[0], Fp, Fm, r);
            epilogue<DIR>(a, ql, DIR == 0 ? i : i + l, DIR == 0 ? j + l : j, k, r);
        }
        return;
    }
    // faces p-5/2 .. p+5/2: the fourth- and sixth-order corrected flux is
    // Fh = c2 F-2 + c1 F-1 + c0 F0 + c1 F+1 + c2 F+2 with c0 = 6402/5760,
    // c1 = -348/5760, c2 = 27/5760; val = -coef (Fh[p] - Fh[p-1])
    const F2 e0 = pk(27.0f / 5760) * coef, e1 = pk((-348.0f - 27.0f) / 5760) * coef,
             e2 = pk((6402.0f + 348.0f) / 5760) * coef;
#pragma unroll
    for (int v = 0; v < 9; v++) {
        const F2 *f = sL + v * SC_THREADS + t;
        val[v] = fma2(e2, f[-STEP] - f[0], fma2(e1, f[-2 * STEP] - f[STEP], e0 * (f[-3 * STEP] - f[2 * STEP])));
    }
    epilogue2<DIR>(a, q, i, j, k, two, val);
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

template <int DIR, int NPOS, int NL>
static cudaError_t tile_attr()
{
    return cudaFuncSetAttribute(k_sc_tile<DIR, NPOS, NL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sc_tile_smem(NPOS, NL));
}

cudaError_t sc_dir_prepare()
{
    CUDA_TRY((tile_attr<0, SCX_NPOS, SCX_NL>()));
    CUDA_TRY((tile_attr<1, SCY_NPOS, SCY_NL>()));
    CUDA_TRY((tile_attr<2, SCY_NPOS, SCY_NL>()));
    return cudaSuccess;
}

cudaError_t launch_sc_dir(int dir, ScDirArgs a, const ScTiling &t, cudaStream_t st)
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
