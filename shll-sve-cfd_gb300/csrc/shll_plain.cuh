// Plain SHLL kernels: the reference's arithmetic, one fused launch per time step.
//
// Included by plain_fast.cu (compiled with fused multiply-add allowed: SHLL_PREC_F64) and by
// plain_exact.cu (compiled with -fmad=false: SHLL_PREC_F64_EXACT and SHLL_PREC_F32_EXACT,
// bit-identical to the reference's gcc builds).  SHLL_PLAIN_NS names the namespace.
//
// Each expression follows the reference's evaluation order and promotions:
//   Compute_P_from_U   base-c/base_shll.c:161-177, base-c/base_shll_2d.c:302-319
//   Compute_F_from_P   base-c/base_shll.c:130-159, base-c/base_shll_2d.c:239-300
//   Update_U_from_F    base-c/base_shll.c:87-128 (reflective walls), base-c/base_shll_2d.c:139-237,
//                      base-c/2nd_order_base_shll.c:203-459 (minmod slopes, outflow walls)
// D(x) widens an operand that the reference promotes to double (a double literal or sqrt()
// touches it); with REAL = double it is a no-op.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "exact_math.cuh"
#include "shll_internal.h"

namespace SHLL_PLAIN_NS {

#define D(x) ((double)(x))

// A grid constant (DT_ON_DX and the like), and whether it is a power of two (the reference's
// 0.25 / (R + 1)), so that products with it are exact.
template <typename REAL>
struct Factor {
    REAL v;
    bool pow2;
};
template <typename REAL>
__host__ Factor<REAL> make_factor(REAL v) {
    Factor<REAL> f;
    int ex = 0;
    f.v = v;
    f.pow2 = std::frexp((double)v, &ex) == 0.5 && ex > -500 && ex < 500;
    return f;
}

template <typename REAL>
struct Gas {
    REAL R, GAMMA, CV, DT_ON_DX, DT_ON_DY, alpha;
    int limiter;
    // derived (finish_gas)
    bool R_one;                                        // R == 1: products with it are skipped
    REAL gR;                                           // GAMMA * R
    REAL rCV;                                          // about 1 / CV (float arithmetic)
    exact_math::Divisor cv;                            // CV as a divisor (FP64 arithmetic)
    bool plain;                                        // the constants suit the cells' main path
    Factor<REAL> lx, ly, hlx, hly;                     // DT_ON_DX, DT_ON_DY and 0.5 times them
    Factor<REAL> sx, sy, hsx, hsy;                     // the same for fluxes as cell1 and cell2 scale them
};

// The split fluxes of cell1 and cell2 are kFluxScale times the reference's: in FP64 twice (the factors
// 0.5 of Z1, Z2 and Z3 are left out, and half the grid constants make up for it, all exactly).
template <typename REAL>
constexpr REAL kFluxScale = sizeof(REAL) == 8 ? (REAL)2 : (REAL)1;

template <typename REAL>
__host__ void finish_gas(Gas<REAL>& g) {
    g.R_one = g.R == (REAL)1;
    g.gR = g.GAMMA * g.R;
    g.rCV = (REAL)1 / g.CV;
    g.cv = exact_math::divisor((double)g.CV);
    g.lx = make_factor<REAL>(g.DT_ON_DX);
    g.ly = make_factor<REAL>(g.DT_ON_DY);
    g.hlx = make_factor<REAL>((REAL)0.5 * g.DT_ON_DX);
    g.hly = make_factor<REAL>((REAL)0.5 * g.DT_ON_DY);
    g.sx = make_factor<REAL>(g.DT_ON_DX / kFluxScale<REAL>);
    g.sy = make_factor<REAL>(g.DT_ON_DY / kFluxScale<REAL>);
    g.hsx = make_factor<REAL>((REAL)0.5 * g.DT_ON_DX / kFluxScale<REAL>);
    g.hsy = make_factor<REAL>((REAL)0.5 * g.DT_ON_DY / kFluxScale<REAL>);
    const double c[3] = {(double)g.CV, (double)g.R, (double)g.gR};
    g.plain = true;
    for (double v : c) g.plain = g.plain && v > 1e-9 && v < 1e9;
}

template <typename REAL>
__host__ Gas<REAL> make_gas(const PlainArgs& a) {
    Gas<REAL> g;
    g.R = (REAL)a.R; g.GAMMA = (REAL)a.GAMMA; g.CV = (REAL)a.CV;
    g.DT_ON_DX = (REAL)a.DT_ON_DX; g.DT_ON_DY = (REAL)a.DT_ON_DY;
    g.alpha = (REAL)a.mc_alpha; g.limiter = a.limiter;
    finish_gas(g);
    return g;
}

// ---- the reference's expressions, FP64 ----
// FP64 instructions are the scarce resource of these kernels (19 clocks per warp instruction per
// SM), so divisions, square roots, comparisons and power-of-two scalings run on the integer pipes
// (exact_math.cuh) with the same results; the float arithmetic does without FP64.  Measured, by
// itself: one 2D step of 256 x 256 cells in FP64 40.3 -> 25.9 us, of 301 x 277 in float (second order)
// 29.5 -> 13.4 us, one 1D step of 3001 cells (FP64, second order) 20.5 -> 16.4 us; with the tile kernel
// and the 1D runs of plain_resident.cuh these are 13.7, 7.6 and 2.4 us.
__device__ __forceinline__ double half_of(double x) { return exact_math::scale_pow2(x, -1, 0.5); }
__device__ __forceinline__ float half_of(float x) { return 0.5f * x; }
// 0.5 * (x + c) (the scaling is exact: one fused operation rounds like the sum)
__device__ __forceinline__ double half_sum(double x, double c) { return __fma_rn(0.5, x, 0.5 * c); }
__device__ __forceinline__ float half_sum(float x, float c) { return __fmul_rn(0.5f, __fadd_rn(x, c)); }
__device__ __forceinline__ bool positive(double x) {
    const long long b = __double_as_longlong(x);
    return b > 0 && b <= 0x7ff0000000000000ll;
}
__device__ __forceinline__ bool positive(float x) { return x > 0.f; }
// u - f * x.  With f a power of two f * x is exact unless it is subnormal, so that one fused operation
// rounds like the product and the difference; *special where it may be subnormal (then sub_scaled).
__device__ __forceinline__ double sub_scaled_plain(double u, const Factor<double>& f, double x, bool* special) {
#if SHLL_PLAIN_FMA
    return __fma_rn(-f.v, x, u);
#else
    if (!f.pow2) return u - f.v * x;
    const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
    *special = *special || (h < (600u << 20) && (h | (unsigned)__double2loint(x)) != 0u);
    return __fma_rn(-f.v, x, u);
#endif
}
__device__ __forceinline__ double sub_scaled(double u, const Factor<double>& f, double x) {
    bool special = false;
    const double r = sub_scaled_plain(u, f, x, &special);
    return special ? u - f.v * x : r;
}
__device__ __forceinline__ float sub_scaled_plain(float u, const Factor<float>& f, float x, bool*) { return u - f.v * x; }
__device__ __forceinline__ float sub_scaled(float u, const Factor<float>& f, float x) { return u - f.v * x; }
// (REAL)(D(u) - 0.5 * D(lambda) * D(x)), f = 0.5 * lambda
__device__ __forceinline__ double sub_half_scaled_plain(double u, const Factor<double>& f, double x, bool* special) {
    return sub_scaled_plain(u, f, x, special);
}
__device__ __forceinline__ float sub_half_scaled_plain(float u, const Factor<float>& f, float x, bool*) {
    return exact_math::sub_product_ref(u, f.v, x);
}
__device__ __forceinline__ double sub_half_scaled(double u, const Factor<double>& f, double x) {
    return sub_scaled(u, f, x);
}
__device__ __forceinline__ float sub_half_scaled(float u, const Factor<float>& f, float x) {
    return exact_math::sub_product_ref(u, f.v, x);
}
// a divisor used for several quotients
template <typename REAL>
struct Den;
template <>
struct Den<double> {
    exact_math::Divisor d;
    __device__ __forceinline__ explicit Den(double b) : d(exact_math::divisor(b)) {}
    __device__ __forceinline__ double divide(double a) const { return exact_math::divide(a, d); }
};
template <>
struct Den<float> {
    float b;
    __device__ __forceinline__ explicit Den(float x) : b(x) {}
    __device__ __forceinline__ float divide(float a) const { return a / b; }
};
// sqrt of a REAL argument as the reference evaluates it: sqrt(double) rounded to REAL.  For
// float this equals the correctly rounded sqrtf (53 >= 2*24+2, so the double rounding is exact).
__device__ __forceinline__ float sqrt_ref(float x) { return sqrtf(x); }
__device__ __forceinline__ double sqrt_ref(double x) { return exact_math::square_root(x); }
// the Z2 of a split flux, (REAL)(0.5 * D(a) * (1.0 - D(M * M)))
__device__ __forceinline__ double z2(double a, double M) { return half_of(a) * (1.0 - M * M); }
__device__ __forceinline__ float z2(float a, float M) { return exact_math::z2_ref(a, M * M); }
// temperature from the specific energy e, (REAL)((D(e) - 0.5 * kinetic) / D(CV)): 1D kinetic =
// D(p1) * D(p1) (0.5 * D(p1) taken first), 2D the REAL p1 * p1 + p2 * p2
__device__ __forceinline__ double temp1(const Gas<double>& g, double e, double p1) {
    return exact_math::divide(e - half_of(p1) * p1, g.cv);
}
__device__ __forceinline__ float temp1(const Gas<float>& g, float e, float p1) {
    const float kh = __fmul_rn(p1, p1);
    return exact_math::temperature_ref(e, 0.5f * kh, 0.5f * __fmaf_rn(p1, p1, -kh), g.CV, g.rCV);
}
__device__ __forceinline__ double temp2(const Gas<double>& g, double e, double p1, double p2) {
    return exact_math::divide(e - half_of(p1 * p1 + p2 * p2), g.cv);
}
__device__ __forceinline__ float temp2(const Gas<float>& g, float e, float p1, float p2) {
    return exact_math::temperature_ref(e, 0.5f * (p1 * p1 + p2 * p2), 0.f, g.CV, g.rCV);
}
template <typename REAL>
__device__ __forceinline__ REAL times_R(const Gas<REAL>& g, REAL x) { return g.R_one ? x : x * g.R; }

// ---------------- 1D ----------------
// P from U (base_shll.c:171-176); returns p1 (velocity), p2 (temperature), a (sound speed)
template <typename REAL>
__device__ __forceinline__ void prim1(const Gas<REAL>& g, REAL u0, REAL u1, REAL u2, REAL& p1, REAL& p2, REAL& a) {
    const Den<REAL> rho(u0);
    p1 = rho.divide(u1);
    p2 = temp1(g, rho.divide(u2), p1);
    a = sqrt_ref(g.gR * p2);
}

// split fluxes (base_shll.c:134-158) from P (p0 = u0) and U
template <typename REAL>
__device__ __forceinline__ void flux1(const Gas<REAL>& g, REAL u0, REAL u1, REAL u2, REAL p1, REAL p2, REAL a,
                                      REAL fp[3], REAL fm[3]) {
    REAL M = Den<REAL>(a).divide(p1);
    REAL Z1 = half_sum(M, (REAL)1);
    REAL Z2 = z2(a, M);
    REAL Z3 = half_sum(M, (REAL)-1);
    REAL P = times_R(g, u0) * p2;
    REAL f0 = u1, f1 = u1 * p1 + P, f2 = p1 * (u2 + P);
    fp[0] = f0 * Z1 + u0 * Z2; fp[1] = f1 * Z1 + u1 * Z2; fp[2] = f2 * Z1 + u2 * Z2;
    fm[0] = -f0 * Z3 - u0 * Z2; fm[1] = -f1 * Z3 - u1 * Z2; fm[2] = -f2 * Z3 - u2 * Z2;
}

// ---- a cell of the fused kernels, 1D ----
// Split fluxes (kFluxScale times) of a cell with conserved state u; returns whether its density or
// temperature is not positive.  The main path is free of branches and special cases: it holds for
// states and constants whose exponents are well inside the range (a momentum may be zero); any other
// cell takes the general functions.
// (a value, not through pointers, which would keep the main path's fluxes in local memory)
template <typename REAL, int NF>
struct CellFlux {
    REAL f[NF];
    int bad;
};
template <typename REAL>
__device__ __noinline__ CellFlux<REAL, 6> cell1_general(const Gas<REAL>& g, REAL u0, REAL u1, REAL u2) {
    CellFlux<REAL, 6> c;
    REAL p1, p2, a;
    prim1(g, u0, u1, u2, p1, p2, a);
    flux1(g, u0, u1, u2, p1, p2, a, c.f, c.f + 3);
    for (int k = 0; k < 6; k++) c.f[k] *= kFluxScale<REAL>;
    c.bad = !positive(u0) || !positive(p2);
    return c;
}
__device__ __forceinline__ unsigned hi_word(double x) { return (unsigned)__double2hiint(x); }
__device__ __forceinline__ bool is_zero(double x) { return ((hi_word(x) << 1) | (unsigned)__double2loint(x)) == 0u; }
// exponent (biased) in [lo, lo + n) and positive
__device__ __forceinline__ bool in_range(double x, unsigned lo, unsigned n) { return (hi_word(x) >> 20) - lo < n; }
__device__ __forceinline__ bool in_range(float x, unsigned lo, unsigned n) { return (__float_as_uint(x) >> 23) - lo < n; }
// momentum: zero, or of a magnitude whose quotients and products stay normal
__device__ __forceinline__ bool momentum_plain(double x) {
    return ((hi_word(x) & 0x7fffffffu) >> 20) - 323u < 800u || is_zero(x);
}
__device__ __forceinline__ bool momentum_plain(float x) {
    return ((__float_as_uint(x) & 0x7fffffffu) >> 23) - 67u < 120u || x == 0.f;
}
__device__ __forceinline__ bool all_ones(float x) { return (__float_as_uint(x) & 0x7fffffu) == 0x7fffffu; }
__device__ __forceinline__ double divide_or_zero(double a, const exact_math::Divisor& d) {
    const double q = exact_math::divide_plain(a, d);
    return is_zero(a) ? a : q;
}
// x y + z, rounded once where products and sums may be fused.  Written out in cell1 and cell1_lanes: a
// run's steps are taken by one or the other, as its length has it, and any split of a run into calls gives
// the same bits only if both fuse the same products.
__device__ __forceinline__ double product_sum(double x, double y, double z) {
#if SHLL_PLAIN_FMA
    return __fma_rn(x, y, z);
#else
    return x * y + z;
#endif
}

__device__ __forceinline__ int cell1(const Gas<double>& g, const double u[3], double fp[3], double fm[3]) {
    const exact_math::Divisor rho = exact_math::divisor(u[0]);
    const double p1 = divide_or_zero(u[1], rho);
    const double e = exact_math::divide_plain(u[2], rho);
    // e - 0.5 * p1 * p1 (the scaling is exact beside a normal e)
    const double t = __fma_rn(-0.5, __dmul_rn(p1, p1), e);
    const double p2 = exact_math::divide_plain(t, g.cv);
    exact_math::Divisor snd;
    const double a = exact_math::square_root_plain(g.gR * p2, &snd);
    const double M = divide_or_zero(p1, snd);
    const double Z1 = M + 1.0, Z3 = M - 1.0, Z2 = a * product_sum(-M, M, 1.0);   // twice the reference's
    const double rR = times_R(g, u[0]), P = rR * p2;
    const double F[3] = {u[1], product_sum(u[1], p1, P), p1 * product_sum(rR, p2, u[2])};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double w = u[k] * Z2;
        fp[k] = product_sum(F[k], Z1, w);
        fm[k] = product_sum(-F[k], Z3, -w);
    }
    if (g.plain && in_range(u[0], 923, 200) && in_range(u[2], 923, 200) && momentum_plain(u[1]) && in_range(t, 900, 250))
        return 0;
    const auto c = cell1_general(g, u[0], u[1], u[2]);
#pragma unroll
    for (int k = 0; k < 3; k++) { fp[k] = c.f[k]; fm[k] = c.f[3 + k]; }
    return c.bad;
}
// The same by a group of four lanes, FP64: lane k < 3 of the group evaluates component k alone (lane 3
// doubles lane 0), so that one lane issues 17 FP64 instructions and not 32 (25 and not 40 without fused
// operations): a scheduler starts one FP64 warp instruction in about 70 clocks whatever its
// dependences, which is what a step of a small tube waits for.  u: this lane's component.
__device__ __forceinline__ int cell1_lanes(const Gas<double>& g, double u, double& fp, double& fm) {
    const int k = threadIdx.x & 3;
    const double u0 = __shfl_sync(0xffffffffu, u, 0, 4), u1 = __shfl_sync(0xffffffffu, u, 1, 4),
                 u2 = __shfl_sync(0xffffffffu, u, 2, 4);
    const exact_math::Divisor rho = exact_math::divisor(u0);
    const double q = exact_math::divide_plain(k == 2 ? u2 : u1, rho);
    const double q1 = __shfl_sync(0xffffffffu, q, 1, 4), e = __shfl_sync(0xffffffffu, q, 2, 4);
    const double p1 = is_zero(u1) ? u1 : q1;
    const double t = __fma_rn(-0.5, __dmul_rn(p1, p1), e);
    const double p2 = exact_math::divide_plain(t, g.cv);
    exact_math::Divisor snd;
    const double a = exact_math::square_root_plain(g.gR * p2, &snd);
    const double M = divide_or_zero(p1, snd);
    const double Z1 = M + 1.0, Z3 = M - 1.0, Z2 = a * product_sum(-M, M, 1.0);   // twice the reference's
    const double rR = times_R(g, u0), P = rR * p2;
    // F = u1, u1 p1 + P, p1 (u2 + P)
    double F = product_sum(k == 2 ? rR : u1, k == 2 ? p2 : p1, k == 2 ? u2 : P);
    const double F2 = p1 * F;
    F = k == 1 ? F : k == 2 ? F2 : u1;
    const double w = (k == 1 ? u1 : k == 2 ? u2 : u0) * Z2;
    fp = product_sum(F, Z1, w);
    fm = product_sum(-F, Z3, -w);
    if (g.plain && in_range(u0, 923, 200) && in_range(u2, 923, 200) && momentum_plain(u1) && in_range(t, 900, 250)) return 0;
    const auto c = cell1_general(g, u0, u1, u2);
    fp = k == 1 ? c.f[1] : k == 2 ? c.f[2] : c.f[0];
    fm = k == 1 ? c.f[4] : k == 2 ? c.f[5] : c.f[3];
    return c.bad;
}
__device__ __forceinline__ int cell1(const Gas<float>& g, const float u[3], float fp[3], float fm[3]) {
    const float y = exact_math::reciprocal_plain(u[0], exact_math::em_rcp(u[0]));
    const float p1 = exact_math::divide_plain(u[1], u[0], y), e = exact_math::divide_plain(u[2], u[0], y);
    // A rounding that the FP32 forms leave open takes the general functions, too: one branch at the end
    // and none in the chain (1024 cells: 0.44 -> 0.40 us a step, second order 0.77 -> 0.73; the same in
    // Cell2<float> gains nothing: 512 x 480 cells, second order, 14.0 us both, 301 x 277 7.6 -> 7.8).
    bool ok = true;
    const float kh = __fmul_rn(p1, p1);
    const float p2 = exact_math::temperature_plain(e, 0.5f * kh, 0.5f * __fmaf_rn(p1, p1, -kh), g.CV, g.rCV, &ok);
    const float x = g.gR * p2;
    float ya;
    const float a = exact_math::square_root_plain(x, &ya);
    const float M = exact_math::divide_plain(p1, a, exact_math::reciprocal_plain(a, ya));
    const float Z1 = half_sum(M, 1.f), Z3 = half_sum(M, -1.f), Z2 = exact_math::z2_plain(a, M * M, &ok);
    const float P = times_R(g, u[0]) * p2;
    const float F[3] = {u[1], u[1] * p1 + P, p1 * (u[2] + P)};
#pragma unroll
    for (int k = 0; k < 3; k++) { fp[k] = F[k] * Z1 + u[k] * Z2; fm[k] = -F[k] * Z3 - u[k] * Z2; }
    // (a divisor of all-ones significand is the exception of the residual step)
    if (ok && g.plain && in_range(u[0], 97, 60) && !all_ones(u[0]) && in_range(u[2], 87, 80) && momentum_plain(u[1]) &&
        in_range(x, 87, 80) && !all_ones(a))
        return 0;
    const auto c = cell1_general(g, u[0], u[1], u[2]);
#pragma unroll
    for (int k = 0; k < 3; k++) { fp[k] = c.f[k]; fm[k] = c.f[3 + k]; }
    return c.bad;
}

// minmod (2nd_order_base_shll.c:191-201)
__device__ __forceinline__ double minmod(double l, double r, bool* special) {
    return exact_math::minmod_plain(l, r, special);
}
__device__ __forceinline__ float minmod(float l, float r, bool*) {
    if (__fmul_rn(l, r) < 0.f) return 0.f;
    return fabsf(l) < fabsf(r) ? l : r;
}
// slope of a split flux at an interior cell from the differences l = fc - fl and r = fr - fc (and
// c = fr - fl): minmod, or the MC limiter of base-omp/2nd_order_base_shll.c:316-325.  Where *special
// comes back set, slope_general decides.
template <typename REAL>
__device__ __forceinline__ REAL slope_plain(const Gas<REAL>& g, REAL fl, REAL fc, REAL fr, bool* special) {
    const REAL m = minmod(fc - fl, fr - fc, special);
    return g.limiter == 1 ? minmod(half_of(fr - fl), g.alpha * m, special) : m;
}
template <typename REAL>
__device__ __noinline__ REAL slope_general(const Gas<REAL>& g, REAL fl, REAL fc, REAL fr, REAL inv_scale) {
    if constexpr (sizeof(REAL) == 4) return slope_plain(g, fl, fc, fr, nullptr);
    else {
        const REAL m = exact_math::minmod_general(fc - fl, fr - fc, inv_scale);
        return g.limiter == 1 ? exact_math::minmod_general(half_of(fr - fl), g.alpha * m, inv_scale) : m;
    }
}
template <typename REAL>
__device__ __forceinline__ REAL slope(const Gas<REAL>& g, REAL fl, REAL fc, REAL fr,
                                      REAL inv_scale = (REAL)1 / kFluxScale<REAL>) {
    bool special = false;
    const REAL s = slope_plain(g, fl, fc, fr, &special);
    return special ? slope_general(g, fl, fc, fr, inv_scale) : s;
}

constexpr int T1 = 256;  // cells per block (1D)

// One fused time step in 1D: P and split fluxes for the block's cells plus halo (in shared
// memory), slopes (order 2), then the reference's per-cell update.  Uin/Uout: 3 planes of n.
// Body of one 1D block: cells [b0, b0+T1) of a tube of n cells whose component k lives at
// U[k*stride + c].
template <typename REAL, int ORDER>
__device__ __forceinline__ void step1_block(const REAL* __restrict__ Uin, REAL* __restrict__ Uout, int n, long stride,
                                            const Gas<REAL>& g, int* __restrict__ flag, int b0) {
    constexpr int H = ORDER;
    constexpr int W = T1 + 2 * H;
    __shared__ REAL sfp[3][W], sfm[3][W];
    __shared__ REAL sdp[3][ORDER == 2 ? T1 + 2 : 1], sdm[3][ORDER == 2 ? T1 + 2 : 1];
    int bad = 0;
    for (int t = threadIdx.x; t < W; t += T1) {
        int c = b0 - H + t;
        REAL fp[3] = {0, 0, 0}, fm[3] = {0, 0, 0};
        if (c >= 0 && c < n) {
            const REAL u[3] = {Uin[c], Uin[stride + c], Uin[2 * stride + c]};
            bad |= cell1(g, u, fp, fm);
        }
#pragma unroll
        for (int k = 0; k < 3; k++) { sfp[k][t] = fp[k]; sfm[k][t] = fm[k]; }
    }
    __syncthreads();
    if (ORDER == 2) {
        for (int t = threadIdx.x; t < T1 + 2; t += T1) {
            int c = b0 - 1 + t, s = t + 1;  // shared index of cell c
#pragma unroll
            for (int k = 0; k < 3; k++) {
                REAL dp = 0, dm = 0;
                if (c > 0 && c < n - 1) {
                    dp = slope(g, sfp[k][s - 1], sfp[k][s], sfp[k][s + 1]);
                    dm = slope(g, sfm[k][s - 1], sfm[k][s], sfm[k][s + 1]);
                }
                sdp[k][t] = dp; sdm[k][t] = dm;
            }
        }
        __syncthreads();
    }
    const int i = b0 + threadIdx.x;
    if (bad) atomicOr(flag, SHLL_FLAG_NONPOSITIVE);
    if (i >= n) return;
    const int s = threadIdx.x + H;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        REAL fp = sfp[k][s], fm = sfm[k][s], L, Rr, u = Uin[k * stride + i];
        if (ORDER == 1) {
            const REAL sg = (k == 1) ? (REAL)1 : (REAL)-1;  // reflective wall (base_shll.c:93-110)
            if (i == 0) { L = sg * fm; Rr = sfm[k][s + 1]; }
            else if (i == n - 1) { L = sfp[k][s - 1]; Rr = sg * fp; }
            else { L = sfp[k][s - 1]; Rr = sfm[k][s + 1]; }
            u = sub_scaled(u, g.sx, fp - fm + Rr - L);
        } else {
            const int d = threadIdx.x + 1;  // slope index of cell i
            REAL Ldf, Rdf;
            if (i == 0) { L = fp; Rr = sfm[k][s + 1]; Ldf = 0; Rdf = sdm[k][d + 1]; }
            else if (i == n - 1) { L = sfp[k][s - 1]; Rr = fm; Ldf = sdp[k][d - 1]; Rdf = 0; }
            else { L = sfp[k][s - 1]; Rr = sfm[k][s + 1]; Ldf = sdp[k][d - 1]; Rdf = sdm[k][d + 1]; }
            u = sub_scaled(u, g.sx, fp - fm + Rr - L);
            u = sub_half_scaled(u, g.hsx, sdp[k][d] + sdm[k][d] - Rdf - Ldf);
        }
        Uout[k * stride + i] = u;
    }
}

template <typename REAL, int ORDER>
__global__ void __launch_bounds__(T1) k_step1(const REAL* __restrict__ Uin, REAL* __restrict__ Uout, int n,
                                              Gas<REAL> g, int* __restrict__ flag) {
    step1_block<REAL, ORDER>(Uin, Uout, n, n, g, flag, blockIdx.x * T1);
}

// ---------------- 2D ----------------
template <typename REAL>
__device__ __forceinline__ void prim2(const Gas<REAL>& g, REAL u0, REAL u1, REAL u2, REAL u3, REAL& p1, REAL& p2,
                                      REAL& p3, REAL& a) {
    const Den<REAL> rho(u0);
    p1 = rho.divide(u1);
    p2 = rho.divide(u2);
    p3 = temp2(g, rho.divide(u3), p1, p2);
    a = sqrt_ref(g.gR * p3);
}

// x and y split fluxes (base_shll_2d.c:243-299)
template <typename REAL>
__device__ __forceinline__ void flux2(const Gas<REAL>& g, const REAL u[4], REAL p1, REAL p2, REAL p3, REAL a,
                                      REAL fp[4], REAL fm[4], REAL hp[4], REAL hm[4]) {
    REAL P = times_R(g, u[0]) * p3;
    const Den<REAL> da(a);
    REAL M = da.divide(p1);
    REAL Z1 = half_sum(M, (REAL)1);
    REAL Z2 = z2(a, M);
    REAL Z3 = half_sum(M, (REAL)-1);
    REAL f[4] = {u[1], u[1] * p1 + P, u[1] * p2, p1 * (u[3] + P)};
#pragma unroll
    for (int k = 0; k < 4; k++) { fp[k] = f[k] * Z1 + u[k] * Z2; fm[k] = -f[k] * Z3 - u[k] * Z2; }
    M = da.divide(p2);
    Z1 = half_sum(M, (REAL)1);
    Z2 = z2(a, M);
    Z3 = half_sum(M, (REAL)-1);
    REAL h[4] = {u[2], u[2] * p1, u[2] * p2 + P, p2 * (u[3] + P)};
#pragma unroll
    for (int k = 0; k < 4; k++) { hp[k] = h[k] * Z1 + u[k] * Z2; hm[k] = -h[k] * Z3 - u[k] * Z2; }
}

// a cell of the fused kernels, 2D (see cell1)
template <typename REAL>
__device__ __noinline__ CellFlux<REAL, 16> cell2_general(const Gas<REAL>& g, REAL u0, REAL u1, REAL u2, REAL u3) {
    const REAL u[4] = {u0, u1, u2, u3};
    CellFlux<REAL, 16> c;
    REAL p1, p2, p3, a;
    prim2(g, u0, u1, u2, u3, p1, p2, p3, a);
    flux2(g, u, p1, p2, p3, a, c.f, c.f + 4, c.f + 8, c.f + 12);
    for (int k = 0; k < 16; k++) c.f[k] *= kFluxScale<REAL>;
    c.bad = !positive(u0) || !positive(p3);
    return c;
}
// What both directions' split fluxes of a cell need; plain: the main path holds for this cell.
template <typename REAL>
struct Cell2;
template <>
struct Cell2<double> {
    double p[2], P, a;
    exact_math::Divisor snd;
    bool plain;
    __device__ __forceinline__ Cell2(const Gas<double>& g, const double u[4]) {
        const exact_math::Divisor rho = exact_math::divisor(u[0]);
        p[0] = divide_or_zero(u[1], rho);
        p[1] = divide_or_zero(u[2], rho);
        const double e = exact_math::divide_plain(u[3], rho);
        // (symmetric in the two velocities, so that a cell's y flux is the x flux of its mirror image)
        const double t = __fma_rn(-0.5, __dadd_rn(__dmul_rn(p[0], p[0]), __dmul_rn(p[1], p[1])), e);
        const double p3 = exact_math::divide_plain(t, g.cv);
        a = exact_math::square_root_plain(g.gR * p3, &snd);
        P = times_R(g, u[0]) * p3;
        plain = g.plain && in_range(u[0], 923, 200) && in_range(u[3], 923, 200) && momentum_plain(u[1]) &&
                momentum_plain(u[2]) && in_range(t, 900, 250);
    }
    __device__ __forceinline__ double mach(double pn) const { return divide_or_zero(pn, snd); }
};
template <>
struct Cell2<float> {
    float p[2], P, a, ya;
    bool plain;
    __device__ __forceinline__ Cell2(const Gas<float>& g, const float u[4]) {
        const float y = exact_math::reciprocal_plain(u[0], exact_math::em_rcp(u[0]));
        p[0] = exact_math::divide_plain(u[1], u[0], y);
        p[1] = exact_math::divide_plain(u[2], u[0], y);
        const float p3 = temp2(g, exact_math::divide_plain(u[3], u[0], y), p[0], p[1]), x = g.gR * p3;
        a = exact_math::square_root_plain(x, &ya);
        ya = exact_math::reciprocal_plain(a, ya);
        P = times_R(g, u[0]) * p3;
        plain = g.plain && in_range(u[0], 97, 60) && !all_ones(u[0]) && in_range(u[3], 87, 80) && momentum_plain(u[1]) &&
                momentum_plain(u[2]) && in_range(x, 87, 80) && !all_ones(a);
    }
    __device__ __forceinline__ float mach(float pn) const { return exact_math::divide_plain(pn, a, ya); }
};
__device__ __forceinline__ void z123(double a, double M, double& Z1, double& Z2, double& Z3) {   // twice the reference's
    Z1 = M + 1.0;
    Z2 = a * (1.0 - M * M);
    Z3 = M - 1.0;
}
__device__ __forceinline__ void z123(float a, float M, float& Z1, float& Z2, float& Z3) {
    Z1 = half_sum(M, 1.f);
    Z2 = z2(a, M);
    Z3 = half_sum(M, -1.f);
}
// The split fluxes of a cell in the directions d0..d1 (0 x, 1 y), stored to out[(8 d + 4 pm + k) *
// stride], pm 0 plus and 1 minus.  A loop over the directions and not two copies of its body: the
// cells of a tile's halo need one direction only, and the code stays half as long.
template <typename REAL>
__device__ __forceinline__ int cell2(const Gas<REAL>& g, const REAL u[4], int d0, int d1, REAL* out, int stride) {
    const Cell2<REAL> c(g, u);
    if (c.plain) {
#pragma unroll 1
        for (int d = d0; d <= d1; d++) {
            const REAL un = d ? u[2] : u[1], ut = d ? u[1] : u[2];     // momentum along d and across
            const REAL pn = d ? c.p[1] : c.p[0], pt = d ? c.p[0] : c.p[1];
            REAL Z1, Z2, Z3;
            z123(c.a, c.mach(pn), Z1, Z2, Z3);
            const REAL f[4] = {un, un * pn + c.P, un * pt, pn * (u[3] + c.P)};
            const REAL v[4] = {u[0], un, ut, u[3]};
            REAL* o = out + 8 * d * stride;
            const int at[4] = {0, (1 + d) * stride, (2 - d) * stride, 3 * stride};
#pragma unroll
            for (int k = 0; k < 4; k++) {
                o[at[k]] = f[k] * Z1 + v[k] * Z2;
                o[at[k] + 4 * stride] = -f[k] * Z3 - v[k] * Z2;
            }
        }
        return 0;
    }
    const auto q = cell2_general(g, u[0], u[1], u[2], u[3]);
#pragma unroll
    for (int k = 0; k < 16; k++)
        if (k / 8 >= d0 && k / 8 <= d1) out[k * stride] = q.f[k];
    return q.bad;
}

// ---- one 2D step of a TI x 32 tile ----
// Window: the tile and ORDER cells on each side, without the corners.  Threads: one per tile cell (both
// directions' fluxes), then one per cell of the halo rows (x flux only) and of the halo columns (y only).
constexpr int TJ = 32;           // tile extent along j (contiguous)
constexpr int kBatchTI = 8;      // tile extent along i of the batches
constexpr int kTileThreads = 768;

__host__ __device__ constexpr int tile_threads(int TI, int H) { return (TI * TJ + 2 * H * TJ + TI * 2 * H + 31) / 32 * 32; }

template <typename REAL>
constexpr size_t smem2(int TI, int H) {
    const size_t flux = (size_t)16 * (TI + 2 * H) * (TJ + 2 * H);
    const size_t slopes = H == 2 ? (size_t)8 * ((TI + 2) * TJ + TI * (TJ + 2)) : 0;
    return (flux + slopes) * sizeof(REAL);
}

// One fused 2D time step on a TI x TJ tile.  Shared memory holds fp, fm, hp, hm (4 components
// each) for the tile plus an ORDER-wide halo, then (order 2) the x and y slopes.
// Body of one 2D tile with origin (i0, j0) of an nx x ny domain whose component k lives at
// U[k*stride + i*ny + j].  STAGED: Update_U_from_F, the split fluxes read from the planes of
// Compute_F_from_P instead of evaluated (Uin == Uout: a cell reads only its own state).
template <typename REAL, int ORDER, bool STAGED = false>
__device__ __forceinline__ void step2_tile(const REAL* Uin, REAL* Uout, int nx, int ny,
                                           long stride, const Gas<REAL>& g, int* __restrict__ flag, int i0, int j0,
                                           const int TI, const REAL* const* planes = nullptr) {
    constexpr int H = ORDER, WJ = TJ + 2 * H;
    constexpr REAL kInvScale = STAGED ? (REAL)1 : (REAL)1 / kFluxScale<REAL>;
    const Factor<REAL>& fx = STAGED ? g.lx : g.sx;
    const Factor<REAL>& fy = STAGED ? g.ly : g.sy;
    const Factor<REAL>& hfx = STAGED ? g.hlx : g.hsx;
    const Factor<REAL>& hfy = STAGED ? g.hly : g.hsy;
    const int CELLS = (TI + 2 * H) * WJ;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    REAL* sf = reinterpret_cast<REAL*>(smem_raw);      // [16][CELLS]: fp0..3 fm0..3 hp0..3 hm0..3
    REAL* sd = sf + 16 * CELLS;                          // order 2 slopes
    const int NXS = (TI + 2) * TJ, NYS = TI * (TJ + 2);
    const long n = stride;
    const int tid = threadIdx.x, nthreads = blockDim.x;
    const int ty = tid / TJ, tx = tid % TJ;
    int bad = 0;
    REAL u[4] = {1, 0, 0, 1};
    {
        int li, lj, d0 = 0, d1 = 1;
        const int h = tid - TI * TJ;                     // index among the halo cells
        if (h < 0) { li = ty + H; lj = tx + H; }
        else if (h < 2 * H * TJ) { li = h / TJ; li += li < H ? 0 : TI; lj = tx + H; d1 = 0; }
        else { const int q = h - 2 * H * TJ, m = q % (2 * H); li = q / (2 * H) + H; lj = m < H ? m : TJ + m; d0 = 1; }
        const int i = i0 - H + li, j = j0 - H + lj;
        if (li < TI + 2 * H && (d0 == 0 || li < TI + H) && i >= 0 && i < nx && j >= 0 && j < ny) {
            const long c = (long)i * ny + j;
            if constexpr (STAGED) {
                if (h < 0) {
#pragma unroll
                    for (int k = 0; k < 4; k++) u[k] = Uin[k * n + c];
                }
#pragma unroll
                for (int q = 0; q < 16; q++)
                    if (q / 8 >= d0 && q / 8 <= d1) sf[q * CELLS + li * WJ + lj] = planes[q / 4][(q % 4) * n + c];
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) u[k] = Uin[k * n + c];
                bad = cell2(g, u, d0, d1, sf + li * WJ + lj, CELLS);
            }
        }
    }
    __syncthreads();
    auto F = [&](int q, int k, int li, int lj) -> REAL { return sf[(q * 4 + k) * CELLS + li * WJ + lj]; };
    if (ORDER == 2) {
        // x slopes for local rows -1..TI (cells i0-1..i0+TI), cols 0..TJ-1
        for (int t = tid; t < NXS; t += nthreads) {
            int r = t / TJ, lj = t % TJ;
            int i = i0 - 1 + r, j = j0 + lj, li = r - 1 + H, ljj = lj + H;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                REAL dp = 0, dm = 0;
                if (i > 0 && i < nx - 1 && j < ny) {
                    dp = slope(g, F(0, k, li - 1, ljj), F(0, k, li, ljj), F(0, k, li + 1, ljj), kInvScale);
                    dm = slope(g, F(1, k, li - 1, ljj), F(1, k, li, ljj), F(1, k, li + 1, ljj), kInvScale);
                }
                sd[k * NXS + t] = dp; sd[(4 + k) * NXS + t] = dm;
            }
        }
        // y slopes for rows 0..TI-1, cols -1..TJ
        for (int t = tid; t < NYS; t += nthreads) {
            int r = t / (TJ + 2), c2 = t % (TJ + 2);
            int i = i0 + r, j = j0 - 1 + c2, li = r + H, lj = c2 - 1 + H;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                REAL dp = 0, dm = 0;
                if (j > 0 && j < ny - 1 && i < nx) {
                    dp = slope(g, F(2, k, li, lj - 1), F(2, k, li, lj), F(2, k, li, lj + 1), kInvScale);
                    dm = slope(g, F(3, k, li, lj - 1), F(3, k, li, lj), F(3, k, li, lj + 1), kInvScale);
                }
                sd[8 * NXS + k * NYS + t] = dp; sd[8 * NXS + (4 + k) * NYS + t] = dm;
            }
        }
        __syncthreads();
    }
    if (bad) atomicOr(flag, SHLL_FLAG_NONPOSITIVE);
    const int i = i0 + ty, j = j0 + tx;
    if (ty >= TI || i >= nx || j >= ny) return;
    const long c = (long)i * ny + j;
    const int li = ty + H, lj = tx + H;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        REAL v = u[k];
        REAL fp = F(0, k, li, lj), fm = F(1, k, li, lj), hp = F(2, k, li, lj), hm = F(3, k, li, lj);
        if (ORDER == 1) {
            // reflective walls: x flips components 0,2,3; y flips 0,1,3 (base_shll_2d.c:150-216)
            const REAL sx = (k == 1) ? (REAL)1 : (REAL)-1, sy = (k == 2) ? (REAL)1 : (REAL)-1;
            REAL L, Rr, B, Tt;
            if (i == 0) { L = sx * fm; Rr = F(1, k, li + 1, lj); }
            else if (i == nx - 1) { L = F(0, k, li - 1, lj); Rr = sx * fp; }
            else { L = F(0, k, li - 1, lj); Rr = F(1, k, li + 1, lj); }
            if (j == 0) { B = sy * hm; Tt = F(3, k, li, lj + 1); }
            else if (j == ny - 1) { B = F(2, k, li, lj - 1); Tt = sy * hp; }
            else { B = F(2, k, li, lj - 1); Tt = F(3, k, li, lj + 1); }
            v = sub_scaled(v, fx, fp - fm + Rr - L);
            v = sub_scaled(v, fy, hp - hm + Tt - B);
        } else {
            // outflow walls, slopes zero on edge cells (2nd_order_base_shll.c:210-458)
            auto DX_ = [&](int q, int r) -> REAL { return sd[(q * 4 + k) * NXS + r * TJ + tx]; };
            auto DY_ = [&](int q, int cc) -> REAL {
                return sd[8 * NXS + (q * 4 + k) * NYS + ty * (TJ + 2) + cc];
            };
            const int r = ty + 1, cc = tx + 1;
            REAL L, Rr, Ldf, Rdf, B, Tt, Bdf, Tdf;
            if (i == 0) { L = fp; Rr = F(1, k, li + 1, lj); Ldf = 0; Rdf = DX_(1, r + 1); }
            else if (i == nx - 1) { L = F(0, k, li - 1, lj); Rr = fm; Ldf = DX_(0, r - 1); Rdf = 0; }
            else { L = F(0, k, li - 1, lj); Rr = F(1, k, li + 1, lj); Ldf = DX_(0, r - 1); Rdf = DX_(1, r + 1); }
            if (j == 0) { B = hp; Tt = F(3, k, li, lj + 1); Bdf = 0; Tdf = DY_(1, cc + 1); }
            else if (j == ny - 1) { B = F(2, k, li, lj - 1); Tt = hm; Bdf = DY_(0, cc - 1); Tdf = 0; }
            else { B = F(2, k, li, lj - 1); Tt = F(3, k, li, lj + 1); Bdf = DY_(0, cc - 1); Tdf = DY_(1, cc + 1); }
            v = sub_scaled(v, fx, fp - fm + Rr - L);
            v = sub_half_scaled(v, hfx, DX_(0, r) + DX_(1, r) - Rdf - Ldf);
            v = sub_scaled(v, fy, hp - hm + Tt - B);
            v = sub_half_scaled(v, hfy, DY_(0, cc) + DY_(1, cc) - Tdf - Bdf);
        }
        Uout[k * n + c] = v;
    }
}

// The grid of a domain's tiles: columns along x, rows along y and, as a domain may have more of them than
// the y axis holds (65535: 393210 cells with 6-row tiles), along z.  (All along x, with a division in the
// kernel, cost 301 x 277 cells 7.61 -> 7.74 us a step.)  A block past the last row holds no cell of the
// domain and stores nothing.
static dim3 tile_grid(int nx, int ny, int TI) {
    const int rows = (nx + TI - 1) / TI, layers = (rows + 65534) / 65535;
    return dim3((unsigned)((ny + TJ - 1) / TJ), (unsigned)((rows + layers - 1) / layers), (unsigned)layers);
}
__device__ __forceinline__ int tile_i0(int TI) { return (int)(blockIdx.y + blockIdx.z * gridDim.y) * TI; }

// Consecutive steps are chained by programmatic dependent launch: the next step's blocks are resident
// and past their launch when this grid completes (griddepcontrol.wait).  Uin is written while this grid already
// runs, so it must not be declared read-only (const __restrict__): such loads may take the non-coherent
// path, and may be moved above the wait.
template <typename REAL, int ORDER>
__global__ void __launch_bounds__(kTileThreads) k_step2(const REAL* Uin, REAL* Uout, int nx, int ny,
                                                        const __grid_constant__ Gas<REAL> g, int* flag, int TI) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    step2_tile<REAL, ORDER>(Uin, Uout, nx, ny, (long)nx * ny, g, flag, tile_i0(TI), blockIdx.x * TJ, TI);
}

static int device_sm_count() {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 1;
    return sms;
}

// Tile height of a domain.  FP64: the one with the least work on the busiest SM, counting a halo cell
// as 0.6 of a tile cell (one direction of two) and two rows' worth of fixed cost per tile (256 x 256
// cells on 152 SMs: 14 rows, one tile per SM, 13.7 us a step, where 8 rows take 15.7 and 12 rows
// 22.5).  Float steps are bound by latency, which several small tiles on an SM hide from each
// other: 6 rows (256 x 256, first order: 4.3 us against 5.0 with 14), second order 8 rows (301 x 277:
// 7.6 us against 8.7 with 10) unless one tile per SM will do (256 x 256: 6.2 us against 7.2 with 8).
// On large domains the redundant halo rows count for more: 6 / 8 / 12 rows, first order, 700 x 700 12.2 / 11.8 /
// 11.7 us, 1024 x 1024 23.2 / 22.3 / 21.5, 2048 x 2048 87.9 / 84.0 / 80.5; second order 8 / 16 rows 23.0 / 22.3, 44.9 /
// 42.3, 175 / 161.  The rule does not follow that yet.
static int tile_rows(int nx, int ny, int H, int sms, bool wide) {
    int best = kBatchTI;
    long best_tiles = 0;
    double best_t = 1e30;
    for (int TI = 4; tile_threads(TI, H) <= kTileThreads && TI <= 20; TI++) {
        const long tiles = (long)((nx + TI - 1) / TI) * ((ny + TJ - 1) / TJ);
        const double t = (double)((tiles + sms - 1) / sms) * (TI + 0.6 * 2 * H + 0.6 * 2 * H * TI / TJ + 2.0);
        if (t < best_t) { best_t = t; best = TI; best_tiles = tiles; }
    }
    if (wide) return best;
    return H == 1 ? 6 : best_tiles <= sms ? best : 8;
}

// ---------------- staged kernels (the reference's separate stages) ----------------
// Compute_U_from_P: base_shll.c:76-80 / base_shll_2d.c:126-131.  P: nv planes (+ a plane).
template <typename REAL>
__global__ void k_u_from_p(const REAL* __restrict__ P, REAL* __restrict__ U, long n, int dim, Gas<REAL> g) {
    for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < n; c += (long)gridDim.x * blockDim.x) {
        if (dim == 1) {
            REAL p0 = P[c], p1 = P[n + c], p2 = P[2 * n + c];
            U[c] = p0; U[n + c] = p0 * p1;
            U[2 * n + c] = (REAL)(D(p0) * (D(p2 * g.CV) + 0.5 * D(p1) * D(p1)));
        } else {
            REAL p0 = P[c], p1 = P[n + c], p2 = P[2 * n + c], p3 = P[3 * n + c];
            U[c] = p0; U[n + c] = p0 * p1; U[2 * n + c] = p0 * p2;
            U[3 * n + c] = (REAL)(D(p0) * (D(p3 * g.CV) + 0.5 * D(p1 * p1 + p2 * p2)));
        }
    }
}

// Compute_P_from_U: P planes rho, u, [v,] T and the sound-speed plane a after them.
template <typename REAL>
__global__ void k_p_from_u(const REAL* __restrict__ U, REAL* __restrict__ P, long n, int dim, Gas<REAL> g,
                           int* __restrict__ flag) {
    int bad = 0;
    for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < n; c += (long)gridDim.x * blockDim.x) {
        if (dim == 1) {
            REAL u0 = U[c], p1, p2, a;
            prim1(g, u0, U[n + c], U[2 * n + c], p1, p2, a);
            P[c] = u0; P[n + c] = p1; P[2 * n + c] = p2; P[3 * n + c] = a;
            bad |= !positive(u0) || !positive(p2);
        } else {
            REAL u0 = U[c], p1, p2, p3, a;
            prim2(g, u0, U[n + c], U[2 * n + c], U[3 * n + c], p1, p2, p3, a);
            P[c] = u0; P[n + c] = p1; P[2 * n + c] = p2; P[3 * n + c] = p3; P[4 * n + c] = a;
            bad |= !positive(u0) || !positive(p3);
        }
    }
    if (bad) atomicOr(flag, SHLL_FLAG_NONPOSITIVE);
}

// Primitives handed over as planes of doubles: refused as a whole (worst, nothing else written) when a
// density or temperature is not positive, ...
template <typename REAL>
__global__ void k_check_planes(const double* __restrict__ in, long n, int nv, int* __restrict__ worst) {
    for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < n; c += (long)gridDim.x * blockDim.x)
        if (!positive(in[c]) || !positive(in[(nv - 1) * n + c])) {
            atomicMax(worst, (int)(n - c));
            return;   // (a thread's later cells have higher indices)
        }
}
// ... else taken over as main() does (base_shll.c:202-205): P rounded to REAL, U from P, P from U
// (ends: density and temperature, `reach` values apart, and mid: the velocities, each as handed over or, in
// ends, already in P; a cell's values are read before they are written)
template <typename REAL, typename ENDS>
__global__ void k_load_planes(const ENDS* ends, long reach, const double* __restrict__ mid, REAL* P, REAL* __restrict__ U,
                              long n, int dim, const __grid_constant__ Gas<REAL> g, const int* __restrict__ worst,
                              int* __restrict__ flag) {
    if (*worst > 0) return;
    int bad = 0;
    for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < n; c += (long)gridDim.x * blockDim.x) {
        const REAL p0 = (REAL)ends[c], q1 = (REAL)mid[c], qT = (REAL)ends[reach + c];
        if (dim == 1) {
            const REAL u1 = p0 * q1, u2 = (REAL)(D(p0) * (D(qT * g.CV) + 0.5 * D(q1) * D(q1)));
            REAL p1, p2, a;
            prim1(g, p0, u1, u2, p1, p2, a);
            U[c] = p0; U[n + c] = u1; U[2 * n + c] = u2;
            P[c] = p0; P[n + c] = p1; P[2 * n + c] = p2; P[3 * n + c] = a;
            bad |= !positive(p0) || !positive(p2);
        } else {
            const REAL q2 = (REAL)mid[n + c];
            const REAL u1 = p0 * q1, u2 = p0 * q2;
            const REAL u3 = (REAL)(D(p0) * (D(qT * g.CV) + 0.5 * D(q1 * q1 + q2 * q2)));
            REAL p1, p2, p3, a;
            prim2(g, p0, u1, u2, u3, p1, p2, p3, a);
            U[c] = p0; U[n + c] = u1; U[2 * n + c] = u2; U[3 * n + c] = u3;
            P[c] = p0; P[n + c] = p1; P[2 * n + c] = p2; P[3 * n + c] = p3; P[4 * n + c] = a;
            bad |= !positive(p0) || !positive(p3);
        }
    }
    if (bad) atomicOr(flag, SHLL_FLAG_NONPOSITIVE);
}
// one plane taken over as REAL, unless worst says that the state is refused
template <typename REAL, typename IN>
__global__ void k_take_plane(const IN* __restrict__ in, REAL* __restrict__ out, long n, const int* __restrict__ worst) {
    if (worst && *worst > 0) return;
    for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < n; c += (long)gridDim.x * blockDim.x) out[c] = (REAL)in[c];
}
template <typename REAL>
__global__ void k_dump_planes(const REAL* __restrict__ P, double* __restrict__ out, long words) {
    for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < words; c += (long)gridDim.x * blockDim.x)
        out[c] = D(P[c]);
}

// Compute_F_from_P from the stored P (and its a plane) and U, as the reference reads both.
template <typename REAL>
__global__ void k_f_from_p(const REAL* __restrict__ U, const REAL* __restrict__ P, REAL* __restrict__ fp,
                           REAL* __restrict__ fm, REAL* __restrict__ hp, REAL* __restrict__ hm, long n, int dim,
                           Gas<REAL> g) {
    for (long c = blockIdx.x * (long)blockDim.x + threadIdx.x; c < n; c += (long)gridDim.x * blockDim.x) {
        if (dim == 1) {
            REAL a[3], b[3];
            flux1(g, U[c], U[n + c], U[2 * n + c], P[n + c], P[2 * n + c], P[3 * n + c], a, b);
            for (int k = 0; k < 3; k++) { fp[k * n + c] = a[k]; fm[k * n + c] = b[k]; }
        } else {
            REAL u[4] = {U[c], U[n + c], U[2 * n + c], U[3 * n + c]}, a[4], b[4], e[4], f[4];
            // the reference evaluates P = p0*R*p3 with p0 from the P array (equal to u0)
            flux2(g, u, P[n + c], P[2 * n + c], P[3 * n + c], P[4 * n + c], a, b, e, f);
            for (int k = 0; k < 4; k++) {
                fp[k * n + c] = a[k]; fm[k * n + c] = b[k]; hp[k * n + c] = e[k]; hm[k * n + c] = f[k];
            }
        }
    }
}

// Update_U_from_F from stored split-flux planes (in place: each cell reads only its own U).  2D: the
// tile kernel's slopes and update (a cell's slopes evaluated once and not for each of the three cells
// that use them: 512 x 480 cells, FP64, second order, 73.6 -> 59.5 us).
template <typename REAL, int ORDER>
__global__ void __launch_bounds__(kTileThreads) k_update2_staged(REAL* U, const REAL* fp, const REAL* fm, const REAL* hp,
                                                                 const REAL* hm, int nx, int ny,
                                                                 const __grid_constant__ Gas<REAL> g, int TI) {
    const REAL* const planes[4] = {fp, fm, hp, hm};
    step2_tile<REAL, ORDER, true>(U, U, nx, ny, (long)nx * ny, g, nullptr, tile_i0(TI), blockIdx.x * TJ, TI, planes);
}
template <typename REAL>
__global__ void k_update1_staged(REAL* __restrict__ U, const REAL* __restrict__ fp, const REAL* __restrict__ fm, int n,
                                 int order, const __grid_constant__ Gas<REAL> g) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        for (int k = 0; k < 3; k++) {
            const REAL* Fp = fp + (long)k * n; const REAL* Fm = fm + (long)k * n;
            REAL u = U[(long)k * n + i];
            if (order == 1) {
                const REAL sx = (k == 1) ? (REAL)1 : (REAL)-1;
                REAL L, Rr;
                if (i == 0) { L = sx * Fm[i]; Rr = Fm[i + 1]; }
                else if (i == n - 1) { L = Fp[i - 1]; Rr = sx * Fp[i]; }
                else { L = Fp[i - 1]; Rr = Fm[i + 1]; }
                u = sub_scaled(u, g.lx, Fp[i] - Fm[i] + Rr - L);
            } else {
                auto sl = [&](const REAL* f, int c) -> REAL {
                    if (c <= 0 || c >= n - 1) return (REAL)0;
                    return slope(g, f[c - 1], f[c], f[c + 1], (REAL)1);
                };
                REAL L, Rr, Ldf, Rdf;
                if (i == 0) { L = Fp[i]; Rr = Fm[i + 1]; Ldf = 0; Rdf = sl(Fm, i + 1); }
                else if (i == n - 1) { L = Fp[i - 1]; Rr = Fm[i]; Ldf = sl(Fp, i - 1); Rdf = 0; }
                else { L = Fp[i - 1]; Rr = Fm[i + 1]; Ldf = sl(Fp, i - 1); Rdf = sl(Fm, i + 1); }
                u = sub_scaled(u, g.lx, Fp[i] - Fm[i] + Rr - L);
                u = sub_half_scaled(u, g.hlx, sl(Fp, i) + sl(Fm, i) - Rdf - Ldf);
            }
            U[(long)k * n + i] = u;
        }
    }
}

#undef D

// ---------------- host launchers ----------------
template <typename REAL>
static cudaError_t step_t(const PlainArgs& a) {
    shll_count_launches(1);
    Gas<REAL> g = make_gas<REAL>(a);
    const REAL* Uin = static_cast<const REAL*>(a.Uin);
    REAL* Uout = static_cast<REAL*>(a.Uout);
    if (a.dim == 1) {
        dim3 grid((a.nx + T1 - 1) / T1);
        if (a.order == 1) k_step1<REAL, 1><<<grid, T1, 0, a.stream>>>(Uin, Uout, a.nx, g, a.flag);
        else k_step1<REAL, 2><<<grid, T1, 0, a.stream>>>(Uin, Uout, a.nx, g, a.flag);
    } else {
        cudaError_t e = cudaSuccess;
        const int TI = tile_rows(a.nx, a.ny, a.order, device_sm_count(), sizeof(REAL) == 8);
        auto* kern = a.order == 1 ? k_step2<REAL, 1> : k_step2<REAL, 2>;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = tile_grid(a.nx, a.ny, TI);
        cfg.blockDim = dim3((unsigned)tile_threads(TI, a.order));
        cfg.dynamicSmemBytes = smem2<REAL>(TI, a.order);
        cfg.stream = a.stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = a.chained ? 1 : 0;
        if (e == cudaSuccess && !a.chained)
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2<REAL>(20, a.order));
        if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, kern, Uin, Uout, a.nx, a.ny, g, a.flag, TI);
        if (e != cudaSuccess) return e;
    }
    return cudaGetLastError();
}

template <typename REAL>
static cudaError_t stage_t(const PlainArgs& a, int which) {
    shll_count_launches(1);
    Gas<REAL> g = make_gas<REAL>(a);
    const long n = (long)a.nx * (a.dim == 2 ? a.ny : 1);
    const int threads = 256;
    int blocks = (int)std::min<long>((n + threads - 1) / threads, 152L * 16);
    REAL* U = static_cast<REAL*>(a.Uout);
    REAL* P = static_cast<REAL*>(a.P);
    switch (which) {
        case STAGE_U_FROM_P: k_u_from_p<REAL><<<blocks, threads, 0, a.stream>>>(P, U, n, a.dim, g); break;
        case STAGE_P_FROM_U: k_p_from_u<REAL><<<blocks, threads, 0, a.stream>>>(U, P, n, a.dim, g, a.flag); break;
        case STAGE_F_FROM_P:
            k_f_from_p<REAL><<<blocks, threads, 0, a.stream>>>(U, P, static_cast<REAL*>(a.fp), static_cast<REAL*>(a.fm),
                                                             static_cast<REAL*>(a.hp), static_cast<REAL*>(a.hm), n,
                                                             a.dim, g);
            break;
        case STAGE_UPDATE: {
            const REAL *fp = static_cast<const REAL*>(a.fp), *fm = static_cast<const REAL*>(a.fm);
            if (a.dim == 1) {
                k_update1_staged<REAL><<<blocks, threads, 0, a.stream>>>(U, fp, fm, a.nx, a.order, g);
                break;
            }
            const int TI = tile_rows(a.nx, a.ny, a.order, device_sm_count(), sizeof(REAL) == 8);
            auto* kern = a.order == 1 ? k_update2_staged<REAL, 1> : k_update2_staged<REAL, 2>;
            cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem2<REAL>(20, a.order));
            if (e != cudaSuccess) return e;
            kern<<<tile_grid(a.nx, a.ny, TI), tile_threads(TI, a.order), smem2<REAL>(TI, a.order), a.stream>>>(
                U, fp, fm, static_cast<const REAL*>(a.hp), static_cast<const REAL*>(a.hm), a.nx, a.ny, g, TI);
            break;
        }
        case STAGE_LOAD:
            k_check_planes<REAL><<<blocks, threads, 0, a.stream>>>(a.planes, n, a.dim == 2 ? 4 : 3, a.worst);
            k_load_planes<REAL, double><<<blocks, threads, 0, a.stream>>>(a.planes, (a.dim + 1) * n, a.planes + n, P, U, n, a.dim,
                                                                         g, a.worst, a.flag);
            shll_count_launches(1);
            break;
        case STAGE_DUMP:
            k_dump_planes<REAL><<<blocks, threads, 0, a.stream>>>(P, a.planes, n * (a.dim == 2 ? 4 : 3));
            break;
        default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

// `work` holds two planes of doubles (2D), or one and a plane of REAL (1D).  Density and temperature are checked
// before anything of the state is written (in 1D the density waits as REAL beside the temperature).
// Against planes for all four at once (2D, pinned memory): 401 x 397 cells 75 -> 89 us, 700 x 700 131 -> 140,
// 1400 x 1400 385 -> 399; one plane at a time 115, 171, 432.
template <typename REAL>
static cudaError_t load_by_planes_t(const PlainArgs& a, const double* const* in, void* work) {
    const Gas<REAL> g = make_gas<REAL>(a);
    const long n = (long)a.nx * (a.dim == 2 ? a.ny : 1);
    const int threads = 256, blocks = (int)std::min<long>((n + threads - 1) / threads, 152L * 16);
    double* plane = static_cast<double*>(work);
    REAL* P = static_cast<REAL*>(a.P);
    REAL* PT = P + (a.dim + 1) * n;
    cudaError_t e = cudaSuccess;
    auto copy = [&](double* to, const double* from) {
        if (e == cudaSuccess) e = cudaMemcpyAsync(to, from, sizeof(double) * n, cudaMemcpyHostToDevice, a.stream);
    };
    copy(plane, in[0]);
    if (a.dim == 2) {
        copy(plane + n, in[3]);
        k_check_planes<REAL><<<blocks, threads, 0, a.stream>>>(plane, n, 2, a.worst);
        k_take_plane<REAL, double><<<blocks, threads, 0, a.stream>>>(plane, P, n, a.worst);
        k_take_plane<REAL, double><<<blocks, threads, 0, a.stream>>>(plane + n, PT, n, a.worst);
    } else {
        REAL* held = reinterpret_cast<REAL*>(plane + n);
        k_check_planes<REAL><<<blocks, threads, 0, a.stream>>>(plane, n, 1, a.worst);
        k_take_plane<REAL, double><<<blocks, threads, 0, a.stream>>>(plane, held, n, nullptr);
        copy(plane, in[2]);
        k_check_planes<REAL><<<blocks, threads, 0, a.stream>>>(plane, n, 1, a.worst);
        k_take_plane<REAL, REAL><<<blocks, threads, 0, a.stream>>>(held, P, n, a.worst);
        k_take_plane<REAL, double><<<blocks, threads, 0, a.stream>>>(plane, PT, n, a.worst);
    }
    for (int k = 0; k < a.dim; k++) copy(plane + k * n, in[1 + k]);
    k_load_planes<REAL, REAL><<<blocks, threads, 0, a.stream>>>(P, (a.dim + 1) * n, plane, P, static_cast<REAL*>(a.Uout), n, a.dim,
                                                                g, a.worst, a.flag);
    shll_count_launches(a.dim == 2 ? 4 : 6);
    return e == cudaSuccess ? cudaGetLastError() : e;
}
template <typename REAL>
static cudaError_t dump_by_planes_t(const PlainArgs& a, double* const* out, void* work) {
    const long n = (long)a.nx * (a.dim == 2 ? a.ny : 1);
    const int blocks = (int)std::min<long>((n + 255) / 256, 152L * 16);
    double* plane = static_cast<double*>(work);
    cudaError_t e = cudaSuccess;
    for (int k = 0; k < a.dim + 2 && e == cudaSuccess; k += a.dim) {   // a.dim planes at a time
        const int m = std::min(a.dim, a.dim + 2 - k);
        k_dump_planes<REAL><<<blocks, 256, 0, a.stream>>>(static_cast<const REAL*>(a.P) + k * n, plane, m * n);
        shll_count_launches(1);
        for (int q = 0; q < m && e == cudaSuccess; q++)
            if (out[k + q]) e = cudaMemcpyAsync(out[k + q], plane + q * n, sizeof(double) * n, cudaMemcpyDeviceToHost, a.stream);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    return e == cudaSuccess ? cudaStreamSynchronize(a.stream) : e;
}

}  // namespace SHLL_PLAIN_NS
