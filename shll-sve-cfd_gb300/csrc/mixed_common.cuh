// Device helpers of the mixed-precision engine: FP32-pair (compensated) arithmetic and the
// split fluxes of a cell evaluated in FP32 as deviations from an anchor state.
//
// Split fluxes (base-c/base_shll.c:134-158):  M = u/a, Z1 = (M+1)/2, Z2 = a(1-M^2)/2,
// Z3 = (M-1)/2 = Z1 - 1, P = rho R T, F = (m, m u + P, u (E + P)),
// fp = F Z1 + U Z2, fm = -F Z3 - U Z2.  Every quantity q is written as q* + dq with q* the
// anchor value; the deviations obey exact identities, e.g.
//   du = (dm - u* drho)/rho,  de = (dE - e* drho)/rho,  dT = (de - (u + u*) du / 2)/CV,
//   da = gamma R dT/(a + a*),  dM = (du - M* da)/a,  dZ2 = (da (1-M^2) - a* (M + M*) dM)/2,
//   dP = (gamma-1)(dE - (dm u + m* du)/2),  dfp = dF Z1 + F* dZ1 + dU Z2 + U* dZ2,
//   dfm = dF - dfp,
// in which the anchor values only multiply deviations.  Rounding errors are therefore relative
// to |U - U*|; reciprocals and square roots may use the fast approximations.
#pragma once
#include <cuda_runtime.h>

struct AnchorCoef {
    float rho, u, v, e, T, a, M, P, Z1, Z2, gR, R, cvinv;
    float F[4], Uf[4];
};

// h + l += v (TwoSum; the rounding error goes to l)
__device__ __forceinline__ void two_sum_acc(float& h, float& l, float v) {
    float s = __fadd_rn(h, v);
    float bp = __fadd_rn(s, -h);
    float e = __fadd_rn(__fadd_rn(h, -__fadd_rn(s, -bp)), __fadd_rn(v, -bp));
    h = s;
    l = __fadd_rn(l, e);
}

__device__ __forceinline__ void split2(double d, float& h, float& l) {
    h = (float)d;
    l = (float)(d - (double)h);
}

// (oh, ol) = (ah + al) + (bh + bl), renormalised
__device__ __forceinline__ void ff_add(float ah, float al, float bh, float bl, float& oh, float& ol) {
    float s = __fadd_rn(ah, bh);
    float bp = __fadd_rn(s, -ah);
    float e = __fadd_rn(__fadd_rn(ah, -__fadd_rn(s, -bp)), __fadd_rn(bh, -bp));
    e = __fadd_rn(e, __fadd_rn(al, bl));
    oh = __fadd_rn(s, e);
    ol = __fadd_rn(e, -__fadd_rn(oh, -s));
}
__device__ __forceinline__ void ff_sub(float ah, float al, float bh, float bl, float& oh, float& ol) {
    ff_add(ah, al, -bh, -bl, oh, ol);
}

__device__ __forceinline__ float fast_rcp(float x) { return __fdividef(1.0f, x); }

// ---- packed FP32x2: two cells per thread, one f32x2 instruction per operation --------------
// (__fadd2_rn / __fmul2_rn / __ffma2_rn: the sm_100-family packed FP32 instructions, each lane
// rounded to nearest exactly like the scalar operation, so a packed lane and a scalar evaluation
// of the same formula give identical bits)
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
// a - b per lane: the packed subtract (sub.rn.f32x2), the same bits as a + (-b).  Written out
// because the compiler does not fold the negation of a packed operand into the packed add (the
// resident 1D sweep ran 1.5 % faster with this form on GB300)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    unsigned long long d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d)
        : "l"(*reinterpret_cast<const unsigned long long*>(&a)), "l"(*reinterpret_cast<const unsigned long long*>(&b)));
    return *reinterpret_cast<const float2*>(&d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
// a * b per lane, never fused into a sum that follows: a product whose only use is a packed sum is
// fused with it by the assembler, even as mul.rn (the same value unless the product is subnormal, where
// a fused term would differ from the one that the neighbouring cell or the record of a tile edge sees).
// A fused multiply-add of zero rounds like the product and costs the same.
__device__ __forceinline__ float2 mul2_alone(float2 a, float2 b) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d)
        : "l"(*reinterpret_cast<const unsigned long long*>(&a)), "l"(*reinterpret_cast<const unsigned long long*>(&b)), "l"(0ull));
    return *reinterpret_cast<const float2*>(&d);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 rcp2(float2 a) { return make_float2(fast_rcp(a.x), fast_rcp(a.y)); }
__device__ __forceinline__ float2 rsqrt2(float2 a) { return make_float2(rsqrtf(a.x), rsqrtf(a.y)); }
// the same operations on one cell, with the same names so that both forms share one text (V = float2 or
// float below)
__device__ __forceinline__ float neg2(float a) { return -a; }
__device__ __forceinline__ float add2(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub2(float a, float b) { return __fadd_rn(a, -b); }
__device__ __forceinline__ float mul2(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fma2(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ float rcp2(float a) { return fast_rcp(a); }
__device__ __forceinline__ float rsqrt2(float a) { return rsqrtf(a); }
template <class V>
__device__ __forceinline__ V splat(float a);
template <>
__device__ __forceinline__ float2 splat<float2>(float a) { return f2(a); }
template <>
__device__ __forceinline__ float splat<float>(float a) { return a; }
// lane q of a float2 (q a compile-time constant after unrolling)
__device__ __forceinline__ float lane(float2 v, int q) { return q ? v.y : v.x; }
__device__ __forceinline__ void set_lane(float2& v, int q, float x) { if (q) v.y = x; else v.x = x; }

// h + l += v per lane (TwoSum)
template <class V>
__device__ __forceinline__ void two_sum_acc2(V& h, V& l, V v) {
    const V s = add2(h, v);
    const V bp = sub2(s, h);
    const V e = add2(sub2(h, sub2(s, bp)), sub2(v, bp));
    h = s;
    l = add2(l, e);
}
// h + l -= v per lane: the same bits as two_sum_acc2(h, l, -v) (negation commutes with rounding
// to nearest: (-v) - bp = -(v + bp))
template <class V>
__device__ __forceinline__ void two_diff_acc2(V& h, V& l, V v) {
    const V s = sub2(h, v);
    const V bp = sub2(s, h);
    const V e = sub2(sub2(h, sub2(s, bp)), add2(v, bp));
    h = s;
    l = add2(l, e);
}

// minmod(a, b): the smaller magnitude with the common sign when a and b have the same sign,
// else 0.  Three integer/min-max operations: t = min(|a|,|b|) carrying sign(a) xor sign(b)
// (PTX min.xorsign.abs), r = max(t, 0) (0 unless the signs agree), then sign(a) on r.
// Symmetric in a and b up to the sign of a zero result, so threads that evaluate the same slope
// get the same value.
__device__ __forceinline__ float minmod_s(float a, float b) {
    float t;
    asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(t) : "f"(a), "f"(b));
    const float r = fmaxf(t, 0.f);
    return __uint_as_float(__float_as_uint(r) | (__float_as_uint(a) & 0x80000000u));
}
__device__ __forceinline__ float2 minmod2(float2 a, float2 b) {
    return make_float2(minmod_s(a.x, b.x), minmod_s(a.y, b.y));
}
// limited slope from the backward and forward differences a = f_j - f_{j-1}, b = f_{j+1} - f_j:
// minmod (LIM = 0) or the MC limiter minmod((a+b)/2, alpha minmod(a,b)) (LIM = 1,
// base-omp/2nd_order_base_shll.c:316-325)
template <int LIM>
__device__ __forceinline__ float slope_s(float a, float b, float alpha) {
    if (LIM == 1) return minmod_s(__fmul_rn(0.5f, __fadd_rn(a, b)), __fmul_rn(alpha, minmod_s(a, b)));
    return minmod_s(a, b);
}
template <int LIM>
__device__ __forceinline__ float2 slope2(float2 a, float2 b, float alpha) {
    if (LIM == 1) return minmod2(mul2(f2(0.5f), add2(a, b)), mul2(f2(alpha), minmod2(a, b)));
    return minmod2(a, b);
}

// anchor coefficients of a 1D frame, each duplicated into both lanes (negated where the
// formulas subtract them)
template <class V>
struct CoefV {
    V rho, u, nu, ne, T, a, na, M, nM, Z1, Z2, P, gR, R, cvinv, gm1;
    V F[3], Uf[3];
};
template <class V>
__device__ __forceinline__ CoefV<V> coef2(const AnchorCoef& c) {
    CoefV<V> k;
    const auto f2 = [](float a) { return splat<V>(a); };
    k.rho = f2(c.rho); k.u = f2(c.u); k.nu = f2(-c.u); k.ne = f2(-c.e); k.T = f2(c.T); k.a = f2(c.a); k.na = f2(-c.a);
    k.M = f2(c.M); k.nM = f2(-c.M); k.Z1 = f2(c.Z1); k.Z2 = f2(c.Z2); k.P = f2(c.P); k.gR = f2(c.gR);
    k.R = f2(c.R);
    k.cvinv = f2(c.cvinv);
    k.gm1 = f2(__fmul_rn(c.R, c.cvinv));   // R / CV = gamma - 1
    for (int i = 0; i < 3; i++) { k.F[i] = f2(c.F[i]); k.Uf[i] = f2(c.Uf[i]); }
    return k;
}

// 1D split-flux deviations of two cells at once (the conserved deviations d = (drho, dm, dE) of
// both cells as the lanes of FP32x2 registers; V = float: of one cell)
template <class V>
__device__ __forceinline__ void dflux1x2(const CoefV<V>& c, const V d[3], V dfp[3], V dfm[3]) {
    const V drho = d[0], dm = d[1], dE = d[2];
    const V rho = add2(c.rho, drho);
    const V r = rcp2(rho);
    const V du = mul2(fma2(c.nu, drho, dm), r);
    const V u = add2(c.u, du);
    const V de = mul2(fma2(c.ne, drho, dE), r);
    const V dT = mul2(fma2(splat<V>(-0.5f), mul2(add2(u, c.u), du), de), c.cvinv);
    const V T = add2(c.T, dT);
    const V gRT = mul2(c.gR, T);
    const V ainv = rsqrt2(gRT);
    const V da = mul2(mul2(c.gR, dT), rcp2(fma2(gRT, ainv, c.a)));   // (a = gRT ainv)
    const V dM = mul2(fma2(c.nM, da, du), ainv);
    const V M = add2(c.M, dM);
    const V dZ1 = mul2(splat<V>(0.5f), dM);
    const V Z1 = add2(c.Z1, dZ1);
    // (negations folded into the operations: -M = (-M*) - dM and -(a* s dM) = ((-a*) s) dM, the
    // same bits as negating the results)
    const V omm = fma2(sub2(c.nM, dM), M, splat<V>(1.0f));
    const V dZ2 = mul2(splat<V>(0.5f), fma2(da, omm, mul2(mul2(c.na, add2(M, c.M)), dM)));
    const V Z2 = add2(c.Z2, dZ2);
    // P = (gamma-1)(E - m u / 2): dP = (gamma-1)(dE - (dm u + m* du) / 2).  At a contact (P and u
    // continuous) this cancels kinetic-energy-sized terms, where R (drho T + rho* dT) would cancel
    // internal-energy-sized ones
    const V x = fma2(splat<V>(-0.5f), fma2(dm, u, mul2(c.Uf[1], du)), dE);   // dP = gm1 x
    const V P = fma2(c.gm1, x, c.P);
    const V E = add2(c.Uf[2], dE);
    V dF[3];
    dF[0] = dm;
    dF[1] = fma2(c.gm1, x, fma2(dm, u, mul2(c.Uf[1], du)));
    dF[2] = fma2(du, add2(E, P), mul2(c.u, fma2(c.gm1, x, dE)));
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const V a1 = fma2(dF[k], Z1, mul2(c.F[k], dZ1));
        const V a2 = fma2(d[k], Z2, mul2(c.Uf[k], dZ2));
        dfp[k] = add2(a1, a2);
        // fp + fm = F (Z1 - Z3 = 1).  Besides saving the minus-flux products, the difference keeps
        // dfp + dfm = dF to one rounding, which the separately rounded form -(dF Z3 + F* dZ1 + d Z2)
        // did not: on strong tubes with supersonic flow (where this split amplifies perturbations)
        // the FP32-flux error fell from about 1e-2 to 3e-6 against FP64
        dfm[k] = sub2(dF[k], dfp[k]);
    }
}

// ---- FP64 <-> FP32 conversions on the integer pipes --------------------------------------
// GB300 executes FP64 arithmetic and F2F conversions at 2 lanes per clock per SM, so the
// once-per-sweep conversions are done with bit operations instead (IEEE-754 layouts:
// float = s | e8 | m23, double = s | e11 | m52; exponent biases 127 and 1023).

// float -> double, exact for normal floats and zero; subnormal floats become signed zero,
// infinities and NaNs stay non-finite
__device__ __forceinline__ double f2d_bits(float f) {
    const unsigned b = __float_as_uint(f);
    const unsigned e = (b >> 23) & 0xffu;
    unsigned hi = (b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + ((1023u - 127u) << 20));
    unsigned lo = b << 29;
    if (e == 0u) { hi = b & 0x80000000u; lo = 0u; }
    if (e == 0xffu) hi |= 0x7ff00000u;
    return __hiloint2double((int)hi, (int)lo);
}

// double -> FP32 pair (h, l): h = x truncated to 24 significant bits, l = x - h (29 bits)
// rounded to nearest FP32, so |x - (h + l)| <= 2^-48 |x|.  |x| < 2^-126 gives (0, 0) and
// 2^-126 <= |x| < 2^-74 gives l = 0 (absolute error below 2^-97); |x| >= 2^128 and
// non-finite x give a NaN h.
__device__ __forceinline__ void d2ff_bits(double x, float& h, float& l) {
    const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
    const unsigned e = (hi >> 20) & 0x7ffu;
    const unsigned s = hi & 0x80000000u;
    // h: sign | (e - 896) << 23 | top 23 mantissa bits (20 from hi, 3 from lo)
    const unsigned hb = s | ((((hi & 0x7fffffffu) - (896u << 20)) << 3) & 0x7fffffffu) | (lo >> 29);
    // l: the low 29 mantissa bits as an integer r, times 2^(e - 1075); r is converted exactly in
    // two 23-bit halves through the 2^23 magic-number trick, the final fma rounds once
    const unsigned r = lo & 0x1fffffffu;
    const float rh = __fadd_rn(__uint_as_float(0x4b000000u | (r >> 6)), -8388608.0f);
    const float rl = __fadd_rn(__uint_as_float(0x4b000000u | (r & 63u)), -8388608.0f);
    const float rf = __fmaf_rn(rh, 64.0f, rl);
    const float scale = __uint_as_float((e - 948u) << 23);  // 2^(e - 1075), valid for e in [949, 1202]
    const float lf = __uint_as_float(__float_as_uint(__fmul_rn(rf, scale)) | s);
    if (e < 897u) { h = __uint_as_float(s); l = __uint_as_float(s); }
    else if (e > 1150u) { h = __uint_as_float(0x7fc00000u); l = 0.f; }
    else { h = __uint_as_float(hb); l = e < 949u ? __uint_as_float(s) : lf; }
}
__device__ __forceinline__ float d2f_bits(double x) {  // truncation to FP32 (same range rules)
    float h, l;
    d2ff_bits(x, h, l);
    return h;
}

// ---- double-FP32 ("float-float") arithmetic on packed FP32x2 lanes ----------------------------
// A value is an unevaluated sum h + l of two FP32 numbers (about 48 significant bits).  Products
// use the exact FMA residual (fma(a, b, -a*b) is the rounding error of a*b), sums the TwoSum
// error-free transformation; the absolute error of a sum or product is about 2^-46 of its largest
// operand.  Used by the first-order sweeps of chunks in supersonic flow, where the reference scheme
// amplifies per-step rounding errors (its split gives the u - a wave the negative numerical
// viscosity a(1 - M)/2 once M > 1), so that FP32 rounding is not enough there.
template <class V>
struct FFV {
    V h, l;
};
using FF2 = FFV<float2>;
using FFS = FFV<float>;   // one cell or lane (a scalar instruction takes half the issue time of a packed one)
template <class V = float2>
__device__ __forceinline__ FFV<V> ffv(float h, float l) { return {splat<V>(h), splat<V>(l)}; }
// a * s for a power of two s (exact)
template <class V>
__device__ __forceinline__ FFV<V> ffscale(FFV<V> a, float s) { return {mul2(a.h, splat<V>(s)), mul2(a.l, splat<V>(s))}; }
// renormalisation of p + e with |e| small against |p|
template <class V>
__device__ __forceinline__ FFV<V> ffnorm(V p, V e) {
    const V h = add2(p, e);
    return {h, sub2(e, sub2(h, p))};
}
// renormalisation of p + x y, the product unrounded
template <class V>
__device__ __forceinline__ FFV<V> ffnorm_mul(V p, V x, V y) {
    const V h = fma2(x, y, p);
    return {h, fma2(x, y, sub2(p, h))};
}
// sum without the final renormalisation: (s, e) with e = the rounding error of the high parts plus
// the low parts; for sums that feed another sum or a product
template <class V>
__device__ __forceinline__ FFV<V> ffadd_u(FFV<V> a, FFV<V> b) {
    const V s = add2(a.h, b.h);
    const V bp = sub2(s, a.h);
    const V e = add2(sub2(a.h, sub2(s, bp)), sub2(b.h, bp));
    return {s, add2(e, add2(a.l, b.l))};
}
template <class V>
__device__ __forceinline__ FFV<V> ffadd(FFV<V> a, FFV<V> b) {
    const FFV<V> t = ffadd_u(a, b);
    return ffnorm(t.h, t.l);
}
// ffadd(a, -b), written with packed subtracts: a packed operand's negation is not folded, it costs an
// instruction per lane
template <class V>
__device__ __forceinline__ FFV<V> ffsub(FFV<V> a, FFV<V> b) {
    const V s = sub2(a.h, b.h);
    const V bp = sub2(s, a.h);
    const V e = sub2(sub2(a.h, sub2(s, bp)), add2(b.h, bp));
    return ffnorm(s, add2(e, sub2(a.l, b.l)));
}
// product left unnormalised, (p, e) with |e| <= about 2^-22 |p|; for products that feed a sum or
// another product, which renormalise
template <class V>
__device__ __forceinline__ FFV<V> ffmul_u(FFV<V> a, FFV<V> b) {
    const V p = mul2(a.h, b.h);
    V e = fma2(a.h, b.h, neg2(p));
    e = fma2(a.h, b.l, e);
    return {p, fma2(a.l, b.h, e)};
}
template <class V>
__device__ __forceinline__ FFV<V> ffmul(FFV<V> a, FFV<V> b) {
    const FFV<V> t = ffmul_u(a, b);
    return ffnorm(t.h, t.l);
}
// 1/a: r0 = approximate FP32 reciprocal, e = 1 - a r0 (FMA residuals), r = r0 (1 + e + e^2)
template <class V>
__device__ __forceinline__ FFV<V> ffrcp(FFV<V> a) {
    const V r0 = rcp2(a.h);
    V e = fma2(neg2(a.h), r0, splat<V>(1.0f));
    e = fma2(neg2(a.l), r0, e);
    return ffnorm_mul(r0, r0, fma2(e, e, e));
}
// sqrt(a), a > 0: FP32 estimate s0 from a Newton-refined reciprocal square root y, then
// s = s0 + (a - s0^2) y / 2 (the residual a - s0^2 from an FMA)
template <class V>
__device__ __forceinline__ FFV<V> ffsqrt(FFV<V> a) {
    V y = rsqrt2(a.h);
    y = mul2(y, fma2(mul2(splat<V>(-0.5f), a.h), mul2(y, y), splat<V>(1.5f)));
    const V s0 = mul2(a.h, y);
    const V e = add2(fma2(neg2(s0), s0, a.h), a.l);
    return ffnorm_mul(s0, mul2(splat<V>(0.5f), e), y);
}

// The split fluxes of two cells (FP32x2 lanes) with conserved state U (pairs), evaluated directly
// in double-FP32 arithmetic (base-c/base_shll.c:134-158 with P = (gamma-1)(E - m u / 2), which
// equals rho R T, and a^2 = gamma R T = gamma (gamma-1) (E - m u / 2) / rho).  Absolute errors are
// about 2^-45 of the flux magnitudes, so no deviation form is needed.  gg1 = gamma (gamma-1),
// gm1 = gamma - 1, as pairs.
template <class V>
__device__ __forceinline__ void flux1x2_ff(const FFV<V> U[3], FFV<V> gg1, FFV<V> gm1, FFV<V> fp[3], FFV<V> fm[3]) {
    const FFV<V> r = ffrcp(U[0]);
    const FFV<V> u = ffmul(U[1], r);
    const FFV<V> mu = ffmul_u(U[1], u);
    const FFV<V> eint = ffsub(U[2], ffscale(mu, 0.5f));
    const FFV<V> P = ffmul(gm1, eint);
    const FFV<V> a = ffsqrt(ffmul(gg1, ffmul_u(eint, r)));
    const FFV<V> M = ffmul(u, ffrcp(a));
    const FFV<V> Z1 = ffscale(ffadd(M, ffv<V>(1.0f, 0.0f)), 0.5f);
    const FFV<V> Z2 = ffmul(ffscale(a, 0.5f), ffsub(ffv<V>(1.0f, 0.0f), ffmul_u(M, M)));
    FFV<V> F[3];
    F[0] = U[1];
    F[1] = ffadd(mu, P);
    F[2] = ffmul(u, ffadd_u(U[2], P));
#pragma unroll
    for (int k = 0; k < 3; k++) {
        fp[k] = ffadd(ffmul_u(F[k], Z1), ffmul_u(U[k], Z2));
        fm[k] = ffsub(F[k], fp[k]);
    }
}

// minmod of two pairs per lane, as the reference's minmod (base-c/2nd_order_base_shll.c:191-201):
// 0 unless both have the same sign, else the one of smaller magnitude (the second on a tie); a
// pair's sign is that of its high part and magnitudes compare by high, then low parts
__device__ __forceinline__ float2 ffsel(bool q0, bool q1, float2 a, float2 b) {
    return make_float2(q0 ? a.x : b.x, q1 ? a.y : b.y);
}
__device__ __forceinline__ FF2 ffminmod(FF2 a, FF2 b) {
    bool pick_a[2], zero[2];
#pragma unroll
    for (int q = 0; q < 2; q++) {
        const float ah = lane(a.h, q), al = lane(a.l, q), bh = lane(b.h, q), bl = lane(b.l, q);
        zero[q] = !((ah > 0.f && bh > 0.f) || (ah < 0.f && bh < 0.f));
        const float sa = ah < 0.f ? -1.f : 1.f, sb = bh < 0.f ? -1.f : 1.f;
        const float mah = fabsf(ah), mbh = fabsf(bh);
        pick_a[q] = mah < mbh || (mah == mbh && __fmul_rn(sa, al) < __fmul_rn(sb, bl));
    }
    FF2 r = {ffsel(pick_a[0], pick_a[1], a.h, b.h), ffsel(pick_a[0], pick_a[1], a.l, b.l)};
    r.h = ffsel(zero[0], zero[1], f2(0.f), r.h);
    r.l = ffsel(zero[0], zero[1], f2(0.f), r.l);
    return r;
}
// limited slope from the differences a = f_j - f_{j-1}, b = f_{j+1} - f_j: minmod (LIM = 0) or the
// MC limiter minmod((a+b)/2, alpha minmod(a, b)) (LIM = 1, base-omp/2nd_order_base_shll.c:316-325)
template <int LIM>
__device__ __forceinline__ FF2 ffslope(FF2 a, FF2 b, float alpha) {
    if (LIM == 1) return ffminmod(ffscale(ffadd(a, b), 0.5f), ffmul(ffv(alpha, 0.f), ffminmod(a, b)));
    return ffminmod(a, b);
}
