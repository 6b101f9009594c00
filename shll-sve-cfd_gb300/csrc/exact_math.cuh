// Correctly rounded FP64 division and square root on the integer pipes, and the reference's mixed
// float/double expressions in FP32 only.
//
// GB300 executes FP64 arithmetic, comparisons and conversions at 1.68 lanes per clock per SM (one
// warp instruction every 19 clocks per SM, 64 clocks of latency), 32-bit integer operations at about
// 108.  An FP64 division or square root on the FP64 pipe takes about 600 clocks (measured), as long as nine
// dependent FP64 operations; the integer forms here are about 60 integer operations (about 250 clocks),
// with the same correctly rounded results bit for bit.  They are long division / digit-by-digit square root in
// a large radix (Knuth, TAOCP vol. 2, 4.3.1): a first partial result of 30 bits from a 32-bit
// reciprocal (Newton's iteration on the FP32 seed), the exact 64-bit remainder, a second partial
// result of 23 bits, and a final correction by the sign of the exact remainder.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>

namespace exact_math {

// (host forms of the primitives, so that the same arithmetic can be checked and constants prepared
// on the CPU)
#define EM_FN __host__ __device__ __forceinline__
#ifdef __CUDA_ARCH__
#define EM_PICK(device, host) return device
#else
#define EM_PICK(device, host) return host
#endif
template <class To, class From>
EM_FN To em_cast(From x) {
    To y;
    memcpy(&y, &x, sizeof(y));
    return y;
}
EM_FN uint32_t em_mulhi(uint32_t a, uint32_t b) { EM_PICK(__umulhi(a, b), (uint32_t)(((uint64_t)a * b) >> 32)); }
EM_FN float em_rcp(float x) { EM_PICK(__fdividef(1.0f, x), 1.0f / x); }
EM_FN float em_rsqrt(float x) { EM_PICK(rsqrtf(x), (float)(1.0 / sqrt((double)x))); }
EM_FN uint32_t em_fbits(float x) { EM_PICK(__float_as_uint(x), em_cast<uint32_t>(x)); }
EM_FN float em_bitsf(uint32_t x) { EM_PICK(__uint_as_float(x), em_cast<float>(x)); }
EM_FN uint64_t em_dbits(double x) { EM_PICK((uint64_t)__double_as_longlong(x), em_cast<uint64_t>(x)); }
EM_FN double em_bitsd(uint64_t x) { EM_PICK(__longlong_as_double((long long)x), em_cast<double>(x)); }
EM_FN double em_hwdiv(double a, double b) { EM_PICK(__ddiv_rn(a, b), a / b); }
EM_FN double em_hwsqrt(double a) { EM_PICK(__dsqrt_rn(a), sqrt(a)); }
// (never contracted into a fused multiply-add)
EM_FN float em_add(float a, float b) { EM_PICK(__fadd_rn(a, b), a + b); }
EM_FN float em_mul(float a, float b) { EM_PICK(__fmul_rn(a, b), a * b); }
EM_FN float em_fma(float a, float b, float c) { EM_PICK(__fmaf_rn(a, b, c), fmaf(a, b, c)); }
EM_FN double em_add(double a, double b) { EM_PICK(__dadd_rn(a, b), a + b); }
EM_FN double em_mul(double a, double b) { EM_PICK(__dmul_rn(a, b), a * b); }

constexpr uint64_t kOne52 = 1ull << 52;

// an approximation of a value in (0.5, 1] as a 24-bit fixed-point number (x 2^24), clamped to
// [2^23, 2^24 - 1]
EM_FN uint32_t em_seed(float x) {
    int d = (int)em_fbits(x) - 0x3f000000;
    d = d < 0 ? 0 : d > 0x7fffff ? 0x7fffff : d;
    return (uint32_t)d + 0x800000u;
}

// A divisor b: its significand mb in [2^52, 2^53), a 32-bit reciprocal r <= 2^84 / mb (relative
// error below 2^-29), its bits.
struct Divisor {
    uint64_t mb, bits;
    uint32_t r;
};

EM_FN uint64_t em_significand(uint64_t bits) { return (bits & (kOne52 - 1)) | kOne52; }
EM_FN int em_exponent(uint64_t bits) { return (int)(bits >> 52) & 0x7ff; }

EM_FN Divisor divisor(double b) {
    Divisor d;
    d.bits = em_dbits(b);
    d.mb = em_significand(d.bits);
    // seed: 1 / beta, beta = mb / 2^52 cut to 24 bits, as a 24-bit fixed-point number R0 / 2^24
    const float bf = em_bitsf(0x3f800000u | ((uint32_t)(d.mb >> 29) & 0x7fffffu));
    const uint32_t R0 = em_seed(em_rcp(bf));
    // 1 - beta R0 / 2^24 = -D / 2^76 with |D| < 2^56: the low 64 bits of mb R0 are all of it
    const int32_t Dh = (int32_t)((int64_t)(d.mb * R0) >> 24);
    // one Newton step, scaled to 2^32 and lowered so that it never reaches 1 / beta
    d.r = (R0 << 8) - (uint32_t)((int32_t)(((int64_t)(int32_t)R0 * Dh) >> 32) >> 12) - 3u;
    return d;
}

// a / b, correctly rounded, for normal a and b whose quotient is normal (the exponents of both, and
// their difference, well inside the range; anything else gives a meaningless value and no fault)
EM_FN double divide_plain(double a, const Divisor& d) {
    const uint64_t ab = em_dbits(a);
    const uint64_t ma = em_significand(ab);
    const bool less = ma < d.mb;
    const uint64_t N = less ? ma + ma : ma;              // N / mb in [1, 2)
    // first 30 fraction bits, too small by a few units
    const uint32_t q1 = em_mulhi((uint32_t)(N >> 22), d.r);
    const int64_t rem1 = (int64_t)((N << 30) - (uint64_t)q1 * d.mb);
    // the next 22 bits, rounded: rem1 2^22 / mb = rem1 r / 2^62
    const int32_t q2 = (int32_t)(((int64_t)(int32_t)(rem1 >> 25) * (int32_t)(d.r >> 1)) >> 32);
    const int32_t r = (q2 + 8) >> 4;
    const int64_t rem2 = 2 * (int64_t)(((uint64_t)rem1 << 22) - (uint64_t)((int64_t)r * (int64_t)d.mb));
    uint64_t Q = ((uint64_t)q1 << 22) + (int64_t)r;
    // the quotient of two 53-bit numbers is never half way between two 53-bit numbers
    if (rem2 > (int64_t)d.mb) Q++;
    if (rem2 < -(int64_t)d.mb) Q--;
    // (Q's bit 52 adds one to the exponent field)
    const uint32_t hi = (uint32_t)(Q >> 32) + (uint32_t)((ab >> 32) & 0xfff00000u) - (uint32_t)((d.bits >> 32) & 0xfff00000u) +
                        ((less ? 1021u : 1022u) << 20);
    return em_bitsd(((uint64_t)hi << 32) | (uint32_t)Q);
}

// a / b, correctly rounded (round to nearest even); every special case as the hardware's
EM_FN double divide(double a, const Divisor& d) {
    const uint64_t ab = em_dbits(a);
    const int ea = em_exponent(ab), eb = em_exponent(d.bits);
    // (the plain division takes the divisor's sign for 0: flipped in below)
    if ((unsigned)(ea - 1) < 2046u && (unsigned)(eb - 1) < 2046u && (unsigned)(ea - eb + 1021) < 2043u) {
        Divisor p = d;
        p.bits &= ~(1ull << 63);
        return em_bitsd(em_dbits(divide_plain(a, p)) ^ (d.bits & (1ull << 63)));
    }
    // a zero dividend is common (gas at rest)
    if ((ab << 1) == 0 && (unsigned)(eb - 1) < 2046u) return em_bitsd((ab ^ d.bits) & (1ull << 63));
    return em_hwdiv(a, em_bitsd(d.bits));
}

// sqrt(a), correctly rounded, for a normal positive a; *root: it as a divisor (its reciprocal is a
// by-product)
EM_FN double square_root_plain(double a, Divisor* root) {
    const uint64_t ab = em_dbits(a);
    const int ea = (int)(ab >> 52);
    const int odd = (ea & 1) ^ 1;                        // unbiased exponent odd
    const uint64_t M = em_significand(ab) << odd;        // X = M / 2^52 in [1, 4)
    const uint32_t Mh = (uint32_t)(M >> 22);             // X 2^30
    // seed 1 / sqrt(X), one Newton step: y <- y + y (1 - X y^2) / 2, to about 2^-30
    const float xf = em_bitsf(0x3f800000u + ((uint32_t)odd << 23) + ((uint32_t)((ab & (kOne52 - 1)) >> 29)));
    const uint32_t Y0 = em_seed(em_rsqrt(xf));
    const uint32_t T = (uint32_t)(((uint64_t)Y0 * Y0) >> 16);   // y^2 2^32
    const int64_t e0 = (int64_t)((1ull << 62) - (uint64_t)T * Mh);   // (1 - X y^2) 2^62, |.| < 2^43
    const int64_t t = (int64_t)(int32_t)Y0 * (int32_t)(e0 >> 20);    // y e0 2^(24 + 42)
    const uint32_t y = (Y0 << 8) + (uint32_t)((int32_t)(t >> 32) >> 3) - 4u;   // y (1 + e0 / 2) 2^32
    // first 30 fraction bits, then 22 more from the exact remainder
    const uint32_t s1 = em_mulhi(Mh, y);
    const int64_t rem1 = (int64_t)((M << 8) - (uint64_t)s1 * s1);
    const int64_t s2 = (int64_t)(int32_t)(rem1 >> 6) * (int32_t)(y >> 1);   // rem1 y 2^25
    const int32_t r = ((int32_t)(s2 >> 32) + 2) >> 2;    // rem1 2^22 / (2 s1) = rem1 y / 2^41, y = y' / 2^32
    uint64_t S = ((uint64_t)s1 << 22) + (int64_t)r;
    const int64_t rem = (int64_t)((M << 52) - S * S);
    if (rem > (int64_t)S) S++;
    if (rem <= -(int64_t)S) S--;
    const int e = ((ea - odd - 1023) >> 1) + 1023;
    root->mb = S;
    root->r = y;
    root->bits = ((uint64_t)(uint32_t)(e - 1) << 52) + S;
    return em_bitsd(root->bits);
}

// sqrt(a), correctly rounded; every special case as the hardware's
EM_FN double square_root(double a) {
    Divisor root;
    if ((unsigned)((int)(em_dbits(a) >> 52) - 1) < 2046u) return square_root_plain(a, &root);
    return em_hwsqrt(a);
}

// x 2^k for a power of two the reference multiplies by (k small): the exponent field moves; zeros
// stay, subnormal operands or results and non-finite operands take the multiplication
EM_FN double scale_pow2(double x, int k, double pow2k) {
    const uint64_t b = em_dbits(x);
    const int e = (int)(b >> 52) & 0x7ff;
    if ((unsigned)(e + k - 1) < 2046u && (unsigned)(e - 1) < 2046u) return em_bitsd(b + ((int64_t)k << 52));
    return (b << 1) == 0 ? x : em_mul(x, pow2k);
}

// minmod(l, r): 0 when l * r < 0.0, else the one of smaller magnitude (r on a tie, or when l or r
// is a NaN), without FP64 instructions.  Sets *special where the sign of the FP64 product must be
// asked (non-finite operands, or a product that may underflow to zero): minmod_general.
EM_FN double minmod_plain(double l, double r, bool* special) {
    const uint64_t lb = em_dbits(l), rb = em_dbits(r);
    const uint64_t la = lb << 1, ra = rb << 1;
    const int el = (int)(la >> 53), er = (int)(ra >> 53);
    // (1080: a subnormal's exponent, 0 here, stands for up to 52 less; and l and r may be scaled by 2 each)
    *special = *special || (el + er < 1080 && la != 0 && ra != 0) || el == 2047 || er == 2047;
    const bool negative = (int32_t)((lb ^ rb) >> 32) < 0 && la != 0 && ra != 0;
    const uint64_t m = la < ra ? lb : rb;
    return em_bitsd(negative ? 0 : m);
}
// (inv_scale: 1 / the scale of l and r, for the product)
EM_FN double minmod_general(double l, double r, double inv_scale) {
    if (em_mul(em_mul(l, inv_scale), em_mul(r, inv_scale)) < 0.0) return 0.0;
    return fabs(l) < fabs(r) ? l : r;
}

// ---- the published arithmetic's double expressions of float values, in FP32 -----------------
// The reference's float solver widens some expressions to double (its 0.5 and 1.0 literals, sqrt) and
// rounds the result back to float.  Each value below is first evaluated in FP32 as an unevaluated sum
// R + rem that is exact to 2^-18 of half a unit in R's last place (half_ulp; 2^-21 where no
// cancellation magnifies the rounding of a low part, up to 2^4 is let through); when rem is
// clear of the half-way points the rounded double expression can only be R, otherwise (a chance of
// about 2^-17) the double expression itself decides.

// the double expressions themselves, out of line so that none of their FP64 instructions is issued
// ahead of the branch that needs them
#ifdef __CUDACC__
#define EM_SLOW __host__ __device__ __noinline__
#else
#define EM_SLOW inline
#endif
static EM_SLOW float temperature_slow(float e, float kh, float kl, float c) {
    return (float)em_hwdiv(em_add((double)e, -((double)kh + (double)kl)), (double)c);
}
static EM_SLOW float z2_slow(float a, float t) { return (float)em_mul(0.5 * (double)a, em_add(1.0, -(double)t)); }
static EM_SLOW float sub_product_slow(float u, float c, float s) {
    return (float)em_add((double)u, -em_mul((double)c, (double)s));
}

// true when R + rem (exact as above) certainly rounds to R, R in the middle of the range
EM_FN bool rounds_to(float R, float rem) {
    const uint32_t b = em_fbits(R), e = b & 0x7f800000u;
    const float half_ulp = em_bitsf(e - (24u << 23));
    const float lim = (b & 0x7fffffu) == 0u ? 0.49f : 0.99999237060546875f;   // 1 - 2^-17
    return e > (40u << 23) && e < (240u << 23) && fabsf(rem) < lim * half_ulp;
}
// s + e = a + b exactly
EM_FN float two_sum(float a, float b, float& e) {
    const float s = em_add(a, b), bp = em_add(s, -a);
    e = em_add(em_add(a, -em_add(s, -bp)), em_add(b, -bp));
    return s;
}

// FP32 quotients and square roots, correctly rounded, for operands and results well inside the range
// (a zero dividend included): a residual step with a refined reciprocal (Markstein, IBM J. Res. Dev. 34
// (1990) 111), without the range branches of the general forms.
// y: 1 / b, refined
EM_FN float reciprocal_plain(float b, float y) { return em_fma(em_fma(-b, y, 1.0f), y, y); }
EM_FN float divide_plain(float a, float b, float y) {
    const float q = em_mul(a, y);
    return em_fma(em_fma(-q, b, a), y, q);
}
// *y: about 1 / sqrt(x)
EM_FN float square_root_plain(float x, float* y) {
    float r = em_rsqrt(x);
    r = em_fma(em_mul(0.5f, r), em_fma(-em_mul(x, r), r, 1.0f), r);
    const float s = em_mul(x, r);
    *y = r;
    return em_fma(em_fma(-s, s, x), em_mul(0.5f, r), s);
}

// (float)((D(e) - k) / D(c)) with k = kh + kl the exact subtrahend (D(k) a double of at most 48
// bits) and rc an approximation of 1 / c
// (*ok cleared: the value may be the other neighbour, temperature_slow decides)
EM_FN float temperature_plain(float e, float kh, float kl, float c, float rc, bool* ok) {
    float sl;
    const float sh = two_sum(e, -kh, sl);
    sl = em_add(sl, -kl);
    const float qh = em_mul(sh, rc);
    const float ql = em_mul(em_add(em_fma(-qh, c, sh), sl), rc);
    const float R = em_add(qh, ql);
    const float rem = em_add(ql, -em_add(R, -qh));
    // (no large cancellation, which would magnify the rounding of sl)
    *ok = *ok && rounds_to(R, rem) && fabsf(kh) < 16.0f * fabsf(sh);
    return R;
}
EM_FN float temperature_ref(float e, float kh, float kl, float c, float rc) {
    bool ok = true;
    const float R = temperature_plain(e, kh, kl, c, rc, &ok);
    return ok ? R : temperature_slow(e, kh, kl, c);
}

// (float)(0.5 * D(a) * (1.0 - D(t)))
EM_FN float z2_plain(float a, float t, bool* ok) {
    float wl;
    const float wh = two_sum(1.0f, -t, wl);
    const float ph = em_mul(a, wh);
    const float pl = em_fma(a, wl, em_fma(a, wh, -ph));
    const float R = em_add(ph, pl);
    const float rem = em_add(pl, -em_add(R, -ph));
    *ok = *ok && rounds_to(R, rem);
    return em_mul(0.5f, R);
}
EM_FN float z2_ref(float a, float t) {
    bool ok = true;
    const float z = z2_plain(a, t, &ok);
    return ok ? z : z2_slow(a, t);
}

// (float)(D(u) - D(c) * D(s)) for a float c (the product is exact in double)
EM_FN float sub_product_ref(float u, float c, float s) {
    const float ph = em_mul(c, s), pl = em_fma(c, s, -ph);
    float sl;
    const float sh = two_sum(u, -ph, sl);
    // c a power of two: one exact product, and a double rounding of a float sum is the float sum
    if (pl == 0.0f && (fabsf(ph) > 1.0e-30f || s == 0.0f)) return sh;
    sl = em_add(sl, -pl);
    const float R = em_add(sh, sl);
    const float rem = em_add(sl, -em_add(R, -sh));
    if (rounds_to(R, rem) && fabsf(ph) < 16.0f * fabsf(sh)) return R;
    return sub_product_slow(u, c, s);
}

}  // namespace exact_math
