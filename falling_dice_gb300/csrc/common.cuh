// common.cuh -- shared device helpers: FP64 vector/quaternion algebra, deterministic
// block reductions, launch geometry.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "kernels.h"

namespace mcg {

constexpr int kBlock = 256;          // threads per CTA for the streaming kernels
constexpr double kPiD = 3.1415926535897932384626433832795;

// ---- FP64 3-vectors and quaternions ----------------------------------------------------
// Same algebra as the reference's Vec3/Quat (MC/include/core.hpp:37-41): a vector divided
// by s is a multiplication with 1/s, and rotation is v + w t + q x t with t = 2 q x v.
struct d3 { double x, y, z; };
struct q4 { double w, x, y, z; };

__device__ __forceinline__ d3 operator+(d3 a, d3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ d3 operator-(d3 a, d3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ d3 operator-(d3 a) { return {-a.x, -a.y, -a.z}; }
__device__ __forceinline__ d3 operator*(d3 a, double s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ double dot(d3 a, d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ d3 cross(d3 a, d3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ double len2(d3 v) { return dot(v, v); }
__device__ __forceinline__ double len(d3 v) { return sqrt(len2(v)); }
__device__ __forceinline__ d3 unit(d3 v) {
    const double l2 = len2(v);
    return (isfinite(l2) && l2 > 1e-30) ? v * (1.0 / sqrt(l2)) : d3{0, 1, 0};
}
__device__ __forceinline__ double clampd(double x, double lo, double hi) { return fmax(lo, fmin(hi, x)); }
__device__ __forceinline__ double sqr(double x) { return x * x; }

__device__ __forceinline__ q4 conj(q4 q) { return {q.w, -q.x, -q.y, -q.z}; }
__device__ __forceinline__ q4 qnorm(q4 q) {
    const double n = sqrt(q.w * q.w + q.x * q.x + q.y * q.y + q.z * q.z);
    if (n < 1e-30) return q4{1, 0, 0, 0};
    return {q.w / n, q.x / n, q.y / n, q.z / n};
}
__device__ __forceinline__ q4 qmul(q4 a, q4 b) {
    return {a.w * b.w - a.x * b.x - a.y * b.y - a.z * b.z,
            a.w * b.x + a.x * b.w + a.y * b.z - a.z * b.y,
            a.w * b.y - a.x * b.z + a.y * b.w + a.z * b.x,
            a.w * b.z + a.x * b.y - a.y * b.x + a.z * b.w};
}
__device__ __forceinline__ d3 qrot(q4 q, d3 v) {
    const d3 u{q.x, q.y, q.z};
    const d3 t = cross(u, v) * 2.0;
    return (v + t * q.w) + cross(u, t);
}

// Unit quaternion of the rotation vector v (MC/include/core.hpp:51 quatExp, :42 quatAxisAngle).
__device__ __forceinline__ q4 exp_map(d3 v) {
    const double a = len(v);
    if (a < 1e-12) return qnorm(q4{1 - .125 * a * a, .5 * v.x, .5 * v.y, .5 * v.z});
    const d3 axis = unit(v * (1.0 / a));
    double s, c;
    sincos(.5 * a, &s, &c);
    return qnorm(q4{c, axis.x * s, axis.y * s, axis.z * s});
}
// J_l^{-T}(p) v, the SO(3) left-Jacobian inverse transpose applied to v
// (MC/include/core.hpp:53): v + p x v / 2 + A p x (p x v) with
// A(a) = 1/a^2 - (1 + cos a) / (2 a sin a) = 1/a^2 - cot(a/2) / (2a).
// Below a = 0.5 A is evaluated from its Taylor series (the Laurent series of cot, whose
// coefficients are Bernoulli numbers): 1/12 + a^2/720 + a^4/30240 + ...; eight terms leave
// a truncation error below 2e-18 relative there, and avoid both the sine/cosine and the
// cancellation of the closed form, which loses about log10(12/a^2) digits at small a.
// Above it the closed form is used as the reference writes it.
__device__ __forceinline__ double jl_coef(double a2) {
    double A = 3617.0 / 10670622842880000.0;
    A = fma(A, a2, 1.0 / 74724249600.0);
    A = fma(A, a2, 691.0 / 1307674368000.0);
    A = fma(A, a2, 1.0 / 47900160.0);
    A = fma(A, a2, 1.0 / 1209600.0);
    A = fma(A, a2, 1.0 / 30240.0);
    A = fma(A, a2, 1.0 / 720.0);
    return fma(A, a2, 1.0 / 12.0);
}
__device__ __forceinline__ d3 jl_inv_t(d3 p, d3 v) {
    const double a2 = len2(p);
    const d3 c1 = cross(p, v);
    const d3 c2 = cross(p, c1);
    double A;
    if (a2 < 0.25) {
        A = jl_coef(a2);
    } else {
        const double a = sqrt(a2);
        double s, c;
        sincos(a, &s, &c);
        A = 1 / (a * a) - (1 + c) / (2 * a * s);
    }
    return (v + c1 * .5) + c2 * A;
}

// ---- FP64 arithmetic for a narrow FP64 pipe -----------------------------------------------
// A sub-partition issues one FP64 warp instruction per 64 cycles when one or two of an SM's four do,
// per 76 when all do: one per 19 cycles and SM (measured: adds, multiplies and fused multiply-adds
// alike, compares too; conversions from FP64 keep the 64), while the integer and FP32 pipes idle
// beside it.  So comparisons, sign changes, halvings and conversions are done on the bit patterns,
// and square roots start from the FP32 estimate.

// v > 0 (false for NaN, as the comparison).
__device__ __forceinline__ bool positive(double v) {
    return (unsigned long long)(__double_as_longlong(v) - 1) < 0x7ff0000000000000ULL;
}
// a < b for non-negative a and b (false where a is NaN).
__device__ __forceinline__ bool less_bits(double a, double b) { return __double_as_longlong(a) < __double_as_longlong(b); }
__device__ __forceinline__ bool negative_sign(double v) { return __double2hiint(v) < 0; }
// v with the sign bit of s xored in.
__device__ __forceinline__ double xor_sign(double v, double s) {
    return __hiloint2double(__double2hiint(v) ^ (__double2hiint(s) & int(0x80000000u)), __double2loint(v));
}
// v / 2 for a normal v above the smallest exponent.
__device__ __forceinline__ double half_of(double v) {
    return __hiloint2double(__double2hiint(v) - 0x00100000, __double2loint(v));
}
// |v - 1| <= 2^-28 (2^25 numbers below one, 2^24 above it): a squared norm whose inverse square root
// is 1 - (v - 1) / 2 to FP64 precision (what is left out, 3 (v - 1)^2 / 8, is below 2^-57).
__device__ __forceinline__ bool near_one(double v) {
    constexpr long long one = 0x3ff0000000000000LL;
    return (unsigned long long)(__double_as_longlong(v) - (one - (1LL << 25))) <= (1ULL << 25) + (1ULL << 24);
}
// a in [2^-111, 2^98): its FP32 estimate below neither overflows nor loses bits.
__device__ __forceinline__ bool rsqrt_range(double a) {
    return unsigned(__double2hiint(a)) - 0x39000000u < 0x0d100000u;
}
// 1 / sqrt(a), a in rsqrt_range: the FP32 estimate y0 of the truncated a (relative error below
// 2^-21), then one third-order step y = y0 (1 + e / 2 + 3 e^2 / 8), e = 1 - a y0^2 (the binomial
// series of (1 - e)^(-1/2); what is left is of order e^3 < 2^-60).  Five FP64 instructions.
__device__ __forceinline__ double rsqrt_est(double a) {
    const float f = __int_as_float(int(__funnelshift_l(__double2loint(a), __double2hiint(a) - 0x38000000, 3)));
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
    const int b = __float_as_int(y);
    const double y0 = __hiloint2double((b >> 3) + 0x38000000, b << 29);
    const double e = fma(-(a * y0), y0, 1.0);
    return fma(y0 * e, fma(.375, e, .5), y0);
}
// sqrt(a) from y = rsqrt_est(a): a y corrected by its residual (P. Markstein, IBM J. Res. Dev.
// 34 (1990) 111), correctly rounded but for rare cases.
__device__ __forceinline__ double sqrt_from(double a, double y) {
    const double g = a * y;
    return fma(fma(-g, g, a), half_of(y), g);
}
__device__ __forceinline__ double rsqrt_any(double a) { return rsqrt_range(a) ? rsqrt_est(a) : rsqrt(a); }

// Conversions on the bit patterns; values outside FP32's normal range (zero among them, which
// stays cheap) take the instruction.
enum class RoundTo { kNearest, kDown, kUp };
template <RoundTo M>
__device__ __forceinline__ float to_float(double v) {
    const int hi = __double2hiint(v), lo = __double2loint(v);
    const unsigned mag = unsigned(hi) & 0x7fffffffu;
    if (mag - 0x38100000u >= 0x0fe00000u) {  // not in [2^-126, 2^128)
        if ((mag | unsigned(lo)) == 0) return __int_as_float(hi);
        return M == RoundTo::kNearest ? __double2float_rn(v) : M == RoundTo::kDown ? __double2float_rd(v) : __double2float_ru(v);
    }
    unsigned t = __funnelshift_l(unsigned(lo), mag - 0x38000000u, 3);
    const unsigned rest = unsigned(lo) & 0x1fffffffu;
    if (M == RoundTo::kNearest) t += rest + (t & 1u) > 0x10000000u;
    else t += rest != 0 && (hi < 0) == (M == RoundTo::kDown);
    return __int_as_float(int(t | (unsigned(hi) & 0x80000000u)));
}
__device__ __forceinline__ double to_double(float v) {
    const unsigned b = unsigned(__float_as_int(v)), mag = b & 0x7fffffffu;
    if (mag - 0x00800000u >= 0x7f000000u) return mag == 0 ? __hiloint2double(int(b), 0) : double(v);
    return __hiloint2double(int((b & 0x80000000u) | ((mag >> 3) + 0x38000000u)), int(b << 29));
}

// exp of the rotation vector v as a unit quaternion, for |v| <= 1 (v2 = |v|^2): cos(a / 2) and
// sin(a / 2) / a as polynomials in a^2 (Chebyshev interpolation on [0, 1], errors 6e-18 and
// 9e-19), so that neither a square root nor a division nor a sine is taken.
__device__ __forceinline__ q4 exp_map_small(d3 v, double v2) {
    double c = 0x1.1d8d32755f8fbp-41, s = 0x1.5fac6e0083f22p-46;
    c = fma(c, v2, -0x1.27e40964b47d4p-32); s = fma(s, v2, -0x1.ae63543245d1fp-37);
    c = fma(c, v2, 0x1.a01a00fb1bc6fp-24); s = fma(s, v2, 0x1.71de39fd64b1fp-28);
    c = fma(c, v2, -0x1.6c16c16bdd04ep-16); s = fma(s, v2, -0x1.a01a019ffb337p-20);
    c = fma(c, v2, 0x1.5555555555421p-9); s = fma(s, v2, 0x1.11111111110bfp-12);
    c = fma(c, v2, -0x1.fffffffffffffp-4); s = fma(s, v2, -0x1.5555555555555p-6);
    c = fma(c, v2, 0x1p+0); s = fma(s, v2, 0x1p-1);
    return {c, v.x * s, v.y * s, v.z * s};
}
// Products with explicit fused multiply-adds, for units compiled without contraction: the
// compiler then cannot fuse the same formula differently in two variants of a kernel, whose
// results must agree bit for bit.
__device__ __forceinline__ double fdot(d3 a, d3 b) { return fma(a.z, b.z, fma(a.y, b.y, a.x * b.x)); }
__device__ __forceinline__ d3 fcross(d3 a, d3 b) {
    return {fma(a.y, b.z, -(a.z * b.y)), fma(a.z, b.x, -(a.x * b.z)), fma(a.x, b.y, -(a.y * b.x))};
}
__device__ __forceinline__ d3 fmadd(d3 a, double s, d3 c) { return {fma(a.x, s, c.x), fma(a.y, s, c.y), fma(a.z, s, c.z)}; }
__device__ __forceinline__ q4 fqmul(q4 a, q4 b) {
    return {fma(-a.z, b.z, fma(-a.y, b.y, fma(-a.x, b.x, a.w * b.w))),
            fma(-a.z, b.y, fma(a.y, b.z, fma(a.x, b.w, a.w * b.x))),
            fma(a.z, b.x, fma(a.y, b.w, fma(-a.x, b.z, a.w * b.y))),
            fma(a.z, b.w, fma(-a.y, b.x, fma(a.x, b.y, a.w * b.z)))};
}
// Unit quaternion of q: by one step when |q| differs from one by little (rounding, usually; near_one),
// else qnorm.
__device__ __forceinline__ q4 qnorm_near(q4 q) {
    const double n2 = fma(q.z, q.z, fma(q.y, q.y, fma(q.x, q.x, q.w * q.w)));
    if (!near_one(n2)) return qnorm(q);
    const double r = fma(-.5, n2, 1.5);
    return {q.w * r, q.x * r, q.y * r, q.z * r};
}

struct m3 { d3 r0, r1, r2; };
__device__ __forceinline__ d3 fmrot(const m3& m, d3 v) { return d3{fdot(m.r0, v), fdot(m.r1, v), fdot(m.r2, v)}; }

// ---- vectors in fixed point ----------------------------------------------------------------
// An FP64 instruction occupies a sub-partition for 76 cycles, a 32 x 32 -> 64-bit multiply-add for a
// few: sums of products of numbers of a few units (rotation matrices, unit quaternions and vectors,
// rotation vectors; sums up to 32, numbers below 8) are cheaper on the integer pipe, which stands
// idle beside FP64.
// A number is (h 2^30 + l) 2^-58, |l| <= 2^29: products of two upper halves, and of an upper and a
// lower one, sum up in 64 bits each; the lower halves' products, below 2^-58, are left out.  A sum
// of three products is off by at most 2^-56 = 1.4e-17 (FP64 additions near one: 1.1e-16 each).
// "Units" are 64-bit integers of 2^-58.
// A number far below one has few bits above 2^-58, where FP64 keeps 53 of them whatever its size.  So
// vectors of free magnitude (a rotation's vector part and its matrix less the identity, deviations
// of directors from chords, rotation vectors, strains) have an exponent e for their components
// together: units times 2^e, the largest component in [1/4, 1/2) where e was made for the vector.
// Sums align their terms to the larger exponent, so that a result is off by 2^-55 of its largest
// term, where FP64's rounding is 2^-53 of it.  With e = 0 throughout the moment of two rotations of
// 1e-3 was off by 6e-15 of itself, of 1e-6 by 6e-12; with exponents 1e-16 (FP64: 2e-16).
struct fx { int h, l; };
struct u3 { long long x, y, z; };  // units
struct fx3 { fx x, y, z; };
struct fx4 { fx w, x, y, z; };
constexpr long long kFxOne = 1LL << 58;
__device__ __forceinline__ fx fx_of(long long n) {
    const int h = int((n + (1 << 29)) >> 30);
    return fx{h, int(unsigned(n) - (unsigned(h) << 30))};
}
__device__ __forceinline__ fx operator-(fx a) { return fx{-a.h, -a.l}; }
// m 2^-s or m 2^s of a 53-bit mantissa; 0 from 2^-63 on.
__device__ __forceinline__ unsigned long long shift_mantissa(unsigned long long m, int s) {
    return s >= 0 ? m << min(s, 11) : m >> min(-s, 63);
}
// v in units of 2^(scale - 1075) ... for a double's mantissa m 2^(e - 1075): m 2^(e - scale).
__device__ __forceinline__ unsigned long long fixed_magnitude(double v, int scale) {
    const unsigned hi = unsigned(__double2hiint(v));
    const unsigned long long m = (unsigned long long)(hi & 0xfffffu | 0x100000u) << 32 | unsigned(__double2loint(v));
    return shift_mantissa(m, int(hi >> 20 & 0x7ffu) - scale);
}
// v (|v| < 8 2^e) in units times 2^e, rounded toward zero; some integer when v is larger or not finite.
__device__ __forceinline__ long long fx_units(double v, int e = 0) {
    const long long n = (long long)fixed_magnitude(v, 1017 + e);
    return __double2hiint(v) < 0 ? -n : n;
}
// The exponent of a vector: its largest component is in [1/4, 1/2) 2^e; kFxLeast for a smaller one
// (or zero), above kFxMost for one that is larger or not finite.
constexpr int kFxLeast = -700, kFxMost = 700;
__device__ __forceinline__ int fx_exponent(d3 v) {
    const auto exponent = [](double a) { return int(unsigned(__double2hiint(a)) >> 20 & 0x7ffu); };
    return max(max(exponent(v.x), max(exponent(v.y), exponent(v.z))) - 1021, kFxLeast);
}
// n 2^e2, rounded to nearest; 2^-900 < the magnitude < 2^900 or zero.
__device__ __forceinline__ double fx_double(long long n, int e2 = -58) {
    const unsigned long long a = n < 0 ? 0ULL - (unsigned long long)n : (unsigned long long)n;
    const int z = __clzll((long long)(a | 1));
    const unsigned long long m = a << z;
    unsigned long long b = ((unsigned long long)(1023 + 62 - z + e2) << 52) + (m >> 11) + (m >> 10 & 1);
    if (n == 0) b = 0;
    return __longlong_as_double((long long)(n < 0 ? b | 0x8000000000000000ULL : b));
}
__device__ __forceinline__ double fx_double(fx a, int e2 = -58) { return fx_double((long long)a.h * (1 << 30) + a.l, e2); }
__device__ __forceinline__ d3 fx_double(u3 n, int e2 = -58) { return d3{fx_double(n.x, e2), fx_double(n.y, e2), fx_double(n.z, e2)}; }
__device__ __forceinline__ u3 fx_units(d3 v, int e = 0) { return u3{fx_units(v.x, e), fx_units(v.y, e), fx_units(v.z, e)}; }
// n 2^-s, rounded down; s >= 0.
__device__ __forceinline__ long long fx_shr(long long n, int s) { return n >> min(s, 63); }
__device__ __forceinline__ u3 fx_shr(u3 n, int s) { return u3{fx_shr(n.x, s), fx_shr(n.y, s), fx_shr(n.z, s)}; }
__device__ __forceinline__ long long fx_hh(fx a, fx b) { return (long long)a.h * b.h; }
__device__ __forceinline__ long long fx_hl(fx a, fx b) { return (long long)a.h * b.l + (long long)a.l * b.h; }
__device__ __forceinline__ long long fx_sum(long long hh, long long hl) { return hh * 4 + ((hl + (1 << 27)) >> 28); }
__device__ __forceinline__ long long fx_dot(const fx3& a, const fx3& b) {
    return fx_sum(fx_hh(a.x, b.x) + fx_hh(a.y, b.y) + fx_hh(a.z, b.z), fx_hl(a.x, b.x) + fx_hl(a.y, b.y) + fx_hl(a.z, b.z));
}
__device__ __forceinline__ long long fx_dot(const fx4& a, const fx4& b) {
    return fx_sum(fx_hh(a.w, b.w) + fx_hh(a.x, b.x) + fx_hh(a.y, b.y) + fx_hh(a.z, b.z),
                  fx_hl(a.w, b.w) + fx_hl(a.x, b.x) + fx_hl(a.y, b.y) + fx_hl(a.z, b.z));
}
__device__ __forceinline__ fx3 fx_of(u3 n) { return fx3{fx_of(n.x), fx_of(n.y), fx_of(n.z)}; }
__device__ __forceinline__ long long fx_mul(fx a, fx b) { return fx_sum(fx_hh(a, b), fx_hl(a, b)); }
__device__ __forceinline__ u3 fx_cross(const fx3& a, const fx3& b) {
    const auto minor = [](fx p, fx q, fx r, fx s) { return fx_sum(fx_hh(p, q) - fx_hh(r, s), fx_hl(p, q) - fx_hl(r, s)); };
    return u3{minor(a.y, b.z, a.z, b.y), minor(a.z, b.x, a.x, b.z), minor(a.x, b.y, a.y, b.x)};
}
// 2 (a b + c d)
__device__ __forceinline__ long long fx_twice(fx a, fx b, fx c, fx d) {
    return (fx_hh(a, b) + fx_hh(c, d)) * 8 + ((fx_hl(a, b) + fx_hl(c, d) + (1 << 26)) >> 27);
}
// n scaled by 1 - d / 2, d in units (the square of a length that is one but for rounding, less one).
__device__ __forceinline__ long long fx_renorm(long long n, int d) { return n - (((n >> 30) * d) >> 29); }

// A record of four numbers is stored as four doubles' bits.
__device__ __forceinline__ double fx_bits(fx a) { return __hiloint2double(a.h, a.l); }
__device__ __forceinline__ fx fx_load(double v) { return fx{__double2hiint(v), __double2loint(v)}; }

// A node's rotation in fixed point: the unit quaternion, its vector part with an exponent e <= 0, and
// the matrix less the identity (2 (w [v] + [v]^2), of the vector part's size) with the same.  A
// quaternion that is not finite has w.h = kFxInvalid.
struct FxRot {
    fx3 r0, r1, r2;  // rows of R - I, times 2^e
    int e;
};
// The matrix rows with e beside the first, and the quaternion, as the node's four records; q
// normalized to rounding already, here to 2^-56.
__device__ __forceinline__ void store_rotation(q4 q, double4_32a* __restrict__ rec) {
    const d3 qv{q.x, q.y, q.z};
    const int e = min(fx_exponent(qv), 0);
    const long long uw = fx_units(q.w);
    u3 uv = fx_units(qv, e);
    fx w = fx_of(uw);
    fx3 v = fx_of(uv);  // times 2^e
    const int d = int(fx_mul(w, w) + fx_shr(fx_dot(v, v), -2 * e) - kFxOne);
    w = fx_of(fx_renorm(uw, d));
    uv = u3{fx_renorm(uv.x, d), fx_renorm(uv.y, d), fx_renorm(uv.z, d)};
    v = fx_of(uv);
    const fx3 a = fx_of(fx_shr(uv, -e));  // the vector part itself
    const auto entry = [](long long n) { return fx_bits(fx_of(n)); };
    rec[0] = make_double4_32a(entry(-fx_twice(a.y, v.y, a.z, v.z)), entry(fx_twice(a.x, v.y, -w, v.z)),
                              entry(fx_twice(a.x, v.z, w, v.y)), fx_bits(fx{e, 0}));
    rec[1] = make_double4_32a(entry(fx_twice(a.x, v.y, w, v.z)), entry(-fx_twice(a.x, v.x, a.z, v.z)),
                              entry(fx_twice(a.y, v.z, -w, v.x)), 0.0);
    rec[2] = make_double4_32a(entry(fx_twice(a.x, v.z, -w, v.y)), entry(fx_twice(a.y, v.z, w, v.x)),
                              entry(-fx_twice(a.x, v.x, a.y, v.y)), 0.0);
    const bool ok = isfinite(q.w) && isfinite(q.x) && isfinite(q.y) && isfinite(q.z);
    if (!ok) w.h = kFxInvalid;
    rec[3] = make_double4_32a(fx_bits(w), fx_bits(v.x), fx_bits(v.y), fx_bits(v.z));
}
__device__ __forceinline__ fx3 load_fx3(const double4_32a* rec) {
    const double4_32a v = *rec;
    return fx3{fx_load(v.x), fx_load(v.y), fx_load(v.z)};
}
__device__ __forceinline__ fx4 load_fx4(const double4_32a* rec) {
    const double4_32a v = *rec;
    return fx4{fx_load(v.x), fx_load(v.y), fx_load(v.z), fx_load(v.w)};
}
__device__ __forceinline__ FxRot load_rotation(const double4_32a* rec) {
    const double4_32a v = *rec;
    return FxRot{fx3{fx_load(v.x), fx_load(v.y), fx_load(v.z)}, load_fx3(rec + 1), load_fx3(rec + 2), fx_load(v.w).h};
}
__device__ __forceinline__ m3 fx_matrix(const FxRot& r) {
    const auto row = [&](const fx3& v) { return d3{fx_double(v.x, r.e - 58), fx_double(v.y, r.e - 58), fx_double(v.z, r.e - 58)}; };
    m3 m{row(r.r0), row(r.r1), row(r.r2)};
    m.r0.x += 1;
    m.r1.y += 1;
    m.r2.z += 1;
    return m;
}
// Any vector as fixed point times 2^(e - 1022): its components to one exponent, 58 bits below the
// largest; false when that is tiny (zero, usually) or huge.
__device__ __forceinline__ bool block_units(d3 v, u3& n, int& e) {
    const auto exponent = [](double a) { return int(unsigned(__double2hiint(a)) >> 20 & 0x7ffu); };
    e = max(exponent(v.x), max(exponent(v.y), exponent(v.z)));
    // the largest component in [1/2, 1): its exponent 1022
    const auto units = [e](double a) {
        const long long m = (long long)fixed_magnitude(a, e - 5);
        return __double2hiint(a) < 0 ? -m : m;
    };
    n = u3{units(v.x), units(v.y), units(v.z)};
    return unsigned(e - 300) <= 1400u;
}
// R v, v in units times 2^(e - 1022): v and (R - I) v.
__device__ __forceinline__ d3 fx_rotate(const FxRot& r, u3 v, int e) {
    const fx3 f = fx_of(v);
    const u3 n{v.x + fx_shr(fx_dot(r.r0, f), -r.e), v.y + fx_shr(fx_dot(r.r1, f), -r.e), v.z + fx_shr(fx_dot(r.r2, f), -r.e)};
    return fx_double(n, e - 1022 - 58);
}

// ---- deterministic reductions ------------------------------------------------------------
// Fixed shuffle tree inside a warp, fixed order across warps: the same inputs in the same
// threads always give the same bits.  The warp results are complete in lane 0 only; at
// each level only the lanes whose sums lane 0 still needs add (the FP64 pipe is narrow).
__device__ __forceinline__ double warp_sum(double v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_down_sync(0xffffffffu, v, o);
        if (lane < o) v += y;
    }
    return v;
}
// Sums of four values over the warp with six FP64 additions instead of twenty: at the first two
// steps the lanes pass half of their values on and keep the other half.  Lane 0 holds the sum of
// a, lane 8 of b, lane 16 of c, lane 24 of d (as do the seven lanes after each).
__device__ __forceinline__ double warp_sum4(double a, double b, double c, double d) {
    const int lane = threadIdx.x & 31;
    const bool up = lane & 16, mid = lane & 8;
    const double k0 = (up ? c : a) + __shfl_xor_sync(0xffffffffu, up ? a : c, 16);
    const double k1 = (up ? d : b) + __shfl_xor_sync(0xffffffffu, up ? b : d, 16);
    double v = (mid ? k1 : k0) + __shfl_xor_sync(0xffffffffu, mid ? k0 : k1, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}
// Sums of two values: lane 0 holds the sum of a, lane 16 of b.
__device__ __forceinline__ double warp_sum2(double a, double b) {
    const bool up = threadIdx.x & 16;
    double v = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_down_sync(0xffffffffu, v, o);
        if (lane < o) v = fmax(v, y);
    }
    return v;
}

// Sums NV values per thread over the block; thread 0 receives the totals.  `smem` needs
// NV * (blockDim.x / 32) doubles.  blockDim.x must be a multiple of 32.
template <int NV>
__device__ __forceinline__ void block_sum(double (&v)[NV], double* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) v[k] = warp_sum(v[k]);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) smem[k * nw + warp] = v[k];
    __syncthreads();
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) {
            double s = 0;
            for (int w = 0; w < nw; w++) s += smem[k * nw + w];
            v[k] = s;
        }
    __syncthreads();
}

// Sums NV values per thread over the block into thread 0 with few FP64 warp instructions
// (GB300's FP64 pipe is narrow): the values go through shared memory, warp w reduces values
// w, w + 8, ...: lane l adds entries l, l + 32, ... in order, then the warp's shuffle tree.
// `smem` needs NV * blockDim.x doubles.  blockDim.x must be a multiple of 32.
template <int NV>
__device__ __forceinline__ void block_sum_t(double (&v)[NV], double* smem) {
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++) smem[k * nt + tid] = v[k];
    __syncthreads();
    for (int k = warp; k < NV; k += nw) {
        const double* a = smem + k * nt;
        double s = a[lane];
        for (int j = lane + 32; j < nt; j += 32) s += a[j];
        s = warp_sum(s);
        __syncwarp();
        if (lane == 0) smem[k * nt] = s;
    }
    __syncthreads();
    if (tid == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] = smem[k * nt];
    __syncthreads();
}

__device__ __forceinline__ double block_max(double v, double* smem) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    v = warp_max(v);
    if (lane == 0) smem[warp] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double m = smem[0];
        for (int w = 1; w < nw; w++) m = fmax(m, smem[w]);
        v = m;
    }
    __syncthreads();
    return v;
}

// ---- maxima on the integer pipe -------------------------------------------------------------
// Floats and doubles as integers of the same order; NaN counts as the lowest value, as fmax
// skips it.
__device__ __forceinline__ int order_key(float v) {
    const int b = __float_as_int(v);
    return v == v ? b ^ ((b >> 31) & 0x7fffffff) : int(0x80000000u);
}
__device__ __forceinline__ float order_value(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }
__device__ __forceinline__ long long order_key(double v) {
    const long long b = __double_as_longlong(v);
    const bool nan = (unsigned long long)(b & 0x7fffffffffffffffLL) > 0x7ff0000000000000ULL;
    return nan ? (long long)0x8000000000000000ULL : b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
__device__ __forceinline__ double order_value(long long k) {
    return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL));
}
__device__ __forceinline__ int warp_max_key(int k) { return __reduce_max_sync(0xffffffffu, k); }
__device__ __forceinline__ long long warp_max_key(long long k) {
    const int hi = __reduce_max_sync(0xffffffffu, int(k >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, int(k >> 32) == hi ? unsigned(k) : 0u);
    return ((long long)hi << 32) | lo;
}

// ---- node state: bounds and block partials, shared by the FP64 and the mixed form ------------
// Single-precision bounds of a node's position in the contact grid's frame (the instance's
// offset added with outward rounding), and the extrema of the bounding box: x and z from the
// outward-rounded bounds (they contain the FP64 positions), y exact (the permanent set reads it).
struct StateBounds {
    int f[4] = {int(0x80000000u), int(0x80000000u), int(0x80000000u), int(0x80000000u)};  // -min x, -min z, max x, max z
    long long y[2] = {(long long)0x8000000000000000ULL, (long long)0x8000000000000000ULL};  // -min y, max y
    __device__ __forceinline__ void take(double xx, double xy, double xz, float2 o, float4& xf_lo, float4& xf_hi) {
        const float4 lo = make_float4(__fadd_rd(to_float<RoundTo::kDown>(xx), o.x), to_float<RoundTo::kDown>(xy),
                                      __fadd_rd(to_float<RoundTo::kDown>(xz), o.y), 0.f);
        const float4 hi = make_float4(__fadd_ru(to_float<RoundTo::kUp>(xx), o.x), to_float<RoundTo::kUp>(xy),
                                      __fadd_ru(to_float<RoundTo::kUp>(xz), o.y), 0.f);
        xf_lo = lo;
        xf_hi = hi;
        f[0] = order_key(-lo.x);
        f[1] = order_key(-lo.z);
        f[2] = order_key(hi.x);
        f[3] = order_key(hi.z);
        y[0] = order_key(-xy);
        y[1] = order_key(xy);
    }
};
// Whether a node may have moved farther than `skin` from its position at the list's build: the
// displacement bounded from its FP32 interval [l, h] and the stored lower end r of its interval at
// the build (one FP32 ulp wide at most), all rounded upward.  A list built with boxes grown by
// `skin` holds every pair whose boxes overlap at any state where no node has moved farther than
// skin (Euclidean, so no farther on any axis): each current box lies inside the build's.
__device__ __forceinline__ bool moved_beyond(float skin, float4 l, float4 h, float4 r) {
    const float ulp = 1.2e-7f * fmaxf(fmaxf(fabsf(r.x), fabsf(r.y)), fabsf(r.z)) + 1e-30f;
    const float dx = __fadd_ru(fmaxf(__fsub_ru(h.x, r.x), __fsub_ru(r.x, l.x)), ulp);
    const float dy = __fadd_ru(fmaxf(__fsub_ru(h.y, r.y), __fsub_ru(r.y, l.y)), ulp);
    const float dz = __fadd_ru(fmaxf(__fsub_ru(h.z, r.z), __fsub_ru(r.z, l.z)), ulp);
    const float d2 = __fadd_ru(__fadd_ru(__fmul_ru(dx, dx), __fmul_ru(dy, dy)), __fmul_ru(dz, dz));
    return !(__fsqrt_ru(d2) <= skin);  // also when not finite
}
// All threads of the block: asks for a build when one of its nodes has moved.
__device__ __forceinline__ void ask_build(const BuildArgs& b, bool moved) {
    if (__any_sync(0xffffffffu, moved) && (threadIdx.x & 31) == 0) b.flags[1] = 1u;
}
struct StateParts {
    double sum[3][kEvalBlock / 32];
    long long y[2][kEvalBlock / 32];
    int f[4][kEvalBlock / 32];
};
// The block's nine partials (sum, -min, max of the positions) into q.
__device__ __forceinline__ void state_block_parts(const double (&acc)[3], const StateBounds& b, StateParts& sm, double* q) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const double v = warp_sum4(acc[0], acc[1], acc[2], 0.0);
    if ((lane & 7) == 0 && lane < 24) sm.sum[lane >> 3][warp] = v;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int m = warp_max_key(b.f[k]);
        if (lane == 0) sm.f[k][warp] = m;
    }
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const long long m = warp_max_key(b.y[k]);
        if (lane == 0) sm.y[k][warp] = m;
    }
    __syncthreads();
    constexpr int nw = kEvalBlock / 32;
    const int t = threadIdx.x;
    if (t < 3) {
        double s = sm.sum[t][0];
        for (int w = 1; w < nw; w++) s += sm.sum[t][w];
        q[t] = s;
    } else if (t < 5) {
        long long m = sm.y[t - 3][0];
        for (int w = 1; w < nw; w++) m = max(m, sm.y[t - 3][w]);
        q[t == 3 ? 4 : 7] = order_value(m);
    } else if (t < 9) {
        int m = sm.f[t - 5][0];
        for (int w = 1; w < nw; w++) m = max(m, sm.f[t - 5][w]);
        q[t == 5 ? 3 : t == 6 ? 5 : t == 7 ? 6 : 8] = double(order_value(m));
    }
}

// Whether this is the last of `total` blocks to arrive at a counter; then every
// block's earlier writes are visible.  All threads call it.
__device__ __forceinline__ bool last_block(unsigned* counter, unsigned total) {
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(counter, 1u) == total - 1u;
        if (last) *counter = 0;  // for the next pass
    }
    __syncthreads();
    if (last) __threadfence();
    return last;
}

inline unsigned grid_for(long long n, int block = kBlock) {
    long long g = (n + block - 1) / block;
    return unsigned(g < 1 ? 1 : g);
}

}  // namespace mcg
