// exact64.cuh -- FP64 results of the reference's expressions in fewer FP64 instructions:
// limited slopes and fluxes, quotients by shared divisors, ghost interpolation. Only
// arithmetic: the CPU compiles it too, with stand-ins for the bit and rounding
// intrinsics (tests/exact64_host.cpp).
#pragma once
#include <cstdint>

namespace falcon {
namespace impl {

#ifdef __CUDACC__
__device__ __forceinline__ float rcp_approx(float x) {   // infinity of what FP32 flushes to 0
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
#endif

// ---- exact FP64 results with fewer instructions on the FP64 pipe -------------
// GB300 issues one FP64 warp instruction per 16 cycles and SM; compares, minima,
// sign and exponent changes of doubles run on the integer pipes instead (a
// positive double orders as its bit pattern), and a division by a value that
// many cells share goes through its reciprocal. Every function below gives the
// bits of the expression that it stands for; face_flux_h does so for speeds within
// 2^-590 .. 2^440, between which the halvings that it moves are exact (a face's
// speed is at least two sound speeds).
__device__ __forceinline__ int exp_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ unsigned long long abs_bits(double x) {
    return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ bool is_zero(double x) { return abs_bits(x) == 0ull; }
__device__ __forceinline__ double with_sign_of(unsigned long long mag, double s) {
    return __longlong_as_double((long long)(mag | ((unsigned long long)__double_as_longlong(s) & 0x8000000000000000ull)));
}
constexpr unsigned long long kExpOne = 1ull << 52;   // one step of the exponent field: a factor of 2

// A positive divisor b and y = RN(1/b). lim: 0 sends every quotient to the
// plain division (b outside 2^-300 .. 2^300).
struct Divisor {
    double b, y;
    unsigned lim;
};
__device__ __forceinline__ Divisor divisor(double b) {
    return Divisor{b, 1.0 / b, b > 0.0 && (unsigned)(exp_field(b) - 723) <= 600u ? 1000u : 0u};
}
// a / b correctly rounded in 5 FP64 instructions instead of the about 10 of a
// division (P. Markstein, IBM J. R&D 34 (1990) 111): with y = RN(1/b) and q
// within one ulp of a/b, RN(q + (a - b q) y) = RN(a/b), the residual a - b q
// being exact in an FMA. The first correction brings q = RN(a y) within an
// ulp. Quotients whose residual could underflow (exponent of a outside
// 2^-523 .. 2^477) are divided; a zero keeps its sign.
// The rare divisions are calls: inlined, the compiler runs their FP64
// instructions for every warp that holds a zero.
static __device__ __noinline__ double div_plain(double a, double b) { return a / b; }
__device__ __forceinline__ double div_by(double a, const Divisor& d) {
    double q = a * d.y;
    q = fma(fma(-d.b, q, a), d.y, q);
    q = fma(fma(-d.b, q, a), d.y, q);
    if ((unsigned)(exp_field(a) - 500) >= d.lim) {
        if (is_zero(a) && d.lim) q = a;
        else q = div_plain(a, d.b);
    }
    return q;
}

// Half the minmod slope of a cell (minmod() times 0.5) from its
// differences dl = u - ul, dr = ur - u and da = ur - ul. With a = da/2, b =
// 2 dr, c = 2 dl the selector max(0,ab) max(0,bc) 1e10 >= 1e-30 needs equal
// signs and |a| |b|^2 |c| >= 1e-40: the exponents' sum E puts that product in
// [2^E, 2^(E+4)), which decides it unless E is -136 .. -133 (1e-40 = 2^-132.88).
// The minimum and the factors of 2 are integer operations on the bit patterns.
// Magnitudes above 2^200, infinities and NaNs and the undecided products take
// the formula itself.
static __device__ __noinline__ double half_minmod_formula(double dl, double dr, double da) {
    const double a = da * 0.5, b = 2.0 * dr, c = 2.0 * dl;
    const double t = fmax(0.0, a * b) * fmax(0.0, b * c) * 1.e10 - (double)1.e-30f;
    return ((copysign(0.5, t) + 0.5) * copysign(fmin(fmin(fabs(a), fabs(b)), fabs(c)), a)) * 0.5;
}
__device__ __forceinline__ double half_minmod(double dl, double dr, double da) {
    const int ea = exp_field(da), eb = exp_field(dr), ec = exp_field(dl);
    const int E = ea + 2 * eb + ec - 4 * 1023 + 2;   // a: -1, b twice: +2, c: +1
    if (max(max(ea, eb), ec) > 1223 || (unsigned)(E + 136) <= 3u) return half_minmod_formula(dl, dr, da);
    const int ha = __double2hiint(da);
    const bool same = ((ha ^ __double2hiint(dr)) | (ha ^ __double2hiint(dl))) >= 0;
    // min(|da|/2, 2 |dr|, 2 |dl|) / 2, each factor on the exponent of |da|
    unsigned long long m = min(abs_bits(da), min(abs_bits(dr), abs_bits(dl)) + 2 * kExpOne) - 2 * kExpOne;
    if (!same || E < -132) m = 0ull;
    return with_sign_of(m, da);
}
// -phi/4 = -(0.5 (num/den - 1) + 0.25) for magnitudes an, ad (as bits) with 1/2 <
// an/ad < 1, num/den correctly rounded: with Q = RN(2^53 an/ad) the rest is exact, and
// the result -(Q - 2^52) 2^-54. Q - 2^52 = RN(2^52 N / B), B ad's significand and N what
// an/ad exceeds 1/2 by, is formed digit by digit (18, 17 and 17 bits) from FP32 estimates
// and 64-bit remainders, in place of the about 11 FP64 instructions of a division and
// the FMA: faces whose limiter acts are rare, but hardly any warp has none. (A quotient
// of two 53-bit numbers never lies halfway between two.) 442k cells, the diffusion: 768
// -> 587 us in 8^3 blocks, 970 -> 731 in 16^3.
__device__ __forceinline__ double quarter_phi(unsigned long long an, unsigned long long ad) {
    const unsigned long long top = 1ull << 52, B = (ad & (top - 1)) | top, A = (an & (top - 1)) | top;
    long long R = (long long)(((an ^ ad) >> 52 & 1ull) ? A : A << 1) - (long long)B;   // N; exponents equal or one apart
    // 2^k / B for the digits: y = 2^52 / B from its leading 24 bits
    const float y = rcp_approx(__int_as_float(0x3f800000 | (int)((B >> 29) & 0x7fffffull)));
    // round(R 2^bits / B), off by at most 1; R becomes the remainder (both products leave 64
    // bits, their difference does not: modulo 2^64)
    auto digit = [&](int bits) {
        const float t = __fmul_rn(__fmul_rn((float)(int)(R >> 22), y), __int_as_float((127 + bits - 30) << 23));
        const int k = __float_as_int(__fadd_rn(t, 12582912.f)) - 0x4B400000;
        R = (long long)(((unsigned long long)R << bits) - (unsigned long long)(long long)k * B);
        return (long long)k;
    };
    long long K = digit(18) * (1ll << 34);
    K += digit(17) * (1ll << 17);
    K += digit(17);
    K += (2 * R > (long long)B) - (2 * R < -(long long)B);
    // K as a double: 2^52 + K less 2^52; K = 0 and K = 2^52 keep the form's values
    const double d = __longlong_as_double((long long)(0x4330000000000000ull + (unsigned long long)K)) - 4503599627370496.0;
    return K == 0 ? -0.0 : __longlong_as_double((__double_as_longlong(d) - (54ll << 52)) ^ (long long)0x8000000000000000ull);
}
// The limited flux through a face (3_6/ModDiffusion.f90:40-60) from the cell values fl,
// fr, their difference den = fr - fl, the half slopes and the sum of the two
// cells' speeds. phi = max(0, 1 + 2 (num/den - 1)) is 0 unless num/den > 1/2 --
// decided by sign and magnitude, and 0/0 counts as 0 -- and 1 for num = den
// (both slopes 0), so only the faces near an extremum divide. Halving is exact,
// so -(phi/2 num) speed / 2 is formed as (-phi/4 num) speed.
static __device__ __noinline__ double flux_formula(double num, double den, double speed) {
    return -(0.5 * fmax(0.0, 1.0 + 2.0 * (num / den - 1.0)) * num) * speed * 0.5;
}
__device__ __forceinline__ double face_flux_h(double fl, double fr, double den, double hL, double hR, double speed) {
    const double num = ((fr - hR) - fl) - hL;
    const unsigned long long an = abs_bits(num), ad = abs_bits(den);
    const bool opposite = (__double2hiint(num) ^ __double2hiint(den)) < 0;
    double q;   // -phi/4
    if ((an | ad) == 0ull) {
        q = -0.0;   // 0/0
    } else if (ad - 600 * kExpOne >= 1000 * kExpOne || an >= 1600 * kExpOne) {
        // den tiny or huge, or a value that is not finite: the formula
        return flux_formula(num, den, speed);
    } else if (opposite || an <= ad - kExpOne) {
        q = -0.0;
    } else if (an == ad) {
        q = -0.25;
    } else {
        q = quarter_phi(an, ad);
    }
    return q * num * speed;
}

// ---- FP64 ghost interpolation ------------------------------------------------
// The reference's trilinear sum of a ghost entry: eight corners of three products
// each, rounded operation by operation, 31 FP64 instructions a value at one warp
// instruction in 16 cycles per SM. But nearly every entry lies on its source's grid
// lines along two or three axes, up to the rounding of the coordinates: its weights
// there are within some 1e-14 of 0 and 1 ("near" axes). Products with the small of
// two such weights matter only to the last bits of the sum, and the exact bits of
//   a (1 - D 2^-53)         a's significand less its D 2^-53, rounded, and
//   S + t, |t| < 2^-35 |S|  S's significand plus t in units of its last place, rounded
// follow from 32-bit integer and FP32 arithmetic, unless the exact result lies too
// close to the middle between two numbers to tell, or near the end of a binade; then,
// and for zeros, denormals and what is not finite, the value takes the reference's
// form. 442k cells in 8^3 blocks, 604k entries a stage: 351 -> 121 us an exchange; what bounds it
// now is half FP64 (entries near along one axis or none), half latency.
constexpr unsigned kNearD = 1u << 13;   // a factor within kNearD 2^-53 of 1 is near

// Weights of one entry. lo, hi: factors of the base and of the +1 corner along i, j, k.
struct GhostWeights {
    double lo[3], hi[3];
    unsigned D[3];       // near axes: 1 - (the large factor), in units of 2^-53
    unsigned near, up;   // bit a: axis a is near; its large factor is the +1 corner's
};
__device__ __forceinline__ GhostWeights ghost_weights(const double* w) {
    GhostWeights g;
    g.near = g.up = 0u;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        g.hi[a] = w[a];
        g.lo[a] = 1.0 - w[a];
        const unsigned long long one = 0x3ff0000000000000ull;
        const unsigned long long dl = one - (unsigned long long)__double_as_longlong(g.lo[a]);
        const unsigned long long dh = one - (unsigned long long)__double_as_longlong(g.hi[a]);
        g.D[a] = 0u;
        if (dl <= kNearD) {
            g.near |= 1u << a;
            g.D[a] = (unsigned)dl;
        } else if (dh <= kNearD) {
            g.near |= 1u << a;
            g.up |= 1u << a;
            g.D[a] = (unsigned)dh;
        }
    }
    return g;
}
// the reference's form (f: the base corner; w: the weights)
static __device__ __noinline__ double ghost_plain(const double* f, const double* w, int nip, int pl) {
    const double wi = w[0], wj = w[1], wk = w[2], ui = 1.0 - wi, uj = 1.0 - wj, uk = 1.0 - wk;
    return f[0] * ui * uj * uk + f[1] * wi * uj * uk + f[nip] * ui * wj * uk + f[pl] * ui * uj * wk +
           f[1 + nip] * wi * wj * uk + f[nip + pl] * ui * wj * wk + f[1 + pl] * wi * uj * wk + f[1 + nip + pl] * wi * wj * wk;
}
// a's significand's leading 32 bits
__device__ __forceinline__ unsigned top_bits(double a) {
    return __funnelshift_l((unsigned)__double2loint(a), (unsigned)__double2hiint(a), 11) | 0x80000000u;
}
// round(M D 2^-53) for the significand M with leading bits Mt (M may have moved by
// 2^16 since): the product of Mt and D has 32 fraction bits and is off by less than
// D + 64 of their units; false if that leaves the rounding open
__device__ __forceinline__ bool near_units(unsigned Mt, unsigned D, int& k) {
    const unsigned long long x = (unsigned long long)Mt * D + 0x80000000ull;
    k = (int)(x >> 32);
    return (unsigned)x + (D + 64u) > 2u * (D + 64u);
}
// f W in units of the last place of a number with a's exponent and sign (W: times
// 2^52), relative error 2^-22 beyond W's; 0 for an f beyond 2^-126 below it. d: f's exponent
// less a's
__device__ __forceinline__ float small_units(double f, float W, double a, int& d) {
    const int hf = __double2hiint(f), ha = __double2hiint(a);
    d = exp_field(f) - exp_field(a);
    const unsigned m = __funnelshift_l((unsigned)__double2loint(f), (unsigned)hf, 3) & 0x7fffffu;
    const unsigned bits = m | (unsigned)(d + 127) << 23 | ((unsigned)(hf ^ ha) & 0x80000000u);
    return d < -126 ? 0.f : __fmul_rn(__int_as_float((int)bits), W);
}
// round(x) for an x off by less than 2^-21 m (m >= |x|); false if that leaves it open
__device__ __forceinline__ bool round_units(float x, float m, int& k) {
    const float r = __fadd_rn(x, 12582912.f);   // ulp 1: the integer in its low bits
    k = (int)((unsigned)__float_as_int(r) - 0x4B400000u);
    return __fmaf_rn(m, 4.7683716e-7f, fabsf(__fsub_rn(x, __fsub_rn(r, 12582912.f)))) < 0.499999f;
}
// exponents in the middle of the range: no underflow in the products, and what is
// not finite lies more than 60 above
__device__ __forceinline__ bool mid_range(double a) { return (unsigned)(exp_field(a) - 100) < 1800u; }

// Entries near along all axes. Every rounding moves the large corner's significand by
// a whole number of units that does not depend on the others, as long as the binade
// does not end within 2^20 units: the three products with 1 - D 2^-53, the sum of the
// terms before the large corner (the corners below it along its `up` axes), and each
// term after it. Corners off along two or three axes are left out: added after the
// large corner they move nothing, being less than half a unit; before it (`up` set
// along j or k) they are part of the sum that is rounded, and count as its error.
struct NearEntry {
    unsigned D[3], up;
    int at, step[3];   // the large corner from the base, and from it to its neighbours
    float W[3];        // weights of these, times 2^52
};
__device__ __forceinline__ NearEntry near_entry(const GhostWeights& g, int nip, int pl) {
    NearEntry n;
    n.up = g.up;
    n.at = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int st = a == 0 ? 1 : a == 1 ? nip : pl;
        const bool up = g.up >> a & 1u;
        n.D[a] = g.D[a];
        n.at += up ? st : 0;
        n.step[a] = up ? -st : st;
        n.W[a] = (float)(up ? g.lo[a] : g.hi[a]) * 4503599627370496.f;
    }
    return n;
}
__device__ __forceinline__ double ghost_near(const double* f, const double* w, const NearEntry& n, int nip, int pl) {
    const double* fc = f + n.at;
    const double a = fc[0];
    double v[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) v[q] = fc[n.step[q]];
    const int s01 = n.step[0] + n.step[1], s2 = n.step[2];
    // the corners off along several axes: weights up to kNearD^2 2^-106 = 2^-80. With
    // exponents up to `rise` above a's their sum is below 2^(rise - 25) units of a's last place
    const int hx = max(max(__double2hiint(fc[s01]) & 0x7ff00000, __double2hiint(fc[n.step[0] + s2]) & 0x7ff00000),
                       max(__double2hiint(fc[n.step[1] + s2]) & 0x7ff00000, __double2hiint(fc[s01 + s2]) & 0x7ff00000));
    const unsigned Mt = top_bits(a);
    const int rise = (hx - (__double2hiint(a) & 0x7ff00000)) >> 20;
    bool ok = mid_range(a) & (Mt - 0x80000001u < 0x7ffffffeu) & (rise < 20);
    unsigned sum = 0u;   // (modulo 2^32: a term out of range fails a test below)
    int k;
    // (pre_m counts 2^-21 of itself as error)
    float pre = 0.f, pre_m = n.up > 1u ? __int_as_float((127 - 4 + min(max(rise, -100), 20)) << 23) : 0.f, all_m = 0.f;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        ok &= near_units(Mt, n.D[q], k);
        sum -= (unsigned)k;
        int d;
        const float y = small_units(v[q], n.W[q], a, d);
        ok &= d < 60;
        all_m += fabsf(y);
        const bool before = n.up >> q & 1u;
        pre += before ? y : 0.f;
        pre_m += before ? fabsf(y) : 0.f;
        ok &= round_units(before ? 0.f : y, fabsf(y), k);
        sum += (unsigned)k;
    }
    ok &= round_units(pre, pre_m, k) & (all_m < 131072.f);
    sum += (unsigned)k;
    return ok ? __longlong_as_double(__double_as_longlong(a) + (long long)(int)sum) : ghost_plain(f, w, nip, pl);
}

// Entries near along some axes. The main corners (all near factors large) are formed
// in FP64 along the other axes; the rest are small terms, rounded one by one.
__device__ __forceinline__ double move_units(double a, int k, bool& ok) {
    const long long r = (long long)((unsigned long long)__double_as_longlong(a) + (unsigned long long)(long long)k);
    ok &= (((int)(r >> 32) ^ __double2hiint(a)) >> 20 == 0) & (((unsigned long long)r << 12) != 0ull);   // inside the binade
    return __longlong_as_double(r);
}
__device__ __forceinline__ constexpr int ghost_order(int p) { return 0x75634210 >> (4 * p) & 7; }   // the reference's order of summation
struct MixedEntry {
    GhostWeights g;
    unsigned main;     // bit c: corner c (bit a of c: +1 along a) is a main corner
    float W[8];        // the others: product of factors, times 2^52
};
__device__ __forceinline__ MixedEntry mixed_entry(const GhostWeights& g) {
    MixedEntry n;
    n.g = g;
    n.main = 0xffu;
    float lo[3], hi[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const unsigned base = a == 0 ? 0x55u : a == 1 ? 0x33u : 0x0fu;   // corners with bit a clear
        if (g.near >> a & 1u) n.main &= g.up >> a & 1u ? ~base : base;
        lo[a] = (float)g.lo[a];
        hi[a] = (float)g.hi[a];
    }
#pragma unroll
    for (int c = 0; c < 8; ++c)
        n.W[c] = ((c & 1 ? hi[0] : lo[0]) * (c & 2 ? hi[1] : lo[1])) * (c & 4 ? hi[2] : lo[2]) * 4503599627370496.f;
    return n;
}
__device__ __forceinline__ double ghost_mixed(const double* f, const double* w, const MixedEntry& n, int nip, int pl) {
    double v[8], S = 0.0;
#pragma unroll
    for (int c = 0; c < 8; ++c) v[c] = f[(c & 1) + (c & 2 ? nip : 0) + (c & 4 ? pl : 0)];
    bool ok = true;
    auto main_term = [&](int c) {
        double x = v[c];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (n.g.near >> a & 1u) {
                int k;
                ok &= near_units(top_bits(x), n.g.D[a], k) & mid_range(x);
                x = move_units(x, -k, ok);
            } else {
                x = x * (c >> a & 1 ? n.g.hi[a] : n.g.lo[a]);
            }
        }
        ok &= mid_range(x);
        return x;
    };
    // the small terms before the first main corner are added to it when it is known
    unsigned pending = 0u;
    bool first = true;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
        const int c = ghost_order(p);
        int k, d;
        if (n.main >> c & 1u) {
            const double t = main_term(c);
            if (first) {
                S = t;
                first = false;
                if (pending) {
                    float x = 0.f, m = 0.f;
#pragma unroll
                    for (int q = 0; q < p; ++q) {
                        const int e = ghost_order(q);
                        const float y = small_units(v[e], n.W[e], S, d);
                        ok &= d < 60;
                        x += y;
                        m += fabsf(y);
                    }
                    ok &= round_units(x, 2.f * m, k);
                    S = move_units(S, k, ok);
                }
            } else {
                S = S + t;
                ok &= mid_range(S);
            }
        } else if (first) {
            pending = 1u;
        } else {
            const float y = small_units(v[c], n.W[c], S, d);
            ok &= (d < 60) & round_units(y, 2.f * fabsf(y), k);   // (W: three rounded factors)
            S = move_units(S, k, ok);
        }
    }
    return ok ? S : ghost_plain(f, w, nip, pl);
}

}  // namespace impl
}  // namespace falcon
