// exact64.cuh compiled for the CPU: every form against the expression that it stands
// for, bit by bit. Usage: exact64_host FORM COUNT SEED; prints the values that differ.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>

#define __device__
#define __forceinline__ inline
#define __noinline__
using std::max;
using std::min;
template <class To, class From> static To bits(From x) {
    To r;
    static_assert(sizeof(To) == sizeof(From), "same size");
    std::memcpy(&r, &x, sizeof r);
    return r;
}
static long long __double_as_longlong(double x) { return bits<long long>(x); }
static double __longlong_as_double(long long x) { return bits<double>(x); }
static int __double2hiint(double x) { return (int)(bits<unsigned long long>(x) >> 32); }
static int __double2loint(double x) { return (int)bits<unsigned long long>(x); }
static float __int_as_float(int x) { return bits<float>(x); }
static int __float_as_int(float x) { return bits<int>(x); }
static unsigned __funnelshift_l(unsigned lo, unsigned hi, int s) {
    return (unsigned)(((unsigned long long)hi << 32 | lo) << s >> 32);
}
static float __fadd_rn(float a, float b) { return a + b; }
static float __fsub_rn(float a, float b) { return a - b; }
static float __fmul_rn(float a, float b) { return a * b; }
static float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
namespace falcon {
namespace impl {
static int estimate_off;   // the reciprocal's error, in units of its last place
static float rcp_approx(float x) { return __int_as_float(__float_as_int(1.f / x) + estimate_off); }
}  // namespace impl
}  // namespace falcon
using std::copysign;
using std::fabs;
using std::fma;
using std::fmax;
using std::fmin;
#include "../falcon_gb300/csrc/exact64.cuh"

using namespace falcon::impl;
static std::mt19937_64 rng;
static double unit() { return (double)(rng() >> 11) * 0x1p-53; }             // [0, 1)
static double sym() { return 2.0 * unit() - 1.0; }
static double wide(int lo, int hi) { return std::ldexp(sym(), lo + (int)(rng() % (unsigned)(hi - lo))); }
static long bad;
static void same(const char* what, double a, double b, const double* v, int n) {
    if (bits<uint64_t>(a) == bits<uint64_t>(b) || (a != a && b != b)) return;
    if (bad++ < 5) {
        std::printf("%s: %a, expression %a, of", what, a, b);
        for (int q = 0; q < n; ++q) std::printf(" %a", v[q]);
        std::printf("\n");
    }
}

// three cells in a row: smooth, few values, many binades, near the selector's threshold
static void cells(double (&u)[4]) {
    const int kind = (int)(rng() % 5);
    const double base = sym();
    for (double& x : u)
        x = kind == 0 ? base + 1e-6 * sym() : kind == 1 ? (double)((int)(rng() % 3) - 1) : kind == 2 ? wide(-200, 120)
          : kind == 3 ? 0x1p-33 * wide(-2, 3) : sym();
}
static void slopes() {
    double u[4];
    cells(u);
    const double a = (u[2] - u[0]) * 0.5, b = 2.0 * (u[2] - u[1]), c = 2.0 * (u[1] - u[0]);
    const double t = fmax(0.0, a * b) * fmax(0.0, b * c) * 1.e10 - (double)1.e-30f;
    const double slope = (copysign(0.5, t) + 0.5) * copysign(fmin(fmin(fabs(a), fabs(b)), fabs(c)), a);
    same("half_minmod", half_minmod(u[1] - u[0], u[2] - u[1], u[2] - u[0]), slope * 0.5, u, 3);
}
static void fluxes() {
    double u[4];
    cells(u);
    const double hL = half_minmod(u[1] - u[0], u[2] - u[1], u[2] - u[0]);
    const double hR = half_minmod(u[2] - u[1], u[3] - u[2], u[3] - u[1]);
    const double num = ((u[2] - hR) - u[1]) - hL, den = u[2] - u[1], speed = std::ldexp(1.0 + unit(), (int)(rng() % 40) - 20);
    const double phi = fmax(0.0, 1.0 + 2.0 * (num / den - 1.0));
    estimate_off = (int)(rng() % 5) - 2;
    same("face_flux_h", face_flux_h(u[1], u[2], den, hL, hR, speed), -(0.5 * phi * num) * speed * 0.5, u, 4);
}
static void quotients() {
    const double v[2] = {wide(-700, 700), std::ldexp(1.0 + unit(), (int)(rng() % 500) - 250)};
    const double a = rng() % 64 ? v[0] : rng() % 2 ? 0.0 : -0.0;
    same("div_by", div_by(a, divisor(v[1])), a / v[1], v, 2);
}
// phi near its ends, and quotients of any two significands
static void limiters() {
    double v[2] = {1.0 + unit(), 1.0 + unit()};   // num, den with 1/2 < num/den < 1
    if (rng() % 4 == 0) v[0] = v[1] * (rng() % 2 ? 1.0 - 0x1p-52 * (double)(rng() % 9) : 0.5 + 0x1p-53 * (double)(rng() % 9));
    if (v[0] >= v[1]) v[0] *= 0.5;
    if (!(v[0] > 0.5 * v[1] && v[0] < v[1])) return;
    estimate_off = (int)(rng() % 5) - 2;
    same("quarter_phi", quarter_phi(abs_bits(v[0]), abs_bits(v[1])), -(0.5 * (v[0] / v[1] - 1.0) + 0.25), v, 2);
}

static double interpolate(const double (&v)[8], const double (&w)[3]) {
    const double wi = w[0], wj = w[1], wk = w[2], ui = 1.0 - wi, uj = 1.0 - wj, uk = 1.0 - wk;
    return v[0] * ui * uj * uk + v[1] * wi * uj * uk + v[2] * ui * wj * uk + v[4] * ui * uj * wk + v[3] * wi * wj * uk +
           v[6] * ui * wj * wk + v[5] * wi * uj * wk + v[7] * wi * wj * wk;
}
static void ghost(const double (&v)[8], const double (&w)[3]) {
    const GhostWeights g = ghost_weights(w);
    double all[11];
    std::copy(w, w + 3, all);
    std::copy(v, v + 8, all + 3);
    if (g.near == 7u) same("ghost_near", ghost_near(v, w, near_entry(g, 2, 4), 2, 4), interpolate(v, w), all, 11);
    else if (g.near) same("ghost_mixed", ghost_mixed(v, w, mixed_entry(g), 2, 4), interpolate(v, w), all, 11);
}
static void ghosts() {
    double v[8], w[3];
    for (double& x : w) {
        const int kind = (int)(rng() % 8);
        const double e = (double)(rng() % (rng() % 2 ? 60 : kNearD)) * 0x1p-53;
        x = kind < 3 ? e : kind < 6 ? 1.0 - (e > 0 ? e : 0x1p-53) : kind == 6 ? 0.0 : unit();
    }
    const int kind = (int)(rng() % 8);
    const double scale = wide(-60, 60), b0 = 1.0 + unit();
    for (double& x : v)
        x = kind == 0 ? sym() * scale : kind == 1 ? (b0 + 1e-3 * sym()) * scale : kind == 2 ? (b0 + 1e-12 * sym()) * scale
          : kind == 3 ? (double)(int)(rng() % 3) * scale : kind == 4 ? wide(-200, 200)
          : kind == 5 ? (1.0 + (double)(rng() % 7) * 0x1p-52) * scale : kind == 6 ? (2.0 - (double)(1 + rng() % 90) * 0x1p-52) * scale
          : rng() % 64 ? sym() : bits<double>((uint64_t)rng());
    ghost(v, w);
}
// all three axes near, with factors over the whole accepted range, and corners far
// above the large one: those off along several axes reach its rounding
static void far_ghosts() {
    double v[8], w[3];
    const int large = (int)(rng() % 8);
    for (int a = 0; a < 3; ++a) {
        const double e = (double)(1 + rng() % kNearD) * 0x1p-53;
        w[a] = large >> a & 1 ? 1.0 - e : e;
    }
    for (int c = 0; c < 8; ++c) v[c] = c == large ? 1.0 + unit() : wide(-3, 21);
    ghost(v, w);
}
// a sum within 2^-9 of a unit of the middle between two numbers
static void far_ghost_case() {
    const double w[3] = {0x1.ffffffffff82p-1, 0x1.fffffffffff1p-1, 0.0};
    const double v[8] = {-0x1.ffffffffffffcp+30, -0x1.aaaa34ep+6,      0x1.0000000000002p+5,  -0x1.4688ff63e2b77p+11,
                         0x1.0000000000002p+21,  -0x1.e5396d33293fep+26, 0x1.ffffffffffffdp+20, -0x1.cc5025p+34};
    ghost(v, w);
}

int main(int argc, char** argv) {
    const char* form = argc > 1 ? argv[1] : "";
    const long n = argc > 2 ? std::atol(argv[2]) : 1;
    rng.seed(argc > 3 ? (unsigned long)std::atol(argv[3]) : 1);
    for (long q = 0; q < n; ++q) {
        if (!std::strcmp(form, "slopes")) slopes();
        else if (!std::strcmp(form, "fluxes")) fluxes();
        else if (!std::strcmp(form, "quotients")) quotients();
        else if (!std::strcmp(form, "limiters")) limiters();
        else if (!std::strcmp(form, "ghosts")) ghosts();
        else if (!std::strcmp(form, "far_ghosts")) far_ghosts();
        else if (!std::strcmp(form, "far_ghost_case")) far_ghost_case();
        else return 2;
    }
    std::printf("%s: %ld of %ld differ\n", form, bad, n);
    return bad ? 1 : 0;
}
