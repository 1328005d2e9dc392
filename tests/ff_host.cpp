// ff.cuh compiled for the CPU: the error of FFSum, the sum of products that the solver's
// operator and dot products use, beside that of float-float additions, both against
// long double and relative to the sum of the magnitudes. Usage: ff_host TERMS KIND;
// prints rms and largest error of either, in units of 2^-48.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#define __device__
#define __forceinline__ inline
struct float2 { float x, y; };
static float2 make_float2(float x, float y) { return float2{x, y}; }
using std::fmaf;
#include "../falcon_gb300/csrc/ff.cuh"
using namespace falcon::sv;

int main(int argc, char** argv) {
    const int terms = argc > 1 ? std::atoi(argv[1]) : 7, kind = argc > 2 ? std::atoi(argv[2]) : 0;
    std::mt19937_64 rng(5);
    std::uniform_real_distribution<double> unit(0.0, 1.0);
    double rms[2] = {0, 0}, worst[2] = {0, 0};
    const int n = 200000;
    for (int q = 0; q < n; ++q) {
        FFSum sum;
        float2 chain = make_float2(0.f, 0.f);
        long double exact = 0, mag = 0;
        for (int t = 0; t < terms; ++t) {
            // kind 0: signs of a Laplacian, a smooth vector; 1: positive; 2: any sign and binade
            const double c = kind == 0 ? (t == 0 ? -6.0 : 1.0) * (1.0 + 0.01 * unit(rng)) : unit(rng) + 0.5;
            const double z = kind == 2 ? std::ldexp(2.0 * unit(rng) - 1.0, -(int)(rng() % 12)) : 1.0 + 0.01 * unit(rng);
            const float2 a = ff_from(c), b = ff_from(z);
            sum.add(a, b);
            chain = ff_add(chain, ff_mul(a, b));
            const long double p = ((long double)a.x + a.y) * ((long double)b.x + b.y);
            exact += p;
            mag += std::fabs(p);
        }
        const float2 v[2] = {sum.value(), chain};
        for (int k = 0; k < 2; ++k) {
            const double e = (double)(std::fabs((long double)v[k].x + v[k].y - exact) / mag) * 0x1p48;
            rms[k] += e * e / n;
            worst[k] = std::max(worst[k], e);
        }
    }
    std::printf("%.17g %.17g %.17g %.17g\n", std::sqrt(rms[0]), worst[0], std::sqrt(rms[1]), worst[1]);
}
