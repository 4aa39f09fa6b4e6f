// Host-side check of div_r with the reciprocals that FP64 segments hand it
// (imc_math64.cuh): quotients that are not the IEEE ones, among operands of all
// sizes and among those whose quotient lies next to a tie.  Driven by
// tests/test_div64.py.
#define IMC_HD inline
#include "../../mixedprecisionimc.jl_gb300/csrc/imc_math64.cuh"

#include <cstdio>
#include <random>

using namespace imc::m64;

int main() {
    std::mt19937_64 g(4711);
    long any = 0, near_tie = 0;
    auto wrong = [](double a, double b) { return div_r(a, b, rcp64(b)) != a / b; };
    for (int i = 0; i < 1000000; ++i) {
        const double a = std::ldexp(1.0 + (double)(g() >> 12) * 0x1p-52, (int)(g() % 60) - 30);
        // cosines, widths, constants; every other one where a reciprocal's error weighs most
        const double m = i & 1 ? 2.0 - (double)(g() >> 17) * 0x1p-52 : 1.0 + (double)(g() >> 12) * 0x1p-52;
        const double b = std::ldexp(g() & 1 ? m : -m, (int)(g() % 60) - 30);
        any += wrong(a, b);
    }
    // a = (q + half a unit) b rounded: quotients next to a tie
    for (int i = 0; i < 1000000; ++i) {
        const double b = 2.0 - (double)((g() >> 17) | 1u) * 0x1p-52;
        const double q = 1.0 + (double)(g() >> 12) * 0x1p-52;
        const long double a = ((long double)q + 0x1p-53L) * (long double)b;
        near_tie += wrong((double)a, b) + wrong(std::nextafter((double)a, 4.0), b) + wrong(std::nextafter((double)a, 0.0), b);
    }
    printf("any %ld\nnear_tie %ld\n", any, near_tie);
    return 0;
}
