// Host-side check of imc_math64.cuh: largest errors, in units in the last
// place of the exact value, against long double (64-bit mantissa or wider).
// Prints one line per function; driven by tests/test_math64.py.
#define IMC_HD inline
#include "../../mixedprecisionimc.jl_gb300/csrc/imc_math64.cuh"

#include <cmath>
#include <cstdio>
#include <random>

using namespace imc::m64;

static double ulp(long double v) {
    int e;
    std::frexp((double)v, &e);
    return std::ldexp(1.0, e - 53);
}

int main() {
    std::mt19937_64 g(20240607);
    const uint64_t top = 1ull << 53;
    double wl = 0.0, we = 0.0, wr = 0.0, ws = 0.0;
    long bad_div = 0, bad_u = 0;
    auto log_at = [&](uint64_t k) {
        const long double ex = -logl((long double)k / 9007199254740992.0L);
        wl = std::fmax(wl, (double)(fabsl((long double)neglog_k53(k) - ex) / ulp(ex)));
    };
    // every table row's ends, the ends of the range, then uniforms, small and near-1 ones
    for (int row = 0; row < 256; ++row)
        for (int d = -2; d <= 2; ++d) log_at((((uint64_t)(256 + row) << 44) + d) & (top - 1));
    for (uint64_t k = 1; k < 64; ++k) { log_at(k); log_at(top - k); }
    for (int i = 0; i < 200000; ++i) {
        const uint64_t k = (g() >> 11) | 1ull;
        log_at(k);
        log_at((k >> (g() % 53)) | 1ull);
        log_at(top - 1 - 2 * (k >> (2 + g() % 50)));
    }
    for (int i = 0; i < 400000; ++i) {
        const double y = std::ldexp((double)((g() >> 11) | 1ull), -53 + (int)(g() % 47) - 40);
        const long double ex = expm1l(-(long double)y);
        we = std::fmax(we, (double)(fabsl((long double)expm1_neg(y) - ex) / ulp(ex)));
        const double a = std::ldexp(1.0 + (double)(g() >> 12) * 0x1p-52, (int)(g() % 60) - 30);
        double b = std::ldexp(1.0 + (double)(g() >> 12) * 0x1p-52, (int)(g() % 60) - 30);
        if (g() & 1) b = -b;
        if (div_r(a, b, 1.0 / b) != a / b) ++bad_div;
        const uint64_t k = i < 4 ? (i == 0 ? 0 : i == 1 ? top - 1 : (top >> 1) - (i == 2)) : g() >> 11;
        const double u = (double)k * 0x1p-53;
        if (u53(k) != u || one_minus_2u53(k) != 1.0 - 2.0 * u) ++bad_u;
    }
    // reciprocals, and the two kinds of addends of the 128-bit sum, in units of
    // the sum (or, of large addends, of their last kept bit)
    for (int i = 0; i < 400000; ++i) {
        const int wide = i & 1 ? 1000 : 3;
        double b = std::ldexp(1.0 + (double)(g() >> 12) * 0x1p-52, (int)(g() % (2 * wide)) - wide);
        if (g() & 1) b = -b;
        const long double ex = 1.0L / (long double)b;
        wr = std::fmax(wr, (double)(fabsl((long double)rcp64(b) - ex) / ulp(ex)));
        const int at = -300 + (int)(g() % 20), down = (int)(g() % 90);
        const double x = std::ldexp(1.0 + (double)(g() >> 12) * 0x1p-52, at - down / 2);
        const double y = -std::ldexp(1.0 + (double)(g() >> 12) * 0x1p-52, -(down - down / 2));
        const int unit = at - 92;
        Sum128 one, two;
        one.clear();
        two.clear();
        if (!one.add(x, unit) || !two.add_minus_product(x, y, unit) || !two.add(-x, unit)) ws = INFINITY;
        const long double v1 = (long double)one.hi * 0x1p64L + (long double)one.lo;
        const unsigned __int128 t = ((unsigned __int128)(uint64_t)~two.hi << 64 | (uint64_t)~two.lo) + 1;  // -two
        const long double v2 = two.hi < 0 ? -(long double)t : (long double)two.hi * 0x1p64L + (long double)two.lo;
        const long double e1 = ldexpl((long double)x, -unit);
        const long double e2 = ldexpl(-(long double)x * (long double)y - (long double)x, -unit);
        const long double scale = fmaxl(1.0L, e1 * 0x1p-60L);
        ws = std::fmax(ws, (double)(fmaxl(fabsl(v1 - e1), fabsl(v2 - e2)) / scale));
    }
    Sum128 none;
    none.clear();
    const bool refused = !none.add(INFINITY, 0) && !none.add(NAN, 0) && !none.add(1.0, -95) && none.add(0.0, 0) &&
                         none.add(0x1p-1060, -900) && none.lo == 0 && none.hi == 0;
    printf("reciprocal %.6f\nsum %.6f\nrefused %d\n", wr, ws, refused);
    printf("log %.6f\nexpm1 %.6f\ndiv %ld\nuniform %ld\n", wl, we, bad_div, bad_u);
    printf("limits %d\n", expm1_neg(0.0) == 0.0 && expm1_neg(INFINITY) == -1.0 && expm1_neg(64.0) == -1.0 &&
                             expm1_neg(1e300) == -1.0 && expm1_neg(NAN) != expm1_neg(NAN) && neglog_k53(top >> 1) == M_LN2);
    return 0;
}
