// Checks of m64::pow_law (imc_math64.cuh), built and driven by
// tests/test_pow_law.py: the largest errors, in units in the last place,
// against long double (64-bit mantissa or wider), on the host or on the GPU,
// and whether the limits are pow's.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "../../mixedprecisionimc.jl_gb300/csrc/imc_device.cuh"

using namespace imc;

static const double kPowers[] = {-3.0, -2.0, -1.0, 0.0, 1.0, 2.0, 3.0};
// beyond the products' range, and where a power leaves the range of doubles
static const double kEnds[] = {0.0, -0.0, INFINITY, -INFINITY, NAN, 0x1p-301, -0x1p-301, 0x1.8p301, 0x1p-1074, -0x1.8p-1022, 0x1p1023, -0x1p350};

__global__ void k_pow(int n, const double *x, const double *p, double *o, double *want) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    o[i] = m64::pow_law(x[i], p[i]);
    want[i] = pow(x[i], p[i]);
}

int main(int argc, char **argv) {
    const int per = 100000, np = 7, ne = (int)(sizeof(kEnds) / sizeof(kEnds[0])), n = np * (per + ne);
    std::vector<double> x(n), p(n), o(n), want(n);
    std::mt19937_64 g(31337);
    for (int q = 0; q < np; ++q)
        for (int i = 0; i < per + ne; ++i) {
            const int at = q * (per + ne) + i;
            p[at] = kPowers[q];
            // temperatures, then the whole range that products serve, both signs
            const double m = 1.0 + (double)(g() >> 12) * 0x1p-52;
            const int e = i & 1 ? (int)(g() % 14) - 10 : (int)(g() % 600) - 300;
            x[at] = i < per ? std::ldexp(g() & 1 ? m : -m, e) : kEnds[i - per];
        }
    for (int i = 0; i < n; ++i) {
        o[i] = m64::pow_law(x[i], p[i]);
        want[i] = pow(x[i], p[i]);
    }
    if (argc > 1 && !strcmp(argv[1], "device")) {
        double *d[4];
        for (auto &v : d)
            if (cudaMalloc(&v, 8 * (size_t)n)) return 2;
        cudaMemcpy(d[0], x.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
        cudaMemcpy(d[1], p.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
        k_pow<<<(n + 255) / 256, 256>>>(n, d[0], d[1], d[2], d[3]);
        if (cudaDeviceSynchronize() != cudaSuccess) return 3;
        cudaMemcpy(o.data(), d[2], 8 * (size_t)n, cudaMemcpyDeviceToHost);
        cudaMemcpy(want.data(), d[3], 8 * (size_t)n, cudaMemcpyDeviceToHost);
    }
    long bad = 0;
    for (int q = 0; q < np; ++q) {
        long double worst = 0.0L;
        for (int i = 0; i < per + ne; ++i) {
            const int at = q * (per + ne) + i;
            if (i >= per) {  // p = 0 and 1 as the mathematics, the rest as pow has it
                bad += memcmp(&o[at], &want[at], 8) != 0 && !(o[at] != o[at] && want[at] != want[at]);
                continue;
            }
            const long double v = x[at];
            long double ex = 1.0L;
            for (int k = 0; k < (int)std::fabs(p[at]); ++k) ex *= v;
            if (p[at] < 0.0) ex = 1.0L / ex;
            int e;
            std::frexp((double)ex, &e);
            worst = fmaxl(worst, fabsl((long double)o[at] - ex) / ldexpl(1.0L, e - 53));
        }
        printf("%d %.4Lf\n", (int)kPowers[q], worst);
    }
    printf("limits %ld\n", bad);
    return 0;
}
