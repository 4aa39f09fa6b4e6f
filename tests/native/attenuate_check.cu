// Checks of m64::attenuate (imc_math64.cuh), the weight that an FP64 history
// carries on, built and driven by tests/test_attenuate64.py.
//   host     the largest relative errors of the weight by ranges of y = sigma_a
//            f d, in units of 2^-53 (of the least normal number where the weight is
//            below it), against long double (64-bit mantissa or wider)
//   device   the same inputs on the GPU: results that are not the host's
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>
#include "../../mixedprecisionimc.jl_gb300/csrc/imc_device.cuh"

using namespace imc;

// name, range of y
struct Range { const char *name; double lo, hi; };
static const Range kRanges[] = {{"tiny", 1e-12, 1e-3}, {"thin", 1e-3, 0.5}, {"near_half", 0.5, 0.9}, {"near_one", 0.9, 1.1},
                                {"to_two", 1.0, 2.0}, {"cutoff", 2.0, 4.6051702}, {"deep", 4.6, 64.0}, {"far", 64.0, 700.0},
                                {"past_census", -1e-6, -1e-16}, {"negative", -4.0, -1e-6}};

__global__ void k_attenuate(int n, const double *E, const double *y, double *w, double *em1) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) w[i] = m64::attenuate(E[i], y[i], &em1[i]);
}

int main(int argc, char **argv) {
    const int per = 200000, nr = (int)(sizeof(kRanges) / sizeof(kRanges[0])), n = per * nr;
    std::vector<double> E(n), y(n), w(n), em1(n);
    std::mt19937_64 g(20250311);
    for (int i = 0; i < n; ++i) {
        const Range &r = kRanges[i / per];
        const double u = (double)(g() >> 11) * 0x1p-53;
        y[i] = i % per == 0 ? r.lo : i % per == 1 ? r.hi : r.lo + (r.hi - r.lo) * u;
        E[i] = std::ldexp(1.0 + (double)(g() >> 12) * 0x1p-52, (int)(g() % 40) - 20);
        w[i] = m64::attenuate(E[i], y[i], &em1[i]);
    }
    if (argc > 1 && !strcmp(argv[1], "device")) {
        double *d[4];
        for (auto &p : d)
            if (cudaMalloc(&p, 8 * (size_t)n)) return 2;
        cudaMemcpy(d[0], E.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
        cudaMemcpy(d[1], y.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
        k_attenuate<<<(n + 255) / 256, 256>>>(n, d[0], d[1], d[2], d[3]);
        if (cudaDeviceSynchronize() != cudaSuccess) return 3;
        std::vector<double> gw(n), ge(n);
        cudaMemcpy(gw.data(), d[2], 8 * (size_t)n, cudaMemcpyDeviceToHost);
        cudaMemcpy(ge.data(), d[3], 8 * (size_t)n, cudaMemcpyDeviceToHost);
        long differ = 0;
        // from 0 up to 64 the same integers and FP64 operations on both sides
        for (int i = 0; i < n; ++i) differ += y[i] >= 0.0 && y[i] < 64.0 && (gw[i] != w[i] || ge[i] != em1[i]);
        printf("differ %ld\n", differ);
        w = gw;
    }
    for (int r = 0; r < nr; ++r) {
        long double worst = 0.0L;
        for (int i = r * per; i < (r + 1) * per; ++i) {
            const long double ex = (long double)E[i] * expl(-(long double)y[i]);
            worst = fmaxl(worst, fabsl((long double)w[i] - ex) / fmaxl(ex, 0x1p-1022L) * 0x1p53L);
        }
        printf("%s %.4Lf\n", kRanges[r].name, worst);
    }
    return 0;
}
