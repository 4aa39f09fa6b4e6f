// Checks of the FP32 segment's building blocks in imc_device.cuh, built and
// driven by tests/test_gpu_segment.py; prints "<name> <mismatches>" lines.
//   words    on the host: Words<5> and Words<7> against Stream
//   device   on the GPU: reciprocals and quotients against the IEEE division,
//            the FP64 functions against their host path (the reciprocal within
//            one unit in the last place of the IEEE quotient)
#include <cstdio>
#include <cstring>
#include <vector>
#include "../../mixedprecisionimc.jl_gb300/csrc/imc_device.cuh"

using namespace imc;

static uint32_t mix(uint32_t &s) { return s = s * 1664525u + 1013904223u; }

// histories of `segments` draws of one or two words, topped up where the
// transport does: below 2 before every segment (M = 5), below 4 before every
// second one (M = 7)
template <int M> static long long words_differ() {
    long long bad = 0;
    uint32_t rnd = 12345u + M;
    for (uint32_t pid = 0; pid < 400; ++pid) {
        const uint64_t seed = 0x9E3779B97F4A7C15ull * (pid + 1);
        RoundKeys rk;
        rk.set(seed);
        Stream rs;
        rs.init(seed, 3u, pid, 1u);
        Words<M> ws;
        if (pid & 1) ws.init_full(pid, rk, 3u, 1u);
        else ws.init(pid);
        for (int seg = 0; seg < 60; ++seg) {
            if (M == 5 ? ws.n < 2 : seg % 2 == 0 && ws.n < 4) ws.refill(rk, 3u, 1u);
            if (ws.n < 2) return -1;
            const bool two = (mix(rnd) >> 16) & 1;
            bad += ws.w[0] != rs.next();
            if (two) bad += ws.w[1] != rs.next();
            ws.drop(two);
        }
    }
    return bad;
}

__device__ bool same(float a, float b) { return __float_as_uint(a) == __float_as_uint(b) || (a != a && b != b); }
__device__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16; x *= 0x7FEB352Du; x ^= x >> 15; x *= 0x846CA68Bu; x ^= x >> 16;
    return x;
}

// grid of exactly 2^24 threads
__global__ void k_floats(unsigned long long *bad) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    // every mantissa, both signs, at the middle and the ends of rcp_mid's range
    const float m = __uint_as_float(0x3F800000u | (i & 0x7FFFFFu)) * (i >> 23 ? -1.0f : 1.0f);
    const float scales[3] = {1.0f, 0x1p-90f, 0x1p89f};
    for (int k = 0; k < 3; ++k)
        if (!same(rcp_mid(m * scales[k]), 1.0f / (m * scales[k]))) atomicAdd(bad + 0, 1ull);
    // every cosine
    const float mu = Rand<float>::cosine(i << 8);
    if (mu != 0.0f && !same(rcp_mid(mu), 1.0f / mu)) atomicAdd(bad + 0, 1ull);
    // every exponent, zeros, subnormals, infinities and NaN
    const float any = __uint_as_float(hash32(i));
    if (!same(rcp_any(any), 1.0f / any)) atomicAdd(bad + 1, 1ull);
    // quotients by what may be a cosine or any float
    for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t h = hash32(8u * i + k + 0x5bd1e995u);
        float a = __uint_as_float(hash32(h));
        if (k & 1) a = ldexpf(1.0f + (float)(h >> 9) * 0x1p-23f, (int)(h & 127u) - 100);
        const float b = k < 6 ? Rand<float>::cosine(hash32(h + 1u)) : __uint_as_float(hash32(h + 2u));
        if (!same(div_mid(a, b, face_rcp(b)), a / b)) atomicAdd(bad + 2, 1ull);
    }
}

// out[3 i ..]: the FP64 functions at input i of n
__global__ void k_doubles(int n, const uint64_t *in, double *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[3 * i] = m64::neglog_k53((in[i] >> 11) | 1u);
    out[3 * i + 1] = m64::expm1_neg(m64::u53(in[i] >> 11) * ldexp(1.0, (int)(in[i] & 7u) - 2));
    out[3 * i + 2] = m64::rcp64(m64::from_bits(in[i]));
}

int main(int argc, char **argv) {
    if (argc > 1 && !strcmp(argv[1], "words")) {
        printf("words5 %lld\nwords7 %lld\n", words_differ<5>(), words_differ<7>());
        return 0;
    }
    const int n = 1 << 20;
    std::vector<uint64_t> in(n);
    uint32_t s = 77u;
    for (int i = 0; i < n; ++i) {
        const uint64_t hi = mix(s), lo = mix(s);
        in[i] = (hi << 32) ^ (lo << 13) ^ (lo >> 19);
        if (i < 2048) in[i] = (uint64_t)i << 53;                // zeros, exact powers, infinities
        else if (i < 4096) in[i] = ~0ull >> (i & 63) << (i & 7);  // runs of ones
    }
    unsigned long long *bad, h_bad[3];
    uint64_t *d_in;
    double *d_out;
    std::vector<double> out(3 * (size_t)n);
    if (cudaMalloc(&bad, sizeof(h_bad)) || cudaMalloc(&d_in, 8 * (size_t)n) || cudaMalloc(&d_out, 24 * (size_t)n)) return 2;
    cudaMemset(bad, 0, sizeof(h_bad));
    cudaMemcpy(d_in, in.data(), 8 * (size_t)n, cudaMemcpyHostToDevice);
    k_floats<<<(1 << 24) / 256, 256>>>(bad);
    k_doubles<<<(n + 255) / 256, 256>>>(n, d_in, d_out);
    if (cudaDeviceSynchronize() != cudaSuccess) return 3;
    cudaMemcpy(h_bad, bad, sizeof(h_bad), cudaMemcpyDeviceToHost);
    cudaMemcpy(out.data(), d_out, 24 * (size_t)n, cudaMemcpyDeviceToHost);
    long long diff[3] = {0, 0, 0};
    for (int i = 0; i < n; ++i) {
        const double want[3] = {m64::neglog_k53((in[i] >> 11) | 1u),
                                m64::expm1_neg(m64::u53(in[i] >> 11) * ldexp(1.0, (int)(in[i] & 7u) - 2)),
                                1.0 / m64::from_bits(in[i])};
        for (int k = 0; k < 3; ++k) {
            // (the reciprocal's first guess is the hardware's: its neighbour at most)
            const double got = out[3 * (size_t)i + k];
            const long long off = (long long)m64::bits(got) - (long long)m64::bits(want[k]);
            diff[k] += !(got != got && want[k] != want[k]) && (k == 2 ? off < -1 || off > 1 : off != 0);
        }
    }
    printf("rcp_mid %llu\nrcp_any %llu\ndiv_mid %llu\nneglog_k53 %lld\nexpm1_neg %lld\nrcp64 %lld\n", h_bad[0], h_bad[1],
           h_bad[2], diff[0], diff[1], diff[2]);
    return 0;
}
