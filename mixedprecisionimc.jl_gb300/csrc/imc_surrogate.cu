// imc_surrogate.cu -- training data, training and test entry points of the
// learned thick-cell surrogate (model in imc_surrogate.cuh).
//
//   k_surr_datagen  the analog in-cell walk (the physics of Transport.MC inside
//                   one cell, src/imc_transport.jl:72-193, in mean free paths)
//                   from random walk states; its outcomes are the training
//                   targets and, in the tests, the yardstick of the sampled ones
//   k_surr_grad     forward + backward of a 64-sample slice in FP32: the loss
//                   (cross entropy of the outcome + pinball losses of the
//                   outcome's quantile heads) and per-block weight gradients
//   k_surr_adam     sums the per-block gradients in block order (deterministic)
//                   and takes the Adam step on FP32 master weights
//   k_surr_reduce   the sums alone
//   k_surr_forward  the transport kernel's tensor-core forward pass on given
//                   inputs (for the tests)
//   k_surr_sample   inverse-transform sampling of the network's outputs, as
//                   the transport kernel samples them (for the tests)
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "imc.h"  // include/imc.h (on the -I path)
#include "imc_device.cuh"
#include "imc_internal.h"
#include "imc_surrogate.cuh"

using namespace imc;
using namespace imc::surr;

namespace {

constexpr uint32_t kStageSurrData = 3;   // Philox stage tag of training walks
constexpr uint32_t kStageSurrTest = 4;   // stage tag of test sampling
constexpr int kWalkCapFactor = 8;        // flight cap: 8 * lmax + 64

// ----------------------------------------------------------- in-cell walk
// Analog walk from (d_n, d_f, mu', lmax), all in mean free paths, near face at
// 0, far face at d_n + d_f, one flight at a time.  Ends with the outcome and
// its two targets: for an exit ln(path / lmax) and |mu|, for truncation the
// displacement toward the far face / sqrt(lmax) and the final mu'.
struct Walk {
    float d_n, W, mu, lmax, pos, path;
    float den, rden;  // |mu| as the divisor of the face distance, and 1 / den where that serves (inf otherwise)
    int left;         // flights left before the cap
    Words<5> ws;
    __device__ __forceinline__ void aim(float m) {
        mu = m;
        den = m > 0.0f ? m : -m;
        rden = den >= 0x1p-40f && den <= 1.0f ? rcp_mid(den) : INFINITY;
    }
    __device__ __forceinline__ void start(float dn, float df, float m, float L, const Stream &rs) {
        d_n = dn; W = dn + df; lmax = L; pos = dn; path = 0.0f;
        left = kWalkCapFactor * (int)L + 64;
        aim(m);
        // the rest of the stream's block, then its next ones
        ws.pid = rs.pid; ws.block = rs.block; ws.n = 4 - rs.idx;
        ws.w[0] = rs.idx == 0 ? rs.buf[0] : rs.idx == 1 ? rs.buf[1] : rs.idx == 2 ? rs.buf[2] : rs.buf[3];
        ws.w[1] = rs.idx == 0 ? rs.buf[1] : rs.idx == 1 ? rs.buf[2] : rs.buf[3];
        ws.w[2] = rs.idx == 0 ? rs.buf[2] : rs.buf[3];
        ws.w[3] = rs.buf[3];
    }
    __device__ __forceinline__ int truncated(float *y0, float *y1) const {
        *y0 = (pos - d_n) / sqrtf(lmax);
        *y1 = mu;
        return kTrunc;
    }
    // one flight; the outcome, or -1 while the walk goes on
    __device__ __forceinline__ int flight(const SeedKeys &key, float *y0, float *y1) {
        if (left <= 0) return truncated(y0, y1);
        if (ws.n < 2) ws.refill(key, 0u, kStageSurrData);
        const float s = -logf((float)((ws.w[0] >> 8) | 1u) * 0x1p-24f);
        // the distance to the face ahead, num / den: the quotient's residual
        // corrects num * rden to the IEEE quotient (Markstein, IBM J. Res.
        // Dev. 34, 1990) while nothing leaves binary32's middle range
        const float num = mu > 0.0f ? W - pos : pos;
        const float q = num * rden;
        float dface = fmaf(fmaf(-q, den, num), rden, q);
        if (!(fabsf(q) >= 0x1p-60f && fabsf(q) <= 0x1p60f)) dface = num / den;
        const float rem = lmax - path;
        if (rem <= s && rem <= dface) {
            pos += mu * rem;
            return truncated(y0, y1);
        }
        if (dface <= s) {
            path += dface;
            *y0 = logf(fmaxf(path, 1e-30f) / lmax);
            *y1 = fabsf(mu);
            return mu > 0.0f ? kFar : kNear;
        }
        pos += mu * s;
        path += s;
        float m = Rand<float>::cosine(ws.w[1]);
        for (int r = 1; r < 64 && m == 0.0f; ++r) {
            ws.drop(false);
            if (ws.n < 2) ws.refill(key, 0u, kStageSurrData);
            m = Rand<float>::cosine(ws.w[1]);
        }
        aim(m == 0.0f ? 1.0f : m);
        ws.drop(true);
        --left;
        return -1;
    }
};

// Random walk states covering the states the transport kernel asks about
// (lmax >= 32, cells >= 8 mean free paths, expected collisions
// min(lmax, 1.5 d_n d_f) >= 64) with a margin: lmax log-uniform on
// [40, 1.2e4]; cell width W log-uniform on [12, 2.5 lmax] for half of the
// states and on [12, min(2.5 lmax, 20 sqrt(lmax))] for the other half, so that
// cells thin enough for walks to cross them (diffusion length sqrt(lmax)) are
// well represented; the start uniform in the nearer half of the cell, redrawn
// (at most 16 times, then the cell centre) until 1.5 d_n d_f >= 48; mu'
// uniform on [-1, 1].
__device__ void draw_state(Stream &rs, float *d_n, float *d_f, float *mu, float *lmax) {
    const float lo = 1.6020600f, hi = 4.0791812f;  // log10 40, log10 1.2e4
    const float L = exp10f(lo + (hi - lo) * Rand<float>::u(rs));
    const float top = Rand<float>::u(rs) < 0.5f ? fminf(2.5f * L, 20.0f * sqrtf(L)) : 2.5f * L;
    const float lw0 = 1.0791812f, lw1 = log10f(fmaxf(top, 12.0f));  // log10 12
    const float W = exp10f(lw0 + (lw1 - lw0) * Rand<float>::u(rs));
    float dn = 0.5f * W;
    for (int r = 0; r < 16; ++r) {
        const float v = 0.5f * W * Rand<float>::u(rs);
        if (1.5f * v * (W - v) >= 48.0f) { dn = v; break; }
    }
    float m = 0.0f;
    for (int r = 0; r < 64 && m == 0.0f; ++r) m = 1.0f - 2.0f * Rand<float>::u(rs);
    if (m == 0.0f) m = 1.0f;
    *d_n = dn; *d_f = W - dn; *mu = m; *lmax = L;
}

// The walks, a lane each: a lane whose walk has ended takes the next sample from
// the counter, once four of a warp's lanes wait (walks are 1 to 1e4 flights
// long; a thread per sample left most lanes waiting for the longest walk of
// their warp: 2^18 walks 12.3 ms).  Every sample has its own stream, so who walks it
// changes nothing.
constexpr int kDatagenThreads = 256;
// samples a lane walks on average until the grid has its four blocks an SM (2^18
// walks: 171 blocks): fewer leave the lanes idle behind the longest walks (3: 9.2
// ms for 2^18 walks), more leave SMs short of warps (12: 11.2 ms); 8.4 ms
constexpr int kDatagenPerLane = 6;
__global__ void __launch_bounds__(kDatagenThreads, 4) k_surr_datagen(unsigned long long seed, long long n,
                                                                     const float *state_in, float *x, int *cls,
                                                                     float *tgt, unsigned long long *counter) {
    const int lane = threadIdx.x & 31;
    const SeedKeys key(seed);
    Walk w{};
    long long i = -1;   // the sample under way (-1: none)
    bool more = true;   // warp-uniform: the counter has samples left
    while (true) {
        const unsigned idle = __ballot_sync(0xFFFFFFFFu, i < 0);
        if (more && (__popc(idle) >= 4)) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(counter, (unsigned long long)__popc(idle));
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            more = (long long)base + __popc(idle) < n;
            const long long mine = (long long)base + __popc(idle & ((1u << lane) - 1u));
            if (i < 0 && mine < n) {
                i = mine;
                Stream rs;
                rs.init(seed, 0u, (uint32_t)i, kStageSurrData);
                float dn, df, mu, L;
                if (state_in) {
                    dn = state_in[4 * i]; df = state_in[4 * i + 1]; mu = state_in[4 * i + 2]; L = state_in[4 * i + 3];
                } else {
                    draw_state(rs, &dn, &df, &mu, &L);
                }
                float f[kIn];
                features(dn, df, mu, L, f);
                for (int k = 0; k < kIn; ++k) x[kIn * i + k] = f[k];
                w.start(dn, df, mu, L, rs);
            }
        } else if (idle == 0xFFFFFFFFu) {
            return;
        }
        if (i >= 0) {
            float y0, y1;
            const int c = w.flight(key, &y0, &y1);
            if (c >= 0) {
                cls[i] = c;
                tgt[2 * i] = y0;
                tgt[2 * i + 1] = y1;
                i = -1;
            }
        }
    }
}

// ------------------------------------------------------------- training
constexpr int kSlice = 64;        // samples per block
constexpr int kTileThreads = 256;  // the layers' products
constexpr int kTrainThreads = kTileThreads + kSlice;
constexpr int kQMax = kQL + kQM;  // knots of an outcome's two heads, at most

// shared-memory layout of k_surr_grad (floats).  Weights W2..W4 as they are in
// the parameters and activations by sample, both with rows of 68 floats: 16
// threads reading one float4 each from 16 consecutive rows (weights) or from
// one row meet no bank twice, and two rows four apart lie 16 banks apart.
constexpr int kLd = 68;
constexpr int kSmW1 = 0;                           // [64][4]
constexpr int kSmW2 = kSmW1 + kHid * kIn;          // [64][68] each
constexpr int kSmW3 = kSmW2 + kHid * kLd;
constexpr int kSmW4 = kSmW3 + kHid * kLd;
constexpr int kSmB = kSmW4 + kHid * kLd;           // biases b1..b4 (256)
constexpr int kSmX = kSmB + 4 * kHid;              // inputs [64][4]
constexpr int kSmA1 = kSmX + kSlice * kIn;         // activations [64][68] x 3
constexpr int kSmA2 = kSmA1 + kSlice * kLd;
constexpr int kSmA3 = kSmA2 + kSlice * kLd;
constexpr int kSmO = kSmA3 + kSlice * kLd;         // outputs, then their gradients
constexpr int kSmD = kSmO + kSlice * kLd;          // back-propagated deltas
constexpr int kSmQ = kSmD + kSlice * kLd;          // per sample and knot: softplus, sigmoid, loss term
constexpr int kSmTotal = kSmQ + 3 * kSlice * kQMax;
constexpr int kGradSmemBytes = kSmTotal * 4;
static_assert(kSmW2 % 4 == 0 && kSmB % 4 == 0 && kSmX % 4 == 0 && kSmA1 % 4 == 0, "float4 rows");

// Gradient of a sample's quantile losses with respect to its raw outputs, in
// place (O: its row; the three logits are left alone), by four neighbouring
// threads (q = 0..3).  The transcendentals and the loss terms of the knots are
// spread over the four threads; the two heads' sums run in the order of a
// single thread, one thread each.  sp, sg, tm: the sample's kQMax entries of
// each; tm is left with the loss terms.  valid: the sample exists (a padding
// row's gradient is zero).
static_assert(kNearL == 3, "the logits are the first three outputs");
__device__ __forceinline__ void heads_grad(float *O, int q, bool valid, int c, float y0, float y1, float *sp, float *sg,
                                           float *tm) {
    int h0 = 0, k0 = 0, h1 = 0, k1 = 0;
    heads_of(c, &h0, &k0, &h1, &k1);
    const int off = q == 0 ? 0 : k0, K = q == 0 ? k0 : k1, head = q == 0 ? h0 : h1;
    if (valid) {
        for (int e = q; e < k0 + k1; e += 4) {
            const float h = O[e < k0 ? h0 + e : h1 + e - k0];
            if (e != 0 && e != k0) {
                sp[e] = softplusf(h);
                sg[e] = 1.0f / (1.0f + expf(-h));
            } else {
                sp[e] = h;  // the head's first knot
            }
        }
    }
    __syncwarp();
    if (q == 0) O[3] = 0.0f;
    for (int j = q == 0 ? 16 : 4 * q; j < kOut; j += 16)
        *reinterpret_cast<float4 *>(O + j) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (valid && q < 2) {
        // the knots of one of the outcome's two heads
        float acc = sp[off];
#pragma unroll 5
        for (int k = 1; k < K; ++k) {
            acc += sp[off + k];
            sp[off + k] = acc;
        }
    }
    __syncwarp();
    if (valid) {
        // pinball losses; sp becomes d loss / d q_k
        for (int e = q; e < k0 + k1; e += 4) {
            const bool second = e >= k0;
            const float tau = second ? level(e - k0, k1) : level(e, k0), u = (second ? y1 : y0) - sp[e];
            tm[e] = u >= 0.0f ? tau * u : (tau - 1.0f) * u;
            sp[e] = (u < 0.0f ? 1.0f : 0.0f) - tau;
        }
    }
    __syncwarp();
    if (valid && q < 2) {
        // back through q_k = h_0 + sum_{j<=k, j>=1} softplus(h_j)
        float tail = 0.0f;
#pragma unroll 5
        for (int k = K - 1; k >= 1; --k) {
            tail += sp[off + k];
            O[head + k] = tail * sg[off + k];
        }
        O[head] = tail + sp[off];
    }
}

// The cross entropy of a sample's outcome, by one thread: leaves the gradient
// in the three logits and returns the loss.
__device__ __forceinline__ float outcome_grad(float *O, bool valid, int c) {
    float d0 = 0.0f, d1 = 0.0f, d2 = 0.0f, loss = 0.0f;
    if (valid) {
        const float m = fmaxf(O[0], fmaxf(O[1], O[2]));
        const float e0 = expf(O[0] - m), e1 = expf(O[1] - m), e2 = expf(O[2] - m);
        const float z = e0 + e1 + e2;
        loss = -(O[c] - m - logf(z));
        d0 = e0 / z - (c == 0 ? 1.0f : 0.0f);
        d1 = e1 / z - (c == 1 ? 1.0f : 0.0f);
        d2 = e2 / z - (c == 2 ? 1.0f : 0.0f);
    }
    O[0] = d0;
    O[1] = d1;
    O[2] = d2;
    return loss;
}

// The three products of a layer, each thread a 4 x 4 tile of the result in
// registers: two shared float4 loads feed 32 multiplies and adds, where one
// result per thread and step loaded two floats for one of each.  Every sum runs
// over its index in order, one product at a time, a multiply and an add each, as
// the library is built without contraction.  (FP32 issue bounds them: 256 threads x
// 16 sums x 64 products x 2 instructions are 4096 cycles a product on an SM; they
// take 5200 to 5800 whatever the mapping, prefetch or layout tried.  The
// histories need the separate roundings, these sums do not: fused they would be
// 2048 cycles, with parameters that differ in rounding; not tried.)
__device__ __forceinline__ float lane4(const float4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// z[s][j] = b[j] + sum_k W[j][k] a[s][k], the 64 x 64 outputs of a layer:
// outputs tj + 16 jj, samples 4 ts + i
template <int K>
__device__ __forceinline__ void dense_fwd(const float *W, int ldw, const float *b, const float *a, int lda, float *z,
                                          bool relu) {
    const int tj = threadIdx.x & 15, ts = threadIdx.x >> 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) acc[i][jj] = b[tj + 16 * jj];
#pragma unroll 4
    for (int k = 0; k < K; k += 4) {
        float4 w[4], v[4];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) w[jj] = *reinterpret_cast<const float4 *>(W + (tj + 16 * jj) * ldw + k);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = *reinterpret_cast<const float4 *>(a + (4 * ts + i) * lda + k);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) acc[i][jj] += lane4(w[jj], kk) * lane4(v[i], kk);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) z[(4 * ts + i) * kLd + tj + 16 * jj] = relu ? fmaxf(acc[i][jj], 0.0f) : acc[i][jj];
}

// weight gradients of one layer: gW[j][k] = sum_s dz[s][j] a[s][k]
__device__ __forceinline__ void dense_wgrad(const float *dz, const float *a, float *gW) {
    const int tk = threadIdx.x & 15, tj = threadIdx.x >> 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) acc[i][kk] = 0.0f;
#pragma unroll 8
    for (int s = 0; s < kSlice; ++s) {
        const float4 d = *reinterpret_cast<const float4 *>(dz + s * kLd + 4 * tj);
        const float4 v = *reinterpret_cast<const float4 *>(a + s * kLd + 4 * tk);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) acc[i][kk] += lane4(d, i) * lane4(v, kk);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4 *>(gW + (4 * tj + i) * kHid + 4 * tk) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}

// the first layer's weight gradients, one a thread
__device__ __forceinline__ void input_wgrad(const float *dz, const float *x, float *gW) {
    static_assert(kHid * kIn == kTileThreads, "one weight a thread");
    const int k = threadIdx.x % kIn, j = threadIdx.x / kIn;
    float acc = 0.0f;
#pragma unroll 16
    for (int s = 0; s < kSlice; ++s) acc += dz[s * kLd + j] * x[s * kIn + k];
    gW[threadIdx.x] = acc;
}

// bias gradient j of one layer
__device__ __forceinline__ void bias_grad(const float *dz, int j, float *gb) {
    float acc = 0.0f;
#pragma unroll 16
    for (int s = 0; s < kSlice; ++s) acc += dz[s * kLd + j];
    gb[j] = acc;
}

// delta of the layer below: da[s][k] = sum_j W[j][k] dz[s][j], masked by ReLU
__device__ __forceinline__ void dense_bwd(const float *W, const float *dz, const float *a_below, float *da) {
    const int tk = threadIdx.x & 15, ts = threadIdx.x >> 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) acc[i][kk] = 0.0f;
#pragma unroll 4
    for (int j = 0; j < kHid; j += 4) {
        float4 w[4], d[4];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) w[jj] = *reinterpret_cast<const float4 *>(W + (j + jj) * kLd + 4 * tk);
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = *reinterpret_cast<const float4 *>(dz + (4 * ts + i) * kLd + j);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) acc[i][kk] += lane4(w[jj], kk) * lane4(d[i], jj);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 m = *reinterpret_cast<const float4 *>(a_below + (4 * ts + i) * kLd + 4 * tk);
        *reinterpret_cast<float4 *>(da + (4 * ts + i) * kLd + 4 * tk) =
            make_float4(m.x > 0.0f ? acc[i][0] : 0.0f, m.y > 0.0f ? acc[i][1] : 0.0f, m.z > 0.0f ? acc[i][2] : 0.0f,
                        m.w > 0.0f ? acc[i][3] : 0.0f);
    }
}

// 16 bytes to shared memory, without a register
__device__ __forceinline__ void copy16(float *smem, const float *from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(from) : "memory");
}
__device__ __forceinline__ void copies_issued() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_arrived() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

// Forward + backward of samples [off + 64 b, off + 64 b + 64) clipped to n;
// writes this block's gradient sums (kParams floats) and loss sum.  One block
// an SM; a batch of 8192 walks is 128 of them.  The first 256 threads run the
// layers' products and the quantile heads; the last 64, one sample or one
// output each, the serial sums beside them: cross entropy, bias gradients, loss.
// The weights of a layer arrive while the layer before it runs.  (With the sums
// after the products on the same threads, the first layer's gradients on 16
// threads and the weights waited for at the start: 33.5 us against 30.6; the
// barriers at block scope, which both roles share, add 0.4.)
__global__ void __launch_bounds__(kTrainThreads) k_surr_grad(const float *P, const float *x, const int *cls,
                                                             const float *tgt, long long n, long long off,
                                                             float *gpart, float *lpart) {
    extern __shared__ __align__(16) float sm[];
    float *W1 = sm + kSmW1, *W2 = sm + kSmW2, *W3 = sm + kSmW3, *W4 = sm + kSmW4, *B = sm + kSmB, *X = sm + kSmX;
    float *A1 = sm + kSmA1, *A2 = sm + kSmA2, *A3 = sm + kSmA3, *O = sm + kSmO, *D = sm + kSmD;
    float *SP = sm + kSmQ, *SG = SP + kSlice * kQMax, *TM = SG + kSlice * kQMax;
    __shared__ float sloss[kSlice];
    const long long s0 = off + (long long)blockIdx.x * kSlice;
    float *g = gpart + (size_t)blockIdx.x * kParams;
    // the two roles; every barrier is the whole block's
    const bool tiles = threadIdx.x < kTileThreads;
    const int j = threadIdx.x - kTileThreads;  // the serial sums' sample and output
    // this thread's sample of the output gradient
    const int smp = tiles ? threadIdx.x >> 2 : j;
    const bool valid = s0 + smp < n;
    int c = 0;
    float y0 = 0.0f, y1 = 0.0f, l = 0.0f;
    if (tiles) {
        static_assert(kHid * kIn == kTileThreads && kSlice * kIn == kTileThreads, "one element a thread");
        const long long i = s0 + threadIdx.x / kIn;
        const float w1 = P[kW1 + threadIdx.x], x1 = i < n ? x[i * kIn + threadIdx.x % kIn] : 0.0f;
        auto fetch = [&](float *W, const float *from) {
#pragma unroll
            for (int r = 0; r < kHid * kHid; r += 4 * kTileThreads) {
                const int e = r + 4 * threadIdx.x;
                copy16(W + (e / kHid) * kLd + e % kHid, from + e);
            }
            copies_issued();
        };
        fetch(W2, P + kW2);
        fetch(W3, P + kW3);
        fetch(W4, P + kW4);
        W1[threadIdx.x] = w1;
        X[threadIdx.x] = x1;
        if (valid) { c = cls[s0 + smp]; y0 = tgt[2 * (s0 + smp)]; y1 = tgt[2 * (s0 + smp) + 1]; }
    } else {
        if (valid) c = cls[s0 + smp];
        B[j] = P[kB1 + j]; B[kHid + j] = P[kB2 + j]; B[2 * kHid + j] = P[kB3 + j]; B[3 * kHid + j] = P[kB4 + j];
    }
    __syncthreads();
    if (tiles) {
        dense_fwd<kIn>(W1, kIn, B, X, kIn, A1, true);
        copies_arrived<2>();
    }
    __syncthreads();
    if (tiles) {
        dense_fwd<kHid>(W2, kLd, B + kHid, A1, kLd, A2, true);
        copies_arrived<1>();
    }
    __syncthreads();
    if (tiles) {
        dense_fwd<kHid>(W3, kLd, B + 2 * kHid, A2, kLd, A3, true);
        copies_arrived<0>();
    }
    __syncthreads();
    if (tiles) dense_fwd<kHid>(W4, kLd, B + 3 * kHid, A3, kLd, O, false);
    __syncthreads();
    if (tiles)
        heads_grad(O + smp * kLd, threadIdx.x & 3, valid, c, y0, y1, SP + smp * kQMax, SG + smp * kQMax, TM + smp * kQMax);
    else
        l = outcome_grad(O + j * kLd, valid, c);
    __syncthreads();
    if (tiles) {
        dense_wgrad(O, A3, g + kW4);
        dense_bwd(W4, O, A3, D);  // delta at layer 3 output
    } else {
        bias_grad(O, j, g + kB4);
        if (valid) {
            int h0, k0, h1, k1;
            heads_of(c, &h0, &k0, &h1, &k1);
            for (int k = 0; k < k0 + k1; ++k) l += TM[j * kQMax + k];
        }
        sloss[j] = l;
    }
    __syncthreads();
    if (tiles) {
        dense_wgrad(D, A2, g + kW3);
        dense_bwd(W3, D, A2, O);  // delta at layer 2 output (reuses O)
    } else {
        bias_grad(D, j, g + kB3);
        if (j == 0) {
            float sum = 0.0f;
#pragma unroll 16
            for (int s = 0; s < kSlice; ++s) sum += sloss[s];
            lpart[blockIdx.x] = sum;
        }
    }
    __syncthreads();
    if (tiles) {
        dense_wgrad(O, A1, g + kW2);
        dense_bwd(W2, O, A1, D);  // delta at layer 1 output
    } else {
        bias_grad(O, j, g + kB2);
    }
    __syncthreads();
    if (tiles) input_wgrad(D, X, g + kW1);
    else bias_grad(D, j, g + kB1);
}

// scale * sum_b gpart[b][p], in block order (the loads of 64 blocks in flight:
// their latency bounds it, 5.2 us for 128 blocks, 5.8 with 16)
constexpr int kReduceThreads = 64;
template <int N> __device__ __forceinline__ void add_blocks(const float *gpart, int p, int *b, float *acc) {
    float v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = gpart[(size_t)(*b + i) * kParams + p];
#pragma unroll
    for (int i = 0; i < N; ++i) *acc += v[i];
    *b += N;
}
__device__ __forceinline__ float reduce_param(const float *gpart, int nblk, float scale, int p) {
    float acc = 0.0f;
    int b = 0;
    while (b + 64 <= nblk) add_blocks<64>(gpart, p, &b, &acc);
    while (b + 16 <= nblk) add_blocks<16>(gpart, p, &b, &acc);
    for (; b < nblk; ++b) acc += gpart[(size_t)b * kParams + p];
    return acc * scale;
}

__global__ void __launch_bounds__(kReduceThreads) k_surr_reduce(const float *gpart, int nblk, float scale, float *grad) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < kParams) grad[p] = reduce_param(gpart, nblk, scale, p);
}

// the reduction and the Adam step of each parameter
__global__ void __launch_bounds__(kReduceThreads) k_surr_adam(float *P, float *m, float *v, const float *gpart, int nblk,
                                                              float scale, float lr, float b1t, float b2t) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kParams) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float gr = reduce_param(gpart, nblk, scale, p);
    const float mm = b1 * m[p] + (1.0f - b1) * gr;
    const float vv = b2 * v[p] + (1.0f - b2) * gr * gr;
    m[p] = mm;
    v[p] = vv;
    P[p] -= lr * (mm / (1.0f - b1t)) / (sqrtf(vv / (1.0f - b2t)) + eps);
}

// He-uniform weights, zero biases; deterministic in the seed
__global__ void k_surr_init(float *P, unsigned long long seed) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kParams) return;
    int fan_in;
    bool is_w = true;
    if (p < kB1) fan_in = kIn;
    else if (p < kW2) is_w = false;
    else if (p < kB2) fan_in = kHid;
    else if (p < kW3) is_w = false;
    else if (p < kB3) fan_in = kHid;
    else if (p < kW4) is_w = false;
    else if (p < kB4) fan_in = kHid;
    else is_w = false;
    if (!is_w) { P[p] = 0.0f; return; }
    Stream rs;
    rs.init(seed, 1u, (uint32_t)p, kStageSurrData);
    const float bound = sqrtf(6.0f / (float)fan_in);
    float w = (2.0f * Rand<float>::u(rs) - 1.0f) * bound;
    if (p >= kW4) w *= 0.1f;  // small initial outputs
    P[p] = w;
}

// ------------------------------------------------------ tensor-core tests
constexpr int kFwdWarps = 4;
constexpr int kFwdSmemBytes = kImageBytes + kFwdWarps * kStageFloats * 4;

// network outputs of n given inputs, 16 rows per warp per pass
__global__ void __launch_bounds__(32 * kFwdWarps) k_surr_forward(const float *P, const float *x, long long n,
                                                                 float *out) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t *frag = reinterpret_cast<uint32_t *>(smem);
    float *bias = reinterpret_cast<float *>(frag + kFragWords);
    float *stage = bias + kBiasFloats + (threadIdx.x >> 5) * kStageFloats;
    float *xin = stage, *yout = stage + 16 * kIn;
    build_image(P, frag, bias);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long nwarps = (long long)gridDim.x * kFwdWarps;
    for (long long r0 = ((long long)blockIdx.x * kFwdWarps + (threadIdx.x >> 5)) * 16; r0 < n; r0 += nwarps * 16) {
        for (int e = lane; e < 16 * kIn; e += 32) {
            const long long r = r0 + e / kIn;
            xin[e] = r < n ? x[r * kIn + e % kIn] : 0.0f;
        }
        __syncwarp();
        forward16(frag, bias, xin, yout);
        for (int e = lane; e < 16 * kOut; e += 32) {
            const long long r = r0 + e / kOut;
            if (r < n) out[r * kOut + e % kOut] = yout[e];
        }
        __syncwarp();
    }
}

// outcomes sampled from the network at n walk states (d_n, d_f, mu', lmax)
__global__ void __launch_bounds__(32 * kFwdWarps) k_surr_sample(const float *P, unsigned long long seed,
                                                                const float *state, long long n, int *cls,
                                                                float *y0, float *y1) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t *frag = reinterpret_cast<uint32_t *>(smem);
    float *bias = reinterpret_cast<float *>(frag + kFragWords);
    float *stage = bias + kBiasFloats + (threadIdx.x >> 5) * kStageFloats;
    float *xin = stage, *yout = stage + 16 * kIn;
    build_image(P, frag, bias);
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const long long nwarps = (long long)gridDim.x * kFwdWarps;
    for (long long r0 = ((long long)blockIdx.x * kFwdWarps + (threadIdx.x >> 5)) * 16; r0 < n; r0 += nwarps * 16) {
        if (lane < 16) {
            const long long r = r0 + lane;
            float f[kIn] = {0.0f, 0.0f, 0.0f, 0.0f};
            if (r < n) features(state[4 * r], state[4 * r + 1], state[4 * r + 2], state[4 * r + 3], f);
            for (int k = 0; k < kIn; ++k) xin[lane * kIn + k] = f[k];
        }
        __syncwarp();
        forward16(frag, bias, xin, yout);
        if (lane < 16 && r0 + lane < n) {
            const long long r = r0 + lane;
            Stream rs;
            rs.init(seed, 0u, (uint32_t)r, kStageSurrTest);
            const float u0 = Rand<float>::u(rs), u1 = Rand<float>::u(rs), u2 = Rand<float>::u(rs);
            float a, b;
            cls[r] = sample_outcome(yout + lane * kOut, u0, u1, u2, &a, &b);
            y0[r] = a;
            y1[r] = b;
        }
        __syncwarp();
    }
}

}  // namespace

// ------------------------------------------------------------ entry points
namespace {

// device buffers of one call, released on every return path
struct DevScope {
    std::vector<void *> ptrs;
    cudaStream_t stream = nullptr;
    ~DevScope() {
        if (stream) cudaStreamSynchronize(stream);
        for (void *p : ptrs) cudaFree(p);
        if (stream) cudaStreamDestroy(stream);
    }
    template <class T> T *alloc(size_t count) {
        void *p = nullptr;
        if (count == 0) count = 1;
        if (cudaMalloc(&p, count * sizeof(T)) != cudaSuccess) return nullptr;
        ptrs.push_back(p);
        return static_cast<T *>(p);
    }
};

int surr_device(DevScope &ds) {
    int dev = 0, major = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return IMC_ERR_NO_DEVICE;
    if (cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, dev) != cudaSuccess || major < 10)
        return IMC_ERR_NO_DEVICE;
    if (cudaStreamCreateWithFlags(&ds.stream, cudaStreamNonBlocking) != cudaSuccess) return IMC_ERR_CUDA;
    return IMC_OK;
}

int h2d(void *d, const void *h, size_t bytes, cudaStream_t s) {
    return cudaMemcpyAsync(d, h, bytes, cudaMemcpyHostToDevice, s) == cudaSuccess ? IMC_OK : IMC_ERR_CUDA;
}
int d2h(void *h, const void *d, size_t bytes, cudaStream_t s) {
    return cudaMemcpyAsync(h, d, bytes, cudaMemcpyDeviceToHost, s) == cudaSuccess ? IMC_OK : IMC_ERR_CUDA;
}
int finish(cudaStream_t s) {
    if (cudaGetLastError() != cudaSuccess) return IMC_ERR_CUDA;
    return cudaStreamSynchronize(s) == cudaSuccess ? IMC_OK : IMC_ERR_CUDA;
}

int grid_of(long long n, int per_block, int cap) {
    long long b = (n + per_block - 1) / per_block;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

// n walks on a grid of at most four blocks an SM
int launch_datagen(DevScope &ds, unsigned long long seed, long long n, const float *state, float *x, int *cls,
                   float *tgt) {
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return IMC_ERR_CUDA;
    unsigned long long *counter = ds.alloc<unsigned long long>(1);
    if (!counter) return IMC_ERR_OOM;
    if (cudaMemsetAsync(counter, 0, sizeof(*counter), ds.stream) != cudaSuccess) return IMC_ERR_CUDA;
    k_surr_datagen<<<grid_of(n, kDatagenPerLane * kDatagenThreads, 4 * sms), kDatagenThreads, 0, ds.stream>>>(seed, n, state, x, cls, tgt,
                                                                                          counter);
    return IMC_OK;
}

// per-slice gradients and the block-order reduction: grad = mean over n
int launch_grad(const float *P, const float *x, const int *cls, const float *tgt, long long n, long long off,
                float *gpart, float *lpart, float *grad, cudaStream_t s) {
    const int nblk = (int)((n + kSlice - 1) / kSlice);
    k_surr_grad<<<nblk, kTrainThreads, kGradSmemBytes, s>>>(P, x, cls, tgt, off + n, off, gpart, lpart);
    k_surr_reduce<<<(kParams + kReduceThreads - 1) / kReduceThreads, kReduceThreads, 0, s>>>(gpart, nblk,
                                                                                             1.0f / (float)n, grad);
    return cudaGetLastError() == cudaSuccess ? IMC_OK : IMC_ERR_CUDA;
}

bool smem_optin() {
    static bool done = false;
    if (done) return true;
    if (cudaFuncSetAttribute(k_surr_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, kGradSmemBytes) != cudaSuccess)
        return false;
    done = true;
    return true;
}

}  // namespace

extern "C" {

int imc_surrogate_param_count(int *count) {
    if (!count) return IMC_ERR_INVALID_ARG;
    *count = kParams;
    return IMC_OK;
}

int imc_surrogate_walk(uint64_t seed, const float *state, int64_t n, float *x, int32_t *cls, float *tgt) {
    if (n < 0 || (n > 0 && (!x || !cls || !tgt)) || n > (int64_t)0xFFFFFFFF) return IMC_ERR_INVALID_ARG;
    if (n == 0) return IMC_OK;
    DevScope ds;
    int rc = surr_device(ds);
    if (rc) return rc;
    float *dstate = nullptr;
    if (state) {
        if (!(dstate = ds.alloc<float>(4 * n))) return IMC_ERR_OOM;
        if ((rc = h2d(dstate, state, 16 * (size_t)n, ds.stream))) return rc;
    }
    float *dx = ds.alloc<float>(kIn * n), *dt = ds.alloc<float>(2 * n);
    int *dc = ds.alloc<int>(n);
    if (!dx || !dt || !dc) return IMC_ERR_OOM;
    if ((rc = launch_datagen(ds, seed, n, dstate, dx, dc, dt))) return rc;
    if ((rc = d2h(x, dx, 4 * kIn * (size_t)n, ds.stream)) || (rc = d2h(cls, dc, 4 * (size_t)n, ds.stream)) ||
        (rc = d2h(tgt, dt, 8 * (size_t)n, ds.stream)))
        return rc;
    return finish(ds.stream);
}

int imc_surrogate_grad(const float *params, const float *x, const int32_t *cls, const float *tgt, int64_t n,
                       float *grad, double *loss) {
    if (!params || !x || !cls || !tgt || !grad || n <= 0) return IMC_ERR_INVALID_ARG;
    for (int64_t i = 0; i < n; ++i)
        if (cls[i] < 0 || cls[i] > 2) return IMC_ERR_INVALID_ARG;
    DevScope ds;
    int rc = surr_device(ds);
    if (rc) return rc;
    if (!smem_optin()) return IMC_ERR_CUDA;
    const int nblk = (int)((n + kSlice - 1) / kSlice);
    float *dP = ds.alloc<float>(kParams), *dx = ds.alloc<float>(kIn * n), *dt = ds.alloc<float>(2 * n);
    int *dc = ds.alloc<int>(n);
    float *gpart = ds.alloc<float>((size_t)nblk * kParams), *lpart = ds.alloc<float>(nblk);
    float *dg = ds.alloc<float>(kParams);
    if (!dP || !dx || !dt || !dc || !gpart || !lpart || !dg) return IMC_ERR_OOM;
    if ((rc = h2d(dP, params, 4 * (size_t)kParams, ds.stream)) || (rc = h2d(dx, x, 4 * kIn * (size_t)n, ds.stream)) ||
        (rc = h2d(dc, cls, 4 * (size_t)n, ds.stream)) || (rc = h2d(dt, tgt, 8 * (size_t)n, ds.stream)))
        return rc;
    if ((rc = launch_grad(dP, dx, dc, dt, n, 0, gpart, lpart, dg, ds.stream))) return rc;
    std::vector<float> lp(nblk);
    if ((rc = d2h(grad, dg, 4 * (size_t)kParams, ds.stream)) || (rc = d2h(lp.data(), lpart, 4 * (size_t)nblk, ds.stream)))
        return rc;
    if ((rc = finish(ds.stream))) return rc;
    if (loss) {
        double l = 0.0;
        for (float v : lp) l += v;
        *loss = l / (double)n;
    }
    return IMC_OK;
}

int imc_surrogate_train(const ImcSurrogateTrainConfig *cfg, float *params, float *loss_history) {
    if (!cfg || !params) return IMC_ERR_INVALID_ARG;
    const long long n = cfg->n_samples;
    const int B = cfg->batch;
    if (n <= 0 || n > (int64_t)0xFFFFFFFF || B <= 0 || B % kSlice || n % B || cfg->iterations <= 0 ||
        !(cfg->lr > 0.0f) || cfg->lr_min < 0.0f)
        return IMC_ERR_INVALID_ARG;
    DevScope ds;
    int rc = surr_device(ds);
    if (rc) return rc;
    if (!smem_optin()) return IMC_ERR_CUDA;
    const int nblk = B / kSlice;
    float *dx = ds.alloc<float>(kIn * n), *dt = ds.alloc<float>(2 * n);
    int *dc = ds.alloc<int>(n);
    float *dP = ds.alloc<float>(kParams), *dm = ds.alloc<float>(kParams), *dv = ds.alloc<float>(kParams);
    float *gpart = ds.alloc<float>((size_t)nblk * kParams);
    float *lpart = ds.alloc<float>((size_t)nblk * cfg->iterations);
    if (!dx || !dt || !dc || !dP || !dm || !dv || !gpart || !lpart) return IMC_ERR_OOM;
    if ((rc = launch_datagen(ds, cfg->seed, n, nullptr, dx, dc, dt))) return rc;
    k_surr_init<<<(kParams + 255) / 256, 256, 0, ds.stream>>>(dP, cfg->seed);
    if (cudaMemsetAsync(dm, 0, 4 * (size_t)kParams, ds.stream) != cudaSuccess ||
        cudaMemsetAsync(dv, 0, 4 * (size_t)kParams, ds.stream) != cudaSuccess)
        return IMC_ERR_CUDA;
    double b1t = 1.0, b2t = 1.0;
    const double pi = 3.14159265358979323846;
    for (int it = 0; it < cfg->iterations; ++it) {
        const long long off = ((long long)it * B) % n;
        k_surr_grad<<<nblk, kTrainThreads, kGradSmemBytes, ds.stream>>>(dP, dx, dc, dt, off + B, off, gpart,
                                                                        lpart + (size_t)it * nblk);
        b1t *= 0.9;
        b2t *= 0.999;
        const double lr = cfg->lr_min + 0.5 * (cfg->lr - cfg->lr_min) * (1.0 + cos(pi * it / cfg->iterations));
        k_surr_adam<<<(kParams + kReduceThreads - 1) / kReduceThreads, kReduceThreads, 0, ds.stream>>>(
            dP, dm, dv, gpart, nblk, 1.0f / (float)B, (float)lr, (float)b1t, (float)b2t);
        if (cudaGetLastError() != cudaSuccess) return IMC_ERR_CUDA;
    }
    if ((rc = d2h(params, dP, 4 * (size_t)kParams, ds.stream))) return rc;
    std::vector<float> lp;
    if (loss_history) {
        lp.resize((size_t)nblk * cfg->iterations);
        if ((rc = d2h(lp.data(), lpart, 4 * lp.size(), ds.stream))) return rc;
    }
    if ((rc = finish(ds.stream))) return rc;
    if (loss_history) {
        for (int it = 0; it < cfg->iterations; ++it) {
            double l = 0.0;
            for (int b = 0; b < nblk; ++b) l += lp[(size_t)it * nblk + b];
            loss_history[it] = (float)(l / B);
        }
    }
    return IMC_OK;
}

int imc_surrogate_forward(const float *params, const float *x, int64_t n, float *out) {
    if (!params || n < 0 || (n > 0 && (!x || !out))) return IMC_ERR_INVALID_ARG;
    if (n == 0) return IMC_OK;
    DevScope ds;
    int rc = surr_device(ds);
    if (rc) return rc;
    float *dP = ds.alloc<float>(kParams), *dx = ds.alloc<float>(kIn * n), *dout = ds.alloc<float>(kOut * n);
    if (!dP || !dx || !dout) return IMC_ERR_OOM;
    if ((rc = h2d(dP, params, 4 * (size_t)kParams, ds.stream)) || (rc = h2d(dx, x, 4 * kIn * (size_t)n, ds.stream)))
        return rc;
    k_surr_forward<<<grid_of(n, 16 * kFwdWarps, 1024), 32 * kFwdWarps, kFwdSmemBytes, ds.stream>>>(dP, dx, n, dout);
    if ((rc = d2h(out, dout, 4 * kOut * (size_t)n, ds.stream))) return rc;
    return finish(ds.stream);
}

int imc_surrogate_sample(const float *params, uint64_t seed, const float *state, int64_t n, int32_t *cls, float *y0,
                         float *y1) {
    if (!params || n < 0 || n > (int64_t)0xFFFFFFFF || (n > 0 && (!state || !cls || !y0 || !y1)))
        return IMC_ERR_INVALID_ARG;
    if (n == 0) return IMC_OK;
    DevScope ds;
    int rc = surr_device(ds);
    if (rc) return rc;
    float *dP = ds.alloc<float>(kParams), *dst = ds.alloc<float>(4 * n);
    float *d0 = ds.alloc<float>(n), *d1 = ds.alloc<float>(n);
    int *dc = ds.alloc<int>(n);
    if (!dP || !dst || !d0 || !d1 || !dc) return IMC_ERR_OOM;
    if ((rc = h2d(dP, params, 4 * (size_t)kParams, ds.stream)) || (rc = h2d(dst, state, 16 * (size_t)n, ds.stream)))
        return rc;
    k_surr_sample<<<grid_of(n, 16 * kFwdWarps, 1024), 32 * kFwdWarps, kFwdSmemBytes, ds.stream>>>(dP, seed, dst, n, dc,
                                                                                                d0, d1);
    if ((rc = d2h(cls, dc, 4 * (size_t)n, ds.stream)) || (rc = d2h(y0, d0, 4 * (size_t)n, ds.stream)) ||
        (rc = d2h(y1, d1, 4 * (size_t)n, ds.stream)))
        return rc;
    return finish(ds.stream);
}

}  // extern "C"
