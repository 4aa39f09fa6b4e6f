// imc_kernels.cu -- the O(ncells) stages (FP64) and the particle-list stages
// around transport.
//
//   k_update           <- Update.update                 src/imc_update.jl:12-56
//   k_source_slots     <- Sourcing.sourcing, energies     src/imc_sourcing.jl:56-121
//                         (the step sequence: with Update.update in the launch)
//   k_source_counts    <- Sourcing.sourcing, total/budget/counts src/imc_sourcing.jl:121-157
//   k_source_emit      <- Sourcing.sourcing, births        src/imc_sourcing.jl:159-366
//   k_compact_*        <- Clean.clean                    src/imc_clean.jl:6-19
//   k_tally            <- Tally.tally                    src/imc_tally.jl:22-142
//   k_energycheck      <- EnergyCheck.energychecker      src/imc_energycheck.jl:19-38
//   k_timestep         <- timestep                       src/MixedPrecisionIMC.jl:181-222
//   k_tally_check      the step sequence: finalize, tally, energy check, clock
//
// Sums over cells are exact to 93 bits below the largest term inside a warp's
// unit of 32, then over the units' partials in the last block to finish --
// deterministic, and within a rounding of the exact sum.  Every launch has a fixed grid and reads its sizes from
// device scalars, so a whole step can be captured once as a CUDA graph.
#include <cstdint>
#include "imc_device.cuh"
#include "imc_internal.h"
#include "imc_state.cuh"
#include "imc_transport.cuh"

namespace imc {

// GB300 executes FP64 at 1/64 of the FP32 rate, so a per-cell FP64 stage runs as
// one warp, or one warp for each of an SM's four FP64 units, a block, spread over
// the SMs, and keeps what it can in integers; sums run over a fixed partition of
// the cells (units of kCellThreads).

// x / s for an energy scale s: the scales in use are 1 and powers of two, whose
// quotients need no division
__device__ __forceinline__ double div_scale(double x, double s) {
    const uint64_t b = d2u(s);
    if (b == 0x3FF0000000000000ull) return x;
    const int ex = (int)(b >> 52);  // s > 0
    if ((b & 0xFFFFFFFFFFFFFull) == 0 && ex >= 1 && ex <= 2045) return x * m64::from_bits((uint64_t)(2046 - ex) << 52);
    return x / s;
}

// v 2^e: by the exponent bits where both are normal numbers
__device__ __forceinline__ double times_pow2(double v, int e) {
    const uint64_t b = d2u(v);
    const int ex = (int)((b >> 52) & 0x7FFu), to = ex + e;
    if (ex == 0 || ex == 0x7FF || to <= 0 || to >= 0x7FF) return ldexp(v, e);
    return m64::from_bits(b + ((uint64_t)(int64_t)e << 52));
}

// ---- sums over the lanes of a warp
// A double as up to 93 bits of a fixed-point number whose top bit is that of
// the largest exponent present: four signed 24-bit digits.  32 or more such
// digits add up in 32 bits with the warp's integer reduction, so a sum costs a
// handful of FP64 instructions (the digits back to two doubles) where a tree
// of double-double adds took 40 (each as long as 64 FP32 instructions: half of
// the step's tail).  What lies 93 bits below the largest term is rounded away, as a
// double-double sum's is.
struct Digits {
    int d[4];
    __device__ __forceinline__ void clear() { d[0] = d[1] = d[2] = d[3] = 0; }
    // emax: the largest biased exponent (1..2046)
    __device__ __forceinline__ void add(double x, int emax) {
        const uint64_t b = d2u(x);
        const int ex = (int)((b >> 52) & 0x7FFu);
        uint64_t man = b & 0xFFFFFFFFFFFFFull;
        if (ex) man |= 0x10000000000000ull;
        const int sh = emax - (ex ? ex : 1);
        uint64_t hi = man >> 24, lo = man << 40;  // man 2^40 in 128 bits
        if (sh >= 64) {
            lo = sh < 128 ? hi >> (sh - 64) : 0ull;
            hi = 0ull;
        } else if (sh > 0) {
            lo = (lo >> sh) | (hi << (64 - sh));
            hi >>= sh;
        }
        const int sg = (long long)b < 0 ? -1 : 1;
        d[0] += sg * (int)(lo & 0xFFFFFFull);
        d[1] += sg * (int)((lo >> 24) & 0xFFFFFFull);
        d[2] += sg * (int)((lo >> 48) | ((hi & 0xFFull) << 16));
        d[3] += sg * (int)(hi >> 8);
    }
    __device__ __forceinline__ void warp_sum() {
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = __reduce_add_sync(0xFFFFFFFFu, d[i]);
    }
    // emax as in add, at least kDigitsExpMin: the scales are normal numbers
    __device__ __forceinline__ DD value(int emax) const {
        const long long top = ((long long)d[3] << 24) + d[2], low = ((long long)d[1] << 24) + d[0];
        // units 2^(emax - 1075 - 40) and, of top, 2^48 of them
        const double u = m64::from_bits((uint64_t)(emax - 1075 - 40 + 1023) << 52);
        const double a = (double)top * (u * 0x1p48), c = (double)low * u;
        DD r;
        r.hi = a + c;
        r.lo = c - (r.hi - a);
        return r;
    }
};
constexpr int kDigitsExpMin = 128;
__device__ __forceinline__ int biased_exp(double x) { return (int)((d2u(x) >> 52) & 0x7FFu); }
// digits serve for finite terms that are not all tiny
__device__ __forceinline__ bool digits_serve(int emax) { return emax >= kDigitsExpMin && emax < 0x7FF; }

// the bits of the largest of the lanes' doubles, none of them negative or NaN
__device__ __forceinline__ unsigned long long warp_max_bits(double v) {
    const uint64_t b = d2u(v);
    const unsigned hi = __reduce_max_sync(0xFFFFFFFFu, (unsigned)(b >> 32));
    const unsigned lo = __reduce_max_sync(0xFFFFFFFFu, (unsigned)(b >> 32) == hi ? (unsigned)b : 0u);
    return ((unsigned long long)hi << 32) | lo;
}

// sum of one double-double a lane over the warp, by shuffles (any values)
__device__ __forceinline__ DD warp_sum_tree(DD d) {
    for (int off = 16; off > 0; off >>= 1) {
        DD o;
        o.hi = __shfl_down_sync(0xFFFFFFFFu, d.hi, off);
        o.lo = __shfl_down_sync(0xFFFFFFFFu, d.lo, off);
        if ((int)(threadIdx.x & 31) < off) d.add(o);
    }
    d.hi = __shfl_sync(0xFFFFFFFFu, d.hi, 0);
    d.lo = __shfl_sync(0xFFFFFFFFu, d.lo, 0);
    return d;
}

// sum of one double a lane over the warp, on every lane
__device__ __forceinline__ DD warp_sum(double x) {
    const int emax = __reduce_max_sync(0xFFFFFFFFu, biased_exp(x));
    if (!__any_sync(0xFFFFFFFFu, x != 0.0)) {
        DD z;
        z.clear();
        return z;
    }
    if (!digits_serve(emax)) {
        DD d;
        d.hi = x;
        d.lo = 0.0;
        return warp_sum_tree(d);
    }
    Digits g;
    g.clear();
    g.add(x, emax);
    g.warp_sum();
    return g.value(emax);
}

// Sum of the double-double partials of one group by one warp (lane l takes
// partials l, l + 32, ...), on every lane: digits again, summed in 64 bits, as
// there may be thousands of partials.  Deterministic.
__device__ __forceinline__ double warp_sum_partials(const double *part, int nb, int stride, int g) {
    const int lane = threadIdx.x & 31;
    int emax = 0;
    for (int bb = lane; bb < nb; bb += 32) emax = max(emax, biased_exp(part[(bb * stride + g) * 2]));
    emax = __reduce_max_sync(0xFFFFFFFFu, emax);
    if (emax == 0) return 0.0;  // (subnormal sums are no energies)
    if (nb < (1 << 16) && digits_serve(emax)) {
        long long t[4] = {0, 0, 0, 0};
        for (int bb = lane; bb < nb; bb += 32) {
            Digits d;
            d.clear();
            d.add(part[(bb * stride + g) * 2], emax);
            d.add(part[(bb * stride + g) * 2 + 1], emax);
#pragma unroll
            for (int i = 0; i < 4; ++i) t[i] += d.d[i];
        }
        for (int off = 16; off > 0; off >>= 1)
#pragma unroll
            for (int i = 0; i < 4; ++i) t[i] += __shfl_xor_sync(0xFFFFFFFFu, t[i], off);
        // carries up: t[0..2] in [0, 2^24), t[3] signed, below 2^38
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            t[i + 1] += t[i] >> 24;
            t[i] &= 0xFFFFFFll;
        }
        const long long top = t[3] * (1ll << 24) + t[2], low = (t[1] << 24) + t[0];
        const double u = m64::from_bits((uint64_t)(emax - 1075 - 40 + 1023) << 52);
        const double a = (double)(top >> 32) * (u * 0x1p80), b = (double)(top & 0xFFFFFFFFll) * (u * 0x1p48);
        const double s = a + b;
        return s + ((b - (s - a)) + (double)low * u);
    }
    DD d;
    d.clear();
    for (int bb = lane; bb < nb; bb += 32) {
        DD p;
        p.hi = part[(bb * stride + g) * 2];
        p.lo = part[(bb * stride + g) * 2 + 1];
        d.add(p);
    }
    return warp_sum_tree(d).val();
}

// ------------------------------------------------------------------ update
struct CellLaws { double T, f, sa; };
// Update.update for cell i (src/imc_update.jl:12-56); WRITE: also leaves the
// fields and the transport's table row
template <bool WRITE>
__device__ __forceinline__ CellLaws update_cell(const CellArgs &ca, double dt, int i) {
    const double a = ca.a, c = ca.c;
    const double one[1] = {1.0};
    CellLaws u;
    const double T = ca.temp[i];
    const double T3 = T * T * T;
    double beta;
    if (ca.linearized) {
        if (WRITE) ca.bee[i] = (4.0 * a) * T3;
        beta = 1.0;
    } else {
        beta = ((4.0 * a) * T3) / ca.bee[i];
    }
    const double Tc = (ca.temp_floor > 0.0 && T < ca.temp_floor) ? ca.temp_floor : T;
    double sa = ca.sa_val[i] * m64::pow_law(Tc, ca.sa_pow[i]);
    if (ca.marshak) sa = ca.sa_val[i] / Tc / Tc / Tc;
    double v[6] = {ca.ds, ca.alpha, beta, c, dt, sa};
    int j;
    const double prod = sorter_n<0, 6>(v, one, 1, &j);
    u.T = T;
    u.sa = sa;
    u.f = 1.0 / (1.0 + prod);
    if (WRITE) {
        const double ss = ca.ss_val[i] * m64::pow_law(Tc, ca.ss_pow[i]);
        ca.beta[i] = beta;
        ca.sa[i] = sa;
        ca.ss[i] = ss;
        ca.fleck[i] = u.f;
        if (ca.prec == 0) store_tab<double>(ca, i, sa, u.f, ss);
        else store_tab<float>(ca, i, sa, u.f, ss);
    }
    return u;
}

__global__ void __launch_bounds__(kCellThreads) k_update(CellArgs ca, Scalars *sc) {
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->flags = 0;
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ca.nc) update_cell<true>(ca, sc->dt, i);
}

__global__ void __launch_bounds__(kCellThreads) k_table(CellArgs ca) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ca.nc) return;
    if (ca.prec == 0) store_tab<double>(ca, i, ca.sa[i], ca.fleck[i], ca.ss[i]);
    else store_tab<float>(ca, i, ca.sa[i], ca.fleck[i], ca.ss[i]);
}

void launch_update(const CellArgs &ca, Scalars *sc, cudaStream_t st) {
    k_update<<<ca.nblk_cell, kCellThreads, 0, st>>>(ca, sc);
}

void launch_table(const CellArgs &ca, cudaStream_t st) {
    k_table<<<ca.nblk_cell, kCellThreads, 0, st>>>(ca);
}

// ---------------------------------------------------------------- sourcing

__device__ __forceinline__ int nsurf_slots(const CellArgs &ca) {
    return ca.geometry == 1 ? 2 : 2 * ca.nx + 2 * ca.ny;
}

// source-slot groups for the energy sums: 0 body, 1 radiation source,
// 2..5 the faces bottom, top, left, right (2D); 1D surfaces are added directly
__device__ __forceinline__ int slot_group(const CellArgs &ca, int s) {
    const int ns = nsurf_slots(ca);
    if (s >= ns + ca.nc) return 1;
    if (s >= ns) return 0;
    if (ca.geometry == 1) return -1;
    if (s < ca.nx) return 2;
    if (s < 2 * ca.nx) return 3;
    if (s < 2 * ca.nx + ca.ny) return 4;
    return 5;
}

// Energies per source slot (src/imc_sourcing.jl:56-111).  Slot order is the
// reference's push! order: 1D [left, right, body cells, source cells]; 2D
// [bottom x, top x, left y, right y, body cells, source cells].  Two warps for
// 32 slots, as FP64 and the sorter's chain of exchanges bound it: one the
// slots' energies, the other the body cells' emitted energy densities.  Each
// unit of 32 slots leaves double-double partial sums of e/escale per slot
// group; the block that finishes last sums those (src/imc_sourcing.jl:121).
// UPDATE: the step sequence, with Update.update of the body cells in the same
// launch (both warps compute it, the first keeps it).
constexpr int kSlotThreads = 128;
template <int G, int SEL, bool UPDATE>
__global__ void __launch_bounds__(kSlotThreads) k_source_slots(CellArgs ca, Scalars *sc) {
    __shared__ int s_last;
    const double a = ca.a, c = ca.c, ds = ca.ds, dt = sc->dt;
    const int ns = nsurf_slots(ca), nc = ca.nc, K = ca.K;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int unit = blockIdx.x * (kSlotThreads / 64) + (warp >> 1), s = unit * 32 + lane;
    const bool body = s >= ns && s < ns + nc;
    // flags of this launch: with UPDATE the step's first kernel, whose last
    // block starts the step's flags from them
    unsigned *flags = UPDATE ? ca.src_flags : &sc->flags;
    CellLaws u{};
    if (body) {
        const int i = s - ns;
        if (UPDATE) {
            if (warp & 1) u = update_cell<false>(ca, dt, i);
            else u = update_cell<true>(ca, dt, i);
        } else {
            u.T = ca.temp[i]; u.f = ca.fleck[i]; u.sa = ca.sa[i];
        }
    }
    if (warp & 1) {
        if (body) {
            // emitted energy density (src/imc_sourcing.jl:69-70)
            const int i = s - ns;
            double ve[10] = {u.f, u.sa, a, c, u.T, u.T, u.T, u.T, dt, ds};
            int je;
            const double em = sorter_n<SEL, 10>(ve, ca.scales, K, &je);
            for (int k = 0; k < K; ++k) ca.emitted[(size_t)k * nc + i] = k == je ? em : 0.0;
            if (je < 0) atomicOr(flags, 1u << 5);
        }
    } else {
        double q = 0.0;
        int grp = -2;
        if (s < ca.nslots) {
            double e = 0.0;
            int j = -1;
            if (s < ns) {
                double Ts = ca.tsurf[s], w = 0.0;
                if (G == 1) {
                    double v[8] = {a, c, Ts, Ts, Ts, Ts, dt, 0.25};
                    e = sorter_n<SEL, 8>(v, ca.scales, K, &j);
                } else {
                    if (s < 2 * ca.nx) w = ca.dx[s % ca.nx];
                    else w = ca.dy[(s - 2 * ca.nx) % ca.ny];
                    double v[9] = {a, c, Ts, Ts, Ts, Ts, w, dt, 0.25};
                    e = sorter_n<SEL, 9>(v, ca.scales, K, &j);
                }
            } else if (body) {
                const int i = s - ns;
                const int ix = G == 1 ? i : i % ca.nx;
                const int iy = G == 1 ? 0 : i / ca.nx;
                if (G == 1) {
                    double v[11] = {u.f, u.sa, a, c, u.T, u.T, u.T, u.T, ca.dx[i], dt, ds};
                    e = sorter_n<SEL, 11>(v, ca.scales, K, &j);
                } else {
                    double v[12] = {u.f, u.sa, a, c, u.T, u.T, u.T, u.T, ca.dx[ix], ca.dy[iy], dt, ds};
                    e = sorter_n<SEL, 12>(v, ca.scales, K, &j);
                }
            } else {
                const int i = s - ns - nc;
                const int ix = G == 1 ? i : i % ca.nx;
                const int iy = G == 1 ? 0 : i / ca.nx;
                if (G == 1) {
                    double v[3] = {ca.radsource[i], ca.dx[i], dt};
                    e = sorter_n<SEL, 3>(v, ca.scales, K, &j);
                } else {
                    double v[4] = {ca.radsource[i], ca.dx[ix], ca.dy[iy], dt};
                    e = sorter_n<SEL, 4>(v, ca.scales, K, &j);
                }
            }
            if (j < 0) atomicOr(flags, 1u << 5);
            const double sv = j >= 0 ? ca.scales[j] : 0.0;
            q = j >= 0 ? div_scale(e, sv) : e / sv;
            ca.slot_e[s] = e;
            ca.slot_j[s] = j;
            ca.slot_q[s] = q;
            grp = slot_group(ca, s);
        }
        for (int g = 0; g < 6; ++g) {
            // most units hold one group: reduce only the groups present
            DD r;
            r.clear();
            if (__any_sync(0xFFFFFFFFu, grp == g)) r = warp_sum(grp == g ? q : 0.0);
            if (lane == 0 && unit < ca.nblk_slot) {
                ca.part_src[(unit * 6 + g) * 2] = r.hi;
                ca.part_src[(unit * 6 + g) * 2 + 1] = r.lo;
            }
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&sc->tally_blocks_done, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    // 1D needs only the body and radiation-source groups; its two surfaces are
    // added directly
    for (int g = warp; g < (G == 1 ? 2 : 6); g += kSlotThreads / 32) {
        const double v = warp_sum_partials(ca.part_src, ca.nblk_slot, 6, g);
        if (lane == 0) sc->src_group[g] = v;
    }
    if (threadIdx.x == 0) {
        sc->tally_blocks_done = 0u;
        if (UPDATE) {
            sc->flags = *ca.src_flags;
            *ca.src_flags = 0u;
        }
    }
}

__device__ __forceinline__ long long round_count(double q, double n_source, double E, bool withmin,
                                                 double cellmin) {
    double r = rint((q * n_source) / E);
    if (withmin) r = fmax(r, cellmin);
    return (long long)r;
}

// Total energy (src/imc_sourcing.jl:121) and particle budget (:132-136) from
// the group sums, in a fixed order: every block of k_source_counts computes
// the same values.
__device__ __forceinline__ void source_total(const CellArgs &ca, const Scalars *sc, double &E, double &n_source) {
    const double *g = sc->src_group;
    double e_surface;
    if (ca.geometry == 1) {
        e_surface = ca.slot_q[0] + ca.slot_q[1];
    } else {
        e_surface = 0.0;
        e_surface += g[2];
        e_surface += g[3];
        e_surface += g[4];
        e_surface += g[5];
    }
    E = g[0] + g[1] + e_surface;
    const long long n_census = sc->n_census;
    n_source = (double)ca.n_input;
    if (ca.n_input + n_census > ca.n_max) {
        double lenN = ca.geometry == 1 ? 1.0 : 2.0;
        n_source = fmax(ca.cellmin, (double)(ca.n_max - n_census) - lenN - 1.0);
    }
}

// Births per slot (src/imc_sourcing.jl:138-157) and per-particle energy, and
// their exclusive scan: each block's births from its own start (slot_off), and
// in the block that finishes last the blocks' starts (blk_off), the capacity
// check and the fixed-point exponents; block 0 also records the step's total
// energy and budget.  One launch and no pass over the slots by a single block
// (the scan alone took 7 us for 4002 slots, 15 us for 11,560).
__global__ void __launch_bounds__(kCountThreads) k_source_counts(CellArgs ca, Scalars *sc) {
    constexpr int W = kCountThreads / 32;
    __shared__ unsigned long long s_max[W];
    __shared__ long long s_tot[W], s_run;
    __shared__ int s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int ns = nsurf_slots(ca), nc = ca.nc;
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    // everything the slot needs, asked for before the first use
    const bool slot = q < ca.nslots;
    const double eq = slot ? ca.slot_e[q] : 0.0, qq = slot ? ca.slot_q[q] : 0.0;
    const double qb = slot && ca.geometry == 2 && q >= ns + nc ? ca.slot_q[q - nc] : 0.0;
    const int jq = slot ? ca.slot_j[q] : -1;
    double E, n_source;
    source_total(ca, sc, E, n_source);
    const double scale = jq >= 0 ? ca.scales[jq] : 1.0;
    const bool ok = (E > 0.0) && isfinite(E);
    double my = 0.0;
    long long n = 0;
    if (slot) {
        long long nd = 0;
        if (ok) {
            if (q < ns) {
                if (eq > 0) n = round_count(qq, n_source, E, ca.geometry == 2, ca.cellmin);
                nd = n;
            } else if (q < ns + nc) {
                n = round_count(qq, n_source, E, true, ca.cellmin);
                nd = n;
            } else if (eq > 0) {
                n = round_count(qq, n_source, E, true, ca.cellmin);
                nd = n;
                // 2D births n_body particles per source cell (src/imc_sourcing.jl:357)
                if (ca.geometry == 2 && n > 0) n = round_count(qb, n_source, E, true, ca.cellmin);
            }
            if (n < 0) n = 0;
        }
        const double nrg = n > 0 ? eq / (double)nd : 0.0;
        ca.slot_nrg[q] = nrg;
        ca.slot_nrg_f[q] = (float)nrg;
        // the largest birth energy in true units (see scale_exp)
        if (n > 0 && nrg > 0.0) my = times_pow2(nrg, -scale_exp(scale));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->totalenergy = E;
        sc->n_source = n_source;
        if (!ok) atomicOr(&sc->flags, 1u << 4);
    }
    // the block's scan and maximum
    long long x = n;
    for (int off = 1; off < 32; off <<= 1) {
        const long long y = __shfl_up_sync(0xFFFFFFFFu, x, off);
        if (lane >= off) x += y;
    }
    unsigned long long most = warp_max_bits(my);
    if (lane == 31) s_tot[warp] = x;
    if (lane == 0) s_max[warp] = most;
    __syncthreads();
    long long before = 0, total = 0;
    for (int w = 0; w < W; ++w) {
        before += w < warp ? s_tot[w] : 0;
        total += s_tot[w];
        most = s_max[w] > most ? s_max[w] : most;
    }
    if (q < ca.nslots) ca.slot_off[q] = before + x - n;
    if (threadIdx.x == 0) {
        ca.blk_off[blockIdx.x] = total;
        ca.part_emax[blockIdx.x] = m64::from_bits(most);
    }
    const long long n_census = sc->n_census;  // live particles
    const long long len = sc->n_particles;    // list length, holes included
    const int ce = sc->emax_census_exp;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&sc->tally_blocks_done, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) s_run = 0;
    double emax = 0.0;  // (energies: not negative, ordered as their bits)
    const int nb = gridDim.x;
    for (int base = 0; base < nb; base += kCountThreads) {
        const int b = base + threadIdx.x;
        const long long v = b < nb ? ca.blk_off[b] : 0;
        if (b < nb && d2u(ca.part_emax[b]) > d2u(emax)) emax = ca.part_emax[b];
        long long y = v;
        for (int off = 1; off < 32; off <<= 1) {
            const long long o = __shfl_up_sync(0xFFFFFFFFu, y, off);
            if (lane >= off) y += o;
        }
        __syncthreads();  // s_tot and s_run as the round before left them
        if (lane == 31) s_tot[warp] = y;
        __syncthreads();
        long long start = s_run;
        for (int w = 0; w < warp; ++w) start += s_tot[w];
        if (b < nb) ca.blk_off[b] = start + y - v;
        __syncthreads();
        if (threadIdx.x == kCountThreads - 1) s_run = start + y;
    }
    most = warp_max_bits(emax);
    if (lane == 0) s_max[warp] = most;
    __syncthreads();
    if (threadIdx.x == 0) {
        sc->tally_blocks_done = 0u;
        for (int w = 0; w < W; ++w) most = s_max[w] > most ? s_max[w] : most;
        emax = m64::from_bits(most);
        long long n_new = s_run;
        unsigned fl = 0;
        if (len + n_new > ca.capacity) {
            n_new = ca.capacity - len;
            if (n_new < 0) n_new = 0;
            fl |= 1u << 3;
        }
        emax = fmax(ce == kNoExp ? 0.0 : exp_top(ce), emax);
        sc->n_census_in = n_census;
        sc->n_sourced = n_new;
        sc->birth_base = len;
        sc->n_particles = len + n_new;
        sc->emax = emax;
        sc->emax_census_exp = kNoExp;
        sc->segments = 0ull;
        sc->surrogate_calls = 0ull;
        sc->killed = 0ull;
        sc->work_next = 0ull;
        for (int r = 0; r <= 2 * kSurrRounds; ++r) sc->qcount[r] = 0ull;
        const int b = fix_exponent(emax);
        sc->b_dep = ca.vol_min == 1.0 ? b : fix_exponent(emax / ca.vol_min);
        sc->b_lost = b;
        sc->b_rad = b;
        if (fl) atomicOr(&sc->flags, fl);
    }
}

template <class T> struct RT;
template <> struct RT<float> { static __device__ float sqrt_(float x) { return sqrtf(x); } };
template <> struct RT<double> { static __device__ double sqrt_(double x) { return sqrt(x); } };

// What every birth of a slot has in common, found once per slot.
enum { kLeft1D, kRight1D, kBody1D, kBottom2D, kTop2D, kLeft2D, kRight2D, kBody2D };
template <class T> struct BirthSlot {
    int kind, cell, k;
    T E0;
    T wx, wy;      // widths that the drawn coordinates are multiplied by
    T x0, y0;      // fixed coordinates of the surface births
    T cx, cy;      // the cell's widths * DISTANCESCALE (FP16 state: the stored unit)
};
// binary32 copies of the widths for FP32 / FP16 births
template <class T> __device__ __forceinline__ T width_x(const CellArgs &ca, int i) { return sizeof(T) == 4 ? (T)ca.dxf[i] : (T)ca.dx[i]; }
template <class T> __device__ __forceinline__ T width_y(const CellArgs &ca, int i) { return sizeof(T) == 4 ? (T)ca.dyf[i] : (T)ca.dy[i]; }

template <class St>
__device__ __forceinline__ BirthSlot<typename St::T> birth_slot(const CellArgs &ca, int q) {
    typedef typename St::T T;
    const int ns = nsurf_slots(ca), nc = ca.nc, nx = ca.nx, ny = ca.ny;
    // the surface births' fixed positions, the same for every birth of a
    // face (computed on the host, CellArgs::surf_f / surf_d)
    auto surf = [&](int w) -> T { return sizeof(T) == 4 ? (T)ca.surf_f[w] : (T)ca.surf_d[w]; };
    BirthSlot<T> b;
    b.E0 = sizeof(T) == 4 ? (T)ca.slot_nrg_f[q] : (T)ca.slot_nrg[q];
    const int j = ca.slot_j[q];
    b.k = j < 0 ? 0 : j;
    b.wx = b.wy = b.x0 = b.y0 = b.cx = b.cy = (T)0;
    int ix, iy = 0;
    if (ca.geometry == 1) {
        if (q < 2) {
            b.kind = q == 0 ? kLeft1D : kRight1D;
            ix = q == 0 ? 0 : nx - 1;
            b.x0 = surf(q);
        } else {
            b.kind = kBody1D;
            ix = q < ns + nc ? q - ns : q - ns - nc;
            b.wx = width_x<T>(ca, ix);
        }
    } else if (q < ns) {
        if (q < 2 * nx) {
            const bool top = q >= nx;
            b.kind = top ? kTop2D : kBottom2D;
            ix = top ? q - nx : q;
            iy = top ? ny - 1 : 0;
            b.wx = width_x<T>(ca, ix);
            b.y0 = surf(top ? 5 : 4);
        } else {
            const bool right = q >= 2 * nx + ny;
            b.kind = right ? kRight2D : kLeft2D;
            iy = right ? q - 2 * nx - ny : q - 2 * nx;
            ix = right ? nx - 1 : 0;
            b.x0 = surf(right ? 3 : 2);
            // the reference scales y by mesh.dx[j] (src/imc_sourcing.jl:301,316)
            b.wy = iy < nx ? width_x<T>(ca, iy) : width_y<T>(ca, iy);
        }
    } else {
        const int cell = q < ns + nc ? q - ns : q - ns - nc;
        b.kind = kBody2D;
        iy = cell / nx;
        ix = cell - iy * nx;
        b.wx = width_x<T>(ca, ix);
        b.wy = width_y<T>(ca, iy);
    }
    b.cell = ix + iy * nx;
    if (St::half) {
        b.cx = width_x<T>(ca, ix) * (T)ca.ds_f;
        if (ca.geometry == 2) b.cy = width_y<T>(ca, iy) * (T)ca.ds_f;
    }
    return b;
}

template <class St>
__device__ __forceinline__ void store_birth(int geometry, PBuf<St> &pb, long long pid, typename St::T t,
                                            typename St::T x, typename St::T y, typename St::T ux,
                                            typename St::T uy, const BirthSlot<typename St::T> &b, float dtf) {
    typedef typename St::S S;
    if (St::half) {
        st_v(pb.x + pid, (float)x / (float)b.cx);
        if (geometry == 2) {
            st_v(pb.y + pid, (float)y / (float)b.cy);
            st_v(pb.uy + pid, (float)uy);
        }
        st_v(pb.t + pid, (float)t / dtf);
        st_v(pb.ux + pid, (float)ux);
        st_v(pb.E + pid, 1.0f);
        pb.E0[pid] = (float)b.E0;
    } else {
        pb.t[pid] = (S)t;
        pb.x[pid] = (S)x;
        pb.ux[pid] = (S)ux;
        if (geometry == 2) { pb.y[pid] = (S)y; pb.uy[pid] = (S)uy; }
        pb.E[pid] = (S)b.E0;
        pb.E0[pid] = (typename St::E0S)b.E0;
    }
    pb.cs[pid] = b.cell | (b.k << 24);
    pb.alive[pid] = 1;
}

// the uniforms of one birth, in the stream's order: for binary32 the words of a
// block made at once (four serve a birth but for a redraw)
template <class T> struct BirthDraws;
template <> struct BirthDraws<float> {
    Words<5> ws;
    const CellArgs &ca;
    unsigned step;
    __device__ __forceinline__ BirthDraws(const CellArgs &c, unsigned st, uint32_t pid) : ca(c), step(st) {
        ws.init_full(pid, ca.rk, step, kStageSource);
    }
    __device__ __forceinline__ uint32_t word() {
        if (ws.n == 0) ws.refill(ca.rk, step, kStageSource);
        const uint32_t w = ws.w[0];
        ws.drop(false);
        return w;
    }
    __device__ __forceinline__ float u() { return Rand<float>::u(word()); }
    __device__ __forceinline__ float cosine() { return Rand<float>::cosine(word()); }
};
template <> struct BirthDraws<double> {
    Stream rs;
    __device__ __forceinline__ BirthDraws(const CellArgs &ca, unsigned step, uint32_t pid) {
        rs.init(ca.seed, step, pid, kStageSource);
    }
    __device__ __forceinline__ double u() { return Rand<double>::u(rs); }
    __device__ __forceinline__ double cosine() { return Rand<double>::cosine(rs); }
};

// One thread per newborn particle; its stream is keyed by its list index.
// (33 B are stored for 190 instructions a warp's birth, 20 us each for the
// channel's 4e6 births; with the latency of the slot searches and the nine
// streams of stores it takes 37.  With the slot looked up and decoded for each
// birth, 250 instructions: 49.)
constexpr int kEmitThreads = 256;
template <class St, int G>
__global__ void __launch_bounds__(kEmitThreads) k_source_emit(CellArgs ca, Scalars *sc, PBufPair bufs) {
    typedef typename St::T T;
    PBuf<St> pb(bufs.b[sc->cur]);
    const long long n_new = sc->n_sourced, n_census = sc->birth_base;
    const unsigned step = sc->step;
    const T dtT = (T)sc->dt, dsT = Consts<T>::ds(ca);
    const int nslots = ca.nslots;
    const double pd = 3.141592653589793;
    // Each block takes an equal run of consecutive births, thread l the births
    // base + l + 256 i: the block writes one stretch of every array, where runs
    // of each warp wrote eight times as many at once (2D: 45 us for 4e6 births
    // against 37, 121 for 1e7 against 93; blocks of 1024: 41 and 91).  A lane finds the slot of its
    // first birth by binary search over the slot offsets (slot = last q whose
    // first birth is at or below j) and the later ones by galloping forward
    // from there (q + 1, q + 2, q + 4, ... then bisection) once the slot's
    // last birth is behind it.
    auto off = [&](int s) { return ca.slot_off[s] + ca.blk_off[s / kCountThreads]; };
    const long long per_block = (n_new + gridDim.x - 1) / gridDim.x;
    const long long run = (per_block + kEmitThreads - 1) & ~(long long)(kEmitThreads - 1);
    const long long end = min((blockIdx.x + 1) * run, n_new);
    int q = -1;
    long long next = -1;  // the first birth beyond slot q
    BirthSlot<T> b{};
    for (long long j = blockIdx.x * run + threadIdx.x; j < end; j += kEmitThreads) {
        if (next <= j) {
            int lo, hi;
            if (q < 0) {
                // the last block that starts at or below j, then its last such slot
                lo = 0;
                hi = ca.nblk_count;
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (ca.blk_off[mid] <= j) lo = mid;
                    else hi = mid;
                }
                const long long rest = j - ca.blk_off[lo];
                lo *= kCountThreads;
                hi = min(lo + kCountThreads, nslots);
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (ca.slot_off[mid] <= rest) lo = mid;
                    else hi = mid;
                }
            } else {
                int stride = 2;
                lo = q + 1;  // off(lo) <= j
                hi = q + 2;
                while (hi < nslots && off(hi) <= j) {
                    lo = hi;
                    stride <<= 1;
                    hi = q + stride;
                }
                if (hi > nslots) hi = nslots;  // off(hi) > j, or hi == nslots
                while (hi - lo > 1) {
                    const int mid = (lo + hi) >> 1;
                    if (off(mid) <= j) lo = mid;
                    else hi = mid;
                }
            }
            q = lo;
            next = q + 1 < nslots ? off(q + 1) : n_new;
            b = birth_slot<St>(ca, q);
        }
        const long long pid = n_census + j;
        BirthDraws<T> d(ca, step, (uint32_t)pid);
        if (G == 1) {
            T xpos, mu;
            if (b.kind == kBody1D) {
                // body / source births (src/imc_sourcing.jl:193-236)
                xpos = b.wx * d.u() * dsT;
                mu = d.cosine();
                for (int r1 = 1; r1 < 64 && mu == (T)0; ++r1) mu = d.cosine();
                if (mu == (T)0) mu = (T)1;
            } else {
                // surface births (src/imc_sourcing.jl:161-189)
                xpos = b.x0;
                mu = RT<T>::sqrt_(d.u());
                for (int r1 = 1; r1 < 64 && mu == (T)0; ++r1) mu = RT<T>::sqrt_(d.u());
                if (mu == (T)0) mu = (T)1;
                if (b.kind == kRight1D) mu = -mu;
            }
            const T st = dtT * d.u();
            store_birth<St>(1, pb, pid, st, xpos, (T)0, mu, (T)0, b, (float)dtT);
        } else {
            T st, xpos, ypos, ang;
            // the angles are the reference's Float64 products rounded to T
            // (binary32: pi_n24 or two_pi_u24 of the uniform's integer m,
            // the same value without FP64)
            if (b.kind == kBody2D) {
                // body / source births (src/imc_sourcing.jl:326-366)
                xpos = b.wx * d.u() * dsT;
                ypos = b.wy * d.u() * dsT;
                if constexpr (sizeof(T) == 4) ang = two_pi_u24(d.word() >> 8);
                else ang = (T)(2.0 * pd * (double)d.u());
                st = dtT * d.u();
            } else {
                // surface births (src/imc_sourcing.jl:265-323)
                st = dtT * d.u();
                const bool horizontal = b.kind == kBottom2D || b.kind == kTop2D;
                const T along = (horizontal ? b.wx : b.wy) * d.u() * dsT;
                xpos = horizontal ? along : b.x0;
                ypos = horizontal ? b.y0 : along;
                if constexpr (sizeof(T) == 4) {
                    const uint32_t m = d.word() >> 8;
                    if (b.kind == kBottom2D) ang = (T)pd * ((T)m * 0x1p-24f);
                    else if (b.kind == kTop2D) ang = -pi_n24((int)m);
                    else if (b.kind == kLeft2D) ang = pi_n24((1 << 23) - (int)m);
                    else ang = (T)(pd * (0.5 + (double)((T)m * 0x1p-24f)));
                } else {
                    const T u = d.u();
                    if (b.kind == kBottom2D) ang = (T)((T)pd * u);
                    else if (b.kind == kTop2D) ang = (T)(-pd * (double)u);
                    else if (b.kind == kLeft2D) ang = (T)(pd * (0.5 - (double)u));
                    else ang = (T)(pd * (0.5 + (double)u));
                }
            }
            T ux, uy;
            if (sizeof(T) == 4) { float s_, c_; sincosf((float)ang, &s_, &c_); ux = (T)c_; uy = (T)s_; }
            else { double s_, c_; sincos((double)ang, &s_, &c_); ux = (T)c_; uy = (T)s_; }
            store_birth<St>(2, pb, pid, st, xpos, ypos, ux, uy, b, (float)dtT);
        }
    }
}

template <bool UPDATE> static void launch_slots(const CellArgs &ca, Scalars *sc, cudaStream_t st) {
    // one instantiation per geometry and scale-selection precision, so each
    // holds only its own unrolled sorters
    auto slots = ca.geometry == 1
                     ? (ca.sel_prec == 2 ? k_source_slots<1, 2, UPDATE> : ca.sel_prec == 1 ? k_source_slots<1, 1, UPDATE> : k_source_slots<1, 0, UPDATE>)
                     : (ca.sel_prec == 2 ? k_source_slots<2, 2, UPDATE> : ca.sel_prec == 1 ? k_source_slots<2, 1, UPDATE> : k_source_slots<2, 0, UPDATE>);
    const int units = kSlotThreads / 64;
    slots<<<(ca.nblk_slot + units - 1) / units, kSlotThreads, 0, st>>>(ca, sc);
}

void launch_source(const CellArgs &ca, Scalars *sc, int prec, PBufPair buf, int grid, bool update, cudaStream_t st) {
    if (update) launch_slots<true>(ca, sc, st);
    else launch_slots<false>(ca, sc, st);
    k_source_counts<<<ca.nblk_count, kCountThreads, 0, st>>>(ca, sc);
    auto emit = ca.geometry == 1
                    ? (prec == 0 ? k_source_emit<StF64, 1> : prec == 1 ? k_source_emit<StF32, 1> : k_source_emit<StF16, 1>)
                    : (prec == 0 ? k_source_emit<StF64, 2> : prec == 1 ? k_source_emit<StF32, 2> : k_source_emit<StF16, 2>);
    emit<<<grid, kEmitThreads, 0, st>>>(ca, sc, buf);
}

// ------------------------------------------------------------- compaction
// Stable compaction in two launches: per-tile alive counts and, in the block
// that finishes last, their exclusive scan; then a per-tile block scan that
// scatters the survivors in order into the other buffer.  Whether this step
// compacts follows from the transport's kills (census carried in + births -
// removed), so the holes are known without reading the alive bytes and every
// block decides alike; a step that does not compact leaves at once.  The blocks
// stride over the tiles: one per tile of the buffer's capacity, the launches
// cost 5 us each on the 2000-cell slab's 5900 tiles with nothing to do.
constexpr int kCompactBlocksPerSM = 8;
__global__ void __launch_bounds__(kCompactThreads) k_compact_count(Scalars *sc, PBufPair bufs, long long *tile_cnt,
                                                                   long long *tile_off, long long *n_before, int force) {
    constexpr int W = kCompactThreads / 32;
    __shared__ int wt[W];
    __shared__ long long s_tot[W], s_run;
    __shared__ int s_last;
    const long long n = sc->n_particles;
    const long long live = sc->n_census_in + sc->n_sourced - (long long)sc->killed;
    if (!force && (n - live) * kDeferHoles <= n) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            sc->compact_now = 0;
            sc->n_census = live;
        }
        return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint8_t *alive = bufs.b[sc->cur].alive;
    const long long ntiles = (n + kCompactTile - 1) / kCompactTile;
    for (long long tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const long long base = tile * kCompactTile;
        int cnt = 0;
        if (base + kCompactTile <= n) {
            // a full tile: 16 alive bytes per thread in one 16-byte load (tiles
            // start at multiples of 4096 bytes, so every load is aligned)
            static_assert(kCompactTile == 16 * kCompactThreads, "one uint4 per thread");
            const uint4 v = reinterpret_cast<const uint4 *>(alive + base)[threadIdx.x];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            for (int q = 0; q < 4; ++q)
                for (int b = 0; b < 4; ++b) cnt += ((w[q] >> (8 * b)) & 0xFFu) != 0u;
        } else {
            for (int r = threadIdx.x; r < kCompactTile; r += blockDim.x) {
                long long i = base + r;
                if (i < n && alive[i]) ++cnt;
            }
        }
        cnt = __reduce_add_sync(0xFFFFFFFFu, (unsigned)cnt);
        if (lane == 0) wt[warp] = cnt;
        __syncthreads();
        if (threadIdx.x == 0) {
            long long t = 0;
            for (int w = 0; w < W; ++w) t += wt[w];
            tile_cnt[tile] = t;
        }
        __syncthreads();
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&sc->tally_blocks_done, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) s_run = 0;
    for (long long base = 0; base < ntiles; base += kCompactThreads) {
        const long long q = base + threadIdx.x;
        const long long v = q < ntiles ? tile_cnt[q] : 0;
        long long x = v;
        for (int off = 1; off < 32; off <<= 1) {
            const long long y = __shfl_up_sync(0xFFFFFFFFu, x, off);
            if (lane >= off) x += y;
        }
        __syncthreads();  // s_tot and s_run as the round before left them
        if (lane == 31) s_tot[warp] = x;
        __syncthreads();
        long long start = s_run;
        for (int w = 0; w < warp; ++w) start += s_tot[w];
        if (q < ntiles) tile_off[q] = start + x - v;
        __syncthreads();
        if (threadIdx.x == kCompactThreads - 1) s_run = start + x;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        sc->tally_blocks_done = 0u;
        sc->compact_now = 1;
        *n_before = n;
        sc->n_census = s_run;
        sc->compact_src = sc->cur;
        sc->cur ^= 1;
        sc->n_particles = s_run;
    }
}

template <class St>
__global__ void __launch_bounds__(kCompactThreads) k_compact_scatter(int geometry, const Scalars *sc,
                                                                     const long long *tile_off, PBufPair bufs,
                                                                     const long long *n_before) {
    if (!sc->compact_now) return;
    PBuf<St> src(bufs.b[sc->compact_src]), dst(bufs.b[sc->compact_src ^ 1]);
    __shared__ unsigned short src_idx[kCompactTile];
    __shared__ int wt[kCompactThreads / 32];
    __shared__ int s_tot;
    const long long n = *n_before;
    for (long long tile = blockIdx.x; tile * kCompactTile < n; tile += gridDim.x) {
    const long long base = tile * kCompactTile;
    const int tile_n = (int)((n - base) < kCompactTile ? (n - base) : kCompactTile);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // survivor list of the tile, in order: thread t owns tile positions
    // [16t, 16t + 16) and reads their alive bytes with one 16-byte load
    constexpr int kPer = kCompactTile / kCompactThreads;
    static_assert(kPer == 16, "one uint4 of alive bytes per thread");
    const int first = threadIdx.x * kPer;
    unsigned char flags[kPer];
    const uint8_t *ap = src.alive + base + first;
    if (first + kPer <= tile_n && (((uintptr_t)ap) & 15u) == 0) {
        uint4 v = *reinterpret_cast<const uint4 *>(ap);
        const unsigned w[4] = {v.x, v.y, v.z, v.w};
        for (int q = 0; q < kPer; ++q) flags[q] = (unsigned char)((w[q >> 2] >> (8 * (q & 3))) & 0xFFu);
    } else {
        for (int q = 0; q < kPer; ++q) flags[q] = first + q < tile_n ? ap[q] : 0;
    }
    int mine = 0;
    for (int q = 0; q < kPer; ++q) mine += flags[q] ? 1 : 0;
    int incl = mine;
    for (int off = 1; off < 32; off <<= 1) {
        int y = __shfl_up_sync(0xFFFFFFFFu, incl, off);
        if (lane >= off) incl += y;
    }
    if (lane == 31) wt[warp] = incl;
    __syncthreads();
    if (threadIdx.x == 0) {
        int acc = 0;
        for (int w = 0; w < kCompactThreads / 32; ++w) { int v = wt[w]; wt[w] = acc; acc += v; }
        s_tot = acc;
    }
    __syncthreads();
    int pos = wt[warp] + incl - mine;
    for (int q = 0; q < kPer; ++q)
        if (flags[q]) src_idx[pos++] = (unsigned short)(first + q);
    const int run = s_tot;
    __syncthreads();
    const int cnt = run;
    const long long out = tile_off[tile];
    // Every field of a survivor in one pass: stores coalesced, loads gathered
    // from the tile (whole sectors when most entries survive; when most are
    // holes, only the sectors that hold a survivor), all fields' loads of a
    // survivor in flight together.
    for (int j = threadIdx.x; j < cnt; j += blockDim.x) {
        const long long f = base + src_idx[j], d = out + j;
        const auto t = src.t[f], x = src.x[f], ux = src.ux[f];
        const auto E = src.E[f];
        const auto E0 = src.E0[f];
        const int cs = src.cs[f];
        if (geometry == 2) {
            const auto y = src.y[f], uy = src.uy[f];
            dst.y[d] = y;
            dst.uy[d] = uy;
        }
        dst.t[d] = t; dst.x[d] = x; dst.ux[d] = ux;
        dst.E[d] = E;
        dst.E0[d] = E0;
        dst.cs[d] = cs;
        dst.alive[d] = 1;
    }
    __syncthreads();  // the tile's shared arrays are read
    }
}

void launch_compact(const CellArgs &ca, Scalars *sc, int prec, PBufPair bufs, long long *tile_cnt,
                    long long *tile_off, long long ntiles_cap, int sms, bool force, cudaStream_t st) {
    // tile_off has ntiles_cap + 1 entries; the last holds the pre-compaction length
    long long *n_before = tile_off + ntiles_cap;
    const long long most = (long long)sms * kCompactBlocksPerSM;
    const unsigned grid = (unsigned)(ntiles_cap < most ? ntiles_cap : most);
    k_compact_count<<<grid, kCompactThreads, 0, st>>>(sc, bufs, tile_cnt, tile_off, n_before, force ? 1 : 0);
    if (prec == 0)
        k_compact_scatter<StF64><<<grid, kCompactThreads, 0, st>>>(ca.geometry, sc, tile_off, bufs, n_before);
    else if (prec == 1)
        k_compact_scatter<StF32><<<grid, kCompactThreads, 0, st>>>(ca.geometry, sc, tile_off, bufs, n_before);
    else
        k_compact_scatter<StF16><<<grid, kCompactThreads, 0, st>>>(ca.geometry, sc, tile_off, bufs, n_before);
}

void launch_compact(const CellArgs &ca, Scalars *sc, int prec, PBufRaw src, PBufRaw dst, long long *tile_cnt,
                    long long *tile_off, long long ntiles_cap, int sms, cudaStream_t st) {
    PBufPair p;
    p.b[0] = src;
    p.b[1] = dst;
    launch_compact(ca, sc, prec, p, tile_cnt, tile_off, ntiles_cap, sms, true, st);
}

// ------------------------------------------------------------------- tally
__device__ __forceinline__ double cell_vol(const CellArgs &ca, int i) {
    return ca.geometry == 1 ? ca.dx[i] : ca.dx[i % ca.nx] * ca.dy[i / ca.nx];
}

// fix_value with the power of two applied to its two halves
__device__ __forceinline__ double fix_value_fast(const long long *a, int b) {
    if (b < -960 || b > 800) return fix_value(a, b);
    uint64_t hi = (uint64_t)a[0], lo = 0;
    const uint64_t lo1 = (uint64_t)a[1] << 32, lo2 = (uint64_t)a[2];
    lo = lo1 + lo2;
    hi += (uint64_t)(a[1] >> 32) + (a[2] < 0 ? ~0ull : 0ull) + (lo < lo1 ? 1ull : 0ull);
    const double u = m64::from_bits((uint64_t)(1023 + b) << 52);
    return (double)(long long)hi * (u * 0x1p64) + (double)lo * u;
}

// Converts this transport's fixed-point tallies to FP64 mesh fields and
// clears the accumulators: energydep as Transport.MC leaves it
// (src/imc_transport.jl:198-205), and the census radiation energy density of
// src/imc_tally.jl:81-113, for cell i.
__device__ __forceinline__ void finalize_cell(const CellArgs &ca, Scalars *sc, int i) {
    const int nc = ca.nc, K = ca.K;
    const int b_dep = sc->b_dep, b_rad = sc->b_rad;
    if (i < nc) {
        const double vol = cell_vol(ca, i);
        double r = 0.0;
        for (int k = 0; k < K; ++k) {
            const size_t idx = (size_t)k * nc + i;
            const double s = ca.scales[k];
            const int se = scale_exp(s);
            long long *d = ca.dep_acc + 3 * idx;
            // FP64 histories deposit energies, FP32 ones densities
            const double dep = fix_value_fast(d, b_dep + se);
            ca.energydep[idx] = ca.prec == 0 ? dep / vol : dep;
            d[0] = d[1] = d[2] = 0;
            long long *g = ca.rad_acc + 3 * idx;
            r += fix_value_fast(g, b_rad + se) / (d2u(s) == 0x3FF0000000000000ull ? vol : vol * s);
            g[0] = g[1] = g[2] = 0;
        }
        ca.radenergydens[i] = r;
    }
}

// the escaped energy and the segment statistics, by one thread
__device__ __forceinline__ void finalize_scalars(const CellArgs &ca, Scalars *sc) {
    const int b_lost = sc->b_lost;
    double lost = 0.0;
    for (int k = 0; k < ca.K; ++k) {
        long long *d = ca.lost_acc + 3 * k;
        const double s = ca.scales[k];
        if (d[0] | d[1] | d[2]) lost += div_scale(fix_value_fast(d, b_lost + scale_exp(s)), s);
        d[0] = d[1] = d[2] = 0;
    }
    sc->lost_step = lost;
    // mean transport segments per history of this step: the next
    // transport picks its lane schedule from it
    const double hist = (double)(sc->n_census_in + sc->n_sourced);
    sc->seg_per_hist = hist > 0.0 ? (float)((double)sc->segments / hist) : 0.0f;
    sc->lostenergy += lost;
}

// Tally.tally per cell (src/imc_tally.jl:29-75); each unit of 32 cells leaves
// partial sums of the deposited energy per scale and of the radiation energy.
__device__ __forceinline__ void tally_cell(const CellArgs &ca, Scalars *sc, int i, int unit) {
    const int nc = ca.nc, K = ca.K;
    const double a = ca.a, c = ca.c, dt = sc->dt;
    const bool first = sc->t == 0.0;
    const double one[1] = {1.0};
    double vol = 0.0;
    if (i < nc) {
        vol = cell_vol(ca, i);
        if (first) {
            double T = ca.temp[i];
            double v[10] = {ca.fleck[i], ca.sa[i], a, c, T, T, T, T, dt, ca.ds};
            int j;
            ca.matenergydens[i] = sorter_n<0, 10>(v, one, 1, &j);
        }
        double inc = 0.0;
        for (int k = 0; k < K; ++k)
            inc += div_scale(ca.energydep[(size_t)k * nc + i] - ca.emitted[(size_t)k * nc + i], ca.scales[k]);
        double m = ca.matenergydens[i] + inc;
        ca.matenergydens[i] = m;
        // the fourth root as two square roots: 3/4 of a unit in the last place
        // at most, in a third of pow's instructions
        if (ca.linearized) ca.temp[i] = sqrt(sqrt(m));
        else ca.temp[i] = ca.temp[i] + inc / ca.bee[i];
    }
    const int np = K + 1;
    for (int k = 0; k <= K; ++k) {
        double x = 0.0;
        if (i < nc)
            x = k < K ? div_scale(ca.energydep[(size_t)k * nc + i] * vol, ca.scales[k]) : ca.radenergydens[i] * vol;
        const DD r = warp_sum(x);
        if ((threadIdx.x & 31) == 0) {
            ca.part_tally[(unit * np + k) * 2] = r.hi;
            ca.part_tally[(unit * np + k) * 2 + 1] = r.lo;
        }
    }
}

__global__ void __launch_bounds__(kCellThreads) k_finalize(CellArgs ca, Scalars *sc) {
    finalize_cell(ca, sc, blockIdx.x * blockDim.x + threadIdx.x);
    if (blockIdx.x == 0 && threadIdx.x == 0) finalize_scalars(ca, sc);
}

__global__ void __launch_bounds__(kCellThreads) k_tally(CellArgs ca, Scalars *sc) {
    tally_cell(ca, sc, blockIdx.x * blockDim.x + threadIdx.x, blockIdx.x);
}

void launch_finalize(const CellArgs &ca, Scalars *sc, cudaStream_t st) {
    k_finalize<<<ca.nblk_cell, kCellThreads, 0, st>>>(ca, sc);
}

void launch_tally(const CellArgs &ca, Scalars *sc, cudaStream_t st) {
    k_tally<<<ca.nblk_cell, kCellThreads, 0, st>>>(ca, sc);
}

// timestep (src/MixedPrecisionIMC.jl:181-222), FP64 on the device so a run
// can replay without host round trips.
__device__ __forceinline__ void advance_clock(const CellArgs &ca, Scalars *sc) {
    double t = sc->t, dt = sc->dt;
    const double t_end = ca.t_end;
    if (t == t_end) {
        t = t_end + dt;
    } else if (ca.timestepping == 0) {
        if (t + dt > t_end) { dt = t_end - t; t = t_end; }
        else t = t + dt;
    } else {
        if (dt < ca.dtmax) {
            dt = dt * ca.kfac;
            if (dt > ca.dtmax) dt = ca.dtmax;
        }
        if (t + dt > t_end) { dt = t_end - t; t = t_end; }
        else t = t + dt;
    }
    sc->t = t;
    sc->dt = dt;
    sc->finished = t > t_end ? 1 : 0;
    sc->step += 1u;
}

// EnergyCheck.energychecker (src/imc_energycheck.jl:19-38) from the sums of
// the tally's per-block partials (g[k]: deposited energy of scale k, g[K]:
// radiation energy), by one thread: the balance, the step's statistics, the
// learned surrogate's gate, and with STEP the clock.
__device__ void energycheck_done(const CellArgs &ca, Scalars *sc, DevStats *stats, long long stats_cap,
                                 const double *g, bool step) {
    double totdep = 0.0;
    for (int k = 0; k < ca.K; ++k) totdep += g[k];
    const double radenergy = g[ca.K];
    sc->totalenergydep = totdep;
    double err = (sc->totalenergy - totdep - (radenergy - sc->radenergyold) - sc->lostenergy) / sc->totalenergy;
    if (stats && stats_cap > 0) {
        DevStats d;
        d.t = sc->t; d.dt = sc->dt;
        d.total_energy = sc->totalenergy;
        d.energy_dep = totdep;
        d.rad_energy = radenergy;
        d.rad_energy_old = sc->radenergyold;
        d.lost_energy = sc->lostenergy;
        d.energy_error = err;
        d.n_census_in = sc->n_census_in;
        d.n_sourced = sc->n_sourced;
        d.n_census_out = sc->n_census;
        d.segments = (long long)sc->segments;
        d.surrogate_calls = (long long)sc->surrogate_calls;
        d.error_flags = sc->flags;
        d.step_index = sc->step;
        stats[sc->step % (unsigned long long)stats_cap] = d;
        if (step && ca.mirror) {
            ca.mirror->last = d;
            ca.mirror->n_particles = sc->n_particles;
        }
    }
    sc->energy_err = err;
    sc->radenergy = radenergy;
    sc->radenergyold = radenergy;
    sc->lostenergy = 0.0;
    // Learned surrogate gate for the next step.  Its extra passes (a query
    // pass and an analog resume pass after the list pass) pay only when a
    // step holds enough queries to fill the GPU about twice over; with
    // fewer, the passes' latency outweighs the collisions the queries save
    // (measured on the 256-deck ensemble).  A step that ran with the gate
    // open keeps it open only if it made ca.surr_min_calls queries.  A
    // closed gate opens again to measure when the step's histories have
    // doubled since it closed (a census still filling up) and every
    // kSurrProbe-th step.  The decision uses the step's own counts, so runs
    // stay reproducible.
    if (ca.surr_image) {
        const long long hist = sc->n_census_in + sc->n_sourced;
        if (sc->surr_gate) {
            sc->surr_gate = (long long)sc->surrogate_calls >= ca.surr_min_calls ? 1 : 0;
            if (!sc->surr_gate) sc->surr_closed_h = hist;
        } else if (hist >= 2 * sc->surr_closed_h) {
            sc->surr_gate = 1;
        }
        if ((sc->step + 1u) % kSurrProbe == 0u) sc->surr_gate = 1;
    }
    if (step) advance_clock(ca, sc);  // the step sequence: timestep in the same launch
}

// EnergyCheck.energychecker as its own launch: one warp per partial-sum
// group (K deposition scales, then the radiation energy).
__global__ void __launch_bounds__(544) k_energycheck(CellArgs ca, Scalars *sc, DevStats *stats, long long stats_cap) {
    __shared__ double g[17];
    const int warp = threadIdx.x >> 5, np = ca.K + 1;
    if (warp < np) {
        double v = warp_sum_partials(ca.part_tally, ca.nblk_cell, np, warp);
        if ((threadIdx.x & 31) == 0) g[warp] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) energycheck_done(ca, sc, stats, stats_cap, g, false);
}

// Finalize + tally per cell, then, in the block that finishes last, the
// energy check and the timestep: one launch for the step's tail.  The tally of
// cell i reads only what the finalize of cell i wrote, in the same thread, and
// nothing that the compaction between them in the reference's order changes.
// Blocks of four warps, one for each of an SM's FP64 units; each publishes its
// partial sums before taking a ticket, and the last block's warps sum a group
// each over every unit of cells.  (FP64 latency bounds it, an FP64
// instruction taking as long as 64 in FP32: 2000 cells 24 us with double-double
// trees, pow and divisions by the scales, one warp a block, against 14 to 15.)
constexpr int kTailThreads = 128;
__global__ void __launch_bounds__(kTailThreads) k_tally_check(CellArgs ca, Scalars *sc, DevStats *stats,
                                                             long long stats_cap) {
    __shared__ double g[17];
    __shared__ int s_last;
    const int warp = threadIdx.x >> 5, unit = blockIdx.x * (kTailThreads / 32) + warp;
    if (unit < ca.nblk_cell) {
        const int i = unit * 32 + (threadIdx.x & 31);
        finalize_cell(ca, sc, i);
        tally_cell(ca, sc, i, unit);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&sc->tally_blocks_done, 1u) == gridDim.x - 1u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int np = ca.K + 1;
    if (warp == 3 && (threadIdx.x & 31) == 0) finalize_scalars(ca, sc);
    for (int q = warp; q < np; q += kTailThreads / 32) {
        const double v = warp_sum_partials(ca.part_tally, ca.nblk_cell, np, q);
        if ((threadIdx.x & 31) == 0) g[q] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        sc->tally_blocks_done = 0u;
        energycheck_done(ca, sc, stats, stats_cap, g, true);
    }
}

__global__ void k_timestep(CellArgs ca, Scalars *sc) { advance_clock(ca, sc); }

void launch_timestep(const CellArgs &ca, Scalars *sc, cudaStream_t st) { k_timestep<<<1, 1, 0, st>>>(ca, sc); }

void launch_energycheck(const CellArgs &ca, Scalars *sc, DevStats *stats, long long stats_cap, cudaStream_t st) {
    k_energycheck<<<1, 32 * (ca.K + 1), 0, st>>>(ca, sc, stats, stats_cap);
}

void launch_tally_check_timestep(const CellArgs &ca, Scalars *sc, DevStats *stats, long long stats_cap,
                                 cudaStream_t st) {
    const int warps = kTailThreads / 32;
    k_tally_check<<<(ca.nblk_cell + warps - 1) / warps, kTailThreads, 0, st>>>(ca, sc, stats, stats_cap);
}

// Transport of a list that was set directly (no sourcing this step): take the
// fixed-point exponents from the census maximum.
__global__ void k_prepare_transport(CellArgs ca, Scalars *sc) {
    const int ce = sc->emax_census_exp;
    const double emax = ce == kNoExp ? 0.0 : exp_top(ce);
    sc->emax = emax;
    sc->emax_census_exp = kNoExp;
    sc->segments = 0ull;
    sc->surrogate_calls = 0ull;
    sc->killed = 0ull;
    sc->work_next = 0ull;
    for (int r = 0; r <= 2 * kSurrRounds; ++r) sc->qcount[r] = 0ull;
    sc->n_census_in = sc->n_census;
    sc->n_sourced = 0;
    sc->birth_base = sc->n_particles;
    sc->b_dep = fix_exponent(emax / ca.vol_min);
    sc->b_lost = fix_exponent(emax);
    sc->b_rad = fix_exponent(emax);
}

void launch_prepare_transport(const CellArgs &ca, Scalars *sc, cudaStream_t st) {
    k_prepare_transport<<<1, 1, 0, st>>>(ca, sc);
}

}  // namespace imc
