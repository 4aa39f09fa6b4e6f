// imc_transport.cuh -- device helpers shared by the transport kernels
// (imc_transport.cu, imc_transport_surr.cu): math overloads of the particle
// type, the segment arithmetic, the sums of a cell's deposits, exact fixed-point
// tally flushes into global or block-shared accumulators, the work split, the
// per-cell table and the end-of-kernel counter reduction.
#pragma once
#include <cstdint>
#include "imc_device.cuh"
#include "imc_internal.h"
#include "imc_state.cuh"
#include "imc_surrogate.cuh"

namespace imc {

__device__ __forceinline__ float m_abs(float x) { return fabsf(x); }
__device__ __forceinline__ double m_abs(double x) { return fabs(x); }
__device__ __forceinline__ void m_sincos(double a, double *s, double *c) { sincos(a, s, c); }

// e^x - 1 in the FP32 segment arithmetic: for |x| <= 1/16 the Taylor series
// to x^7 in Horner form with fused multiply-adds (the dropped terms are below
// 1e-13 of the result; rounding within about one ulp), else expm1f.  Segments
// of sigma_a f d below 1/16 -- every segment of the slab decks -- take the
// series.  The oracle's FP32 path evaluates the same expression.
__device__ __forceinline__ float expm1_seg(float x) {
    float p = fmaf(x, 1.0f / 5040.0f, 1.0f / 720.0f);
    p = fmaf(p, x, 1.0f / 120.0f);
    p = fmaf(p, x, 1.0f / 24.0f);
    p = fmaf(p, x, 1.0f / 6.0f);
    p = fmaf(p, x, 0.5f);
    p = fmaf(p * x, x, x);
    if (fabsf(x) > 0.0625f) p = expm1f(x);
    return p;
}

// Neumaier compensated add; all deposit terms are non-negative.
template <class T> __device__ __forceinline__ void nadd(T &s, T &c, T x) {
    T t = s + x;
    if (s >= x) c += (s - t) + x;
    else c += (x - t) + s;
    s = t;
}
// the same sums without a branch (two of them for lanes that part)
template <> __device__ __forceinline__ void nadd<float>(float &s, float &c, float x) {
    const float t = s + x;
    c += (fmaxf(s, x) - t) + fminf(s, x);
    s = t;
}
// Limb adds into global memory (64-bit integer reductions in L2) or into the
// block's private copy of the tally in shared memory.
//
// A shared-memory slot is six 32-bit words: the running sums of the three
// limb positions (w[0..2], same order as Limbs l0..l2, wrapping modulo 2^32)
// and their signed carry counts (cy[0..2]).  Each limb is added with a native
// 32-bit shared atomic; the returned old sum shows whether the add wrapped,
// and only then the carry count is bumped (a negative limb l is added as
// 2^32 + l with a carry of -1).  flush_block_tallies folds the carries into
// the next limb up.  Exact for any order of adds, like the 64-bit form, at
// the cost of a 32-bit atomic instead of a 64-bit one (which shared memory
// does not add natively).  The carry counts stay below 2^31 in magnitude
// while a block adds fewer than 2^31 limbs to one slot in one launch.
__device__ __forceinline__ void add_word_smem(unsigned *w, int *cy, long long l) {
    const unsigned u = (unsigned)l;
    const unsigned old = atomicAdd_block(w, u);
    const int c = (old + u < old ? 1 : 0) - (l < 0 ? 1 : 0);
    if (c) atomicAdd_block(cy, c);
}

// A positive FP32 value into a shared slot, without the signed three-limb
// split: its 24-bit mantissa occupies at most two adjacent 32-bit words of the
// 96-bit fixed-point value (f32_words), so at most two word adds (slot word
// 2 - j holds bits 32j..32j+31, as in add_limbs).  The same integers as
// fix_split + add_limbs<true>, so the same sums.  False (nothing added) for a
// value the general path must handle (see f32_words).  The adds and their
// carries are predicated and both sums are asked for before either is looked
// at: with a branch for each and in turn, the heat wave, which flushes in
// nearly every iteration, took 132 instead of 128 ms, the 2000-cell slab's
// transport 398 instead of 382 us.
__device__ __forceinline__ void add_words_u(unsigned addr, unsigned lo, unsigned hi) {
    asm volatile("{\n\t.reg .pred p, q, r;\n\t.reg .u32 o, n, o2, n2;\n\t"
                 "setp.ne.u32 q, %2, 0;\n\t"
                 "mov.u32 o2, 0;\n\t"
                 "atom.shared.add.u32 o, [%0], %1;\n\t"
                 "@q atom.shared.add.u32 o2, [%0 + -4], %2;\n\t"
                 "add.u32 n, o, %1;\n\t"
                 "setp.lt.u32 p, n, o;\n\t"
                 "@p red.shared.add.u32 [%0 + 12], 1;\n\t"
                 "add.u32 n2, o2, %2;\n\t"
                 "setp.lt.u32 r, n2, o2;\n\t"
                 "@r red.shared.add.u32 [%0 + 8], 1;\n\t}"
                 :: "r"(addr), "r"(lo), "r"(hi) : "memory");
}
// slot: its address in the shared window
__device__ __forceinline__ bool add_f32_smem(unsigned slot, float v, int b) {
    int j;
    uint32_t lo, hi;
    if (!f32_words(v, b, j, lo, hi)) return false;
    add_words_u(slot + 8u - 4u * (unsigned)j, lo, hi);
    return true;
}
__device__ __forceinline__ bool add_f32_smem(long long *slot, float v, int b) {
    return add_f32_smem((unsigned)__cvta_generic_to_shared(slot), v, b);
}

// the same two words into a global slot's 64-bit accumulators (one flush per
// census particle, seldom two of a warp's to one slot at once)
__device__ __forceinline__ bool add_f32_global(long long *slot, float v, int b) {
    int j;
    uint32_t lo, hi;
    if (!f32_words(v, b, j, lo, hi)) return false;
    unsigned long long *a = reinterpret_cast<unsigned long long *>(slot) + 2 - j;
    atomicAdd(a, (unsigned long long)lo);
    if (hi) atomicAdd(a - 1, (unsigned long long)hi);
    return true;
}

template <bool SMT> __device__ __forceinline__ void add_limbs(long long *a, const Limbs &L) {
    if (SMT) {
        // the pointer is known to address shared memory
        unsigned *w = reinterpret_cast<unsigned *>(a);
        int *cy = reinterpret_cast<int *>(a) + 3;
        if (L.l0) add_word_smem(w + 0, cy + 0, L.l0);
        if (L.l1) add_word_smem(w + 1, cy + 1, L.l1);
        if (L.l2) add_word_smem(w + 2, cy + 2, L.l2);
    } else {
        // Warp-aggregated: the lanes flushing to the same slot at this moment
        // add their limbs in registers (integer sums, exact in any order) and
        // one of them sends the reduction to L2.
        const unsigned active = __activemask();
        const unsigned peers = __match_any_sync(active, (unsigned long long)a);
        const int lane = threadIdx.x & 31;
        long long s0 = L.l0, s1 = L.l1, s2 = L.l2;
        if (peers != (1u << lane)) {
            const int rank = __popc(peers & ((1u << lane) - 1u));
            const int n = __popc(peers);
            for (int off = 1; off < n; off <<= 1) {
                const int pr = rank + off;
                const int src = pr < n ? (int)__fns(peers, 0u, pr + 1) : lane;
                const long long o0 = __shfl_sync(peers, s0, src);
                const long long o1 = __shfl_sync(peers, s1, src);
                const long long o2 = __shfl_sync(peers, s2, src);
                if ((rank & (2 * off - 1)) == 0 && pr < n) { s0 += o0; s1 += o1; s2 += o2; }
            }
            if (rank != 0) return;
        }
        if (s0) atomicAdd((unsigned long long *)(a + 0), (unsigned long long)s0);
        if (s1) atomicAdd((unsigned long long *)(a + 1), (unsigned long long)s1);
        if (s2) atomicAdd((unsigned long long *)(a + 2), (unsigned long long)s2);
    }
}

// bytes of the per-cell transport table at the start of dynamic shared memory
// (1D: one 32-byte Tab1 per cell for either type)
__host__ __device__ __forceinline__ int table_bytes(const CellArgs &ca, int tsz) {
    // 1D: 32-byte Tab1 rows; 2D: 16-byte Tab2 rows, then x and y Face rows
    int b = ca.geometry == 1 ? 32 * ca.nx : 16 * ca.nc + 2 * tsz * (ca.nx + ca.ny);
    return (b + 15) & ~15;
}
__host__ __device__ __forceinline__ int table_bytes(const Deck1DArgs &ca, int) { return (32 * ca.nx + 15) & ~15; }

__device__ __forceinline__ long long *tally_smem(unsigned char *smem, int table) {
    return reinterpret_cast<long long *>(smem + table);
}

// Adds the block's shared tallies (deposition, then census energy, in the
// same 3-limb layout as the global accumulators) to the global ones: limb
// q of a slot gets its word sum plus the carries out of the limb below it.
// with_rad false: the block holds only the deposition tallies.
template <class CA>
__device__ __forceinline__ void flush_block_tallies(const CA &ca, const long long *sm, bool with_rad) {
    __syncthreads();
    const int n = ca.K * ca.nc;
    for (int i = threadIdx.x; i < (with_rad ? 2 * n : n); i += blockDim.x) {
        const unsigned *w = reinterpret_cast<const unsigned *>(sm + 3 * (size_t)i);
        const int *cy = reinterpret_cast<const int *>(w + 3);
        long long *g = (i < n ? ca.dep_acc : ca.rad_acc) + 3 * (size_t)(i < n ? i : i - n);
        const long long v0 = (long long)w[0] + (long long)cy[1] + (long long)cy[0] * 4294967296ll;
        const long long v1 = (long long)w[1] + (long long)cy[2];
        const long long v2 = (long long)w[2];
        if (v0) atomicAdd((unsigned long long *)(g + 0), (unsigned long long)v0);
        if (v1) atomicAdd((unsigned long long *)(g + 1), (unsigned long long)v1);
        if (v2) atomicAdd((unsigned long long *)(g + 2), (unsigned long long)v2);
    }
}

// a value that add_f32_smem did not take: its exact conversion and adds in the
// general form
template <class T, bool SMT>
__device__ __forceinline__ void flush_rest(long long *acc, int slot, T v, int b, unsigned &flags) {
    if (v == (T)0) return;
    Limbs A;
    if (!fix_split(v, b, A)) {
        flags |= (v != v) ? 1u /*NAN*/ : (1u << 5) /*FIXPOINT_RANGE*/;
        return;
    }
    add_limbs<SMT>(acc + 3 * (size_t)slot, A);
}

// The deposits of the cell a history is in: a compensated pair of binary32
// densities, or an exact sum of energies (FP64).
template <class T> struct CellSum;
template <> struct CellSum<float> {
    float s, c;
    __device__ __forceinline__ void clear() { s = 0.0f; c = 0.0f; }
    __device__ __forceinline__ void add(float x) { nadd(s, c, x); }
};
template <> struct CellSum<double> {
    m64::Sum128 v;
    __device__ __forceinline__ void clear() { v.clear(); }
    // dead: all of E, else E's share -em1; b: the tally's exponent
    __device__ __forceinline__ void add(double E, double em1, bool dead, int b, unsigned &flags) {
        const bool ok = dead ? v.add(E, b) : v.add_minus_product(E, em1, b);
        if (!ok) flags |= (E != E || em1 != em1) ? 1u /*NAN*/ : (1u << 5) /*FIXPOINT_RANGE*/;
    }
    template <bool SMT> __device__ __forceinline__ void flush(long long *acc, int slot, unsigned &flags) const {
        if ((v.lo | (uint64_t)v.hi) == 0) return;
        bool neg;
        uint64_t l, h;
        if (!v.magnitude(neg, l, h)) {
            flags |= 1u << 5;  // FIXPOINT_RANGE
            return;
        }
        Limbs A;
        A.l2 = (long long)(l & 0xFFFFFFFFull);
        A.l1 = (long long)(l >> 32);
        A.l0 = (long long)h;
        if (neg) { A.l0 = -A.l0; A.l1 = -A.l1; A.l2 = -A.l2; }
        add_limbs<SMT>(acc + 3 * (size_t)slot, A);
    }
};

template <class T, bool SMT>
__device__ __forceinline__ void flush_one(long long *acc, int slot, T v, int b, unsigned &flags) {
    if constexpr (SMT && sizeof(T) == 4)
        if (add_f32_smem(acc + 3 * (size_t)slot, v, b)) return;
    flush_rest<T, SMT>(acc, slot, v, b, flags);
}

// flush a compensated pair: the Neumaier result s + c, converted once
template <class T, bool SMT>
__device__ __forceinline__ void flush_pair(long long *acc, int slot, T s, T c, int b, unsigned &flags) {
    flush_one<T, SMT>(acc, slot, s + c, b, flags);
}

// Work split of the transport over the particle list (or a resume pass's
// queue): warps take chunks in order from a counter (Scalars::work_next,
// zeroed before each transport and by each query pass) -- kListChunk1D- or
// kListChunk-entry chunks in the short-history schedule of the 1D and 2D
// kernels, 32-entry chunks in the refill schedule -- so the blocks (one per
// SM) run out of work together.  Measured against a fixed grid stride over 7/8
// of the list with the rest from the counter: the same on the slab (+0.7 %),
// 29 % faster transport on the 2D channel, whose history costs vary along the
// list.  256-entry chunks: 1.7 % faster 1D transport on the slab than 128,
// 2-4 % slower 2D transport on the channel.
constexpr int kListChunk = 128;
constexpr int kListChunk1D = 256;
// A short list is cut finer, so that every warp of the grid takes about four
// chunks (at least one 32-entry chunk): 1e5 FP64 histories are 390 chunks of
// 256, which left 134 of 152 SMs without work.
__device__ __forceinline__ int list_chunk(long long n, int most) {
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    const long long per = (n / (4 * warps)) & ~31ll;
    return per >= most ? most : per < 32 ? 32 : (int)per;
}
// the counter's next value for the warp (warp-uniform; every lane calls)
__device__ __forceinline__ long long warp_counter_next(unsigned long long *counter) {
    unsigned long long c = 0;
    if ((threadIdx.x & 31) == 0) c = atomicAdd(counter, 1ull);
    return (long long)__shfl_sync(0xFFFFFFFFu, c, 0);
}

// where the transport kernels add their tallies
enum { kTallyGlobal = 0, kTallyShared = 1, kTallySharedDep = 2 };

// threads per block of the shared-tally transport kernels: FP32 / FP16 state
// and FP64 state (one block per SM: the table and the private tallies take
// most of the shared memory)
constexpr int kSmtBlock32 = 1024;
constexpr int kSmtBlock64 = 512;
// threads per block of the global-tally kernels (meshes whose private
// tallies do not fit): FP32 / FP16 state as one 1024-thread block per SM,
// FP64 in 256-thread blocks
constexpr int kGlbBlock32 = 1024;
// the 1D long-history kernels of FP32 / FP16 state: 80 registers a thread keep
// the history and its random words out of local memory, and the schedule loses
// nothing by eight warps less (heat wave 163 -> 162 ms, thick slab 51.9 -> 50.3
// ms at 768 against 1024 threads; the short-history kernel 402 -> 452 us)
constexpr int kLongBlock32 = 768;
constexpr int kGlbBlock64 = 256;

// 1D per-cell table: sigma_a f, effective scatter, width * distancescale;
// the FP32 table adds the width and the reciprocals its arithmetic multiplies
// by, the FP64 table 1/seff (its deposits are energies, not densities, so it
// needs no width)
template <class T> struct Tab1;
template <> struct Tab1<double> { double saf, seff, rseff, dxs; };
template <> struct Tab1<float> { float saf, seff, dxs, dxT, rseff, rdxT, pad0, pad1; };
static_assert(sizeof(Tab1<double>) == 32 && sizeof(Tab1<float>) == 32, "32-byte table rows");

// The rows are written once per step with the cells' update (store_tab) and copied to
// shared memory by every transport block (load_tab): built by each block,
// they cost every SM the FP64 conversions and divisions of all cells.
template <class T>
__device__ __forceinline__ Tab1<T> make_tab1(double sa, double f, double ss, double dx, T ds) {
    Tab1<T> e;
    const T saT = (T)sa, fT = (T)f, ssT = (T)ss;
    e.saf = saT * fT;
    e.seff = saT * ((T)1 - fT) + ssT;
    e.dxs = (T)dx * ds;
    if constexpr (sizeof(T) == 8) {
        e.rseff = 1.0 / e.seff;
    } else {
        e.dxT = (T)dx;
        e.rseff = 1.0f / e.seff;  // inf for a zero opacity: the flight is then inf, as seff/0 is
        e.rdxT = 1.0f / e.dxT;
        e.pad0 = e.pad1 = 0.0f;
    }
    return e;
}

// Segment arithmetic of Transport.MC (src/imc_transport.jl:84-123).  FP32
// (and FP16 state) evaluates the collision distance as -log(v) * (1/seff)
// with the hardware logarithm, the weight after the segment as E + E
// expm1(-sigma_a f d) -- one transcendental for both the attenuation and the
// deposit, so the two add up to E up to one rounding -- and reciprocals
// instead of divisions.  FP64 evaluates the same quantities from the functions
// of imc_math64.cuh.  The FP64 pipe bounds it (an FP64 instruction takes as
// long as 64 in FP32), so a segment holds as few of them as its
// accuracy allows: logarithm and exponential in 64-bit integers, the deposits
// of a cell summed as energies and divided by the cell's volume once, when the
// tally is finalised, and comparisons on the bits.  2000-cell slab at 2e6
// histories: 1.24 ms per launch with CUDA's exp, expm1 and log, five divisions
// and FP64 compares; 0.55 with table-driven FP64 functions and corrected
// products; 0.35 with the functions in integers.  The weight after the segment
// is E + E (exp(-y) - 1) while that cancels nothing and E exp(-y) from y = ln 2
// on (m64::attenuate).
template <class T> struct SegMath;
template <> struct SegMath<double> {
    // inf for a zero opacity (rseff inf), as el / 0 is
    static __device__ __forceinline__ double flight(Stream &rs, double seff, double rseff) {
        const double el = Rand<double>::exp1(rs), q = el * rseff;
        const double d = fma(fma(-q, seff, el), rseff, q);
        // opacities of zero, infinity, beyond 2^1022 or below 0: the division
        return m64::hi32(rseff) - 0x00100000u < 0x7FE00000u - 0x00100000u ? d : el / seff;
    }
    static __device__ __forceinline__ double flight(Stream &rs, const Tab1<double> &ce) {
        return flight(rs, ce.seff, ce.rseff);
    }
    // new weight; *em1 = minus the share of it deposited
    static __device__ __forceinline__ double attenuate(double E, double saf, double d, double *em1) {
        return m64::attenuate(E, saf * d, em1);
    }
};
// the least of three, NaN if one is NaN (jmin of jmin; one instruction)
__device__ __forceinline__ float min3_nan(float a, float b, float c) {
    float r;
    asm("min.NaN.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
// c, DISTANCESCALE and 1 / (DISTANCESCALE c) in the arithmetic type
template <class T> struct Consts;
template <> struct Consts<float> {
    template <class CA> static __device__ __forceinline__ float c(const CA &ca) { return ca.c_f; }
    template <class CA> static __device__ __forceinline__ float ds(const CA &ca) { return ca.ds_f; }
    template <class CA> static __device__ __forceinline__ float rdsc(const CA &ca) { return ca.rdsc_f; }
};
template <> struct Consts<double> {
    template <class CA> static __device__ __forceinline__ double c(const CA &ca) { return ca.c; }
    template <class CA> static __device__ __forceinline__ double ds(const CA &ca) { return ca.ds; }
    template <class CA> static __device__ __forceinline__ double rdsc(const CA &) { return 0.0; }  // divides
};
// the round keys of a launch's seed
__device__ __forceinline__ const RoundKeys &round_keys(const CellArgs &ca) { return ca.rk; }
__device__ __forceinline__ SeedKeys round_keys(const Deck1DArgs &ca) { return SeedKeys(ca.seed); }

// The shortest of the distances of an FP64 segment, and which of them it is
// (ties give every one): bit comparisons when all are in [+0, inf], else
// (odd) the reference's NaN-propagating minimum.
__device__ __forceinline__ bool plain64(double v) { return m64::hi32(v) <= 0x7FF00000u; }
__device__ __forceinline__ double min64(double a, double b) {
    const uint64_t x = m64::bits(a), y = m64::bits(b);
    return m64::from_bits(x < y ? x : y);
}
// v > 0 for v not NaN, without the FP64 pipe
__device__ __forceinline__ bool pos64(double v) { return (long long)m64::bits(v) > 0; }
// a <= b: the bits ordered for two numbers of [+0, inf], else (energies below 0,
// born where a cell emits them, and NaN) the comparison itself
__device__ __forceinline__ bool le64(double a, double b) {
    return plain64(a) && plain64(b) ? m64::bits(a) <= m64::bits(b) : a <= b;
}
template <> struct SegMath<float> {
    static __device__ __forceinline__ float flight(uint32_t w, float rseff) {
        const float v = (float)((w >> 8) | 1u) * 0x1p-24f;
        return -log_fast(v) * rseff;
    }
    static __device__ __forceinline__ float flight(uint32_t w, const Tab1<float> &ce) {
        return flight(w, ce.rseff);
    }
    static __device__ __forceinline__ float attenuate(float E, const Tab1<float> &ce, float d, float *dep) {
        const float em1 = expm1_seg(-ce.saf * d);
        *dep = -(E * ce.rdxT) * em1;
        return E + E * em1;
    }
    static __device__ __forceinline__ float all_in(float E, const Tab1<float> &ce) { return E * ce.rdxT; }
};
// 2D per-cell table: sigma_a f, effective scatter; FP32 adds 1/seff and the
// reciprocal cell area
template <class T> struct Tab2;
template <> struct Tab2<double> { double saf, seff; };
template <> struct Tab2<float> { float saf, seff, rseff, rarea; };
static_assert(sizeof(Tab2<double>) == 16 && sizeof(Tab2<float>) == 16, "16-byte table rows");
template <class T> struct Face { T ws, wT; };  // width * distancescale, width
template <class T>
__device__ __forceinline__ Tab2<T> make_tab2(double sa_, double f_, double ss_, double dx, double dy) {
    const T sa = (T)sa_, f = (T)f_, ss = (T)ss_;
    Tab2<T> e;
    e.saf = sa * f;
    e.seff = sa * ((T)1 - f) + ss;
    if constexpr (sizeof(T) == 4) {
        e.rseff = 1.0f / e.seff;
        e.rarea = 1.0f / ((float)dx * (float)dy);
    }
    return e;
}
// row i of the table in global memory
template <class T>
__device__ __forceinline__ void store_tab(const CellArgs &ca, int i, double sa, double f, double ss) {
    if (ca.geometry == 1) {
        static_cast<Tab1<T> *>(ca.tab)[i] = make_tab1<T>(sa, f, ss, ca.dx[i], (T)ca.ds);
    } else {
        const Tab2<T> e = make_tab2<T>(sa, f, ss, ca.dx[i % ca.nx], ca.dy[i / ca.nx]);
        static_cast<Tab2<T> *>(ca.tab)[i] = e;
        if constexpr (sizeof(T) == 8) ca.tab_rs[i] = 1.0 / e.seff;
    }
}
// `rows` table rows of R from global memory into shared memory
template <class R> __device__ __forceinline__ void load_tab(R *dst, const void *src, int rows) {
    const uint4 *s = static_cast<const uint4 *>(src);
    uint4 *d = reinterpret_cast<uint4 *>(dst);
    for (int v = threadIdx.x; v < rows * (int)(sizeof(R) / 16); v += blockDim.x) d[v] = s[v];
}

// end-of-kernel reduction of per-thread counters: one atomic per warp
// (segments, histories removed from the list, error flags, and the census
// maximum as the exponent of its true energy, see scale_exp)
__device__ __forceinline__ void finish_counters(Scalars *sc, unsigned long long segs, unsigned long long killed,
                                                unsigned flags, int emax_e) {
    const unsigned full = 0xFFFFFFFFu;
    for (int off = 16; off > 0; off >>= 1) {
        segs += __shfl_down_sync(full, segs, off);
        killed += __shfl_down_sync(full, killed, off);
        flags |= __shfl_down_sync(full, flags, off);
        const int o = __shfl_down_sync(full, emax_e, off);
        emax_e = o > emax_e ? o : emax_e;
    }
    if ((threadIdx.x & 31) == 0) {
        if (segs) atomicAdd(&sc->segments, segs);
        if (killed) atomicAdd(&sc->killed, killed);
        if (flags) atomicOr(&sc->flags, flags);
        if (emax_e != kNoExp) atomicMax(&sc->emax_census_exp, emax_e);
    }
}

// the exponents scale_exp(scale_k) of the deck's energy scales, in shared
// memory (every thread calls; a barrier must follow before use)
template <class CA> __device__ __forceinline__ void load_scale_exps(const CA &ca, int *s_sexp) {
    for (int i = threadIdx.x; i < ca.K; i += blockDim.x) s_sexp[i] = scale_exp(ca.scales[i]);
}

// ------------------------------------------------ learned surrogate: when to ask
// The walk's state in mean free paths, for the network (imc_surrogate.cuh).
struct Query {
    float W, dn, df, mup, L;
    bool near_left;  // the nearer face is the left one
    bool cut;        // the 1 % energy cut-off ends the walk at L (truncation = kill)
    bool census;     // census ends the walk at L
};

enum { kAnalog = 0, kAsk = 1, kCertainKill = 2 };

// Whether a history at (x, mu, t, E) in a cell should walk analog, ask the
// network, or die here for certain (no face within reach before the cut-off).
template <class T>
__device__ __forceinline__ int surr_decide(const Tab1<T> &ce, T x, T mu, T t, T E, T minenergy, T c, T ds, T dt,
                                           Query &q) {
    using namespace surr;
    const float seff = (float)ce.seff;
    const float W = (float)ce.dxs * seff;
    if (!(W >= kCellMin)) return kAnalog;
    const float lcen = seff * (float)(c * (dt - t) * ds);
    const float lcut = ce.saf > (T)0 ? logf((float)E / (float)minenergy) * seff / (float)ce.saf : INFINITY;
    const float L = fminf(lcen, lcut);
    if (!(L >= kLmaxMin)) return kAnalog;
    const float xm = (float)x * seff;
    q.W = W;
    q.near_left = xm <= 0.5f * W;
    q.dn = fmaxf(q.near_left ? xm : W - xm, 0.0f);
    q.df = W - q.dn;
    q.mup = q.near_left ? (float)mu : -(float)mu;
    q.cut = lcut <= lcen && lcut <= kLmaxMax;
    q.census = !q.cut && lcen <= kLmaxMax;
    q.L = fminf(L, kLmaxMax);
    if (q.cut && q.dn >= q.L) return kCertainKill;
    return expected_collisions(q.dn, q.df, q.L) >= kMinGain ? kAsk : kAnalog;
}

// Per-cell gate of the analog passes: the least distance from the nearer
// face, in mean free paths, at which a history of this cell can want a query
// this step (infinity where none can: cell narrower than kCellMin mean free
// paths, or lmax below kMinGain even at the step's start with full energy).
// With lmax at most Lc = min(census path seff c dt ds, cut-off path
// ln(100) seff / (sigma_a f)), asking needs 1.95 d_n sqrt(Lc) >= kMinGain,
// so histories nearer the face than kMinGain / (1.95 sqrt(Lc)) skip the test.
template <class T>
__device__ __forceinline__ void fill_gate(const CellArgs &ca, float *gate, T ds, T c, T dt) {
    using namespace surr;
    for (int i = threadIdx.x; i < ca.nx; i += blockDim.x) {
        const float sa = (float)ca.sa[i], f = (float)ca.fleck[i], ss = (float)ca.ss[i];
        const float saf = sa * f, seff = sa * (1.0f - f) + ss;
        const float W = (float)ca.dx[i] * (float)ds * seff;
        const float lcen = seff * (float)(c * dt * ds);
        const float lcut = saf > 0.0f ? 4.6051702f * seff / saf : INFINITY;
        const float Lc = fminf(lcen, lcut);
        gate[i] = (W >= kCellMin && Lc >= kMinGain) ? kMinGain / (1.95f * sqrtf(Lc)) : INFINITY;
    }
}

// whether this thread's share of the filled gate holds an open cell
__device__ __forceinline__ bool gate_open(const CellArgs &ca, const float *gate) {
    bool open = false;
    for (int i = threadIdx.x; i < ca.nx; i += blockDim.x) open |= gate[i] < INFINITY;
    return open;
}

// shared-memory bytes of the 1D analog kernel: table, private tallies (SMT),
// and the per-cell gate when histories may be set aside for queries
template <class CA>
__host__ __device__ __forceinline__ int analog1d_smem(const CA &ca, int tsz, bool smt, bool gate) {
    return table_bytes(ca, tsz) + (smt ? 48 * ca.K * ca.nc : 0) + (gate ? ((4 * ca.nx + 15) & ~15) : 0);
}

}  // namespace imc
