// imc_transport.cu -- history-based particle transport, one thread per history.
//
//   k_transport1d        <- Transport.MC   (src/imc_transport.jl:13-210)
//   k_transport1d_multi     the same over many decks' lists in one launch
//   k_transport2d        <- Transport.MC2D (src/imc_transport.jl:483-732)
//
// One kernel for lists of short histories (a warp walks 32 consecutive entries
// at a time), one for long ones (lanes refill from the list as their histories
// end); both are launched and the one that the last step's histories do not call
// for returns at once, as each holds only its own schedule's registers.  FP64 2D
// has both in one kernel.
//
// A persistent grid, no larger than the list has warps' worth of entries,
// walks the particle list in chunks of consecutive entries that warps take from
// a counter, so every warp loads 32 consecutive particles (coalesced
// structure-of-arrays loads) and the blocks run out of work together; a history
// stays in registers: each particle's state is read once and written once per
// step.  Every block copies the step's per-cell transport table (sigma_a f,
// effective scatter opacity, its reciprocal, widths) to shared memory.
//
// Tallies: a history accumulates its deposits for the cell it is in as a
// Neumaier-compensated pair (FP32) or a 128-bit fixed-point sum (FP64), and
// flushes it when it leaves the cell or ends, as exact fixed-point limbs (imc_device.cuh) with
// 64-bit integer atomics.  Census energy and escaped energy are tallied the
// same way.  All tallies are therefore independent of scheduling.
//
// The event logic restates the reference line by line: distances to the face,
// to collision (randexp over the effective scatter opacity) and to census; the
// minimum wins; events are tested by float equality in the reference's
// if/if/if order, so ties run every matching branch, as they do there.
#include <cstdint>
#include "imc_transport.cuh"

namespace imc {

// segments per history at and above which lanes refill.  Measured with both
// schedules in one kernel: the refill made the heat wave (12 segments) 15 %
// faster and the slab (1.5) 22 % slower, the channel (2.4) 30 %.
constexpr float kRefillSegments = 3.0f;

// 1D analog kernel modes: the plain transport, and the passes of the
// surrogate transport (imc_transport_surr.cu) -- the list pass and the resume
// passes set aside histories that want a network query; the last resume
// pass walks everything to its end.
enum { kModePlain = 0, kModeList = 1, kModeResume = 2, kModeResumeLast = 3 };

// The transport of one deck's list by one block (every thread calls; the
// block's dynamic shared memory at smem_raw).  TM: where the flushes go
// (kTallyGlobal, kTallyShared, or kTallySharedDep: deposition tallies shared,
// census tallies global; the plain pass only).  The block's shared tallies
// and counters are flushed to the deck's before it returns; the caller puts a
// barrier between two calls.  chunk: list entries a warp takes at a time in the
// short-history schedule (0: by the list's length, list_chunk).
template <class St, int BLOCK, int TM, int MODE, bool LONG, class CA, class BP>
__device__ __forceinline__ void transport1d_block(const CA &ca, Scalars *sc, const BP &bufs, const SurrWave &w,
                                                  int round, unsigned char *smem_raw, int chunk) {
    constexpr bool SMT = TM != kTallyGlobal;      // deposition flushes to shared memory
    constexpr bool RAD_SMT = TM == kTallyShared;  // census flushes to shared memory
    typedef typename St::T T;
    typedef SegMath<T> M;
    constexpr bool kFromQueue = MODE == kModeResume || MODE == kModeResumeLast;
    constexpr bool kPause = MODE == kModeList || MODE == kModeResume;
    const long long n = kFromQueue ? (long long)sc->qcount[2 * round + 1] : sc->n_particles;
    if (kFromQueue && n == 0) return;
    if (chunk == 0) chunk = list_chunk(n, kListChunk1D);
    PBuf<St> pb(bufs.b[sc->cur]);
    Tab1<T> *tab = reinterpret_cast<Tab1<T> *>(smem_raw);
    const int N = ca.nx;
    const T ds = Consts<T>::ds(ca), c = Consts<T>::c(ca);
    const bool ds_one = ds == (T)1, c_one = c == (T)1;
    const T rdsc = Consts<T>::rdsc(ca);
    const T rds = sizeof(T) == 8 ? (T)1 / ds : (T)0, rc = sizeof(T) == 8 ? (T)1 / c : (T)0;
    long long *dep_acc = ca.dep_acc, *rad_acc = ca.rad_acc;
    if (SMT) {
        dep_acc = tally_smem(smem_raw, table_bytes(ca, sizeof(T)));
        if (RAD_SMT) rad_acc = dep_acc + 3 * (size_t)ca.K * ca.nc;
        for (int i = threadIdx.x; i < (RAD_SMT ? 6 : 3) * ca.K * ca.nc; i += blockDim.x) dep_acc[i] = 0;
    }
    static_assert(TM != kTallySharedDep || MODE == kModePlain, "deposition-only tallies: plain pass only");
    const T endsteptime = (T)sc->dt;
    float *gate = reinterpret_cast<float *>(smem_raw + analog1d_smem(ca, sizeof(T), RAD_SMT, false));
    load_tab(tab, ca.tab, N);
    __shared__ int s_sexp[16];
    load_scale_exps(ca, s_sexp);
    if constexpr (kPause) fill_gate<T>(ca, gate, ds, c, endsteptime);
    // the barrier after the table; with the gate, also whether any cell's
    // gate is open this step (each thread tests the entries it filled; every
    // block fills the whole gate, so all blocks agree): if none is, no
    // history is tested
    bool gating = false;
    if constexpr (kPause) gating = __syncthreads_or(gate_open(ca, gate)) && sc->surr_gate != 0;
    else __syncthreads();
    const int b_dep = sc->b_dep, b_rad = sc->b_rad, b_lost = sc->b_lost;
    const unsigned step = sc->step;
    const unsigned long long seed = ca.seed;
    // segments are counted in 32 bits: a cap beyond them is out of any
    // launch's reach
    const unsigned cap = ca.seg_cap > 0xFFFFFFFEll ? 0xFFFFFFFEu : (unsigned)ca.seg_cap;
    const int nc = ca.nc;
    const bool reflect_r = ca.bc[1] == 1, reflect_l = ca.bc[0] == 1;
    unsigned long long *ask_count = &sc->qcount[kFromQueue ? 2 * round + 2 : 0];
    const uint32_t stage = kFromQueue ? kStageResume + (uint32_t)round : kStageTransport;
    unsigned long long segs = 0, calls = 0, killed = 0;
    unsigned flags = 0;
    int emax_e = kNoExp;
    // Lane state of the history in flight (cs: as stored in the list; the
    // current cell and scale are cell, k).  Deposits go to the sum of the
    // current cell, flushed when it is left.
    long long i = 0;
    int cs = 0, cell = 0, k = 0, se = 0;  // se: scale k's exponent
    // shared tallies: scale k's deposition slots, and from there to its census slots
    const unsigned dep_shared = SMT ? (unsigned)__cvta_generic_to_shared(dep_acc) : 0u;
    unsigned slots_k = 0;
    T t = (T)0, x = (T)0, mu = (T)0, E = (T)0, E0 = (T)0, minenergy = (T)0, rmu = (T)0;
    CellSum<T> dep_sum;
    unsigned seg = 0;
    Stream rs;  // FP64
    Words<LONG ? 7 : 5> ws;  // FP32
    int need = 2;            // words a segment starts with: 2, or 2 and 4 in turn for the whole warp
    auto start = [&](int cs_now) {
        cell = cs_now & 0xFFFFFF;
        k = cs_now >> 24;
        se = s_sexp[k];
        if constexpr (SMT) slots_k = dep_shared + 24u * (unsigned)(k * nc);
        if constexpr (sizeof(T) == 8) rs.init(seed, step, (uint32_t)i, stage);
        else if constexpr (LONG) ws.init((uint32_t)i);
        else ws.init_full((uint32_t)i, round_keys(ca), step, stage);
        minenergy = cutoff_energy(E0);  // (T)(0.01 * (double)E0), without FP64 in binary32
        dep_sum.clear();
        seg = 0;
        rmu = rcp_any(mu);  // the face distance as a product (reset at each new direction)
    };
    // one entry of the list (or of the resume queue): false if it holds no history
    auto load = [&](long long e, int &cs_now, T &lt, T &lx, T &lmu, T &lE, T &lE0, long long &li, int &lcs) -> bool {
        if (kFromQueue) {
            li = w.resume.idx[e];
            lcs = w.resume.cs_list[e];
            cs_now = w.resume.cs[e];
            lt = (T)w.resume.t[e]; lx = (T)w.resume.x[e]; lmu = (T)w.resume.mu[e];
            lE = (T)w.resume.E[e]; lE0 = (T)w.resume.E0[e];
            return true;
        }
        if (!pb.alive[e]) return false;
        li = e;
        lcs = cs_now = pb.cs[e];
        lE0 = (T)pb.E0[e];
        if (St::half) {
            lt = ld_f(pb.t + e) * (float)endsteptime;
            lx = ld_f(pb.x + e) * (float)tab[cs_now & 0xFFFFFF].dxs;
            lmu = ld_f(pb.ux + e);
            lE = ld_f(pb.E + e) * (float)lE0;
        } else {
            lt = (T)pb.t[e]; lx = (T)pb.x[e]; lmu = (T)pb.ux[e]; lE = (T)pb.E[e];
        }
        return true;
    };
    // the deposits of the cell the history leaves, or ends in
    auto flush_cell = [&]() {
        if constexpr (sizeof(T) == 4) {
            const T v = dep_sum.s + dep_sum.c;
            if constexpr (SMT)
                if (add_f32_smem(slots_k + 24u * (unsigned)cell, v, b_dep + se)) return;
            flush_rest<T, SMT>(dep_acc, k * nc + cell, v, b_dep + se, flags);
        } else {
            dep_sum.template flush<SMT>(dep_acc, k * nc + cell, flags);
        }
    };
    // one pass of the reference's while loop; 0 = go on, 1 = killed, 2 =
    // census, 3 = set aside for a query (kPause), 4 = escaped through a
    // vacuum face.  The census write and the escape tally are left to
    // finish(), which the warp runs converged once per history.
    auto segment = [&]() -> int {
        if (gating && (float)(x < tab[cell].dxs - x ? x : tab[cell].dxs - x) * (float)tab[cell].seff >= gate[cell]) {
            Query q;
            const int kind = surr_decide<T>(tab[cell], x, mu, t, E, minenergy, c, ds, endsteptime, q);
            if (kind == kCertainKill) {
                if constexpr (sizeof(T) == 4) dep_sum.add(M::all_in(E, tab[cell]));
                ++seg;
                ++calls;
                return 1;
            }
            if (kind == kAsk) return 3;
        }
        if (++seg > cap) {
            flags |= (1u << 2);
            return 1;
        }
        const Tab1<T> ce = tab[cell];
        int end = 0;
        if constexpr (sizeof(T) == 4) {
            // Written without branches but for the rare cases and the flush: a
            // warp's lanes collide, cross and end in one and the same segment,
            // and each branch would run for a few of them at a time.
            if (ws.n < need) ws.refill(round_keys(ca), step, stage);
            const bool right = mu > (T)0;
            const T dist_col = M::flight(ws.w[0], ce);
            const T dist_b = right ? (ce.dxs - x) * rmu : m_abs(x * rmu);
            const T dist_cen = c * (endsteptime - t) * ds;
            const T dist = min3_nan(dist_b, dist_col, dist_cen);
            if (dist != dist) {
                flags |= 1u;
                return 1;
            }
            T dep;
            const T newenergy = M::attenuate(E, ce, dist, &dep);
            const bool dead = newenergy <= minenergy;
            dep_sum.add(dead ? M::all_in(E, ce) : dep);
            x += mu * dist;
            t += dist * rdsc;
            E = newenergy;
            // the events in the reference's order: face, collision, census
            const bool at_b = !dead && dist == dist_b;
            const int next = cell + (right ? 1 : -1);
            const bool inside = (unsigned)next < (unsigned)N;
            if (at_b && inside) {
                flush_cell();
                dep_sum.clear();
                cell = next;
                x = right ? (T)0 : tab[next].dxs;
            }
            bool escaped = false;
            if (at_b && !inside) {
                // the escape, or the reflection, which leaves a right mover on
                // its face (the reference steps out and back in)
                escaped = !(right ? reflect_r : reflect_l);
                mu = -mu;
                rmu = -rmu;
                if (right) x = ce.dxs;
            }
            const bool turn = dist == dist_col;
            // mu = 1 - 2*rand, redrawn while zero (src/imc_transport.jl:178-181);
            // a zero needs rand == 0.5 exactly, so 64 redraws never run out
            auto new_direction = [&]() {
                T m = Rand<T>::cosine(ws.w[1]);
                if (turn && m == (T)0) {
                    for (int r = 1; r < 64 && m == (T)0; ++r) {
                        ws.drop(false);
                        if (ws.n < 2) ws.refill(round_keys(ca), step, stage);
                        m = Rand<T>::cosine(ws.w[1]);
                    }
                    if (m == (T)0) m = (T)1;
                }
                const T rm = rcp_mid(m);
                mu = turn ? m : mu;
                rmu = turn ? rm : rmu;
                ws.drop(turn);
            };
            if constexpr (LONG) {
                new_direction();
            } else {
                // a short history seldom collides
                if (turn) new_direction();
                else ws.drop(false);
            }
            // census: t = 0 and the state written back by finish()
            // (src/imc_transport.jl:185-193)
            end = dead ? 1 : escaped ? 4 : dist == dist_cen ? 2 : 0;
        } else {
            // FP64: every FP64 instruction costs more than a branch
            T dist_b, dist_cen, dist, em1;
            bool at_b, at_col, at_cen;
            const T dist_col = M::flight(rs, ce);
            const bool fwd = pos64(mu);
            dist_b = m64::div_r(fwd ? ce.dxs - x : x, mu, rmu);
            if (!fwd) dist_b = m_abs(dist_b);
            dist_cen = endsteptime - t;
            if (!c_one) dist_cen = c * dist_cen;
            if (!ds_one) dist_cen = dist_cen * ds;
            // odd: a distance below +0 or not a number
            const bool odd = !(plain64(dist_b) && plain64(dist_col) && plain64(dist_cen));
            if (!odd) {
                dist = min64(min64(dist_b, dist_col), dist_cen);
                at_b = m64::bits(dist) == m64::bits(dist_b);
                at_col = m64::bits(dist) == m64::bits(dist_col);
                at_cen = m64::bits(dist) == m64::bits(dist_cen);
            } else {
                dist_b = mu > (T)0 ? (ce.dxs - x) / mu : m_abs(x / mu);
                dist = jmin(jmin(dist_b, dist_col), dist_cen);
                at_b = dist == dist_b;
                at_col = dist == dist_col;
                at_cen = dist == dist_cen;
                if (dist != dist) {
                    flags |= 1u;
                    return 1;
                }
            }
            const T newenergy = M::attenuate(E, ce.saf, dist, &em1);
            const bool dead = le64(newenergy, minenergy);
            dep_sum.add(E, em1, dead, b_dep + se, flags);
            if (dead) return 1;
            x = fma(mu, dist, x);
            T dt_seg = ds_one ? dist : m64::div_r(dist, ds, rds);
            if (!c_one) dt_seg = m64::div_r(dt_seg, c, rc);
            t += dt_seg;
            E = newenergy;
            if (at_b) {
                const bool right = mu > (T)0;
                const int next = cell + (right ? 1 : -1);
                if ((unsigned)next < (unsigned)N) {
                    flush_cell();
                    dep_sum.clear();
                    cell = next;
                    x = right ? (T)0 : tab[next].dxs;
                } else if (right ? reflect_r : reflect_l) {
                    mu = -mu;
                    rmu = -rmu;
                    if (right) x = ce.dxs;
                } else {
                    return 4;
                }
            }
            if (at_col) {
                mu = (T)0;
                for (int r = 0; r < 64 && mu == (T)0; ++r) mu = Rand<T>::cosine(rs);
                if (mu == (T)0) mu = (T)1;
                rmu = rcp_any(mu);
            }
            if (at_cen) end = 2;
        }
        return end;
    };
    auto finish = [&](int end) {
        flush_cell();
        if (end == 2) {
            // census: t = 0, write the state back (src/imc_transport.jl:185-193)
            T Est = E;
            if (St::half) {
                st_v(pb.t + i, 0.0f);
                st_v(pb.x + i, (float)x / (float)tab[cell].dxs);
                st_v(pb.ux + i, (float)mu);
                __half ef = __float2half_rn((float)E / (float)E0);
                pb.E[i] = ef;
                Est = __half2float(ef) * (float)E0;
            } else {
                pb.t[i] = (typename St::S)0;
                pb.x[i] = (typename St::S)x;
                pb.ux[i] = (typename St::S)mu;
                pb.E[i] = (typename St::S)E;
            }
            if (cell != (cs & 0xFFFFFF)) pb.cs[i] = cell | (k << 24);
            bool flushed = false;
            if constexpr (RAD_SMT && sizeof(T) == 4)
                flushed = add_f32_smem(slots_k + 24u * (unsigned)(ca.K * nc + cell), Est, b_rad + se);
            if (!flushed) flush_rest<T, RAD_SMT>(rad_acc, k * nc + cell, Est, b_rad + se, flags);
            const int ee = exp_bound(Est) - se;
            emax_e = ee > emax_e ? ee : emax_e;
        } else if (end == 3) {
            // set aside with its state for the query pass (its deposits flushed)
            const unsigned long long j = atomicAdd(ask_count, 1ull);
            w.ask.x[j] = (float)x; w.ask.mu[j] = (float)mu; w.ask.t[j] = (float)t; w.ask.E[j] = (float)E;
            w.ask.E0[j] = (float)E0; w.ask.cs[j] = cell | (k << 24); w.ask.cs_list[j] = cs; w.ask.idx[j] = i;
        } else {
            // killed, or escaped with E through a vacuum face
            if (end == 4) flush_one<T, false>(ca.lost_acc, k, E, b_lost + se, flags);
            pb.alive[i] = 0;
            ++killed;
        }
        segs += (unsigned long long)seg;
    };
    const int lane = threadIdx.x & 31;
    if constexpr (!LONG) {
        // Short histories (the last transport averaged fewer than
        // kRefillSegments segments each): each lane walks one history to its
        // end, and the warp moves on together to 32 consecutive entries, so
        // every load and store of the list is coalesced.
        if constexpr (!kFromQueue) {
            // the list in chunks from the counter; the next entry's fields
            // are loaded while the current history walks (measured on the
            // 2000-cell slab, 0.496 -> 0.474 ms per launch)
            typedef typename St::S S;
            typedef typename St::E0S E0S;
            uint8_t pa = 0;
            int pcs = 0;
            S pt = (S)0.0f, px = (S)0.0f, pmu = (S)0.0f, pE = (S)0.0f;
            E0S pE0 = (E0S)0;
            auto fetch = [&](long long e) {
                pa = e < n ? pb.alive[e] : (uint8_t)0;
                if (pa) { pcs = pb.cs[e]; pt = pb.t[e]; px = pb.x[e]; pmu = pb.ux[e]; pE = pb.E[e]; pE0 = pb.E0[e]; }
            };
            for (long long base = warp_counter_next(&sc->work_next) * chunk; base < n;
                 base = warp_counter_next(&sc->work_next) * chunk) {
                fetch(base + lane);
                for (int r = 0; r < chunk; r += 32) {
                    const long long e = base + r + lane;
                    const bool a = pa != 0;
                    const int ccs = pcs;
                    E0 = (T)pE0;
                    if constexpr (St::half) {
                        t = __half2float(pt) * endsteptime;
                        x = a ? __half2float(px) * tab[ccs & 0xFFFFFF].dxs : 0.0f;
                        mu = __half2float(pmu);
                        E = __half2float(pE) * E0;
                    } else {
                        t = (T)pt; x = (T)px; mu = (T)pmu; E = (T)pE;
                    }
                    if (r + 32 < chunk) fetch(e + 32);
                    if (a) {
                        i = e;
                        cs = ccs;
                        start(ccs);
                        int end;
                        do end = segment(); while (!end);
                        finish(end);
                    }
                }
            }
        } else {
            // a resume pass's queue in chunks from the counter
            for (long long base = warp_counter_next(&sc->work_next) * chunk; base < n;
                 base = warp_counter_next(&sc->work_next) * chunk)
                for (int r = 0; r < chunk; r += 32) {
                    const long long e = base + r + lane;
                    int cs_now;
                    if (e >= n || !load(e, cs_now, t, x, mu, E, E0, i, cs)) continue;
                    start(cs_now);
                    int end;
                    do end = segment(); while (!end);
                    finish(end);
                }
        }
    } else {
        // Long histories of unequal length: each lane starts the next history
        // as soon as its current one ends.  The warp reads the entries in
        // chunks of 32 (coalesced: lane l prefetches entry 32 c + l into
        // registers); idle lanes take the chunk's entries in order through
        // register shuffles.
        const unsigned lt = (1u << lane) - 1u;
        const long long nchunks = (n + 31) / 32;
        // chunks of the list (or of a resume pass's queue) from the counter
        long long chunk = warp_counter_next(&sc->work_next);
        auto advance = [&]() { chunk = warp_counter_next(&sc->work_next); };
        int p_now = -1, p_cs = 0;  // prefetched entry (p_now -1: none / dead)
        long long p_i = 0;
        T p_t = (T)0, p_x = (T)0, p_mu = (T)0, p_E = (T)0, p_E0 = (T)0;
        auto prefetch = [&]() {
            const long long e = chunk * 32 + lane;
            p_now = -1;
            if (e < n) {
                int cn;
                if (load(e, cn, p_t, p_x, p_mu, p_E, p_E0, p_i, p_cs)) p_now = cn;
            }
        };
        bool more = chunk < nchunks;  // warp-uniform: the current chunk has entries left
        int pos = 0;                  // warp-uniform: next entry of the chunk to hand out
        if (more) prefetch();
        bool has = false;
        while (true) {
            unsigned idle = __ballot_sync(0xFFFFFFFFu, !has);
            while (idle && more) {
                const int r = __popc(idle & lt);
                const int avail = 32 - pos;
                const int sl = (pos + r) & 31;
                const int q_now = __shfl_sync(0xFFFFFFFFu, p_now, sl);
                const int q_cs = __shfl_sync(0xFFFFFFFFu, p_cs, sl);
                const long long q_i = __shfl_sync(0xFFFFFFFFu, p_i, sl);
                const T q_t = __shfl_sync(0xFFFFFFFFu, p_t, sl), q_x = __shfl_sync(0xFFFFFFFFu, p_x, sl);
                const T q_mu = __shfl_sync(0xFFFFFFFFu, p_mu, sl), q_E = __shfl_sync(0xFFFFFFFFu, p_E, sl);
                const T q_E0 = __shfl_sync(0xFFFFFFFFu, p_E0, sl);
                if (!has && r < avail && q_now >= 0) {
                    i = q_i;
                    cs = q_cs;
                    t = q_t; x = q_x; mu = q_mu; E = q_E; E0 = q_E0;
                    start(q_now);
                    has = true;
                }
                const int nidle = __popc(idle);
                pos += nidle < avail ? nidle : avail;
                if (pos >= 32) {
                    advance();
                    more = chunk < nchunks;
                    pos = 0;
                    if (more) prefetch();
                }
                idle = __ballot_sync(0xFFFFFFFFu, !has);
            }
            if (idle == 0xFFFFFFFFu) break;  // no history left for this warp
            need ^= 6;
            if (!has) continue;
            const int end = segment();
            if (end) {
                finish(end);
                has = false;
            }
        }
    }
    if (SMT) flush_block_tallies(ca, dep_acc, RAD_SMT);
    if (kPause) {
        for (int off = 16; off > 0; off >>= 1) calls += __shfl_down_sync(0xFFFFFFFFu, calls, off);
        if (lane == 0 && calls) atomicAdd(&sc->surrogate_calls, calls);
    }
    finish_counters(sc, segs, killed, flags, emax_e);
}

enum { kShortSchedule = 0, kLongSchedule = 1, kBothSchedules = 2 };
// The two lane schedules are kernels of their own, so that neither holds the
// other's registers and each has its own block size; a step launches both and
// the one whose schedule the step does not take returns at once (~2 us).
// The short one is bound by instruction issue (FP32 slab of 2000 cells: 80 % of
// the issue slots, 27 of 32 lanes; 200 steps filling to 2e7 histories take 348
// us a launch, 432 with both schedules in one kernel, words drawn on demand and
// a branch per face), the long one by the length of its longest histories (heat
// wave: 1100 segments, 15 of 32 lanes on average).
__device__ __forceinline__ bool long_histories(const Scalars *sc) { return sc->seg_per_hist >= kRefillSegments; }

template <class St, int BLOCK, int TM, int MODE, bool LONG>
__global__ void __launch_bounds__(BLOCK) k_transport1d(CellArgs ca, Scalars *sc, PBufPair bufs, SurrWave w,
                                                       int round) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (long_histories(sc) != LONG) return;
    transport1d_block<St, BLOCK, TM, MODE, LONG>(ca, sc, bufs, w, round, smem_raw, 0);
}

// One transport launch over the lists of many 1D decks (the fused batch,
// imc_run_batch_fused), whose arguments sit in constant memory.  Blocks go
// through the decks in turn, each from its own; a block sets up a deck (its cell
// table and private tallies) only while the deck's work counter still has
// chunks, takes chunks from that counter like the single-deck kernel, and
// flushes the deck's tallies and counters before it moves on.  Every history runs the
// single-deck code with the deck's own streams and exact tallies, so each
// deck's result is bit-identical to its own launch's.
__constant__ Deck1DArgs c_multi_ca[kFusedMaxDecks];
__constant__ PBufPair1D c_multi_bufs[kFusedMaxDecks];
__constant__ Scalars *c_multi_sc[kFusedMaxDecks];

template <class St, int BLOCK, bool LONG>
__global__ void __launch_bounds__(BLOCK) k_transport1d_multi(int ndecks) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    static_assert(kFusedMaxDecks == 256 && BLOCK >= kFusedMaxDecks, "eight decks a lane, one a thread");
    __shared__ float s_work[kFusedMaxDecks];
    __shared__ int s_at;
    // Each block starts at the deck that lies at its share of the step's
    // segments (as many of them a history as the last step had), so that a
    // deck's histories are walked by full blocks; with every block starting at
    // the first deck, a small deck left each a warp or two and the wait for
    // their longest history (24 small decks 246 ms against 231, 256 decks 18.4 s
    // against 16.1; giving a block only the decks that its share meets, and others
    // while they have four entries a thread: 234 ms, 16.5 s).
    if (threadIdx.x < kFusedMaxDecks) {
        float work = 0.0f;
        if ((int)threadIdx.x < ndecks) {
            const Scalars *sc = c_multi_sc[threadIdx.x];
            if (long_histories(sc) == LONG) work = (float)sc->n_particles * fmaxf(sc->seg_per_hist, 1.0f);
        }
        s_work[threadIdx.x] = work;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        float mine = 0.0f;
        for (int i = 0; i < 8; ++i) mine += s_work[8 * lane + i];
        float incl = mine;
        for (int off = 1; off < 32; off <<= 1) {
            const float o = __shfl_up_sync(0xFFFFFFFFu, incl, off);
            if (lane >= off) incl += o;
        }
        const float share = __shfl_sync(0xFFFFFFFFu, incl, 31) * ((float)blockIdx.x + 0.5f) / (float)gridDim.x;
        const unsigned before = __ballot_sync(0xFFFFFFFFu, incl <= share);  // lanes that end below it
        if (lane == min(__popc(before), 31)) {
            float acc = incl - mine;
            int d = 8 * lane;
            while (d < 8 * lane + 7 && acc + s_work[d] <= share) acc += s_work[d++];
            s_at = min(d, ndecks - 1);
        }
    }
    __syncthreads();
    int at = s_at;
    // then each deck once, in turn, that has chunks left
    for (int visit = 0; visit < ndecks; ++visit) {
        __syncthreads();
        if (threadIdx.x == 0) s_at = ndecks;
        __syncthreads();
        if ((int)threadIdx.x < ndecks) {
            const int d = at + (int)threadIdx.x < ndecks ? at + (int)threadIdx.x : at + (int)threadIdx.x - ndecks;
            if (s_work[d] > 0.0f) {
                // a stale, low counter only costs a setup
                const Scalars *sc = c_multi_sc[d];
                const unsigned long long used = *(volatile const unsigned long long *)&sc->work_next;
                const long long per = LONG ? 32 : kListChunk1D;
                if ((long long)used * per < sc->n_particles) atomicMin(&s_at, (int)threadIdx.x);
            }
        }
        __syncthreads();
        if (s_at == ndecks) return;
        at = at + s_at < ndecks ? at + s_at : at + s_at - ndecks;
        transport1d_block<St, BLOCK, kTallyShared, kModePlain, LONG>(c_multi_ca[at], c_multi_sc[at], c_multi_bufs[at],
                                                                SurrWave{}, 0, smem_raw, kListChunk1D);
    }
}

// TM, where the flushes go: kTallyGlobal, kTallyShared (deposition and
// census tallies block-private in shared memory) or kTallySharedDep (the
// deposition tallies only; census energy, one flush per census particle, to
// global memory)
// SCHED: the short- or the long-history schedule, or both in one kernel (FP64,
// whose registers hold both; the launch that does nothing costs it 3 %).
template <class St, int BLOCK, int TM, int SCHED>
__global__ void __launch_bounds__(BLOCK) k_transport2d(CellArgs ca, Scalars *sc, PBufPair bufs) {
    const bool long_step = long_histories(sc);
    if (SCHED != kBothSchedules && long_step != (SCHED == kLongSchedule)) return;
    constexpr bool SMT = TM != kTallyGlobal;        // deposition flushes to shared memory
    constexpr bool RAD_SMT = TM == kTallyShared;    // census flushes to shared memory
    typedef typename St::T T;
    PBuf<St> pb(bufs.b[sc->cur]);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int NX = ca.nx, NY = ca.ny, nc = ca.nc;
    Tab2<T> *tab = reinterpret_cast<Tab2<T> *>(smem_raw);
    Face<T> *fx = reinterpret_cast<Face<T> *>(tab + nc);
    Face<T> *fy = fx + NX;
    const T ds = Consts<T>::ds(ca), c = Consts<T>::c(ca);
    const bool ds_one = ds == (T)1, c_one = c == (T)1;
    const T rdsc = Consts<T>::rdsc(ca);
    const T rds = sizeof(T) == 8 ? (T)1 / ds : (T)0, rc = sizeof(T) == 8 ? (T)1 / c : (T)0;
    long long *dep_acc = ca.dep_acc, *rad_acc = ca.rad_acc;
    if (SMT) {
        dep_acc = tally_smem(smem_raw, table_bytes(ca, sizeof(T)));
        if (RAD_SMT) rad_acc = dep_acc + 3 * (size_t)ca.K * ca.nc;
        for (int i = threadIdx.x; i < (RAD_SMT ? 6 : 3) * ca.K * ca.nc; i += blockDim.x) dep_acc[i] = 0;
    }
    load_tab(tab, ca.tab, nc);
    for (int i = threadIdx.x; i < NX; i += blockDim.x) { fx[i].wT = (T)ca.dx[i]; fx[i].ws = fx[i].wT * ds; }
    for (int i = threadIdx.x; i < NY; i += blockDim.x) { fy[i].wT = (T)ca.dy[i]; fy[i].ws = fy[i].wT * ds; }
    __shared__ int s_sexp[16];
    load_scale_exps(ca, s_sexp);
    __syncthreads();
    const T dtT = (T)sc->dt;
    const long long n = sc->n_particles;
    const int b_dep = sc->b_dep, b_rad = sc->b_rad, b_lost = sc->b_lost;
    const unsigned step = sc->step;
    const unsigned long long seed = ca.seed;
    const unsigned cap = ca.seg_cap > 0xFFFFFFFEll ? 0xFFFFFFFEu : (unsigned)ca.seg_cap;
    const bool refl_l = ca.bc[0] == 1, refl_r = ca.bc[1] == 1, refl_t = ca.bc[2] == 1, refl_b = ca.bc[3] == 1;
    unsigned long long segs = 0, killed = 0;
    unsigned flags = 0;
    int emax_e = kNoExp;
    // Lane state of the history in flight.
    long long i = 0;
    int cs = 0, xi = 0, yi = 0, k = 0, se = 0;  // se: scale k's exponent
    const unsigned dep_shared = SMT ? (unsigned)__cvta_generic_to_shared(dep_acc) : 0u;
    unsigned slots_k = 0;  // shared tallies: scale k's deposition slots
    // c / NX as the high word of c times this (exact: c NX < 2^32, as the
    // table of all cells fits in shared memory)
    const unsigned rNX = NX > 1 ? 0xFFFFFFFFu / (unsigned)NX + 1u : 0u;
    auto row_of = [&](int c) { return NX > 1 ? (int)__umulhi((unsigned)c, rNX) : c; };
    T t = (T)0, xp = (T)0, yp = (T)0, vx = (T)0, vy = (T)0, E = (T)0, E0 = (T)0, minenergy = (T)0;
    CellSum<T> dep_sum;
    T rvx = (T)0, rvy = (T)0;  // 1/vx, 1/vy (FP32: inf where div_mid is to divide)
    unsigned seg = 0;
    Stream rs;     // FP64
    Words<5> ws;   // FP32
    auto start = [&]() {
        const int cell0 = cs & 0xFFFFFF;
        k = cs >> 24;
        yi = row_of(cell0);
        xi = cell0 - yi * NX;
        se = s_sexp[k];
        if constexpr (SMT) slots_k = dep_shared + 24u * (unsigned)(k * nc);
        if constexpr (sizeof(T) == 8) rs.init(seed, step, (uint32_t)i, kStageTransport);
        else if constexpr (SCHED == kLongSchedule) ws.init((uint32_t)i);
        else ws.init_full((uint32_t)i, round_keys(ca), step, kStageTransport);
        minenergy = cutoff_energy(E0);  // (T)(0.01 * (double)E0), without FP64 in binary32
        dep_sum.clear();
        seg = 0;
        rvx = face_rcp(vx);
        rvy = face_rcp(vy);
    };
    auto load = [&](long long e, int &lcs, T &lt, T &lx, T &ly, T &lvx, T &lvy, T &lE, T &lE0) -> bool {
        if (!pb.alive[e]) return false;
        lcs = pb.cs[e];
        const int c0 = lcs & 0xFFFFFF;
        lE0 = (T)pb.E0[e];
        if (St::half) {
            lt = ld_f(pb.t + e) * (float)dtT;
            const int r0 = row_of(c0);
            lx = ld_f(pb.x + e) * (float)fx[c0 - r0 * NX].ws;
            ly = ld_f(pb.y + e) * (float)fy[r0].ws;
            lvx = ld_f(pb.ux + e);
            lvy = ld_f(pb.uy + e);
            lE = ld_f(pb.E + e) * (float)lE0;
        } else {
            lt = (T)pb.t[e]; lx = (T)pb.x[e]; ly = (T)pb.y[e];
            lvx = (T)pb.ux[e]; lvy = (T)pb.uy[e]; lE = (T)pb.E[e];
        }
        return true;
    };
    // the deposits of the cell the history leaves, or ends in
    auto flush_cell = [&]() {
        const int cell = xi + yi * NX;
        if constexpr (sizeof(T) == 4) {
            const T v = dep_sum.s + dep_sum.c;
            if constexpr (SMT)
                if (add_f32_smem(slots_k + 24u * (unsigned)cell, v, b_dep + se)) return;
            flush_rest<T, SMT>(dep_acc, k * nc + cell, v, b_dep + se, flags);
        } else {
            dep_sum.template flush<SMT>(dep_acc, k * nc + cell, flags);
        }
    };
    // one pass of the reference's while loop (src/imc_transport.jl:533-717);
    // 0 = go on, 1 = killed, 2 = census, 4 = escaped through a vacuum face.
    // The census write and the escape tally are left to finish(), which
    // the warp runs converged once per history.  Both axes and both directions
    // share one path through the face: a warp's lanes cross all four.
    auto segment = [&]() -> int {
        if (++seg > cap) { flags |= (1u << 2); return 1; }
        const int cell = xi + yi * NX;
        const Tab2<T> ce = tab[cell];
        T dist_bx, dist_by, dist_col, dist_cen, dist, newenergy;
        bool at_b, at_col, at_cen, dead;
        const bool right = vx > (T)0, up = vy > (T)0;
        if constexpr (sizeof(T) == 4) {
            if (ws.n < 2) ws.refill(round_keys(ca), step, kStageTransport);
            dist_col = SegMath<T>::flight(ws.w[0], ce.rseff);
            dist_cen = c * (dtT - t) * ds;
            // the reference's quotients |num / v|
            dist_bx = m_abs(div_mid(right ? fx[xi].ws - xp : xp, vx, rvx));
            dist_by = m_abs(div_mid(up ? fy[yi].ws - yp : yp, vy, rvy));
            dist = min3_nan(fminf(dist_bx, dist_by), dist_col, dist_cen);
            if (dist != dist) { flags |= 1u; return 1; }
            at_b = dist == dist_bx || dist == dist_by;
            at_col = dist == dist_col;
            at_cen = dist == dist_cen;
            const float em1 = expm1_seg(-ce.saf * dist);
            newenergy = E + E * em1;
            const float Edens = E * ce.rarea;
            dead = newenergy <= minenergy;
            dep_sum.add(dead ? Edens : -Edens * em1);
        } else {
            // FP64: SegMath<double>'s formulation; the deposits are energies
            dist_col = SegMath<double>::flight(rs, ce.seff, ca.tab_rs[cell]);
            dist_cen = dtT - t;
            if (!c_one) dist_cen = c * dist_cen;
            if (!ds_one) dist_cen = dist_cen * ds;
            dist_bx = m_abs(m64::div_r(right ? fx[xi].ws - xp : xp, vx, rvx));
            dist_by = m_abs(m64::div_r(up ? fy[yi].ws - yp : yp, vy, rvy));
            const bool odd = !(plain64(dist_bx) && plain64(dist_by) && plain64(dist_col) && plain64(dist_cen));
            if (!odd) {
                dist = min64(min64(dist_bx, dist_by), min64(dist_col, dist_cen));
                const uint64_t b = m64::bits(dist);
                at_b = b == m64::bits(dist_bx) || b == m64::bits(dist_by);
                at_col = b == m64::bits(dist_col);
                at_cen = b == m64::bits(dist_cen);
            } else {
                // by the reference's expressions and order
                dist_bx = vx > (T)0 ? m_abs((fx[xi].ws - xp) / vx) : m_abs(xp / vx);
                dist_by = vy > (T)0 ? m_abs((fy[yi].ws - yp) / vy) : m_abs(yp / vy);
                T dist_b;
                if (dist_bx != dist_bx) dist_b = dist_by;
                else if (dist_by != dist_by) dist_b = dist_bx;
                else dist_b = jmin(dist_bx, dist_by);
                dist = jmin(jmin(dist_b, dist_col), dist_cen);
                at_b = dist == dist_bx || dist == dist_by;
                at_col = dist == dist_col;
                at_cen = dist == dist_cen;
                if (dist != dist) { flags |= 1u; return 1; }
            }
            double em1;
            newenergy = SegMath<double>::attenuate(E, ce.saf, dist, &em1);
            dead = le64(newenergy, minenergy);
            dep_sum.add(E, em1, dead, b_dep + se, flags);
        }
        if (dead) return 1;
        if constexpr (sizeof(T) == 4) {
            xp += dist * vx;
            yp += dist * vy;
            t += dist * rdsc;
        } else {
            xp = fma(dist, vx, xp);
            yp = fma(dist, vy, yp);
            T dt_seg = ds_one ? dist : m64::div_r(dist, ds, rds);
            if (!c_one) dt_seg = m64::div_r(dt_seg, c, rc);
            t += dt_seg;
        }
        E = newenergy;
        if (at_b) {
            if constexpr (sizeof(T) == 4) ws.drop(false);
            const bool ax = dist_bx < dist_by, fwd = ax ? right : up;
            const int next = (ax ? xi : yi) + (fwd ? 1 : -1);
            if ((unsigned)next < (unsigned)(ax ? NX : NY)) {
                flush_cell();
                dep_sum.clear();
                const T at = fwd ? (T)0 : (ax ? fx : fy)[next].ws;
                if (ax) { xi = next; xp = at; }
                else { yi = next; yp = at; }
                return 0;
            }
            if (!(ax ? (fwd ? refl_r : refl_l) : (fwd ? refl_t : refl_b))) return 4;
            if (ax) { vx = -vx; rvx = -rvx; }
            else { vy = -vy; rvy = -rvy; }
            return 0;
        }
        if (at_col) {
            // isotropic re-emission: angle 2*pi*rand in Float64, rounded to T
            // (binary32: two_pi_u24, the same value without FP64; the
            // hardware sine and cosine)
            if constexpr (sizeof(T) == 4) {
                __sincosf(two_pi_u24(ws.w[1] >> 8), &vy, &vx);
                ws.drop(true);
            } else {
                m_sincos((T)(6.283185307179586 * (double)Rand<T>::u(rs)), &vy, &vx);
            }
            rvx = face_rcp(vx);
            rvy = face_rcp(vy);
        }
        // census: t = 0 and the state written back by finish()
        if (at_cen) return 2;
        return 0;
    };
    auto finish = [&](int end) {
        flush_cell();
        if (end == 2) {
            // census: t = 0, write the state back (src/imc_transport.jl:700-717)
            const int cellf = xi + yi * NX;
            T Est = E;
            if (St::half) {
                st_v(pb.t + i, 0.0f);
                st_v(pb.x + i, (float)xp / (float)fx[xi].ws);
                st_v(pb.y + i, (float)yp / (float)fy[yi].ws);
                st_v(pb.ux + i, (float)vx);
                st_v(pb.uy + i, (float)vy);
                __half ef = __float2half_rn((float)E / (float)E0);
                pb.E[i] = ef;
                Est = __half2float(ef) * (float)E0;
            } else {
                pb.t[i] = (typename St::S)0;
                pb.x[i] = (typename St::S)xp;
                pb.y[i] = (typename St::S)yp;
                pb.ux[i] = (typename St::S)vx;
                pb.uy[i] = (typename St::S)vy;
                pb.E[i] = (typename St::S)E;
            }
            if (cellf != (cs & 0xFFFFFF)) pb.cs[i] = cellf | (k << 24);
            bool flushed = false;
            if constexpr (sizeof(T) == 4) {
                if constexpr (RAD_SMT) flushed = add_f32_smem(slots_k + 24u * (unsigned)(ca.K * nc + cellf), Est, b_rad + se);
                else flushed = add_f32_global(rad_acc + 3 * (size_t)(k * nc + cellf), Est, b_rad + se);
            }
            if (!flushed) flush_rest<T, RAD_SMT>(rad_acc, k * nc + cellf, Est, b_rad + se, flags);
            const int ee = exp_bound(Est) - se;
            emax_e = ee > emax_e ? ee : emax_e;
        } else {
            // killed, or escaped with E through a vacuum face
            if (end == 4) flush_one<T, false>(ca.lost_acc, k, E, b_lost + se, flags);
            pb.alive[i] = 0;
            ++killed;
        }
        segs += (unsigned long long)seg;
    };
    if (SCHED == kShortSchedule || (SCHED == kBothSchedules && !long_step)) {
        // short histories: one history per lane to its end (see k_transport1d)
        auto walk = [&](long long e) {
            if (!load(e, cs, t, xp, yp, vx, vy, E, E0)) return;
            i = e;
            start();
            int end;
            do end = segment(); while (!end);
            finish(end);
        };
        // the list in chunks from the counter
        const int lane = threadIdx.x & 31, chunk = list_chunk(n, kListChunk);
        for (long long base = warp_counter_next(&sc->work_next) * chunk; base < n;
             base = warp_counter_next(&sc->work_next) * chunk)
            for (int r = 0; r < chunk; r += 32)
                if (base + r + lane < n) walk(base + r + lane);
    } else {
        // long histories: lanes refill from 32-entry chunks (see k_transport1d)
        const int lane = threadIdx.x & 31;
        const unsigned lt = (1u << lane) - 1u;
        const long long nchunks = (n + 31) / 32;
        // chunks from the counter
        long long chunk = warp_counter_next(&sc->work_next);
        auto advance = [&]() { chunk = warp_counter_next(&sc->work_next); };
        int p_cs = -1;
        T p_t = (T)0, p_x = (T)0, p_y = (T)0, p_vx = (T)0, p_vy = (T)0, p_E = (T)0, p_E0 = (T)0;
        auto prefetch = [&]() {
            const long long e = chunk * 32 + lane;
            int lcs = -1;
            if (!(e < n && load(e, lcs, p_t, p_x, p_y, p_vx, p_vy, p_E, p_E0))) lcs = -1;
            p_cs = lcs;
        };
        bool more = chunk < nchunks;
        int pos = 0;
        if (more) prefetch();
        bool has = false;
        while (true) {
            unsigned idle = __ballot_sync(0xFFFFFFFFu, !has);
            while (idle && more) {
                const int r = __popc(idle & lt);
                const int avail = 32 - pos;
                const int sl = (pos + r) & 31;
                const int q_cs = __shfl_sync(0xFFFFFFFFu, p_cs, sl);
                const T q_t = __shfl_sync(0xFFFFFFFFu, p_t, sl), q_x = __shfl_sync(0xFFFFFFFFu, p_x, sl);
                const T q_y = __shfl_sync(0xFFFFFFFFu, p_y, sl), q_vx = __shfl_sync(0xFFFFFFFFu, p_vx, sl);
                const T q_vy = __shfl_sync(0xFFFFFFFFu, p_vy, sl), q_E = __shfl_sync(0xFFFFFFFFu, p_E, sl);
                const T q_E0 = __shfl_sync(0xFFFFFFFFu, p_E0, sl);
                if (!has && r < avail && q_cs >= 0) {
                    i = chunk * 32 + pos + r;
                    cs = q_cs;
                    t = q_t; xp = q_x; yp = q_y; vx = q_vx; vy = q_vy; E = q_E; E0 = q_E0;
                    start();
                    has = true;
                }
                const int nidle = __popc(idle);
                pos += nidle < avail ? nidle : avail;
                if (pos >= 32) {
                    advance();
                    more = chunk < nchunks;
                    pos = 0;
                    if (more) prefetch();
                }
                idle = __ballot_sync(0xFFFFFFFFu, !has);
            }
            if (idle == 0xFFFFFFFFu) break;
            if (!has) continue;
            const int end = segment();
            if (end) {
                finish(end);
                has = false;
            }
        }
    }
    if (SMT) flush_block_tallies(ca, dep_acc, RAD_SMT);
    finish_counters(sc, segs, killed, flags, emax_e);
}

// Launch shape of the transport kernel.  When the table and the block's
// private tallies fit in shared memory the kernel runs one large block per
// SM with shared tallies (kSmtBlock32 threads for FP32 / FP16 state,
// kSmtBlock64 for FP64).  When only the table and the deposition tallies fit
// in the opt-in maximum, the deposition tallies are shared and the census
// flushes (one per census particle) go to global memory (the analog passes
// of the surrogate transport then keep every tally global).
// Otherwise every flush goes to global memory (kGlbBlock32 / kGlbBlock64
// threads).
constexpr int kSmemBudget = 200 * 1024;
constexpr int kSmemOptInMax = 227 * 1024;  // sm_100-family dynamic shared memory per block

TransportShape transport_shape(const CellArgs &ca, int prec) {
    TransportShape sh{};
    const int tsz = prec == 0 ? 8 : 4;
    const int table = table_bytes(ca, tsz);
    const long long dep = 3ll * 8 * (long long)ca.K * ca.nc;
    sh.smem_tally = table + 2 * dep <= kSmemBudget;
    sh.dep_only = !sh.smem_tally && table + dep <= kSmemOptInMax;
    sh.smem = table + (int)(sh.smem_tally ? 2 * dep : sh.dep_only ? dep : 0);
    const bool shared = sh.smem_tally || sh.dep_only;
    sh.block = shared ? (prec == 0 ? kSmtBlock64 : kSmtBlock32) : (prec == 0 ? kGlbBlock64 : kGlbBlock32);
    sh.block_long = prec == 0 ? sh.block : kLongBlock32;
    return sh;
}

template <class St> struct StBlocks {
    static constexpr bool fp64 = sizeof(typename St::T) == 8;
    static constexpr int smt = fp64 ? kSmtBlock64 : kSmtBlock32;
    static constexpr int glb = fp64 ? kGlbBlock64 : kGlbBlock32;
    static constexpr int smt_long = fp64 ? kSmtBlock64 : kLongBlock32;
    static constexpr int glb_long = fp64 ? kGlbBlock64 : kLongBlock32;
};

// the transport kernels of one state type and tally mode: short histories, long
// histories
template <class St, int TM> struct Kernels {
    static constexpr int block = TM == kTallyGlobal ? StBlocks<St>::glb : StBlocks<St>::smt;
    static constexpr int block_long = TM == kTallyGlobal ? StBlocks<St>::glb_long : StBlocks<St>::smt_long;
    static constexpr bool two = !StBlocks<St>::fp64;  // 2D: a kernel for each schedule
    static const void *ptr(int geometry, bool lng) {
        if (geometry == 2)
            return lng ? (const void *)k_transport2d<St, block_long, TM, two ? kLongSchedule : kBothSchedules>
                       : (const void *)k_transport2d<St, block, TM, two ? kShortSchedule : kBothSchedules>;
        if (lng) return (const void *)k_transport1d<St, block_long, TM, kModePlain, true>;
        return (const void *)k_transport1d<St, block, TM, kModePlain, false>;
    }
    static void launch(const CellArgs &ca, Scalars *sc, PBufPair buf, TransportGrid g, int smem, cudaStream_t st) {
        if (ca.geometry == 2) {
            k_transport2d<St, block, TM, two ? kShortSchedule : kBothSchedules><<<g.grid, block, smem, st>>>(ca, sc, buf);
            if constexpr (two) k_transport2d<St, block_long, TM, kLongSchedule><<<g.grid_long, block_long, smem, st>>>(ca, sc, buf);
            return;
        }
        k_transport1d<St, block, TM, kModePlain, false><<<g.grid, block, smem, st>>>(ca, sc, buf, SurrWave{}, 0);
        k_transport1d<St, block_long, TM, kModePlain, true><<<g.grid_long, block_long, smem, st>>>(ca, sc, buf,
                                                                                                SurrWave{}, 0);
    }
};

template <class St> static const void *kernel_of(const CellArgs &ca, const TransportShape &sh, bool lng) {
    if (sh.smem_tally) return Kernels<St, kTallyShared>::ptr(ca.geometry, lng);
    if (sh.dep_only) return Kernels<St, kTallySharedDep>::ptr(ca.geometry, lng);
    return Kernels<St, kTallyGlobal>::ptr(ca.geometry, lng);
}

template <class St>
static void launch_of(const CellArgs &ca, const TransportShape &sh, Scalars *sc, PBufPair buf, TransportGrid g,
                      cudaStream_t st) {
    if (sh.smem_tally) Kernels<St, kTallyShared>::launch(ca, sc, buf, g, sh.smem, st);
    else if (sh.dep_only) Kernels<St, kTallySharedDep>::launch(ca, sc, buf, g, sh.smem, st);
    else Kernels<St, kTallyGlobal>::launch(ca, sc, buf, g, sh.smem, st);
}

const void *transport_kernel_ptr(const CellArgs &ca, int prec, bool lng) {
    TransportShape sh = transport_shape(ca, prec);
    if (prec == 0) return kernel_of<StF64>(ca, sh, lng);
    if (prec == 1) return kernel_of<StF32>(ca, sh, lng);
    return kernel_of<StF16>(ca, sh, lng);
}

void launch_transport(const CellArgs &ca, Scalars *sc, int prec, PBufPair buf, TransportGrid g, cudaStream_t st) {
    TransportShape sh = transport_shape(ca, prec);
    if (prec == 0) launch_of<StF64>(ca, sh, sc, buf, g, st);
    else if (prec == 1) launch_of<StF32>(ca, sh, sc, buf, g, st);
    else launch_of<StF16>(ca, sh, sc, buf, g, st);
}

template <class St> static const void *multi_ptr(bool lng) {
    if (lng) return (const void *)k_transport1d_multi<St, StBlocks<St>::smt_long, true>;
    return (const void *)k_transport1d_multi<St, StBlocks<St>::smt, false>;
}
const void *transport_multi_ptr(int prec, bool lng) {
    return prec == 0 ? multi_ptr<StF64>(lng) : prec == 1 ? multi_ptr<StF32>(lng) : multi_ptr<StF16>(lng);
}

int transport_multi_block(int prec, bool lng) {
    return prec == 0 ? kSmtBlock64 : lng ? kLongBlock32 : kSmtBlock32;
}

cudaError_t set_transport_multi_decks(const Deck1DArgs *ca, const PBufPair1D *bufs, Scalars *const *sc, int n,
                                      cudaStream_t st) {
    if (n < 0 || n > kFusedMaxDecks) return cudaErrorInvalidValue;
    cudaError_t e = cudaMemcpyToSymbolAsync(c_multi_ca, ca, sizeof(Deck1DArgs) * (size_t)n, 0,
                                            cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbolAsync(c_multi_bufs, bufs, sizeof(PBufPair1D) * (size_t)n, 0, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbolAsync(c_multi_sc, sc, sizeof(Scalars *) * (size_t)n, 0, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    return e;
}


// ------------------------------------------- analog passes of the surrogate transport
// which: 0 the list pass, 1 a resume pass that sets aside, 2 the last resume pass
template <class St, bool SMT, int MODE> struct WaveKernels {
    static constexpr int tm = SMT ? kTallyShared : kTallyGlobal;
    static constexpr int block = SMT ? kSmtBlock32 : kGlbBlock32;
    static const void *ptr(bool lng) {
        if (lng) return (const void *)k_transport1d<St, kLongBlock32, tm, MODE, true>;
        return (const void *)k_transport1d<St, block, tm, MODE, false>;
    }
    static void launch(const CellArgs &ca, Scalars *sc, PBufPair bufs, const SurrWave &w, int round, TransportGrid g,
                       int smem, cudaStream_t st) {
        k_transport1d<St, block, tm, MODE, false><<<g.grid, block, smem, st>>>(ca, sc, bufs, w, round);
        k_transport1d<St, kLongBlock32, tm, MODE, true><<<g.grid_long, kLongBlock32, smem, st>>>(ca, sc, bufs, w, round);
    }
};

template <class St, bool SMT> static const void *wave_ptr(int which, bool lng) {
    if (which == 0) return WaveKernels<St, SMT, kModeList>::ptr(lng);
    if (which == 1) return WaveKernels<St, SMT, kModeResume>::ptr(lng);
    return WaveKernels<St, SMT, kModeResumeLast>::ptr(lng);
}

const void *surr_analog_ptr(const CellArgs &ca, int prec, int which, bool lng) {
    const bool smt = transport_shape(ca, prec).smem_tally;
    if (prec == 2) return smt ? wave_ptr<StF16, true>(which, lng) : wave_ptr<StF16, false>(which, lng);
    return smt ? wave_ptr<StF32, true>(which, lng) : wave_ptr<StF32, false>(which, lng);
}

int surr_analog_smem(const CellArgs &ca, int prec) {
    return analog1d_smem(ca, 4, transport_shape(ca, prec).smem_tally, true);
}

template <class St, bool SMT>
static void wave_one(const CellArgs &ca, Scalars *sc, PBufPair bufs, const SurrWave &w, int which, int round,
                     TransportGrid g, int smem, cudaStream_t st) {
    if (which == 0) WaveKernels<St, SMT, kModeList>::launch(ca, sc, bufs, w, round, g, smem, st);
    else if (which == 1) WaveKernels<St, SMT, kModeResume>::launch(ca, sc, bufs, w, round, g, smem, st);
    else WaveKernels<St, SMT, kModeResumeLast>::launch(ca, sc, bufs, w, round, g, smem, st);
}

void launch_surr_analog(const CellArgs &ca, Scalars *sc, int prec, PBufPair bufs, const SurrWave &w, int which,
                        int round, TransportGrid g, int smem, cudaStream_t st) {
    const bool smt = transport_shape(ca, prec).smem_tally;
    if (prec == 2) {
        if (smt) wave_one<StF16, true>(ca, sc, bufs, w, which, round, g, smem, st);
        else wave_one<StF16, false>(ca, sc, bufs, w, which, round, g, smem, st);
    } else {
        if (smt) wave_one<StF32, true>(ca, sc, bufs, w, which, round, g, smem, st);
        else wave_one<StF32, false>(ca, sc, bufs, w, which, round, g, smem, st);
    }
}

}  // namespace imc
