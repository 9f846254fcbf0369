// gathers.cuh -- the four gather kernels of the two-scale step (densities of both
// scales, low-res force + advance + split marks, high-res force + integrate +
// tether), templated on the batch form B, the walk G (gather.cuh) and the
// arithmetic policy A (arith.cuh).  sph.cu instantiates them with ExactArith (the
// reference's bits), sph_fast.cu with FastArith (within the step's tolerance).
//
// Particles are in (cell, id) order.  Because the arrays are sorted by cell, the
// candidates of one row of the 3x3 (or wider cross-scale) cell window are one
// contiguous span [off[row + cx0], off[row + cx1 + 1]).  Each particle's sums take
// its candidates in the reference's order (cells row by row, particles in cell
// order), which keeps every FP32 sum identical to the reference's for the same
// list order.  A particle is taken in one of three ways (gather.cuh): by one thread,
// consecutive threads with overlapping windows so that neighbour loads are shared
// through L1 (the throughput form); by a group of 8 or 4 lanes, where a list is too
// short to fill the GPU that way (by_size); or by a warp, a launch shape of its own.
// All give the same bits.
//
// Each kernel's per-particle work is an inlined function of the particle's Params:
// the kernel's own constants for a single scene, the scene's table row for a
// batch.  The row is read through a reference, so each field is loaded where it is
// used: a copy of the whole row kept every field live in registers across the
// neighbour loops, and the batched gathers spilled and ran 5 % slower.  A scene's
// cell windows index its grid at its cell base in the global cell space, so one
// sort and one offset table serve all scenes of a batch.
#pragma once
#include "arith.cuh"
#include "gather.cuh"
#include "sph.cuh"

namespace tss {

namespace gather_detail {
__device__ __forceinline__ int nthreads() { return gridDim.x * blockDim.x; }
__device__ __forceinline__ int tid() { return blockIdx.x * blockDim.x + threadIdx.x; }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return sub2(a, b); }
__device__ __forceinline__ float2 vel_of(float4 vq) { return make_float2(vq.x, vq.y); }
__device__ __forceinline__ void add_density(float& d, float t) { d += t; }

// The particles of a gather, one per thread (G = PerThread) or one per group of lanes
// (PerGroup, every lane of a group taking the same particle).  f(i, valid): the
// groups of a warp come together, those past the end with the last particle and
// valid = false.
// Taken by `blocks` blocks, of which this one is the `block`-th.
template <class G, class F>
__device__ __forceinline__ void for_each_particle(int n, int block, int blocks, F&& f) {
    const int t0 = block * blockDim.x + threadIdx.x, step = blocks * blockDim.x;
    if constexpr (G::kLanes > 1) {
        constexpr int per = 32 / G::kLanes;  // particles per warp
        for (int base = (t0 >> 5) * per; base < n; base += (step >> 5) * per) {
            const int i = base + (static_cast<int>(threadIdx.x) & 31) / G::kLanes;
            f(min(i, n - 1), i < n);
        }
    } else {
        for (int i = t0; i < n; i += step) f(i, true);
    }
}
template <class G, class F>
__device__ __forceinline__ void for_each_particle(int n, F&& f) {
    for_each_particle<G>(n, blockIdx.x, gridDim.x, f);
}

// f(form, n) with the form that takes n particles: the launch's own, except that one
// particle per thread becomes one per group of lanes for a short list (sph.cuh).
template <class G, bool Force, class F>
__device__ __forceinline__ void by_size(int n, F&& f) {
    if constexpr (G::kLanes == 1) {
        if (n <= (Force ? kForce8Max : kDensity8Max)) {
            f(PerGroup<8>{}, n);
            return;
        }
        if constexpr (Force) {
            if (n <= kForce4Max) {
                f(PerGroup<4>{}, n);
                return;
            }
        }
    }
    f(G{}, n);
}
}  // namespace gather_detail
using namespace gather_detail;

// Neighbour lists (ScaleView::nbr).  The density pass records the same-scale
// candidates that a particle's window accepts, in window order, and the force pass of the same step walks that list instead of its window: the
// force's own candidates are a subset of the density's (same positions and
// states, cutoff d < r and d != 0 against d <= r, the same lambda masks), so
// testing each listed candidate again with the force's test gives the force's
// candidates in the same order -- the same sums, bit for bit -- without scanning
// the ~36 candidates of the window, of which about a third are accepted.  A particle
// with more than kMaxNbr neighbours is marked kNbrCrowd: its list holds the first of
// them, and the force walks its window from the last one listed.  One with an offset that
// does not fit 16 bits is marked kNbrOverflow and walks its whole window.
//
// The density pass takes a particle's same-scale window in two phases.  The first
// walks the window and only tests: it leaves the accepted candidates' offsets in
// shared memory (`col`: the thread's column of a kNbrRows x kNbrCols array, stride
// kNbrCols), a few instructions per candidate.  The second walks that short list,
// evaluates the pairs' terms in order and writes the list out.  A warp's lanes
// accept different candidates of the ~34 in their windows, so a walk that evaluates
// a pair as soon as its test passes runs the pair arithmetic for nearly every
// candidate with a third of the lanes active; here it runs once per list entry with
// almost all of them (the lists are 10-14 long).  A window of more particles than a list
// holds is taken column by column (nbr_crowd).  A dam break of 1.0M low-res and
// 1.0M high-res particles, exact / tolerance arithmetic, against a walk that
// evaluated at once: low-res density 96 -> 61 / 73 -> 51 us, high-res density 117 ->
// 86 / 92 -> 67 us (with the longer lists, kMaxNbr); a 5,000-particle scene 16 -> 13
// and 18 -> 12 us.  Warp instructions of the exact low-res density 94 -> 53 M, active
// lanes 17 -> 26 of 32; issue still bounds it (79 % of cycles), DRAM a few percent.
constexpr int kNbrCols = 256;          // the gathers' largest block
constexpr int kNbrRows = kMaxNbr + 5;  // the particle itself, and one trip of four past a full list

// Phase one: the candidates k of the window with key(k) <= T (a NaN key fails), in
// window order, as k - i in the column.  Returns their number; kNbrFar when an offset
// does not fit 16 bits; or, when there are more than the list holds, minus the number
// found before the search stopped, at candidate k of row cy.
constexpr int kNbrFar = -0x10000;

template <class Key>
__device__ __forceinline__ int nbr_search(const int* off, int dimx, int csx, int cex, int& cy, int cey, int& k, int i,
                                          float T, int16_t* col, Key&& key) {
    int16_t* c = col;
    int16_t* const full = col + (kMaxNbr + 1) * kNbrCols;
    const auto put = [&](int j, float x) {
        if (x <= T) {
            *c = static_cast<int16_t>(j - i);
            c += kNbrCols;
        }
    };
    for (; cy <= cey; ++cy) {
        const int row = cy * dimx;
        k = off[row + csx];
        const int b = off[row + cex + 1];
        if (k - i < -32768 || b - i > 32768) return kNbrFar;
        for (; k + 3 < b; k += 4) {
            const float x0 = key(k), x1 = key(k + 1), x2 = key(k + 2), x3 = key(k + 3);
            put(k, x0);
            put(k + 1, x1);
            put(k + 2, x2);
            put(k + 3, x3);
            if (c > full) {
                k += 4;
                return -(static_cast<int>(c - col) / kNbrCols);
            }
        }
        if (k + 1 < b) {
            const float x0 = key(k), x1 = key(k + 1);
            put(k, x0);
            put(k + 1, x1);
            k += 2;
        }
        if (k < b) {
            put(k, key(k));
            ++k;
        }
        if (c > full) return -(static_cast<int>(c - col) / kNbrCols);
    }
    return static_cast<int>(c - col) / kNbrCols;
}

// The rest of a window that holds more than a list: adds the terms of the n entries in
// the column, searches on from candidate k of row cy until the column is full again, and
// so on, so that a warp's lanes evaluate their pairs together here too; its first kMaxNbr
// neighbours go to the list.  Returns false when it comes to a row that does not fit 16 bits.  With a support of 3 lattice spacings
// (28 neighbours, 81 candidates) the exact low-res density of 700,000 particles takes 123
// us without the list and 135 with it, of 4 spacings (50, 144) 156 and 168 us; a walk that
// evaluates at once took 125 and 203 us, and after a search that gave up 320 and 430 us.
template <class A, class Key>
__device__ __forceinline__ bool nbr_crowd(const Params& P, const ScaleView& S, const int* off, int dimx, int csx,
                                          int cex, int cy, int cey, int k, int i, float2 p, float T, int16_t* col,
                                          int n, float& sum, Key&& key) {
    int16_t* const full = col + (kMaxNbr + 1) * kNbrCols;
    int16_t* c = col + n * kNbrCols;
    int b = off[cy * dimx + cex + 1];
    bool fit = true, done = false;
    int m = 0;
    while (!done) {
        for (const int16_t* q = col; q < c; q += kNbrCols) {
            const int d = *q;
            sum += A::density(P, sq(sub(p, S.pos[i + d])));
            if (d != 0 && m < kMaxNbr) S.nbr[m++ * S.nbr_stride + i] = static_cast<int16_t>(d);
        }
        c = col;
        done = !fit || cy > cey;
        while (fit && cy <= cey && c <= full) {
            if (k + 3 < b) {
                const float x0 = key(k), x1 = key(k + 1), x2 = key(k + 2), x3 = key(k + 3);
                const auto put = [&](int j, float x) {
                    if (x <= T) {
                        *c = static_cast<int16_t>(j - i);
                        c += kNbrCols;
                    }
                };
                put(k, x0);
                put(k + 1, x1);
                put(k + 2, x2);
                put(k + 3, x3);
                k += 4;
            } else if (k < b) {
                if (key(k) <= T) {
                    *c = static_cast<int16_t>(k - i);
                    c += kNbrCols;
                }
                ++k;
            } else if (++cy <= cey) {
                k = off[cy * dimx + csx];
                b = off[cy * dimx + cex + 1];
                fit = k - i >= -32768 && b - i <= 32768;
            }
        }
    }
    return fit;
}

// Phase two: adds the terms of the n entries in the column to `sum`, in order, and
// writes the entries other than the particle itself to its neighbour list.  The column
// holds one entry more than the list; the particle itself is not always among them, for
// the relaxation moves children after the grid is built.  Only the entry past the last
// pair can be one too many (a bound tested at every entry put 1 % on a step of 1.0M +
// 1.0M particles).
template <class A>
__device__ __forceinline__ void nbr_density(const Params& P, const ScaleView& S, int i, float2 p, int n,
                                            const int16_t* col, float& sum) {
    int16_t* const first = S.nbr + i;  // 64-bit steps: a pool's capacity times kMaxNbr passes 2^31
    int16_t* dst = first;
    int m = 0;
    const auto entry = [&](int dj, float x) {
        sum += A::density(P, x);
        if (dj != 0) {
            *dst = static_cast<int16_t>(dj);
            dst += S.nbr_stride;
            ++m;
        }
    };
    int c = 0;
    for (; c + 1 < n; c += 2) {
        const int d0 = col[c * kNbrCols], d1 = col[(c + 1) * kNbrCols];
        const float x0 = sq(sub(p, S.pos[i + d0])), x1 = sq(sub(p, S.pos[i + d1]));
        entry(d0, x0);
        entry(d1, x1);
    }
    static_assert(kMaxNbr % 2 == 0, "entry kMaxNbr is not half of a pair");
    if (c < n) {
        const int d0 = col[c * kNbrCols];
        sum += A::density(P, sq(sub(p, S.pos[i + d0])));
        if (d0 != 0) {
            if (m < kMaxNbr) *dst = static_cast<int16_t>(d0);
            ++m;
        }
    }
    S.nnbr[i] = m <= kMaxNbr ? static_cast<uint8_t>(m) : kNbrCrowd;
}

// A same-scale neighbour's state as the force pass reads it.
struct NbrState {
    int k;
    float2 pos;
    float4 vq;
};
__device__ __forceinline__ NbrState fetch_nbr(const ScaleView& S, int k) { return NbrState{k, S.pos[k], S.vq[k]}; }

// The force pass's same-scale pairs: from the list when there is one (test and
// term take the neighbour's NbrState), else `walk`.  Two entries per trip: both
// neighbours' state is loaded before either pair is evaluated, in list order, and the
// next trip's entries before them too, so that no trip waits for its entries and then
// for its neighbours (the force kernels wait mostly on these loads).  An absent second
// entry is taken as offset 0, the particle itself, which every force test rejects.
// On a dam break of 1.0M + 1.0M particles, with a neighbour's velocity, p/rho^2 and
// rho in one vector instead of three arrays (ScaleView::vq), the low-res force took
// 97 -> 91 us (exact) and 68 -> 64 us (tolerance arithmetic), the high-res force 138 ->
// 130 and 91 -> 86 us; one entry per trip instead of two costs 13-18 % of the high-res
// force, four per trip 3-8 % (registers).  Two entries to a 32-bit word took 2 us off
// the low-res force and put 3-5 us on each density.
//
// A group of lanes takes an entry per lane, up to three rounds of entries loaded
// first.
//
// walk(on, from) takes the window's candidates from index `from` on: all of them without
// a list, those after the first kMaxNbr - 1 neighbours in a crowd (a group of lanes walks
// the whole window, 43 us a step of 5,000 such particles; the lists' part of a crowd put
// 1 % on the steps of short lists without one).  With a support of 3
// lattice spacings (28 neighbours) the exact low-res force of 700,000 particles takes 182
// us, against 324 where the whole window is walked; of 4 spacings (50) 371 and 442 us.
template <class G, class T, class Test, class Term, class Add, class Walk>
__device__ __forceinline__ void list_or_walk(bool on, const ScaleView& S, int i, Test&& test, Term&& term, Add&& add,
                                             T& sum, Walk&& walk) {
    int mark = S.nnbr[i];
    const int16_t* src = S.nbr + i;
    if constexpr (G::kLanes > 1) {
        constexpr int kRounds = (kMaxNbr + G::kLanes - 1) / G::kLanes;
        const int m = on && mark <= kMaxNbr ? mark : 0;
        int dj[kRounds];
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            const int c = r * G::kLanes + G::lane();
            dj[r] = c < m ? src[c * S.nbr_stride] : 0;
        }
#pragma unroll
        for (int r = 0; r < kRounds; ++r) {
            if (!G::any(r * G::kLanes < m)) break;
            const NbrState n0 = fetch_nbr(S, i + dj[r]);  // an absent entry is the particle itself: rejected
            T t{};
            const bool ok = r * G::kLanes + G::lane() < m && test(n0);
            if (ok) t = term(n0);
            G::add_lanes(G::ballot(ok), t, add, sum);
        }
        if (G::any(on && mark > kMaxNbr)) walk(on && mark > kMaxNbr);
    } else {
        const int nc = mark <= kMaxNbr ? mark : (mark == kNbrCrowd ? kMaxNbr - 1 : 0);
        int d0 = 0, d1 = 0;
        const auto next = [&](int c) {
            if (c < nc) d0 = *src;
            src += S.nbr_stride;
            d1 = 0;
            if (c + 1 < nc) d1 = *src;
            src += S.nbr_stride;
        };
        next(0);
        for (int c = 0; c < nc; c += 2) {
            const NbrState n0 = fetch_nbr(S, i + d0), n1 = fetch_nbr(S, i + d1);
            next(c + 2);
            if (test(n0)) add(sum, term(n0));
            if (test(n1)) add(sum, term(n1));
        }
        // the mark is loaded again (the index is hidden, or the compiler would keep it): one
        // register less in the list loop, without which the tolerance arithmetic's forces
        // took 4 % longer
        int again = i;
        asm("" : "+r"(again));
        mark = S.nnbr[again];
        if (mark > kMaxNbr) walk(true, mark == kNbrCrowd ? i + S.nbr[(kMaxNbr - 1) * S.nbr_stride + i] : 0);
    }
}

// A particle's same-scale density sum over its window (candidates k with key(k) <= T),
// which also records its neighbour list: in the two phases above, or, by a group of
// lanes, W candidates at a time.
template <class A, class G, class Key>
__device__ __forceinline__ void same_scale_density(bool on, const Params& P, const ScaleView& S, const int* off,
                                                   int dimx, int csx, int cex, int csy, int cey, int i, float2 p,
                                                   float T, int16_t* nbr_col, float& sum, Key&& key) {
    if constexpr (G::kLanes > 1) {
        int n = 0;
        bool fit = true;
        for (int cy = csy; G::any(on && cy <= cey); ++cy) {
            const int row = cy * dimx;
            const bool in = on && cy <= cey;
            const int a = in ? off[row + csx] : 0, b = in ? off[row + cex + 1] : 0;
            if (in && (a - i < -32768 || b - i > 32768)) fit = false;
            for (int base = a; G::any(base < b); base += G::kLanes) {
                const int k = base + G::lane();
                const float x = k < b ? key(k) : INFINITY;
                const bool ok = x <= T;
                const unsigned m = G::ballot(ok);
                const int own = i - base;  // the particle itself is left out of the list
                const unsigned listed = own >= 0 && own < G::kLanes ? m & ~(1u << own) : m;
                if (ok && k != i) {
                    const int c = n + __popc(listed & ((1u << G::lane()) - 1u));
                    if (c < kMaxNbr && fit) S.nbr[c * S.nbr_stride + i] = static_cast<int16_t>(k - i);
                }
                n += __popc(listed);
                G::add_lanes(m, ok ? A::density(P, x) : 0.0f, add_density, sum);
            }
        }
        if (on && G::leader()) S.nnbr[i] = fit ? (n <= kMaxNbr ? static_cast<uint8_t>(n) : kNbrCrowd) : kNbrOverflow;
    } else {
        int cy = csy, at = 0;
        // the lanes leave the search at different candidates; without a barrier here those
        // with too many went on alone (123 -> 195 us in the example at nbr_crowd)
        const unsigned together = __activemask();
        const int n = nbr_search(off, dimx, csx, cex, cy, cey, at, i, T, nbr_col, key);
        __syncwarp(together);
        if (n >= 0) {
            nbr_density<A>(P, S, i, p, n, nbr_col, sum);
            return;
        }
        S.nnbr[i] = kNbrCrowd;
        if (n == kNbrFar || !nbr_crowd<A>(P, S, off, dimx, csx, cex, cy, cey, at, i, p, T, nbr_col, -n, sum, key)) {
            S.nnbr[i] = kNbrOverflow;
            float x = 0.0f;
            sum = 0.0f;
            G::window(
                true, off, dimx, csx, cex, csy, cey,
                [&](int k) {
                    x = key(k);
                    return x <= T;
                },
                [&](int) { return A::density(P, x); }, add_density, sum);
        }
    }
}

// ---------------------------------------------------------------------------
// High-res density + Tait, computeParticleDensityPressureHigh (WCSPHSolver.cu:1426-1516)
// ---------------------------------------------------------------------------
template <class A, class G>
__device__ __forceinline__ void density_high_one(const Params& P, const StepView& V, int i, bool valid, bool hstate0,
                                                 int16_t* nbr_col) {
    const ScaleView& H = V.H;
    const ScaleView& L = V.L;
    const int* offH = H.off + P.cbH;
    const int* offL = L.off + P.cbL;
    const float2 p = H.pos[i];
    const unsigned s = H.st[i];
    float d = 0.0f, dl = 0.0f;
    float x = 0.0f;
    const auto term = [&](int) { return A::density(P, x); };
    int csx, csy, cex, cey;
    grid_coord_s<1>(P, p.x, p.y, -P.rh, csx, csy);
    grid_coord_s<1>(P, p.x, p.y, P.rh, cex, cey);
    // a candidate the lambda mask rejects gets key +inf: no cutoff passes it (the mask
    // passes every candidate of a state-1 particle)
    const auto masked = [&](int k) { return lamHH(s, H.st[k]) ? sq(sub(p, H.pos[k])) : INFINITY; };
    const auto plain = [&](int k) { return sq(sub(p, H.pos[k])); };
    if (!G::any((s & 1u) == 0u))
        same_scale_density<A, G>(valid, P, H, offH, P.dimH[0], csx, cex, csy, cey, i, p, P.Tle_rh, nbr_col, d, plain);
    else
        same_scale_density<A, G>(valid, P, H, offH, P.dimH[0], csx, cex, csy, cey, i, p, P.Tle_rh, nbr_col, d, masked);
    grid_coord_s<0>(P, p.x, p.y, -P.r, csx, csy);
    grid_coord_s<0>(P, p.x, p.y, P.r, cex, cey);
    // With no high-res entry in state 0 in this step (hstate0 false), a state-1
    // particle's Q1 term can take only never-created slots (position (0,0), state 0:
    // lambda_HL rejects every existing state-1 entry), and those only when the
    // particle lies within r_h of (0,0): otherwise the walk adds nothing and is
    // skipped -- the same terms, none.
    const bool q1_live = hstate0 || (s & 1u) == 0u || sq(p) <= P.Tle_rh;
    const bool q1 = valid && P.q1 && q1_live;
    if (G::any(q1)) {
        // The reference reads the HIGH sorted list at LOW-grid ranges of its own
        // scene; past the scene's n_high that list still holds its initial identity
        // (slot t at position t).  A row's range [a, b) of low-list positions t
        // (t - baseL >= 0: offsets only grow) is taken in two runs, in order: the
        // positions below baseL + n_high, which are the high-list entries
        // t - baseL + baseH, and the rest, through the slot map.
        const int baseL = offL[0], baseH = offH[0];
        const int nHs = offH[P.CHs] - baseH;
        const int tH = baseL + nHs;   // first position past the scene's high-res list
        const int dH = baseH - baseL;  // low-list position -> high-list entry
        for (int cy = csy; G::any(q1 && cy <= cey); ++cy) {
            const int row = cy * P.dimL[0];
            const bool in = q1 && cy <= cey;
            const int a = in ? offL[row + csx] : 0, b = in ? offL[row + cex + 1] : 0;
            const int m = min(b, max(a, tH));
            G::span(
                a + dH, m + dH,
                [&](int k) {
                    if (!lamHL(s, H.st[k])) return false;
                    x = sq(sub(p, H.pos[k]));
                    return x <= P.Tle_rh;
                },
                term, add_density, d);
            G::span(
                m, b,
                [&](int t) {
                    const int tl = t - baseL;
                    const int slot = 4 * P.sbL + tl;
                    const int k = (tl < 4 * P.nLs && slot < P.slotsH) ? H.map[slot] : -1;
                    float2 pj = make_float2(0.0f, 0.0f);
                    unsigned sj = 0;
                    if (k >= 0) {
                        pj = H.pos[k];
                        sj = H.st[k];
                    }
                    if (!lamHL(s, sj)) return false;
                    x = sq(sub(p, pj));
                    return x <= P.Tle_rh;
                },
                term, add_density, d);
        }
    }
    if (G::any(valid && !P.q1)) {
        G::window(
            valid && !P.q1, offL, P.dimL[0], csx, cex, csy, cey,
            [&](int k) {
                if (!lamHL(s, L.st[k])) return false;
                x = sq(sub(p, L.pos[k]));
                return x <= P.Tle_rh;
            },
            term, add_density, dl);
    }
    d *= P.mH;
    dl *= P.mL;
    d += dl;
    const float pr = tait(d, P);
    if (valid && G::leader()) {
        H.dens[i] = d;
        H.pres[i] = pr;
        *reinterpret_cast<float2*>(&H.vq[i].z) = make_float2(pr / (d * d), d);
        if (!isfinite(d) || !isfinite(pr)) atomicOr(&V.cnt->err, kErrNumeric);
    }
}

template <bool B, class G, class A>
__global__ void __launch_bounds__(256, B ? (A::kFast ? 6 : 5) : (A::kFast ? 8 : 6)) k_density_high(Params P0, StepView V) {
    __shared__ int16_t s_nbr[G::kLanes > 1 ? 1 : kNbrRows * kNbrCols];
    int16_t* const nbr_col = s_nbr + (G::kLanes > 1 ? 0 : threadIdx.x);
    const bool hstate0 = V.cnt->h_state0 != 0;
    by_size<G, false>(V.cnt->cur[1], [&](auto form, int n) {
        using F = decltype(form);
        for_each_particle<F>(n, [&](int i, bool valid) {
            if constexpr (B) {
                const Params& P = V.table[V.scH[i]];
                density_high_one<A, F>(P, V, i, valid, hstate0, nbr_col);
            } else {
                density_high_one<A, F>(P0, V, i, valid, hstate0, nbr_col);
            }
        });
    });
}

// ---------------------------------------------------------------------------
// Wall term of a force sum (updateAccCell 562-579 / updateAccCellComplementHigh
// 867-884): every wall particle of the window's cells, in cell order.  Pairs with
// sqrtf(x) > rad have q >= 2 and add exactly zero, so they are skipped.  S selects
// the scale: 0 the low-res radius r, 1 the high-res radius rh.  `cell`: the particle's
// cell of the low-res grid.
// ---------------------------------------------------------------------------
template <class A, class G, int S>
__device__ __forceinline__ float2 wall_sum(bool on, const Params& P, const StepView& V, float2 p, int cell) {
    float2 accB = make_float2(0.f, 0.f);
    // the window reaches at most two cells from the particle's own (near_cells): with no
    // wall particle within two cells of that, the sum is empty
    on = on && (!P.near_cells || V.wnear[P.cbL + cell]);
    if (!G::any(on)) return accB;
    int csx, csy, cex, cey;
    grid_coord_s<0>(P, p.x, p.y, -P.r, csx, csy);
    grid_coord_s<0>(P, p.x, p.y, P.r, cex, cey);
    const float Tle = S ? P.Tle_rh : P.Tle_r, cB = S ? P.cBH : P.cBL;
    const float2* wpos = V.wpos + P.wb;
    float2 pik = make_float2(0.f, 0.f);
    float x = 0.0f;
    G::window(
        on, V.woff + P.cbL, P.dimL[0], csx, cex, csy, cey,
        [&](int k) {
            pik = sub(p, wpos[k]);
            x = sq(pik);
            return !(x > Tle);  // NaN passes: the reference's 0 * NaN offset propagates it
        },
        [&](int) { return A::template wall<S>(P, pik, x, cB); },
        [](float2& a, float2 t) {
            a.x += t.x;
            a.y += t.y;
        },
        accB);
    return accB;
}

// The wall terms of lists short enough for groups of lanes.  They need the positions
// alone, so blocks of their own take them in the low-res density's launch, and the force
// reads them (acc holds them until it writes the accelerations).  A particle near a wall
// has some 36 candidates and 20 pairs there, and a short list's step waits for it.
// A step took, with the tether radius out of FP64 too, 37.2 -> 34.8 us at 5,000
// particles (34.8 -> 31.9 us a step of a graph of eight), 43.6 -> 39.6 us at 22,000
// (tolerance arithmetic).  A long list's step hides its walls' warps; taken here they
// made one of 1.0M low-res particles slower (180 -> 183 us), as did a launch of their
// own beside the densities for the steps of graphs of several (34.4 -> 36.4 us).
template <bool B, class A, int S>
__device__ __forceinline__ void wall_scale(const Params& P0, const StepView& V, const ScaleView& X, const uint16_t* sc,
                                           int block, int blocks) {
    using G = PerGroup<8>;
    const int n = V.cnt->cur[S];
    if (n > kForce4Max) return;
    const auto one = [&](const Params& P, int i, bool valid) {
        const float2 p = X.pos[i];
        const float2 accB = wall_sum<A, G, S>(valid, P, V, p, cell_hash_s<0>(P, p));
        if (valid && G::leader()) X.acc[i] = accB;
    };
    for_each_particle<G>(n, block, blocks, [&](int i, bool valid) {
        if constexpr (B) one(V.table[sc[i]], i, valid);
        else one(P0, i, valid);
    });
}

template <class A, class G, int S>
__device__ __forceinline__ float2 wall_term(bool valid, const Params& P, const StepView& V, const ScaleView& X, int i,
                                            float2 p, int cell) {
    if constexpr (G::kLanes == 8 || G::kLanes == 4) return X.acc[i];  // by_size's lists: wall_scale
    else return wall_sum<A, G, S>(valid, P, V, p, cell);
}

// ---------------------------------------------------------------------------
// Low-res density + Tait, computeParticleDensityPressure (WCSPHSolver.cu:1342-1424)
// ---------------------------------------------------------------------------
template <class A, class G>
__device__ __forceinline__ void density_low_one(const Params& P, const StepView& V, int i, bool valid, bool cross,
                                                int16_t* nbr_col) {
    const ScaleView& H = V.H;
    const ScaleView& L = V.L;
    const float2 p = L.pos[i];
    const unsigned s = L.st[i];
    float d = 0.0f, dh = 0.0f;
    float x = 0.0f;
    const auto term = [&](int) { return A::density(P, x); };
    int csx, csy, cex, cey;
    grid_coord_s<0>(P, p.x, p.y, -P.r, csx, csy);
    grid_coord_s<0>(P, p.x, p.y, P.r, cex, cey);
    same_scale_density<A, G>(valid, P, L, L.off + P.cbL, P.dimL[0], csx, cex, csy, cey, i, p, P.Tle_r, nbr_col, d,
                             [&](int k) { return sq(sub(p, L.pos[k])); });
    if (cross) {  // only state-0 high-res particles can contribute (lambda_LH)
        grid_coord_s<1>(P, p.x, p.y, -P.r, csx, csy);
        grid_coord_s<1>(P, p.x, p.y, P.r, cex, cey);
        G::window(
            valid, H.off + P.cbH, P.dimH[0], csx, cex, csy, cey,
            [&](int k) {
                if (!lamLH(s, H.st[k])) return false;
                x = sq(sub(p, H.pos[k]));
                return x <= P.Tle_r;
            },
            term, add_density, dh);
    }
    d *= P.mL;
    dh *= P.mH;
    const float rho = d + dh;
    const float pr = tait(rho, P);
    if (valid && G::leader()) {
        L.dens[i] = rho;
        L.pres[i] = pr;
        *reinterpret_cast<float2*>(&L.vq[i].z) = make_float2(pr / (rho * rho), rho);
        if (!isfinite(rho) || !isfinite(pr)) atomicOr(&V.cnt->err, kErrNumeric);
    }
}

template <bool B, class G, class A>
__global__ void __launch_bounds__(256, B ? 6 : 8) k_density_low(Params P0, StepView V) {
    __shared__ int16_t s_nbr[G::kLanes > 1 ? 1 : kNbrRows * kNbrCols];
    int16_t* const nbr_col = s_nbr + (G::kLanes > 1 ? 0 : threadIdx.x);
    const int blocks = gridDim.x - V.wallL - V.wallH;  // then the walls' blocks
    const int block = static_cast<int>(blockIdx.x);
    if (block >= blocks) {
        if (block < blocks + V.wallL) wall_scale<B, A, 0>(P0, V, V.L, V.scL, block - blocks, V.wallL);
        else wall_scale<B, A, 1>(P0, V, V.H, V.scH, block - blocks - V.wallL, V.wallH);
        return;
    }
    const bool cross = V.cnt->h_state0 != 0;
    // the split counts of the low-res force's tiles, zero before it
    for (int t = block * blockDim.x + threadIdx.x; t < (V.cnt->cur[0] + kSplitTile - 1) / kSplitTile;
         t += blocks * blockDim.x)
        V.split_tile[t] = 0u;
    by_size<G, false>(V.cnt->cur[0], [&](auto form, int n) {
        using F = decltype(form);
        for_each_particle<F>(n, block, blocks, [&](int i, bool valid) {
            if constexpr (B) {
                const Params& P = V.table[V.scL[i]];
                density_low_one<A, F>(P, V, i, valid, cross, nbr_col);
            } else {
                density_low_one<A, F>(P0, V, i, valid, cross, nbr_col);
            }
        });
    });
}

// ---------------------------------------------------------------------------
// Low-res force + advance + split test: computeParticleAcceleration
// (WCSPHSolver.cu:1648-1865) with advance (1604-1646) fused; its predicted position
// is the advanced position bit for bit.  The fluid and wall sums are independent
// accumulators.  The new position also gives the entry's
// key for the next step's grid.  Returns the split flag.
// ---------------------------------------------------------------------------
template <class A, class G>
__device__ __forceinline__ bool force_low_one(const Params& P, const StepView& V, int i, bool valid, bool cross,
                                              bool deleted) {
    const ScaleView& H = V.H;
    const ScaleView& L = V.L;
    const float4 own = L.vq[i];
    float2 p = L.pos[i], v = vel_of(own);
    const unsigned s = L.st[i];
    const float qi = own.z, dens = own.w;
    PairTerms fl{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};  // (acc, accT)
    float2 pij = make_float2(0.f, 0.f);
    float x = 0.0f;
    int csx, csy, cex, cey;  // found where they are used: few values live through the list loop
    {
        const auto test = [&](int k) {
            pij = sub(p, L.pos[k]);
            x = sq(pij);
            return x != 0.0f && x <= P.Tlt_r && notDeleted(L.st[k]);
        };
        const auto term = [&](int j) {
            const float4 o = L.vq[j];
            return A::template pair<kHLow>(P, pij, x, sub(v, vel_of(o)), qi, o.z, dens, o.w);
        };
        const auto test_n = [&](const NbrState& n) {
            pij = sub(p, n.pos);
            x = sq(pij);
            return x != 0.0f && x <= P.Tlt_r && (!deleted || notDeleted(L.st[n.k]));
        };
        const auto term_n = [&](const NbrState& n) {
            return A::template pair<kHLow>(P, pij, x, sub(v, vel_of(n.vq)), qi, n.vq.z, dens, n.vq.w);
        };
        list_or_walk<G>(valid, L, i, test_n, term_n, add_terms, fl, [&](bool on, auto... from) {
            grid_coord_s<0>(P, p.x, p.y, -P.r, csx, csy);
            grid_coord_s<0>(P, p.x, p.y, P.r, cex, cey);
            G::window(on, L.off + P.cbL, P.dimL[0], csx, cex, csy, cey, test, term, add_terms, fl, from...);
        });
    }
    const int cell = cell_hash_s<0>(P, p);
    const float2 accB = wall_term<A, G, 0>(valid, P, V, L, i, p, cell);
    PairTerms fh{make_float2(0.f, 0.f), fl.t};  // (accH, accT): the sigma sum continues
    if (cross) {
        grid_coord_s<1>(P, p.x, p.y, -P.r, csx, csy);
        grid_coord_s<1>(P, p.x, p.y, P.r, cex, cey);
        G::window(
            valid, H.off + P.cbH, P.dimH[0], csx, cex, csy, cey,
            [&](int k) {
                if (!lamLH(s, H.st[k])) return false;
                pij = sub(p, H.pos[k]);
                x = sq(pij);
                return x != 0.0f && x <= P.Tlt_r;
            },
            [&](int j) {
                const float4 o = H.vq[j];
                return A::template pair<kHCross>(P, pij, x, sub(v, vel_of(o)), qi, o.z, dens, o.w);
            },
            add_terms, fh);
    }
    float2 acc = fl.a, accH = fh.a;
    const float2 accT = fh.t;
    acc.x *= -P.mL;
    acc.y *= -P.mL;
    accH.x *= -P.mH;
    accH.y *= -P.mH;
    acc.x += accH.x;
    acc.y += accH.y;
    acc.x -= P.sigma * accT.x;
    acc.y -= P.sigma * accT.y;
    acc.x += accB.x;
    acc.y += accB.y;
    acc.y -= P.g;
    v.x += P.dt * acc.x;
    v.y += P.dt * acc.y;
    p.x += P.dt * v.x;
    p.y += P.dt * v.y;
    // split test on the predicted position (computeParticleAcceleration 1810-1835)
    // against the ROI of this step; with TSS_FLAG_MERGE a split parent outside it
    // merges back
    const float kf = static_cast<float>(V.cnt->steps - P.step0);
    const float rx0 = P.roi[0] + kf * P.roi_vdt[0], rx1 = P.roi[2] + kf * P.roi_vdt[0];
    const float ry0 = P.roi[1] + kf * P.roi_vdt[1], ry1 = P.roi[3] + kf * P.roi_vdt[1];
    const bool in_roi = rx0 < p.x && p.x < rx1 && ry0 < p.y && p.y < ry1;
    bool flag = false;
    uint8_t ns = static_cast<uint8_t>(s);
    if (s == 0u && in_roi) {
        ns = 1;
        flag = true;
    } else if (P.merge && s == 1u && !in_roi) {
        ns = 0;
    }
    if (valid && G::leader()) {
        L.acc[i] = acc;
        if (!isfinite(acc.x) || !isfinite(acc.y)) atomicOr(&V.cnt->err, kErrNumeric);
        // a split parent's tether radius (adjustPosition, WCSPHSolver.cu:1007-1022), once
        // per parent here instead of once per child in the high-res force.  min(dist,
        // float(R)) == float(min(dist, R)) for a float dist (rounding is monotone), so
        // the children's clamp is unchanged bit for bit.
        if (s == 1u) L.tr[i] = tether_radius(P, dens);
        // the cells of this step's grid that hold an entry in state 0 after the split
        // marks: the only low-res partners of a state-1 child in the high-res force.
        // The entry's cell is the one its key was made from (its position at the
        // start of the step, the same cell function).
        if (ns == 0u) L.cflag[P.cbL + cell] = static_cast<uint8_t>(V.cnt->steps);
        L.npos[i] = p;
        L.nvel[i] = v;
        L.nid[i] = L.id[i];
        grid_key(L.gcount, L.gkey, L.grank, L.gtile, i,
                 P.cbL + cell_hash_s<0>(P, p));
        L.nst[i] = ns;
        V.split_flag[i] = flag ? 1 : 0;
        if (L.ndens) {
            L.ndens[i] = dens;
            L.npres[i] = L.pres[i];
        }
    }
    return flag;
}

// A warp-uniform loop (every lane makes the same number of trips, lanes past n
// inactive) so the ballot that feeds the split compaction sees whole warps; a warp's
// particles lie in one compaction tile (kSplitTile % 32 == 0).
// 48 registers (five blocks per SM) in both forms of the exact arithmetic, 40 (six) in
// the tolerance arithmetic's single-scene form; one block per SM more or fewer was slower.
// The kernel holds the forms for short lists too
// (by_size), and they share the register bound with the long lists' form: it spills 124 /
// 160 bytes (stores / loads) in the exact arithmetic and 88 / 140 in the tolerance one,
// batched 420 / 680 and 164 / 164; without the short forms it would be 48 / 48, 16 / 16,
// 220 / 204 and 36 / 40.
template <bool B, class G, class A>
__global__ void __launch_bounds__(256, (A::kFast && !B) ? 6 : 5) k_force_low(Params P0, StepView V) {
    let_next_start();
    const int n = V.cnt->cur[0];
    const bool cross = V.cnt->h_state0 != 0, deleted = V.cnt->l_deleted != 0;
    by_size<G, true>(n, [&](auto form, int) {
        using F = decltype(form);
        const auto one = [&](int i, bool valid) {
            if constexpr (B) {
                const Params& P = V.table[V.scL[i]];
                return force_low_one<A, F>(P, V, i, valid, cross, deleted);
            } else {
                return force_low_one<A, F>(P0, V, i, valid, cross, deleted);
            }
        };
        const int lane = threadIdx.x & 31;
        if constexpr (F::kLanes > 1) {
            for_each_particle<F>(n, [&](int i, bool valid) {
                const bool flag = one(i, valid);
                const unsigned m = __ballot_sync(0xffffffffu, flag && valid && F::leader());
                // the warp's particles are neighbours; lane 0 has the first of them
                if (lane == 0 && m) atomicAdd(&V.split_tile[i / kSplitTile], __popc(m));
            });
        } else {
            for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
                const int i = base + threadIdx.x;
                const bool flag = i < n && one(i, true);
                const unsigned m = __ballot_sync(0xffffffffu, flag);
                if (lane == 0 && m) atomicAdd(&V.split_tile[(base + (threadIdx.x & ~31)) / kSplitTile], __popc(m));
            }
        }
    });
}

// ---------------------------------------------------------------------------
// High-res force + integrate + tether: computeParticleAccelerationAndAdvanceHigh
// (WCSPHSolver.cu:1867-2033) and adjustOrInjectTransientHighD (1097-1172).
// Reads see the pre-step state (the reference integrates in place, a data race);
// low-res states are read after this step's split marks, as in the reference.
// ---------------------------------------------------------------------------
template <class A, class G>
__device__ __forceinline__ void force_high_one(const Params& P, const StepView& V, int i, bool valid) {
    const ScaleView& H = V.H;
    const ScaleView& L = V.L;
    const float4 own = H.vq[i];
    float2 p = H.pos[i], v = vel_of(own);
    const unsigned s = H.st[i];
    const float qi = own.z, dens = own.w;
    PairTerms fh{make_float2(0.f, 0.f), make_float2(0.f, 0.f)};  // (acc, accT)
    float2 pij = make_float2(0.f, 0.f);
    float x = 0.0f;
    int csx, csy, cex, cey;
    {
        const auto test = [&](int k) {
            if (!lamHH(s, H.st[k])) return false;
            pij = sub(p, H.pos[k]);
            x = sq(pij);
            return x != 0.0f && x <= P.Tlt_rh;
        };
        const auto term = [&](int j) {
            const float4 o = H.vq[j];
            return A::template pair<kHHigh>(P, pij, x, sub(v, vel_of(o)), qi, o.z, dens, o.w);
        };
        const auto test_n = [&](const NbrState& n) {
            pij = sub(p, n.pos);
            x = sq(pij);
            return x != 0.0f && x <= P.Tlt_rh && ((s & 1u) || lamHH(s, H.st[n.k]));
        };
        const auto term_n = [&](const NbrState& n) {
            return A::template pair<kHHigh>(P, pij, x, sub(v, vel_of(n.vq)), qi, n.vq.z, dens, n.vq.w);
        };
        list_or_walk<G>(valid, H, i, test_n, term_n, add_terms, fh, [&](bool on, auto... from) {
            grid_coord_s<1>(P, p.x, p.y, -P.rh, csx, csy);
            grid_coord_s<1>(P, p.x, p.y, P.rh, cex, cey);
            G::window(on, H.off + P.cbH, P.dimH[0], csx, cex, csy, cey, test, term, add_terms, fh, from...);
        });
    }
    const float2 accB = wall_term<A, G, 1>(valid, P, V, H, i, p, cell_hash_s<0>(P, p));
    const int id = H.id[i];
    const int parent = id >> 2;
    int pi = parent >= 0 && parent < P.slotsL ? L.map[parent] : -1;
    if (pi >= 0 && L.st[pi] != 1) pi = -1;  // not a split parent
    grid_coord_s<0>(P, p.x, p.y, -P.r, csx, csy);
    grid_coord_s<0>(P, p.x, p.y, P.r, cex, cey);
    // up to here, nothing of this step's low-res force: this kernel starts while that one's
    // last blocks run.  (The wall term, the parent and the window on this side of the wait:
    // a step of 2,000 particles 30.7 -> 30.1 us, 1.0M + 1.0M in the tolerance arithmetic
    // 277 -> 275 us.)  From here, what it wrote
    wait_for_previous();
    PairTerms fl{make_float2(0.f, 0.f), fh.t};  // (accL, accT): the sigma sum continues
    // A state-1 child pairs only with low-res entries in state 0 (lambda_HL and
    // notDeleted); a row of the window whose cells the low-res force did not stamp
    // in this step holds none, and is skipped.
    const bool odd = (s & 1u) != 0u;
    const uint8_t stamp = static_cast<uint8_t>(V.cnt->steps);
    G::window_if(
        valid, L.off + P.cbL, P.dimL[0], csx, cex, csy, cey,
        [&](int row) {
            if (!odd) return true;
            const uint8_t* f = L.cflag + P.cbL + row;
            for (int cx = csx; cx <= cex; ++cx)
                if (f[cx] == stamp) return true;
            return false;
        },
        [&](int k) {
            const unsigned sj = L.nst[k];  // low-res states after this step's split marks
            if (!(lamHL(s, sj) && notDeleted(sj))) return false;
            pij = sub(p, L.pos[k]);
            x = sq(pij);
            return x != 0.0f && x <= P.Tlt_r;
        },
        [&](int j) {
            const float4 o = L.vq[j];
            return A::template pair<kHCross>(P, pij, x, sub(v, vel_of(o)), qi, o.z, dens, o.w);
        },
        add_terms, fl);
    float2 acc = fh.a, accL = fl.a;
    const float2 accT = fl.t;
    acc.x *= -P.mH;
    acc.y *= -P.mH;
    accL.x *= -P.mL;
    accL.y *= -P.mL;
    acc.x -= P.sigma * accT.x;
    acc.y -= P.sigma * accT.y;
    acc.x += accL.x;
    acc.y += accL.y;
    acc.x += accB.x;
    acc.y += accB.y;
    acc.y -= P.g;
    v.x += P.dt * acc.x;
    v.y += P.dt * acc.y;
    p.x += P.dt * v.x;
    p.y += P.dt * v.y;
    // tether to the parent after the parent's advance (adjustPosition, 1007-1022);
    // with TSS_FLAG_MERGE the children of a parent that merged back in this step
    // are removed instead
    const bool drop = P.merge && pi >= 0 && L.nst[pi] == 0;
    if (pi >= 0 && !drop) {
        const float2 pl = L.npos[pi];
        const float2 pji = sub(p, pl);
        const float dist = vnorm(pji);
        const float lim = fminf(dist, L.tr[pi]);  // the parent's radius, from the low-res force
        if (!(P.tether_guard && dist == 0.0f)) {  // guarded: a child on its parent stays there
            p.x = pl.x + lim / dist * pji.x;
            p.y = pl.y + lim / dist * pji.y;
        }
    }
    if (!valid || !G::leader()) return;
    H.acc[i] = acc;
    if (!isfinite(acc.x) || !isfinite(acc.y)) atomicOr(&V.cnt->err, kErrNumeric);
    H.npos[i] = p;
    H.nvel[i] = v;
    H.nst[i] = static_cast<uint8_t>(drop ? 2u : s);
    H.nid[i] = id;
    if (drop) {  // out of the next grid build, and of the slot map
        H.gkey[i] = -1;
        H.map[id] = -1;
        atomicAdd(&V.cnt->n_drop, 1);
    } else {
        grid_key(H.gcount, H.gkey, H.grank, H.gtile, i, P.cbH + cell_hash_s<1>(P, p));
    }
    if (H.ndens) {
        H.ndens[i] = dens;
        H.npres[i] = H.pres[i];
    }
}

// Registers: 48 (five blocks per SM) in the exact arithmetic's single-scene form and the
// tolerance arithmetic's batched one, 40 (six) and 64 (four) in the other two.  On a dam
// break of 1.0M + 1.0M particles five blocks took 130 us and four 140 (exact), six 86 and
// five 90.5 (tolerance), and one more was slower too.  The batched form reads
// each particle's parameters from the scene table, which is what its registers go to.
// Spills, with the forms for short lists in the same kernel (see k_force_low): 240 / 356
// bytes exact, 128 / 212 in the tolerance arithmetic, batched 40 / 116 and 188 / 224;
// without the short forms 80 / 92, 8 / 8, 28 / 32 and 52 / 56.
template <bool B, class G, class A>
__global__ void __launch_bounds__(256, B ? (A::kFast ? 5 : 4) : (A::kFast ? 6 : 5)) k_force_high(Params P0, StepView V) {
    by_size<G, true>(V.cnt->cur[1], [&](auto form, int n) {
        using F = decltype(form);
        for_each_particle<F>(n, [&](int i, bool valid) {
            if constexpr (B) {
                const Params& P = V.table[V.scH[i]];
                force_high_one<A, F>(P, V, i, valid);
            } else {
                force_high_one<A, F>(P0, V, i, valid);
            }
        });
    });
}

// ---------------------------------------------------------------------------
// Host side: launch gather g (0 high-res density, 1 low-res density, 2 low-res
// force, 3 high-res force) in arithmetic A, and its occupancy.
// ---------------------------------------------------------------------------
template <class A, bool B, class G>
void launch_gather_bg(int g, int blocks, int threads, cudaStream_t s, const Params& P, const StepView& V) {
    switch (g) {
        case 0:
            k_density_high<B, G, A><<<blocks, threads, 0, s>>>(P, V);
            break;
        case 1:
            k_density_low<B, G, A><<<blocks + V.wallL + V.wallH, threads, 0, s>>>(P, V);
            break;
        case 2:
            k_force_low<B, G, A><<<blocks, threads, 0, s>>>(P, V);
            break;
        case 3:
            launch_after(k_force_high<B, G, A>, blocks, threads, s, P, V);
            break;
        default:
            break;
    }
}

template <class A>
void launch_gather_a(int g, bool batched, bool warp, int blocks, int threads, cudaStream_t s, const Params& P,
                     const StepView& V) {
    if (batched) {
        if (warp)
            launch_gather_bg<A, true, PerWarp>(g, blocks, threads, s, P, V);
        else
            launch_gather_bg<A, true, PerThread>(g, blocks, threads, s, P, V);
    } else {
        if (warp)
            launch_gather_bg<A, false, PerWarp>(g, blocks, threads, s, P, V);
        else
            launch_gather_bg<A, false, PerThread>(g, blocks, threads, s, P, V);
    }
}

template <class K>
int occupancy_of(K kernel, int threads) {
    int n = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0) == cudaSuccess ? n : 0;
}

template <class A, bool B, class G>
int gather_occupancy_bg(int g, int threads) {
    switch (g) {
        case 0:
            return occupancy_of(k_density_high<B, G, A>, threads);
        case 1:
            return occupancy_of(k_density_low<B, G, A>, threads);
        case 2:
            return occupancy_of(k_force_low<B, G, A>, threads);
        case 3:
            return occupancy_of(k_force_high<B, G, A>, threads);
        default:
            return 0;
    }
}

template <class A>
int gather_occupancy_a(int g, bool batched, bool warp, int threads) {
    if (batched)
        return warp ? gather_occupancy_bg<A, true, PerWarp>(g, threads) : gather_occupancy_bg<A, true, PerThread>(g, threads);
    return warp ? gather_occupancy_bg<A, false, PerWarp>(g, threads) : gather_occupancy_bg<A, false, PerThread>(g, threads);
}

}  // namespace tss
