// gather.cuh -- the ways a gather walks one particle's cell window.
//
// PerThread: one particle per thread, 32 particles per warp.  Each thread walks its
// window's rows in order, testing each candidate and evaluating an accepted pair
// at once.  This is the throughput form: consecutive threads walk overlapping
// windows, so neighbour loads are shared through L1.  The same-scale sums, which
// are most of the work, are taken from lists instead (nbr_search, gathers.cuh).
//
// PerGroup<W>: one particle per W lanes (W = 32: one per warp).  The lanes test W
// consecutive candidates of a row at a time and evaluate the accepted pairs' terms
// in parallel; then every lane adds the terms in candidate order, taking each from
// the lane that evaluated it (warp shuffles), so every lane ends with the per-thread
// sum, bit for bit.  A rejected candidate's term is +0: a sum that starts at +0 never
// becomes -0 under round-to-nearest, so adding +0 changes no bit of it.  For lists
// too short to fill the GPU, where a step is bound by each thread's chain of
// dependent loads rather than by instruction issue.
//
// A gather is written once against the policy G: G::window / G::window_if /
// G::span take the candidate test (which may leave state for the term: a
// candidate's term is evaluated right after its test by the same lane), the pair
// term, the accumulation, and the running sum.  The groups of a warp stay in step,
// so that the shuffles are whole-warp ones: a sum that only some particles need is
// called for all of them under G::any(needed), with `on` = needed.  Per-particle
// results are stored by G::leader() only.
#pragma once
#include "tss_device.cuh"

namespace tss {

__device__ __forceinline__ float shfl_from(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float2 shfl_from(float2 v, int src) {
    return make_float2(shfl_from(v.x, src), shfl_from(v.y, src));
}
__device__ __forceinline__ PairTerms shfl_from(const PairTerms& v, int src) {
    return PairTerms{shfl_from(v.a, src), shfl_from(v.t, src)};
}

struct PerThread {
    static constexpr int kLanes = 1;
    __device__ __forceinline__ static bool leader() { return true; }
    __device__ __forceinline__ static bool any(bool c) { return c; }

    // the candidates [a, b), in order
    template <class T, class Test, class Term, class Add>
    __device__ __forceinline__ static void span(int a, int b, Test&& test, Term&& term, Add&& add, T& sum) {
        for (int k = a; k < b; ++k)
            if (test(k)) add(sum, term(k));
    }

    // the rows cy of the window for which live(row) holds (row = cy * dimx), candidates
    // below `from` left out.  A row left out must hold no candidate that passes the test:
    // the sum is the same.
    template <class T, class Live, class Test, class Term, class Add>
    __device__ __forceinline__ static void window_if(bool on, const int* off, int dimx, int csx, int cex, int csy,
                                                     int cey, Live&& live, Test&& test, Term&& term, Add&& add,
                                                     T& sum, int from = 0) {
        if (!on) return;
        for (int cy = csy; cy <= cey; ++cy) {
            const int row = cy * dimx;
            if (live(row)) span(max(off[row + csx], from), off[row + cex + 1], test, term, add, sum);
        }
    }

    template <class T, class Test, class Term, class Add>
    __device__ __forceinline__ static void window(bool on, const int* off, int dimx, int csx, int cex, int csy, int cey,
                                                  Test&& test, Term&& term, Add&& add, T& sum, int from = 0) {
        window_if(on, off, dimx, csx, cex, csy, cey, [](int) { return true; }, test, term, add, sum, from);
    }
};

template <int W>
struct PerGroup {
    static_assert(W == 4 || W == 8 || W == 16 || W == 32, "a group is a power of two lanes of a warp");
    static constexpr int kLanes = W;
    __device__ __forceinline__ static int lane() { return static_cast<int>(threadIdx.x) & (W - 1); }
    // the warp lane of the group's first lane
    __device__ __forceinline__ static int first() { return static_cast<int>(threadIdx.x) & (32 - W); }
    __device__ __forceinline__ static bool leader() { return lane() == 0; }
    // whether c holds for a particle of the warp (c is the same in every lane of a group)
    __device__ __forceinline__ static bool any(bool c) {
        if constexpr (W == 32) return c;
        return __any_sync(0xffffffffu, c) != 0;
    }
    // the group's lanes for which ok holds, bit l for its lane l
    __device__ __forceinline__ static unsigned ballot(bool ok) {
        return (__ballot_sync(0xffffffffu, ok) >> first()) & (0xffffffffu >> (32 - W));
    }
    // adds the lanes' terms in lane order; m: the lanes that have one (the others' are +0)
    template <class T, class Add>
    __device__ __forceinline__ static void add_lanes(unsigned m, const T& t, Add&& add, T& sum) {
        if constexpr (W == 32) {
            while (m) {
                const int src = __ffs(m) - 1;
                m &= m - 1u;
                add(sum, shfl_from(t, src));
            }
        } else {
            if (!any(m != 0u)) return;
#pragma unroll
            for (int l = 0; l < W; ++l) add(sum, shfl_from(t, first() + l));
        }
    }

    // a and b are the same in every lane of a group
    template <class T, class Test, class Term, class Add>
    __device__ __forceinline__ static void span(int a, int b, Test&& test, Term&& term, Add&& add, T& sum) {
        for (int base = a; any(base < b); base += W) {
            const int k = base + lane();
            T t{};
            const bool ok = k < b && test(k);
            if (ok) t = term(k);
            add_lanes(ballot(ok), t, add, sum);
        }
    }

    // live(row) is the same in every lane of a group
    template <class T, class Live, class Test, class Term, class Add>
    __device__ __forceinline__ static void window_if(bool on, const int* off, int dimx, int csx, int cex, int csy,
                                                     int cey, Live&& live, Test&& test, Term&& term, Add&& add,
                                                     T& sum) {
        for (int cy = csy; any(on && cy <= cey); ++cy) {
            const int row = cy * dimx;
            const bool in = on && cy <= cey && live(row);
            if (any(in)) span(in ? off[row + csx] : 0, in ? off[row + cex + 1] : 0, test, term, add, sum);
        }
    }

    template <class T, class Test, class Term, class Add>
    __device__ __forceinline__ static void window(bool on, const int* off, int dimx, int csx, int cex, int csy, int cey,
                                                  Test&& test, Term&& term, Add&& add, T& sum) {
        window_if(on, off, dimx, csx, cex, csy, cey, [](int) { return true; }, test, term, add, sum);
    }
};

using PerWarp = PerGroup<32>;

}  // namespace tss
