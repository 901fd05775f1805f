// sweep.cuh - bodies of the phase-1 sweep kernels (decide-and-move, weight
// update and pruning) per degree bin: every function handles the list
// positions of one warp or block, so that one kernel can run a single bin
// (phase1.cu) or whole sweeps (small_level.cu).
#pragma once
#include "common.cuh"
#include "internal.h"

namespace gala {

// Exact 128-bit block sum added to the (lo, hi) counter pair (carry from the
// low word's atomic result, so the total does not depend on the order).
__device__ __forceinline__ void block_add_u128(unsigned __int128 v, unsigned long long *lo, unsigned long long *hi)
{
    __shared__ unsigned long long rlo[32], rhi[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const unsigned long long l = __shfl_xor_sync(GALA_FULL_MASK, (unsigned long long)v, o);
        const unsigned long long h = __shfl_xor_sync(GALA_FULL_MASK, (unsigned long long)(v >> 64), o);
        v += ((unsigned __int128)h << 64) | l;
    }
    if (lane == 0) {
        rlo[wid] = (unsigned long long)v;
        rhi[wid] = (unsigned long long)(v >> 64);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned __int128 t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += ((unsigned __int128)rhi[w] << 64) | rlo[w];
        const unsigned long long l = (unsigned long long)t;
        unsigned long long h = (unsigned long long)(t >> 64);
        if (l) {
            const unsigned long long old = atomicAdd(lo, l);
            if (old + l < old) h += 1;
        }
        if (h) atomicAdd(hi, h);
    }
    __syncthreads();
}

// Square sums of community weights: u64 for int32 weights, exact u128 for
// 64-bit fixed-point weights (Tot^2 up to 2^124).
template <typename WT>
struct SqSum {
    using T = unsigned long long;
    static __device__ __forceinline__ T sq(WT t) { return (T)((long long)t * t); }
    static __device__ __forceinline__ void add(T v, unsigned long long *lo, unsigned long long *)
    {
        block_add_u64(v, lo);
    }
};
template <>
struct SqSum<long long> {
    using T = unsigned __int128;
    static __device__ __forceinline__ T sq(long long t)
    {
        return (T)(unsigned long long)t * (unsigned long long)t;
    }
    static __device__ __forceinline__ void add(T v, unsigned long long *lo, unsigned long long *hi)
    {
        block_add_u128(v, lo, hi);
    }
};

// ------------------------------------------------------------------------
// Decide-and-move
// ------------------------------------------------------------------------
// Labels, totals, sizes and weighted degrees are read-only for a kernel that
// runs one sweep (RO), so their loads may take the non-coherent path; a kernel
// that runs a whole level with grid barriers between its steps (!RO) writes
// them too.
template <typename T, bool RO>
struct SweepPtr {
    using type = const T *__restrict__;
};
template <typename T>
struct SweepPtr<T, false> {
    using type = const T *;
};

template <typename WT, bool RO = true>
struct DecideArgs {
    const int64_t *__restrict__ offs;
    const int32_t *__restrict__ nbr;
    const WT *__restrict__ w;
    typename SweepPtr<int32_t, RO>::type comm;
    typename SweepPtr<WT, RO>::type K;
    typename SweepPtr<WT, RO>::type Self;
    typename SweepPtr<WT, RO>::type Tot;
    typename SweepPtr<int32_t, RO>::type size;
    int32_t *mv_v, *mv_old, *mv_new;
    WT *tot_next;  // !RO: totals after the sweep, moved along with the mover lists
    int *n_movers, *err;
    unsigned long long *fp64_decisions;
    double constant;  // 1 / m2
    long long m2;
    int fp64_only;    // 1 = evaluate every vertex with the FP64 expressions
    float *feat_gain;   // proposal features (null when no proposal mode is on)
    int32_t *feat_ndist;
    // batched graphs (null for one graph): graph of each vertex, its total
    // weight m2 and 1/m2, and the graphs whose phase 1 has stopped
    const int32_t *__restrict__ gid;
    const long long *__restrict__ m2g;
    const double *__restrict__ cg;
    const uint8_t *__restrict__ stop;
};

// Gain scale of a vertex: m2 and 1/m2 of its graph.
struct Scale {
    long long m2;
    double c;
};
template <typename WT, bool RO>
__device__ __forceinline__ Scale scale_of(const DecideArgs<WT, RO> &a, int v)
{
    if (a.gid) {
        const int g = a.gid[v];
        return Scale{a.m2g[g], a.cg[g]};
    }
    return Scale{a.m2, a.constant};
}
// Vertex of a batched graph whose phase 1 has stopped: not decided.
template <typename WT, bool RO>
__device__ __forceinline__ bool stopped(const DecideArgs<WT, RO> &a, int v)
{
    return a.stop && a.stop[a.gid[v]];
}

// Singleton swap guard (kernel_functions.cu:386): two singletons never move
// towards the larger id.
template <typename WT, bool RO>
__device__ __forceinline__ bool guard_ok(const DecideArgs<WT, RO> &a, int cur, int best)
{
    return !(a.size[best] == 1 && a.size[cur] == 1 && best > cur);
}

// ---- gains without FP64 ----------------------------------------------------
// GB300 runs FP64 at 1/64 of its FP32 rate, so a decision is taken without it
// whenever that provably gives what the reference's FP64 expressions give.
//
// int32 weights, exact integers.  The reference's gain
// dq = 2w - 2K((Tot_c - Tot_cur) + K)/m2 equals (2/m2) * X with the integer
// X = w*m2 - K*((Tot_c - Tot_cur) + K), which fits int64 for m2 < 2^31.
// Distinct X differ by at least 2/m2 in dq, while the FP64 evaluation errs by
// at most K * 2^-50; so for K*m2 < 2^49 the FP64 order of distinct X is the
// exact order and the sign of a non-zero X (or of the corrected gain) is
// exact.  Three cases can still round either way and are re-evaluated with
// the FP64 expressions of the reference: equal best X from different weights
// (FP64 may order them by value, not by id), X = 0 when the vertex has no
// other weight in its community, and a corrected gain of exactly 0.
//
// 64-bit fixed-point weights, FP32 bounds.  g = w - K((Tot_c - Tot_cur) + K)/m2
// (half the gain) is evaluated in FP32 from the exact 64-bit integers, with a
// bound e on its distance both from the exact value and from the FP64
// evaluation: each operand is rounded to 2^-23 relative or better and four
// roundings follow, under 2^-20 (w + |p|) for g = w - p; the FP64 evaluation
// errs by under 26 K 2^-53 (its three totals are rounded before they cancel).
// A candidate whose lower bound exceeds every other candidate's upper bound
// is the FP64 maximum, and the move is settled when the corrected gain's
// bound excludes 0; all else goes to the FP64 expressions, which then skip
// the candidates the bounds exclude.  The partition is the same bit for bit.
// Measured on an LFR-style graph of 500k vertices / 13M edges, lognormal
// float weights, where every candidate took 12 FP64 instructions before: the
// decide kernels' summed time goes from 26.8 to 16.6 ms a run.

// Per-vertex terms of the gains.
template <typename WT>
struct GainTerms;
template <>
struct GainTerms<int> {
    long long m2, xbase;  // X = w m2 - K Tot_c - xbase
    int ki;
    __device__ __forceinline__ GainTerms(const Scale &sc, int k, int tcur)
        : m2(sc.m2), xbase((long long)k * ((long long)k - (long long)tcur)), ki(k)
    {
    }
};
template <>
struct GainTerms<long long> {
    long long base;  // K - Tot_cur
    float kc, ek;    // K / m2; the FP64 evaluation's error
    __device__ __forceinline__ GainTerms(const Scale &sc, long long k, long long tcur) : base(k - tcur)
    {
        const float kf = f32_of(k);
        kc = kf * (float)sc.c;
        ek = kf * 0x1p-46f;
    }
    // bounds of g for weight w and total tot
    __device__ __forceinline__ void bounds(long long w, long long tot, float &lo, float &hi) const
    {
        const float wf = f32_of(w), p = kc * f32_of(tot + base), g = wf - p;
        const float e = (wf + fabsf(p)) * 0x1p-20f + ek;
        lo = g - e;
        hi = g + e;
    }
};

// Best candidate so far.  Merging is commutative, so butterfly reductions
// agree on every lane.
template <typename WT>
struct Cand;
template <>
struct Cand<int> {
    long long x;  // largest X (>= 0), -1: no candidate
    int c, w, t;  // its lowest id, that one's weight, tie between different weights
    __device__ __forceinline__ explicit Cand(int cur) : x(-1), c(cur), w(0), t(0) {}
    __device__ __forceinline__ void merge(const Cand &o)
    {
        if (o.x == x) {
            const int tie = t | o.t | (o.w != w);
            if (o.c < c) {
                c = o.c;
                w = o.w;
            }
            t = tie;
        } else if (o.x > x) {
            *this = o;
        }
    }
    __device__ __forceinline__ void offer(const GainTerms<int> &g, int cc, int ww, int tot)
    {
        Cand o(cc);
        o.x = (long long)ww * g.m2 - (long long)g.ki * (long long)tot - g.xbase;
        o.w = ww;
        if (o.x >= 0) merge(o);
    }
    __device__ __forceinline__ Cand shfl_xor(int o) const
    {
        Cand r(__shfl_xor_sync(GALA_FULL_MASK, c, o));
        r.x = __shfl_xor_sync(GALA_FULL_MASK, x, o);
        r.w = __shfl_xor_sync(GALA_FULL_MASK, w, o);
        r.t = __shfl_xor_sync(GALA_FULL_MASK, t, o);
        return r;
    }
    // Could the candidate be the FP64 maximum, given the merged best?
    __device__ __forceinline__ bool fp64_rival(const GainTerms<int> &, int, int) const { return true; }
    // 0 = stay, 1 = move (before the singleton guard), 2 = evaluate in FP64.
    __device__ __forceinline__ int decide(int fp64_only, const Scale &sc, int cur, int w_cur, int self_w, int ki) const
    {
        if (fp64_only || (long long)ki * sc.m2 >= (1LL << 49)) return 2;
        if (c == cur) return 0;  // every candidate has X < 0: every FP64 gain is < 0
        if (x == 0) return w_cur == self_w ? 2 : 0;
        if (t) return 2;
        const long long y = x - (long long)(w_cur - self_w) * sc.m2;
        if (y == 0) return 2;
        return y > 0 ? 1 : 0;
    }
};
template <>
struct Cand<long long> {
    float lo, hi;  // bounds of the candidate with the largest lower bound (-inf: none)
    float hi2;     // largest upper bound of the others
    int c;         // its id
    __device__ __forceinline__ explicit Cand(int cur) : lo(-INFINITY), hi(-INFINITY), hi2(-INFINITY), c(cur) {}
    __device__ __forceinline__ void merge(const Cand &o)
    {
        if (o.lo > lo || (o.lo == lo && o.c < c)) {
            hi2 = fmaxf(fmaxf(hi2, o.hi2), hi);
            lo = o.lo;
            hi = o.hi;
            c = o.c;
        } else {
            hi2 = fmaxf(fmaxf(hi2, o.hi2), o.hi);
        }
    }
    __device__ __forceinline__ void offer(const GainTerms<long long> &g, int cc, long long ww, long long tot)
    {
        Cand o(cc);
        g.bounds(ww, tot, o.lo, o.hi);
        merge(o);
    }
    __device__ __forceinline__ Cand shfl_xor(int o) const
    {
        Cand r(__shfl_xor_sync(GALA_FULL_MASK, c, o));
        r.lo = __shfl_xor_sync(GALA_FULL_MASK, lo, o);
        r.hi = __shfl_xor_sync(GALA_FULL_MASK, hi, o);
        r.hi2 = __shfl_xor_sync(GALA_FULL_MASK, hi2, o);
        return r;
    }
    __device__ __forceinline__ bool fp64_rival(const GainTerms<long long> &g, long long w, long long tot) const
    {
        float l, h;
        g.bounds(w, tot, l, h);
        return h >= fmaxf(lo, 0.f);
    }
    __device__ __forceinline__ int decide(int fp64_only, const Scale &, int, long long w_cur, long long self_w,
                                          long long ki) const
    {
        if (fp64_only) return 2;
        const float top = fmaxf(hi, hi2);
        if (top < 0.f) return 0;  // every FP64 gain is < 0
        // corrected gain / 2 = g - (w_cur - Self), FP64 error again under 13 K 2^-53
        const float d = f32_of(w_cur - self_w);
        const float e = (top + fabsf(d)) * 0x1p-20f + f32_of(ki) * 0x1p-46f;
        if (top - d < -e) return 0;  // whichever candidate wins
        if (hi2 < lo && lo > 0.f && lo - d > e) return 1;
        return 2;
    }
};

// Proposal features of a decided vertex: its best corrected gain
// (max(X, 0) - (w_cur - Self) m2, normalised by K m2) and the number of
// distinct neighbour communities (-1 when the schedule does not count them).
template <typename WT, bool RO>
__device__ __forceinline__ void write_features(const DecideArgs<WT, RO> &a, const Scale &sc, int v, const Cand<WT> &best,
                                               WT w_cur, WT self_w, WT ki, int ndist)
{
    if constexpr (WideOf<WT>::exact) {  // no proposal modes on fixed-point weights
        if (!a.feat_gain) return;
        const long long y = (best.x > 0 ? best.x : 0) - (long long)(w_cur - self_w) * sc.m2;
        a.feat_gain[v] = ki > 0 ? (float)y / ((float)sc.m2 * (float)ki) : 0.f;
        a.feat_ndist[v] = ndist;
    }
}

// FP32 as int32 of the same order.
__device__ __forceinline__ int ordered(float f)
{
    const int i = __float_as_int(f);
    return i ^ ((i >> 31) & 0x7fffffff);
}

// Merge over a whole warp whose lanes hold different communities: the result of
// the butterfly merge below from a few warp reductions (a butterfly step moves
// five or six values).
__device__ __forceinline__ void warp_best(Cand<int> &b)
{
    const int mh = __reduce_max_sync(GALA_FULL_MASK, (int)(b.x >> 32));
    if (mh < 0) return;  // no candidate in any lane (warp-uniform)
    const bool top = (int)(b.x >> 32) == mh;
    const unsigned ml = __reduce_max_sync(GALA_FULL_MASK, top ? (unsigned)b.x : 0u);
    const bool win = top && (unsigned)b.x == ml;
    const unsigned wins = __ballot_sync(GALA_FULL_MASK, win);
    int src = __ffs((int)wins) - 1, t = b.t;
    if (wins & (wins - 1)) {  // equal best X: the lowest id, a tie when the weights differ
        const int w0 = __shfl_sync(GALA_FULL_MASK, b.w, src);
        t = __any_sync(GALA_FULL_MASK, win && (b.t || b.w != w0));
        const unsigned c0 = __reduce_min_sync(GALA_FULL_MASK, win ? (unsigned)b.c : 0xffffffffu);
        src = __ffs((int)__ballot_sync(GALA_FULL_MASK, win && (unsigned)b.c == c0)) - 1;
    }
    b.c = __shfl_sync(GALA_FULL_MASK, b.c, src);
    b.w = __shfl_sync(GALA_FULL_MASK, b.w, src);
    b.t = __shfl_sync(GALA_FULL_MASK, t, src);
    b.x = ((long long)mh << 32) | ml;
}
__device__ __forceinline__ void warp_best(Cand<long long> &b)
{
    const int ml = __reduce_max_sync(GALA_FULL_MASK, ordered(b.lo));
    const int src = __ffs((int)__ballot_sync(GALA_FULL_MASK, ordered(b.lo) == ml)) - 1;
    const bool win = (int)(threadIdx.x & 31) == src;
    const int m2 = __reduce_max_sync(GALA_FULL_MASK, ordered(win ? b.hi2 : fmaxf(b.hi, b.hi2)));
    b.lo = __shfl_sync(GALA_FULL_MASK, b.lo, src);
    b.hi = __shfl_sync(GALA_FULL_MASK, b.hi, src);
    b.c = __shfl_sync(GALA_FULL_MASK, b.c, src);
    b.hi2 = __int_as_float(m2 ^ ((m2 >> 31) & 0x7fffffff));
}

// Merge over `width` lanes: the candidate and the weight to the own community.
template <typename WT>
__device__ __forceinline__ void warp_merge(Cand<WT> &x, WT &wc, int width)
{
    if (width == 32) {
        wc = group_sum(GALA_FULL_MASK, wc);
        warp_best(x);
        return;
    }
    for (int o = width / 2; o >= 1; o >>= 1) {
        wc += __shfl_xor_sync(GALA_FULL_MASK, wc, o);
        x.merge(x.shfl_xor(o));
    }
}

// One candidate and own-community weight per warp of a block, in shared memory.
template <typename WT, int N>
struct CandRow;
template <int N>
struct CandRow<int, N> {
    long long x[N];
    int c[N], w[N], t[N], wc[N];
    __device__ __forceinline__ void put(int i, const Cand<int> &b, int own)
    {
        x[i] = b.x;
        c[i] = b.c;
        w[i] = b.w;
        t[i] = b.t;
        wc[i] = own;
    }
    __device__ __forceinline__ void get(int i, int n, int cur, Cand<int> &b, int &own) const
    {
        b.x = i < n ? x[i] : -1;
        b.c = i < n ? c[i] : cur;
        b.w = i < n ? w[i] : 0;
        b.t = i < n ? t[i] : 0;
        own = i < n ? wc[i] : 0;
    }
};
template <int N>
struct CandRow<long long, N> {
    float lo[N], hi[N], hi2[N];
    int c[N];
    long long wc[N];
    __device__ __forceinline__ void put(int i, const Cand<long long> &b, long long own)
    {
        lo[i] = b.lo;
        hi[i] = b.hi;
        hi2[i] = b.hi2;
        c[i] = b.c;
        wc[i] = own;
    }
    __device__ __forceinline__ void get(int i, int n, int cur, Cand<long long> &b, long long &own) const
    {
        b.lo = i < n ? lo[i] : -INFINITY;
        b.hi = i < n ? hi[i] : -INFINITY;
        b.hi2 = i < n ? hi2[i] : -INFINITY;
        b.c = i < n ? c[i] : cur;
        own = i < n ? wc[i] : 0;
    }
};

constexpr int kStageN = 256;  // staged active-list appends per warp
constexpr int kStageM = 128;  // staged movers per warp

// Totals and sizes of a warp's movers (Tot += Tot_update, size += size_update,
// louvain_main_process.cu:949-953), or one of the two.  Movers of one warp that
// share a source or a target community add to its Tot and size once (many
// movers of a sweep head for the same large community).  All 32 lanes call.
template <typename WT, bool TOT = true, bool SIZE = true>
__device__ __forceinline__ void move_totals(bool valid, int from, int to, WT k, WT *Tot, int32_t *size)
{
    const int lane = threadIdx.x & 31;
    const unsigned mt = __match_any_sync(GALA_FULL_MASK, to);
    const WT kt = TOT ? match_sum(mt, valid, k) : (WT)0;
    if (valid && lane == __ffs(mt) - 1) {
        if (TOT) atomic_add_w(&Tot[to], kt);
        if (SIZE) atomicAdd(&size[to], __popc(mt));
    }
    const unsigned mf = __match_any_sync(GALA_FULL_MASK, from);
    const WT kf = TOT ? match_sum(mf, valid, k) : (WT)0;
    if (valid && lane == __ffs(mf) - 1) {
        if (TOT) atomic_add_w(&Tot[from], (WT)-kf);
        if (SIZE) atomicSub(&size[from], __popc(mf));
    }
}

template <typename WT, bool RO>
__device__ __forceinline__ void append_mover(const DecideArgs<WT, RO> &a, bool move, int v, int cur, int best)
{
    unsigned b = __ballot_sync(GALA_FULL_MASK, move);
    if (b == 0) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(b) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(a.n_movers, __popc(b));
    base = __shfl_sync(GALA_FULL_MASK, base, leader);
    if (move) {
        int p = base + __popc(b & lanemask_lt());
        a.mv_v[p] = v;
        a.mv_old[p] = cur;
        a.mv_new[p] = best;
        if constexpr (!RO) {
            const WT k = a.K[v];
            atomic_add_w(&a.tot_next[best], k);
            atomic_add_w(&a.tot_next[cur], (WT)-k);
        }
    }
}

// A warp's staged movers to the lists; with !RO their totals move too.
template <typename WT, bool RO>
__device__ __forceinline__ void flush_movers(const DecideArgs<WT, RO> &a, WarpStage<kStageM, 3> &stage)
{
    int *const lists[3] = {a.mv_v, a.mv_old, a.mv_new};
    if constexpr (!RO) {
        __syncwarp();
        if (stage.n == 0) return;
        int base = 0;  // its place in the lists, asked for ahead of the totals
        if ((threadIdx.x & 31) == 0) base = atomicAdd(a.n_movers, stage.n);
        for (int i0 = 0; i0 < stage.n; i0 += 32) {
            const int i = i0 + (threadIdx.x & 31);
            const bool valid = i < stage.n;
            int from = -1, to = -1;
            WT k = 0;
            if (valid) {
                k = a.K[stage.buf[i]];
                from = stage.buf[kStageM + i];
                to = stage.buf[2 * kStageM + i];
            }
            move_totals<WT, true, false>(valid, from, to, k, a.tot_next, nullptr);
        }
        stage.store(lists, __shfl_sync(GALA_FULL_MASK, base, 0));
    } else {
        stage.flush(lists, a.n_movers);
    }
}

// Degree <= G: one lane per neighbour.  Lanes holding the same neighbour
// community are found with __match_any_sync (the key carries the group index
// so groups of one warp stay apart) and their weights summed with
// __reduce_add_sync; the lowest lane of each set evaluates the gain.
// A warp takes the tasks (32 / G vertices each) wg, wg + nw, ... of the list.
template <typename WT, int G, bool W, bool RO>
__device__ __forceinline__ void decide_group(const DecideArgs<WT, RO> &a, const int32_t *list, int count, int wg,
                                             int nw, WarpStage<kStageM, 3> &stage)
{
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), gw = lane / G;
    constexpr int GPW = 32 / G;
    int *const mlists[3] = {a.mv_v, a.mv_old, a.mv_new};
    for (int base = wg * GPW; base < count; base += nw * GPW) {
        const int idx = base + gw;
        bool has = idx < count;
        int v = 0, cur = -1, deg = 0;
        WT ki = 0, sf = 0, tcur = 0;
        long long s = 0;
        Scale sc{a.m2, a.constant};
        if (has) {
            v = list[idx];
            has = !stopped(a, v);
        }
        if (has) {
            sc = scale_of(a, v);
            s = a.offs[v];
            deg = (int)(a.offs[v + 1] - s);
            cur = a.comm[v];
            ki = a.K[v];
            sf = a.Self[v];
            tcur = a.Tot[cur];
        }
        const bool valid = has && sub < deg;
        int c = -1;
        WT wt = 0;
        if (valid) {
            c = a.comm[a.nbr[s + sub]];
            wt = W ? a.w[s + sub] : 1;
        }
        // lanes of the group holding the same community: the lowest leads and
        // sums the weights (G - 1 shuffles for small groups, a key match for
        // whole warps)
        WT wsum;
        bool leader;
        if constexpr (G == 32) {
            const unsigned m = __match_any_sync(GALA_FULL_MASK, c);
            wsum = W ? match_sum(m, valid, wt) : (WT)__popc(m);
            leader = valid && (__ffs(m) - 1 == lane);
        } else {
            wsum = wt;
            leader = valid;
#pragma unroll
            for (int o = 1; o < G; ++o) {
                const int osub = (sub + o) & (G - 1);
                const int src = (lane & ~(G - 1)) | osub;
                const int oc = __shfl_sync(GALA_FULL_MASK, c, src);
                const WT ow = W ? __shfl_sync(GALA_FULL_MASK, wt, src) : (WT)1;
                if (oc == c) {
                    wsum += ow;
                    if (osub < sub) leader = false;
                }
            }
        }
        const WT wc_own = (leader && c == cur) ? wsum : 0;
        WT wc = wc_own;
        WT tc = 0;
        Cand<WT> best(cur);
        if (leader && c != cur) {
            tc = a.Tot[c];
            best.offer(GainTerms<WT>(sc, ki, tcur), c, wsum, tc);
        }
        warp_merge(best, wc, G);
        int bc = best.c;
        int dec = 0;
        if (has && sub == 0) dec = best.decide(a.fp64_only, sc, cur, wc, sf, ki);
        const bool fp = dec == 2;
        if (__any_sync(GALA_FULL_MASK, fp)) {
            // the reference's FP64 evaluation of the same candidates
            double dq = 0.0;
            int fc = cur;
            if (leader && c != cur) {
                const double d = gain_dq(wsum, ki, tc, tcur, sc.c);
                if (d > 0.0) {
                    dq = d;
                    fc = c;
                }
            }
#pragma unroll
            for (int o = G / 2; o >= 1; o >>= 1) {
                const double od = __shfl_xor_sync(GALA_FULL_MASK, dq, o);
                const int oc = __shfl_xor_sync(GALA_FULL_MASK, fc, o);
                if (cand_better(od, oc, dq, fc)) {
                    dq = od;
                    fc = oc;
                }
            }
            if (fp) {
                bc = fc;
                dec = (fc != cur && gain_correct(dq, wc, sf) > 0.0) ? 1 : 0;
                atomicAdd(a.fp64_decisions, 1ull);
            }
        }
        const bool move = has && sub == 0 && dec == 1 && guard_ok(a, cur, bc);
        if (a.feat_gain) {
            const unsigned lb = __ballot_sync(GALA_FULL_MASK, leader);
            const unsigned gmask = G == 32 ? GALA_FULL_MASK : (((1u << G) - 1u) << (gw * G));
            if (has && sub == 0) write_features(a, sc, v, best, wc, sf, ki, __popc(lb & gmask));
        }
        const int item[3] = {v, cur, bc};
        if (!RO && stage.n + 32 > kStageM) flush_movers(a, stage);
        stage.push(move, item, mlists, a.n_movers);
    }
}

// Scan a hash table: this thread's best candidate and its share of the
// weight to the own community.
template <typename WT, bool RO>
__device__ __forceinline__ void scan_table_best(const DecideArgs<WT, RO> &a, const GainTerms<WT> &gt, const int *keys,
                                                const WT *vals, int T, int first, int stride, int cur, Cand<WT> &best,
                                                WT &wc)
{
    for (int j = first; j < T; j += stride) {
        const int c = keys[j];
        if (c < 0) continue;
        const WT wv = vals[j];
        if (c == cur)
            wc += wv;
        else
            best.offer(gt, c, wv, a.Tot[c]);
    }
}

// The same scan with the reference's FP64 gains (vertices that Cand::decide
// cannot settle); best: the merged best candidate of the scan.
template <typename WT, bool RO>
__device__ __forceinline__ void scan_table(const DecideArgs<WT, RO> &a, const Scale &sc, const GainTerms<WT> &gt,
                                           const Cand<WT> &best, const int *keys, const WT *vals, int T, int first,
                                           int stride, int cur, WT ki, WT tcur, double &dq, int &bc)
{
    for (int j = first; j < T; j += stride) {
        const int c = keys[j];
        if (c < 0 || c == cur) continue;
        const WT tc = a.Tot[c];
        if (!a.fp64_only && !best.fp64_rival(gt, vals[j], tc)) continue;
        const double d = gain_dq(vals[j], ki, tc, tcur, sc.c);
        if (d > 0.0 && cand_better(d, c, dq, bc)) {
            dq = d;
            bc = c;
        }
    }
}

__device__ __forceinline__ void warp_argmax(double &dq, int &bc)
{
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        double od = __shfl_xor_sync(GALA_FULL_MASK, dq, o);
        int oc = __shfl_xor_sync(GALA_FULL_MASK, bc, o);
        if (cand_better(od, oc, dq, bc)) {
            dq = od;
            bc = oc;
        }
    }
}

// Insert (key, w) into a table of T slots (power of two); returns the slot
// and sets `created` when this call claimed it, -1 when the probe ran out.
template <typename VT>
__device__ __forceinline__ int hash_add_slot(int *keys, VT *vals, int T, int log2t, int key, VT w, bool &created)
{
    // one compare-and-swap per probe: it claims an empty slot or returns the
    // key that holds it
    unsigned h = hash_slot(key, log2t);
    created = false;
    for (int p = 0; p < T; ++p) {
        const int k = atomicCAS(&keys[h], -1, key);
        if (k == -1 || k == key) {
            created = k == -1;
            atomic_add_sm(&vals[h], w);
            return (int)h;
        }
        h = (h + 1) & (unsigned)(T - 1);
    }
    return -1;
}

// Scans over the list of occupied slots (slot indices in occ[0, nocc)).
template <typename WT, bool RO>
__device__ __forceinline__ void scan_list_best(const DecideArgs<WT, RO> &a, const GainTerms<WT> &gt, const int *keys,
                                               const WT *vals, const unsigned short *occ, int nocc, int first,
                                               int stride, int cur, Cand<WT> &best, WT &wc)
{
    for (int q = first; q < nocc; q += stride) {
        const int j = occ[q];
        const int c = keys[j];
        const WT wv = vals[j];
        if (c == cur)
            wc += wv;
        else
            best.offer(gt, c, wv, a.Tot[c]);
    }
}

template <typename WT, bool RO>
__device__ __forceinline__ void scan_list(const DecideArgs<WT, RO> &a, const Scale &sc, const GainTerms<WT> &gt,
                                          const Cand<WT> &best, const int *keys, const WT *vals,
                                          const unsigned short *occ, int nocc, int first, int stride, int cur, WT ki,
                                          WT tcur, double &dq, int &bc)
{
    for (int q = first; q < nocc; q += stride) {
        const int j = occ[q];
        const int c = keys[j];
        if (c == cur) continue;
        const WT tc = a.Tot[c];
        if (!a.fp64_only && !best.fp64_rival(gt, vals[j], tc)) continue;
        const double d = gain_dq(vals[j], ki, tc, tcur, sc.c);
        if (d > 0.0 && cand_better(d, c, dq, bc)) {
            dq = d;
            bc = c;
        }
    }
}

// Degree 33-256: one warp per vertex with a private shared-memory hash table
// of TW slots (one-bin kernels, two launches: 256 slots for rows up to 128
// entries, with eight resident blocks per SM at 32 registers a thread, and 512
// slots for longer rows; small levels: rows up to half the table, 512 slots or 256
// with 64-bit weights, longer ones in the CTA's table).  The table is cleared once per warp; per vertex the slots it claims
// are listed, and only those are scanned and cleared again.
constexpr int kWarpTable = 512;  // the full table; rows up to kWarpTable / 4 use half of it
constexpr int kWarpWarps = 8;  // warps per block
// TW slots per warp for rows up to TW / 2 entries (a vertex claims at most
// as many slots as it has entries)
template <typename WT, int TW>
constexpr size_t warp_smem()
{
    return (size_t)kWarpWarps * (TW * (sizeof(int) + sizeof(WT)) + (TW / 2) * sizeof(unsigned short));
}
// (keys / vals / occ: this warp's empty table, left empty; the warp takes the
// vertices wg, wg + nw, ... of the list)
template <typename WT, bool W, int TW, bool RO>
__device__ __forceinline__ void decide_warp(const DecideArgs<WT, RO> &a, const int32_t *list, int count, int wg, int nw,
                                            int dlo, int dhi, int *keys, WT *vals, unsigned short *occ)
{
    const int lane = threadIdx.x & 31;
    constexpr int TL = TW == 256 ? 8 : 9;
    static_assert((1 << TL) == TW, "table size");
    for (int i = wg; i < count; i += nw) {
        const int v = list[i];
        if (stopped(a, v)) continue;
        const Scale sc = scale_of(a, v);
        const long long s = a.offs[v];
        const int deg = (int)(a.offs[v + 1] - s);
        if (deg <= dlo || deg > dhi) continue;  // the other launch of this bin decides it
        const int cur = a.comm[v];
        int nocc = 0;
        const int32_t *rn = a.nbr + s;
        const WT *rw = W ? a.w + s : nullptr;
        for (int e0 = 0; e0 < deg; e0 += 32) {
            const int e = e0 + lane;
            const bool valid = e < deg;
            int c = -1;
            WT wt = 0;
            if (valid) {
                c = a.comm[rn[e]];
                wt = W ? rw[e] : 1;
            }
            // every entry goes to the table on its own: repeated communities
            // meet at their slot (a warp-level match of equal keys costs more
            // than the repeated adds it saves)
            bool created = false;
            int slot = -1;
            if (valid) {
                slot = hash_add_slot(keys, vals, TW, TL, c, wt, created);
                if (slot < 0) atomicOr(a.err, kErrHashOverflow);
            }
            const unsigned cb = __ballot_sync(GALA_FULL_MASK, created);
            if (created) occ[nocc + __popc(cb & lanemask_lt())] = (unsigned short)slot;
            nocc += __popc(cb);
        }
        __syncwarp();
        const WT ki = a.K[v], tcur = a.Tot[cur], sf = a.Self[v];
        const GainTerms<WT> gt(sc, ki, tcur);
        Cand<WT> best(cur);
        WT wc = 0;
        scan_list_best(a, gt, keys, vals, occ, nocc, lane, 32, cur, best, wc);
        warp_merge(best, wc, 32);
        int bc = best.c;
        int dec = best.decide(a.fp64_only, sc, cur, wc, sf, ki);  // warp-uniform
        if (dec == 2) {
            double dq = 0.0;
            int fc = cur;
            scan_list(a, sc, gt, best, keys, vals, occ, nocc, lane, 32, cur, ki, tcur, dq, fc);
            warp_argmax(dq, fc);
            bc = fc;
            dec = (fc != cur && gain_correct(dq, wc, sf) > 0.0) ? 1 : 0;
            if (lane == 0) atomicAdd(a.fp64_decisions, 1ull);
        }
        const bool move = lane == 0 && dec == 1 && guard_ok(a, cur, bc);
        if (lane == 0) write_features(a, sc, v, best, wc, sf, ki, nocc);
        append_mover(a, move, v, cur, bc);
        __syncwarp();
        for (int q = lane; q < nocc; q += 32) {
            const int j = occ[q];
            keys[j] = -1;
            vals[j] = 0;
        }
        __syncwarp();
    }
}

// Degree 257-8192 (small levels: to 4096, 64-bit weights from 129 to 2048): one
// CTA per vertex with a shared-memory hash table of tmax slots (int keys, WT
// values) and the list of claimed slots, cleared once per CTA and then slot by
// slot after every vertex.
template <typename WT>
constexpr size_t cta_smem(int tmax)
{
    // a vertex claims at most deg <= tmax / 2 slots
    return (size_t)tmax * (sizeof(int) + sizeof(WT)) + (size_t)(tmax / 2) * sizeof(unsigned short);
}
// (keys / vals / occ: the block's empty table of tmax slots, left empty; the
// block takes the vertices b0, b0 + nb, ... of the list)
template <typename WT, int BLOCK, bool W, bool RO>
__device__ __forceinline__ void decide_cta(const DecideArgs<WT, RO> &a, const int32_t *list, int count, int b0, int nb,
                                           int tmax, int dlo, int dhi, int *keys, WT *vals, unsigned short *occ)
{
    __shared__ double r_dq[BLOCK / 32];
    __shared__ int r_c[BLOCK / 32];
    __shared__ CandRow<WT, BLOCK / 32> r_best;
    __shared__ int s_dec, s_bc, s_nocc;
    __shared__ WT s_wc;
    const int lg = __ffs(tmax) - 1;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_nocc = 0;
    __syncthreads();
    for (int i = b0; i < count; i += nb) {
        const int v = list[i];
        if (stopped(a, v)) continue;
        const Scale sc = scale_of(a, v);
        const long long s = a.offs[v];
        const long long e = a.offs[v + 1];
        const int deg = (int)(e - s);
        const int cur = a.comm[v];
        if (deg <= dlo || deg > dhi) continue;  // the other launch of this bin decides it
        if (2LL * deg > tmax) {  // cannot happen for the bin limits; recorded, vertex stays
            if (threadIdx.x == 0) atomicOr(a.err, kErrHashOverflow);
            continue;
        }
        for (long long j0 = s; j0 < e; j0 += BLOCK) {
            const long long j = j0 + threadIdx.x;
            const bool valid = j < e;
            int c = -1;
            WT wt = 0;
            if (valid) {
                c = a.comm[a.nbr[j]];
                wt = W ? a.w[j] : 1;
            }
            bool created = false;
            int slot = -1;
            if (valid) {
                slot = hash_add_slot(keys, vals, tmax, lg, c, wt, created);
                if (slot < 0) atomicOr(a.err, kErrHashOverflow);
            }
            const unsigned cb = __ballot_sync(GALA_FULL_MASK, created);
            if (cb) {
                const int leader = __ffs(cb) - 1;
                int base = 0;
                if (lane == leader) base = atomicAdd(&s_nocc, __popc(cb));
                base = __shfl_sync(GALA_FULL_MASK, base, leader);
                if (created) occ[base + __popc(cb & lanemask_lt())] = (unsigned short)slot;
            }
        }
        __syncthreads();
        const int nocc = s_nocc;
        const WT ki = a.K[v], tcur = a.Tot[cur], sf = a.Self[v];
        constexpr int NW = BLOCK / 32;
        const GainTerms<WT> gt(sc, ki, tcur);
        Cand<WT> best(cur);
        WT wc = 0;
        scan_list_best(a, gt, keys, vals, occ, nocc, threadIdx.x, BLOCK, cur, best, wc);
        warp_merge(best, wc, 32);
        if (lane == 0) r_best.put(wid, best, wc);
        __syncthreads();
        if (wid == 0) {
            r_best.get(lane, NW, cur, best, wc);
            warp_merge(best, wc, 32);
            if (lane == 0) {
                s_dec = best.decide(a.fp64_only, sc, cur, wc, sf, ki);
                s_bc = best.c;
                s_wc = wc;
                r_best.put(0, best, wc);  // the vertex's, for an FP64 evaluation
            }
        }
        __syncthreads();
        if (s_dec == 2) {  // block-uniform: the reference's FP64 evaluation
            double dq = 0.0;
            int fc = cur;
            Cand<WT> top(cur);
            WT unused;
            r_best.get(0, 1, cur, top, unused);
            scan_list(a, sc, gt, top, keys, vals, occ, nocc, threadIdx.x, BLOCK, cur, ki, tcur, dq, fc);
            warp_argmax(dq, fc);
            if (lane == 0) {
                r_dq[wid] = dq;
                r_c[wid] = fc;
            }
            __syncthreads();
            if (wid == 0) {
                dq = lane < NW ? r_dq[lane] : 0.0;
                fc = lane < NW ? r_c[lane] : cur;
                warp_argmax(dq, fc);
                if (lane == 0) {
                    s_bc = fc;
                    s_dec = (fc != cur && gain_correct(dq, s_wc, sf) > 0.0) ? 1 : 0;
                    atomicAdd(a.fp64_decisions, 1ull);
                }
            }
            __syncthreads();
        }
        if (wid == 0) {
            const bool move = lane == 0 && s_dec == 1 && guard_ok(a, cur, s_bc);
            if (lane == 0) write_features(a, sc, v, best, s_wc, sf, ki, nocc);
            append_mover(a, move, v, cur, s_bc);
        }
        for (int q = threadIdx.x; q < nocc; q += BLOCK) {
            const int j = occ[q];
            keys[j] = -1;
            vals[j] = 0;
        }
        __syncthreads();
        if (threadIdx.x == 0) s_nocc = 0;
        __syncthreads();
    }
}

// ------------------------------------------------------------------------
// Hub vertices (degree > 8192, on small levels > 4096 or, with 64-bit weights,
// > 2048): one global hash table per hub, filled by many CTAs in 4096-entry
// chunks of the hub's row, scanned by many CTAs in 4096-slot chunks (each writes
// the best candidate of its chunk), and merged by one warp per hub.  A hub's work
// is spread over all SMs instead of one.
// ------------------------------------------------------------------------
constexpr int kHubChunk = 4096;

// Table slots, row chunks and table chunks of a hub of degree deg (p: the
// caller's cap on the slots, which rows that only a small level makes hubs of
// are spared).
__device__ __forceinline__ void hub_table(const HubPlan &p, long long deg, long long &T, long long &chunks,
                                          long long &tchunks)
{
    T = next_pow2_ll(deg + deg / 2);  // load at most 2/3
    if (p.t_cap > 0 && deg > p.cap_deg && T > p.t_cap) T = p.t_cap;  // capped: inserts may run out of slots
    chunks = (deg + kHubChunk - 1) / kHubChunk;
    tchunks = (T + kHubChunk - 1) / kHubChunk;
}

// Chunk -> hub lists, one warp per hub.
__device__ __forceinline__ void hub_work(const HubPlan &p, int wg, int nw)
{
    const int lane = threadIdx.x & 31;
    for (int i = wg; i < p.H; i += nw) {
        long long o = p.coff[i], k = p.coff[i + 1] - o;
        for (long long j = lane; j < k; j += 32) p.work[o + j] = i;
        o = p.tcoff[i];
        k = p.tcoff[i + 1] - o;
        for (long long j = lane; j < k; j += 32) p.twork[o + j] = i;
    }
}

// Values of a hub table (WT per slot, after the keys of all tables).
template <typename WT>
__device__ __forceinline__ WT *hub_vals(const HubPlan &p, long long i)
{
    return (WT *)(p.pool + p.half) + p.toff[i];
}

template <typename WT, bool W, bool RO>
__device__ __forceinline__ void hub_insert(const DecideArgs<WT, RO> &a, const HubPlan &p, const uint8_t *flag, int bid,
                                           int nb)
{
    // a small shared-memory table in front of the hub's global table: an
    // entry whose community finds a slot within kHubCacheProbe probes is
    // summed there, the rest go to the global table directly; the cached sums
    // are added to the global table at the end of the chunk (integer adds:
    // the totals do not depend on the split)
    constexpr int kHubCache = 512, kHubCacheLog = 9, kHubCacheProbe = 2;
    __shared__ int ckeys[kHubCache];
    __shared__ WT cvals[kHubCache];
    for (int q = threadIdx.x; q < kHubCache; q += blockDim.x) {
        ckeys[q] = -1;
        cvals[q] = 0;
    }
    __syncthreads();
    for (long long wi = bid; wi < p.nwork; wi += nb) {
        const int i = p.work[wi];
        const int v = p.hubs[i];
        if (!flag[v] || stopped(a, v)) continue;  // block-uniform
        const long long e = a.offs[v + 1];
        const long long s = a.offs[v] + (wi - p.coff[i]) * kHubChunk;
        const long long e2 = s + kHubChunk < e ? s + kHubChunk : e;
        const int T = (int)p.T[i];
        const int lg = __ffs(T) - 1;
        int *keys = p.pool + p.toff[i];
        WT *vals = hub_vals<WT>(p, i);
        for (long long b0 = s; b0 < e2; b0 += blockDim.x) {
            const long long j = b0 + threadIdx.x;
            if (j < e2) {
                const int c = a.comm[a.nbr[j]];
                const WT wt = W ? a.w[j] : 1;
                unsigned h = hash_slot(c, kHubCacheLog);
                bool cached = false;
#pragma unroll
                for (int q = 0; q < kHubCacheProbe; ++q) {
                    const int k = atomicCAS(&ckeys[h], -1, c);
                    if (k == -1 || k == c) {
                        atomic_add_sm(&cvals[h], wt);
                        cached = true;
                        break;
                    }
                    h = (h + 1) & (unsigned)(kHubCache - 1);
                }
                if (!cached && !hash_add(keys, vals, T, lg, c, wt)) atomicOr(a.err, kErrHashOverflow);
            }
        }
        __syncthreads();
        for (int q = threadIdx.x; q < kHubCache; q += blockDim.x) {
            const int k = ckeys[q];
            if (k != -1) {
                if (!hash_add(keys, vals, T, lg, k, cvals[q])) atomicOr(a.err, kErrHashOverflow);
                ckeys[q] = -1;
                cvals[q] = 0;
            }
        }
        __syncthreads();
    }
}

// FP64 evaluation needed whatever the candidates: K*m2 out of the range where
// the integer order equals the FP64 order, or FP64 forced.  Fixed-point
// weights always get their chunks' FP64 partials: the bounds leave few
// candidates to evaluate.
template <typename WT, bool RO>
__device__ __forceinline__ bool needs_fp64(const DecideArgs<WT, RO> &a, const Scale &sc, WT ki)
{
    if constexpr (!WideOf<WT>::exact) return true;
    return a.fp64_only || (long long)ki * sc.m2 >= (1LL << 49);
}

// A chunk's best candidate in the plan's partial arrays.
__device__ __forceinline__ void hub_put(const HubPlan &p, long long i, const Cand<int> &b, int wc)
{
    p.px[i] = b.x;
    p.pc[i] = b.c;
    p.pw[i] = b.w;
    p.pt[i] = b.t;
    p.pwc[i] = wc;
}
__device__ __forceinline__ Cand<int> hub_get(const HubPlan &p, long long i, const Cand<int> &, int &wc)
{
    Cand<int> b(p.pc[i]);
    b.x = p.px[i];
    b.w = p.pw[i];
    b.t = p.pt[i];
    wc = p.pwc[i];
    return b;
}
__device__ __forceinline__ void hub_put(const HubPlan &p, long long i, const Cand<long long> &b, long long wc)
{
    ((float2 *)p.px)[i] = make_float2(b.lo, b.hi);
    p.pc[i] = b.c;
    p.pt[i] = __float_as_int(b.hi2);
    ((long long *)p.pwc)[i] = wc;
}
__device__ __forceinline__ Cand<long long> hub_get(const HubPlan &p, long long i, const Cand<long long> &,
                                                   long long &wc)
{
    Cand<long long> b(p.pc[i]);
    const float2 l = ((const float2 *)p.px)[i];
    b.lo = l.x;
    b.hi = l.y;
    b.hi2 = __int_as_float(p.pt[i]);
    wc = ((const long long *)p.pwc)[i];
    return b;
}

template <typename WT, int BLOCK, bool RO>
__device__ __forceinline__ void hub_scan(const DecideArgs<WT, RO> &a, const HubPlan &p, const uint8_t *flag, int bid,
                                         int nb)
{
    __shared__ double r_dq[BLOCK / 32];
    __shared__ int r_c[BLOCK / 32];
    __shared__ CandRow<WT, BLOCK / 32> r_best;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (long long wi = bid; wi < p.ntwork; wi += nb) {
        const int i = p.twork[wi];
        const int v = p.hubs[i];
        if (!flag[v] || stopped(a, v)) continue;
        const Scale sc = scale_of(a, v);
        const int cur = a.comm[v];
        const WT ki = a.K[v], tcur = a.Tot[cur];
        const long long j0 = (wi - p.tcoff[i]) * kHubChunk;
        const long long T = p.T[i];
        const long long j1 = j0 + kHubChunk < T ? j0 + kHubChunk : T;
        const int *keys = p.pool + p.toff[i];
        const WT *vals = hub_vals<WT>(p, i);
        const GainTerms<WT> gt(sc, ki, tcur);
        Cand<WT> best(cur);
        WT wc = 0;
        scan_table_best(a, gt, keys + j0, vals + j0, (int)(j1 - j0), threadIdx.x, blockDim.x, cur, best, wc);
        warp_merge(best, wc, 32);
        if (lane == 0) r_best.put(wid, best, wc);
        __syncthreads();
        if (wid == 0) {
            r_best.get(lane, blockDim.x >> 5, cur, best, wc);
            warp_merge(best, wc, 32);
            if (lane == 0) {
                hub_put(p, wi, best, wc);
                r_best.put(0, best, wc);
            }
        }
        __syncthreads();
        if (needs_fp64(a, sc, ki)) {  // uniform per chunk: the reference's FP64 gains, chunk-wise
            double dq = 0.0;
            int fc = cur;
            r_best.get(0, 1, cur, best, wc);
            scan_table(a, sc, gt, best, keys + j0, vals + j0, (int)(j1 - j0), threadIdx.x, blockDim.x, cur, ki, tcur,
                       dq, fc);
            warp_argmax(dq, fc);
            if (lane == 0) {
                r_dq[wid] = dq;
                r_c[wid] = fc;
            }
            __syncthreads();
            if (wid == 0) {
                const int nwp = blockDim.x >> 5;
                dq = lane < nwp ? r_dq[lane] : 0.0;
                fc = lane < nwp ? r_c[lane] : cur;
                warp_argmax(dq, fc);
                if (lane == 0) {
                    p.pdq[wi] = dq;
                    p.pfc[wi] = fc;
                }
            }
            __syncthreads();
        }
    }
}

// end(i): past hub i's last partial; rescan: the hub's candidates in FP64, by
// the warp.
template <typename WT, bool RO, typename End, typename Rescan>
__device__ __forceinline__ void hub_final(const DecideArgs<WT, RO> &a, const HubPlan &p, const uint8_t *flag, int wg,
                                          int nw, End end, Rescan rescan)
{
    const int lane = threadIdx.x & 31;
    for (int i = wg; i < p.H; i += nw) {
        const int v = p.hubs[i];
        if (!flag[v] || stopped(a, v)) continue;
        const Scale sc = scale_of(a, v);
        const int cur = a.comm[v];
        const WT ki = a.K[v], sf = a.Self[v], tcur = a.Tot[cur];
        Cand<WT> best(cur);
        WT wc = 0;
        const long long q1 = end(i);
        for (long long q = p.tcoff[i] + lane; q < q1; q += 32) {
            WT own;
            best.merge(hub_get(p, q, best, own));
            wc += own;
        }
        warp_merge(best, wc, 32);
        int bc = best.c;
        int dec = best.decide(a.fp64_only, sc, cur, wc, sf, ki);  // warp-uniform
        if (dec == 2) {
            double dq = 0.0;
            int fc = cur;
            if (needs_fp64(a, sc, ki)) {  // chunk-wise FP64 partials from k_hub_scan
                for (long long q = p.tcoff[i] + lane; q < q1; q += 32)
                    if (cand_better(p.pdq[q], p.pfc[q], dq, fc)) {
                        dq = p.pdq[q];
                        fc = p.pfc[q];
                    }
            } else {  // rare rounding cases
                rescan(i, v, sc, GainTerms<WT>(sc, ki, tcur), best, cur, ki, tcur, dq, fc);
            }
            warp_argmax(dq, fc);
            bc = fc;
            dec = (fc != cur && gain_correct(dq, wc, sf) > 0.0) ? 1 : 0;
            if (lane == 0) atomicAdd(a.fp64_decisions, 1ull);
        }
        const bool move = lane == 0 && dec == 1 && guard_ok(a, cur, bc);
        append_mover(a, move, v, cur, bc);
    }
}

// The same over the hubs' tables.
template <typename WT, bool RO>
__device__ __forceinline__ void hub_final(const DecideArgs<WT, RO> &a, const HubPlan &p, const uint8_t *flag, int wg,
                                          int nw)
{
    hub_final(
        a, p, flag, wg, nw, [&](int i) { return p.tcoff[i + 1]; },
        [&](int i, int, const Scale &sc, const GainTerms<WT> &gt, const Cand<WT> &best, int cur, WT ki, WT tcur,
            double &dq, int &fc) {
            scan_table(a, sc, gt, best, p.pool + p.toff[i], hub_vals<WT>(p, i), (int)p.T[i], threadIdx.x & 31, 32, cur,
                       ki, tcur, dq, fc);
        });
}

// ------------------------------------------------------------------------
// Weight update + pruning (compute_In / compute_In_blk,
// kernel_functions.cu:890-1034): In[v] over the new labels, the pruning
// bound, next active lists, sum of In.
// ------------------------------------------------------------------------
template <typename WT, bool RO = true>
struct UpdateArgs {
    const int64_t *__restrict__ offs;
    const int32_t *__restrict__ nbr;
    const WT *__restrict__ w;
    typename SweepPtr<int32_t, RO>::type comm;
    typename SweepPtr<WT, RO>::type K;
    typename SweepPtr<WT, RO>::type Self;
    typename SweepPtr<WT, RO>::type Tot;
    WT *In;
    uint8_t *act_flag;  // per-vertex copy of the next active set
    int32_t *act_list;  // next active list, segment of this bin
    int *act_counter;
    DevStats *st;
    double constant;
    long long m2;
    int next;
    // batched graphs (null for one graph)
    const int32_t *__restrict__ gid;
    const long long *__restrict__ m2g;
    const double *__restrict__ cg;
    const uint8_t *__restrict__ stop;
    const int32_t *__restrict__ min_tot_g;
};

// Per-vertex prune parameters: the graph's m2, 1/m2 and min Tot; `stop` when
// the vertex's graph has stopped (no update, never active).
struct PruneScale {
    long long m2;
    double c;
    long long min_tot;
    bool stop;
};
template <typename WT, bool RO>
__device__ __forceinline__ PruneScale prune_scale(const UpdateArgs<WT, RO> &a, int v, long long min_tot)
{
    if (a.gid) {
        const int g = a.gid[v];
        return PruneScale{a.m2g[g], a.cg[g], a.min_tot_g[g], a.stop[g] != 0};
    }
    return PruneScale{a.m2, a.constant, min_tot, false};
}

// A thread's share of the sweep's sums: In, row entries and vertices of the
// next active set.
struct UpdateSums {
    unsigned long long in = 0, edges = 0;
    int act = 0;
};

// Weight of the own-community entries of a row among the entries first,
// first + G, ...: U entries per lane in flight (predicated, so that a short
// row's loads are all in flight together).
template <typename WT, int G, int U, bool W, bool RO>
__device__ __forceinline__ WT own_weight(const UpdateArgs<WT, RO> &a, long long s, int deg, int first, int cur)
{
    const int32_t *rn = a.nbr + s;
    const WT *rw = W ? a.w + s : nullptr;
    WT sum = 0;
    for (int j0 = first; j0 < deg; j0 += U * G) {
        int u[U];
#pragma unroll
        for (int q = 0; q < U; ++q) u[q] = j0 + q * G < deg ? rn[j0 + q * G] : -1;
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (u[q] >= 0) u[q] = a.comm[u[q]];
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (u[q] == cur) sum += W ? rw[j0 + q * G] : (WT)1;
    }
    return sum;
}

// A warp takes the tasks (32 / G vertices each) wg, wg + nw, ... of the list.
template <typename WT, int G, int U, bool W, bool RO>
__device__ __forceinline__ void update_group(const UpdateArgs<WT, RO> &a, const int32_t *list, int count,
                                             long long min_tot, int wg, int nw, WarpStage<kStageN, 1> &stage,
                                             UpdateSums &sums)
{
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), gw = lane / G;
    constexpr int GPW = 32 / G;
    int *const lists[1] = {a.act_list};
    for (int base = wg * GPW; base < count; base += nw * GPW) {
        const int idx = base + gw;
        bool has = idx < count;
        int v = 0, cur = -1;
        long long s = 0, e = 0;
        PruneScale ps{a.m2, a.constant, min_tot, false};
        if (has) {
            v = list[idx];
            ps = prune_scale(a, v, min_tot);
            if (ps.stop) has = false;
        }
        if (has) {
            s = a.offs[v];
            e = a.offs[v + 1];
            cur = a.comm[v];
        }
        WT sum = own_weight<WT, G, U, W>(a, s, (int)(e - s), sub, cur);
#pragma unroll
        for (int o = G / 2; o >= 1; o >>= 1) sum += __shfl_xor_sync(GALA_FULL_MASK, sum, o);
        bool active = false;
        if (ps.stop && sub == 0) a.act_flag[v] = 0;
        if (has && sub == 0) {
            a.In[v] = sum;
            const WT ki = a.K[v];
            active = !prune_bound_fast<WT>(sum, a.Self[v], ki, (WT)ps.min_tot, a.Tot[cur], ps.c, ps.m2);
            a.act_flag[v] = active;
            sums.in += (unsigned long long)sum;
            if (active) {
                sums.edges += (unsigned long long)(e - s);
                sums.act += 1;
            }
        }
        const int item[1] = {v};
        stage.push(active, item, lists, a.act_counter);
    }
    stage.flush(lists, a.act_counter);
}

// The block takes the vertices b0, b0 + nb, ... of the list.
template <typename WT, bool W, bool RO>
__device__ __forceinline__ void update_cta(const UpdateArgs<WT, RO> &a, const int32_t *list, int count,
                                           long long min_tot, int b0, int nb, UpdateSums &sums)
{
    __shared__ WT red[32];
    for (int i = b0; i < count; i += nb) {
        const int v = list[i];
        const PruneScale ps = prune_scale(a, v, min_tot);
        if (ps.stop) {  // block-uniform
            if (threadIdx.x == 0) a.act_flag[v] = 0;
            continue;
        }
        const long long s = a.offs[v], e = a.offs[v + 1];
        const int cur = a.comm[v];
        WT sum = 0;
#pragma unroll 4
        for (long long j = s + threadIdx.x; j < e; j += blockDim.x)
            if (a.comm[a.nbr[j]] == cur) sum += W ? a.w[j] : 1;
        sum = warp_sum(sum);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            sum = 0;
            for (int q = 0; q < (int)(blockDim.x >> 5); ++q) sum += red[q];
            a.In[v] = sum;
            const WT ki = a.K[v];
            bool active = !prune_bound_fast<WT>(sum, a.Self[v], ki, (WT)ps.min_tot, a.Tot[cur], ps.c, ps.m2);
            a.act_flag[v] = active;
            sums.in += (unsigned long long)sum;
            if (active) {
                a.act_list[atomicAdd(a.act_counter, 1)] = v;
                sums.edges += (unsigned long long)(e - s);
                sums.act += 1;
            }
        }
        __syncthreads();
    }
}

// Weight update of the hub bin: In[v] of a hub row summed by many CTAs (one
// per 4096-entry chunk, the chunks of the hub plan) with integer atomics into
// zeroed In, then one thread per hub evaluates the pruning bound.
template <typename WT, bool W, bool RO>
__device__ __forceinline__ void hub_in_partial(const UpdateArgs<WT, RO> &a, const HubPlan &p, int bid, int nb)
{
    __shared__ WT red[32];
    for (long long wi = bid; wi < p.nwork; wi += nb) {
        const int i = p.work[wi];
        const int v = p.hubs[i];
        if (a.gid && a.stop[a.gid[v]]) continue;  // block-uniform
        const long long e = a.offs[v + 1];
        const long long s = a.offs[v] + (wi - p.coff[i]) * kHubChunk;
        const long long e2 = s + kHubChunk < e ? s + kHubChunk : e;
        const int cur = a.comm[v];
        WT sum = 0;
#pragma unroll 4
        for (long long j = s + threadIdx.x; j < e2; j += blockDim.x)
            if (a.comm[a.nbr[j]] == cur) sum += W ? a.w[j] : 1;
        sum = warp_sum(sum);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            WT t = 0;
            for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += red[q];
            if (t) atomic_add_w(&a.In[v], t);
        }
        __syncthreads();
    }
}

template <typename WT, bool RO>
__device__ __forceinline__ void hub_in_final(const UpdateArgs<WT, RO> &a, const HubPlan &p, long long min_tot, int bid,
                                             int nb, UpdateSums &sums)
{
    const int stride = nb * blockDim.x;
    for (int base = bid * blockDim.x; base < p.H; base += stride) {  // warp-uniform trip count
        const int i = base + threadIdx.x;
        bool active = false;
        int v = 0;
        if (i < p.H) {
            v = p.hubs[i];
            const PruneScale ps = prune_scale(a, v, min_tot);
            if (ps.stop) {
                a.act_flag[v] = 0;
            } else {
                const WT sum = a.In[v];
                const WT ki = a.K[v];
                active = !prune_bound_fast<WT>(sum, a.Self[v], ki, (WT)ps.min_tot, a.Tot[a.comm[v]], ps.c, ps.m2);
                a.act_flag[v] = active;
                sums.in += (unsigned long long)sum;
                if (active) {
                    sums.edges += (unsigned long long)(a.offs[v + 1] - a.offs[v]);
                    sums.act += 1;
                }
            }
        }
        warp_append(active, v, a.act_list, a.act_counter);
    }
}

}  // namespace gala
