// batch_cta.cu - a batch of small graphs in one persistent launch: every CTA
// takes graphs from a queue (largest first) and runs the whole multi-round
// Louvain of a graph on its own - phase 1 sweeps, the convergence rule, the
// contraction and the round rule - with block barriers between the steps and
// no host round trip.  Batching has no counterpart in the reference; every
// graph follows the single-graph rules of the reference
// (louvain_main_process.cu:571-1034 for phase 1, build_compressed_graph.cu
// for the contraction, louvain.cu:193-226 for the rounds), so its partition,
// modularity and community count equal its single-graph run.
//
// Decisions follow the single-graph engine: candidates are ordered by the
// exact integer gain numerator X = w m2 - K ((Tot_c - Tot_cur) + K), and the
// cases where the reference's FP64 rounding could decide (equal best X from
// different weights, X = 0, a corrected gain of 0, K m2 >= 2^49) are
// re-evaluated with its FP64 expressions.
//
// A level has at most kCtaMaxN vertices, so its labels (16 bits, old and new)
// and community totals live in shared memory: the gathers that bound a sweep,
// one label per entry and one total per candidate, take a few bank conflicts
// instead of 32 L1 tag lookups.  Neighbour-community weights are summed per
// warp: rows of at most 32 entries by a warp match; longer ones in a dense
// table of the warp when the level has at most kDense communities, in its hash
// table up to kWRow entries, else in a dense global table, read and cleared
// with one atomic exchange per entry.  A warp takes a run of consecutive
// vertices, loads their row bounds and degrees one per lane and has the next
// vertex's first entries in flight while it decides one.
// 4,096 planted-partition graphs of 200-3500 vertices, 121M entries: 31.4 ms
// with labels and totals in global memory and a hash table per row, 15.4 ms
// so (15.6 with the copies of the graphs from page-locked memory).
#include "common.cuh"
#include "internal.h"
#include "scan.cuh"

namespace gala {

namespace {

constexpr int kCtaThreads = 512;
constexpr int kCtaWarps = kCtaThreads / 32;
constexpr int kWT = 256;  // slots of a warp's hash table
constexpr int kWTLog = 8;
constexpr int kWRow = kWT / 2;   // longest row (entries) the hash table takes
constexpr int kDense = 2 * kWT;  // communities of a warp's dense table

// Level graph as seen by one graph's CTA: level 0 reads the union CSR
// (64-bit global offsets, union ids), later levels the graph's own
// contracted CSR (32-bit local starts and lengths, local ids).
struct LevelView {
    const int64_t *o64;
    const int32_t *o32, *len;
    long long obase;
    const int32_t *nbr;
    int shift;
    const int32_t *w;
    __device__ __forceinline__ int beg(int v) const { return o64 ? (int)(o64[v] - obase) : o32[v]; }
    __device__ __forceinline__ int end(int v) const { return o64 ? (int)(o64[v + 1] - obase) : o32[v] + len[v]; }
    __device__ __forceinline__ int nb(int j) const { return nbr[j] - shift; }
    __device__ __forceinline__ int wt(int j) const { return w ? w[j] : 1; }
};

struct CtaShared {
    long long red_ll[kCtaWarps];
    unsigned long long red_u[kCtaWarps];
    int red_i[kCtaWarps];
    long long scan_wt[32];
    long long scan_tot;
    int graph;
    // in dynamic shared memory
    int *tab;               // 2 kWT ints per warp: hash keys and sums, or a dense table
    unsigned short *occ;    // kWRow claimed slots per warp
    int *Tot;               // nmax
    unsigned short *lab, *cur;  // nmax: labels before and after a sweep
    unsigned char *act;     // nmax: active vertices
};
constexpr size_t cta_smem(int nmax)
{
    const size_t n = (size_t)((nmax + 31) & ~31);
    return (size_t)kCtaWarps * (kDense * sizeof(int) + kWRow * sizeof(unsigned short)) + n * (4 + 2 + 2 + 1);
}

__device__ __forceinline__ long long cta_sum_ll(long long v, long long *red)
{
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    long long t = 0;
    for (int q = 0; q < kCtaWarps; ++q) t += red[q];
    return t;
}

__device__ __forceinline__ unsigned long long cta_sum_u64(unsigned long long v, unsigned long long *red)
{
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    unsigned long long t = 0;
    for (int q = 0; q < kCtaWarps; ++q) t += red[q];
    return t;
}

__device__ __forceinline__ int cta_min_int(int v, int *red)
{
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v = min(v, __shfl_xor_sync(GALA_FULL_MASK, v, o));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    int t = 0x7fffffff;
    for (int q = 0; q < kCtaWarps; ++q) t = min(t, red[q]);
    return t;
}

// out[i] = sum_{j<i} f(j) for i < n (block-wide; returns the total).
template <typename F>
__device__ __forceinline__ int cta_exclusive_scan(int n, F f, int *out, long long *wt, long long *tot)
{
    long long carry = 0;
    for (int base = 0; base < n; base += kCtaThreads) {
        const int i = base + threadIdx.x;
        const long long v = i < n ? f(i) : 0;
        const long long ex = block_exclusive_scan<long long>(v, wt, tot);
        if (i < n) out[i] = (int)(carry + ex);
        carry += *tot;
        __syncthreads();
    }
    return (int)carry;
}

// Best candidate across the warp: larger gain, then the lower id.
__device__ __forceinline__ void warp_best(double &dq, int &c)
{
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const double od = __shfl_xor_sync(GALA_FULL_MASK, dq, o);
        const int oc = __shfl_xor_sync(GALA_FULL_MASK, c, o);
        if (cand_better(od, oc, dq, c)) {
            dq = od;
            c = oc;
        }
    }
}

// Q from exact sums with the engine's FP64 expression (sum_in/m2 - t2/m2^2).
__device__ __forceinline__ double q_of_sums(unsigned long long sum_in, unsigned long long sum_tot2, long long m2)
{
    const double c = 1.0 / (double)m2;
    return __dsub_rn(__dmul_rn((double)(long long)sum_in, c), __dmul_rn(__dmul_rn((double)sum_tot2, c), c));
}

// Empty tables: hash keys -1 and sums 0, or all 0 for dense use.
__device__ __forceinline__ void clear_tables(CtaShared &sh, bool dense)
{
    for (int i = threadIdx.x; i < kCtaWarps * kDense; i += kCtaThreads) sh.tab[i] = !dense && (i & kWT) == 0 ? -1 : 0;
}

// Add w to key's slot (claiming an empty one); at most kWRow distinct keys
// go to a table of kWT slots, so the probe always ends.
__device__ __forceinline__ int wt_add(int *tab, int key, int w, bool &created)
{
    unsigned h = ((unsigned)key * 0x9E3779B1u) >> (32 - kWTLog);
    for (int p = 0; p < kWT; ++p) {
        const int k = atomicCAS(&tab[h], -1, key);
        if (k == -1 || k == key) {
            created = k == -1;
            atomicAdd(&tab[kWT + h], w);
            return (int)h;
        }
        h = (h + 1) & (kWT - 1);
    }
    created = false;
    return -1;
}

// Entries of several rows, gathered by a warp: add(j) for every entry j of
// rows r0 .. r1 - 1 ([rb(r), re(r))).  The bounds of 32 rows are loaded at
// once; fn(j, ok) is called by all lanes.
template <typename RB, typename RE, typename FN>
__device__ __forceinline__ void for_entries(int r0, int r1, RB rb, RE re, FN fn)
{
    const int lane = threadIdx.x & 31;
    for (int q0 = r0; q0 < r1; q0 += 32) {
        const int q = q0 + lane;
        int b = 0, e = 0;
        if (q < r1) {
            b = rb(q);
            e = re(q);
        }
        const int rows = r1 - q0 < 32 ? r1 - q0 : 32;
        for (int r = 0; r < rows; ++r) {
            const int rbeg = __shfl_sync(GALA_FULL_MASK, b, r), rend = __shfl_sync(GALA_FULL_MASK, e, r);
            for (int j0 = rbeg; j0 < rend; j0 += 32) fn(j0 + lane, j0 + lane < rend);
        }
    }
}

// Sum the weights per key over the entries of rows [r0, r1) (row r holds
// entries [rb(r), re(r)); entry j has key kf(j) and weight wf(j), positive);
// then emit(key, sum, pos) once per distinct key, pos = 0, 1, ... over the
// keys.  total (warp-uniform) is the number of entries; dense: every key is
// below nkeys <= kDense and the tables are in dense use.  All 32 lanes call;
// returns the number of keys.
template <typename RB, typename RE, typename KF, typename WF, typename EM>
__device__ __forceinline__ int warp_aggregate(int *tab, unsigned short *occ, int *gacc, bool dense, int nkeys, int r0,
                                              int r1, int total, RB rb, RE re, KF kf, WF wf, EM emit)
{
    const int lane = threadIdx.x & 31;
    int n = 0;
    if (dense) {
        for_entries(r0, r1, rb, re, [&](int j, bool ok) {
            if (ok) atomicAdd(&tab[kf(j)], wf(j));
        });
        __syncwarp();
        for (int c0 = 0; c0 < nkeys; c0 += 32) {
            const int c = c0 + lane;
            const int sum = c < nkeys ? tab[c] : 0;
            const unsigned m = __ballot_sync(GALA_FULL_MASK, sum != 0);
            if (sum != 0) {
                tab[c] = 0;
                emit(c, sum, n + __popc(m & lanemask_lt()));
            }
            n += __popc(m);
        }
        __syncwarp();
    } else if (total <= kWRow) {
        for_entries(r0, r1, rb, re, [&](int j, bool ok) {
            bool cr = false;
            int slot = -1;
            if (ok) slot = wt_add(tab, kf(j), wf(j), cr);
            const unsigned cb = __ballot_sync(GALA_FULL_MASK, cr);
            if (cr) occ[n + __popc(cb & lanemask_lt())] = (unsigned short)slot;
            n += __popc(cb);
        });
        __syncwarp();
        for (int q = lane; q < n; q += 32) {
            const int sl = occ[q];
            const int key = tab[sl], sum = tab[kWT + sl];
            tab[sl] = -1;
            tab[kWT + sl] = 0;
            emit(key, sum, q);
        }
        __syncwarp();
    } else {
        for_entries(r0, r1, rb, re, [&](int j, bool ok) {
            if (ok) atomicAdd(&gacc[kf(j)], wf(j));
        });
        __syncwarp();
        for_entries(r0, r1, rb, re, [&](int j, bool ok) {
            int key = -1, sum = 0;
            if (ok) {
                key = kf(j);
                sum = atomicExch(&gacc[key], 0);
            }
            const unsigned got = __ballot_sync(GALA_FULL_MASK, sum != 0);
            if (sum != 0) emit(key, sum, n + __popc(got & lanemask_lt()));
            n += __popc(got);
        });
        __syncwarp();
    }
    return n;
}

// Candidate merge by exact gain numerator: larger X, then the lower id; t
// records a tie on the best X between different weights.
__device__ __forceinline__ void merge_x(long long &x, int &c, int &w, int &t, long long ox, int oc, int ow)
{
    if (ox == x) {
        t |= ow != w;
        if (oc < c) {
            c = oc;
            w = ow;
        }
    } else if (ox > x) {
        x = ox;
        c = oc;
        w = ow;
        t = 0;
    }
}

// The warp's best of the lanes' candidates (x >= 0, ids distinct over the
// lanes; x = -1: none), by the same rule; c = none when there is none.
__device__ __forceinline__ void warp_best_x(long long &x, int &c, int w, int &t, int none)
{
    const int mh = __reduce_max_sync(GALA_FULL_MASK, (int)(x >> 32));
    if (mh < 0) {  // warp-uniform
        x = -1;
        c = none;
        t = 0;
        return;
    }
    const bool top = (int)(x >> 32) == mh;
    const unsigned ml = __reduce_max_sync(GALA_FULL_MASK, top ? (unsigned)x : 0u);
    const bool win = top && (unsigned)x == ml;
    const unsigned wins = __ballot_sync(GALA_FULL_MASK, win);
    int src = __ffs((int)wins) - 1;
    if (wins & (wins - 1)) {  // several: the lowest id; a tie in any of their lanes or between them counts
        const int bc = (int)__reduce_min_sync(GALA_FULL_MASK, win ? (unsigned)c : 0xffffffffu);
        const int bw = __shfl_sync(GALA_FULL_MASK, w, src);
        t = __any_sync(GALA_FULL_MASK, win && (t || w != bw));
        src = __ffs((int)__ballot_sync(GALA_FULL_MASK, win && c == bc)) - 1;
    } else {
        t = __shfl_sync(GALA_FULL_MASK, t, src);
    }
    c = __shfl_sync(GALA_FULL_MASK, c, src);
    x = ((long long)mh << 32) | ml;
}

// Decision of one vertex by a warp: its new label.
__device__ __forceinline__ int decide_vertex(const LevelView &g, const CtaShared &sh, int *gacc, const int *size,
                                             bool dense, int n, long long m2, int b, int e, int ki, int sf, int cv,
                                             int u0, int w0)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int deg = e - b, tcur = sh.Tot[cv];
    const unsigned short *lab = sh.lab;
    int *tab = sh.tab + wid * kDense;
    unsigned short *occ = sh.occ + wid * kWRow;
    const long long xb = (long long)ki * ((long long)ki - (long long)tcur);
    auto gain = [&](int s, int tot) { return (long long)s * m2 - (long long)ki * (long long)tot - xb; };
    // per lane: its best candidate; for a matched row its one sum
    long long x = -1;
    int bc = cv, bw = 0, bt = 0, wc = 0, ms = 0, mc = -1, mt = 0;
    bool lead = false;
    const bool match = deg <= 32;
    auto rows = [&](auto emit) {
        warp_aggregate(
            tab, occ, gacc, dense, n, 0, 1, deg, [=](int) { return b; }, [=](int) { return e; },
            [&](int j) { return (int)lab[g.nb(j)]; }, [&](int j) { return g.wt(j); }, emit);
    };
    if (match) {
        const bool ok = lane < deg;
        mc = ok ? (int)lab[u0] : -1;
        const unsigned m = __match_any_sync(GALA_FULL_MASK, mc);
        ms = g.w ? match_sum(m, ok, w0) : __popc(m);
        lead = ok && __ffs((int)m) - 1 == lane;
        const unsigned own = __ballot_sync(GALA_FULL_MASK, lead && mc == cv);
        if (own) wc = __shfl_sync(GALA_FULL_MASK, ms, __ffs((int)own) - 1);
        lead = lead && mc != cv;
        if (lead) {
            mt = sh.Tot[mc];
            const long long xx = gain(ms, mt);
            if (xx >= 0) {
                x = xx;
                bc = mc;
                bw = ms;
            }
        }
    } else {
        rows([&](int c, int s, int) {
            if (c == cv) {
                wc += s;
            } else {
                const long long xx = gain(s, sh.Tot[c]);
                if (xx >= 0) merge_x(x, bc, bw, bt, xx, c, s);
            }
        });
        wc = (int)__reduce_add_sync(GALA_FULL_MASK, (unsigned)wc);
    }
    warp_best_x(x, bc, bw, bt, cv);
    // 0 stay, 1 move, 2 the FP64 expressions decide (warp-uniform)
    int dec;
    if ((long long)ki * m2 >= (1LL << 49))
        dec = 2;
    else if (bc == cv)
        dec = 0;
    else if (x == 0)
        dec = wc == sf ? 2 : 0;
    else if (bt)
        dec = 2;
    else {
        const long long y = x - (long long)(wc - sf) * m2;
        dec = y == 0 ? 2 : (y > 0 ? 1 : 0);
    }
    if (dec == 2) {
        const double constant = 1.0 / (double)m2;
        double bdq = 0.0;
        int fc = cv;
        auto offer = [&](int c, int s, int tot) {
            const double d = gain_dq<int>(s, ki, tot, tcur, constant);
            if (d > 0.0 && cand_better(d, c, bdq, fc)) {
                bdq = d;
                fc = c;
            }
        };
        if (match) {
            if (lead) offer(mc, ms, mt);
        } else {
            rows([&](int c, int s, int) {
                if (c != cv) offer(c, s, sh.Tot[c]);
            });
        }
        warp_best(bdq, fc);
        bc = fc;
        dec = (fc != cv && gain_correct<int>(bdq, wc, sf) > 0.0) ? 1 : 0;
    }
    return dec == 1 && !(size[bc] == 1 && size[cv] == 1 && bc > cv) ? bc : cv;
}

// Moves of a sweep into (sign = 1) or out of (-1) the community totals.
__device__ __forceinline__ void move_tot(CtaShared &sh, const int *K, int n, int sign, int *size)
{
    for (int v = threadIdx.x; v < n; v += kCtaThreads) {
        const int to = sh.cur[v], from = sh.lab[v];
        if (to != from) {
            const int k = sign * K[v];
            atomicAdd(&sh.Tot[to], k);
            atomicSub(&sh.Tot[from], k);
            if (size) {
                atomicAdd(&size[to], 1);
                atomicSub(&size[from], 1);
            }
        }
    }
}

// K and Self of level 0: row weight and self-loop weight (the last one listed),
// a group of eight lanes per row.
__device__ void cta_rows0(const LevelView &g, int n, int *K, int *Self)
{
    const int lane = threadIdx.x & 31, sub = lane & 7;
    for (int v0 = (threadIdx.x >> 5) * 4; v0 < n; v0 += kCtaWarps * 4) {
        const int v = v0 + (lane >> 3);
        int k = 0, sf = 0, at = -1;
        if (v < n) {
            const int e = g.end(v);
            for (int j = g.beg(v) + sub; j < e; j += 8) {
                const int w = g.wt(j);
                k += w;
                if (g.nb(j) == v) {
                    sf = w;
                    at = j;
                }
            }
        }
#pragma unroll
        for (int o = 4; o >= 1; o >>= 1) {
            k += __shfl_xor_sync(GALA_FULL_MASK, k, o);
            const int of = __shfl_xor_sync(GALA_FULL_MASK, sf, o), oa = __shfl_xor_sync(GALA_FULL_MASK, at, o);
            if (oa > at) {
                sf = of;
                at = oa;
            }
        }
        if (v < n && sub == 0) {
            K[v] = k;
            Self[v] = sf;
        }
    }
}

// Phase 1 of one level (the oracle's phase1 rule) from given K and Self:
// labels in sh.lab and their totals in sh.Tot on return.
__device__ void cta_phase1(const BatchCtaArgs &a, const LevelView &g, int n, long long m2, int vb, int *gacc,
                           CtaShared &sh, double *q_out, int *iters_out)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int *K = a.K + vb, *Self = a.Self + vb;
    int *size = a.size + vb;
    const double constant = 1.0 / (double)m2;
    const bool dense = n <= kDense;
    clear_tables(sh, dense);
    // Tot = K, label = own id, size 1, every vertex active
    unsigned long long s_in = 0, s_t2 = 0;
    for (int v = threadIdx.x; v < n; v += kCtaThreads) {
        const int k = K[v];
        sh.Tot[v] = k;
        size[v] = 1;
        sh.lab[v] = (unsigned short)v;
        sh.act[v] = 1;
        s_in += (unsigned long long)Self[v];
        s_t2 += (unsigned long long)((long long)k * k);
    }
    s_in = cta_sum_u64(s_in, sh.red_u);
    s_t2 = cta_sum_u64(s_t2, sh.red_u);
    double prev_q = q_of_sums(s_in, s_t2, m2);
    int iters = 0;
    // runs of consecutive vertices per warp and pass, at most 32
    const int passes = (n + kCtaThreads - 1) / kCtaThreads;
    const int run = (n + kCtaWarps * passes - 1) / (kCtaWarps * passes);
    __syncthreads();
    for (;;) {
        // decide-and-move: every decision reads the labels and totals of the
        // previous iteration
        for (int v0 = wid * run; v0 < n; v0 += kCtaWarps * run) {
            const int v = v0 + lane;
            const bool has = lane < run && v < n;
            int b = 0, e = 0, k = 0, sf = 0, l = 0;
            if (has) {
                l = sh.lab[v];
                sh.cur[v] = (unsigned short)l;
                if (sh.act[v]) {
                    b = g.beg(v);
                    e = g.end(v);
                    k = K[v];
                    sf = Self[v];
                }
            }
            __syncwarp();  // lane 0 may write a label again below
            unsigned todo = __ballot_sync(GALA_FULL_MASK, e > b);
            int un = -1, wn = 0;  // the next vertex's first entries
            auto fetch = [&](int i) {
                const int j = __shfl_sync(GALA_FULL_MASK, b, i) + lane;
                const bool ok = j < __shfl_sync(GALA_FULL_MASK, e, i);
                un = ok ? g.nb(j) : 0;
                wn = ok ? g.wt(j) : 0;
            };
            if (todo) fetch(__ffs((int)todo) - 1);
            while (todo) {  // warp-uniform
                const int i = __ffs((int)todo) - 1;
                todo &= todo - 1;
                const int u0 = un, w0 = wn;
                if (todo) fetch(__ffs((int)todo) - 1);
                const int cv = __shfl_sync(GALA_FULL_MASK, l, i);
                const int nl = decide_vertex(g, sh, gacc, size, dense, n, m2, __shfl_sync(GALA_FULL_MASK, b, i),
                                             __shfl_sync(GALA_FULL_MASK, e, i), __shfl_sync(GALA_FULL_MASK, k, i),
                                             __shfl_sync(GALA_FULL_MASK, sf, i), cv, u0, w0);
                if (nl != cv && lane == 0) sh.cur[v0 + i] = (unsigned short)nl;
                __syncwarp();
            }
        }
        __syncthreads();
        move_tot(sh, K, n, 1, size);
        __syncthreads();
        // min Tot over non-empty communities (m2 when none) and sum Tot^2
        int mn = 0x7fffffff;
        s_t2 = 0;
        for (int c = threadIdx.x; c < n; c += kCtaThreads) {
            const int t = sh.Tot[c];
            if (t != 0) {
                mn = min(mn, t);
                s_t2 += (unsigned long long)((long long)t * t);
            }
        }
        mn = cta_min_int(mn, sh.red_i);
        s_t2 = cta_sum_u64(s_t2, sh.red_u);
        const int min_tot = mn == 0x7fffffff ? (int)m2 : mn;
        // weight update and pruning (compute_In): eight lanes per vertex
        unsigned long long my_in = 0;
        const int sub = lane & 7;
        for (int v0 = wid * 4; v0 < n; v0 += kCtaWarps * 4) {
            const int v = v0 + (lane >> 3);
            int b = 0, e = 0, c = -1, s = 0;
            if (v < n) {
                b = g.beg(v);
                e = g.end(v);
                c = sh.cur[v];
            }
            constexpr int U = 4;
            for (int j0 = b + sub; j0 < e; j0 += 8 * U) {
                int u[U];
#pragma unroll
                for (int q = 0; q < U; ++q) u[q] = j0 + 8 * q < e ? g.nb(j0 + 8 * q) : -1;
#pragma unroll
                for (int q = 0; q < U; ++q)
                    if (u[q] >= 0 && (int)sh.cur[u[q]] == c) s += g.wt(j0 + 8 * q);
            }
#pragma unroll
            for (int o = 4; o >= 1; o >>= 1) s += __shfl_xor_sync(GALA_FULL_MASK, s, o);
            if (sub == 0 && e > b) {
                my_in += (unsigned long long)s;
                sh.act[v] = !prune_bound_fast<int>(s, Self[v], K[v], min_tot, sh.Tot[c], constant, m2);
            }
        }
        s_in = cta_sum_u64(my_in, sh.red_u);
        const double q = q_of_sums(s_in, s_t2, m2);
        ++iters;
        if (q - prev_q < a.min_mod) break;  // the iteration's partition is dropped
        prev_q = q;
        __syncthreads();
        if (threadIdx.x == 0) {
            unsigned short *t = sh.lab;
            sh.lab = sh.cur;
            sh.cur = t;
        }
        __syncthreads();
    }
    move_tot(sh, K, n, -1, nullptr);
    __syncthreads();
    *q_out = prev_q;
    *iters_out = iters;
}

// Contraction of a level by its labels (sh.lab): dense renumbering in
// ascending label order, member lists, new rows in buffer `nb` (any order, at
// starts bounded by min(entries, C), lengths apart), K and Self of the new
// vertices.  Returns C; sh.lab receives every vertex's new id.
__device__ int cta_contract(const BatchCtaArgs &a, const LevelView &g, int n, int vb, long long eb, int g_idx, int nb,
                            int *gacc, CtaShared &sh)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int *members = a.members + vb, *ec = a.ec + vb, *moff = a.moff + vb + g_idx;
    int *K = a.K + vb, *Self = a.Self + vb;
    int32_t *noffs = a.loffs[nb] + vb + g_idx, *len = a.llen[nb] + vb;
    int32_t *nnbr = a.lnbr[nb] + eb, *nw = a.lw[nb] + eb;
    // members per label in the tables' memory, then the start of their run
    int *cnt = sh.tab;
    static_assert(kCtaWarps * kDense >= kCtaMaxN, "a count per label");
    for (int c = threadIdx.x; c < n; c += kCtaThreads) {
        cnt[c] = 0;
        ec[c] = 0;
    }
    __syncthreads();
    for (int v = threadIdx.x; v < n; v += kCtaThreads) atomicAdd(&cnt[sh.lab[v]], 1);
    __syncthreads();
    long long carry = 0;  // new ids in the high word, members in the low word
    for (int t = 0; t < n; t += kCtaThreads) {
        const int c = t + threadIdx.x;
        const int k = c < n ? cnt[c] : 0;
        const long long x = carry + block_exclusive_scan<long long>(k ? (1LL << 32) + k : 0, sh.scan_wt, &sh.scan_tot);
        if (k) {
            const int id = (int)(x >> 32);
            sh.cur[c] = (unsigned short)id;
            moff[id] = (int)x;
            cnt[c] = (int)x;
            K[id] = sh.Tot[c];
        }
        carry += sh.scan_tot;
        __syncthreads();
    }
    const int C = (int)(carry >> 32);
    if (threadIdx.x == 0) moff[C] = n;
    for (int v = threadIdx.x; v < n; v += kCtaThreads) {
        const int old = sh.lab[v], c = sh.cur[old];
        members[atomicAdd(&cnt[old], 1)] = v;
        atomicAdd(&ec[c], g.end(v) - g.beg(v));
        sh.lab[v] = (unsigned short)c;
    }
    __syncthreads();
    const bool dense = C <= kDense;
    clear_tables(sh, dense);
    cta_exclusive_scan(C, [&](int c) { return min(ec[c], C); }, noffs, sh.scan_wt, &sh.scan_tot);
    __syncthreads();
    // one warp per community: sums per neighbour community over its members'
    // rows
    for (int c = wid; c < C; c += kCtaWarps) {
        const int o = noffs[c], total = ec[c];
        int self = 0;
        const int k = warp_aggregate(
            sh.tab + wid * kDense, sh.occ + wid * kWRow, gacc, dense, C, moff[c], moff[c + 1], total,
            [&](int mi) { return g.beg(members[mi]); }, [&](int mi) { return g.end(members[mi]); },
            [&](int j) { return (int)sh.lab[g.nb(j)]; }, [&](int j) { return g.wt(j); },
            [&](int d, int s, int pos) {
                nnbr[o + pos] = d;
                nw[o + pos] = s;
                if (d == c) self = s;
            });
        self = (int)__reduce_add_sync(GALA_FULL_MASK, (unsigned)self);
        if (lane == 0) {
            len[c] = k;
            Self[c] = self;
        }
    }
    __syncthreads();
    return C;
}

// to[0, n) = from[0, n) (1 where from is null), from in host memory behind the
// chip-to-chip link: eight loads in flight per thread.
template <typename T, typename Put>
__device__ __forceinline__ void cta_copy(const T *__restrict__ from, int n, Put put)
{
    constexpr int U = 8;
    for (int j0 = threadIdx.x; j0 < n; j0 += U * kCtaThreads) {
        T t[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + u * kCtaThreads;
            t[u] = j < n && from ? from[j] : (T)1;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int j = j0 + u * kCtaThreads;
            if (j < n) put(j, t[u]);
        }
    }
}

// The CTA's graph from host memory to its part of the union CSR.  A gather of
// the whole batch ahead of this kernel runs at the link's rate with the SMs idle
// (4096 graphs, 0.5 GB: 2.9 ms of 20.3); here the other CTAs work meanwhile.
__device__ __forceinline__ void cta_gather(const BatchCtaArgs &a, int gi, int vb, int n0, long long eb, int E0)
{
    int64_t *const o = a.u_offs + vb;
    if (threadIdx.x == 0) o[0] = eb;  // (also the last one of the graph before, with the same value)
    cta_copy(a.src.offs[gi], n0, [&](int v, int64_t x) { o[v + 1] = eb + x; });
    int32_t *const nbr = a.u_nbr + eb;
    cta_copy(a.src.nbr[gi], E0, [&](int j, int32_t x) { nbr[j] = x; });
    if (a.u_w) {
        int32_t *const w = a.u_w + eb;
        cta_copy(a.src.w[gi], E0, [&](int j, int32_t x) { w[j] = x; });
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kCtaThreads, 3) k_batch_cta(const __grid_constant__ BatchCtaArgs a)
{
    extern __shared__ int cta_sm[];
    __shared__ CtaShared sh;
    const int wid = threadIdx.x >> 5;
    const int npad = (a.nmax + 31) & ~31;
    if (threadIdx.x == 0) {
        sh.tab = cta_sm;
        sh.Tot = sh.tab + kCtaWarps * kDense;
        sh.occ = (unsigned short *)(sh.Tot + npad);
        sh.lab = sh.occ + kCtaWarps * kWRow;
        sh.cur = sh.lab + npad;
        sh.act = (unsigned char *)(sh.cur + npad);
    }
    // this warp's dense table for long rows (zero, and left zero by every use)
    int *gacc = a.gacc + ((size_t)blockIdx.x * kCtaWarps + wid) * (size_t)a.nmax;
    for (;;) {
        if (threadIdx.x == 0) {
            const int t = atomicAdd(a.queue, 1);
            sh.graph = t < a.G ? a.order[t] : -1;
        }
        __syncthreads();
        const int gi = sh.graph;
        __syncthreads();
        if (gi < 0) break;
        const int vb = (int)a.vstart[gi], n0 = (int)(a.vstart[gi + 1] - vb);
        const long long eb = a.estart[gi];
        const int E0 = (int)(a.estart[gi + 1] - eb);
        if (a.gather) cta_gather(a, gi, vb, n0, eb, E0);
        LevelView g{a.u_offs + vb, nullptr, nullptr, eb, a.u_nbr + eb, a.gather ? 0 : vb,
                    a.u_w ? a.u_w + eb : nullptr};
        long long m2 = 0;
        if (g.w)
            for (int j = threadIdx.x; j < E0; j += kCtaThreads) m2 += g.wt(j);
        else
            m2 = threadIdx.x == 0 ? E0 : 0;
        m2 = cta_sum_ll(m2, sh.red_ll);
        int32_t *orig = a.labels + vb;
        for (int i = threadIdx.x; i < n0; i += kCtaThreads) orig[i] = i;
        __syncthreads();
        if (m2 <= 0 || m2 > 0x7fffffffLL) {  // no edges: singletons; too heavy for int32 sums: flagged
            if (threadIdx.x == 0) {
                if (m2 > 0) atomicOr(a.err, 1);
                a.q_out[gi] = 0.0;
                a.c_out[gi] = n0;
                a.rounds_out[gi] = 0;
                a.iters_out[gi] = 0;
            }
            __syncthreads();
            continue;
        }
        cta_rows0(g, n0, a.K + vb, a.Self + vb);
        __syncthreads();
        int n = n0, rounds = 0, iters_all = 0, C = n0, buf = 0;
        double prev_mod = -1.0, cur_mod = -1.0;
        for (;;) {
            double q = 0.0;
            int it = 0;
            cta_phase1(a, g, n, m2, vb, gacc, sh, &q, &it);
            iters_all += it;
            C = cta_contract(a, g, n, vb, eb, gi, buf, gacc, sh);
            for (int i = threadIdx.x; i < n0; i += kCtaThreads) orig[i] = sh.lab[orig[i]];
            __syncthreads();
            ++rounds;
            prev_mod = cur_mod;
            cur_mod = q;
            if (!(cur_mod - prev_mod >= a.min_mod)) break;  // louvain.cu:202
            if (a.max_levels > 0 && rounds >= a.max_levels) break;
            g = LevelView{nullptr, a.loffs[buf] + vb + gi, a.llen[buf] + vb, 0, a.lnbr[buf] + eb, 0, a.lw[buf] + eb};
            n = C;
            buf ^= 1;
        }
        if (threadIdx.x == 0) {
            a.q_out[gi] = cur_mod;
            a.c_out[gi] = C;
            a.rounds_out[gi] = rounds;
            a.iters_out[gi] = iters_all;
        }
        __syncthreads();
    }
}

}  // namespace

void batch_cta_configure()
{
    cudaFuncSetAttribute(k_batch_cta, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cta_smem(kCtaMaxN));
}

int batch_cta_grid(int G, int nmax)
{
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_cta, kCtaThreads, cta_smem(nmax));
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long cap = (long long)(per_sm > 0 ? per_sm : 1) * (sms > 0 ? sms : 1);
    return (int)(G < cap ? G : cap);
}

size_t batch_cta_gacc_ints(int grid, int nmax) { return (size_t)grid * kCtaWarps * (size_t)nmax; }

void batch_cta_launch(const BatchCtaArgs &a, int grid, cudaStream_t st)
{
    k_batch_cta<<<grid, kCtaThreads, cta_smem(a.nmax), st>>>(a);
    note_launch(1);
}

}  // namespace gala
