// small_contract.cu - contraction of a small level in one cooperative launch
// (build_compressed_graph.cu:5-173 in the reference).
//
// The general contraction (contract.cu) takes some fifty launches, most of
// them prefix sums, lists and size classes; on a level of few entries each
// finishes in two microseconds and the whole in about 200.  Here one grid runs
// the same steps with a grid barrier between them, eleven in all (three more
// when a community has more than half a CTA table of entries):
//   labels     member counts, dense renumbering in ascending label order
//   entries    entries per community, their prefix, every row of the level
//              copied to its community's range with the neighbours' labels
//   rows       per community the weights summed per neighbour community: a
//              warp match (<= 32 entries), a warp's table, the CTA's table, or
//              a global table filled by many CTAs
//   new level  prefix of the row lengths, rows to their places
// Rows come out in any order, as inside every Louvain run.
#include <algorithm>

#include "common.cuh"
#include "coop.cuh"
#include "internal.h"
#include "scan.cuh"
#include "sweep.cuh"

namespace gala {

namespace {

constexpr int kContractOneCta = 1024;
struct ContractCtl {
    // reset before every launch
    GridBarrier bar;
    int n_cta, n_big;      // communities listed for a CTA / for global tables
    long long big_slots;   // slots of the global tables
    long long part[2][kSmallMaxGrid];  // block sums of the running prefix
};

template <typename WT>
struct ContractArgs {
    int n, n_orig;
    long long E;
    const int64_t *__restrict__ offs;
    const int32_t *__restrict__ nbr;
    const WT *__restrict__ w;
    const int32_t *__restrict__ comm;
    const int32_t *__restrict__ order;
    int bin_start[kNumBins + 1];
    int32_t *cnt, *newid, *lab, *kc, *list;
    long long *ec, *ebase, *taken, *tmp_off;
    long long *long_claim;  // claims of the long rows (degree bins 6 and 7)
    int32_t *skey, *tmp_nbr;
    WT *sw, *tmp_w;
    int32_t *pool;
    long long pool_ints;
    long long *big_T, *big_toff;
    const WT *__restrict__ tot;
    WT *k_out, *self_out;
    int32_t *orig;
    int64_t *new_offs;
    int32_t *new_nbr;
    WT *new_w;
    bool labels_only;
    ContractCtl *ctl;
    unsigned polls;  // of a grid barrier
    DevStats *st;
};

// This block's contiguous part of [0, n).
struct Part {
    int lo, hi;
    __device__ __forceinline__ explicit Part(int n)
    {
        const long long per = ((long long)n + gridDim.x - 1) / gridDim.x;
        lo = (int)min(per * blockIdx.x, (long long)n);
        hi = (int)min(lo + per, (long long)n);
    }
};

// Prefix over the blocks' parts in two steps with a barrier between: every
// block puts the sum of f over its part; then out(i, prefix) is called for
// every i of the part in order.  Returns the total over all blocks.
template <typename F>
__device__ __forceinline__ void part_sum(long long *part, const Part &p, F f)
{
    __shared__ long long ws[32];
    long long s = 0;
    for (int i = p.lo + threadIdx.x; i < p.hi; i += kSmallBlock) s += f(i);
    s = scan_block_sum(s, ws);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}
template <typename F, typename Out>
__device__ __forceinline__ long long part_prefix(const long long *part, const Part &p, F f, Out out)
{
    __shared__ long long ws[32], tot;
    long long before = 0, all = 0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kSmallBlock) {
        const long long x = part[b];
        all += x;
        if (b < (int)blockIdx.x) before += x;
    }
    all = scan_block_sum(all, ws);
    long long carry = scan_block_sum(before, ws);
    constexpr int U = 4;  // consecutive items per thread
    for (int t = p.lo; t < p.hi; t += U * kSmallBlock) {  // block-uniform
        const int i0 = t + threadIdx.x * U;
        long long x[U], s = 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            x[u] = i0 + u < p.hi ? f(i0 + u) : 0;
            s += x[u];
        }
        long long run = carry + block_exclusive_scan<long long>(s, ws, &tot);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (i0 + u < p.hi) out(i0 + u, run);
            run += x[u];
        }
        carry += tot;
        __syncthreads();
    }
    return all;
}

// Adds v to a[c] for every lane with v != 0, equal c of a warp together.  All
// 32 lanes call; v < 2^26.
template <typename T>
__device__ __forceinline__ void add_by_label(T *a, int c, unsigned v)
{
    const unsigned m = __match_any_sync(GALA_FULL_MASK, v ? c : -1);
    const unsigned t = (unsigned)match_sum(m, v != 0, (int)v);
    if (v && (int)(threadIdx.x & 31) == __ffs((int)m) - 1) {
        if constexpr (sizeof(T) == 8)
            atomicAdd((unsigned long long *)&a[c], (unsigned long long)t);
        else
            atomicAdd((int *)&a[c], (int)t);
    }
}

// Rows of a degree bin to their places in the stream: a group of G lanes per
// row, one claim per row.
template <typename WT, int G, bool W>
__device__ __forceinline__ void fill_rows(const ContractArgs<WT> &a, int lo, int hi, int wg, int nw)
{
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), gw = lane / G;
    constexpr int GPW = 32 / G, U = 4;
    for (int base = lo + wg * GPW; base < hi; base += nw * GPW) {
        const int idx = base + gw;
        long long s = 0, d = 0, to = 0;
        if (idx < hi) {
            const int v = a.order[idx];
            s = a.offs[v];
            d = a.offs[v + 1] - s;
            if (sub == 0) {
                const int c = a.lab[v];
                to = a.ebase[c] + (long long)atomicAdd((unsigned long long *)&a.taken[c], (unsigned long long)d);
            }
        }
        to = __shfl_sync(GALA_FULL_MASK, to, lane & ~(G - 1));
        for (long long j = sub; j < d; j += U * G) {
            int u[U];
            WT w[U];
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const bool ok = j + q * G < d;
                u[q] = ok ? a.nbr[s + j + q * G] : -1;
                w[q] = W && ok ? a.w[s + j + q * G] : (WT)1;
            }
#pragma unroll
            for (int q = 0; q < U; ++q)
                if (u[q] >= 0) u[q] = a.lab[u[q]];
#pragma unroll
            for (int q = 0; q < U; ++q)
                if (u[q] >= 0) {
                    a.skey[to + j + q * G] = u[q];
                    if (W) a.sw[to + j + q * G] = w[q];
                }
        }
    }
}

// Long rows: chunks of kHubChunk entries spread over the blocks.
template <typename WT, bool W>
__device__ __forceinline__ void fill_long_rows(const ContractArgs<WT> &a, int lo, int hi)
{
    const int nb = gridDim.x;
    int off = 0;  // chunks of the rows before, modulo the grid
    for (int i = lo; i < hi; ++i) {
        const int v = a.order[i];
        const long long s = a.offs[v], d = a.offs[v + 1] - s;
        const int chunks = (int)((d + kHubChunk - 1) / kHubChunk);
        const int c = a.lab[v];
        const long long to = a.ebase[c] + a.long_claim[i - lo];
        for (int k = (blockIdx.x + nb - off) % nb; k < chunks; k += nb) {
            const long long e = min((long long)(k + 1) * kHubChunk, d);
            for (long long j = (long long)k * kHubChunk + threadIdx.x; j < e; j += kSmallBlock) {
                a.skey[to + j] = a.lab[a.nbr[s + j]];
                if (W) a.sw[to + j] = a.w[s + j];
            }
        }
        off = (off + chunks) % nb;
    }
}

// Aggregates stream entries [e0, e0 + len) of one community in a shared-memory
// table by one warp (NT = 32) or the block (NT = kSmallBlock); claimed slots
// are listed in occ.  Returns their number.
template <typename WT, int NT, int TL>
__device__ __forceinline__ int aggregate(const ContractArgs<WT> &a, const WT *sw, long long e0, int len, int *keys,
                                         WT *vals, unsigned short *occ, int *s_n)
{
    const int t = NT == 32 ? threadIdx.x & 31 : threadIdx.x, lane = threadIdx.x & 31;
    int n = 0;
    for (int j0 = 0; j0 < len; j0 += NT) {
        const int j = j0 + t;
        bool created = false;
        int slot = -1;
        if (j < len) {
            slot = hash_add_slot(keys, vals, 1 << TL, TL, a.skey[e0 + j], sw ? sw[e0 + j] : (WT)1, created);
            if (slot < 0) atomicOr(&a.st->err, kErrHashOverflow);
        }
        const unsigned m = __ballot_sync(GALA_FULL_MASK, created);
        if (NT == 32) {
            if (created) occ[n + __popc(m & lanemask_lt())] = (unsigned short)slot;
            n += __popc(m);
        } else if (m) {
            int base = 0;
            if (lane == 0) base = atomicAdd(s_n, __popc(m));
            base = __shfl_sync(GALA_FULL_MASK, base, 0);
            if (created) occ[base + __popc(m & lanemask_lt())] = (unsigned short)slot;
        }
    }
    if (NT == 32) {
        __syncwarp();
        return n;
    }
    __syncthreads();
    return *s_n;
}

// Rows of 1 ... 32 entries by one warp, equal keys by a match; returns the row
// length.
template <typename WT>
__device__ __forceinline__ int row_match(const ContractArgs<WT> &a, const WT *sw, long long e0, int len, long long to)
{
    const int lane = threadIdx.x & 31;
    const bool ok = lane < len;
    const int key = ok ? a.skey[e0 + lane] : -1;
    const WT w = ok ? (sw ? sw[e0 + lane] : (WT)1) : (WT)0;
    const unsigned m = __match_any_sync(GALA_FULL_MASK, key);
    const WT sum = match_sum(m, ok, w);
    const bool head = ok && __ffs((int)m) - 1 == lane;
    const unsigned hm = __ballot_sync(GALA_FULL_MASK, head);
    if (head) {
        const long long o = to + __popc(hm & lanemask_lt());
        a.tmp_nbr[o] = key;
        a.tmp_w[o] = sum;
    }
    return __popc(hm);
}

template <typename WT, bool W>
__global__ void __launch_bounds__(kSmallBlock, 2) k_contract_small(const __grid_constant__ ContractArgs<WT> a)
{
    using Tab = SmallTable<WT>;
    constexpr int WS = Tab::kWarpSlots, WL = WS == 512 ? 9 : 8, TL = WL + 4;
    static_assert((1 << TL) == Tab::kSlots, "sixteen warp tables");
    extern __shared__ long long small_sm[];
    WT *vals = (WT *)small_sm;
    int *keys = (int *)(vals + Tab::kSlots);
    unsigned short *occ = (unsigned short *)(keys + Tab::kSlots);
    __shared__ int s_n;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int bid = blockIdx.x, nb = gridDim.x;
    const int wg = wib * nb + (nb - 1 - bid), nw = nb * kSmallWarps;  // warp tasks: see small_level.cu
    const int t0 = bid * kSmallBlock + threadIdx.x, nt = nb * kSmallBlock;
    ContractCtl *ctl = a.ctl;
    int *const err = &a.st->err;
    unsigned target = 0;
#define GALA_SYNC()                                          \
    do {                                                     \
        if (!grid_sync(&ctl->bar, target, err, a.polls)) return;      \
    } while (0)
    // (*err is 0: the level's phase 1 cleared it, and an error ends a run)
    for (int i = t0; i < a.n; i += nt) {
        a.cnt[i] = 0;
        if (!a.labels_only) a.ec[i] = a.taken[i] = 0;
    }
    for (int j = threadIdx.x; j < Tab::kSlots; j += kSmallBlock) {
        keys[j] = -1;
        vals[j] = 0;
    }
    GALA_SYNC();

    // ---- labels
    for (int v0 = t0 - lane; v0 < a.n; v0 += nt) {
        const int v = v0 + lane;
        add_by_label(a.cnt, v < a.n ? a.comm[v] : -1, v < a.n ? 1u : 0u);
    }
    GALA_SYNC();
    const Part pv(a.n);
    part_sum(ctl->part[0], pv, [&](int c) { return a.cnt[c] > 0 ? 1LL : 0LL; });
    GALA_SYNC();
    const int C = (int)part_prefix(
        ctl->part[0], pv, [&](int c) { return a.cnt[c] > 0 ? 1LL : 0LL; },
        [&](int c, long long id) {
            if (a.cnt[c] <= 0) return;
            a.newid[c] = (int)id;
            if (a.k_out) a.k_out[id] = a.tot[c];
            if (a.self_out) a.self_out[id] = 0;
        });
    if (bid == 0 && threadIdx.x == 0) a.st->ccount = C;
    GALA_SYNC();
    for (int v = t0; v < a.n; v += nt) a.lab[v] = a.newid[a.comm[v]];
    if (a.labels_only) {
        if (a.orig)
            for (int i = t0; i < a.n_orig; i += nt) a.orig[i] = a.newid[a.comm[a.orig[i]]];
        return;
    }

    // ---- entries per community, over the vertices that have some
    for (int i0 = t0 - lane; i0 < a.bin_start[kNumBins]; i0 += nt) {
        const int i = i0 + lane;
        int c = -1;
        unsigned d = 0;
        if (i < a.bin_start[kNumBins]) {
            const int v = a.order[i];
            c = a.newid[a.comm[v]];
            d = (unsigned)(a.offs[v + 1] - a.offs[v]);
        }
        add_by_label(a.ec, c, d);
    }
    GALA_SYNC();
    const Part pc(C);
    auto cap = [&](int c) { return min(a.ec[c], (long long)C); };
    part_sum(ctl->part[0], pc, [&](int c) { return a.ec[c]; });
    part_sum(ctl->part[1], pc, cap);
    GALA_SYNC();
    part_prefix(ctl->part[0], pc, [&](int c) { return a.ec[c]; }, [&](int c, long long x) { a.ebase[c] = x; });
    part_prefix(ctl->part[1], pc, cap, [&](int c, long long x) { a.tmp_off[c] = x; });
    int32_t *const cta_list = a.list, *const big_list = a.list + a.n;
    for (int c0 = pc.lo; c0 < pc.hi; c0 += kSmallBlock) {  // block-uniform
        const int c = c0 + threadIdx.x;
        const long long e = c < pc.hi ? a.ec[c] : 0;
        warp_append(e > WS / 2 && e <= Tab::kSlots / 2, c, cta_list, &ctl->n_cta);
        warp_append(e > Tab::kSlots / 2, c, big_list, &ctl->n_big);
    }
    // the long rows' places, claimed once for all blocks that copy them
    if (bid == 0) {
        for (int i = a.bin_start[6] + threadIdx.x; i < a.bin_start[kNumBins]; i += kSmallBlock) {
            const int v = a.order[i];
            a.long_claim[i - a.bin_start[6]] = (long long)atomicAdd((unsigned long long *)&a.taken[a.lab[v]],
                                                                    (unsigned long long)(a.offs[v + 1] - a.offs[v]));
        }
    }
    GALA_SYNC();

    // ---- the stream
    fill_long_rows<WT, W>(a, a.bin_start[6], a.bin_start[kNumBins]);
    fill_rows<WT, 32, W>(a, a.bin_start[4], a.bin_start[6], wg, nw);
    fill_rows<WT, 8, W>(a, a.bin_start[2], a.bin_start[4], wg, nw);
    fill_rows<WT, 4, W>(a, a.bin_start[0], a.bin_start[2], wg, nw);
    GALA_SYNC();

    // ---- rows; few communities: fewer than 32 per warp, so that all warps have some
    const int per = min(32, (C + nw - 1) / nw);
    const WT *const sw = W ? a.sw : nullptr;
    const int n_cta = ctl->n_cta, n_big = ctl->n_big;
    if (n_big > 0 && bid == nb - 1) {  // table sizes of the longest rows
        __shared__ long long ws[32], tot;
        long long carry = 0;
        for (int t = 0; t < n_big; t += kSmallBlock) {
            const int i = t + threadIdx.x;
            long long T = 0;
            if (i < n_big) {
                const long long k = cap(big_list[i]);
                T = max(32LL, next_pow2_ll(k + k / 2));  // load at most 2/3
                a.big_T[i] = T;
                a.kc[big_list[i]] = 0;
            }
            const long long x = block_exclusive_scan<long long>(T, ws, &tot);
            if (i < n_big) a.big_toff[i] = carry + x;
            carry += tot;
            __syncthreads();
        }
        if (threadIdx.x == 0) ctl->big_slots = carry;
    }
    for (int i = bid; i < n_cta; i += nb) {
        const int c = cta_list[i];
        if (threadIdx.x == 0) s_n = 0;
        __syncthreads();
        const int k = aggregate<WT, kSmallBlock, TL>(a, sw, a.ebase[c], (int)a.ec[c], keys, vals, occ, &s_n);
        const long long o = a.tmp_off[c];
        for (int q = threadIdx.x; q < k; q += kSmallBlock) {
            const int h = occ[q];
            a.tmp_nbr[o + q] = keys[h];
            a.tmp_w[o + q] = vals[h];
            keys[h] = -1;
            vals[h] = 0;
        }
        if (threadIdx.x == 0) a.kc[c] = k;
        __syncthreads();
    }
    {
        int *const wk = keys + wib * WS;
        WT *const wv = vals + wib * WS;
        unsigned short *const wo = occ + wib * (WS / 2);
        for (int c0 = wg * per; c0 < C; c0 += nw * per) {
            const int cl = c0 + lane;
            const bool mine = lane < per && cl < C;
            const long long el = mine ? a.ec[cl] : 0;
            if (mine && el == 0) a.kc[cl] = 0;
            unsigned todo = __ballot_sync(GALA_FULL_MASK, el > 0 && el <= WS / 2);
            while (todo) {  // warp-uniform
                const int src = __ffs((int)todo) - 1;
                todo &= todo - 1;
                const int c = c0 + src, len = (int)__shfl_sync(GALA_FULL_MASK, el, src);
                const long long e0 = a.ebase[c], o = a.tmp_off[c];
                int k;
                if (len <= 32) {
                    k = row_match(a, sw, e0, len, o);
                } else {
                    k = aggregate<WT, 32, WL>(a, sw, e0, len, wk, wv, wo, nullptr);
                    for (int q = lane; q < k; q += 32) {
                        const int h = wo[q];
                        a.tmp_nbr[o + q] = wk[h];
                        a.tmp_w[o + q] = wv[h];
                        wk[h] = -1;
                        wv[h] = 0;
                    }
                    __syncwarp();
                }
                if (lane == 0) a.kc[c] = k;
            }
        }
    }
    GALA_SYNC();
    if (n_big > 0) {
        const long long slots = ctl->big_slots;
        if (slots * (1 + (long long)(sizeof(WT) / sizeof(int))) > a.pool_ints) {  // the same for every block
            if (bid == 0 && threadIdx.x == 0) atomicOr(err, kErrCapacity);
            return;
        }
        int *const bk = a.pool;
        WT *const bv = (WT *)(a.pool + slots);  // slots: a sum of powers of two >= 32
        for (long long j = t0; j < slots; j += nt) {
            bk[j] = -1;
            bv[j] = 0;
        }
        GALA_SYNC();
        // chunks of half a CTA table: summed in shared memory, then added to
        // the row's table
        constexpr int CH = Tab::kSlots / 2;
        int off = 0;
        for (int i = 0; i < n_big; ++i) {
            const int c = big_list[i];
            const long long E = a.ec[c], T = a.big_T[i];
            const int chunks = (int)((E + CH - 1) / CH), lg = 63 - __clzll(T);
            int *const tk = bk + a.big_toff[i];
            WT *const tv = bv + a.big_toff[i];
            for (int q0 = (bid + nb - off) % nb; q0 < chunks; q0 += nb) {
                if (threadIdx.x == 0) s_n = 0;
                __syncthreads();
                const long long e0 = (long long)q0 * CH;
                const int k = aggregate<WT, kSmallBlock, TL>(a, sw, a.ebase[c] + e0, (int)min((long long)CH, E - e0),
                                                             keys, vals, occ, &s_n);
                for (int q = threadIdx.x; q < k; q += kSmallBlock) {
                    const int h = occ[q];
                    if (!hash_add(tk, tv, (int)T, lg, keys[h], vals[h])) atomicOr(err, kErrHashOverflow);
                    keys[h] = -1;
                    vals[h] = 0;
                }
                __syncthreads();
            }
            off = (off + chunks) % nb;
        }
        GALA_SYNC();
        off = 0;
        for (int i = 0; i < n_big; ++i) {
            const int c = big_list[i];
            const long long T = a.big_T[i];
            const int chunks = (int)((T + kHubChunk - 1) / kHubChunk);
            const int *const tk = bk + a.big_toff[i];
            const WT *const tv = bv + a.big_toff[i];
            for (int q0 = (bid + nb - off) % nb; q0 < chunks; q0 += nb) {
                const long long h1 = min((long long)(q0 + 1) * kHubChunk, T);
                for (long long h0 = (long long)q0 * kHubChunk; h0 < h1; h0 += kSmallBlock) {  // block-uniform
                    const long long h = h0 + threadIdx.x;
                    const int key = h < h1 ? tk[h] : -1;
                    const unsigned m = __ballot_sync(GALA_FULL_MASK, key >= 0);
                    if (!m) continue;
                    int base = 0;
                    if (lane == 0) base = atomicAdd(&a.kc[c], __popc(m));
                    base = __shfl_sync(GALA_FULL_MASK, base, 0);
                    if (key >= 0) {
                        const long long o = a.tmp_off[c] + base + __popc(m & lanemask_lt());
                        a.tmp_nbr[o] = key;
                        a.tmp_w[o] = tv[h];
                    }
                }
            }
            off = (off + chunks) % nb;
        }
        GALA_SYNC();
    }

    // ---- the new level
    part_sum(ctl->part[0], pc, [&](int c) { return (long long)a.kc[c]; });
    GALA_SYNC();
    const long long En = part_prefix(
        ctl->part[0], pc, [&](int c) { return (long long)a.kc[c]; }, [&](int c, long long x) { a.new_offs[c] = x; });
    if (bid == 0 && threadIdx.x == 0) {
        a.new_offs[C] = En;
        a.st->new_entries = En;
    }
    if (a.orig)
        for (int i = t0; i < a.n_orig; i += nt) a.orig[i] = a.lab[a.orig[i]];
    GALA_SYNC();
    for (int c0 = wg * per; c0 < C; c0 += nw * per) {
        const int cl = c0 + lane;
        const int kl = lane < per && cl < C ? a.kc[cl] : 0;
        unsigned todo = __ballot_sync(GALA_FULL_MASK, kl > 0 && kl <= kHubChunk);
        while (todo) {
            const int src = __ffs((int)todo) - 1;
            todo &= todo - 1;
            const int c = c0 + src, k = __shfl_sync(GALA_FULL_MASK, kl, src);
            const long long s = a.tmp_off[c], o = a.new_offs[c];
            for (int q = lane; q < k; q += 32) {
                const int key = a.tmp_nbr[s + q];
                const WT wt = a.tmp_w[s + q];
                a.new_nbr[o + q] = key;
                a.new_w[o + q] = wt;
                if (a.self_out && key == c) a.self_out[c] = wt;
            }
        }
    }
    for (int i = 0; i < n_big; ++i) {  // rows too long for a warp
        const int c = big_list[i], k = a.kc[c];
        if (k <= kHubChunk) continue;
        const long long s = a.tmp_off[c], o = a.new_offs[c];
        for (int q = t0; q < k; q += nt) {
            const int key = a.tmp_nbr[s + q];
            const WT wt = a.tmp_w[s + q];
            a.new_nbr[o + q] = key;
            a.new_w[o + q] = wt;
            if (a.self_out && key == c) a.self_out[c] = wt;
        }
    }
#undef GALA_SYNC
}

template <typename WT, bool W>
cudaError_t launch_contract(ContractArgs<WT> &a, int max_grid, cudaStream_t st)
{
    if (max_grid <= 0) return cudaErrorLaunchOutOfResources;
    // a thread per vertex and per four entries
    const long long items = std::max<long long>(a.n, std::max<long long>(a.E / 4, a.n_orig / 4));
    // (few items stay on one CTA, as in small_level.cu)
    const long long want = items <= kContractOneCta ? 1 : (items + kSmallBlock - 1) / kSmallBlock;
    const long long grid = std::min<long long>(want, max_grid);
    cudaMemsetAsync(a.ctl, 0, offsetof(ContractCtl, part), st);
    void *args[] = {&a};
    const cudaError_t e =
        coop_launch((const void *)k_contract_small<WT, W>, grid, kSmallBlock, args, SmallTable<WT>::kBytes, st);
    note_launch(1);
    return e;
}

template <typename WT>
cudaError_t contract_small_t(const LevelGraph &g, const int32_t *comm, ContractBuffers &b, const int32_t *order,
                             const int *bin_start, int64_t *new_offs, int32_t *new_nbr, void *new_w, int32_t *orig_map,
                             int32_t n_orig, const NextLevelInit &nli, bool labels_only, cudaStream_t st)
{
    ContractArgs<WT> a{};
    a.n = g.n;
    a.n_orig = n_orig;
    a.E = g.E;
    a.offs = g.offs;
    a.nbr = g.nbr;
    a.w = (const WT *)g.w;
    a.comm = comm;
    a.order = order;
    for (int i = 0; i <= kNumBins; ++i) a.bin_start[i] = bin_start[i];
    a.cnt = b.cnt;
    a.newid = b.newid;
    a.lab = b.lab;
    a.kc = b.kc;
    a.list = b.cls_list;
    a.ec = b.ec;
    a.ebase = b.ebase;
    a.taken = b.taken;
    a.long_claim = b.nz_shift;
    a.tmp_off = b.tmp_off;
    a.skey = b.stream_key;
    a.tmp_nbr = b.tmp_nbr;
    a.sw = (WT *)b.stream_w;
    a.tmp_w = (WT *)b.tmp_w;
    a.pool = b.big_pool;
    a.pool_ints = b.big_pool_ints;
    a.big_T = b.big_T;
    a.big_toff = b.big_toff;
    a.tot = (const WT *)nli.tot;
    a.k_out = (WT *)nli.k;
    a.self_out = (WT *)nli.self;
    a.orig = orig_map;
    a.new_offs = new_offs;
    a.new_nbr = new_nbr;
    a.new_w = (WT *)new_w;
    a.labels_only = labels_only;
    a.ctl = (ContractCtl *)b.small_ctl;
    a.polls = b.polls;
    a.st = b.stats;
    const int max_grid = b.coop->contract[weight_kind(g)];
    if (g.w) return launch_contract<WT, true>(a, max_grid, st);
    if constexpr (WideOf<WT>::exact) return launch_contract<WT, false>(a, max_grid, st);
    return cudaErrorInvalidValue;  // fixed-point levels are weighted
}

}  // namespace

void contract_small_configure(CoopGrids &c)
{
    constexpr size_t i = SmallTable<int>::kBytes, l = SmallTable<long long>::kBytes;
    c.contract[0] = coop_grid(k_contract_small<int, false>, kSmallBlock, i, kSmallMaxGrid);
    c.contract[1] = coop_grid(k_contract_small<int, true>, kSmallBlock, i, kSmallMaxGrid);
    c.contract[2] = coop_grid(k_contract_small<long long, true>, kSmallBlock, l, kSmallMaxGrid);
}

size_t contract_ctl_bytes() { return sizeof(ContractCtl); }

cudaError_t contract_small(const LevelGraph &g, const int32_t *comm, ContractBuffers &b, const int32_t *order,
                           const int *bin_start, int64_t *new_offs, int32_t *new_nbr, void *new_w, int32_t *orig_map,
                           int32_t n_orig, const NextLevelInit &nli, bool labels_only, cudaStream_t st)
{
    return g.wide ? contract_small_t<long long>(g, comm, b, order, bin_start, new_offs, new_nbr, new_w, orig_map, n_orig,
                                                nli, labels_only, st)
                  : contract_small_t<int>(g, comm, b, order, bin_start, new_offs, new_nbr, new_w, orig_map, n_orig, nli,
                                          labels_only, st);
}

}  // namespace gala
