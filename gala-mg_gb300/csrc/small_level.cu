// small_level.cu - all sweeps of a small level's phase 1 in one cooperative
// launch (louvain_main_process.cu:571-1034 in the reference, which returns to
// the host between the steps of every iteration), the level init included
// (louvain_main_process.cu:268-375, init_communities kernel_functions.cu:34-73).
//
// A sweep of a small level is bound by its launches: some twenty kernels over
// the degree bins, the events that fork and join their streams, and a host
// read of the counters, about 110 us a sweep whatever the level's size.  Here
// the whole grid (two 512-thread CTAs per SM, fewer for tiny levels) runs
// every step of every sweep and meets at a grid barrier between them, three a
// sweep (six with hub rows):
//   decide          all degree bins, heavy rows first; the movers' totals
//   apply + totals  the movers' labels and sizes; min Tot, sum Tot^2
//   update + prune  In, the next active lists, sum In
// The decide step moves the totals in a second array, so that its own reads
// see those before the sweep, and the next step copies them over while it reads
// them all anyway: one step and one barrier less than with the totals in one
// array (phase 1 at 20k vertices and 0.4M entries 0.88 -> 0.76 ms, at 100k and
// 2.4M 1.48 -> 1.39).  Every CTA takes the convergence decision from the same
// exact sums.
// What bounds it: at 14k entries the barriers (about 3k SM cycles each) and one
// chain of dependent L2 reads per step (18 us a sweep against 110), at 2.4M
// entries the label and total gathers (64 us against 100).  Whole runs,
// separate launches / one launch per level: 1,024-vertex SBM 1.42 / 0.64 ms,
// 50k-vertex float LFR 4.52 / 2.43 ms.  The
// bodies per degree bin are those of the one-bin kernels (sweep.cuh), so the
// partition and every Q are the same bit for bit.
#include <algorithm>

#include "common.cuh"
#include "coop.cuh"
#include "internal.h"
#include "scan.cuh"
#include "sweep.cuh"

namespace gala {

namespace {

// Counters of one sweep; three slots in turn, so that a slot is cleared two
// barriers after its last reader and two before its next writer.
struct SweepSlot {
    unsigned long long sum_in, sum_tot2, sum_tot2_hi, act_edges;
    long long min_tot;
    int act_vertices, n_movers;
    int err;  // error bits of the sweep's decisions: read behind its last barrier, while
              // a faster block may already set bits of the next sweep (in the next slot)
    int act_count[kNumBins];
};

constexpr int kSmallOneCta = 64;
// Hub rows of an unweighted level from which the level is left to the one-bin
// kernels: those take rows of 4097-8192 entries in shared memory, and the level's
// first sweep without tables.  Whole runs, bipartite graphs of k rows of d entries,
// one-bin launches (behind the launch that declines) / one launch (ms): k 200, d 4300
// 1.15 / 1.13, d 9500 1.44 / 1.26; k 300, d 4300 1.45 / 1.49, d 6000 1.22 / 1.28, d 9500
// 1.55 / 1.47; k 400, d 6000 1.26 / 1.46; k 800, d 4300 1.41 / 1.83.  With weights one launch is faster throughout (k 800, d 4300
// 3.28 / 2.91), with 64-bit weights too (k 800, d 4700 3.46 / 2.86).
constexpr int kSmallHubs = 320;
struct SmallCtl {
    // reset before every launch
    GridBarrier bar;
    SmallOut out;
    // reset before a level's first launch
    unsigned long long sum_k, sum_k2, sum_k2_hi, sum_self;
    // kept between a level's launches
    SweepSlot slot[3];
    int bin_start[kNumBins + 1];
    long long half, nwork, ntwork;          // hub plan
    int part[kSmallMaxGrid][kNumBinSlots];  // vertices per block and bin
};

template <typename WT>
struct SmallArgs {
    DecideArgs<WT, false> d;
    UpdateArgs<WT, false> u;
    HubPlan hp;  // arrays; H, half, nwork and ntwork come from the level
    long long pool_ints, work_cap, twork_cap;
    int n;
    BinLimits lim;
    bool ks_ready;        // K and Self are given (else summed over the rows)
    const int32_t *init;  // starting community of every vertex (null: its own)
    int32_t *order;
    int32_t *act[2];
    int32_t *comm, *size;
    WT *K, *Self, *Tot, *In;
    uint8_t *act_flag;
    SmallCtl *ctl;
    unsigned polls;  // of a grid barrier
    double min_mod, prev_q;
    long long m2;  // total weight (0: this level's sum of K)
    int s0;        // first sweep of this launch (1 = the level's first)
};

// Degree bins of a small level: the longest rows that a warp's and the CTA's table
// take, whatever limits the caller gave bins 4 and 5 (they are tuned for the
// one-bin launches; rows of 100 entries in 8M, bin 4 ending at 64: 4.4 ms, so
// 1.9).  A lower limit of bin 6 still makes hubs of the rows above it.
BinLimits small_limits(const BinLimits &lim, bool wide)
{
    const int row4 = (wide ? SmallTable<long long>::kWarpSlots : SmallTable<int>::kWarpSlots) / 2;
    const int row6 = (wide ? SmallTable<long long>::kSlots : SmallTable<int>::kSlots) / 2;
    BinLimits l;
    l.m6 = std::min(lim.m6, row6);
    l.m5 = std::min(l.m5, l.m6);
    l.m4 = std::min(row4, l.m5);
    return l;
}

// (read twice a launch: the steps are timed in SM cycles, since a read of the
// global timer takes a good part of a step of a tiny level)
__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Q from exact sums, the host's expression (q_from_sums in engine.cu) in the
// same order.
__device__ double slot_q(const SweepSlot &s, double c)
{
    const double t2 = __dadd_rn(__dmul_rn((double)s.sum_tot2_hi, 18446744073709551616.0), (double)s.sum_tot2);
    return __dsub_rn(__dmul_rn((double)(long long)s.sum_in, c), __dmul_rn(__dmul_rn(t2, c), c));
}

__device__ void clear_slot(SweepSlot &s, long long min_tot_init)
{
    s.sum_in = s.sum_tot2 = s.sum_tot2_hi = s.act_edges = 0;
    s.min_tot = min_tot_init;
    s.act_vertices = s.n_movers = s.err = 0;
    for (int b = 0; b < kNumBins; ++b) s.act_count[b] = 0;
}

// The movers' labels and sizes; their totals (moved by the decide step into
// a.d.tot_next) only on the way back.
template <typename WT, bool BACK>
__device__ __forceinline__ void apply_moves(const SmallArgs<WT> &a, int nm)
{
    const int lane = threadIdx.x & 31;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < nm; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + lane;
        const bool valid = i < nm;
        int from = -1, to = -1;
        WT k = 0;
        if (valid) {
            const int v = a.d.mv_v[i];
            from = BACK ? a.d.mv_new[i] : a.d.mv_old[i];
            to = BACK ? a.d.mv_old[i] : a.d.mv_new[i];
            if (BACK) k = a.d.K[v];
            a.comm[v] = to;
        }
        move_totals<WT, BACK, true>(valid, from, to, k, a.Tot, a.size);
    }
}

// K and Self of the rows of a list (lane groups of G; a row of a vertex that
// lists itself in several lanes' entries sums those, as k_init_rows_group).
template <typename WT, int G, bool W>
__device__ __forceinline__ void init_rows(const SmallArgs<WT> &a, const int32_t *list, int count, int wg, int nw,
                                          unsigned long long &sk, typename SqSum<WT>::T &sk2, unsigned long long &ss)
{
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), gw = lane / G;
    constexpr int GPW = 32 / G;
    for (int base = wg * GPW; base < count; base += nw * GPW) {
        const int idx = base + gw;
        const bool has = idx < count;
        const int v = has ? list[idx] : 0;
        const long long s = has ? a.d.offs[v] : 0, e = has ? a.d.offs[v + 1] : 0;
        WT k = 0, sf = 0;
        for (long long j = s + sub; j < e; j += G) {
            const WT wt = W ? a.d.w[j] : 1;
            k += wt;
            if (a.d.nbr[j] == v) sf = wt;
        }
#pragma unroll
        for (int o = G / 2; o >= 1; o >>= 1) {
            k += __shfl_xor_sync(GALA_FULL_MASK, k, o);
            sf += __shfl_xor_sync(GALA_FULL_MASK, sf, o);
        }
        if (has && sub == 0) {
            a.K[v] = k;
            a.Tot[v] = k;
            a.Self[v] = sf;
            a.In[v] = sf;
            sk += (unsigned long long)k;
            sk2 += SqSum<WT>::sq(k);
            ss += (unsigned long long)sf;
        }
    }
}

// The same for long rows, a block per row: 256 of its threads, as
// k_init_rows_cta.
template <typename WT, bool W>
__device__ __forceinline__ void init_rows_cta(const SmallArgs<WT> &a, const int32_t *list, int count,
                                              unsigned long long &sk, typename SqSum<WT>::T &sk2,
                                              unsigned long long &ss)
{
    __shared__ WT rk[8], rs[8];
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int v = list[i];
        const long long s = a.d.offs[v], e = a.d.offs[v + 1];
        if (threadIdx.x < 256) {
            WT k = 0, sf = 0;
            for (long long j = s + threadIdx.x; j < e; j += 256) {
                const WT wt = W ? a.d.w[j] : 1;
                k += wt;
                if (a.d.nbr[j] == v) sf = wt;
            }
            k = warp_sum(k);
            sf = warp_sum(sf);
            if ((threadIdx.x & 31) == 0) {
                rk[threadIdx.x >> 5] = k;
                rs[threadIdx.x >> 5] = sf;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            WT k = 0, sf = 0;
            for (int q = 0; q < 8; ++q) {
                k += rk[q];
                sf += rs[q];
            }
            a.K[v] = k;
            a.Tot[v] = k;
            a.Self[v] = sf;
            a.In[v] = sf;
            sk += (unsigned long long)k;
            sk2 += SqSum<WT>::sq(k);
            ss += (unsigned long long)sf;
        }
        __syncthreads();
    }
}

// Level init, one block's contiguous run of vertices.  place = false: labels,
// sizes, totals and the block's vertices per degree bin (ctl->part); place =
// true, after a barrier: the vertices into the bin-ordered list (offsets from
// every block's counts), bin starts into s_bin.
template <typename WT>
__device__ __forceinline__ void level_vertices(const SmallArgs<WT> &a, bool place, int *s_bin)
{
    __shared__ int s_cnt[kNumBinSlots], s_pos[kNumBinSlots];
    SmallCtl *ctl = a.ctl;
    const int nb = gridDim.x, bid = blockIdx.x, lane = threadIdx.x & 31;
    const int per = (a.n + nb - 1) / nb;
    const int v0 = (int)min((long long)per * bid, (long long)a.n), v1 = (int)min((long long)v0 + per, (long long)a.n);
    if (threadIdx.x < kNumBinSlots) s_cnt[threadIdx.x] = s_pos[threadIdx.x] = 0;
    __syncthreads();
    if (place) {
        // s_cnt: vertices per bin; s_pos: those of the blocks before this one
        for (int i = threadIdx.x; i < nb * kNumBinSlots; i += kSmallBlock) {
            const int c = ctl->part[i / kNumBinSlots][i % kNumBinSlots];
            if (c) {
                atomicAdd(&s_cnt[i % kNumBinSlots], c);
                if (i / kNumBinSlots < bid) atomicAdd(&s_pos[i % kNumBinSlots], c);
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            int run = 0;
            for (int k = 0; k < kNumBinSlots; ++k) {
                if (k <= kNumBins) s_bin[k] = run;
                s_pos[k] += run;
                run += s_cnt[k];
            }
            if (bid == 0)
                for (int k = 0; k <= kNumBins; ++k) ctl->bin_start[k] = s_bin[k];
        }
        __syncthreads();
    }
    unsigned long long sk = 0, ss = 0;
    typename SqSum<WT>::T sk2 = 0;
    for (int t = v0; t < v1; t += kSmallBlock) {  // block-uniform
        const int v = t + threadIdx.x;
        int b = -1;
        if (v < v1) {
            b = bin_of_degree(a.d.offs[v + 1] - a.d.offs[v], a.lim);
            if (!place) {
                a.comm[v] = a.init ? a.init[v] : v;
                a.size[v] = a.init ? 0 : 1;
                a.act_flag[v] = 1;
                WT k = 0, sf = 0;
                if (a.ks_ready) {
                    k = a.K[v];
                    sf = a.Self[v];
                    sk += (unsigned long long)k;
                    sk2 += SqSum<WT>::sq(k);
                    ss += (unsigned long long)sf;
                } else {  // the rows' sums follow; vertices without entries stay 0
                    a.K[v] = 0;
                    a.Self[v] = 0;
                }
                a.Tot[v] = a.init ? (WT)0 : k;
                a.In[v] = a.init ? (WT)0 : sf;
            }
        }
#pragma unroll
        for (int k = 0; k < kNumBinSlots; ++k) {
            const unsigned m = __ballot_sync(GALA_FULL_MASK, b == k);
            if (m == 0) continue;
            int p = 0;
            if (lane == __ffs((int)m) - 1) p = atomicAdd(place ? &s_pos[k] : &s_cnt[k], __popc(m));
            p = __shfl_sync(GALA_FULL_MASK, p, __ffs((int)m) - 1);
            if (place && b == k) a.order[p + __popc(m & lanemask_lt())] = v;
        }
        if (place && a.init) {  // Tot and size of the starting communities
            const bool has = v < v1;
            if (has) {
                atomic_add_w(&a.Tot[a.init[v]], a.K[v]);
                atomicAdd(&a.size[a.init[v]], 1);
            }
        }
    }
    if (!place) {
        __syncthreads();
        if (threadIdx.x < kNumBinSlots) ctl->part[bid][threadIdx.x] = s_cnt[threadIdx.x];
        if (a.ks_ready) {
            block_add_u64(sk, &ctl->sum_k);
            SqSum<WT>::add(sk2, &ctl->sum_k2, &ctl->sum_k2_hi);
            block_add_u64(ss, &ctl->sum_self);
        }
    }
}

// Hub plan by one block: table sizes, chunk counts and their prefixes.
template <typename WT>
__device__ __forceinline__ void plan_hubs(const SmallArgs<WT> &a, const HubPlan &p)
{
    __shared__ long long wt[32], tot;
    long long c0 = 0, c1 = 0, c2 = 0;
    for (int t = 0; t < p.H; t += kSmallBlock) {
        const int i = t + threadIdx.x;
        long long T = 0, ch = 0, tc = 0;
        if (i < p.H) {
            const int v = p.hubs[i];
            hub_table(p, a.d.offs[v + 1] - a.d.offs[v], T, ch, tc);
            p.T[i] = T;
        }
        long long x = block_exclusive_scan<long long>(T, wt, &tot);
        if (i < p.H) p.toff[i] = c0 + x;
        c0 += tot;
        __syncthreads();
        x = block_exclusive_scan<long long>(ch, wt, &tot);
        if (i < p.H) p.coff[i] = c1 + x;
        c1 += tot;
        __syncthreads();
        x = block_exclusive_scan<long long>(tc, wt, &tot);
        if (i < p.H) p.tcoff[i] = c2 + x;
        c2 += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        p.toff[p.H] = c0;
        p.coff[p.H] = c1;
        p.tcoff[p.H] = c2;
        a.ctl->half = c0;
        a.ctl->nwork = c1;
        a.ctl->ntwork = c2;
    }
}

// log2 of the rows per warp task of the update, bins 0 to 5.
__device__ constexpr int kUpdShift[6] = {3, 3, 3, 2, 2, 0};

// Warp wg's first task of every bin, one bin per lane (tasks: the bin's, 0 in
// the other lanes), when the bins from the highest down share the nw warps round
// robin.
__device__ __forceinline__ int first_tasks(int tasks, int wg, int nw)
{
    int sum = tasks;  // of this lane's bin and those above
#pragma unroll
    for (int o = 1; o < 8; o *= 2) sum += __shfl_down_sync(GALA_FULL_MASK, sum, o);
    const int w0 = wg - (sum - tasks) % nw;
    return w0 < 0 ? w0 + nw : w0;
}

// The block's share of In, active entries and active vertices to the sweep's
// counters, in one reduction.
__device__ __forceinline__ void block_sums(const UpdateSums &sums, SweepSlot &slot)
{
    __shared__ unsigned long long s_sums[3][kSmallWarps];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    unsigned long long x[3] = {sums.in, sums.edges, (unsigned long long)sums.act};
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; ++k) x[k] += __shfl_xor_sync(GALA_FULL_MASK, x[k], o);
    if (lane < 3) s_sums[lane][wib] = lane == 0 ? x[0] : (lane == 1 ? x[1] : x[2]);
    __syncthreads();
    if (wib == 0) {  // (the sums' next writer comes after a grid barrier)
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            x[k] = s_sums[k][lane & (kSmallWarps - 1)];
#pragma unroll
            for (int o = kSmallWarps / 2; o >= 1; o >>= 1) x[k] += __shfl_xor_sync(GALA_FULL_MASK, x[k], o);
        }
        if (lane == 0) {
            if (x[0]) atomicAdd(&slot.sum_in, x[0]);
            if (x[1]) atomicAdd(&slot.act_edges, x[1]);
            if (x[2]) atomicAdd(&slot.act_vertices, (int)x[2]);
        }
    }
}

template <typename WT, bool W>
__global__ void __launch_bounds__(kSmallBlock, 2) k_small_level(const __grid_constant__ SmallArgs<WT> a)
{
    using Tab = SmallTable<WT>;
    extern __shared__ long long small_sm[];
    __shared__ int stage_buf[kSmallWarps][3 * kStageM];
    __shared__ int s_go, s_bin[kNumBins + 1];
    __shared__ long long s_min[kSmallWarps];
    __shared__ struct {
        long long movers, decisions, cyc0, dec_cyc, upd_cyc;
        unsigned long long entries, ns0;
    } s_stat;  // block 0's
    static_assert(kStageN <= 3 * kStageM, "the two stages share their buffer");
    WT *vals = (WT *)small_sm;
    int *keys = (int *)(vals + Tab::kSlots);
    unsigned short *occ = (unsigned short *)(keys + Tab::kSlots);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int bid = blockIdx.x, nb = gridDim.x;
    const bool boss = bid == 0 && threadIdx.x == 0;
    // warp tasks go over the CTAs first, from the last CTA down (the CTA rows
    // go to the first CTAs)
    const int wg = wib * nb + (nb - 1 - bid), nw = nb * kSmallWarps;
    unsigned target = 0;
    for (int j = threadIdx.x; j < Tab::kSlots; j += kSmallBlock) {
        keys[j] = -1;
        vals[j] = 0;
    }
    SmallCtl *ctl = a.ctl;
    SmallOut *const out = &ctl->out;
    HubPlan hp = a.hp;
    int *const err = &out->err;  // of the barriers
    auto clear_hubs = [&]() {
        int *hk = hp.pool;
        WT *hv = (WT *)(hp.pool + hp.half);
        for (long long j = bid * kSmallBlock + threadIdx.x; j < hp.half; j += (long long)nb * kSmallBlock) {
            hk[j] = -1;
            hv[j] = 0;
        }
    };
    const bool fresh = a.s0 == 1;
    const long long min_tot_cap = WideOf<WT>::exact ? 0x7fffffffLL : 0x7fffffffffffffffLL;
    if (fresh) {
        // ---- level init
        if (boss) a.u.st->err = 0;  // of the level's later kernels
        level_vertices(a, false, s_bin);
        if (!grid_sync(&ctl->bar, target, err, a.polls)) return;
        level_vertices(a, true, s_bin);
    } else {
        if (threadIdx.x <= kNumBins) s_bin[threadIdx.x] = ctl->bin_start[threadIdx.x];
        __syncthreads();
    }
    hp.H = s_bin[8] - s_bin[7];
    hp.hubs = a.order + s_bin[7];
    const bool hubs = hp.H > 0;
    if (!W && fresh && hp.H > kSmallHubs) {  // the same for every block
        if (boss) out->status = 3;
        return;
    }
    if (fresh) {
        if (!a.ks_ready || hubs || a.init) {
            if (!grid_sync(&ctl->bar, target, err, a.polls)) return;
            if (!a.ks_ready) {
                unsigned long long sk = 0, ss = 0;
                typename SqSum<WT>::T sk2 = 0;
                init_rows_cta<WT, W>(a, a.order + s_bin[6], s_bin[8] - s_bin[6], sk, sk2, ss);
                init_rows<WT, 32, W>(a, a.order + s_bin[3], s_bin[6] - s_bin[3], wg, nw, sk, sk2, ss);
                init_rows<WT, 16, W>(a, a.order + s_bin[2], s_bin[3] - s_bin[2], wg, nw, sk, sk2, ss);
                init_rows<WT, 8, W>(a, a.order + s_bin[1], s_bin[2] - s_bin[1], wg, nw, sk, sk2, ss);
                init_rows<WT, 4, W>(a, a.order + s_bin[0], s_bin[1] - s_bin[0], wg, nw, sk, sk2, ss);
                block_add_u64(sk, &ctl->sum_k);
                SqSum<WT>::add(sk2, &ctl->sum_k2, &ctl->sum_k2_hi);
                block_add_u64(ss, &ctl->sum_self);
            }
            if (hubs && bid == nb - 1) plan_hubs(a, hp);
        }
        if (!grid_sync(&ctl->bar, target, err, a.polls)) return;
    }
    const long long m2 = a.m2 ? a.m2 : (long long)ctl->sum_k;
    const double constant = __ddiv_rn(1.0, (double)m2);
    hp.half = ctl->half;
    hp.nwork = ctl->nwork;
    hp.ntwork = ctl->ntwork;
    const long long min_tot_init = min(m2, min_tot_cap);
    double prev_q = a.prev_q;
    if (fresh) {
        const bool fits = !hubs || ((1 + (long long)(sizeof(WT) / sizeof(int))) * hp.half <= a.pool_ints &&
                                    hp.nwork <= a.work_cap && hp.ntwork <= a.twork_cap);
        const bool sum_ok = m2 > 0 && m2 <= min_tot_cap && (long long)ctl->sum_k == m2;
        if (boss) {
            out->sum_k = ctl->sum_k;
            out->nv = s_bin[8];
            for (int k = 0; k <= kNumBins; ++k) out->bin_start[k] = s_bin[k];
            out->hub_slots = hubs ? hp.half : 0;
            out->done = 1;
            out->status = !sum_ok ? 1 : (!fits ? 2 : 0);
        }
        if (!sum_ok || !fits) return;  // the same for every block
        if (!a.init && threadIdx.x == 0) {
            SweepSlot q0;
            q0.sum_in = ctl->sum_self;
            q0.sum_tot2 = ctl->sum_k2;
            q0.sum_tot2_hi = ctl->sum_k2_hi;
            prev_q = slot_q(q0, constant);
            if (bid == 0) out->q0 = prev_q;
        }
        if (boss) {
            clear_slot(ctl->slot[0], min_tot_init);
            clear_slot(ctl->slot[1], min_tot_init);
        }
        if (hubs) {
            hub_work(hp, wg, nw);
            clear_hubs();
        }
        for (int c = bid * kSmallBlock + threadIdx.x; c < a.n; c += nb * kSmallBlock) a.d.tot_next[c] = a.Tot[c];
        if (!grid_sync(&ctl->bar, target, err, a.polls)) return;
    }

    // counts of the run, kept by a thread that has nothing else on its path
    const bool clerk = bid == 0 && threadIdx.x == kSmallBlock - 1;
    if (clerk) s_stat.movers = s_stat.decisions = s_stat.entries = 0;
    if (boss) {
        s_stat.ns0 = now_ns();
        s_stat.cyc0 = clock64();
        s_stat.dec_cyc = s_stat.upd_cyc = 0;
    }
    int upd_w0;  // this warp's first update task per bin, one bin per lane
    {
        int tasks = 0;
        if (lane < 6) {
            const int sh = kUpdShift[lane];
            tasks = (s_bin[lane + 1] - s_bin[lane] + (1 << sh) - 1) >> sh;
        }
        upd_w0 = first_tasks(tasks, wg, nw);
    }
    int done = 0, s = fresh && a.init ? 0 : a.s0;  // sweep 0: In and Q of a starting partition
    for (;; ++s) {
        SweepSlot *const cur = &ctl->slot[s % 3];
        const SweepSlot *const prev = &ctl->slot[(s + 2) % 3];
        const bool first = s == 1;
        const int32_t *const lists = first ? a.order : a.act[(s + 1) & 1];
        // rows of the bins, one bin per lane: one read after the barrier instead
        // of one in front of every bin
        int counts = 0;
        if (lane < kNumBins) counts = first ? s_bin[lane + 1] - s_bin[lane] : prev->act_count[lane];
        auto count = [&](int bin) { return __shfl_sync(GALA_FULL_MASK, counts, bin); };
        if (boss) s_stat.dec_cyc -= s > 0 ? clock64() : 0;

        // ---- decide
        if (s > 0) {
            DecideArgs<WT, false> d = a.d;
            d.n_movers = &cur->n_movers;
            d.err = &cur->err;
            d.m2 = m2;
            d.constant = constant;
            int c = count(6);
            decide_cta<WT, kSmallBlock, W>(d, lists + s_bin[6], c, bid, nb, Tab::kSlots, 0, INT_MAX, keys, vals,
                                           occ);
            const int b5 = bid - (c < nb ? c : c % nb);
            decide_cta<WT, kSmallBlock, W>(d, lists + s_bin[5], count(5), b5 < 0 ? b5 + nb : b5, nb, Tab::kSlots, 0,
                                           INT_MAX, keys, vals, occ);
            if (hubs) hub_insert<WT, W>(d, hp, a.act_flag, nb - 1 - bid, nb);
            WarpStage<kStageM, 3> stage{stage_buf[wib], 0};
            const int w0s = first_tasks(lane < 5 ? (counts + (8 >> min(lane, 3)) - 1) >> (3 - min(lane, 3)) : 0, wg, nw);
            auto start = [&](int bin) { return __shfl_sync(GALA_FULL_MASK, w0s, bin); };
            constexpr int WS = Tab::kWarpSlots;
            c = count(4);
            decide_warp<WT, W, WS>(d, lists + s_bin[4], c, start(4), nw, 0, INT_MAX, keys + wib * WS,
                                   vals + wib * WS, occ + wib * (WS / 2));
            c = count(3);
            decide_group<WT, 32, W>(d, lists + s_bin[3], c, start(3), nw, stage);
            c = count(2);
            decide_group<WT, 16, W>(d, lists + s_bin[2], c, start(2), nw, stage);
            c = count(1);
            decide_group<WT, 8, W>(d, lists + s_bin[1], c, start(1), nw, stage);
            c = count(0);
            decide_group<WT, 4, W>(d, lists + s_bin[0], c, start(0), nw, stage);
            flush_movers(d, stage);
            if (!grid_sync(&ctl->bar, target, err, a.polls)) return;
            if (hubs) {
                hub_scan<WT, kSmallBlock>(d, hp, a.act_flag, bid, nb);
                if (!grid_sync(&ctl->bar, target, err, a.polls)) return;
                hub_final(d, hp, a.act_flag, wg, nw);
                if (!grid_sync(&ctl->bar, target, err, a.polls)) return;
            }
        }
        if (boss && s > 0) s_stat.dec_cyc += clock64();

        // ---- labels and sizes; with hub rows a step of their own, since these
        // rows' In is summed over the new labels in the next one
        const int c0 = bid * kSmallBlock + threadIdx.x;  // (the first total is read ahead)
        WT t = c0 < a.n ? a.d.tot_next[c0] : (WT)0;
        if (s > 0) {
            apply_moves<WT, false>(a, cur->n_movers);
            if (hubs) {
                for (int i = bid * kSmallBlock + threadIdx.x; i < hp.H; i += nb * kSmallBlock) a.In[hp.hubs[i]] = 0;
                if (!grid_sync(&ctl->bar, target, err, a.polls)) return;
            }
        }

        // ---- totals; hub rows' In and their cleared tables on the side
        {
            long long mn = 0x7fffffffffffffffLL;
            typename SqSum<WT>::T s2 = 0;
            int nm = 0, dv = 0;
            unsigned long long de = 0;
            if (clerk) {
                nm = cur->n_movers;
                dv = prev->act_vertices;
                de = prev->act_edges;
            }
            for (int c = c0; c < a.n; c += nb * kSmallBlock) {
                if (c != c0) t = a.d.tot_next[c];
                a.Tot[c] = t;
                if (t != 0) {
                    mn = min(mn, (long long)t);
                    s2 += SqSum<WT>::sq(t);
                }
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) mn = min(mn, __shfl_xor_sync(GALA_FULL_MASK, mn, o));
            if (lane == 0) s_min[wib] = mn;
            SqSum<WT>::add(s2, &cur->sum_tot2, &cur->sum_tot2_hi);  // (block barriers inside)
            if (wib == 0) {
                mn = s_min[lane & (kSmallWarps - 1)];
#pragma unroll
                for (int o = kSmallWarps / 2; o >= 1; o >>= 1) mn = min(mn, __shfl_xor_sync(GALA_FULL_MASK, mn, o));
                if (lane == 0 && mn != 0x7fffffffffffffffLL) atomicMin(&cur->min_tot, mn);
            }
            if (hubs) {
                hub_in_partial<WT, W>(a.u, hp, nb - 1 - bid, nb);
                clear_hubs();
            }
            if (clerk) {
                clear_slot(ctl->slot[(s + 1) % 3], min_tot_init);
                s_stat.movers += nm;
                if (s > 1) {
                    s_stat.decisions += dv;
                    s_stat.entries += de;
                }
            }
        }
        if (!grid_sync(&ctl->bar, target, err, a.polls)) return;
        if (boss) s_stat.upd_cyc -= s > 0 ? clock64() : 0;

        // ---- update and prune
        {
            UpdateArgs<WT, false> u = a.u;
            u.m2 = m2;
            u.constant = constant;
            const long long mt = cur->min_tot;
            UpdateSums sums;
            WarpStage<kStageN, 1> stage{stage_buf[wib], 0};
            auto bin = [&](int b) {  // active list of a bin; this warp's first task
                u.act_list = a.act[s & 1] + s_bin[b];
                u.act_counter = &cur->act_count[b];
                return __shfl_sync(GALA_FULL_MASK, upd_w0, b);
            };
            bin(6);
            update_cta<WT, W>(u, a.order + s_bin[6], s_bin[7] - s_bin[6], mt, bid, nb, sums);
#define GALA_SMALL_UPD(B, G, U)                                                                                      \
    do {                                                                                                             \
        static_assert(32 / G == 1 << kUpdShift[B], "tasks of the bin");                                              \
        const int w0 = bin(B);                                                                                       \
        update_group<WT, G, U, W>(u, a.order + s_bin[B], s_bin[B + 1] - s_bin[B], mt, w0, nw, stage,  \
                               sums);                                                                                \
    } while (0)
            GALA_SMALL_UPD(5, 32, 4);
            GALA_SMALL_UPD(4, 8, 4);
            GALA_SMALL_UPD(3, 8, 4);
            GALA_SMALL_UPD(2, 4, 4);
            GALA_SMALL_UPD(1, 4, 2);
            GALA_SMALL_UPD(0, 4, 1);
#undef GALA_SMALL_UPD
            if (hubs) {
                u.act_list = a.act[s & 1] + s_bin[7];
                u.act_counter = &cur->act_count[7];
                hub_in_final(u, hp, mt, bid, nb, sums);
            }
            block_sums(sums, *cur);
        }
        if (!grid_sync(&ctl->bar, target, err, a.polls)) return;

        // ---- convergence (louvain_main_process.cu:1004-1007)
        const int k = s - a.s0;  // sweeps of this launch before this one
        if (s == 0) {
            if (threadIdx.x == 0) prev_q = slot_q(*cur, constant);
            if (boss) out->q0 = prev_q;
            continue;
        }
        if (threadIdx.x == 0) {
            const int e = *(volatile int *)&cur->err;
            const double q = slot_q(*cur, constant);
            int go = 1;
            if (e)
                go = 0;
            else if (__dsub_rn(q, prev_q) < a.min_mod)
                go = -1;
            else
                prev_q = q;
            s_go = go;
            if (bid == 0) {
                s_stat.upd_cyc += clock64();
                out->trace[k] = q;
            }
        }
        __syncthreads();
        if (s_go < 0) apply_moves<WT, true>(a, cur->n_movers);
        if (s_go <= 0) {
            done = 1;
            break;
        }
        if (k + 1 == kSmallSweeps) break;
        // (every thread reads s_go before the next sweep's barriers let thread
        // 0 write it again)
    }
    if (clerk) {
        out->movers = s_stat.movers;
        out->decisions = s_stat.decisions;
        out->entries = s_stat.entries;
    }
    if (boss) {
        out->q = prev_q;
        out->sweeps = s - a.s0 + 1;
        out->done = done;
        const int e = *(volatile int *)&ctl->slot[s % 3].err;
        if (e) atomicOr(err, e);  // (another block may add that a barrier gave up)
        const double ns = (double)(now_ns() - s_stat.ns0) / (double)max(clock64() - s_stat.cyc0, 1LL);  // per cycle
        out->decide_ns = (unsigned long long)((double)s_stat.dec_cyc * ns);
        out->update_ns = (unsigned long long)((double)s_stat.upd_cyc * ns);
    }
}

template <typename WT, bool W>
cudaError_t launch_small(const LevelGraph &g, SmallArgs<WT> &a, int max_grid, cudaStream_t st)
{
    if (max_grid <= 0) return cudaErrorLaunchOutOfResources;
    // warps a sweep keeps busy: about 1.5 lanes per entry, at most 8 vertices
    // a warp
    const long long tasks = g.E * 3 / 64 + g.n / 32;
    // (a level of few tasks stays on one CTA, which needs no grid barriers and
    // keeps the level in its L1)
    long long grid = tasks <= kSmallOneCta ? 1 : (tasks + kSmallWarps - 1) / kSmallWarps;
    grid = std::max(1LL, std::min<long long>(grid, max_grid));
    cudaMemsetAsync(a.ctl, 0, a.s0 == 1 ? offsetof(SmallCtl, slot) : offsetof(SmallCtl, sum_k), st);
    void *args[] = {&a};
    const cudaError_t e =
        coop_launch((const void *)k_small_level<WT, W>, grid, kSmallBlock, args, SmallTable<WT>::kBytes, st);
    note_launch(1);
    return e;
}

template <typename WT>
cudaError_t small_t(const LevelGraph &g, Phase1Buffers &b, const HubPlan &hp, const SmallRun &r, cudaStream_t st)
{
    SmallArgs<WT> a{};
    DecideArgs<WT, false> &d = a.d;
    d.offs = g.offs;
    d.nbr = g.nbr;
    d.w = (const WT *)g.w;
    d.comm = b.comm;
    d.K = (const WT *)b.K;
    d.Self = (const WT *)b.Self;
    d.Tot = (const WT *)b.Tot;
    d.size = b.size;
    d.tot_next = (WT *)r.tot_next;
    d.mv_v = b.mv_v;
    d.mv_old = b.mv_old;
    d.mv_new = b.mv_new;
    d.fp64_decisions = &b.stats->fp64_decisions;
    d.fp64_only = r.fp64_only;
    UpdateArgs<WT, false> &u = a.u;
    u.offs = g.offs;
    u.nbr = g.nbr;
    u.w = (const WT *)g.w;
    u.comm = b.comm;
    u.K = (const WT *)b.K;
    u.Self = (const WT *)b.Self;
    u.Tot = (const WT *)b.Tot;
    u.In = (WT *)b.In;
    u.act_flag = b.act_flag;
    u.st = b.stats;
    a.hp = hp;
    a.pool_ints = r.pool_ints;
    a.work_cap = r.work_cap;
    a.twork_cap = r.twork_cap;
    a.n = g.n;
    a.lim = small_limits(b.lim, g.wide);
    a.ks_ready = g.ks_ready;
    a.init = r.init;
    a.order = b.order;
    a.act[0] = b.act[0];
    a.act[1] = b.act[1];
    a.comm = b.comm;
    a.size = b.size;
    a.K = (WT *)b.K;
    a.Self = (WT *)b.Self;
    a.Tot = (WT *)b.Tot;
    a.In = (WT *)b.In;
    a.act_flag = b.act_flag;
    a.ctl = (SmallCtl *)r.ctl;
    a.polls = r.polls;
    a.min_mod = r.min_mod;
    a.prev_q = r.prev_q;
    a.m2 = r.m2;
    a.s0 = r.s0;
    if constexpr (WideOf<WT>::exact)
        if (!g.w) return launch_small<WT, false>(g, a, r.max_grid, st);
    return launch_small<WT, true>(g, a, r.max_grid, st);
}

}  // namespace

void small_level_configure(CoopGrids &c)
{
    constexpr size_t i = SmallTable<int>::kBytes, l = SmallTable<long long>::kBytes;
    c.level[0] = coop_grid(k_small_level<int, false>, kSmallBlock, i, kSmallMaxGrid);
    c.level[1] = coop_grid(k_small_level<int, true>, kSmallBlock, i, kSmallMaxGrid);
    c.level[2] = coop_grid(k_small_level<long long, true>, kSmallBlock, l, kSmallMaxGrid);
}

size_t small_ctl_bytes() { return sizeof(SmallCtl); }

const SmallOut *small_ctl_out(const void *ctl) { return &((const SmallCtl *)ctl)->out; }

cudaError_t small_level_run(const LevelGraph &g, Phase1Buffers &b, const HubPlan &hp, const SmallRun &r,
                            cudaStream_t st)
{
    return g.wide ? small_t<long long>(g, b, hp, r, st) : small_t<int>(g, b, hp, r, st);
}

}  // namespace gala
