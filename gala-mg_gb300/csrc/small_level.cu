// small_level.cu - all sweeps of a small level's phase 1 in one cooperative
// launch (louvain_main_process.cu:571-1034 in the reference, which returns to
// the host between the steps of every iteration).
//
// A sweep of a small level is bound by its launches: some twenty kernels over
// the degree bins, the events that fork and join their streams, and a host
// read of the counters, about 110 us a sweep whatever the level's size.  Here
// the whole grid (two 512-thread CTAs per SM, fewer for tiny levels) runs
// every step of every sweep and meets at a grid barrier between them, four a
// sweep (six with hub rows):
//   decide          all degree bins, heavy rows first
//   apply           the movers' labels, totals and sizes
//   totals          min Tot, sum Tot^2
//   update + prune  In, the next active lists, sum In
// and every CTA takes the convergence decision from the same exact sums.
// What bounds it: at 14k entries the barriers and one dependent chain per step
// (21 us a sweep against 110), at 2.4M entries the label and total gathers
// (82 us against 122).  Whole runs, separate launches / one launch per level:
// 1,024-vertex SBM 1.62 / 1.08 ms, 50k-vertex float LFR 5.2 / 3.5 ms.  The
// bodies per degree bin are those of the one-bin kernels (sweep.cuh), so the
// partition and every Q are the same bit for bit.
#include <algorithm>

#include "common.cuh"
#include "internal.h"
#include "sweep.cuh"

namespace gala {

namespace {

constexpr int kSmallBlock = 512;
constexpr int kSmallWarps = kSmallBlock / 32;

// Counters of one sweep; three slots in turn, so that a slot is cleared two
// barriers after its last reader and two before its next writer.
struct SweepSlot {
    unsigned long long sum_in, sum_tot2, sum_tot2_hi, act_edges;
    long long min_tot;
    int act_vertices, n_movers;
    int act_count[kNumBins];
};

struct SmallCtl {
    unsigned arrive;  // grid barrier: arrivals since the launch
    int dead;         // a barrier wait gave up: every CTA leaves
    SweepSlot slot[3];
};

template <typename WT>
struct SmallArgs {
    DecideArgs<WT, false> d;
    UpdateArgs<WT, false> u;
    HubPlan hp;
    int n;
    int bin_start[kNumBins + 1];
    const int32_t *order;
    int32_t *act[2];
    int32_t *comm, *size;
    WT *Tot, *In;
    uint8_t *act_flag;
    SmallCtl *ctl;
    SmallOut *out;
    double min_mod, prev_q;
    long long min_tot_init;
    int s0;  // first sweep of this launch (1 = the level's first)
};

// Warp-table slots per warp: the tables of all warps together are the CTA
// table (rows up to half of it), 53-74 KB, so that two CTAs fit an SM.
template <typename WT>
struct SmallTable {
    static constexpr int kWarpSlots = WideOf<WT>::exact ? 512 : 256;
    static constexpr int kSlots = kWarpSlots * kSmallWarps;
    static constexpr size_t kBytes = (size_t)kSlots * (sizeof(int) + sizeof(WT)) + kSlots / 2 * sizeof(unsigned short);
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned *p)
{
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid barrier (the launch is cooperative: all CTAs are resident).  False when
// the wait gave up after a few seconds, for every thread of the block; the launch
// then ends with kErrBarrier.
__device__ __forceinline__ bool grid_sync(SmallCtl *c, unsigned &target, int *err)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        target += gridDim.x;
        __threadfence();
        atomicAdd(&c->arrive, 1u);
        int ok = 1;
        for (unsigned spin = 0; (int)(ld_acquire(&c->arrive) - target) < 0; ++spin) {
            if (spin > (1u << 22) || *(volatile int *)&c->dead) {
                atomicExch(&c->dead, 1);
                atomicOr(err, kErrBarrier);
                ok = 0;
                break;
            }
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

__device__ __forceinline__ unsigned long long now_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Q from exact sums, the host's expression (q_from_sums in engine.cu) in the
// same order.
__device__ double slot_q(const SweepSlot &s, long long m2)
{
    const double c = __ddiv_rn(1.0, (double)m2);
    const double t2 = __dadd_rn(__dmul_rn((double)s.sum_tot2_hi, 18446744073709551616.0), (double)s.sum_tot2);
    return __dsub_rn(__dmul_rn((double)(long long)s.sum_in, c), __dmul_rn(__dmul_rn(t2, c), c));
}

__device__ void clear_slot(SweepSlot &s, long long min_tot_init)
{
    s.sum_in = s.sum_tot2 = s.sum_tot2_hi = s.act_edges = 0;
    s.min_tot = min_tot_init;
    s.act_vertices = s.n_movers = 0;
    for (int b = 0; b < kNumBins; ++b) s.act_count[b] = 0;
}

template <typename WT>
__device__ __forceinline__ void apply_moves(const SmallArgs<WT> &a, int nm, int sign)
{
    const int lane = threadIdx.x & 31;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < nm; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + lane;
        const bool valid = i < nm;
        int from = -1, to = -1;
        WT k = 0;
        if (valid) {
            const int v = a.d.mv_v[i];
            from = sign > 0 ? a.d.mv_old[i] : a.d.mv_new[i];
            to = sign > 0 ? a.d.mv_new[i] : a.d.mv_old[i];
            k = a.d.K[v];
            a.comm[v] = to;
        }
        move_totals(valid, from, to, k, a.Tot, a.size);
    }
}

template <typename WT, bool W>
__global__ void __launch_bounds__(kSmallBlock, 2) k_small_level(const __grid_constant__ SmallArgs<WT> a)
{
    using Tab = SmallTable<WT>;
    extern __shared__ long long small_sm[];
    __shared__ int stage_buf[kSmallWarps][3 * kStageM];
    __shared__ int s_go;
    static_assert(kStageN <= 3 * kStageM, "the two stages share their buffer");
    WT *vals = (WT *)small_sm;
    int *keys = (int *)(vals + Tab::kSlots);
    unsigned short *occ = (unsigned short *)(keys + Tab::kSlots);
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int bid = blockIdx.x, nb = gridDim.x;
    // warp tasks go over the CTAs first, from the last CTA down (the CTA rows
    // go to the first CTAs)
    const int wg = wib * nb + (nb - 1 - bid), nw = nb * kSmallWarps;
    unsigned target = 0;
    for (int j = threadIdx.x; j < Tab::kSlots; j += kSmallBlock) {
        keys[j] = -1;
        vals[j] = 0;
    }
    SmallCtl *ctl = a.ctl;
    const HubPlan &hp = a.hp;
    const bool hubs = hp.H > 0;
    int *const err = a.d.err;
    auto clear_hubs = [&]() {
        int *hk = hp.pool;
        WT *hv = (WT *)(hp.pool + hp.half);
        for (long long j = bid * kSmallBlock + threadIdx.x; j < hp.half; j += (long long)nb * kSmallBlock) {
            hk[j] = -1;
            hv[j] = 0;
        }
    };
    if (hubs) clear_hubs();
    if (bid == 0 && threadIdx.x == 0) clear_slot(ctl->slot[a.s0 % 3], a.min_tot_init);
    if (!grid_sync(ctl, target, err)) return;

    double prev_q = a.prev_q;
    long long movers = 0, decisions = 0;  // block 0, thread 0
    unsigned long long entries = 0, dec_ns = 0, upd_ns = 0;
    int done = 0, s = a.s0;
    for (;; ++s) {
        SweepSlot *const cur = &ctl->slot[s % 3];
        const SweepSlot *const prev = &ctl->slot[(s + 2) % 3];
        const bool first = s == 1;
        const int32_t *const lists = first ? a.order : a.act[(s + 1) & 1];
        auto count = [&](int bin) { return first ? a.bin_start[bin + 1] - a.bin_start[bin] : prev->act_count[bin]; };
        const bool boss = bid == 0 && threadIdx.x == 0;
        unsigned long long t0 = 0;
        if (boss) t0 = now_ns();

        // ---- decide
        {
            DecideArgs<WT, false> d = a.d;
            d.n_movers = &cur->n_movers;
            int c = count(6);
            decide_cta<WT, kSmallBlock, W>(d, lists + a.bin_start[6], c, bid, nb, Tab::kSlots, 0, INT_MAX, keys, vals,
                                           occ);
            const int off5 = c % nb;
            decide_cta<WT, kSmallBlock, W>(d, lists + a.bin_start[5], count(5), (bid + nb - off5) % nb, nb,
                                           Tab::kSlots, 0, INT_MAX, keys, vals, occ);
            if (hubs) hub_insert<WT, W>(d, hp, a.act_flag, nb - 1 - bid, nb);
            WarpStage<kStageM, 3> stage{stage_buf[wib], 0};
            int off = 0;
            auto start = [&](int tasks) {  // this warp's first task of the next bin
                const int w0 = wg - off;
                off = (off + tasks) % nw;
                return w0 < 0 ? w0 + nw : w0;
            };
            constexpr int WS = Tab::kWarpSlots;
            c = count(4);
            decide_warp<WT, W, WS>(d, lists + a.bin_start[4], c, start(c), nw, 0, INT_MAX, keys + wib * WS,
                                   vals + wib * WS, occ + wib * (WS / 2));
            c = count(3);
            decide_group<WT, 32, W>(d, lists + a.bin_start[3], c, start(c), nw, stage);
            c = count(2);
            decide_group<WT, 16, W>(d, lists + a.bin_start[2], c, start((c + 1) / 2), nw, stage);
            c = count(1);
            decide_group<WT, 8, W>(d, lists + a.bin_start[1], c, start((c + 3) / 4), nw, stage);
            c = count(0);
            decide_group<WT, 4, W>(d, lists + a.bin_start[0], c, start((c + 7) / 8), nw, stage);
            int *const mlists[3] = {a.d.mv_v, a.d.mv_old, a.d.mv_new};
            stage.flush(mlists, &cur->n_movers);
            if (!grid_sync(ctl, target, err)) return;
            if (hubs) {
                hub_scan<WT, kSmallBlock>(d, hp, a.act_flag, bid, nb);
                if (!grid_sync(ctl, target, err)) return;
                hub_final(d, hp, a.act_flag, wg, nw);
                if (!grid_sync(ctl, target, err)) return;
            }
        }
        if (boss) dec_ns += now_ns() - t0;

        // ---- apply
        apply_moves(a, cur->n_movers, +1);
        if (hubs)
            for (int i = bid * kSmallBlock + threadIdx.x; i < hp.H; i += nb * kSmallBlock) a.In[hp.hubs[i]] = 0;
        if (!grid_sync(ctl, target, err)) return;

        // ---- totals; hub rows' In and their cleared tables on the side
        {
            long long mn = 0x7fffffffffffffffLL;
            typename SqSum<WT>::T s2 = 0;
            for (int c = bid * kSmallBlock + threadIdx.x; c < a.n; c += nb * kSmallBlock) {
                const WT t = a.Tot[c];
                if (t != 0) {
                    mn = min(mn, (long long)t);
                    s2 += SqSum<WT>::sq(t);
                }
            }
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) mn = min(mn, __shfl_xor_sync(GALA_FULL_MASK, mn, o));
            if (lane == 0 && mn != 0x7fffffffffffffffLL) atomicMin(&cur->min_tot, mn);
            SqSum<WT>::add(s2, &cur->sum_tot2, &cur->sum_tot2_hi);
            if (hubs) {
                hub_in_partial<WT, W>(a.u, hp, nb - 1 - bid, nb);
                clear_hubs();
            }
            if (boss) {
                clear_slot(ctl->slot[(s + 1) % 3], a.min_tot_init);
                movers += cur->n_movers;
                if (!first) {
                    decisions += prev->act_vertices;
                    entries += prev->act_edges;
                }
            }
        }
        if (!grid_sync(ctl, target, err)) return;
        if (boss) t0 = now_ns();

        // ---- update and prune
        {
            UpdateArgs<WT, false> u = a.u;
            const long long mt = cur->min_tot;
            UpdateSums sums;
            WarpStage<kStageN, 1> stage{stage_buf[wib], 0};
            int off = 0;
            auto bin = [&](int b, int G) {  // list, count and this warp's first task of a bin
                const int c = a.bin_start[b + 1] - a.bin_start[b], tasks = (c + 32 / G - 1) / (32 / G);
                u.act_list = a.act[s & 1] + a.bin_start[b];
                u.act_counter = &cur->act_count[b];
                const int w0 = wg - off;
                off = (off + tasks) % nw;
                return w0 < 0 ? w0 + nw : w0;
            };
            bin(6, 32);
            off = 0;
            update_cta<WT, W>(u, a.order + a.bin_start[6], a.bin_start[7] - a.bin_start[6], mt, bid, nb, sums);
#define GALA_SMALL_UPD(B, G)                                                                                         \
    do {                                                                                                             \
        const int w0 = bin(B, G);                                                                                    \
        update_group<WT, G, W>(u, a.order + a.bin_start[B], a.bin_start[B + 1] - a.bin_start[B], mt, w0, nw, stage,  \
                               sums);                                                                                \
    } while (0)
            GALA_SMALL_UPD(5, 32);
            GALA_SMALL_UPD(4, 8);
            GALA_SMALL_UPD(3, 16);
            GALA_SMALL_UPD(2, 8);
            GALA_SMALL_UPD(1, 8);
            GALA_SMALL_UPD(0, 4);
#undef GALA_SMALL_UPD
            if (hubs) {
                u.act_list = a.act[s & 1] + a.bin_start[7];
                u.act_counter = &cur->act_count[7];
                hub_in_final(u, hp, mt, bid, nb, sums);
            }
            block_add_u64(sums.in, &cur->sum_in);
            block_add_u64(sums.edges, &cur->act_edges);
            block_add_i32(sums.act, &cur->act_vertices);
        }
        if (!grid_sync(ctl, target, err)) return;

        // ---- convergence (louvain_main_process.cu:1004-1007)
        const int k = s - a.s0;  // sweeps of this launch before this one
        if (threadIdx.x == 0) {
            const double q = slot_q(*cur, a.d.m2);
            int go = 1;
            if (*(volatile int *)err)
                go = 0;
            else if (__dsub_rn(q, prev_q) < a.min_mod)
                go = -1;
            else
                prev_q = q;
            s_go = go;
            if (bid == 0) {
                upd_ns += now_ns() - t0;
                a.out->trace[k] = q;
            }
        }
        __syncthreads();
        if (s_go < 0) apply_moves(a, cur->n_movers, -1);
        if (s_go <= 0) {
            done = 1;
            break;
        }
        if (k + 1 == kSmallSweeps) break;
        // (every thread reads s_go before the next sweep's barriers let thread
        // 0 write it again)
    }
    if (bid == 0 && threadIdx.x == 0) {
        SmallOut *o = a.out;
        o->q = prev_q;
        o->sweeps = s - a.s0 + 1;
        o->done = done;
        o->err = *(volatile int *)err;
        o->movers = movers;
        o->decisions = decisions;
        o->entries = entries;
        o->decide_ns = dec_ns;
        o->update_ns = upd_ns;
    }
}

template <typename WT, bool W>
int small_resident()
{
    static int r = 0;
    if (r == 0) {
        int k = 0;
        cudaFuncSetAttribute(k_small_level<WT, W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)SmallTable<WT>::kBytes);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_small_level<WT, W>, kSmallBlock, SmallTable<WT>::kBytes);
        r = k > 0 ? k : -1;
    }
    return r;
}

template <typename WT, bool W>
cudaError_t launch_small(const LevelGraph &g, const Phase1Buffers &b, const HubPlan &hp, const SmallRun &r,
                         const DecideArgs<WT, false> &d, const UpdateArgs<WT, false> &u, cudaStream_t st)
{
    SmallArgs<WT> a;
    a.d = d;
    a.u = u;
    a.hp = hp;
    a.n = g.n;
    long long tasks = 0;  // warps that a sweep over every vertex keeps busy
    const int per[kNumBins] = {8, 4, 2, 1, 1, 1, 1, 1};
    for (int i = 0; i <= kNumBins; ++i) a.bin_start[i] = r.bin_start[i];
    for (int i = 0; i < kNumBins; ++i) {
        const long long c = r.bin_start[i + 1] - r.bin_start[i];
        tasks += i < 5 ? (c + per[i] - 1) / per[i] : c * kSmallWarps;
    }
    if (hp.H > 0) tasks = std::max<long long>(tasks, hp.ntwork * kSmallWarps);
    a.order = b.order;
    a.act[0] = b.act[0];
    a.act[1] = b.act[1];
    a.comm = b.comm;
    a.size = b.size;
    a.Tot = (WT *)b.Tot;
    a.In = (WT *)b.In;
    a.act_flag = b.act_flag;
    a.ctl = (SmallCtl *)r.ctl;
    a.out = r.out;
    a.min_mod = r.min_mod;
    a.prev_q = r.prev_q;
    a.min_tot_init = r.min_tot_init;
    a.s0 = r.s0;
    const int per_sm = small_resident<WT, W>();
    if (per_sm <= 0) return cudaErrorLaunchOutOfResources;
    long long grid = (tasks + kSmallWarps - 1) / kSmallWarps;
    grid = std::max(1LL, std::min<long long>(grid, (long long)hub_grid_size() * per_sm));
    // the barrier's counter (the sweep slots carry over between launches)
    cudaMemsetAsync(r.ctl, 0, offsetof(SmallCtl, slot), st);
    void *args[] = {&a};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void *)k_small_level<WT, W>, dim3((unsigned)grid),
                                                      dim3(kSmallBlock), args, SmallTable<WT>::kBytes, st);
    note_launch(1);
    return e;
}

template <typename WT>
cudaError_t small_t(const LevelGraph &g, Phase1Buffers &b, const HubPlan &hp, const SmallRun &r, cudaStream_t st)
{
    DecideArgs<WT, false> d;
    d.offs = g.offs;
    d.nbr = g.nbr;
    d.w = (const WT *)g.w;
    d.comm = b.comm;
    d.K = (const WT *)b.K;
    d.Self = (const WT *)b.Self;
    d.Tot = (const WT *)b.Tot;
    d.size = b.size;
    d.mv_v = b.mv_v;
    d.mv_old = b.mv_old;
    d.mv_new = b.mv_new;
    d.n_movers = nullptr;  // per sweep
    d.err = &b.stats->err;
    d.fp64_decisions = &b.stats->fp64_decisions;
    d.constant = 1 / (double)r.m2;
    d.m2 = r.m2;
    d.fp64_only = r.fp64_only;
    d.feat_gain = nullptr;
    d.feat_ndist = nullptr;
    d.gid = nullptr;
    d.m2g = nullptr;
    d.cg = nullptr;
    d.stop = nullptr;
    UpdateArgs<WT, false> u;
    u.offs = g.offs;
    u.nbr = g.nbr;
    u.w = (const WT *)g.w;
    u.comm = b.comm;
    u.K = (const WT *)b.K;
    u.Self = (const WT *)b.Self;
    u.Tot = (const WT *)b.Tot;
    u.In = (WT *)b.In;
    u.act_flag = b.act_flag;
    u.act_list = nullptr;  // per bin
    u.act_counter = nullptr;
    u.st = b.stats;
    u.constant = d.constant;
    u.m2 = r.m2;
    u.next = 0;
    u.gid = nullptr;
    u.m2g = nullptr;
    u.cg = nullptr;
    u.stop = nullptr;
    u.min_tot_g = nullptr;
    if constexpr (WideOf<WT>::exact)
        if (!g.w) return launch_small<WT, false>(g, b, hp, r, d, u, st);
    return launch_small<WT, true>(g, b, hp, r, d, u, st);
}

}  // namespace

size_t small_ctl_bytes() { return sizeof(SmallCtl); }

BinLimits small_limits(const BinLimits &lim, bool wide)
{
    BinLimits l = lim;
    const int row4 = (wide ? SmallTable<long long>::kWarpSlots : SmallTable<int>::kWarpSlots) / 2;
    const int row6 = (wide ? SmallTable<long long>::kSlots : SmallTable<int>::kSlots) / 2;
    l.m4 = std::min(l.m4, row4);
    l.m5 = std::min(l.m5, row6);
    l.m6 = std::min(l.m6, row6);
    return l;
}

cudaError_t small_level_run(const LevelGraph &g, Phase1Buffers &b, const HubPlan &hp, const SmallRun &r,
                            cudaStream_t st)
{
    return g.wide ? small_t<long long>(g, b, hp, r, st) : small_t<int>(g, b, hp, r, st);
}

}  // namespace gala
