// phase1.cu - phase-1 kernels of the GB300 Louvain engine (sm_103a).
//
// One phase-1 iteration (louvain_main_process.cu:571-1034 in the reference):
//   decide  : every active vertex aggregates the weights to its neighbour
//             communities, picks the best gain (ties -> lowest id) and, when it
//             moves, appends (v, old, new) to a mover list
//   apply   : movers update comm, Tot and size with integer atomics
//   reduce  : min over non-empty Tot and sum of Tot^2
//   update  : In[v] (weight to the own community) for every vertex, the
//             pruning bound, the next active lists and sum of In
// All reads of a sweep see the previous iteration's labels (synchronous
// semantics, as in the reference), so results do not depend on the order in
// which vertices are processed.
#include "common.cuh"
#include "internal.h"
#include "scan.cuh"
#include "sweep.cuh"

namespace gala {

static int g_num_sms = 0;
static int num_sms()
{
    if (g_num_sms == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_num_sms, cudaDevAttrMultiProcessorCount, dev);
        if (g_num_sms <= 0) g_num_sms = 148;
    }
    return g_num_sms;
}
int hub_grid_size() { return num_sms(); }

constexpr int kCountBlock = 1024;


// ------------------------------------------------------------------------
// Level init: labels = own id, size 1 (louvain_main_process.cu:323-353),
// then a stable counting sort of the vertices into degree bins (the reference
// uses 8 count_if + a radix sort_by_key, :298-375).
// ------------------------------------------------------------------------
template <typename WT>
__global__ void k_init_vertices(int n, int32_t *comm, WT *K, WT *Self, WT *Tot, int32_t *size, WT *In)
{
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        comm[v] = v;
        size[v] = 1;
        K[v] = 0;
        Self[v] = 0;
        Tot[v] = 0;
        In[v] = 0;
    }
}

// Level init of a contracted level whose K and Self the contraction wrote:
// labels and sizes as above, Tot = K, In = Self, and the sums sum(K),
// sum(K^2), sum(Self) of the singleton partition without a row scan.
template <typename WT>
__global__ void __launch_bounds__(256) k_init_vertices_ks(int n, int32_t *comm, const WT *__restrict__ K,
                                                          const WT *__restrict__ Self, WT *Tot, int32_t *size,
                                                          WT *In, DevStats *st)
{
    unsigned long long sk = 0, ss = 0;
    typename SqSum<WT>::T sk2 = 0;
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const WT k = K[v], sf = Self[v];
        comm[v] = v;
        size[v] = 1;
        Tot[v] = k;
        In[v] = sf;
        sk += (unsigned long long)k;
        sk2 += SqSum<WT>::sq(k);
        ss += (unsigned long long)sf;
    }
    block_add_u64(sk, &st->sum_k);
    SqSum<WT>::add(sk2, &st->sum_tot2, &st->sum_tot2_hi);
    block_add_u64(ss, &st->sum_in);
}

__global__ void __launch_bounds__(kCountBlock) k_bin_count(int n, const int64_t *__restrict__ offs,
                                                           int32_t *blockcnt, int nblk, DevStats *st, BinLimits lim)
{
    __shared__ int cnt[kNumBinSlots];
    if (threadIdx.x < kNumBinSlots) cnt[threadIdx.x] = 0;
    __syncthreads();
    int v = blockIdx.x * kCountBlock + threadIdx.x;
    int deg = 0;
    if (v < n) {
        deg = (int)(offs[v + 1] - offs[v]);
        atomicAdd(&cnt[bin_of_degree(deg, lim)], 1);
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) deg = max(deg, __shfl_xor_sync(GALA_FULL_MASK, deg, o));
    if ((threadIdx.x & 31) == 0 && deg > 0) atomicMax(&st->max_deg, deg);
    __syncthreads();
    if (threadIdx.x < kNumBinSlots) blockcnt[threadIdx.x * nblk + blockIdx.x] = cnt[threadIdx.x];
}

__global__ void __launch_bounds__(kCountBlock) k_bin_scatter(int n, const int64_t *__restrict__ offs,
                                                             const int32_t *__restrict__ blockoff, int nblk,
                                                             int32_t *order, DevStats *st, BinLimits lim)
{
    __shared__ int wcnt[kCountBlock / 32][kNumBinSlots];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int v = blockIdx.x * kCountBlock + threadIdx.x;
    int b = -1;
    if (v < n) b = bin_of_degree(offs[v + 1] - offs[v], lim);
    unsigned mine = 0;
#pragma unroll
    for (int bb = 0; bb < kNumBinSlots; ++bb) {
        unsigned bal = __ballot_sync(GALA_FULL_MASK, b == bb);
        if (b == bb) mine = bal;
        if (lane == 0) wcnt[wid][bb] = __popc(bal);
    }
    __syncthreads();
    if (threadIdx.x < kNumBinSlots) {
        int acc = 0;
        for (int w = 0; w < kCountBlock / 32; ++w) {
            int t = wcnt[w][threadIdx.x];
            wcnt[w][threadIdx.x] = acc;
            acc += t;
        }
    }
    __syncthreads();
    if (b >= 0) order[blockoff[b * nblk + blockIdx.x] + wcnt[wid][b] + __popc(mine & lanemask_lt())] = v;
    if (blockIdx.x == 0 && threadIdx.x <= kNumBinSlots)
        st->bin_start[threadIdx.x] = threadIdx.x < kNumBinSlots ? blockoff[threadIdx.x * nblk] : n;
}

// Symmetry hash of one entry: h(v, u, w) - h(u, v, w), summed over all
// entries modulo 2^64 (stats->sym_hash), is 0 when every entry has a mirror.
// Two rounds of the murmur3 finaliser per 32-bit half.
__device__ __forceinline__ unsigned fmix32(unsigned h)
{
    h ^= h >> 16;
    h *= 0x85EBCA6Bu;
    h ^= h >> 13;
    h *= 0xC2B2AE35u;
    return h ^ (h >> 16);
}
__device__ __forceinline__ unsigned long long dir_hash(int a, int b, unsigned long long w)
{
    const unsigned wl = (unsigned)w, wh = (unsigned)(w >> 32);
    const unsigned x = fmix32((unsigned)a ^ fmix32((unsigned)b ^ 0x9E3779B9u) ^ wl);
    const unsigned y = fmix32((unsigned)b + fmix32((unsigned)a + 0x7F4A7C15u) + wh * 0x85EBCA77u + wl);
    return ((unsigned long long)x << 32) | y;
}
__device__ __forceinline__ unsigned long long sym_term(int v, int u, unsigned long long w)
{
    return dir_hash(v, u, w) - dir_hash(u, v, w);
}

// Symmetry hash of a level, summed when a sweep first wants the incremental
// update: summed in every level init it cost 2 % of a run on 2^22 R-MAT
// vertices (17.98 ms against 17.65), which never asks for it.  A warp takes 1024 consecutive entries
// whatever rows they belong to: each lane finds its first entry's row by
// bisection and walks the offsets from there, so that a hub costs no more than
// the same entries in short rows (eight lanes per row cost 0.3 ms on 2^20 R-MAT
// vertices, most of it the hubs' tail).
constexpr int kHashChunk = 1024;
template <typename WT, bool W>
__global__ void __launch_bounds__(256) k_sym_hash(int n, long long E, const int64_t *__restrict__ offs,
                                                  const int32_t *__restrict__ nbr, const WT *__restrict__ w,
                                                  DevStats *st)
{
    constexpr int U = 8;
    const int lane = threadIdx.x & 31;
    const long long c0 = ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kHashChunk;
    const long long c1 = c0 + kHashChunk < E ? c0 + kHashChunk : E;
    unsigned long long hs = 0;
    if (c0 < E) {
        int lo = 0, hi = n;  // offs[lo] <= c0 < offs[hi]
        while (hi - lo > 1) {
            const int mid = lo + ((hi - lo) >> 1);
            if (offs[mid] <= c0) lo = mid;
            else hi = mid;
        }
        int r = lo;
        long long end = offs[r + 1];
        for (long long j = c0 + lane; j < c1; j += U * 32) {
            int u[U];
            WT wt[U];
#pragma unroll
            for (int q = 0; q < U; ++q) {
                const bool in = j + q * 32 < c1;
                u[q] = in ? nbr[j + q * 32] : 0;
                wt[q] = W && in ? w[j + q * 32] : (WT)1;
            }
#pragma unroll
            for (int q = 0; q < U; ++q) {
                if (j + q * 32 >= c1) break;
                while (end <= j + q * 32) end = offs[++r + 1];
                hs += sym_term(r, u[q], (unsigned long long)wt[q]);
            }
        }
    }
    block_add_u64(hs, &st->sym_hash);
}

// Weight, self-loop weight (the last one seen) and, with H, symmetry hash of
// the entries j, j + step, ... < e of vertex v's row.
template <typename WT, bool W, bool H>
__device__ __forceinline__ void row_sums(const int32_t *__restrict__ nbr, const WT *__restrict__ w, long long j,
                                         long long e, int step, int v, WT &k, WT &sf, unsigned long long &hs)
{
    constexpr int U = 4;
    for (; j < e; j += (long long)U * step) {
        int u[U];
        WT wt[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const long long i = j + (long long)q * step;
            u[q] = i < e ? nbr[i] : -1;
            wt[q] = i < e ? (W ? w[i] : (WT)1) : (WT)0;
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
            if (H && u[q] < 0) break;
            k += wt[q];
            if (u[q] == v) sf = wt[q];
            if (H) hs += sym_term(v, u[q], (unsigned long long)wt[q]);
        }
    }
}

// K = row weight sum, Self = self-loop weight (init_communities,
// kernel_functions.cu:34-73); Tot = K, In = Self.  Accumulates sum(K),
// sum(K^2) and sum(Self) for the modularity of the singleton partition and, with
// H, the symmetry hash.  Four entries per lane in flight.
template <typename WT, int G, bool W, bool H>
__global__ void __launch_bounds__(256) k_init_rows_group(const int32_t *__restrict__ list, int count,
                                                         const int64_t *__restrict__ offs,
                                                         const int32_t *__restrict__ nbr,
                                                         const WT *__restrict__ w, WT *K, WT *Self, WT *Tot,
                                                         WT *In, DevStats *st)
{
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), gw = lane / G;
    constexpr int GPW = 32 / G;
    const int wg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long sk = 0, ss = 0, hs = 0;
    typename SqSum<WT>::T sk2 = 0;
    for (int base = wg * GPW; base < count; base += nw * GPW) {
        const int idx = base + gw;
        const bool has = idx < count;
        int v = 0;
        long long s = 0, e = 0;
        if (has) {
            v = list[idx];
            s = offs[v];
            e = offs[v + 1];
        }
        WT k = 0, sf = 0;
        row_sums<WT, W, H>(nbr, w, s + sub, e, G, v, k, sf, hs);
#pragma unroll
        for (int o = G / 2; o >= 1; o >>= 1) {
            k += __shfl_xor_sync(GALA_FULL_MASK, k, o);
            sf += __shfl_xor_sync(GALA_FULL_MASK, sf, o);
        }
        if (has && sub == 0) {
            K[v] = k;
            Tot[v] = k;
            Self[v] = sf;
            In[v] = sf;
            sk += (unsigned long long)k;
            sk2 += SqSum<WT>::sq(k);
            ss += (unsigned long long)sf;
        }
    }
    block_add_u64(sk, &st->sum_k);
    SqSum<WT>::add(sk2, &st->sum_tot2, &st->sum_tot2_hi);
    block_add_u64(ss, &st->sum_in);
    if (H) block_add_u64(hs, &st->sym_hash);
}

template <typename WT, bool W, bool H>
__global__ void __launch_bounds__(256) k_init_rows_cta(const int32_t *__restrict__ list, int count,
                                                       const int64_t *__restrict__ offs,
                                                       const int32_t *__restrict__ nbr,
                                                       const WT *__restrict__ w, WT *K, WT *Self, WT *Tot, WT *In,
                                                       DevStats *st)
{
    __shared__ WT rk[8], rs[8];
    unsigned long long sk = 0, ss = 0, hs = 0;
    typename SqSum<WT>::T sk2 = 0;
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        int v = list[i];
        long long s = offs[v], e = offs[v + 1];
        WT k = 0, sf = 0;
        row_sums<WT, W, H>(nbr, w, s + threadIdx.x, e, blockDim.x, v, k, sf, hs);
        k = warp_sum(k);
        sf = warp_sum(sf);
        if ((threadIdx.x & 31) == 0) {
            rk[threadIdx.x >> 5] = k;
            rs[threadIdx.x >> 5] = sf;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            k = 0;
            sf = 0;
            for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
                k += rk[q];
                sf += rs[q];
            }
            K[v] = k;
            Tot[v] = k;
            Self[v] = sf;
            In[v] = sf;
            sk += (unsigned long long)k;
            sk2 += SqSum<WT>::sq(k);
            ss += (unsigned long long)sf;
        }
        __syncthreads();
    }
    block_add_u64(sk, &st->sum_k);
    SqSum<WT>::add(sk2, &st->sum_tot2, &st->sum_tot2_hi);
    block_add_u64(ss, &st->sum_in);
    if (H) block_add_u64(hs, &st->sym_hash);
}

__global__ void k_reset_level_stats(DevStats *st)
{
    st->sum_in = 0;
    st->sum_tot2 = 0;
    st->sum_tot2_hi = 0;
    st->sum_self = 0;
    st->sum_k = 0;
    st->max_deg = 0;
    st->err = 0;
    st->n_movers = 0;
}

// Symmetry hash of level g (stats->sym_hash).
void p1_sym_hash(const LevelGraph &g, Phase1Buffers &b, cudaStream_t st)
{
    cudaMemsetAsync(&b.stats->sym_hash, 0, sizeof(b.stats->sym_hash), st);
    const int grid = (int)((g.E + 8 * kHashChunk - 1) / (8 * kHashChunk));
    if (grid == 0) return;
    if (g.wide)
        k_sym_hash<long long, true><<<grid, 256, 0, st>>>(g.n, g.E, g.offs, g.nbr, (const long long *)g.w, b.stats);
    else if (g.w)
        k_sym_hash<int, true><<<grid, 256, 0, st>>>(g.n, g.E, g.offs, g.nbr, (const int *)g.w, b.stats);
    else
        k_sym_hash<int, false><<<grid, 256, 0, st>>>(g.n, g.E, g.offs, g.nbr, nullptr, b.stats);
    note_launch(1);
}

void p1_reset_level_stats(Phase1Buffers &b, cudaStream_t st)
{
    k_reset_level_stats<<<1, 1, 0, st>>>(b.stats);
    note_launch(1);
}

template <typename WT, bool H = false>
static void launch_init_rows(const LevelGraph &g, Phase1Buffers &b, int bin, const int32_t *list, int cnt,
                             cudaStream_t st, DevStats *stats = nullptr)
{
    if (cnt <= 0) return;
    if (!stats) stats = b.stats;
    const bool W = g.w != nullptr;
    const WT *w = (const WT *)g.w;
    WT *K = (WT *)b.K, *Self = (WT *)b.Self, *Tot = (WT *)b.Tot, *In = (WT *)b.In;
    const int cap = num_sms() * 8;
    auto grid_for = [&](int G) {
        long long blocks = ((long long)cnt * G + 255) / 256;
        return (int)(blocks < cap ? blocks : cap);
    };
#define GALA_INIT_GROUP(GV)                                                                              \
    do {                                                                                                 \
        if (W)                                                                                           \
            k_init_rows_group<WT, GV, true, H><<<grid_for(GV), 256, 0, st>>>(list, cnt, g.offs, g.nbr,   \
                                                                             w, K, Self, Tot, In, stats); \
        else                                                                                             \
            k_init_rows_group<WT, GV, false, H><<<grid_for(GV), 256, 0, st>>>(list, cnt, g.offs, g.nbr,  \
                                                                              w, K, Self, Tot, In, stats); \
    } while (0)
    switch (bin) {
    case 0: GALA_INIT_GROUP(4); break;
    case 1: GALA_INIT_GROUP(8); break;
    case 2: GALA_INIT_GROUP(16); break;
    case 3:
    case 4:
    case 5: GALA_INIT_GROUP(32); break;
    default: {
        int grid = cnt < cap ? cnt : cap;
        if (W)
            k_init_rows_cta<WT, true, H><<<grid, 256, 0, st>>>(list, cnt, g.offs, g.nbr, w, K, Self, Tot, In, stats);
        else
            k_init_rows_cta<WT, false, H><<<grid, 256, 0, st>>>(list, cnt, g.offs, g.nbr, w, K, Self, Tot, In, stats);
    }
    }
#undef GALA_INIT_GROUP
    note_launch(1);
}

// Level init part 1: labels/sizes, degree-bin counting sort.  The caller reads
// bin_start back before calling p1_level_init_rows.
void p1_level_init(const LevelGraph &g, Phase1Buffers &b, cudaStream_t st)
{
    const int n = g.n;
    const int nblk = (n + kCountBlock - 1) / kCountBlock;
    const int grid = (n + 255) / 256 < 4096 ? (n + 255) / 256 : 4096;
    if (g.ks_ready && g.wide)
        k_init_vertices_ks<long long><<<grid, 256, 0, st>>>(n, b.comm, (const long long *)b.K,
                                                            (const long long *)b.Self, (long long *)b.Tot, b.size,
                                                            (long long *)b.In, b.stats);
    else if (g.ks_ready)
        k_init_vertices_ks<int><<<grid, 256, 0, st>>>(n, b.comm, b.K, b.Self, b.Tot, b.size, b.In, b.stats);
    else if (g.wide)
        k_init_vertices<long long><<<grid, 256, 0, st>>>(n, b.comm, (long long *)b.K, (long long *)b.Self,
                                                         (long long *)b.Tot, b.size, (long long *)b.In);
    else
        k_init_vertices<int><<<grid, 256, 0, st>>>(n, b.comm, b.K, b.Self, b.Tot, b.size, b.In);
    k_bin_count<<<nblk, kCountBlock, 0, st>>>(n, g.offs, b.blockcnt, nblk, b.stats, b.lim);
    exclusive_scan(b.blockcnt, b.blockoff, (long long)kNumBinSlots * nblk, OpIdentity(), b.scan_partial,
                   &b.stats->total, st, &b.stats->err);
    k_bin_scatter<<<nblk, kCountBlock, 0, st>>>(n, g.offs, b.blockoff, nblk, b.order, b.stats, b.lim);
    note_launch(3);
}

// Unweighted level whose rows are still being copied: K = Tot = degree of
// every vertex from the offsets alone, so a vertex's first sweep needs only
// its own row.
__global__ void k_init_degree(int n, const int64_t *__restrict__ offs, int32_t *K, int32_t *Tot)
{
    for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        const int d = (int)(offs[v + 1] - offs[v]);
        K[v] = d;
        Tot[v] = d;
    }
}

// Sub-ranges of the degree bins per row chunk: lo[k][bin] = first position in
// the bin's segment of the order list (ascending ids within a bin) of a vertex
// id >= vstart[k]; cnt[k][bin] = lo[k + 1][bin] - lo[k][bin].
__global__ void k_chunk_bounds(const int32_t *__restrict__ order, const DevStats *__restrict__ st, ChunkStarts vs,
                               int P, int32_t *lo, int32_t *cnt)
{
    const int32_t *vstart = vs.v;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (P + 1) * kNumBins) return;
    const int k = t / kNumBins, bin = t % kNumBins;
    const int bs = st->bin_start[bin], be = st->bin_start[bin + 1];
    auto first_ge = [&](int id) {
        int l = bs, h = be;  // first position in [bs, be) with order >= id
        while (l < h) {
            const int m = (l + h) >> 1;
            if (order[m] < id) l = m + 1;
            else h = m;
        }
        return l - bs;
    };
    const int a = k < P ? first_ge(vstart[k]) : be - bs;
    lo[k * kNumBins + bin] = a;
    if (k < P) cnt[k * kNumBins + bin] = (k + 1 < P ? first_ge(vstart[k + 1]) : be - bs) - a;
}

void p1_init_degree(const LevelGraph &g, Phase1Buffers &b, cudaStream_t st)
{
    const int grid = std::min((g.n + 255) / 256, num_sms() * 8);
    k_init_degree<<<grid > 0 ? grid : 1, 256, 0, st>>>(g.n, g.offs, b.K, b.Tot);
    note_launch(1);
}

void p1_chunk_bounds(Phase1Buffers &b, const ChunkStarts &vs, int P, int32_t *d_lo, int32_t *d_cnt, cudaStream_t st)
{
    const int t = (P + 1) * kNumBins;
    k_chunk_bounds<<<(t + 127) / 128, 128, 0, st>>>(b.order, b.stats, vs, P, d_lo, d_cnt);
    note_launch(1);
}

void p1_init_rows_range(const LevelGraph &g, Phase1Buffers &b, int bin, const int32_t *list, int cnt, DevStats *stats,
                        cudaStream_t st)
{
    if (g.wide)
        launch_init_rows<long long, true>(g, b, bin, list, cnt, st, stats);
    else
        launch_init_rows<int, true>(g, b, bin, list, cnt, st, stats);
}

void p1_level_init_rows(const LevelGraph &g, Phase1Buffers &b, const int *bin_start, cudaStream_t st)
{
    if (g.ks_ready) return;  // K, Self, Tot, In and the sums came with the level init
    for (int bin = 0; bin < kNumBins; ++bin) {
        if (g.wide)
            launch_init_rows<long long>(g, b, bin, b.order + bin_start[bin], bin_start[bin + 1] - bin_start[bin], st);
        else
            launch_init_rows<int>(g, b, bin, b.order + bin_start[bin], bin_start[bin + 1] - bin_start[bin], st);
    }
}

// ------------------------------------------------------------------------
// Decide-and-move: one launch per degree bin
// ------------------------------------------------------------------------
template <typename WT, int G, bool W>
__global__ void __launch_bounds__(256) k_decide_group(DecideArgs<WT> a, const int32_t *__restrict__ list,
                                                      const int *__restrict__ count_ptr)
{
    __shared__ int stage_buf[8][3 * kStageM];
    WarpStage<kStageM, 3> stage{stage_buf[threadIdx.x >> 5], 0};
    decide_group<WT, G, W>(a, list, *count_ptr, (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                           (gridDim.x * blockDim.x) >> 5, stage);
    int *const mlists[3] = {a.mv_v, a.mv_old, a.mv_new};
    stage.flush(mlists, a.n_movers);
}

template <typename WT, bool W, int TW, int MINB>
__global__ void __launch_bounds__(256, MINB) k_decide_warp(DecideArgs<WT> a, const int32_t *__restrict__ list,
                                                     const int *__restrict__ count_ptr, int dlo, int dhi)
{
    extern __shared__ long long wsm_ll[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    WT *vals = (WT *)wsm_ll + wib * TW;
    int *keys = (int *)((WT *)wsm_ll + kWarpWarps * TW) + wib * TW;
    unsigned short *occ =
        (unsigned short *)((int *)((WT *)wsm_ll + kWarpWarps * TW) + kWarpWarps * TW) + wib * (TW / 2);
    for (int j = lane; j < TW; j += 32) {
        keys[j] = -1;
        vals[j] = 0;
    }
    __syncwarp();
    decide_warp<WT, W, TW>(a, list, *count_ptr, (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                           (gridDim.x * blockDim.x) >> 5, dlo, dhi, keys, vals, occ);
}

// 32 registers, so that the threads of an SM's full 64 warps fit whatever the
// block: without the bound the 1024-thread instance took 52 and ran one CTA per SM
// (phase 1 of 8,000 vertices in rows of 3000, 24M entries: 1.80 ms, 1.53 so).
template <typename WT, int BLOCK, bool W>
__global__ void __launch_bounds__(BLOCK, 2048 / BLOCK) k_decide_cta(DecideArgs<WT> a, const int32_t *__restrict__ list,
                                                      const int *__restrict__ count_ptr, int tmax, int dlo,
                                                      int dhi)
{
    extern __shared__ long long dyn_smem_ll[];
    WT *vals = (WT *)dyn_smem_ll;
    int *keys = (int *)(vals + tmax);
    for (int j = threadIdx.x; j < tmax; j += BLOCK) {
        keys[j] = -1;
        vals[j] = 0;
    }
    decide_cta<WT, BLOCK, W>(a, list, *count_ptr, blockIdx.x, gridDim.x, tmax, dlo, dhi, keys, vals,
                             (unsigned short *)(keys + tmax));
}

// Resident 256-thread blocks per SM of the 33-256 kernel (occupancy query,
// cached per instantiation).
template <typename WT, int TW, int MINB>
int warp_resident(bool W)
{
    static int cached[2] = {0, 0};
    int &r = cached[W ? 1 : 0];
    if (r == 0) {
        int k = 0;
        if (W)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_decide_warp<WT, true, TW, MINB>, 256,
                                                          warp_smem<WT, TW>());
        else
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_decide_warp<WT, false, TW, MINB>, 256,
                                                          warp_smem<WT, TW>());
        r = k > 0 ? k : 1;
    }
    return r;
}

// First sweep of a level: every vertex is its own community (comm[u] = u
// after the level init), and rows hold distinct neighbours, so every entry
// is its own candidate community: no aggregation table.  One group of
// GROUP threads (a warp, or the whole CTA) per vertex.
template <typename WT, bool W>
__device__ __forceinline__ void first_scan_best(const DecideArgs<WT> &a, const GainTerms<WT> &gt, long long s, int deg,
                                                int v, int first, int stride, Cand<WT> &best, WT &wc)
{
    for (int j = first; j < deg; j += stride) {
        const int u = a.nbr[s + j];
        const WT w = W ? a.w[s + j] : (WT)1;
        if (u == v)
            wc += w;
        else
            best.offer(gt, u, w, a.Tot[u]);
    }
}

template <typename WT, bool W>
__device__ __forceinline__ void first_scan(const DecideArgs<WT> &a, const Scale &sc, const GainTerms<WT> &gt,
                                           const Cand<WT> &best, long long s, int deg, int v, int first, int stride,
                                           WT ki, WT tcur, double &dq, int &bc)
{
    for (int j = first; j < deg; j += stride) {
        const int u = a.nbr[s + j];
        if (u == v) continue;
        const WT w = W ? a.w[s + j] : (WT)1, tc = a.Tot[u];
        if (!a.fp64_only && !best.fp64_rival(gt, w, tc)) continue;
        const double d = gain_dq(w, ki, tc, tcur, sc.c);
        if (d > 0.0 && cand_better(d, u, dq, bc)) {
            dq = d;
            bc = u;
        }
    }
}

// Degree <= G * U: lane groups of G, U entries per lane in one predicated batch.
// Without the label gather and the search for equal labels: 128 graphs of 58M
// entries 31.1 -> 30.5 ms, 2^22 R-MAT vertices 16.94 -> 16.81.
template <typename WT, int G, int U, bool W>
__global__ void __launch_bounds__(256) k_first_group(DecideArgs<WT> a, const int32_t *__restrict__ list,
                                                     const int *__restrict__ count_ptr)
{
    __shared__ int stage_buf[8][3 * kStageM];
    WarpStage<kStageM, 3> stage{stage_buf[threadIdx.x >> 5], 0};
    int *const mlists[3] = {a.mv_v, a.mv_old, a.mv_new};
    constexpr int GPW = 32 / G;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), gw = lane / G;
    const int count = *count_ptr;
    const int wg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int base = wg * GPW; base < count; base += nw * GPW) {
        const int idx = base + gw;
        bool has = idx < count;
        int v = -1, deg = 0;
        WT ki = 0, sf = 0;
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
            ki = a.K[v];
            sf = a.Self[v];
        }
        const WT tcur = has ? a.Tot[v] : (WT)0;
        int u[U];
        WT wt[U], tc[U], wc = 0;
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const int j = sub + q * G;
            u[q] = j < deg ? a.nbr[s + j] : -1;
            wt[q] = W && j < deg ? a.w[s + j] : (WT)1;
        }
#pragma unroll
        for (int q = 0; q < U; ++q) {
            if (u[q] >= 0 && u[q] == v) {  // own entry: no candidate
                wc += wt[q];
                u[q] = -1;
            }
            tc[q] = u[q] >= 0 ? a.Tot[u[q]] : (WT)0;
        }
        const GainTerms<WT> gt(sc, ki, tcur);
        Cand<WT> best(v);
#pragma unroll
        for (int q = 0; q < U; ++q)
            if (u[q] >= 0) best.offer(gt, u[q], wt[q], tc[q]);
        warp_merge(best, wc, G);
        int bc = best.c, dec = 0;
        if (has && sub == 0) dec = best.decide(a.fp64_only, sc, v, wc, sf, ki);
        const bool fp = dec == 2;
        if (__any_sync(GALA_FULL_MASK, fp)) {
            // the reference's FP64 evaluation of the same candidates
            double dq = 0.0;
            int fc = v;
#pragma unroll
            for (int q = 0; q < U; ++q) {
                if (u[q] < 0) continue;
                const double d = gain_dq(wt[q], ki, tc[q], tcur, sc.c);
                if (d > 0.0 && cand_better(d, u[q], dq, fc)) {
                    dq = d;
                    fc = u[q];
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
                dec = (fc != v && gain_correct(dq, wc, sf) > 0.0) ? 1 : 0;
                atomicAdd(a.fp64_decisions, 1ull);
            }
        }
        const bool move = has && sub == 0 && dec == 1 && guard_ok(a, v, bc);
        if (has && sub == 0) write_features(a, sc, v, best, wc, sf, ki, deg);
        const int item[3] = {v, v, bc};
        stage.push(move, item, mlists, a.n_movers);
    }
    stage.flush(mlists, a.n_movers);
}

template <typename WT, bool W>
__global__ void __launch_bounds__(256) k_first_warp(DecideArgs<WT> a, const int32_t *__restrict__ list,
                                                    const int *__restrict__ count_ptr)
{
    const int lane = threadIdx.x & 31;
    const int count = *count_ptr;
    const int wg = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int i = wg; i < count; i += nw) {
        const int v = list[i];
        if (stopped(a, v)) continue;
        const Scale sc = scale_of(a, v);
        const long long s = a.offs[v];
        const int deg = (int)(a.offs[v + 1] - s);
        const int cur = a.comm[v];  // = v
        const WT ki = a.K[v], tcur = a.Tot[cur], sf = a.Self[v];
        const GainTerms<WT> gt(sc, ki, tcur);
        Cand<WT> best(cur);
        WT wc = 0;
        first_scan_best<WT, W>(a, gt, s, deg, v, lane, 32, best, wc);
        warp_merge(best, wc, 32);
        int bc = best.c;
        int dec = best.decide(a.fp64_only, sc, cur, wc, sf, ki);  // warp-uniform
        if (dec == 2) {
            double dq = 0.0;
            int fc = cur;
            first_scan<WT, W>(a, sc, gt, best, s, deg, v, lane, 32, ki, tcur, dq, fc);
            warp_argmax(dq, fc);
            bc = fc;
            dec = (fc != cur && gain_correct(dq, wc, sf) > 0.0) ? 1 : 0;
            if (lane == 0) atomicAdd(a.fp64_decisions, 1ull);
        }
        const bool move = lane == 0 && dec == 1 && guard_ok(a, cur, bc);
        if (lane == 0) write_features(a, sc, v, best, wc, sf, ki, deg);
        append_mover(a, move, v, cur, bc);
    }
}

template <typename WT, int BLOCK, bool W>
__global__ void __launch_bounds__(BLOCK) k_first_cta(DecideArgs<WT> a, const int32_t *__restrict__ list,
                                                     const int *__restrict__ count_ptr)
{
    __shared__ double r_dq[BLOCK / 32];
    __shared__ int r_c[BLOCK / 32];
    __shared__ CandRow<WT, BLOCK / 32> r_best;
    __shared__ int s_dec, s_bc;
    __shared__ WT s_wc;
    constexpr int NW = BLOCK / 32;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int count = *count_ptr;
    for (int i = blockIdx.x; i < count; i += gridDim.x) {
        const int v = list[i];
        if (stopped(a, v)) continue;
        const Scale sc = scale_of(a, v);
        const long long s = a.offs[v];
        const int deg = (int)(a.offs[v + 1] - s);
        const int cur = a.comm[v];  // = v
        const WT ki = a.K[v], tcur = a.Tot[cur], sf = a.Self[v];
        const GainTerms<WT> gt(sc, ki, tcur);
        Cand<WT> best(cur);
        WT wc = 0;
        first_scan_best<WT, W>(a, gt, s, deg, v, threadIdx.x, BLOCK, best, wc);
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
        if (s_dec == 2) {  // block-uniform
            double dq = 0.0;
            int fc = cur;
            Cand<WT> top(cur);
            WT unused;
            r_best.get(0, 1, cur, top, unused);
            first_scan<WT, W>(a, sc, gt, top, s, deg, v, threadIdx.x, BLOCK, ki, tcur, dq, fc);
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
            if (lane == 0) write_features(a, sc, v, best, s_wc, sf, ki, deg);
            append_mover(a, move, v, cur, s_bc);
        }
        __syncthreads();
    }
}

constexpr int kCtaTable5 = 4096;
constexpr int kCtaTable6 = 16384;
// Resident blocks per SM of a CTA decide kernel with a tmax-slot table (cached).
template <typename WT, int BLOCK>
int cta_resident(bool W, int tmax)
{
    static int cached[2][32] = {};
    int &r = cached[W ? 1 : 0][__builtin_ctz((unsigned)tmax)];
    if (r == 0) {
        int k = 0;
        if (W)
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_decide_cta<WT, BLOCK, true>, BLOCK, cta_smem<WT>(tmax));
        else
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, k_decide_cta<WT, BLOCK, false>, BLOCK,
                                                          cta_smem<WT>(tmax));
        r = k > 0 ? k : 1;
    }
    return r;
}

// Arguments of the decide kernels for the weight type WT.
template <typename WT>
static DecideArgs<WT> decide_args(const LevelGraph &g, Phase1Buffers &b, double constant, long long m2,
                                  int fp64_only)
{
    DecideArgs<WT> a;
    a.offs = g.offs;
    a.nbr = g.nbr;
    a.w = (const WT *)g.w;
    a.comm = b.comm;
    a.K = (const WT *)b.K;
    a.Self = (const WT *)b.Self;
    a.Tot = (const WT *)b.Tot;
    a.size = b.size;
    a.mv_v = b.mv_v;
    a.mv_old = b.mv_old;
    a.mv_new = b.mv_new;
    a.n_movers = &b.stats->n_movers;
    a.err = &b.stats->err;
    a.fp64_decisions = &b.stats->fp64_decisions;
    a.constant = constant;
    a.m2 = m2;
    a.fp64_only = fp64_only;
    a.feat_gain = b.features_on ? b.feat_gain : nullptr;
    a.feat_ndist = b.feat_ndist;
    a.gid = b.gid;
    a.m2g = b.m2g;
    a.cg = b.cg;
    a.stop = b.gstop;
    return a;
}

template <typename WT>
static void decide_t(const LevelGraph &g, Phase1Buffers &b, int bin, const int32_t *list, const int *count_ptr,
                     int level_count, double constant, long long m2, int fp64_only, bool first, cudaStream_t st)
{
    const DecideArgs<WT> a = decide_args<WT>(g, b, constant, m2, fp64_only);
    const bool W = g.w != nullptr;
    const int cap = num_sms() * 8;
    auto grid_lanes = [&](int lanes_per_item) {
        long long blocks = ((long long)level_count * lanes_per_item + 255) / 256;
        return (int)(blocks < cap ? blocks : cap);
    };
#define GALA_FG(GV, UV)                                                                                \
    do {                                                                                               \
        if (W)                                                                                         \
            k_first_group<WT, GV, UV, true><<<grid_lanes(GV), 256, 0, st>>>(a, list, count_ptr);       \
        else                                                                                           \
            k_first_group<WT, GV, UV, false><<<grid_lanes(GV), 256, 0, st>>>(a, list, count_ptr);      \
    } while (0)
    if (first && bin <= 6) {  // singleton partition: no aggregation
        if (bin == 0) {
            GALA_FG(4, 1);
        } else if (bin == 1) {
            GALA_FG(4, 2);
        } else if (bin == 2) {
            GALA_FG(4, 4);
        } else if (bin == 3) {
            GALA_FG(8, 4);
        } else if (bin == 4) {
            if (W)
                k_first_warp<WT, true><<<grid_lanes(32), 256, 0, st>>>(a, list, count_ptr);
            else
                k_first_warp<WT, false><<<grid_lanes(32), 256, 0, st>>>(a, list, count_ptr);
        } else {
            const int grid = level_count < num_sms() * 8 ? level_count : num_sms() * 8;
            if (W)
                k_first_cta<WT, 256, true><<<grid, 256, 0, st>>>(a, list, count_ptr);
            else
                k_first_cta<WT, 256, false><<<grid, 256, 0, st>>>(a, list, count_ptr);
        }
#undef GALA_FG
        note_launch(1);
        return;
    }
#define GALA_DG(GV)                                                                                    \
    do {                                                                                               \
        if (W)                                                                                         \
            k_decide_group<WT, GV, true><<<grid_lanes(GV), 256, 0, st>>>(a, list, count_ptr);          \
        else                                                                                           \
            k_decide_group<WT, GV, false><<<grid_lanes(GV), 256, 0, st>>>(a, list, count_ptr);         \
    } while (0)
    switch (bin) {
    case 0: GALA_DG(4); break;
    case 1: GALA_DG(8); break;
    case 2: GALA_DG(16); break;
    case 3: GALA_DG(32); break;
    case 4: {
        // as many CTAs as can reside (tables and registers): no second wave
        // two launches: rows up to 128 entries with 256-slot tables (more
        // resident warps), longer rows with 512-slot tables
        {
            const int cap4 = num_sms() * warp_resident<WT, kWarpTable / 2, 8>(W);
            const int g4 = grid_lanes(32) < cap4 ? grid_lanes(32) : cap4;
            const size_t sm = warp_smem<WT, kWarpTable / 2>();
            if (W)
                k_decide_warp<WT, true, kWarpTable / 2, 8><<<g4, 256, sm, st>>>(a, list, count_ptr, 0, kWarpTable / 4);
            else
                k_decide_warp<WT, false, kWarpTable / 2, 8><<<g4, 256, sm, st>>>(a, list, count_ptr, 0, kWarpTable / 4);
        }
        {
            const int cap4 = num_sms() * warp_resident<WT, kWarpTable, 1>(W);
            const int g4 = grid_lanes(32) < cap4 ? grid_lanes(32) : cap4;
            const size_t sm = warp_smem<WT, kWarpTable>();
            if (W)
                k_decide_warp<WT, true, kWarpTable, 1><<<g4, 256, sm, st>>>(a, list, count_ptr, kWarpTable / 4, INT_MAX);
            else
                k_decide_warp<WT, false, kWarpTable, 1><<<g4, 256, sm, st>>>(a, list, count_ptr, kWarpTable / 4, INT_MAX);
        }
        note_launch(1);
        break;
    }
    case 5: {  // 256 (default) or 512 threads per vertex
        if (b.b5_block == 256) {
            // two launches: rows up to 1024 entries with a 2048-slot table
            // (more resident CTAs), longer rows with the 4096-slot table
            const int splits[2][3] = {{kCtaTable5 / 2, 0, kCtaTable5 / 4}, {kCtaTable5, kCtaTable5 / 4, INT_MAX}};
            for (const auto &sp : splits) {
                const int cap5 = num_sms() * cta_resident<WT, 256>(W, sp[0]);
                const int grid = level_count < cap5 ? level_count : cap5;
                const size_t sm = cta_smem<WT>(sp[0]);
                if (W)
                    k_decide_cta<WT, 256, true><<<grid, 256, sm, st>>>(a, list, count_ptr, sp[0], sp[1], sp[2]);
                else
                    k_decide_cta<WT, 256, false><<<grid, 256, sm, st>>>(a, list, count_ptr, sp[0], sp[1], sp[2]);
            }
            note_launch(1);
        } else {
            const size_t sm = cta_smem<WT>(kCtaTable5);
            int grid = level_count < num_sms() * 4 ? level_count : num_sms() * 4;
            if (W)
                k_decide_cta<WT, 512, true><<<grid, 512, sm, st>>>(a, list, count_ptr, kCtaTable5, 0, INT_MAX);
            else
                k_decide_cta<WT, 512, false><<<grid, 512, sm, st>>>(a, list, count_ptr, kCtaTable5, 0, INT_MAX);
        }
        break;
    }
    case 6: {
        const int splits[2][3] = {{kCtaTable6 / 2, 0, kCtaTable6 / 4}, {kCtaTable6, kCtaTable6 / 4, INT_MAX}};
        for (const auto &sp : splits) {
            const int cap6 = num_sms() * cta_resident<WT, 1024>(W, sp[0]);
            const int grid = level_count < cap6 ? level_count : cap6;
            const size_t sm = cta_smem<WT>(sp[0]);
            if (W)
                k_decide_cta<WT, 1024, true><<<grid, 1024, sm, st>>>(a, list, count_ptr, sp[0], sp[1], sp[2]);
            else
                k_decide_cta<WT, 1024, false><<<grid, 1024, sm, st>>>(a, list, count_ptr, sp[0], sp[1], sp[2]);
        }
        note_launch(1);
        break;
    }
    default: return;  // hub vertices: p1_hub_decide
    }
#undef GALA_DG
    note_launch(1);
}

void p1_decide(const LevelGraph &g, Phase1Buffers &b, int bin, const int32_t *list, const int *count_ptr,
               int level_count, double constant, long long m2, int fp64_only, bool first, cudaStream_t st)
{
    if (level_count <= 0) return;
    if (g.wide)
        decide_t<long long>(g, b, bin, list, count_ptr, level_count, constant, m2, fp64_only, first, st);
    else
        decide_t<int>(g, b, bin, list, count_ptr, level_count, constant, m2, fp64_only, first, st);
}

template <typename WT>
static void configure_t()
{
    cudaFuncSetAttribute(k_decide_cta<WT, 1024, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)cta_smem<WT>(kCtaTable6));
    cudaFuncSetAttribute(k_decide_cta<WT, 1024, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)cta_smem<WT>(kCtaTable6));
    cudaFuncSetAttribute(k_decide_cta<WT, 512, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)cta_smem<WT>(kCtaTable5));
    cudaFuncSetAttribute(k_decide_cta<WT, 256, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)cta_smem<WT>(kCtaTable5));
    cudaFuncSetAttribute(k_decide_cta<WT, 256, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)cta_smem<WT>(kCtaTable5));
    cudaFuncSetAttribute(k_decide_cta<WT, 512, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)cta_smem<WT>(kCtaTable5));
    cudaFuncSetAttribute(k_decide_warp<WT, true, kWarpTable, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)warp_smem<WT, kWarpTable>());
    cudaFuncSetAttribute(k_decide_warp<WT, false, kWarpTable, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)warp_smem<WT, kWarpTable>());
    cudaFuncSetAttribute(k_decide_warp<WT, true, kWarpTable / 2, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)warp_smem<WT, kWarpTable / 2>());
    cudaFuncSetAttribute(k_decide_warp<WT, false, kWarpTable / 2, 8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)warp_smem<WT, kWarpTable / 2>());
}

void p1_configure_kernels()
{
    configure_t<int>();
    configure_t<long long>();
}

// ------------------------------------------------------------------------
// Apply (sign = +1) or revert (sign = -1) the movers of an iteration
// (Tot += Tot_update, size += size_update, louvain_main_process.cu:949-953).
// ------------------------------------------------------------------------
template <typename WT>
__global__ void k_apply_movers(const int32_t *__restrict__ mv_v, const int32_t *__restrict__ mv_old,
                               const int32_t *__restrict__ mv_new, DevStats *stp, int sign, int32_t *comm, WT *Tot,
                               int32_t *size, const WT *__restrict__ K, int32_t *last_move, int iteration,
                               const int64_t *__restrict__ offs, uint8_t *moved)
{
    const int nm = sign > 0 ? stp->n_movers : stp->prev_movers;
    const int lane = threadIdx.x & 31;
    unsigned long long deg = 0;
    for (int i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < nm; i0 += gridDim.x * blockDim.x) {
        const int i = i0 + lane;
        const bool valid = i < nm;
        int from = -1, to = -1;
        WT k = 0;
        if (valid) {
            const int v = mv_v[i];
            from = sign > 0 ? mv_old[i] : mv_new[i];
            to = sign > 0 ? mv_new[i] : mv_old[i];
            k = K[v];
            comm[v] = to;
            if (last_move && sign > 0) last_move[v] = iteration;
            if (offs) deg += (unsigned long long)(offs[v + 1] - offs[v]);
            if (moved) moved[v] = 1;
        }
        move_totals(valid, from, to, k, Tot, size);
    }
    if (offs) block_add_u64(deg, &stp->mv_edges);
}

void p1_apply_movers(Phase1Buffers &b, int sign, int n, cudaStream_t st, int iteration, const int64_t *offs,
                     uint8_t *moved)
{
    if (sign < 0) offs = nullptr, moved = nullptr;
    int grid = (n + 255) / 256;
    int cap = num_sms() * 4;
    if (grid > cap) grid = cap;
    if (grid < 1) grid = 1;
    if (b.wide)
        k_apply_movers<long long><<<grid, 256, 0, st>>>(b.mv_v, b.mv_old, b.mv_new, b.stats, sign, b.comm,
                                                        (long long *)b.Tot, b.size, (const long long *)b.K, nullptr,
                                                        iteration, offs, moved);
    else
        k_apply_movers<int><<<grid, 256, 0, st>>>(b.mv_v, b.mv_old, b.mv_new, b.stats, sign, b.comm, b.Tot, b.size,
                                                  b.K, b.features_on ? b.last_move : nullptr, iteration, offs, moved);
    note_launch(1);
}

// min over non-empty Tot (Tot_op, kernel_functions.cuh:112-121) and sum Tot^2.
template <typename WT>
__global__ void k_tot_reduce(const WT *__restrict__ Tot, int n, DevStats *st)
{
    long long mn = 0x7fffffffffffffffLL;
    typename SqSum<WT>::T s2 = 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        const WT t = Tot[c];
        if (t != 0) {
            mn = min(mn, (long long)t);
            s2 += SqSum<WT>::sq(t);
        }
    }
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) mn = min(mn, __shfl_xor_sync(GALA_FULL_MASK, mn, o));
    if ((threadIdx.x & 31) == 0 && mn != 0x7fffffffffffffffLL) atomicMin(&st->min_tot, mn);
    SqSum<WT>::add(s2, &st->sum_tot2, &st->sum_tot2_hi);
}

void p1_tot_reduce(Phase1Buffers &b, int n, cudaStream_t st)
{
    int grid = (n + 1023) / 1024;
    int cap = num_sms() * 4;
    if (grid > cap) grid = cap;
    if (grid < 1) grid = 1;
    if (b.wide)
        k_tot_reduce<long long><<<grid, 1024, 0, st>>>((const long long *)b.Tot, n, b.stats);
    else
        k_tot_reduce<int><<<grid, 1024, 0, st>>>(b.Tot, n, b.stats);
    note_launch(1);
}

__global__ void k_iter_reset(DevStats *st, int next, long long min_tot_init)
{
    st->prev_movers = st->n_movers;
    st->n_movers = 0;
    st->mv_edges = 0;
    st->push_mode = 0;
    st->push_len = 0;
    st->batch_running = 0;
    st->batch_rejects = 0;
    st->sum_in = 0;
    st->sum_tot2 = 0;
    st->sum_tot2_hi = 0;
    st->min_tot = min_tot_init;
    st->act_edges[next] = 0;
    st->act_vertices[next] = 0;
    for (int i = 0; i < kNumBins; ++i) st->act_count[next][i] = 0;
}

void p1_iter_reset(Phase1Buffers &b, int next, long long min_tot_init, cudaStream_t st)
{
    k_iter_reset<<<1, 1, 0, st>>>(b.stats, next, min_tot_init);
    note_launch(1);
}

// ------------------------------------------------------------------------
// Weight update + pruning: one launch per degree bin
// ------------------------------------------------------------------------
template <typename WT>
__device__ __forceinline__ void add_update_sums(const UpdateArgs<WT> &a, const UpdateSums &s)
{
    block_add_u64(s.in, &a.st->sum_in);
    block_add_u64(s.edges, &a.st->act_edges[a.next]);
    block_add_i32(s.act, &a.st->act_vertices[a.next]);
}

template <typename WT, int G, int U, bool W>
__global__ void __launch_bounds__(256) k_update_group(UpdateArgs<WT> a, const int32_t *__restrict__ list, int count)
{
    if (a.st->push_mode) return;  // the incremental update runs instead
    __shared__ int stage_buf[8][kStageN];
    WarpStage<kStageN, 1> stage{stage_buf[threadIdx.x >> 5], 0};
    UpdateSums sums;
    update_group<WT, G, U, W>(a, list, count, a.st->min_tot, (blockIdx.x * blockDim.x + threadIdx.x) >> 5,
                           (gridDim.x * blockDim.x) >> 5, stage, sums);
    add_update_sums(a, sums);
}

template <typename WT, bool W>
__global__ void __launch_bounds__(256) k_update_cta(UpdateArgs<WT> a, const int32_t *__restrict__ list, int count)
{
    if (a.st->push_mode) return;  // the incremental update runs instead
    UpdateSums sums;
    update_cta<WT, W>(a, list, count, a.st->min_tot, blockIdx.x, gridDim.x, sums);
    add_update_sums(a, sums);
}

template <typename WT>
static UpdateArgs<WT> update_args(const LevelGraph &g, Phase1Buffers &b, int bin, int next, int bin_start,
                                  double constant, long long m2)
{
    UpdateArgs<WT> a;
    a.offs = g.offs;
    a.nbr = g.nbr;
    a.w = (const WT *)g.w;
    a.comm = b.comm;
    a.K = (const WT *)b.K;
    a.Self = (const WT *)b.Self;
    a.Tot = (const WT *)b.Tot;
    a.In = (WT *)b.In;
    a.act_flag = b.act_flag;
    a.act_list = b.act[next] + bin_start;
    a.act_counter = &b.stats->act_count[next][bin];
    a.st = b.stats;
    a.constant = constant;
    a.m2 = m2;
    a.next = next;
    a.gid = b.gid;
    a.m2g = b.m2g;
    a.cg = b.cg;
    a.stop = b.gstop;
    a.min_tot_g = b.min_tot_g;
    return a;
}

template <typename WT>
static void update_t(const LevelGraph &g, Phase1Buffers &b, int bin, const int32_t *list, int count, int next,
                     int bin_start, double constant, long long m2, cudaStream_t st)
{
    const UpdateArgs<WT> a = update_args<WT>(g, b, bin, next, bin_start, constant, m2);
    const bool W = g.w != nullptr;
    const int cap = num_sms() * 8;
    auto grid_lanes = [&](int G) {
        long long blocks = ((long long)count * G + 255) / 256;
        return (int)(blocks < cap ? blocks : cap);
    };
#define GALA_UG(GV, UV)                                                                                \
    do {                                                                                               \
        if (W)                                                                                         \
            k_update_group<WT, GV, UV, true><<<grid_lanes(GV), 256, 0, st>>>(a, list, count);          \
        else                                                                                           \
            k_update_group<WT, GV, UV, false><<<grid_lanes(GV), 256, 0, st>>>(a, list, count);         \
    } while (0)
    // groups narrower than the rows, with one predicated batch of loads per lane
    // up to 32 entries: a warp serves 8-16 vertices and every load of a row is in
    // flight at once.  Batch of 128 graphs 33.2 -> 31.9 ms, R-MAT scale 22 18.27
    // -> 17.96 ms against groups of 4 / 8 / 8 / 16 lanes whose remainder entries
    // load one after the other (small_level.cu, with half the warps, measured
    // best with groups of 4 / 4 / 4 / 8).
    switch (bin) {
    case 0: GALA_UG(2, 2); break;
    case 1: GALA_UG(2, 4); break;
    case 2: GALA_UG(4, 4); break;
    case 3: GALA_UG(4, 8); break;
    case 4: GALA_UG(8, 8); break;
    case 5: GALA_UG(32, 8); break;
    default: {
        int grid = count < cap ? count : cap;
        if (W)
            k_update_cta<WT, true><<<grid, 256, 0, st>>>(a, list, count);
        else
            k_update_cta<WT, false><<<grid, 256, 0, st>>>(a, list, count);
    }
    }
#undef GALA_UG
    note_launch(1);
}

void p1_update(const LevelGraph &g, Phase1Buffers &b, int bin, const int32_t *list, int count, int next,
               int bin_start, double constant, long long m2, cudaStream_t st)
{
    if (count <= 0) return;
    if (g.wide)
        update_t<long long>(g, b, bin, list, count, next, bin_start, constant, m2, st);
    else
        update_t<int>(g, b, bin, list, count, next, bin_start, constant, m2, st);
}

// ------------------------------------------------------------------------
// Hub vertices: plan of a level, decide and weight update launches
// ------------------------------------------------------------------------
__global__ void k_hub_plan(HubPlan p, const int64_t *__restrict__ offs)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < p.H; i += gridDim.x * blockDim.x) {
        const int v = p.hubs[i];
        hub_table(p, offs[v + 1] - offs[v], p.T[i], p.chunks[i], p.tchunks[i]);
    }
}

__global__ void k_hub_tail(HubPlan p, const DevStats *st)
{
    p.toff[p.H] = st->total;
    p.coff[p.H] = st->total2;
    p.tcoff[p.H] = st->total3;
}

__global__ void k_hub_work(HubPlan p)
{
    hub_work(p, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5);
}

template <typename WT, bool W>
__global__ void __launch_bounds__(256) k_hub_insert(DecideArgs<WT> a, HubPlan p, const uint8_t *__restrict__ flag)
{
    hub_insert<WT, W>(a, p, flag, blockIdx.x, gridDim.x);
}

template <typename WT>
__global__ void __launch_bounds__(256) k_hub_scan(DecideArgs<WT> a, HubPlan p, const uint8_t *__restrict__ flag)
{
    hub_scan<WT, 256>(a, p, flag, blockIdx.x, gridDim.x);
}

template <typename WT>
__global__ void __launch_bounds__(256) k_hub_final(DecideArgs<WT> a, HubPlan p, const uint8_t *__restrict__ flag)
{
    hub_final(a, p, flag, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5);
}

// First sweep of a level, distinct neighbours: a hub's entries are its
// candidates, so its row's chunks are evaluated as they are, without the table
// (its clearing, the label gather, the atomic inserts and a scan over at least
// 1.5 slots per entry).  Partials as hub_scan's, at the first table chunks of
// the hub; 2^22 R-MAT vertices 17.79 ms with the tables, 16.99 without, 2^20 from
// the host 7.54 and 7.31.
template <typename WT, bool W>
__global__ void __launch_bounds__(256) k_hub_first(DecideArgs<WT> a, HubPlan p, const uint8_t *__restrict__ flag)
{
    constexpr int NW = 256 / 32;
    __shared__ double r_dq[NW];
    __shared__ int r_c[NW];
    __shared__ CandRow<WT, NW> r_best;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (long long wi = blockIdx.x; wi < p.nwork; wi += gridDim.x) {
        const int i = p.work[wi];
        const int v = p.hubs[i];
        if (!flag[v] || stopped(a, v)) continue;  // block-uniform
        const Scale sc = scale_of(a, v);
        const int cur = a.comm[v];  // = v
        const WT ki = a.K[v], tcur = a.Tot[cur];
        const long long chunk = wi - p.coff[i], s = a.offs[v] + chunk * kHubChunk, left = a.offs[v + 1] - s;
        const int len = (int)(left < kHubChunk ? left : kHubChunk);
        const long long out = p.tcoff[i] + chunk;
        const GainTerms<WT> gt(sc, ki, tcur);
        Cand<WT> best(cur);
        WT wc = 0;
        first_scan_best<WT, W>(a, gt, s, len, v, threadIdx.x, 256, best, wc);
        warp_merge(best, wc, 32);
        if (lane == 0) r_best.put(wid, best, wc);
        __syncthreads();
        if (wid == 0) {
            r_best.get(lane, NW, cur, best, wc);
            warp_merge(best, wc, 32);
            if (lane == 0) {
                hub_put(p, out, best, wc);
                r_best.put(0, best, wc);
            }
        }
        __syncthreads();
        if (needs_fp64(a, sc, ki)) {  // block-uniform
            double dq = 0.0;
            int fc = cur;
            r_best.get(0, 1, cur, best, wc);
            first_scan<WT, W>(a, sc, gt, best, s, len, v, threadIdx.x, 256, ki, tcur, dq, fc);
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
                    p.pdq[out] = dq;
                    p.pfc[out] = fc;
                }
            }
            __syncthreads();
        }
    }
}

// One warp per hub over its chunks' partials, then over the row itself for the
// rare rounding cases.
template <typename WT, bool W>
__global__ void __launch_bounds__(256) k_hub_first_final(DecideArgs<WT> a, HubPlan p, const uint8_t *__restrict__ flag)
{
    hub_final(
        a, p, flag, (blockIdx.x * blockDim.x + threadIdx.x) >> 5, (gridDim.x * blockDim.x) >> 5,
        [&](int i) { return p.tcoff[i] + p.coff[i + 1] - p.coff[i]; },
        [&](int, int v, const Scale &sc, const GainTerms<WT> &gt, const Cand<WT> &best, int, WT ki, WT tcur, double &dq,
            int &fc) {
            first_scan<WT, W>(a, sc, gt, best, a.offs[v], (int)(a.offs[v + 1] - a.offs[v]), v, threadIdx.x & 31, 32, ki,
                              tcur, dq, fc);
        });
}

// Per level: table sizes, chunk counts and their offsets (the caller reads
// the three totals from the stats block before p1_hub_work_launch).
void p1_hub_plan_launch(const LevelGraph &g, Phase1Buffers &b, HubPlan &p, cudaStream_t st)
{
    const int grid = (p.H + 255) / 256;
    k_hub_plan<<<grid, 256, 0, st>>>(p, g.offs);
    exclusive_scan(p.T, p.toff, p.H, OpIdentity(), b.scan_partial, &b.stats->total, st, &b.stats->err);
    exclusive_scan(p.chunks, p.coff, p.H, OpIdentity(), b.scan_partial, &b.stats->total2, st, &b.stats->err);
    exclusive_scan(p.tchunks, p.tcoff, p.H, OpIdentity(), b.scan_partial, &b.stats->total3, st, &b.stats->err);
    k_hub_tail<<<1, 1, 0, st>>>(p, b.stats);
    note_launch(2);
}

void p1_hub_work_launch(HubPlan &p, cudaStream_t st)
{
    k_hub_work<<<(p.H * 32 + 255) / 256, 256, 0, st>>>(p);
    note_launch(1);
}

template <typename WT>
static void hub_decide_t(const LevelGraph &g, Phase1Buffers &b, const HubPlan &p, double constant, long long m2,
                         int fp64_only, bool first, cudaStream_t st)
{
    const DecideArgs<WT> a = decide_args<WT>(g, b, constant, m2, fp64_only);
    const int cap = num_sms() * 8;
    // (a capped table may hold fewer partials than the row has chunks, and its
    // overflow is to be seen)
    if (first && p.t_cap == 0) {
        const int grid = (int)(p.nwork < cap ? p.nwork : cap), gf = (p.H * 32 + 255) / 256;
        if (g.w) {
            k_hub_first<WT, true><<<grid, 256, 0, st>>>(a, p, b.act_flag);
            k_hub_first_final<WT, true><<<gf, 256, 0, st>>>(a, p, b.act_flag);
        } else {
            k_hub_first<WT, false><<<grid, 256, 0, st>>>(a, p, b.act_flag);
            k_hub_first_final<WT, false><<<gf, 256, 0, st>>>(a, p, b.act_flag);
        }
        note_launch(2);
        return;
    }
    cudaMemsetAsync(p.pool, 0xff, (size_t)p.half * sizeof(int32_t), st);
    cudaMemsetAsync(p.pool + p.half, 0, (size_t)p.half * sizeof(WT), st);
    const int g1 = (int)(p.nwork < cap ? p.nwork : cap);
    if (g.w)
        k_hub_insert<WT, true><<<g1, 256, 0, st>>>(a, p, b.act_flag);
    else
        k_hub_insert<WT, false><<<g1, 256, 0, st>>>(a, p, b.act_flag);
    k_hub_scan<WT><<<(int)(p.ntwork < cap ? p.ntwork : cap), 256, 0, st>>>(a, p, b.act_flag);
    k_hub_final<WT><<<(p.H * 32 + 255) / 256, 256, 0, st>>>(a, p, b.act_flag);
    note_launch(3);
}

// One iteration's decide-and-move of the hub bin.  The values of the hub
// tables follow all keys: p.half int32 keys, then p.half values of the
// weight type (the caller sized the pool for it).
void p1_hub_decide(const LevelGraph &g, Phase1Buffers &b, const HubPlan &p, double constant, long long m2,
                   int fp64_only, bool first, cudaStream_t st)
{
    if (p.H <= 0) return;
    if (g.wide)
        hub_decide_t<long long>(g, b, p, constant, m2, fp64_only, first, st);
    else
        hub_decide_t<int>(g, b, p, constant, m2, fp64_only, first, st);
}

template <typename WT>
__global__ void k_hub_in_zero(HubPlan p, WT *In, const DevStats *st)
{
    if (st->push_mode) return;  // the incremental update runs instead
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < p.H; i += gridDim.x * blockDim.x) In[p.hubs[i]] = 0;
}

template <typename WT, bool W>
__global__ void __launch_bounds__(256) k_hub_in_partial(UpdateArgs<WT> a, HubPlan p)
{
    if (a.st->push_mode) return;  // the incremental update runs instead
    hub_in_partial<WT, W>(a, p, blockIdx.x, gridDim.x);
}

template <typename WT>
__global__ void __launch_bounds__(256) k_hub_in_final(UpdateArgs<WT> a, HubPlan p)
{
    if (a.st->push_mode) return;  // the incremental update runs instead
    UpdateSums sums;
    hub_in_final(a, p, a.st->min_tot, blockIdx.x, gridDim.x, sums);
    add_update_sums(a, sums);
}

template <typename WT>
static void hub_update_t(const LevelGraph &g, Phase1Buffers &b, const HubPlan &p, int next, int bin_start,
                         double constant, long long m2, cudaStream_t st)
{
    UpdateArgs<WT> a = update_args<WT>(g, b, 7, next, bin_start, constant, m2);
    const int cap = num_sms() * 8;
    const int hg = (p.H + 255) / 256;
    k_hub_in_zero<WT><<<hg, 256, 0, st>>>(p, a.In, b.stats);
    const int g1 = (int)(p.nwork < cap ? p.nwork : cap);
    if (g.w)
        k_hub_in_partial<WT, true><<<g1, 256, 0, st>>>(a, p);
    else
        k_hub_in_partial<WT, false><<<g1, 256, 0, st>>>(a, p);
    k_hub_in_final<WT><<<hg, 256, 0, st>>>(a, p);
    note_launch(3);
}

void p1_hub_update(const LevelGraph &g, Phase1Buffers &b, const HubPlan &p, int next, int bin_start, double constant,
                   long long m2, cudaStream_t st)
{
    if (p.H <= 0) return;
    if (g.wide)
        hub_update_t<long long>(g, b, p, next, bin_start, constant, m2, st);
    else
        hub_update_t<int>(g, b, p, next, bin_start, constant, m2, st);
}

}  // namespace gala
