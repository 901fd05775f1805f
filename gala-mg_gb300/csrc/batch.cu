// batch.cu - per-graph reductions of a batch of graphs run as one union
// graph (block-diagonal CSR).  Batching has no counterpart in the reference;
// every graph follows the reference's single-graph rules with its own m2,
// min Tot, modularity and convergence.
//
// The vertices of graph g occupy the contiguous id range [goff[g], goff[g+1])
// at every level: contraction renumbers communities by ascending old id and a
// community never spans two graphs, so the ranges stay contiguous.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace gala {

namespace {

__device__ __forceinline__ unsigned long long block_sum_u64(unsigned long long v, unsigned long long *red)
{
    v = warp_sum(v);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    unsigned long long t = 0;
    if (wid == 0) {
        t = lane < (int)(blockDim.x >> 5) ? red[lane] : 0ull;
        t = warp_sum(t);
    }
    return t;  // valid in thread 0
}

__device__ __forceinline__ int block_min_i32(int v, int *red)
{
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v = min(v, __shfl_xor_sync(GALA_FULL_MASK, v, o));
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    int t = 0x7fffffff;
    if (wid == 0) {
        t = lane < (int)(blockDim.x >> 5) ? red[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) t = min(t, __shfl_xor_sync(GALA_FULL_MASK, t, o));
    }
    return t;
}

// S blocks per graph, each over a slice of its range: the sums `what` asks
// for.  One block per graph writes them (S = 1); several add to values that
// k_graph_sums_zero reset.  Graphs with stop[g] set are left alone (their
// values are final).
__global__ void k_graph_sums_zero(int what, int G, const uint8_t *__restrict__ stop, GraphSums out)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < G; g += gridDim.x * blockDim.x) {
        if (stop && stop[g]) continue;
        if (what & kSumIn) out.sum_in[g] = 0;
        if (what & kSumTot2) out.sum_tot2[g] = 0;
        if (what & kSumK) out.sum_k[g] = 0;
        if (what & kCountComm) out.ncomm[g] = 0;
        if (what & kMinTot) out.min_tot[g] = 0x7fffffff;
    }
}

__device__ __forceinline__ void put_sum(unsigned long long *p, unsigned long long v, bool add)
{
    if (add)
        atomicAdd(p, v);
    else
        *p = v;
}

__global__ void __launch_bounds__(256) k_graph_sums(int what, int G, int S, const int64_t *__restrict__ goff,
                                                    const uint8_t *__restrict__ stop, const int32_t *__restrict__ In,
                                                    const int32_t *__restrict__ Tot, const int32_t *__restrict__ K,
                                                    const int32_t *__restrict__ size, GraphSums out)
{
    __shared__ unsigned long long red[32];
    __shared__ int redi[32];
    const bool add = S > 1;
    for (long long i = blockIdx.x; i < (long long)G * S; i += gridDim.x) {
        const int g = (int)(i / S), slice = (int)(i % S);
        if (stop && stop[g]) continue;
        const long long r0 = goff[g], len = goff[g + 1] - r0;
        const long long v0 = r0 + len * slice / S, v1 = r0 + len * (slice + 1) / S;
        unsigned long long si = 0, st2 = 0, sk = 0, nc = 0;
        int mn = 0x7fffffff;
#pragma unroll 4
        for (long long v = v0 + threadIdx.x; v < v1; v += blockDim.x) {
            if (what & kSumIn) si += (unsigned long long)In[v];
            if (what & (kSumTot2 | kMinTot)) {
                const int t = Tot[v];
                if (t != 0) {
                    st2 += (unsigned long long)((long long)t * t);
                    mn = min(mn, t);
                }
            }
            if (what & kSumK) sk += (unsigned long long)K[v];
            if (what & kCountComm) nc += size[v] > 0;
        }
        if (what & kSumIn) {
            si = block_sum_u64(si, red);
            if (threadIdx.x == 0) put_sum(&out.sum_in[g], si, add);
        }
        if (what & kSumTot2) {
            st2 = block_sum_u64(st2, red);
            if (threadIdx.x == 0) put_sum(&out.sum_tot2[g], st2, add);
        }
        if (what & kSumK) {
            sk = block_sum_u64(sk, red);
            if (threadIdx.x == 0) put_sum(&out.sum_k[g], sk, add);
        }
        if (what & kCountComm) {
            nc = block_sum_u64(nc, red);
            if (threadIdx.x == 0) {
                if (add)
                    atomicAdd(&out.ncomm[g], (int32_t)nc);
                else
                    out.ncomm[g] = (int32_t)nc;
            }
        }
        if (what & kMinTot) {
            mn = block_min_i32(mn, redi);
            if (threadIdx.x == 0) {
                if (add)
                    atomicMin(&out.min_tot[g], mn);
                else
                    out.min_tot[g] = mn;
            }
        }
        __syncthreads();
    }
}

// Convergence of every graph (louvain_main_process.cu:1004-1007): a graph whose
// Q did not grow by min_mod drops this sweep's moves and stops.  Q is the
// host's expression (q_from_sums) in the same order.  The sums of the others go
// back to their starting values.  With the rule on the host a sweep of a batch
// waited for three copies of sums and counters, two of flags and two
// synchronisations (128 graphs, 107 sweeps: 31.95 ms, 30.78 with this).
__global__ void k_batch_converge(int G, GraphSums s, const double *__restrict__ cg, double min_mod, double *prev_q,
                                 uint8_t *stop, uint8_t *reject, DevStats *st)
{
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    bool run = false, rej = false;
    if (g < G) {
        if (!stop[g]) {
            const double c = cg[g], t2 = (double)s.sum_tot2[g];
            const double q =
                __dsub_rn(__dmul_rn((double)(long long)s.sum_in[g], c), __dmul_rn(__dmul_rn(t2, c), c));
            rej = __dsub_rn(q, prev_q[g]) < min_mod;
            run = !rej;
            if (rej)
                stop[g] = 1;
            else
                prev_q[g] = q;
            s.sum_in[g] = 0;
            s.sum_tot2[g] = 0;
            s.min_tot[g] = 0x7fffffff;
        }
        reject[g] = rej;
    }
    const unsigned r = __ballot_sync(GALA_FULL_MASK, run), j = __ballot_sync(GALA_FULL_MASK, rej);
    if ((threadIdx.x & 31) == 0) {
        if (r) atomicAdd(&st->batch_running, __popc(r));
        if (j) atomicAdd(&st->batch_rejects, __popc(j));
    }
}

// Undo this iteration's moves of the graphs flagged in `reject` (their Q
// did not grow by min_mod; louvain_main_process.cu:1004-1007 per graph).
__global__ void k_revert_graphs(const int32_t *__restrict__ mv_v, const int32_t *__restrict__ mv_old,
                                const int32_t *__restrict__ mv_new, const DevStats *__restrict__ stp,
                                const int32_t *__restrict__ gid, const uint8_t *__restrict__ reject, int32_t *comm,
                                int32_t *Tot, int32_t *size, const int32_t *__restrict__ K)
{
    if (stp->batch_rejects == 0) return;
    const int nm = stp->n_movers;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nm; i += gridDim.x * blockDim.x) {
        const int v = mv_v[i];
        if (!reject[gid[v]]) continue;
        const int from = mv_new[i], to = mv_old[i];
        const int k = K[v];
        comm[v] = to;
        atomicAdd(&Tot[to], k);
        atomicSub(&Tot[from], k);
        atomicAdd(&size[to], 1);
        atomicSub(&size[from], 1);
    }
}

__global__ void k_gid_fill(int G, const int64_t *__restrict__ goff, int32_t *gid)
{
    for (int g = blockIdx.x; g < G; g += gridDim.x)
        for (long long v = goff[g] + threadIdx.x; v < goff[g + 1]; v += blockDim.x) gid[v] = g;
}

int sm_count_batch()
{
    static int s = 0;
    if (s == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&s, cudaDevAttrMultiProcessorCount, dev);
        if (s <= 0) s = 148;
    }
    return s;
}

int grid_for(int G) { return G < 65535 ? G : 65535; }

// Graph of union position x: the last g with start[g] <= x.
__device__ __forceinline__ int graph_of(const int64_t *__restrict__ start, int G, long long x)
{
    int lo = 0, hi = G - 1;
    while (lo < hi) {
        const int m = (lo + hi + 1) >> 1;
        if (start[m] <= x)
            lo = m;
        else
            hi = m - 1;
    }
    return lo;
}

// Union CSR of page-locked host graphs, read by the GPU through their
// device-mapped addresses.  A block takes chunks of kGatherChunk union
// entries (or vertices) whatever graphs they lie in, so that one large graph
// does not keep one block busy, with eight loads in flight per thread (host
// memory behind the chip-to-chip link has a long latency).  Ids are shifted
// by their graph's first vertex, offsets by its first entry.
constexpr int kGatherChunk = 8192;
template <typename T, typename Src, typename Put>
__device__ __forceinline__ void gather_chunk(const int64_t *__restrict__ start, int G, long long c0, long long c1,
                                             Src src, Put put)
{
    constexpr int U = 8;
    for (int g = graph_of(start, G, c0); c0 < c1; ++g) {
        const long long b = start[g], e = start[g + 1] < c1 ? start[g + 1] : c1;
        const T *p = src(g);
        for (long long j0 = c0; j0 < e; j0 += (long long)U * blockDim.x) {
            T t[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const long long j = j0 + u * blockDim.x + threadIdx.x;
                t[u] = (j < e && p) ? p[j - b] : (T)1;  // graphs without weights: 1
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const long long j = j0 + u * blockDim.x + threadIdx.x;
                if (j < e) put(g, j, t[u]);
            }
        }
        if (e > c0) c0 = e;
    }
}

__global__ void __launch_bounds__(256) k_batch_gather(int G, BatchSrc s, int64_t *offs, int32_t *nbr, int32_t *w)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) offs[0] = 0;
    const long long n = s.vstart[G], E = s.estart[G];
    const long long ec = (E + kGatherChunk - 1) / kGatherChunk, vc = (n + kGatherChunk - 1) / kGatherChunk;
    const long long all = vc + ec + (w ? ec : 0);
    for (long long c = blockIdx.x; c < all; c += gridDim.x) {
        if (c < vc) {
            const long long c0 = c * kGatherChunk, c1 = c0 + kGatherChunk < n ? c0 + kGatherChunk : n;
            gather_chunk<int64_t>(
                s.vstart, G, c0, c1, [&](int g) { return s.offs[g]; },
                [&](int g, long long v, int64_t x) { offs[v + 1] = s.estart[g] + x; });
            continue;
        }
        const bool wt = c >= vc + ec;
        const long long c0 = (c - vc - (wt ? ec : 0)) * kGatherChunk;
        const long long c1 = c0 + kGatherChunk < E ? c0 + kGatherChunk : E;
        if (wt)
            gather_chunk<int32_t>(
                s.estart, G, c0, c1, [&](int g) { return s.w[g]; },
                [&](int, long long j, int32_t x) { w[j] = x; });
        else
            gather_chunk<int32_t>(
                s.estart, G, c0, c1, [&](int g) { return s.nbr[g]; },
                [&](int g, long long j, int32_t x) { nbr[j] = x + (int32_t)s.vstart[g]; });
    }
}

// In-place shift of a union CSR whose per-graph parts were copied raw:
// graph g's inclusive offsets (at offs[vstart[g]+1 ...]) by its first entry,
// its neighbour ids by its first vertex.
__global__ void __launch_bounds__(256) k_batch_shift(int G, const int64_t *__restrict__ vstart,
                                                     const int64_t *__restrict__ estart, int64_t *offs, int32_t *nbr)
{
    if (blockIdx.x == 0 && threadIdx.x == 0) offs[0] = 0;
    for (int g = blockIdx.x; g < G; g += gridDim.x) {
        const long long v0 = vstart[g], v1 = vstart[g + 1], e0 = estart[g], e1 = estart[g + 1];
        const int32_t shift = (int32_t)v0;
        if (e0 != 0)
            for (long long v = v0 + threadIdx.x; v < v1; v += blockDim.x) offs[v + 1] += e0;
        if (shift != 0)
            for (long long j = e0 + threadIdx.x; j < e1; j += blockDim.x) nbr[j] += shift;
    }
}

// Union community ids -> ids local to each graph (graph g's vertices are
// [vstart[g], vstart[g+1]) of the input; its communities start at goff[g]).
__global__ void k_batch_local_labels(int G, const int64_t *__restrict__ vstart, const int64_t *__restrict__ goff,
                                     int32_t *labels)
{
    for (int g = blockIdx.x; g < G; g += gridDim.x) {
        const int32_t base = (int32_t)goff[g];
        for (long long v = vstart[g] + threadIdx.x; v < vstart[g + 1]; v += blockDim.x) labels[v] -= base;
    }
}

}  // namespace

void batch_gather(int G, const BatchSrc &src, int64_t *offs, int32_t *nbr, int32_t *w, cudaStream_t st)
{
    if (G <= 0) return;
    k_batch_gather<<<sm_count_batch() * 8, 256, 0, st>>>(G, src, offs, nbr, w);
    note_launch(1);
}

void batch_shift(int G, const int64_t *vstart, const int64_t *estart, int64_t *offs, int32_t *nbr, cudaStream_t st)
{
    if (G <= 0) return;
    k_batch_shift<<<grid_for(G), 256, 0, st>>>(G, vstart, estart, offs, nbr);
    note_launch(1);
}

void batch_local_labels(int G, const int64_t *vstart, const int64_t *goff, int32_t *labels, cudaStream_t st)
{
    if (G <= 0) return;
    k_batch_local_labels<<<grid_for(G), 256, 0, st>>>(G, vstart, goff, labels);
    note_launch(1);
}

void batch_sums_reset(int what, int G, const uint8_t *stop, const GraphSums &out, cudaStream_t st)
{
    k_graph_sums_zero<<<(G + 255) / 256, 256, 0, st>>>(what, G, stop, out);
    note_launch(1);
}

void batch_graph_sums(int what, int G, const int64_t *goff, const uint8_t *stop, const Phase1Buffers &b,
                      const GraphSums &out, cudaStream_t st, bool reset)
{
    if (G <= 0) return;
    // few graphs: several blocks each, about eight per SM in all (128 graphs
    // of 2,000-60,000 vertices: 36 us a launch with one block per graph, 6 us
    // with nine, the reset included)
    const int S = std::max(1, std::min(64, sm_count_batch() * 8 / G));
    if (S > 1 && reset) batch_sums_reset(what, G, stop, out, st);
    k_graph_sums<<<grid_for(G * S), 256, 0, st>>>(what, G, S, goff, stop, b.In, b.Tot, b.K, b.size, out);
    note_launch(1);
}

void batch_converge(Phase1Buffers &b, int G, const GraphSums &sums, const double *cg, double min_mod, double *prev_q,
                    uint8_t *stop, uint8_t *reject, const int32_t *gid, int n, cudaStream_t st)
{
    if (G <= 0) return;
    k_batch_converge<<<(G + 255) / 256, 256, 0, st>>>(G, sums, cg, min_mod, prev_q, stop, reject, b.stats);
    note_launch(1);
    int grid = (n + 255) / 256;
    if (grid > 1024) grid = 1024;
    if (grid < 1) grid = 1;
    k_revert_graphs<<<grid, 256, 0, st>>>(b.mv_v, b.mv_old, b.mv_new, b.stats, gid, reject, b.comm, b.Tot, b.size,
                                          b.K);
    note_launch(1);
}

void batch_gid_fill(int G, const int64_t *goff, int32_t *gid, cudaStream_t st)
{
    if (G <= 0) return;
    k_gid_fill<<<grid_for(G), 256, 0, st>>>(G, goff, gid);
    note_launch(1);
}

}  // namespace gala
