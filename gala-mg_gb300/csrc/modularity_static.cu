// modularity_static.cu - modularity of a partition on the device without any
// device allocation.
//
// Some callers of this library cannot call cudaMalloc: a host application
// that hands all device memory to its own pool allocator, or a latency-bound
// path where an allocation (and the synchronisation cudaMalloc/cudaFree can
// cause) is not allowed.  gala_modularity_device_static serves them: the
// caller passes the CSR and the labels (device) and gets Q back, and the
// scratch the computation needs - the total weight of every community and
// four sums - lives in the file-scope arrays below, sized for at most
// kStaticMaxVertices vertices.  Every GPU that loads this library holds that
// memory (8 MB + 40 B) until the process exits.
//
// The computation is the one phase 1 uses for Q: sum of In over vertices and
// total weight m2 as exact 64-bit integers, sum of Tot^2 over communities as
// an exact 128-bit integer (Tot^2 alone passes 2^64 once m2 > 2^32), then Q by
// one FP64 expression.
#include <stdio.h>
#include <string.h>

#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace gala {

constexpr int kStaticMaxVertices = 1 << 20;
constexpr int kStaticMaxDevices = 64;

// Scratch shared by every call on a device: community totals and the sums.
static __device__ __align__(256) unsigned long long g_static_tot[kStaticMaxVertices];
// sum In, sum K, sum Tot^2 (low word), sum Tot^2 (high word), and the error
// bits (bit 0: a label lies outside [0, n); bit 1: a weight is not positive):
// one copy brings all five back
static __device__ __align__(256) unsigned long long g_static_sums[5];

// Device addresses of the two arrays, looked up once per device (in host
// code the symbols are host-side stand-ins, not device addresses).
static unsigned long long *g_tot_ptr[kStaticMaxDevices];
static unsigned long long *g_sums_ptr[kStaticMaxDevices];
static std::mutex g_static_mu;

__global__ void k_static_zero(unsigned long long *tot, int n, unsigned long long *sums)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) tot[i] = 0ull;
    if (blockIdx.x == 0 && threadIdx.x < 5) sums[threadIdx.x] = 0ull;
}

// Weight (W) and own-community weight of the row entries first, first + step,
// ... < deg, U of them in flight.
template <bool W, int U = 4>
__device__ __forceinline__ void static_row(const int32_t *__restrict__ nbr, const int32_t *__restrict__ w,
                                           const int32_t *__restrict__ comm, int n, int c, long long first,
                                           long long deg, int step, unsigned long long &k, unsigned long long &in,
                                           int &bad)
{
    // predicated batches: a short row's loads are in flight together too
    for (; first < deg; first += (long long)U * step) {
        int u[U], wi[U];
#pragma unroll
        for (int q = 0; q < U; ++q) {
            const long long j = first + q * step;
            u[q] = j < deg ? nbr[j] : -1;
            if (W) {
                wi[q] = j < deg ? w[j] : 0;
                if (j < deg && wi[q] <= 0) bad |= 2;
            }
        }
#pragma unroll
        for (int q = 0; q < U; ++q) u[q] = (unsigned)u[q] < (unsigned)n ? comm[u[q]] : ~c;
#pragma unroll
        for (int q = 0; q < U; ++q) {
            if (W) {
                const unsigned long long wt = wi[q] > 0 ? (unsigned long long)wi[q] : 0ull;
                k += wt;
                if (u[q] == c) in += wt;
            } else {
                in += u[q] == c;
            }
        }
    }
}

// K (row weight) and In (weight to the own community) of every vertex;
// community totals by atomics, sums by warp then block reduction.  A group of
// G lanes takes a row, four loads in flight per lane and 32 / G rows per warp;
// rows longer than kStaticLong entries go to the whole warp afterwards, and
// those longer than kStaticBlock (as many as the list holds) to the whole block
// at its end.  One wave of blocks.  300k vertices, 7.2M entries: 59 us with a
// warp per row, 42 us with G = 8, where the label gathers (one 32-byte L2 sector
// each, about 6 TB/s of sectors) bound it: neither more warps nor more loads in
// flight change it.  Few vertices do not fill the chip at G = 8, and long rows
// among them then queue in few warps: a warp per row while that is one wave,
// half a warp up to two (calls of 300 rows of 20,000 entries 74 us with a warp
// per row, 174 at G = 8, 61 so; 1,200 of 5,000: 48 / 76 / 46; 20,000 of 2,000:
// 96 / 98 / 98).  A star of 2^20 vertices: 2.3 ms with its hub's row in one warp,
// 0.31 in a block; 160 rows of 30,000 entries on neighbouring ids among 500,000
// vertices: 0.57 ms with a block's warps on consecutive rows, 0.13 on rows that
// lie a grid apart; 50 rows of 3,800 on neighbouring ids among 42,000: 71 us with a
// warp per row, 95 with four to a warp, 37 by the block.
constexpr int kStaticLong = 512;
constexpr int kStaticBlock = 1024;
constexpr int kStaticList = 16;
template <int G, bool W>
__global__ void __launch_bounds__(256, W ? 5 : 6) k_static_rows(int n, const int64_t *__restrict__ offs,
                                                        const int32_t *__restrict__ nbr,
                                                        const int32_t *__restrict__ w,
                                                        const int32_t *__restrict__ comm, unsigned long long *tot,
                                                        unsigned long long *sums)
{
    __shared__ unsigned long long s_in[8], s_k[8];
    __shared__ int s_rows[kStaticList], s_nrows;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_nrows = 0;
    __syncthreads();
    const int sub = lane & (G - 1), gw = lane / G;
    constexpr int GPW = 32 / G;
    // (consecutive warps' rows in different blocks: long rows often have
    // neighbouring ids)
    const int wg = wid * gridDim.x + blockIdx.x;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    unsigned long long my_in = 0, my_k = 0;
    int bad = 0;
    for (long long v0 = (long long)wg * GPW; v0 < n; v0 += (long long)nw * GPW) {
        const bool has = v0 + gw < n;
        const int v = has ? (int)(v0 + gw) : n - 1;
        const int c = comm[v];
        const long long s = offs[v], deg = has ? offs[v + 1] - s : 0;
        const bool is_long = deg > kStaticLong;
        unsigned long long k = 0, in = 0;
        bool skip = false;
        if (!is_long) static_row<W>(nbr + s, W ? w + s : nullptr, comm, n, c, sub, deg, G, k, in, bad);
        unsigned todo = __ballot_sync(GALA_FULL_MASK, is_long && sub == 0);
        while (todo) {  // warp-uniform
            const int src = __ffs((int)todo) - 1;
            todo &= todo - 1;
            const long long ls = __shfl_sync(GALA_FULL_MASK, s, src), ld = __shfl_sync(GALA_FULL_MASK, deg, src);
            const int lc = __shfl_sync(GALA_FULL_MASK, c, src);
            if (ld > kStaticBlock) {
                int at = 0;
                if (lane == 0) at = atomicAdd(&s_nrows, 1);
                at = __shfl_sync(GALA_FULL_MASK, at, 0);
                if (at < kStaticList) {
                    if (lane == src) {
                        s_rows[at] = v;
                        skip = true;
                    }
                    continue;
                }
            }
            unsigned long long lk = 0, lin = 0;
            static_row<W, W ? 4 : 8>(nbr + ls, W ? w + ls : nullptr, comm, n, lc, lane, ld, 32, lk, lin, bad);
            if (W) lk = warp_sum(lk);
            lin = warp_sum(lin);
            if (lane == src) {
                k = lk;
                in = lin;
            }
        }
#pragma unroll
        for (int o = G / 2; o >= 1; o >>= 1) {
            if (W) k += __shfl_xor_sync(GALA_FULL_MASK, k, o);
            in += __shfl_xor_sync(GALA_FULL_MASK, in, o);
        }
        if (has && sub == 0 && !skip) {
            if (!W) k = (unsigned long long)deg;
            if ((unsigned)c < (unsigned)n)
                atomicAdd(&tot[c], k);
            else
                bad |= 1;
            my_in += in;
            my_k += k;
        }
    }
    __syncthreads();
    for (int i = 0; i < min(s_nrows, kStaticList); ++i) {
        const int v = s_rows[i], c = comm[v];
        const long long s = offs[v], deg = offs[v + 1] - s;
        unsigned long long k = 0, in = 0;
        static_row<W, 8>(nbr + s, W ? w + s : nullptr, comm, n, c, threadIdx.x, deg, 256, k, in, bad);
        if (!W) k = threadIdx.x == 0 ? (unsigned long long)deg : 0;
        k = warp_sum(k);
        if (lane == 0 && k) {
            if ((unsigned)c < (unsigned)n)
                atomicAdd(&tot[c], k);
            else
                bad |= 1;
            my_k += k;
        }
        my_in += in;
    }
    if (bad) atomicOr(&sums[4], (unsigned long long)bad);
    my_in = warp_sum(my_in);
    my_k = warp_sum(my_k);
    if (lane == 0) {
        s_in[wid] = my_in;
        s_k[wid] = my_k;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long a = 0, b = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
            a += s_in[q];
            b += s_k[q];
        }
        if (a) atomicAdd(&sums[0], a);
        if (b) atomicAdd(&sums[1], b);
    }
}

// Sum of Tot^2 over communities, exact in 128 bits: Tot < 2^64, so a square
// needs up to 128 bits; each block adds its sum to the (lo, hi) pair, the
// carry taken from the low word's atomic result (order independent).
__global__ void __launch_bounds__(256) k_static_tot2(int n, const unsigned long long *__restrict__ tot,
                                                     unsigned long long *sums)
{
    __shared__ unsigned long long rlo[8], rhi[8];
    unsigned __int128 s = 0;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x)
        s += (unsigned __int128)tot[c] * tot[c];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        const unsigned long long l = __shfl_xor_sync(GALA_FULL_MASK, (unsigned long long)s, o);
        const unsigned long long h = __shfl_xor_sync(GALA_FULL_MASK, (unsigned long long)(s >> 64), o);
        s += ((unsigned __int128)h << 64) | l;
    }
    if ((threadIdx.x & 31) == 0) {
        rlo[threadIdx.x >> 5] = (unsigned long long)s;
        rhi[threadIdx.x >> 5] = (unsigned long long)(s >> 64);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned __int128 t = 0;
        for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += ((unsigned __int128)rhi[q] << 64) | rlo[q];
        const unsigned long long l = (unsigned long long)t;
        unsigned long long h = (unsigned long long)(t >> 64);
        if (l) {
            const unsigned long long old = atomicAdd(&sums[2], l);
            if (old + l < old) h += 1;
        }
        if (h) atomicAdd(&sums[3], h);
    }
}

}  // namespace gala

using namespace gala;

extern "C" gala_status gala_modularity_device_static(int32_t n, const int64_t *d_offsets, const int32_t *d_neighbors,
                                                     const int32_t *d_weights, const int32_t *d_community,
                                                     double *modularity)
{
    clear_error();
    if (n <= 0 || !d_offsets || !d_neighbors || !d_community || !modularity) {
        set_error("gala_modularity_device_static: bad arguments");
        return GALA_ERR_INVALID;
    }
    if (n > kStaticMaxVertices) {
        set_error("gala_modularity_device_static: %d vertices exceed the static maximum of %d", n,
                  kStaticMaxVertices);
        return GALA_ERR_CAPACITY;
    }
    int dev = 0;
    cudaError_t ce = cudaGetDevice(&dev);
    if (ce != cudaSuccess) return cuda_fail(ce, "gala_modularity_device_static: no device");
    if (dev < 0 || dev >= kStaticMaxDevices) {
        set_error("gala_modularity_device_static: device %d out of range", dev);
        return GALA_ERR_INVALID;
    }
    unsigned long long *tot = nullptr, *sums = nullptr;
    {
        // first call on this device (with it current): look up the device
        // addresses of the static arrays
        std::lock_guard<std::mutex> lock(g_static_mu);
        if (!g_tot_ptr[dev]) {
            void *p = nullptr, *q = nullptr;
            if ((ce = cudaGetSymbolAddress(&p, g_static_tot)) != cudaSuccess ||
                (ce = cudaGetSymbolAddress(&q, g_static_sums)) != cudaSuccess)
                return cuda_fail(ce, "gala_modularity_device_static: symbol address");
            g_sums_ptr[dev] = (unsigned long long *)q;
            g_tot_ptr[dev] = (unsigned long long *)p;
        }
        tot = g_tot_ptr[dev];
        sums = g_sums_ptr[dev];
    }
    // the scratch keeps the previous call's contents: clear it first
    const int grid = (n + 255) / 256 < 1024 ? (n + 255) / 256 : 1024;
    k_static_zero<<<grid, 256>>>(tot, n, sums);
    const long long wave = (long long)hub_grid_size() * (d_weights ? 5 : 6);
    auto rows = [&](auto lanes) {
        constexpr int G = decltype(lanes)::value;
        const long long blocks = ((long long)n * G + 255) / 256;
        const int rgrid = (int)(blocks < wave ? blocks : wave);
        if (d_weights)
            k_static_rows<G, true><<<rgrid, 256>>>(n, d_offsets, d_neighbors, d_weights, d_community, tot, sums);
        else
            k_static_rows<G, false><<<rgrid, 256>>>(n, d_offsets, d_neighbors, nullptr, d_community, tot, sums);
    };
    // (lanes per row: see k_static_rows)
    if ((long long)n * 32 <= wave * 256)
        rows(std::integral_constant<int, 32>());
    else if ((long long)n * 16 <= wave * 256 * 2)
        rows(std::integral_constant<int, 16>());
    else
        rows(std::integral_constant<int, 8>());
    k_static_tot2<<<grid, 256>>>(n, tot, sums);
    note_launch(3);
    // a launch that failed for its configuration would leave the previous
    // call's sums in the scratch: report it instead of reading them
    if ((ce = cudaGetLastError()) != cudaSuccess) return cuda_fail(ce, "gala_modularity_device_static: launch");
    unsigned long long h[5] = {0, 0, 0, 0, 0};
    if ((ce = cudaMemcpy(h, sums, sizeof(h), cudaMemcpyDeviceToHost)) != cudaSuccess)
        return cuda_fail(ce, "gala_modularity_device_static");
    const int hbad = (int)h[4];
    if (hbad & 1) {
        set_error("gala_modularity_device_static: a community label lies outside [0, %d)", n);
        return GALA_ERR_INVALID;
    }
    if (hbad & 2) {
        set_error("gala_modularity_device_static: a weight is not positive");
        return GALA_ERR_INVALID;
    }
    if (h[1] == 0) {
        set_error("gala_modularity_device_static: graph has no edges");
        return GALA_ERR_INVALID;
    }
    // Q = sum In / m2 - sum Tot^2 / m2^2, the 128-bit sum converted as
    // hi * 2^64 + lo (the engine's expression)
    const double c = 1.0 / (double)h[1];
    const double t2 = (double)h[3] * 18446744073709551616.0 + (double)h[2];
    *modularity = (double)h[0] * c - t2 * c * c;
    return GALA_OK;
}
