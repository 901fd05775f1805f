// coop.cuh - pieces shared by the kernels that run a whole small level in one
// cooperative launch (small_level.cu, small_contract.cu).
#pragma once
#include <algorithm>

#include "common.cuh"

namespace gala {

constexpr int kSmallBlock = 512;
constexpr int kSmallWarps = kSmallBlock / 32;
constexpr int kSmallMaxGrid = 1024;

// Shared-memory table: the warps' tables (one each) together are the CTA's
// table (rows up to half of it), 53-74 KB, so that two CTAs fit an SM.
template <typename WT>
struct SmallTable {
    static constexpr int kWarpSlots = WideOf<WT>::exact ? 512 : 256;
    static constexpr int kSlots = kWarpSlots * kSmallWarps;
    static constexpr size_t kBytes = (size_t)kSlots * (sizeof(int) + sizeof(WT)) + kSlots / 2 * sizeof(unsigned short);
};

// Blocks of a cooperative kernel that the current device holds at once, at most
// `cap`; smem: its dynamic shared memory, opted in here.  0: it cannot run.
template <typename K>
int coop_grid(K kernel, int threads, size_t smem, int cap)
{
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (smem > 0) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
    return std::min(sms * per_sm, cap);
}

// Cooperative launch of at most `grid` blocks.  A stream may hold fewer than its
// device (a green context's stream has part of the SMs): the grid is halved
// until it is accepted, and every grid gives the same results.
inline cudaError_t coop_launch(const void *kernel, long long grid, int threads, void **args, size_t smem,
                               cudaStream_t st)
{
    for (;;) {
        const cudaError_t e =
            cudaLaunchCooperativeKernel(kernel, dim3((unsigned)grid), dim3((unsigned)threads), args, smem, st);
        if (e != cudaErrorCooperativeLaunchTooLarge || grid <= 1) return e;
        cudaGetLastError();
        grid = (grid + 1) / 2;
    }
}

struct GridBarrier {
    unsigned arrive;  // arrivals since the launch
    int dead;         // a wait gave up: every CTA leaves
};

// Grid barrier (the launch is cooperative: all CTAs are resident).  False when
// the wait gave up after `polls` looks (kBarrierPolls: a few seconds), for every
// thread of the block, which then leaves the kernel; *err gets kErrBarrier, which
// the host reads after the launch.  A block passes only when all have arrived,
// so what it reads behind the barrier is whole even while others give up, and
// none passes the next one.  The block's writes are released with its
// arrival, the others' acquired by one fence after the last poll (the polls
// are relaxed: an acquire per poll invalidates the L1 each time).
__device__ __forceinline__ bool grid_sync(GridBarrier *c, unsigned &target, int *err, unsigned polls)
{
    __shared__ int s_ok;
    __syncthreads();
    if (gridDim.x == 1) return true;  // one CTA: its L1 stays warm
    if (threadIdx.x == 0) {
        target += gridDim.x;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&c->arrive) : "memory");
        int ok = 1;
        for (unsigned spin = 1;; ++spin) {
            unsigned v;
            asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&c->arrive) : "memory");
            if ((int)(v - target) >= 0) break;
            if (spin >= polls || ((spin & 63) == 0 && *(volatile int *)&c->dead)) {
                atomicExch(&c->dead, 1);
                atomicOr(err, kErrBarrier);
                ok = 0;
                break;
            }
        }
        asm volatile("fence.acq_rel.gpu;" ::: "memory");
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

}  // namespace gala
