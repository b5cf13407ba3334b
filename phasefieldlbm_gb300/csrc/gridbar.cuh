// gridbar.cuh - bounded grid-wide barrier of cooperative launches.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

namespace pflbm {

// Self-resetting: the last CTA to arrive clears the count and advances the
// generation.
struct GridBar {
    unsigned int count;
    unsigned int gen;
    unsigned int never;  // the test build's flag that nothing sets
    unsigned int pad;
};

// Bounded polls of the grid barrier, each a sleep of 64 ns and a load from L2:
// a few seconds in all, far above the difference between the CTAs of any sweep.
constexpr uint32_t kGridWaitLimit = 1u << 22;

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int *p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Grid-wide barrier of a cooperative launch, every poll bounded: on a
// timeout the CTA sets bit 2 of the error word and gets false (the caller
// returns; CTAs still waiting on it time out the same way). Thread 0 makes
// the CTA's writes visible (fence after the block barrier) before arriving.
// The test build -DPFLBM_TEST_DEAD_GRID waits instead on a flag that
// nothing sets, with a short limit.
__device__ __forceinline__ bool grid_barrier(GridBar *gb, unsigned int nblocks, unsigned int *err, int *s_ok) {
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0) {
        bool ok = true;
        const unsigned int g0 = ld_acquire_gpu(&gb->gen);
        __threadfence();
        const unsigned int arrived = atomicAdd(&gb->count, 1u) + 1u;
#ifdef PFLBM_TEST_DEAD_GRID
        (void)arrived;
        (void)nblocks;
        (void)g0;
        ok = false;
        for (uint32_t i = 0; i < (1u << 12); ++i)
            if (ld_acquire_gpu(&gb->never) != 0u) {
                ok = true;
                break;
            }
        if (!ok) atomicOr(err, 2u);
#else
        if (arrived == nblocks) {
            atomicExch(&gb->count, 0u);
            __threadfence();
            atomicAdd(&gb->gen, 1u);
        } else {
            ok = false;
            for (uint32_t i = 0; i < kGridWaitLimit; ++i) {
                if (ld_acquire_gpu(&gb->gen) != g0) {
                    ok = true;
                    break;
                }
                __nanosleep(64);
            }
            if (!ok) atomicOr(err, 2u);
        }
#endif
        __threadfence();
        *s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return *s_ok != 0;
}

// The same for short phases, where the barrier is most of the time: barrier
// `k` of a launch whose count `arrived` is 0 when it starts. The count only
// grows, so a CTA makes one release and then polls for the k+1-th full round;
// nothing is reset and no generation is read or advanced (about 7000 -> 2800
// cycles for 128 CTAs). In two halves, between which a CTA can do what nobody
// waits for. Up to 2^31 arrivals in a launch; every poll bounded as above.
__device__ __forceinline__ void grid_arrive(unsigned int *arrived) {
    __syncthreads();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(arrived) : "memory");
}

__device__ __forceinline__ bool grid_wait(unsigned int *arrived, unsigned int nblocks, unsigned int k,
                                          unsigned int *err, int *s_ok) {
    if (threadIdx.x == 0) {
        bool ok = false;
#ifndef PFLBM_TEST_DEAD_GRID
        const unsigned int goal = (k + 1u) * nblocks;
        for (uint32_t i = 0; i < kGridWaitLimit; ++i) {
            if (int(ld_acquire_gpu(arrived) - goal) >= 0) {
                ok = true;
                break;
            }
            if (i >= 64) __nanosleep(64);
        }
#endif
        if (!ok) atomicOr(err, 2u);
        *s_ok = ok ? 1 : 0;
    }
    __syncthreads();
    return *s_ok != 0;
}

}  // namespace pflbm
