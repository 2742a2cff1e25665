// qew_gridsync.cuh -- bounded grid barrier for cooperative persistent kernels.
//
// Thread 0 of each CTA arrives on a counter that only grows, with release
// order, and polls it with acquire order until every CTA has arrived: a
// barrier is one round trip to L2 behind the last arrival (a counter that the
// last arrival resets and a generation word that it bumps cost two more). The
// polls are bounded in number. A wait that gives up sets `err` (every other
// CTA then stops waiting too) and the barrier returns false, so a kernel can
// leave its loop and the host can report QEW_ERR_TIMEOUT instead of hanging.
// Only use it in kernels launched with cudaLaunchCooperativeKernel, which
// guarantees that every CTA is resident.
#pragma once

#include "qew_internal.cuh"

constexpr long long kGridBarrierPolls = 1LL << 26;  // some 20 s of round trips to L2

struct GridSync {
    unsigned int count;   // arrivals so far (wraps)
    unsigned int pad;
    int err;              // set when a wait gave up
    int skip_block;       // a CTA that never arrives (a test's injected fault), -1: none
    long long max_polls;  // polls before a wait gives up
};

// Fresh barrier state for one launch, with the context's limits.
static __global__ void k_gridsync_init(GridSync *s, long long max_polls, int skip_block) {
    s->count = 0;
    s->pad = 0;
    s->err = 0;
    s->skip_block = skip_block;
    s->max_polls = max_polls;
}
static inline qew_status qew_gridsync_init(qew_ctx *ctx, GridSync *s) {
    k_gridsync_init<<<1, 1, 0, ctx->stream>>>(s, ctx->barrier_polls, ctx->barrier_skip);
    return qew_launch_check(ctx, "gridsync_init");
}

// `arrivals`: this thread's count of the grid's arrivals, 0 before its first
// barrier; the same in every thread.
__device__ __forceinline__ bool grid_sync_bounded(GridSync *s, unsigned int nblocks,
                                                  unsigned int &arrivals) {
    __syncthreads();
    __shared__ int s_ok;
    arrivals += nblocks;
    if (threadIdx.x == 0) {
        if ((int)blockIdx.x == s->skip_block) {
            s_ok = 0;  // leaves without arriving: the other CTAs' waits run out
        } else {
            const long long limit = s->max_polls;
            __threadfence();
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&s->count) : "memory");
            long long polls = 0;
            int ok = 1;
            for (;;) {
                unsigned int c;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];"
                             : "=r"(c)
                             : "l"(&s->count)
                             : "memory");
                if ((int)(c - arrivals) >= 0) break;
                if ((polls & 15) == 15 && *(volatile int *)&s->err) {
                    ok = 0;
                    break;
                }
                if (++polls > limit) {
                    atomicExch(&s->err, 1);
                    ok = 0;
                    break;
                }
                __nanosleep(20);
            }
            __threadfence();
            s_ok = ok;
        }
    }
    __syncthreads();
    return s_ok != 0;
}
