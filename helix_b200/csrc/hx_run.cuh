// What the kernels that run whole integrator steps in one launch share
// (small_step_kernel in hx_small.cu, herm_run_kernel in hx_herm_run.cu): the
// barrier over the grid and the reduction of the observables by one warp.
#ifndef HX_RUN_CUH
#define HX_RUN_CUH

#include <cuda_runtime.h>

#include <cstdint>

#include "hx_internal.h"

namespace hx {

// Grid barrier: every CTA is resident (cooperative launch).  One arrival
// counter, zero when a launch begins: barrier k = 1, 2, ... of the launch waits
// until it reaches k G.  The block's writes are ordered before thread 0's
// arrival by the block barrier and a GPU-scope fence; the wait polls the
// counter with acquire loads, bounded.  The launch puts the counter back to
// zero at its end, so no host-side count is involved (a captured launch replays
// correctly).
//
// A barrier is passed by every CTA or by none, so rho ends at the same step in
// all slabs: the CTA that gives up at barrier k replaces the counter by
// kRunAborted + k G, in one exchange that fails when the last arrival comes
// first.  Who arrives later finds the mark and gives up at once, at the same
// barrier; who still polls for an earlier one passes it.  (At most G - 1
// arrivals follow a mark, so k stays readable.)  The mark stays until the host
// has read the error word: launches already enqueued find it at their first
// arrival and leave rho alone.
constexpr unsigned kRunAborted = 1u << 31;

// The counter before this CTA's arrival (thread 0).
__device__ __forceinline__ unsigned grid_arrive(unsigned* count)
{
    __syncthreads();
    if (threadIdx.x != 0) return 0u;
    __threadfence();
    return atomicAdd(count, 1u);
}

// Barrier k (from 1); false when it was given up.
__device__ __forceinline__ bool grid_barrier(unsigned* count, unsigned k, const StepWait& w)
{
    const unsigned all = k * gridDim.x;
    int late = 0;
    // looked at only where a mark is found, so that the polling does not wait for it (0.2 us a barrier: 6 ADOs at d = 32
    // 15.2 us a step, 14.4 so)
    const unsigned before = grid_arrive(count);
    if (threadIdx.x == 0) {
        const unsigned target = all + w.skew;
        for (uint32_t it = 0;; ++it) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
            if (static_cast<int>(v - target) >= 0 && !(v & kRunAborted)) break;
            if (v & kRunAborted) {
                late = (v & ~kRunAborted) < all + gridDim.x || (before & kRunAborted);
                break;
            }
            if (it >= w.max_polls && atomicCAS(count, v, kRunAborted | all) == v) {
                late = 1;
                break;
            }
        }
    }
    return __syncthreads_or(late) == 0;
}

// A barrier that was not passed, after a stage of step `step` (its last one: the step is in rho): the error
// word, and the steps of the launch that rho does not hold.
__device__ __forceinline__ void run_gave_up(int* error_flag, const StepWait& w, int nsteps, int step, bool last_stage)
{
    if (threadIdx.x != 0) return;
    if (blockIdx.x == 0 && w.lost) atomicAdd(w.lost, nsteps - step - (last_stage ? 1 : 0));
    atomicExch(error_flag, 1);
}

// The counter goes back to zero for the next launch: by the watching CTA,
// whose last wait saw every arrival, or by the last CTA to get here once every
// CTA has passed every barrier (one less than the stages of the run).
__device__ __forceinline__ void grid_reset(unsigned* count, bool watch, bool watcher, unsigned stages)
{
    if (watch) {
        if (watcher && threadIdx.x == 0) atomicExch(count, 0u);
    } else if (threadIdx.x == 0 && atomicAdd(count, 1u) == stages * gridDim.x - 1u) {
        atomicExch(count, 0u);
    }
}

// Energy and trace of rho_0 by one warp, in the summation order of
// observables_kernel (hx_stage.cu); at(r, c) returns an element of rho_0 (the
// real part alone counts off the diagonal).
template <int LOGD, typename At>
__device__ __forceinline__ void warp_observables(const double* hdiag, const double* hflip, At at, double* out)
{
    constexpr int D = 1 << LOGD;
    const int lane = threadIdx.x & 31;
    double sum[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int r0 = 0; r0 < D; r0 += 32) {  // 32 rows at a time, as the warps of that kernel
        const int r = r0 + lane;
        double en = 0.0, tr = 0.0, ti = 0.0;
        if (r < D) {
            const double2 dg = at(r, r);
            en = fma(__ldg(hdiag + r), dg.x, en);
            tr += dg.x;
            ti += dg.y;
#pragma unroll
            for (int i = 0; i < LOGD; ++i) en = fma(__ldg(hflip + i), at(r ^ (1 << i), r).x, en);
        }
        for (int off = 16; off > 0; off >>= 1) {
            en += __shfl_down_sync(0xffffffffu, en, off);
            tr += __shfl_down_sync(0xffffffffu, tr, off);
            ti += __shfl_down_sync(0xffffffffu, ti, off);
        }
        sum[0] += en;
        sum[1] += tr;
        sum[2] += ti;
    }
    if (lane == 0)
        for (int q = 0; q < 3; ++q) out[q] = sum[q];
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

}  // namespace hx

#endif  // HX_RUN_CUH
