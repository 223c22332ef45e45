// Self-check of the bounded waits (failure detection without a GPU fault).
//
// A wait in a kernel of this library has a limit; when it passes, the kernel
// raises kErrWaitTimeout in the grid's error word and returns, and the host
// reports SGB_ETIMEOUT with the context intact.  The one such wait is the grid
// barrier of the small-solve kernel for 4^3 chunks (counter_wait_bounded);
// everything else is ordered by hardware cluster barriers, CTA barriers and
// launches.  This entry point runs that wait, and one on an mbarrier phase, on
// conditions that nothing ever satisfies (a counter nobody increments, a phase
// with no arrivals), each with a short limit, so a test can see the path work.
#include "common.cuh"
#include "internal.h"

namespace sgb {

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait on an mbarrier phase: gives up after about `limit_ns`
// nanoseconds, raises kErrWaitTimeout in *err and returns false.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, unsigned* err,
                                                  uint64_t limit_ns = 2000000000ull) {
    if (mbar_try_wait(bar, parity)) return true;
    const uint64_t t0 = global_timer_ns();
    for (uint32_t it = 0;; ++it) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((it & 63u) == 63u && global_timer_ns() - t0 > limit_ns) {
            atomicOr(err, kErrWaitTimeout);
            return false;
        }
    }
}

__global__ void k_probe_waits(uint64_t limit_ns, unsigned* err, unsigned* counter) {
    __shared__ uint64_t bar;
    if (threadIdx.x != 0) return;
    mbar_init(&bar, 1);
    mbar_fence_init();
    // phase 0 never completes: nobody arrives
    mbar_wait_bounded(&bar, 0, err, limit_ns);
    // the counter stays 0: nobody increments it
    counter_wait_bounded(counter, 1u, err, limit_ns);
}

}  // namespace sgb

using namespace sgb;

extern "C" int sgb_probe_bounded_waits(int64_t limit_ns, int device, sgb_stream stream) {
    if (limit_ns <= 0 || limit_ns > 1000000000ll) return SGB_EINVAL;
    DeviceGuard dg(device);
    SGB_CUDA(dg.status);
    cudaStream_t s = (cudaStream_t)stream;
    unsigned* d = nullptr;
    SGB_CUDA(cudaMalloc(&d, 8));
    unsigned h[2] = {0, 0};
    cudaError_t e = cudaMemsetAsync(d, 0, 8, s);
    if (e == cudaSuccess) {
        k_probe_waits<<<1, 32, 0, s>>>((uint64_t)limit_ns, d, d + 1);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, d, 8, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(d);
    if (e != cudaSuccess) return cuda_status(e, "sgb_probe_bounded_waits");
    if (h[0] & kErrWaitTimeout) {
        set_error("a bounded wait gave up (as this probe intends)");
        return SGB_ETIMEOUT;
    }
    return SGB_OK;
}
