// Device-side helpers: cp.async copies, bounded waits, programmatic launches, searches.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "internal.h"

namespace sgb {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ uint64_t global_timer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait for an arrival counter to reach `target`: gives up after about `limit_ns` nanoseconds, raises
// kErrWaitTimeout in *err and returns false.
__device__ __forceinline__ bool counter_wait_bounded(const unsigned* counter, unsigned target, unsigned* err,
                                                     uint64_t limit_ns = 2000000000ull) {
    const uint64_t t0 = global_timer_ns();
    for (uint32_t it = 0;; ++it) {
        if (*reinterpret_cast<const volatile unsigned*>(counter) >= target) return true;
        if ((it & 63u) == 63u && global_timer_ns() - t0 > limit_ns) {
            atomicOr(err, kErrWaitTimeout);
            return false;
        }
    }
}

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// Wait until at most N of this thread's committed cp.async groups are pending.
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The next launch may begin while this one drains.
__device__ __forceinline__ void grid_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Waits for the launch before this one; the returned value orders the loads that use it behind the wait.
__device__ __forceinline__ int64_t grid_dependency_wait() {
    int64_t z;
    asm volatile("griddepcontrol.wait;\n\tmov.u64 %0, 0;" : "=l"(z)::"memory");
    return z;
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Binary search of a chunk key in the sorted index; -1 when absent
// (vector_sparse_gpu_ker::_branchfree_search returns the background
// position instead, map_vector_sparse_cuda_ker.cuh:75-92).
__device__ __forceinline__ int64_t find_key(const int64_t* keys, int64_t n, int64_t key) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (keys[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    return (lo < n && keys[lo] == key) ? lo : -1;
}

// Number of keys strictly below `key` in a sorted array.
__device__ __forceinline__ int64_t lower_bound_i64(const int64_t* keys, int64_t n, int64_t key) {
    int64_t lo = 0, hi = n;
    while (lo < hi) {
        int64_t mid = (lo + hi) >> 1;
        if (keys[mid] < key) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

}  // namespace sgb
