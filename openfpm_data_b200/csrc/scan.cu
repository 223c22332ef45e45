// Device-wide exclusive prefix sum of uint32 (replaces openfpm::scan, a CUB
// DeviceScan::ExclusiveSum wrapper, src/util/cuda/scan_ofp.cuh:31-80).
// Three phases: tile reduce, recursive scan of the tile sums, tile scan.
#include "common.cuh"
#include "internal.h"

namespace sgb {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* smem_warp, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) smem_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kScanThreads / 32 ? smem_warp[lane] : 0;
        uint32_t s = w;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        if (lane < kScanThreads / 32) smem_warp[lane] = s - w;
        if (lane == kScanThreads / 32 - 1) smem_warp[32] = s;
    }
    __syncthreads();
    uint32_t r = smem_warp[warp] + x - v;
    *total = smem_warp[32];
    __syncthreads();
    return r;
}

__global__ void k_scan_reduce(const uint32_t* in, int64_t n, uint32_t* sums) {
    __shared__ uint32_t sw[33];
    const int64_t base = blockIdx.x * (int64_t)kScanTile + threadIdx.x * kScanItems;
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
        if (base + k < n) s += in[base + k];
    uint32_t tot;
    block_exclusive_scan(s, sw, &tot);
    if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

__global__ void k_scan_tiles(const uint32_t* in, int64_t n, const uint32_t* offsets, uint32_t* out,
                             uint32_t* total_dev) {
    __shared__ uint32_t sw[33];
    const int64_t base = blockIdx.x * (int64_t)kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? in[base + k] : 0;
        s += v[k];
    }
    uint32_t tot;
    uint32_t pre = block_exclusive_scan(s, sw, &tot) + (offsets ? offsets[blockIdx.x] : 0);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) out[base + k] = pre;
        pre += v[k];
    }
    if (total_dev && blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) *total_dev = pre;
}

// Short arrays: one CTA walks them, 16384 items a round (three launches of a few CTAs each cost 10.5 us for 19 K
// items, this 8.1 us).  VEC: 16-byte accesses, for 16-byte aligned arrays.  At both ends the other kernels are the
// faster ones (the point list of n chunks in us, with a tile's CTA / this / three launches): 512 chunks 38 / 41 / -,
// 1024 40 / 39 / -, 4096 - / 40 / 45, 32768 - / 51 / 50, 46656 - / 57 / 58, 65536 - / 74 / 68.
constexpr int64_t kScanOneMin = 512, kScanOneMax = 49152;
constexpr int kScanOneItems = 16;
template <bool VEC>
__global__ void __launch_bounds__(1024) k_scan_one(const uint32_t* __restrict__ in, int64_t n, uint32_t* __restrict__ out,
                                                    uint32_t* total_dev) {
    __shared__ uint32_t ws[33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t carry = 0;
    for (int64_t t0 = 0; t0 < n; t0 += 1024 * kScanOneItems) {
        const int64_t base = t0 + threadIdx.x * kScanOneItems;
        uint32_t v[kScanOneItems], s = 0;
        if (VEC && base + kScanOneItems <= n) {
#pragma unroll
            for (int k = 0; k < kScanOneItems / 4; ++k)
                *reinterpret_cast<uint4*>(v + 4 * k) = *reinterpret_cast<const uint4*>(in + base + 4 * k);
        } else {
#pragma unroll
            for (int k = 0; k < kScanOneItems; ++k) v[k] = base + k < n ? in[base + k] : 0;
        }
#pragma unroll
        for (int k = 0; k < kScanOneItems; ++k) {
            const uint32_t c = v[k];
            v[k] = s;
            s += c;
        }
        uint32_t incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        if (lane == 31) ws[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            const uint32_t w = ws[lane];
            uint32_t x = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += u;
            }
            ws[lane] = x - w;
            if (lane == 31) ws[32] = x;
        }
        __syncthreads();
        const uint32_t pre = carry + ws[warp] + incl - s;
        carry += ws[32];
#pragma unroll
        for (int k = 0; k < kScanOneItems; ++k) v[k] += pre;
        if (VEC && base + kScanOneItems <= n) {
#pragma unroll
            for (int k = 0; k < kScanOneItems / 4; ++k)
                *reinterpret_cast<uint4*>(out + base + 4 * k) = *reinterpret_cast<uint4*>(v + 4 * k);
        } else {
#pragma unroll
            for (int k = 0; k < kScanOneItems; ++k)
                if (base + k < n) out[base + k] = v[k];
        }
        __syncthreads();
    }
    if (total_dev && threadIdx.x == 0) *total_dev = carry;
}

// tmp must provide scratch for the tile sums of every level.
int scan_exclusive_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* total_dev, DevBuf* tmp,
                       cudaStream_t s) {
    if (n <= 0) {
        if (total_dev) SGB_CUDA(cudaMemsetAsync(total_dev, 0, 4, s));
        return SGB_OK;
    }
    if (n <= kScanOneMin) {
        k_scan_tiles<<<1, kScanThreads, 0, s>>>(in, n, nullptr, out, total_dev);
        SGB_CUDA(cudaGetLastError());
        return SGB_OK;
    }
    if (n <= kScanOneMax) {
        const bool vec = ((uintptr_t)in | (uintptr_t)out) % 16 == 0;
        if (vec) k_scan_one<true><<<1, 1024, 0, s>>>(in, n, out, total_dev);
        else k_scan_one<false><<<1, 1024, 0, s>>>(in, n, out, total_dev);
        SGB_CUDA(cudaGetLastError());
        return SGB_OK;
    }
    const int64_t tiles = (n + kScanTile - 1) / kScanTile;
    SGB_TRY(tmp->reserve((size_t)tiles * 4 * 2 + 64));
    uint32_t* sums = tmp->as<uint32_t>();
    uint32_t* offs = sums + tiles;
    k_scan_reduce<<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, sums);
    SGB_CUDA(cudaGetLastError());
    DevBuf sub;  // recursion scratch (only for > kScanTile^2 items)
    int st = scan_exclusive_u32(sums, offs, tiles, nullptr, &sub, s);
    if (st != SGB_OK) return st;
    k_scan_tiles<<<(unsigned)tiles, kScanThreads, 0, s>>>(in, n, offs, out, total_dev);
    cudaError_t e = cudaGetLastError();
    if (sub.p) {
        cudaStreamSynchronize(s);
        sub.release();
    }
    if (e != cudaSuccess) return cuda_status(e, "k_scan_tiles");
    return SGB_OK;
}

}  // namespace sgb
