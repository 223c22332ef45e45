// Flush of staged point inserts into the sorted block map.
//
// Replaces vector_sparse::flush -> flush_on_gpu_insert (src/Vector/
// map_vector_sparse.hpp:1193-1226): make_continuos + reorder_indexes (CUB
// radix sort) + merge_indexes (Thrust merge) + BlockFunctor::solve_conflicts
// (src/SparseGridGpu/BlockMapGpu_kernels.cuh:701-807).
//
// The reference stages one whole chunk slot per inserted point and reduces
// chunk slots; a chunk slot that carries a single point reduces to a per-point
// fold, so this path stages points only:
//   1. stable LSD radix sort of (point id, insertion index)
//   2. per point: A = first insert, A = op(A, next) in insertion order
//   3. unique chunk ids, looked up in the current index
//   4. when new chunks appear: merged index, old chunks moved to their new
//      positions (128-bit copies), new chunks set to background / empty mask
//   5. per point: A = op(A, old) when the point exists, mask |= EXIST
// One device->host read of three counters and the error word sizes the new
// map.
#include <algorithm>
#include <cstring>

#include "common.cuh"
#include "internal.h"

namespace sgb {

constexpr int kRsWarps = 8;
constexpr int kRsThreads = kRsWarps * 32;
// Items per thread of a tile, RR: sixteen, or four while such tiles do not outnumber the CTAs that the chip holds:
// a tile's time is mostly its ranking rounds and latencies (the ghost exchange of 84 K points: 363 us with
// sixteen, 350 with four).
constexpr int kRsRounds = 16, kRsRoundsFew = 4;

constexpr int kRsMaxBuckets = 1024;  // digits of up to 10 bits

// Digit counts of every tile, hist[tile][digit].  T: the staged 64-bit linear ids in pass 0, K afterwards.
template <int RR, typename T, typename K>
__global__ void __launch_bounds__(kRsThreads) k_rs_hist(const T* __restrict__ keys, int64_t n, int shift, unsigned dmask,
                                                         int nbuckets, uint32_t* __restrict__ hist) {
    __shared__ uint32_t h[kRsMaxBuckets];
    for (int i = threadIdx.x; i < nbuckets; i += kRsThreads) h[i] = 0;
    const int64_t base = (int64_t)blockIdx.x * (kRsThreads * RR) + threadIdx.x;
    K k[RR];  // all loads in flight at once
#pragma unroll
    for (int r = 0; r < RR; ++r) k[r] = base + r * kRsThreads < n ? (K)keys[base + r * kRsThreads] : K(0);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RR; ++r)
        if (base + r * kRsThreads < n) atomicAdd(&h[(unsigned)(k[r] >> shift) & dmask], 1u);
    __syncthreads();
    for (int d = threadIdx.x; d < nbuckets; d += kRsThreads) hist[(size_t)blockIdx.x * nbuckets + d] = h[d];
}

// Counts to exclusive prefixes over the tiles, digit by digit, in place; tot[d]: the digit's count over all
// tiles.  A CTA takes 32 digits (one per lane) and splits the tiles over its 32 warps; every access is one
// coalesced line.
__global__ void __launch_bounds__(1024) k_rs_rowscan(uint32_t* hist, int ntiles, int nbuckets, uint32_t* tot) {
    __shared__ uint32_t sums[32][33];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int d = blockIdx.x * 32 + lane;
    const int per = (ntiles + 31) / 32, t0 = min(ntiles, w * per), t1 = min(ntiles, t0 + per);
    uint32_t sum = 0;
    if (d < nbuckets)
#pragma unroll 8
        for (int t = t0; t < t1; ++t) sum += hist[(size_t)t * nbuckets + d];
    sums[w][lane] = sum;
    __syncthreads();
    uint32_t run = 0;
    for (int k = 0; k < w; ++k) run += sums[k][lane];
    if (d >= nbuckets) return;
    if (w == 31) tot[d] = run + sum;
    for (int t = t0; t < t1; t += 8) {
        uint32_t c[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) c[k] = t + k < t1 ? hist[(size_t)(t + k) * nbuckets + d] : 0;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (t + k < t1) {
                hist[(size_t)(t + k) * nbuckets + d] = run;
                run += c[k];
            }
    }
}

// Exclusive scan of one value per thread over the CTA; wsum: one word per warp.
__device__ __forceinline__ uint32_t rs_block_scan(uint32_t v, uint32_t* wsum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += u;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    uint32_t run = incl - v;
    for (int w = 0; w < warp; ++w) run += wsum[w];
    return run;
}

// The warp's lanes with the same digit, by one ballot per digit bit (__match_any_sync, whose time grows with the
// distinct values in the warp, makes a 2 M key pass with random digits 4 us longer).
__device__ __forceinline__ unsigned digit_peers(unsigned d, bool valid, unsigned dmask) {
    unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
    for (int b = 0; b < 10; ++b) {
        if (!(dmask >> b & 1u)) break;  // uniform
        const unsigned m = __ballot_sync(0xffffffffu, d >> b & 1u);
        peers &= (d >> b & 1u) ? m : ~m;
    }
    return peers;
}

// Stable scatter: items keep their order inside each digit.  Tile order is
// (warp, round, lane) == index order; ranks inside a warp come from the peer
// groups of equal digits, counts across warps from a shared prefix.
// The tile is then staged in shared memory in digit order and written out
// run by run, so that consecutive threads store consecutive positions of a
// digit's output range instead of one scattered 4-byte store per item.
//
// Bound by latency (ranking rounds, shared memory), 3.3 CTAs per SM at 2 M
// keys: 25-30 us (50 us with __match_any_sync, the loads inside the ranking
// rounds and one uncoalesced offset read per item).  The keys of a tile all go
// out before the first ranking round, the digits' output positions are read
// once per digit, coalesced, and 64 registers let four CTAs share an SM.
template <int RR, typename K>
__host__ __device__ constexpr size_t rs_union_bytes() {
    constexpr int kRsTile = kRsThreads * RR;
    return (size_t)kRsWarps * kRsMaxBuckets * 4 > (size_t)kRsTile * (sizeof(K) + 4)
               ? (size_t)kRsWarps * kRsMaxBuckets * 4
               : (size_t)kRsTile * (sizeof(K) + 4);
}
template <int RR, typename K>
__host__ __device__ constexpr size_t rs_scatter_smem() {
    return rs_union_bytes<RR, K>() + (size_t)kRsMaxBuckets * 8 + 2 * kRsWarps * 4;
}

template <int RR, typename T, typename K>
__global__ void __launch_bounds__(kRsThreads, sizeof(K) == 4 ? 4 : 2) k_rs_scatter(const T* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                            K* __restrict__ kout, uint32_t* __restrict__ vout, int64_t n,
                                                            int shift, unsigned dmask, int nbuckets,
                                                            const uint32_t* __restrict__ offs,
                                                            const uint32_t* __restrict__ tot_g) {
    constexpr int kRsTile = kRsThreads * RR;
    extern __shared__ __align__(16) unsigned char rs_smem[];
    auto wcnt = reinterpret_cast<uint32_t(*)[kRsMaxBuckets]>(rs_smem);  // [kRsWarps][kRsMaxBuckets]
    K* sk = reinterpret_cast<K*>(rs_smem);                              // the same bytes, once wcnt is done
    uint32_t* sv = reinterpret_cast<uint32_t*>(rs_smem + (size_t)kRsTile * sizeof(K));
    uint32_t* dstart = reinterpret_cast<uint32_t*>(rs_smem + rs_union_bytes<RR, K>());  // digit's first place in the tile
    uint32_t* gdst = dstart + kRsMaxBuckets;  // output position of the digit's items minus dstart
    uint32_t* wsum = gdst + kRsMaxBuckets;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t tbase = (int64_t)blockIdx.x * kRsTile;
    const int64_t base = tbase + warp * (32 * RR) + lane;
    K key[RR];
    uint32_t rank[RR];
#pragma unroll
    for (int r = 0; r < RR; ++r) {
        const int64_t i = base + r * 32;
        key[r] = i < n ? (K)kin[i] : K(0);
    }
    for (int i = threadIdx.x; i < kRsWarps * kRsMaxBuckets / 4; i += kRsThreads)
        reinterpret_cast<uint4*>(&wcnt[0][0])[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const unsigned lt = lanemask_lt();
#pragma unroll
    for (int r = 0; r < RR; ++r) {
        const bool valid = base + r * 32 < n;
        const unsigned d = (unsigned)(key[r] >> shift) & dmask;
        const unsigned peers = digit_peers(d, valid, dmask);
        uint32_t cnt = 0;
        if (valid) cnt = wcnt[warp][d];
        rank[r] = cnt + __popc(peers & lt);
        __syncwarp();
        if (valid && lane == __ffs(peers) - 1) wcnt[warp][d] = cnt + __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    uint32_t val[RR];  // needed from here on
#pragma unroll
    for (int r = 0; r < RR; ++r) {
        const int64_t i = base + r * 32;
        val[r] = i < n ? (vin ? vin[i] : (uint32_t)i) : 0u;
    }
    // per digit: the warps' counts become prefixes; thread t owns digits kPer t .. kPer t + kPer - 1
    constexpr int kPer = kRsMaxBuckets / kRsThreads;
    uint32_t tot[kPer], tsum = 0, gtot[kPer], gsum = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int d = threadIdx.x * kPer + k;
        uint32_t run = 0;
        gtot[k] = d < nbuckets ? tot_g[d] : 0;
        if (d < nbuckets)
#pragma unroll
            for (int w = 0; w < kRsWarps; ++w) {
                const uint32_t c = wcnt[w][d];
                wcnt[w][d] = run;
                run += c;
            }
        tot[k] = run;
        tsum += run;
        gsum += gtot[k];
    }
    // the digits' first positions in the tile and in the output: exclusive scans of the threads' sums
    uint32_t run = rs_block_scan(tsum, wsum), grun = rs_block_scan(gsum, wsum + kRsWarps);
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const int d = threadIdx.x * kPer + k;
        if (d < nbuckets) {
            dstart[d] = run;
            gdst[d] = grun + offs[(size_t)blockIdx.x * nbuckets + d] - run;
        }
        run += tot[k];
        grun += gtot[k];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RR; ++r) {
        if (base + r * 32 < n) {
            const unsigned d = (unsigned)(key[r] >> shift) & dmask;
            rank[r] += dstart[d] + wcnt[warp][d];  // position in the tile, digit order
        }
    }
    __syncthreads();  // wcnt is read no more: its bytes take the staged tile
#pragma unroll
    for (int r = 0; r < RR; ++r) {
        if (base + r * 32 < n) {
            sk[rank[r]] = key[r];
            sv[rank[r]] = val[r];
        }
    }
    __syncthreads();
    const int tn = (int)(n - tbase < kRsTile ? n - tbase : kRsTile);
#pragma unroll 4
    for (int j = threadIdx.x; j < tn; j += kRsThreads) {
        const K k = sk[j];
        const uint32_t pos = gdst[(unsigned)(k >> shift) & dmask] + (uint32_t)j;
        kout[pos] = k;
        vout[pos] = sv[j];
    }
}

struct PropSet {
    unsigned char* p[kMaxProps];
    int type[kMaxProps];
    int op[kMaxProps];
    int nprop;
};

template <typename T>
__device__ __forceinline__ T op_apply(int op, T a, T b) {
    switch (op) {
        case SGB_OP_RIGHT: return b;                  // rightOperand_t
        case SGB_OP_LEFT: return a;                   // leftOperand_t
        case SGB_OP_ADD: return a + b;                // plus_t
        case SGB_OP_MAX: return a > b ? a : b;        // maximum_t
        case SGB_OP_MIN: return a < b ? a : b;        // minimum_t
        default: return b;
    }
}

// Elements of any property type travel as raw 64-bit words.
__device__ __forceinline__ uint64_t load_raw(int type, const unsigned char* p, int64_t i) {
    switch (type) {
        case SGB_F64: return reinterpret_cast<const uint64_t*>(p)[i];
        case SGB_U8: return p[i];
        default: return reinterpret_cast<const uint32_t*>(p)[i];
    }
}
__device__ __forceinline__ void store_raw(int type, unsigned char* p, int64_t i, uint64_t v) {
    switch (type) {
        case SGB_F64: reinterpret_cast<uint64_t*>(p)[i] = v; break;
        case SGB_U8: p[i] = (unsigned char)v; break;
        default: reinterpret_cast<uint32_t*>(p)[i] = (uint32_t)v;
    }
}
// op(a, b) on raw elements of type `type` (both operands exist).
__device__ __forceinline__ uint64_t op_raw(int type, int op, uint64_t a, uint64_t b) {
    if (op == SGB_OP_RIGHT) return b;
    if (op == SGB_OP_LEFT) return a;
    switch (type) {
        case SGB_F32: return __float_as_uint(op_apply(op, __uint_as_float((uint32_t)a), __uint_as_float((uint32_t)b)));
        case SGB_F64:
            return (uint64_t)__double_as_longlong(
                op_apply(op, __longlong_as_double((long long)a), __longlong_as_double((long long)b)));
        case SGB_I32: {
            const int32_t x = (int32_t)(uint32_t)a, y = (int32_t)(uint32_t)b;
            return (uint32_t)(op == SGB_OP_OR ? (x | y) : op_apply(op, x, y));
        }
        default: {
            const uint8_t x = (uint8_t)a, y = (uint8_t)b;
            return (uint8_t)(op == SGB_OP_OR ? (uint8_t)(x | y) : op_apply(op, x, y));
        }
    }
}

// The rest of a point's inserts folded into its first one, in insertion order: one branch on the operation per run and
// three values in flight (one point inserted 8192 times with an addition, the whole flush: 2053 us with a branch per
// insert and a value at a time, 898 so and with run_end).  With four values the kernels that call this spill more:
// 0.3 % of the 1024^3 rebuild, whose points have few inserts, for 7-30 % of such runs.  A call: inlined into the
// unrolled rounds of its users it takes 218 registers.
template <int OP, typename T, typename I>
__device__ __forceinline__ T fold_loop(int type, T first, const T* vals, const I* sidx, uint32_t len) {
    constexpr int N = 3;
    uint64_t acc = first;
    for (uint32_t j = 1; j < len; j += N) {
        T v[N];
#pragma unroll
        for (int k = 0; k < N; ++k) v[k] = j + k < len ? vals[sidx[j + k]] : T(0);
#pragma unroll
        for (int k = 0; k < N; ++k)
            if (j + k < len) acc = op_raw(type, OP, acc, (uint64_t)v[k]);
    }
    return (T)acc;
}
template <typename T, typename I>
__device__ __noinline__ T fold_rest(int type, int op, T first, const T* vals, const I* sidx, uint32_t len) {
    switch (op) {  // one branch per run and not per insert
        case SGB_OP_ADD: return fold_loop<SGB_OP_ADD>(type, first, vals, sidx, len);
        case SGB_OP_MAX: return fold_loop<SGB_OP_MAX>(type, first, vals, sidx, len);
        case SGB_OP_MIN: return fold_loop<SGB_OP_MIN>(type, first, vals, sidx, len);
        default: return fold_loop<SGB_OP_OR>(type, first, vals, sidx, len);
    }
}

// The first item from e on (in sorted order) that is not k: doubling steps, as a point may fill the whole list (100 K
// inserts of one point: a quarter of the flush's time item by item).
template <typename K, typename I>
__device__ __forceinline__ I run_end(const K* sk, I n, I e, K k) {
    while (e < n && sk[e] == k) {
        for (I step = 1; e + step < n && sk[e + step] == k; step <<= 1) e += step;
        ++e;
    }
    return e;
}

// Segment heads of the sorted ids: the first item of every point and of every chunk.  A tile of 1024 items
// is four rounds of a 256-thread CTA in index order (eight rounds: 8 us more per 2 M points, fewer CTAs in flight).
constexpr int kHdThreads = 256, kHdRounds = 4, kHdTile = kHdThreads * kHdRounds;

template <typename K>
__device__ __forceinline__ void heads_of(const K* __restrict__ sk, int64_t n, int64_t i, int bs_shift, K& k, bool& pt,
                                         bool& blk) {
    pt = blk = false;
    k = K(0);
    if (i < n) {
        k = sk[i];
        const K prev = i ? sk[i - 1] : k;
        pt = i == 0 || prev != k;
        blk = i == 0 || (prev >> bs_shift) != (k >> bs_shift);
    }
}

// Points and chunks that begin in every tile.
template <typename K>
__global__ void __launch_bounds__(kHdThreads) k_heads_count(const K* __restrict__ sk, int64_t n, int bs_shift,
                                                             uint2* __restrict__ cnt) {
    __shared__ uint32_t np, nb;
    if (threadIdx.x == 0) np = nb = 0;
    __syncthreads();
    uint32_t p = 0, b = 0;
#pragma unroll
    for (int r = 0; r < kHdRounds; ++r) {
        K k;
        bool hp, hb;
        heads_of(sk, n, (int64_t)blockIdx.x * kHdTile + r * kHdThreads + threadIdx.x, bs_shift, k, hp, hb);
        p += hp;
        b += hb;
    }
    p = __reduce_add_sync(0xffffffffu, p);
    b = __reduce_add_sync(0xffffffffu, b);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&np, p);
        atomicAdd(&nb, b);
    }
    __syncthreads();
    if (threadIdx.x == 0) cnt[blockIdx.x] = make_uint2(np, nb);
}

// Exclusive scan of the tiles' counts by one CTA, in place.  WHICH 0: (points, chunks) pairs, totals to
// counters[0], [1].  WHICH 1: new chunks per 1024-chunk tile, as many tiles as counters[1] chunks take, total to
// counters[2]; the device error word goes along to counters[3].
constexpr int kLkTile = 1024;
template <int WHICH>
__global__ void __launch_bounds__(1024) k_tile_scan(uint2* cnt, int64_t ntiles, uint32_t* counters, const unsigned* err) {
    __shared__ uint32_t wx[32], wy[32];
    if (WHICH == 1) ntiles = ((int64_t)counters[1] + kLkTile - 1) / kLkTile;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t cx = 0, cy = 0;
    for (int64_t t0 = 0; t0 < ntiles; t0 += 1024) {
        const int64_t t = t0 + threadIdx.x;
        const uint2 v = t < ntiles ? cnt[t] : make_uint2(0, 0);
        uint32_t x = v.x, y = v.y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t a = __shfl_up_sync(0xffffffffu, x, o), b = __shfl_up_sync(0xffffffffu, y, o);
            if (lane >= o) {
                x += a;
                y += b;
            }
        }
        if (lane == 31) {
            wx[warp] = x;
            wy[warp] = y;
        }
        __syncthreads();
        uint32_t bx = cx, by = cy;
        for (int w = 0; w < 32; ++w) {
            if (w < warp) {
                bx += wx[w];
                by += wy[w];
            }
            cx += wx[w];
            cy += wy[w];
        }
        if (t < ntiles) cnt[t] = make_uint2(bx + x - v.x, by + y - v.y);
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        if (WHICH == 0) {
            counters[0] = cx;
            counters[1] = cy;
        } else {
            counters[2] = cx;
            counters[3] = *err;
        }
    }
}

// Per point: fold its inserts in insertion order (the sort is stable).  The point's chunk (its rank among the
// touched chunks) and offset go to upt, the reduced values to vals_out, the touched chunks' ids to ublk_key.
template <typename K>
__global__ void __launch_bounds__(kHdThreads, 4) k_fold(const K* __restrict__ sk, const uint32_t* __restrict__ sidx, int64_t n,
                                                      int bs_shift, const uint2* __restrict__ tile_off, PropSet vals,
                                                      PropSet out, uint2* __restrict__ upt, int64_t* __restrict__ ublk_key) {
    constexpr int W = kHdThreads / 32;
    __shared__ uint32_t pre[kHdRounds * W];  // points | chunks << 16 that begin before (round, warp) in the tile
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t base = (int64_t)blockIdx.x * kHdTile + threadIdx.x;
    K key[kHdRounds];
    unsigned pb[kHdRounds], bb[kHdRounds];
#pragma unroll
    for (int r = 0; r < kHdRounds; ++r) {
        bool hp, hb;
        heads_of(sk, n, base + r * kHdThreads, bs_shift, key[r], hp, hb);
        pb[r] = __ballot_sync(0xffffffffu, hp);
        bb[r] = __ballot_sync(0xffffffffu, hb);
        if (lane == 0) pre[r * W + warp] = __popc(pb[r]) | __popc(bb[r]) << 16;
    }
    __syncthreads();
    static_assert(kHdRounds * W == 32, "one entry per lane");
    if (warp == 0) {
        const uint32_t a = pre[lane];
        uint32_t incl = a;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        pre[lane] = incl - a;
    }
    __syncthreads();
    const uint2 off = tile_off[blockIdx.x];
    const unsigned lt = lanemask_lt(), le = lt | 1u << lane;
    // round by round: the point's rank, how many inserts it has, and its first and last one's staging index
    uint32_t u[kHdRounds], len[kHdRounds], first[kHdRounds], last[kHdRounds];
#pragma unroll
    for (int r = 0; r < kHdRounds; ++r) {
        len[r] = 0;
        if (!(pb[r] >> lane & 1u)) continue;
        const int64_t i = base + r * kHdThreads;
        const K k = key[r];
        const uint32_t pr = pre[r * W + warp];
        const uint32_t b = off.y + (pr >> 16) + __popc(bb[r] & le) - 1;
        u[r] = off.x + (pr & 0xffffu) + __popc(pb[r] & lt);
        upt[u[r]] = make_uint2(b, (uint32_t)(k & (((K)1 << bs_shift) - 1)));
        if (bb[r] >> lane & 1u) ublk_key[b] = (int64_t)(k >> bs_shift);
        const unsigned next = pb[r] & ~le;  // the next point begins at that lane, or past the warp's items
        uint32_t c = next ? (uint32_t)(__ffs(next) - 1 - lane) : (uint32_t)(32 - lane);
        if (!next) c = (uint32_t)(run_end(sk, n, i + c, k) - i);
        len[r] = i + c < n ? c : (uint32_t)(n - i);
        first[r] = sidx[i];
        last[r] = len[r] > 1 ? sidx[i + len[r] - 1] : first[r];
    }
    for (int p = 0; p < vals.nprop; ++p) {
        const int op = vals.op[p], t = vals.type[p];
        if (op == SGB_OP_NONE) continue;
        auto reduce = [&](auto zero) {
            using T = decltype(zero);
            const T* src = reinterpret_cast<const T*>(vals.p[p]);
            T* dst = reinterpret_cast<T*>(out.p[p]);
            T v[kHdRounds];  // all of the thread's values in flight at once
#pragma unroll
            for (int r = 0; r < kHdRounds; ++r) v[r] = len[r] ? src[op == SGB_OP_RIGHT ? last[r] : first[r]] : zero;
            if (op != SGB_OP_RIGHT && op != SGB_OP_LEFT)
#pragma unroll
                for (int r = 0; r < kHdRounds; ++r)
                    if (len[r] > 1) v[r] = fold_rest(t, op, v[r], src, sidx + base + r * kHdThreads, len[r]);
#pragma unroll
            for (int r = 0; r < kHdRounds; ++r)
                if (len[r]) dst[u[r]] = v[r];
        };
        if (t == SGB_F64) reduce(uint64_t(0));
        else if (t == SGB_U8) reduce(uint8_t(0));
        else reduce(uint32_t(0));
    }
}

// The touched chunks in the current index: 2 x (old chunks below its id) + (1 when it is new), and the number of
// new ones per 1024-chunk tile.  How many there are is known on the device only.
__global__ void __launch_bounds__(kLkTile) k_lookup(const int64_t* __restrict__ ublk_key, const uint32_t* __restrict__ counters,
                                                 const int64_t* __restrict__ keys, int64_t n, int64_t* __restrict__ place,
                                                 uint2* __restrict__ cnt) {
    __shared__ uint32_t nnew;
    const int64_t nb = counters[1];
    for (int64_t t = blockIdx.x; t * kLkTile < nb; t += gridDim.x) {
        if (threadIdx.x == 0) nnew = 0;
        __syncthreads();
        uint32_t c = 0;
        const int64_t b = t * kLkTile + threadIdx.x;
        if (b < nb) {
            const int64_t key = ublk_key[b];
            const int64_t lo = lower_bound_i64(keys, n, key);
            const bool isnew = !(lo < n && keys[lo] == key);
            place[b] = 2 * lo + isnew;
            c = isnew;
        }
        c = __reduce_add_sync(0xffffffffu, c);
        if ((threadIdx.x & 31) == 0) atomicAdd(&nnew, c);
        __syncthreads();
        if (threadIdx.x == 0) cnt[t] = make_uint2(nnew, 0);
        __syncthreads();
    }
}

// Positions in the merged map: (old chunks below) + (new chunks below).  place[b] becomes 2 x that; the new
// chunks also enter the new-key list and the merged index.
__global__ void __launch_bounds__(kLkTile) k_merge_pos(const int64_t* __restrict__ ublk_key, int64_t nb, int64_t* place,
                                                        const uint2* __restrict__ tile_off, int64_t* __restrict__ newkeys,
                                                        int64_t* __restrict__ keys_out, int32_t* __restrict__ srcpos) {
    __shared__ uint32_t wsum[32];
    const int64_t b = (int64_t)blockIdx.x * kLkTile + threadIdx.x;
    const int64_t v = b < nb ? place[b] : 0;
    const uint32_t isnew = (uint32_t)(v & 1);
    const uint32_t rank = tile_off[blockIdx.x].x + rs_block_scan(isnew, wsum);
    if (b >= nb) return;
    const int64_t pos = (v >> 1) + rank;
    place[b] = 2 * pos;
    if (isnew) {
        const int64_t key = ublk_key[b];
        newkeys[rank] = key;
        keys_out[pos] = key;
        srcpos[pos] = -1;
    }
}

// New position of every old chunk: j + #(new keys below its key).
__global__ void k_old_pos(const int64_t* __restrict__ keys, int64_t n, const int64_t* __restrict__ newkeys, int64_t nnew,
                          int64_t* __restrict__ keys_out, int32_t* __restrict__ srcpos) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int64_t k = keys[j];
    const int64_t pos = j + lower_bound_i64(newkeys, nnew, k);
    srcpos[pos] = (int32_t)j;
    keys_out[pos] = k;
}

struct MapSet {
    const uint4* src[kMaxProps + 1];
    uint4* dst[kMaxProps + 1];
    uint4 fill[kMaxProps + 1];
    int shift[kMaxProps + 1];  // a chunk holds 2^shift 16-byte words
    int count;
};

// The merged map, all properties and the masks: a warp per chunk of it copies the old chunk there or fills a new
// one (and the background chunk at position n) with backgrounds and a zero mask.  Bound by HBM: 6.8 TB/s.
__global__ void __launch_bounds__(256) k_merge_map(MapSet ms, const int32_t* __restrict__ srcpos, int64_t n) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; c <= n; c += nw) {
        const int64_t s = c < n ? srcpos[c] : -1;
        for (int p = 0; p < ms.count; ++p) {
            const int words = 1 << ms.shift[p];
            uint4* d = ms.dst[p] + (c << ms.shift[p]);
            if (s < 0) {
                for (int w = lane; w < words; w += 32) d[w] = ms.fill[p];
                continue;
            }
            const uint4* q = ms.src[p] + (s << ms.shift[p]);
            if (words == 128) {
                uint4 v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] = __ldcs(q + lane + 32 * k);  // the old map is read once
#pragma unroll
                for (int k = 0; k < 4; ++k) d[lane + 32 * k] = v[k];
            } else {
                for (int w = lane; w < words; w += 32) d[w] = __ldcs(q + w);
            }
        }
    }
}

// The element pattern of es bytes repeated over a 16-byte word.
static uint4 replicate16(uint64_t pattern, int es) {
    unsigned char b[16];
    for (int i = 0; i < 16; ++i) b[i] = (unsigned char)(pattern >> (8 * (i % es)));
    uint4 w;
    std::memcpy(&w, b, 16);
    return w;
}

// A unique point: reduce with the existing value, write, set EXIST.
__device__ __forceinline__ void write_point(uint2 q, int64_t u, int bs_shift, const int64_t* place, const PropSet& upv,
                                            const PropSet& data, uint8_t* mask, int any_listed) {
    const int64_t idx = (place[q.x] >> 1 << bs_shift) + q.y;
    const uint8_t om = mask[idx];
    for (int p = 0; p < data.nprop; ++p) {
        const int op = data.op[p], t = data.type[p];
        if (op == SGB_OP_NONE) continue;
        if ((om & 1) && op == SGB_OP_RIGHT) continue;  // op(new, old) = old
        uint64_t v = load_raw(t, upv.p[p], u);
        if ((om & 1) && op != SGB_OP_LEFT) v = op_raw(t, op, v, load_raw(t, data.p[p], idx));  // BlockMapGpu_kernels.cuh:294-305
        store_raw(t, data.p[p], idx, v);
    }
    if (any_listed && !(om & 1)) mask[idx] = om | 1u;
}

__global__ void k_scatter(const uint2* __restrict__ upt, int64_t nu, int bs_shift, const int64_t* __restrict__ place,
                          PropSet upv, PropSet data, uint8_t* mask, int any_listed) {
    const int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (u < nu) write_point(upt[u], u, bs_shift, place, upv, data, mask, any_listed);
}

// ------------------------------------------------------------------ small flushes in one launch
// Up to 8192 staged points: one CTA sorts them in shared memory (digits of at most 8 bits, eight items per thread),
// folds the points' inserts, looks the touched chunks up and, when none of them is new, writes the results back --
// what the kernels above do in 14 launches of a few CTAs, each bound by its launch and memory latency.  (5003
// points into a 128^3 map, whole call: 123 us with those, 92 us so.)  The limit is what the CTA's shared memory holds;
// the kernels above are as fast from fewer points on when many properties are listed, since one CTA folds and writes
// them all.  Insert and flush in us, here / by those kernels, points in existing chunks and in new ones: 1 property
// 8192 points 86 / 103 and 89 / 117; 3 properties 5120 points 102 / 111 and 99 / 129, 8192 points 129 / 111 and
// 114 / 129; 6 properties 4096 points 128 / 123 and 118 / 147, 8192 points 188 / 124 and 154 / 146 (8^3 chunks; 4^3
// chunks and 64-bit ids within 15 %).
constexpr int kSmThreads = 1024, kSmItems = 8, kSmMax = kSmThreads * kSmItems, kSmBuckets = 256;

template <typename K>
constexpr size_t small_smem() {
    // keys, indexes, per-warp digit counts, digit starts
    return (size_t)kSmMax * (sizeof(K) + 2) + (size_t)32 * kSmBuckets * 2 + (size_t)kSmBuckets * 4 * 5;
}

template <typename K>
__global__ void __launch_bounds__(kSmThreads) k_flush_small(const int64_t* __restrict__ lin, int n, int passes, int dbits,
                                                             int bs_shift, PropSet vals, PropSet out, PropSet data,
                                                             uint8_t* mask, int any_listed, const int64_t* __restrict__ keys,
                                                             int64_t nold, uint2* upt, int64_t* ublk_key, int64_t* place,
                                                             uint2* ltile, uint32_t* counters, const unsigned* err) {
    extern __shared__ __align__(16) unsigned char sm_raw[];
    K* sk = reinterpret_cast<K*>(sm_raw);
    uint16_t* si = reinterpret_cast<uint16_t*>(sk + kSmMax);
    auto wcnt = reinterpret_cast<uint16_t(*)[kSmBuckets]>(si + kSmMax);  // [32 warps]
    auto part = reinterpret_cast<uint32_t(*)[kSmBuckets]>(wcnt + 32);    // [4]: sums of eight warps each
    uint32_t* dstart = &part[4][0];
    __shared__ uint32_t ws[33];
    __shared__ unsigned bad;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = lanemask_lt(), dmask = (1u << dbits) - 1u;
    if (tid == 0) bad = *err & (kErrOutOfDomain | kErrPoolOverflow);
    K key[kSmItems];
    uint32_t idx[kSmItems], rank[kSmItems];
    const int rounds = (n + kSmThreads - 1) / kSmThreads;  // the same for every warp
    const int base = warp * 32 * rounds + lane;  // items in (warp, round, lane) order
#pragma unroll
    for (int r = 0; r < kSmItems; ++r) {
        const int i = r < rounds ? base + 32 * r : n;
        key[r] = i < n ? (K)lin[i] : K(0);
        idx[r] = (uint32_t)i;
    }
    for (int ps = 0; ps < passes; ++ps) {
        const int shift = ps * dbits;
        reinterpret_cast<uint4*>(wcnt)[tid] = make_uint4(0, 0, 0, 0);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSmItems; ++r) {
            if (r >= rounds) break;  // uniform
            const bool valid = base + 32 * r < n;
            const unsigned d = (unsigned)(key[r] >> shift) & dmask;
            const unsigned peers = digit_peers(d, valid, dmask);
            uint32_t c = 0;
            if (valid) c = wcnt[warp][d];
            rank[r] = c + __popc(peers & lt);
            __syncwarp();
            if (valid && lane == __ffs(peers) - 1) wcnt[warp][d] = (uint16_t)(c + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        {  // counts to prefixes over the warps: a thread takes one digit of eight warps
            const int d = tid & (kSmBuckets - 1), q = tid >> 8;
            uint32_t sum = 0;
#pragma unroll
            for (int w = 0; w < 8; ++w) sum += wcnt[q * 8 + w][d];
            part[q][d] = sum;
            __syncthreads();
            uint32_t run = 0;
            for (int k = 0; k < q; ++k) run += part[k][d];
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                const uint32_t c = wcnt[q * 8 + w][d];
                wcnt[q * 8 + w][d] = (uint16_t)run;
                run += c;
            }
            if (warp == 0) {  // the digits' starts: eight digits per lane
                uint32_t t[8], s = 0;
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    const int e = lane * 8 + k;
                    t[k] = s;
                    s += part[0][e] + part[1][e] + part[2][e] + part[3][e];
                }
                uint32_t incl = s;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
                    if (lane >= o) incl += u;
                }
#pragma unroll
                for (int k = 0; k < 8; ++k) dstart[lane * 8 + k] = t[k] + incl - s;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSmItems; ++r)
            if (r < rounds && base + 32 * r < n) {
                const unsigned d = (unsigned)(key[r] >> shift) & dmask;
                const uint32_t pos = dstart[d] + wcnt[warp][d] + rank[r];
                sk[pos] = key[r];
                si[pos] = (uint16_t)idx[r];
            }
        __syncthreads();
        if (ps + 1 < passes)
#pragma unroll
            for (int r = 0; r < kSmItems; ++r)
                if (r < rounds && base + 32 * r < n) {
                    key[r] = sk[base + 32 * r];
                    idx[r] = si[base + 32 * r];
                }
    }
    // heads: a thread takes eight consecutive items; ranks by one scan (points | chunks << 16)
    const int i0 = tid * kSmItems;
    uint32_t hp = 0, hb = 0;  // bit k: item i0 + k begins a point / a chunk
#pragma unroll
    for (int k = 0; k < kSmItems; ++k) {
        const int i = i0 + k;
        if (i < n) {
            const K c = sk[i], p = i ? sk[i - 1] : c;
            if (i == 0 || c != p) hp |= 1u << k;
            if (i == 0 || (c >> bs_shift) != (p >> bs_shift)) hb |= 1u << k;
        }
    }
    const uint32_t mine = __popc(hp) | (uint32_t)__popc(hb) << 16;
    const uint32_t before = rs_block_scan(mine, ws);
    if (tid == kSmThreads - 1) ws[32] = before + mine;
    __syncthreads();
    const uint32_t U = ws[32] & 0xffffu, B = ws[32] >> 16;
    uint32_t len[kSmItems], first[kSmItems], last[kSmItems];
    const uint32_t u0 = before & 0xffffu, b0 = before >> 16;
#pragma unroll
    for (int k = 0; k < kSmItems; ++k) {
        len[k] = 0;
        if (!(hp >> k & 1u)) continue;
        const int i = i0 + k;
        const K c = sk[i];
        const uint32_t b = b0 + __popc(hb & ((2u << k) - 1u)) - 1;
        upt[u0 + __popc(hp & ((1u << k) - 1u))] = make_uint2(b, (uint32_t)(c & (((K)1 << bs_shift) - 1)));
        if (hb >> k & 1u) ublk_key[b] = (int64_t)(c >> bs_shift);
        const int e = run_end(sk, n, i + 1, c);
        len[k] = (uint32_t)(e - i);
        first[k] = si[i];
        last[k] = si[e - 1];
    }
    for (int p = 0; p < vals.nprop; ++p) {
        const int op = vals.op[p], t = vals.type[p];
        if (op == SGB_OP_NONE) continue;
        auto reduce = [&](auto zero) {
            using T = decltype(zero);
            const T* src = reinterpret_cast<const T*>(vals.p[p]);
            T* dst = reinterpret_cast<T*>(out.p[p]);
            T v[kSmItems];
#pragma unroll
            for (int k = 0; k < kSmItems; ++k) v[k] = len[k] ? src[op == SGB_OP_RIGHT ? last[k] : first[k]] : zero;
            if (op != SGB_OP_RIGHT && op != SGB_OP_LEFT)
#pragma unroll
                for (int k = 0; k < kSmItems; ++k)
                    if (len[k] > 1) v[k] = fold_rest(t, op, v[k], src, si + i0 + k, len[k]);
#pragma unroll
            for (int k = 0; k < kSmItems; ++k)
                if (len[k]) dst[u0 + __popc(hp & ((1u << k) - 1u))] = v[k];
        };
        if (t == SGB_F64) reduce(uint64_t(0));
        else if (t == SGB_U8) reduce(uint8_t(0));
        else reduce(uint32_t(0));
    }
    __syncthreads();
    // the touched chunks in the current index (as k_lookup), 1024 at a time
    uint32_t nnew = 0;
    for (uint32_t t = 0; t * kLkTile < B; ++t) {
        const uint32_t b = t * kLkTile + tid;
        bool isnew = false;
        if (b < B) {
            const int64_t k = ublk_key[b], lo = lower_bound_i64(keys, nold, k);
            isnew = !(lo < nold && keys[lo] == k);
            place[b] = 2 * lo + isnew;
        }
        if (tid == 0) ltile[t] = make_uint2(nnew, 0);
        nnew += (uint32_t)__syncthreads_count(isnew);
    }
    if (tid == 0) {
        counters[0] = U;
        counters[1] = B;
        counters[2] = nnew;
        counters[3] = *err;
    }
    if (nnew == 0 && !bad)  // every chunk is there: write the points back now
        for (uint32_t u = tid; u < U; u += kSmThreads) write_point(upt[u], u, bs_shift, place, out, data, mask, any_listed);
}

static inline unsigned nblk(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

template <int RR, typename T, typename K>
static int radix_pass(const T* kin, const uint32_t* vin, K* kout, uint32_t* vout, int64_t n, int shift, unsigned dmask,
                      int nbuckets, uint32_t* hist, uint32_t* tot, int ntiles, cudaStream_t s) {
    k_rs_hist<RR, T, K><<<ntiles, kRsThreads, 0, s>>>(kin, n, shift, dmask, nbuckets, hist);
    k_rs_rowscan<<<(nbuckets + 31) / 32, 1024, 0, s>>>(hist, ntiles, nbuckets, tot);
    constexpr size_t smem = rs_scatter_smem<RR, K>();
    if (smem > 48 * 1024)
        SGB_CUDA(cudaFuncSetAttribute(k_rs_scatter<RR, T, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_rs_scatter<RR, T, K><<<ntiles, kRsThreads, smem, s>>>(kin, vin, kout, vout, n, shift, dmask, nbuckets, hist, tot);
    SGB_CUDA(cudaGetLastError());
    return SGB_OK;
}

template <int RR, typename K>
static int radix_sort(sgb_grid* g, int64_t n, int bits, K** keys_out, uint32_t** vals_out, cudaStream_t s) {
    DevBuf& kA = g->scratch[0];
    DevBuf& kB = g->scratch[1];
    DevBuf& vA = g->scratch[2];
    DevBuf& vB = g->scratch[3];
    DevBuf& hist = g->scratch[4];
    SGB_TRY(kA.ensure((size_t)n * sizeof(K)));
    SGB_TRY(kB.ensure((size_t)n * sizeof(K)));
    SGB_TRY(vA.ensure((size_t)n * 4));
    SGB_TRY(vB.ensure((size_t)n * 4));
    const int ntiles = (int)((n + kRsThreads * RR - 1) / (kRsThreads * RR));
    // as few passes as digits of at most 10 bits allow, the digit width spread evenly over them
    const int passes = bits <= 0 ? 1 : (bits + 9) / 10;
    const int dbits = bits <= 0 ? 1 : (bits + passes - 1) / passes;
    const int nbuckets = 1 << dbits;
    const unsigned dmask = (unsigned)nbuckets - 1u;
    SGB_TRY(hist.ensure(((size_t)ntiles + 1) * nbuckets * 4));
    uint32_t* h = hist.as<uint32_t>();
    uint32_t* tot = h + (size_t)ntiles * nbuckets;
    K* kbuf[2] = {kA.as<K>(), kB.as<K>()};
    uint32_t* vbuf[2] = {vA.as<uint32_t>(), vB.as<uint32_t>()};
    // pass 0 takes the staged ids as they are and ranks the insertion index itself
    SGB_TRY((radix_pass<RR, int64_t, K>(g->pend_lin.as<int64_t>(), nullptr, kbuf[0], vbuf[0], n, 0, dmask, nbuckets, h, tot,
                                    ntiles, s)));
    for (int ps = 1; ps < passes; ++ps)
        SGB_TRY((radix_pass<RR, K, K>(kbuf[(ps + 1) & 1], vbuf[(ps + 1) & 1], kbuf[ps & 1], vbuf[ps & 1], n, ps * dbits, dmask,
                                  nbuckets, h, tot, ntiles, s)));
    *vals_out = vbuf[(passes + 1) & 1];
    *keys_out = kbuf[(passes + 1) & 1];
    return SGB_OK;
}

template <typename K>
static int flush_impl(sgb_grid* g, const int* ops, int bits, cudaStream_t s) {
    const int64_t n = g->npend;
    const int bs = g->geo.bs;
    const int bs_shift = bs == 512 ? 9 : 6;
    const bool small = n <= kSmMax;

    DevBuf& tiles = g->scratch[7];
    DevBuf& ubuf = g->scratch[9];
    DevBuf& uval = g->scratch[10];
    DevBuf& cnt = g->scratch[11];
    const int64_t htiles = (n + kHdTile - 1) / kHdTile, ltiles = (n + kLkTile - 1) / kLkTile;
    SGB_TRY(tiles.ensure((size_t)(htiles + ltiles) * 8));
    SGB_TRY(cnt.ensure(64));
    uint2* htile = tiles.as<uint2>();
    uint2* ltile = htile + htiles;
    uint32_t* counters = cnt.as<uint32_t>();  // [0] U, [1] B, [2] NB, [3] error word

    // unique points / chunks: at most n of each
    size_t uval_bytes = 0;
    for (int p = 0; p < g->nprop; ++p) uval_bytes += ((size_t)n * elem_size(g->ptype[p]) + 15) & ~(size_t)15;
    SGB_TRY(uval.ensure(uval_bytes + 64));
    // ubuf: upt[n] uint2 | ublk_key[n] int64 | place[n] int64 | newkeys[n] int64
    SGB_TRY(ubuf.ensure((size_t)n * 32 + 256));
    uint2* upt = ubuf.as<uint2>();
    int64_t* ublk_key = reinterpret_cast<int64_t*>(upt + n);
    int64_t* place = ublk_key + n;
    int64_t* newkeys = place + n;

    PropSet vals{}, upv{}, data{};
    vals.nprop = upv.nprop = data.nprop = g->nprop;
    size_t off = 0;
    int any_listed = 0;
    for (int p = 0; p < g->nprop; ++p) {
        vals.p[p] = g->pend_val[p].as<unsigned char>();
        upv.p[p] = uval.as<unsigned char>() + off;
        off += ((size_t)n * elem_size(g->ptype[p]) + 15) & ~(size_t)15;
        vals.type[p] = upv.type[p] = data.type[p] = g->ptype[p];
        vals.op[p] = upv.op[p] = data.op[p] = ops[p];
        any_listed |= ops[p] != SGB_OP_NONE;
    }
    for (int p = 0; p < g->nprop; ++p) data.p[p] = g->data[p].as<unsigned char>();
    if (small) {
        const int passes = std::max(1, (bits + 7) / 8), dbits = std::max(1, (bits + passes - 1) / passes);
        constexpr size_t smem = small_smem<K>();
        SGB_CUDA(cudaFuncSetAttribute(k_flush_small<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        k_flush_small<K><<<1, kSmThreads, smem, s>>>(g->pend_lin.as<int64_t>(), (int)n, passes, dbits, bs_shift, vals, upv, data,
                                                     g->mask.as<uint8_t>(), any_listed, g->keys.as<int64_t>(), g->n, upt,
                                                     ublk_key, place, ltile, counters, g->err.as<unsigned>());
    } else {
        K* sk = nullptr;
        uint32_t* sidx = nullptr;
        if (n <= (int64_t)g->num_sms * 4 * kRsThreads * kRsRoundsFew)
            SGB_TRY((radix_sort<kRsRoundsFew, K>(g, n, bits, &sk, &sidx, s)));
        else
            SGB_TRY((radix_sort<kRsRounds, K>(g, n, bits, &sk, &sidx, s)));
        k_heads_count<K><<<(unsigned)htiles, kHdThreads, 0, s>>>(sk, n, bs_shift, htile);
        k_tile_scan<0><<<1, 1024, 0, s>>>(htile, htiles, counters, nullptr);
        k_fold<K><<<(unsigned)htiles, kHdThreads, 0, s>>>(sk, sidx, n, bs_shift, htile, vals, upv, upt, ublk_key);
        k_lookup<<<(unsigned)std::min<int64_t>(ltiles, (int64_t)g->num_sms * 2), kLkTile, 0, s>>>(
            ublk_key, counters, g->keys.as<int64_t>(), g->n, place, ltile);
        k_tile_scan<1><<<1, 1024, 0, s>>>(ltile, 0, counters, g->err.as<unsigned>());
    }
    SGB_CUDA(cudaGetLastError());
    SGB_TRY(g->hscratch.ensure(64));
    SGB_CUDA(cudaMemcpyAsync(g->hscratch.p, counters, 16, cudaMemcpyDeviceToHost, s));
    SGB_CUDA(cudaStreamSynchronize(s));
    const int64_t U = ((uint32_t*)g->hscratch.p)[0];
    const int64_t B = ((uint32_t*)g->hscratch.p)[1];
    const int64_t NB = ((uint32_t*)g->hscratch.p)[2];
    // out-of-domain points were flagged at insert time; nothing of the map has been touched yet
    const unsigned e = ((uint32_t*)g->hscratch.p)[3];
    if (e & (kErrOutOfDomain | kErrPoolOverflow)) {
        SGB_CUDA(cudaMemsetAsync(g->err.p, 0, 4, s));
        set_error((e & kErrOutOfDomain)
                      ? "an inserted point lies outside the grid domain; the staged inserts were dropped"
                      : "an insert pool counted more points than its slots; the staged inserts were dropped");
        return SGB_ERANGE;
    }

    if (NB > 0) {
        const int64_t nold = g->n, nn_ = nold + NB;
        // second buffer set for the new map (contents are rebuilt): kept while it holds the map,
        // otherwise allocated for twice the map, so that a growing map reallocates rarely (each
        // reallocation frees and maps gigabytes and stalls the device)
        int64_t cap2 = std::min<int64_t>((int64_t)(g->keys2.bytes / 8), (int64_t)(g->mask2.bytes / bs) - 1);
        for (int p = 0; p < g->nprop; ++p)
            cap2 = std::min<int64_t>(cap2, (int64_t)(g->data2[p].bytes / ((size_t)bs * elem_size(g->ptype[p]))) - 1);
        if (cap2 < nn_) {
            cap2 = std::max<int64_t>(2 * nn_, 16);
            SGB_TRY(g->keys2.ensure((size_t)cap2 * 8));
            SGB_TRY(g->mask2.ensure((size_t)(cap2 + 1) * bs));
            for (int p = 0; p < g->nprop; ++p)
                SGB_TRY(g->data2[p].ensure((size_t)(cap2 + 1) * bs * elem_size(g->ptype[p])));
        }
        DevBuf& posbuf = g->scratch[5];
        SGB_TRY(posbuf.ensure((size_t)nn_ * 4 + 64));
        int32_t* srcpos = posbuf.as<int32_t>();
        k_merge_pos<<<(unsigned)((B + kLkTile - 1) / kLkTile), kLkTile, 0, s>>>(ublk_key, B, place, ltile, newkeys,
                                                                                 g->keys2.as<int64_t>(), srcpos);
        if (nold > 0)
            k_old_pos<<<nblk(nold), 256, 0, s>>>(g->keys.as<int64_t>(), nold, newkeys, NB, g->keys2.as<int64_t>(), srcpos);
        SGB_CUDA(cudaGetLastError());
        MapSet ms{};
        ms.count = g->nprop + 1;
        for (int p = 0; p <= g->nprop; ++p) {
            const int es = p < g->nprop ? elem_size(g->ptype[p]) : 1;
            ms.src[p] = p < g->nprop ? g->data[p].as<uint4>() : g->mask.as<uint4>();
            ms.dst[p] = p < g->nprop ? g->data2[p].as<uint4>() : g->mask2.as<uint4>();
            uint64_t pat = 0;
            if (p < g->nprop) std::memcpy(&pat, g->bck[p], es);
            ms.fill[p] = replicate16(pat, es);
            while ((16 << ms.shift[p]) < bs * es) ++ms.shift[p];  // chunk edges are powers of two
        }
        k_merge_map<<<(unsigned)std::min<int64_t>((nn_ + 8) / 8, (int64_t)g->num_sms * 8), 256, 0, s>>>(ms, srcpos, nn_);
        SGB_CUDA(cudaGetLastError());
        // swap buffer sets
        std::swap(g->keys, g->keys2);
        std::swap(g->mask, g->mask2);
        for (int p = 0; p < g->nprop; ++p) {
            std::swap(g->data[p], g->data2[p]);
            if (g->exposed[p] && nold > 0) g->clean[p] = false;  // what the caller wrote has moved along
            g->exposed[p] = false;
        }
        g->cap = cap2;
        g->n = nn_;
    }
    if (small && NB == 0) return SGB_OK;  // written back already
    for (int p = 0; p < g->nprop; ++p) data.p[p] = g->data[p].as<unsigned char>();
    k_scatter<<<nblk(U), 256, 0, s>>>(upt, U, bs_shift, place, upv, data, g->mask.as<uint8_t>(), any_listed);
    SGB_CUDA(cudaGetLastError());
    return SGB_OK;
}

}  // namespace sgb

using namespace sgb;

extern "C" int sgb_flush(sgb_grid* g, const int* ops, sgb_stream stream) {
    if (!g || !ops) return SGB_EINVAL;
    for (int p = 0; p < g->nprop; ++p) {
        if (ops[p] < SGB_OP_NONE || ops[p] > SGB_OP_OR) return SGB_EINVAL;
        if (ops[p] == SGB_OP_OR && (g->ptype[p] == SGB_F32 || g->ptype[p] == SGB_F64)) return SGB_EINVAL;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (g->npend == 0) return SGB_OK;
    const int64_t maxlin = key_space(g->geo) * g->geo.bs;
    int bits = 0;
    while (bits < 63 && (int64_t(1) << bits) < maxlin) ++bits;
    int st;
    if (bits <= 32) st = flush_impl<uint32_t>(g, ops, bits, s);
    else st = flush_impl<uint64_t>(g, ops, bits, s);
    g->npend = 0;
    if (st == SGB_ERANGE) return st;  // rejected: the map is as it was, and so is what was made from it
    g->nn_valid[0] = g->nn_valid[1] = false;
    g->nnhash_ok = false;
    g->bits_valid = false;
    g->epts_valid = false;
    return st;
}
