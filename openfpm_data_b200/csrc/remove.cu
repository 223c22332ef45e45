// Point removal by boxes and enumeration of the existing points.
//
// remove(box) + removePoints (src/SparseGridGpu/SparseGridGpu.hpp:3417-3489,
// 3528-3531; SparseGridGpu_kernels.cuh:1235-1340): every existing point
// inside one of the queued boxes loses its mask byte; the chunks stay.  The
// reference tests points against Box<dim, unsigned int>, so the int boxes are
// converted to unsigned int here too.  The removed points also get their
// properties' backgrounds, which keeps the grid's background invariant.
//
// The enumeration lists the existing points in (chunk position, offset in the
// chunk) order, the order in which the reference's iterators
// (src/SparseGridGpu/Iterators/SparseGridGpu_iterator.hpp:17-304) visit them.
#include <cstring>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace sgb {

struct UBox {
    uint32_t lo[3], hi[3];
};

struct BckSet {
    unsigned char* p[kMaxProps];
    uint64_t pat[kMaxProps];
    int es[kMaxProps];
    int nprop;
};

// Boxes of a call: in the launch's parameters while they fit, else in device memory.
constexpr int kParamBoxes = 64;
struct UBoxes {
    UBox b[kParamBoxes];
};

// A CTA takes 32 chunks: its first warp tests them against the boxes, one chunk per lane, then the warps share
// the chunks that a box touches, bs / 32 consecutive points per lane.  (A CTA per chunk, tests and all: 53 us
// for six one-layer slabs of a 512^3 grid of 18.9 K chunks, 17 us so.)  A box cuts a chunk's x rows to one bit
// mask, so a touched chunk costs a few operations per box and row.  Boxes are taken 64 at a time through shared
// memory, with a bit per chunk for each that meets it: a grid of few chunks has few CTAs, and each would wait for
// memory box by box (1000 boxes on 216 chunks, the whole call: 582 us, 1009 with boxes read from memory, 660 with a
// CTA per chunk).
template <int P>  // points per lane: 16 (8^3 chunks) or 2 (4^3)
__global__ void __launch_bounds__(256) k_remove_boxes(const int64_t* __restrict__ keys, int64_t n, Geometry geo, uint8_t* mask,
                                                       const __grid_constant__ UBoxes pb, const UBox* __restrict__ db, int nb,
                                                       const __grid_constant__ BckSet bck) {
    constexpr int bs = P * 32, e = P == 16 ? 8 : 4;
    __shared__ int hits[32];
    __shared__ uint32_t org[32][3];
    __shared__ unsigned long long touched[32];  // the boxes of the round that meet the chunk
    __shared__ int nhits;
    __shared__ UBox boxes[kParamBoxes];  // indexed reads of the parameters would go through memory
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t c0 = (int64_t)blockIdx.x * 32;
    if (warp == 0 && c0 + lane < n) {
        int64_t o[3];
        chunk_origin(geo, keys[c0 + lane], o);
        for (int d = 0; d < 3; ++d) org[lane][d] = (uint32_t)o[d];
    }
    for (int k0 = 0; k0 < nb; k0 += kParamBoxes) {
        const int nk = nb - k0 < kParamBoxes ? nb - k0 : kParamBoxes;
        const uint32_t* from = reinterpret_cast<const uint32_t*>(nb <= kParamBoxes ? pb.b : db + k0);
        __syncthreads();  // the round before has read its boxes
        for (int i = threadIdx.x; i < nk * 6; i += 256) reinterpret_cast<uint32_t*>(boxes)[i] = from[i];
        __syncthreads();
        if (warp == 0) {
            unsigned long long in = 0;
            if (c0 + lane < n) {
                uint32_t clo[3];
                for (int d = 0; d < 3; ++d) clo[d] = org[lane][d];
                for (int k = 0; k < nk; ++k) {
                    bool t = true;
                    for (int d = 0; d < 3; ++d) t = t && !(clo[d] + (e - 1) < boxes[k].lo[d] || clo[d] > boxes[k].hi[d]);
                    in |= (unsigned long long)t << k;
                }
                touched[lane] = in;
            }
            const unsigned t = __ballot_sync(0xffffffffu, in != 0);
            if (in) hits[__popc(t & lanemask_lt())] = lane;
            if (lane == 0) nhits = __popc(t);
        }
        __syncthreads();
        for (int h = warp; h < nhits; h += 8) {
            const int j = hits[h];
            const int64_t first = (c0 + j) * bs + lane * P;
            union {
                uint4 v;
                uint16_t s;
                uint8_t b[16];
            } m;
            if (P == 16) m.v = *reinterpret_cast<const uint4*>(mask + first);
            else m.s = *reinterpret_cast<const uint16_t*>(mask + first);
            uint32_t gone = 0;  // the lane's points inside a box, then the existing ones of them
            for (unsigned long long left = touched[j]; left; left &= left - 1) {
                const int k = __ffsll((long long)left) - 1;
                int lo[3], hi[3];  // the box in the chunk's coordinates, clipped to it
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const int64_t o = org[j][d], l = (int64_t)boxes[k].lo[d] - o, u = (int64_t)boxes[k].hi[d] - o;
                    lo[d] = l < 0 ? 0 : l > e ? e : (int)l;
                    hi[d] = u < -1 ? -1 : u > e - 1 ? e - 1 : (int)u;
                }
                if (lo[0] > hi[0]) continue;
                const uint32_t xm = (2u << hi[0]) - (1u << lo[0]);
                if (P == 16) {  // two x rows
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int y = (2 * lane + r) & 7, z = (2 * lane + r) >> 3;
                        if (y >= lo[1] && y <= hi[1] && z >= lo[2] && z <= hi[2]) gone |= xm << (8 * r);
                    }
                } else {  // half an x row
                    const int y = lane >> 1 & 3, z = lane >> 3;
                    if (y >= lo[1] && y <= hi[1] && z >= lo[2] && z <= hi[2]) gone |= xm >> (2 * (lane & 1)) & 3u;
                }
            }
            uint32_t ex = 0;
#pragma unroll
            for (int i = 0; i < P; ++i) ex |= (uint32_t)(m.b[i] & 1) << i;
            gone &= ex;
            if (!gone) continue;
#pragma unroll
            for (int i = 0; i < P; ++i)
                if (gone >> i & 1u) m.b[i] = 0;
            if (P == 16) *reinterpret_cast<uint4*>(mask + first) = m.v;
            else *reinterpret_cast<uint16_t*>(mask + first) = m.s;
            for (int p = 0; p < bck.nprop; ++p) {
                unsigned char* q = bck.p[p] + (size_t)first * bck.es[p];
                const uint64_t pat = bck.pat[p];
                for (uint32_t w = gone; w; w &= w - 1) {
                    const int i = __ffs(w) - 1;
                    if (bck.es[p] == 4) reinterpret_cast<uint32_t*>(q)[i] = (uint32_t)pat;
                    else if (bck.es[p] == 8) reinterpret_cast<uint64_t*>(q)[i] = pat;
                    else q[i] = (unsigned char)pat;
                }
            }
        }
    }
}

__device__ __forceinline__ bool in_ibox(const int64_t* box, int64_t x, int64_t y, int64_t z) {
    return x >= box[0] && x <= box[3] && y >= box[1] && y <= box[4] && z >= box[2] && z <= box[5];
}

struct IBox {
    int64_t b[6];
    int has;
};

// Existing points per chunk (inside the box when there is one): one warp per chunk.
__global__ void k_count_points(const int64_t* __restrict__ keys, int64_t n, Geometry geo, const uint8_t* __restrict__ mask,
                               IBox box, uint32_t* counts) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int bs = geo.bs, e = geo.edge;
    for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; c < n; c += nw) {
        int64_t o[3];
        chunk_origin(geo, keys[c], o);
        uint32_t cnt = 0;
        for (int pt = lane; pt < bs; pt += 32) {
            bool ex = mask[c * bs + pt] & 1;
            if (box.has) ex = ex && in_ibox(box.b, o[0] + pt % e, o[1] + (pt / e) % e, o[2] + pt / (e * e));
            cnt += __popc(__ballot_sync(0xffffffffu, ex));
        }
        if (lane == 0) counts[c] = cnt;
    }
}

// Coordinates of those points at their scanned offsets, in offset order inside each chunk.
__global__ void k_emit_points(const int64_t* __restrict__ keys, int64_t n, Geometry geo, const uint8_t* __restrict__ mask,
                              IBox box, const uint32_t* __restrict__ offs, int32_t* out) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int bs = geo.bs, e = geo.edge;
    for (int64_t c = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; c < n; c += nw) {
        int64_t o[3];
        chunk_origin(geo, keys[c], o);
        uint32_t base = offs[c];
        for (int pt = lane; pt < bs; pt += 32) {
            const int64_t x = o[0] + pt % e, y = o[1] + (pt / e) % e, z = o[2] + pt / (e * e);
            bool ex = mask[c * bs + pt] & 1;
            if (box.has) ex = ex && in_ibox(box.b, x, y, z);
            const unsigned bal = __ballot_sync(0xffffffffu, ex);
            if (ex) {
                const uint32_t k = base + __popc(bal & lanemask_lt());
                out[(size_t)k * 3 + 0] = (int32_t)x;
                out[(size_t)k * 3 + 1] = (int32_t)y;
                out[(size_t)k * 3 + 2] = (int32_t)z;
            }
            base += __popc(bal);
        }
    }
}

static unsigned warp_blocks(const sgb_grid* g, int64_t n) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((int64_t)g->num_sms * 8, (n + 7) / 8));
}

}  // namespace sgb

using namespace sgb;

extern "C" int sgb_remove_boxes(sgb_grid* g, int64_t nboxes, const int64_t* boxes_host, sgb_stream stream) {
    if (!g || nboxes < 0 || (nboxes > 0 && !boxes_host)) return SGB_EINVAL;
    if (g->geo.dim != 3) {
        set_error("removal by boxes is implemented for 3-D grids");
        return SGB_ENOTSUP;
    }
    if (nboxes == 0 || g->n == 0) return SGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    std::vector<UBox> hb((size_t)nboxes);
    for (int64_t k = 0; k < nboxes; ++k)
        for (int d = 0; d < 3; ++d) {
            hb[k].lo[d] = (uint32_t)(int32_t)boxes_host[k * 6 + d];  // Box<dim,int> -> Box<dim,unsigned int>
            hb[k].hi[d] = (uint32_t)(int32_t)boxes_host[k * 6 + 3 + d];
        }
    UBoxes pb{};
    const UBox* db = nullptr;
    if (nboxes <= kParamBoxes) {
        std::memcpy(pb.b, hb.data(), hb.size() * sizeof(UBox));
    } else {
        SGB_TRY(g->scratch[0].ensure(hb.size() * sizeof(UBox)));
        SGB_TRY(g->hscratch.ensure(hb.size() * sizeof(UBox)));
        std::memcpy(g->hscratch.p, hb.data(), hb.size() * sizeof(UBox));
        SGB_CUDA(cudaMemcpyAsync(g->scratch[0].p, g->hscratch.p, hb.size() * sizeof(UBox), cudaMemcpyHostToDevice, s));
        db = g->scratch[0].as<UBox>();
    }
    BckSet bk{};
    bk.nprop = g->nprop;
    for (int p = 0; p < g->nprop; ++p) {
        bk.p[p] = g->data[p].as<unsigned char>();
        bk.pat[p] = bck_pattern(g, p);
        bk.es[p] = elem_size(g->ptype[p]);
    }
    const unsigned blocks = (unsigned)((g->n + 31) / 32);
    if (g->geo.edge == 8)
        k_remove_boxes<16><<<blocks, 256, 0, s>>>(g->keys.as<int64_t>(), g->n, g->geo, g->mask.as<uint8_t>(), pb, db,
                                                  (int)nboxes, bk);
    else
        k_remove_boxes<2><<<blocks, 256, 0, s>>>(g->keys.as<int64_t>(), g->n, g->geo, g->mask.as<uint8_t>(), pb, db,
                                                 (int)nboxes, bk);
    SGB_CUDA(cudaGetLastError());
    // the host copy of the boxes must outlive the asynchronous upload
    SGB_CUDA(cudaStreamSynchronize(s));
    // existence changed; chunks, neighbours and backgrounds did not
    g->bits_valid = false;
    g->epts_valid = false;
    return SGB_OK;
}

extern "C" int sgb_existing_points(sgb_grid* g, const int64_t* box_host, int32_t* coords_dev, int64_t capacity,
                                   int64_t* count, sgb_stream stream) {
    if (!g || !count || capacity < 0 || (capacity > 0 && !coords_dev)) return SGB_EINVAL;
    if (g->geo.dim != 3) {
        set_error("point enumeration is implemented for 3-D grids");
        return SGB_ENOTSUP;
    }
    *count = 0;
    if (g->n == 0) return SGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    IBox box{};
    if (box_host) {
        std::memcpy(box.b, box_host, sizeof(box.b));
        box.has = 1;
    }
    const int64_t n = g->n;
    SGB_TRY(g->scratch[1].ensure((size_t)n * 4 + 16));
    SGB_TRY(g->scratch[2].ensure((size_t)(n + 1) * 4 + 16));
    uint32_t* counts = g->scratch[1].as<uint32_t>();
    uint32_t* offs = g->scratch[2].as<uint32_t>();
    k_count_points<<<warp_blocks(g, n), 256, 0, s>>>(g->keys.as<int64_t>(), n, g->geo, g->mask.as<uint8_t>(), box,
                                                     counts);
    SGB_CUDA(cudaGetLastError());
    SGB_TRY(scan_exclusive_u32(counts, offs, n, offs + n, &g->scratch[6], s));
    SGB_TRY(g->hscratch.ensure(64));
    SGB_CUDA(cudaMemcpyAsync(g->hscratch.p, offs + n, 4, cudaMemcpyDeviceToHost, s));
    SGB_CUDA(cudaStreamSynchronize(s));
    const int64_t total = *(uint32_t*)g->hscratch.p;
    *count = total;
    if (total == 0 || capacity < total) return SGB_OK;  // the caller sizes the buffer from *count
    k_emit_points<<<warp_blocks(g, n), 256, 0, s>>>(g->keys.as<int64_t>(), n, g->geo, g->mask.as<uint8_t>(), box,
                                                    offs, coords_dev);
    SGB_CUDA(cudaGetLastError());
    return SGB_OK;
}
