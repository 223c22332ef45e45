// Packing of sub-boxes of a grid for ghost exchange, and unpacking.
//
// Format of one packed box, the reference's (SparseGridGpu.hpp:2984-3040
// packCalculate, 3244-3300 pack, SparseGridGpu_kernels.cuh:1658-1697
// pack_data), with indexT = int64:
//   uint64 n_cnk;  int32 start[3];  int32 size[3];
//   int64  chunk_id[n_cnk]                 (the chunks holding packed points, index order)
//   uint32 scan[n_cnk + 1]                 (first packed point of each chunk; scan[n_cnk] = n_pnt)
//   data: for each packed property, n_pnt elements of its type, back to back
//   int16  offset[n_pnt]                   (the point's offset inside its chunk)
//   uint8  mask[n_pnt]
// where the scan, the data block, the offsets and the masks are each padded
// to a multiple of 8 bytes.  Packed points are the existing points inside the
// inclusive box.  Inside a chunk the reference orders them by a shared-memory
// atomic counter (any order); here they are in offset order.
//
// Unpacking stages the points of every box of a buffer as inserts at their
// coordinates plus a shift (the caller then flushes with the reduction it
// wants, e.g. sRight_ to overwrite): the unpack-then-merge step of the
// reference's ghost exchange (unpack 3665-3750 + removeAddUnpackFinalize).
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.cuh"
#include "internal.h"

namespace sgb {

__host__ __device__ inline int64_t pad8(int64_t b) { return (b + 7) & ~(int64_t)7; }

struct PackLayout {
    int64_t n_cnk, n_pnt;
    int64_t off_ids, off_scan, off_data, off_offs, off_mask, bytes, data_bytes;
    int64_t prop_off[kMaxProps];
};

__host__ __device__ inline PackLayout layout_of(int64_t n_cnk, int64_t n_pnt, int np, const int* es) {
    PackLayout L{};
    L.n_cnk = n_cnk;
    L.n_pnt = n_pnt;
    int64_t o = 8 + 2 * 3 * 4;
    L.off_ids = o;
    o += 8 * n_cnk;
    L.off_scan = o;
    o += pad8(4 * (n_cnk + 1));
    L.off_data = o;
    int64_t d = 0;
    for (int p = 0; p < np; ++p) {
        L.prop_off[p] = d;
        d += n_pnt * es[p];
    }
    L.data_bytes = d;
    o += pad8(d);
    L.off_offs = o;
    o += pad8(2 * n_pnt);
    L.off_mask = o;
    o += pad8(n_pnt);
    L.bytes = o;
    return L;
}

__device__ __forceinline__ void origin_of(const Geometry& geo, int64_t key, int64_t* o) { chunk_origin(geo, key, o); }

struct Box6 {
    int64_t b[6];
};

// A box and the block coordinates of the chunks it meets: lo = floor(low / edge), hi = floor(high / edge),
// clamped to the grid's.
struct HitBox {
    Box6 box;
    int64_t lo[3], hi[3];
};

// The packed points come from few chunks, so the chunks are found first: which chunks each box meets, as bitmaps
// of 32 chunks (a warp per 32 chunks, a lane per chunk, all boxes), then a list of the hits in (box, chunk) order.
// The point work that follows takes a warp per hit and not a warp per chunk of the grid (six one-layer slabs of a
// 512^3 grid meet 1.7 K of 6 x 18.9 K (box, chunk) pairs: count 54 -> 28 us, emission 64 -> 14 us).  The boxes are
// split over the grid's second dimension, since few chunks make few warps (request and pack of 200 boxes on 216
// chunks 555 us with all boxes in one warp, 335 so).
__global__ void __launch_bounds__(256) k_pack_hits(const int64_t* __restrict__ keys, int64_t n, Geometry geo,
                                                    const HitBox* __restrict__ boxes, int nb, int64_t words,
                                                    uint32_t* __restrict__ bits, uint32_t* __restrict__ cnt) {
    const int lane = threadIdx.x & 31;
    const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    if (w >= words) return;
    const int64_t c = w * 32 + lane;
    int64_t bc[3] = {-1, -1, -1};  // below every box's range
    if (c < n) block_coords(geo, keys[c], bc);
    for (int k = blockIdx.y; k < nb; k += gridDim.y) {
        const HitBox& b = boxes[k];
        const bool in = bc[0] >= b.lo[0] && bc[0] <= b.hi[0] && bc[1] >= b.lo[1] && bc[1] <= b.hi[1] && bc[2] >= b.lo[2] &&
                        bc[2] <= b.hi[2];
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (lane == 0) {
            bits[(int64_t)k * words + w] = m;
            cnt[(int64_t)k * words + w] = (uint32_t)__popc(m);
        }
    }
}

struct Hit {
    int32_t c;    // chunk position
    int32_t box;
};

__global__ void k_pack_list(const uint32_t* __restrict__ bits, const uint32_t* __restrict__ start, int64_t words,
                            int64_t len, Hit* __restrict__ hits) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= len) return;
    uint32_t m = bits[i], h = start[i];
    const int32_t k = (int32_t)(i / words), c0 = (int32_t)(i % words) * 32;
    while (m) {
        hits[h++] = Hit{c0 + __ffs(m) - 1, k};
        m &= m - 1;
    }
}

// The part of a box inside a chunk, in the chunk's own coordinates (empty when lo > hi in a dimension).
struct LocalBox {
    int lo[3], hi[3];
};
__device__ __forceinline__ LocalBox local_box(const Geometry& geo, int64_t key, const Box6& bx) {
    int64_t o[3];
    chunk_origin(geo, key, o);
    LocalBox L;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int64_t lo = bx.b[d] - o[d], hi = bx.b[d + 3] - o[d];
        L.lo[d] = lo < 0 ? 0 : lo > 8 ? 8 : (int)lo;
        L.hi[d] = hi < -1 ? -1 : hi > 8 ? 8 : (int)hi;
    }
    return L;
}
__device__ __forceinline__ bool inside_local(const LocalBox& L, int pt, int e, int sh) {
    const int x = pt & (e - 1), y = pt >> sh & (e - 1), z = pt >> 2 * sh;
    return x >= L.lo[0] && x <= L.hi[0] && y >= L.lo[1] && y <= L.hi[1] && z >= L.lo[2] && z <= L.hi[2];
}

// Per hit: its points inside the box.  A CTA takes 32 consecutive hits, a warp each (grid-stride; the number of
// hits is on the device), and leaves the points and non-empty chunks before each hit in the tile, and the tile's
// totals.
constexpr int kHitTile = 32;
__global__ void __launch_bounds__(kHitTile * 32) k_pack_points(const Hit* __restrict__ hits, const uint32_t* __restrict__ nhits,
                                                      const int64_t* __restrict__ keys, Geometry geo,
                                                      const uint8_t* __restrict__ mask, const HitBox* __restrict__ boxes,
                                                      uint2* __restrict__ pre, uint2* __restrict__ tiles) {
    __shared__ uint32_t cnt[kHitTile];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t H = *nhits;
    const int bs = geo.bs, e = geo.edge, sh = e == 8 ? 3 : 2;
    for (int64_t t = blockIdx.x; t * kHitTile < H; t += gridDim.x) {
        const int64_t h = t * kHitTile + warp;
        uint32_t c = 0;
        if (h < H) {
            const Hit q = hits[h];
            const LocalBox L = local_box(geo, keys[q.c], boxes[q.box].box);
            const uint8_t* m = mask + (int64_t)q.c * bs;
            uint8_t mv[16];  // the lane's mask bytes, all loads in flight at once (bs <= 512)
#pragma unroll
            for (int i = 0; i < 16; ++i) mv[i] = lane + 32 * i < bs ? m[lane + 32 * i] : 0;
#pragma unroll
            for (int i = 0; i < 16; ++i) c += (mv[i] & 1) && inside_local(L, lane + 32 * i, e, sh);
            c = __reduce_add_sync(0xffffffffu, c);
        }
        if (lane == 0) cnt[warp] = c;
        __syncthreads();
        if (warp == 0) {  // points and non-empty chunks before each
            const uint32_t a = cnt[lane];
            uint32_t x = a, y = a != 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t u = __shfl_up_sync(0xffffffffu, x, o), v = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= o) {
                    x += u;
                    y += v;
                }
            }
            const int64_t hl = t * kHitTile + lane;
            if (hl < H) pre[hl] = make_uint2(x - a, y - (a != 0));
            if (lane == 31) tiles[t] = make_uint2(x, y);
        }
        __syncthreads();
    }
}

// Exclusive scan of the tiles (one CTA, in place; tiles[number of tiles] = the totals), then the row starts:
// rows[2 k], rows[2 k + 1] = points and non-empty chunks before box k (k = nb: all).
__global__ void __launch_bounds__(1024) k_pack_rows(uint2* tiles, const uint32_t* __restrict__ nhits,
                                                     const uint32_t* __restrict__ start, const uint2* __restrict__ pre,
                                                     int64_t words, int nb, uint32_t* rows) {
    __shared__ uint32_t wx[32], wy[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t H = *nhits, nt = (H + kHitTile - 1) / kHitTile;
    uint32_t cx = 0, cy = 0;
    for (int64_t t0 = 0; t0 < nt; t0 += 1024) {
        const int64_t t = t0 + threadIdx.x;
        const uint2 v = t < nt ? tiles[t] : make_uint2(0, 0);
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
        if (t < nt) tiles[t] = make_uint2(bx + x - v.x, by + y - v.y);
        __syncthreads();
    }
    for (int k = threadIdx.x; k <= nb; k += 1024) {
        const int64_t h = k < nb ? (int64_t)start[(int64_t)k * words] : H;
        uint2 r = make_uint2(cx, cy);
        if (h < H) {
            const uint2 t = tiles[h / kHitTile], p = pre[h];
            r = make_uint2(t.x + p.x, t.y + p.y);
        }
        rows[2 * k] = r.x;
        rows[2 * k + 1] = r.y;
    }
    if (threadIdx.x == 0) tiles[nt] = make_uint2(cx, cy);
}

struct PackProps {
    const unsigned char* src[kMaxProps];
    int es[kMaxProps];
    int wide[kMaxProps];  // 1: the property's packed block is aligned to its element size
    int np;
};

// One packed box: its place in the output, its layout, its box.
struct PackBox {
    Box6 box;
    int64_t base;  // byte offset of the box in the output
    PackLayout L;
    uint32_t pnt0, cnk0;  // the box's row starts in the scans
};

// A warp per hit.
__global__ void __launch_bounds__(256) k_pack_emit(const Hit* __restrict__ hits, const uint32_t* __restrict__ nhits,
                                                    const int64_t* __restrict__ keys, Geometry geo,
                                                    const uint8_t* __restrict__ mask, const PackBox* __restrict__ pbs,
                                                    const uint2* __restrict__ pre, const uint2* __restrict__ tiles,
                                                    PackProps pp, unsigned char* out) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5, H = *nhits;
    const int bs = geo.bs, e = geo.edge, sh = e == 8 ? 3 : 2;
    for (int64_t h = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; h < H; h += nw) {
        const Hit q = hits[h];
        const int64_t c = q.c, key = keys[c];
        const PackBox& P = pbs[q.box];
        const LocalBox L = local_box(geo, key, P.box);
        uint8_t mv[16];  // the lane's mask bytes, all loads in flight at once (bs <= 512)
#pragma unroll
        for (int i = 0; i < 16; ++i) mv[i] = lane + 32 * i < bs ? mask[c * bs + lane + 32 * i] : 0;
        uint32_t any = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if ((mv[i] & 1) && inside_local(L, lane + 32 * i, e, sh)) any |= 1u << i;
        if (__reduce_or_sync(0xffffffffu, any) == 0) continue;  // no packed point in this chunk (uniform)
        const uint2 t = tiles[h / kHitTile], p0 = pre[h];
        uint32_t base = t.x + p0.x - P.pnt0;
        const uint32_t slot = t.y + p0.y - P.cnk0;
        unsigned char* b = out + P.base;
        if (lane == 0) {
            reinterpret_cast<int64_t*>(b + P.L.off_ids)[slot] = key;
            reinterpret_cast<uint32_t*>(b + P.L.off_scan)[slot] = base;
        }
        int16_t* offs = reinterpret_cast<int16_t*>(b + P.L.off_offs);
        uint8_t* msk = b + P.L.off_mask;
        uint32_t place[16];  // the lane's points' places in the box
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const unsigned bal = __ballot_sync(0xffffffffu, any >> i & 1u);
            place[i] = base + __popc(bal & lanemask_lt());
            base += __popc(bal);
        }
        const int64_t idx = c * bs + lane;
        for (int p = 0; p < pp.np; ++p) {
            unsigned char* d = b + P.L.off_data + P.L.prop_off[p];
            const unsigned char* sp = pp.src[p];
            auto copy = [&](auto zero) {  // all of the lane's values in flight at once
                using T = decltype(zero);
                T v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = any >> i & 1u ? reinterpret_cast<const T*>(sp)[idx + 32 * i] : zero;
#pragma unroll
                for (int i = 0; i < 16; ++i)
                    if (any >> i & 1u) {
                        if (pp.wide[p]) {
                            reinterpret_cast<T*>(d)[place[i]] = v[i];
                        } else {
                            for (int u = 0; u < (int)sizeof(T); ++u)
                                d[(int64_t)place[i] * sizeof(T) + u] = (unsigned char)((uint64_t)v[i] >> (8 * u));
                        }
                    }
            };
            if (pp.es[p] == 4) copy(uint32_t(0));
            else if (pp.es[p] == 8) copy(uint64_t(0));
            else copy(uint8_t(0));
        }
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (any >> i & 1u) {
                offs[place[i]] = (int16_t)(lane + 32 * i);
                msk[place[i]] = mv[i];
            }
    }
}

// Per box: the header, scan[n_cnk] = n_pnt, and zeros in the padding tails.
__global__ void k_pack_finish(const PackBox* __restrict__ pbs, int nb, int32_t sx, int32_t sy, int32_t sz,
                              unsigned char* out) {
    const int k = blockIdx.x;
    if (k >= nb) return;
    const PackBox& P = pbs[k];
    unsigned char* b = out + P.base;
    const PackLayout& L = P.L;
    const int t = threadIdx.x;
    if (t == 0) {
        *reinterpret_cast<uint64_t*>(b) = (uint64_t)L.n_cnk;
        int32_t* h = reinterpret_cast<int32_t*>(b + 8);
        h[0] = (int32_t)P.box.b[0];
        h[1] = (int32_t)P.box.b[1];
        h[2] = (int32_t)P.box.b[2];
        h[3] = sx;
        h[4] = sy;
        h[5] = sz;
        reinterpret_cast<uint32_t*>(b + L.off_scan)[L.n_cnk] = (uint32_t)L.n_pnt;
    }
    // tails: [end of section, next section) for scan, data, offsets, masks
    const int64_t ends[4] = {L.off_scan + 4 * (L.n_cnk + 1), L.off_data + L.data_bytes, L.off_offs + 2 * L.n_pnt,
                             L.off_mask + L.n_pnt};
    const int64_t next[4] = {L.off_data, L.off_offs, L.off_mask, L.bytes};
    if (t < 32) {
        const int s = t >> 3, q = t & 7;
        if (ends[s] + q < next[s]) b[ends[s] + q] = 0;
    }
}

struct UnpackDst {
    unsigned char* p[kMaxProps];  // staged values of the k-th packed property
};

// Staged inserts of the packed points of one box at their coordinates + shift.
__global__ void k_unpack_stage(const unsigned char* __restrict__ buf, PackLayout L, Geometry src_geo, Geometry dst_geo,
                               int64_t sx, int64_t sy, int64_t sz, int64_t* out_lin, PackProps pp, UnpackDst dst,
                               unsigned* err) {
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= L.n_pnt) return;
    const int64_t* ids = reinterpret_cast<const int64_t*>(buf + L.off_ids);
    const uint32_t* scan = reinterpret_cast<const uint32_t*>(buf + L.off_scan);
    const int16_t* offs = reinterpret_cast<const int16_t*>(buf + L.off_offs);
    // the chunk of point j: the last c with scan[c] <= j
    int64_t lo = 0, hi = L.n_cnk;
    while (hi - lo > 1) {
        const int64_t mid = (lo + hi) >> 1;
        if (scan[mid] <= (uint32_t)j) lo = mid;
        else hi = mid;
    }
    int64_t o[3];
    origin_of(src_geo, ids[lo], o);
    const int e = src_geo.edge, pt = offs[j];
    const int64_t c[3] = {o[0] + pt % e + sx, o[1] + (pt / e) % e + sy, o[2] + pt / (e * e) + sz};
    bool ok = pt >= 0 && pt < src_geo.bs;
    for (int d = 0; d < 3; ++d) ok = ok && c[d] >= 0 && c[d] < dst_geo.size[d];
    int64_t lin = -1;
    if (ok) {
        int64_t b, l;
        point_key_in(dst_geo, c, &b, &l);
        lin = b * dst_geo.bs + l;
    } else {
        atomicOr(err, kErrOutOfDomain);
    }
    out_lin[j] = lin;
    for (int p = 0; p < pp.np; ++p) {
        const int es = pp.es[p];
        const unsigned char* s = buf + L.off_data + L.prop_off[p] + j * es;
        for (int b = 0; b < es; ++b) dst.p[p][j * es + b] = s[b];
    }
}

// One packed box of a buffer, as found by k_unpack_walk.
struct UnpackBox {
    int64_t pos;       // byte offset of the box in the buffer
    int64_t n_cnk, n_pnt;
    int64_t start[3];  // packed box lower corner
    int64_t size[3];   // packing grid size
    int64_t pnt0;      // points of the boxes before this one
    int64_t shift[3];  // destination - packed coordinates
    int32_t bad;       // 1: the header does not fit the buffer
};

struct ElemSizes {
    int es[kMaxProps];
    int np;
};

// Walk the headers of nb packed boxes (one thread: each box's place follows
// from the sizes of the boxes before it).
__global__ void k_unpack_walk(const unsigned char* __restrict__ buf, int64_t nbytes, int nb, ElemSizes es,
                              UnpackBox* out) {
    if (blockIdx.x != 0 || threadIdx.x != 0) return;
    int64_t pos = 0, pts = 0;
    for (int k = 0; k < nb; ++k) {
        UnpackBox B{};
        B.pos = pos;
        B.pnt0 = pts;
        B.bad = 1;
        if (nbytes - pos >= 40) {
            const uint64_t nc = *reinterpret_cast<const uint64_t*>(buf + pos);
            if (nc <= (uint64_t)(nbytes - pos - 36) / 12) {
                const int32_t* h = reinterpret_cast<const int32_t*>(buf + pos + 8);
                const uint32_t np_ = *reinterpret_cast<const uint32_t*>(buf + pos + 32 + 12 * (int64_t)nc);
                const PackLayout L = layout_of((int64_t)nc, np_, es.np, es.es);
                bool ok = L.bytes <= nbytes - pos && !(nc == 0 && np_ != 0);
                for (int d = 0; d < 3; ++d) ok = ok && h[3 + d] >= 1;
                if (ok) {
                    B.n_cnk = (int64_t)nc;
                    B.n_pnt = np_;
                    for (int d = 0; d < 3; ++d) {
                        B.start[d] = h[d];
                        B.size[d] = h[3 + d];
                    }
                    B.bad = 0;
                    pos += L.bytes;
                    pts += np_;
                }
            }
        }
        out[k] = B;
        if (B.bad) {
            for (int j = k + 1; j < nb; ++j) out[j].bad = 1;
            return;
        }
    }
}

// Staged inserts of every packed point of the boxes: thread j finds its box
// by the point offsets, then proceeds as k_unpack_stage.
__global__ void k_unpack_stage_all(const unsigned char* __restrict__ buf, const UnpackBox* __restrict__ boxes, int nb,
                                   int64_t total, ElemSizes es, Geometry dst_geo, int64_t* out_lin, UnpackDst dst,
                                   unsigned* err) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= total) return;
    int lo = 0, hi = nb;
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (boxes[mid].pnt0 <= t) lo = mid;
        else hi = mid;
    }
    const UnpackBox& B = boxes[lo];
    const PackLayout L = layout_of(B.n_cnk, B.n_pnt, es.np, es.es);
    const int64_t j = t - B.pnt0;
    const unsigned char* b = buf + B.pos;
    const int64_t* ids = reinterpret_cast<const int64_t*>(b + L.off_ids);
    const uint32_t* scan = reinterpret_cast<const uint32_t*>(b + L.off_scan);
    const int16_t* offs = reinterpret_cast<const int16_t*>(b + L.off_offs);
    int64_t clo = 0, chi = L.n_cnk;
    while (chi - clo > 1) {
        const int64_t mid = (clo + chi) >> 1;
        if (scan[mid] <= (uint32_t)j) clo = mid;
        else chi = mid;
    }
    Geometry src = dst_geo;
    for (int d = 0; d < 3; ++d) {
        src.size[d] = B.size[d];
        src.bsz[d] = (B.size[d] + src.edge - 1) / src.edge;
    }
    int64_t o[3];
    origin_of(src, ids[clo], o);
    const int e = src.edge, pt = offs[j];
    const int64_t c[3] = {o[0] + pt % e + B.shift[0], o[1] + (pt / e) % e + B.shift[1],
                          o[2] + pt / (e * e) + B.shift[2]};
    bool ok = pt >= 0 && pt < src.bs;
    for (int d = 0; d < 3; ++d) ok = ok && c[d] >= 0 && c[d] < dst_geo.size[d];
    int64_t lin = -1;
    if (ok) {
        int64_t kb, kl;
        point_key_in(dst_geo, c, &kb, &kl);
        lin = kb * dst_geo.bs + kl;
    } else {
        atomicOr(err, kErrOutOfDomain);
    }
    out_lin[t] = lin;
    for (int p = 0; p < es.np; ++p) {
        const int sz = es.es[p];
        const unsigned char* sp = b + L.off_data + L.prop_off[p] + j * sz;
        for (int q = 0; q < sz; ++q) dst.p[p][t * sz + q] = sp[q];
    }
}

static unsigned wgrid(const sgb_grid* g, int64_t n) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((int64_t)g->num_sms * 8, (n + 7) / 8));
}

// The device state of a counting pass, in the grid's scratch.
struct PackScratch {
    HitBox* boxes;      // scratch[0]
    uint32_t *bits, *cnt, *start;  // scratch[1]: [len], [len]; scratch[2]: [len + 1], the number of hits last
    Hit* hits;          // scratch[3]
    uint2 *pre, *tiles;  // scratch[4]
    uint32_t* rows;     // scratch[8]
    int64_t words, len;
};

// The counting pass over all boxes: the hits, their places and the row starts (rows: 2 * (nb + 1), on the host).
static int pack_counts(sgb_grid* g, int64_t nboxes, const int64_t* boxes_host, std::vector<uint32_t>& rows, PackScratch& ps,
                       cudaStream_t s) {
    const int64_t n = g->n;
    ps.words = (n + 31) / 32;
    ps.len = nboxes * ps.words;
    rows.assign(2 * (nboxes + 1), 0);
    if (nboxes == 0 || n == 0) return SGB_OK;
    if (nboxes * (n + 1) >= (int64_t(1) << 31)) {
        set_error("too many boxes x chunks in one pack call");
        return SGB_ERANGE;
    }
    // the hits are at most the boxes' block-coordinate volumes, and the chunks of the grid, per box
    const size_t hb = std::max<size_t>((size_t)nboxes * sizeof(HitBox), rows.size() * 4);
    SGB_TRY(g->hscratch.ensure(hb));
    HitBox* hbx = static_cast<HitBox*>(g->hscratch.p);
    int64_t maxhits = 0;
    const int e = g->geo.edge;
    for (int64_t k = 0; k < nboxes; ++k) {
        std::memcpy(hbx[k].box.b, boxes_host + 6 * k, sizeof(hbx[k].box.b));
        double vol = 1;
        for (int d = 0; d < 3; ++d) {
            auto fl = [e](int64_t v) { return v >= 0 ? v / e : -((-(v + 1)) / e) - 1; };
            const int64_t lo = std::max<int64_t>(fl(boxes_host[6 * k + d]), 0);
            const int64_t hi = std::min<int64_t>(fl(boxes_host[6 * k + 3 + d]), g->geo.bsz[d] - 1);
            hbx[k].lo[d] = lo;
            hbx[k].hi[d] = hi;
            vol *= lo <= hi ? (double)(hi - lo + 1) : 0.0;
        }
        maxhits += vol < (double)n ? (int64_t)vol : n;
    }
    const int64_t ntiles = (maxhits + kHitTile - 1) / kHitTile;
    SGB_TRY(g->scratch[0].ensure((size_t)nboxes * sizeof(HitBox)));
    SGB_TRY(g->scratch[1].ensure((size_t)ps.len * 8 + 16));
    SGB_TRY(g->scratch[2].ensure((size_t)(ps.len + 1) * 4 + 16));
    SGB_TRY(g->scratch[3].ensure((size_t)maxhits * sizeof(Hit) + 16));
    SGB_TRY(g->scratch[4].ensure((size_t)(maxhits + ntiles + 1) * 8 + 16));
    SGB_TRY(g->scratch[8].ensure(rows.size() * 4));
    ps.boxes = g->scratch[0].as<HitBox>();
    ps.bits = g->scratch[1].as<uint32_t>();
    ps.cnt = ps.bits + ps.len;
    ps.start = g->scratch[2].as<uint32_t>();
    ps.hits = g->scratch[3].as<Hit>();
    ps.pre = g->scratch[4].as<uint2>();
    ps.tiles = ps.pre + maxhits;
    ps.rows = g->scratch[8].as<uint32_t>();
    SGB_CUDA(cudaMemcpyAsync(ps.boxes, hbx, (size_t)nboxes * sizeof(HitBox), cudaMemcpyHostToDevice, s));
    uint32_t* nhits = ps.start + ps.len;
    // boxes are shared out over the grid's second dimension until the chip holds no more CTAs
    const int64_t hx = (ps.words + 7) / 8;
    const int64_t hy = std::max<int64_t>(1, std::min<int64_t>({nboxes, (int64_t)g->num_sms * 8 / hx, 65535}));
    k_pack_hits<<<dim3((unsigned)hx, (unsigned)hy), 256, 0, s>>>(g->keys.as<int64_t>(), n, g->geo, ps.boxes, (int)nboxes,
                                                               ps.words, ps.bits, ps.cnt);
    SGB_CUDA(cudaGetLastError());
    SGB_TRY(scan_exclusive_u32(ps.cnt, ps.start, ps.len, nhits, &g->scratch[6], s));
    k_pack_list<<<(unsigned)((ps.len + 255) / 256), 256, 0, s>>>(ps.bits, ps.start, ps.words, ps.len, ps.hits);
    const unsigned tgrid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ntiles, (int64_t)g->num_sms * 2));
    k_pack_points<<<tgrid, kHitTile * 32, 0, s>>>(ps.hits, nhits, g->keys.as<int64_t>(), g->geo, g->mask.as<uint8_t>(), ps.boxes,
                                        ps.pre, ps.tiles);
    k_pack_rows<<<1, 1024, 0, s>>>(ps.tiles, nhits, ps.start, ps.pre, ps.words, (int)nboxes, ps.rows);
    SGB_CUDA(cudaGetLastError());
    SGB_CUDA(cudaMemcpyAsync(g->hscratch.p, ps.rows, rows.size() * 4, cudaMemcpyDeviceToHost, s));
    SGB_CUDA(cudaStreamSynchronize(s));
    std::memcpy(rows.data(), g->hscratch.p, rows.size() * 4);
    return SGB_OK;
}

static int check_props(const sgb_grid* g, int nprops, const int* props, int* es) {
    if (nprops < 0 || nprops > kMaxProps || (nprops > 0 && !props)) return SGB_EINVAL;
    for (int k = 0; k < nprops; ++k) {
        if (props[k] < 0 || props[k] >= g->nprop) return SGB_EINVAL;
        es[k] = elem_size(g->ptype[props[k]]);
    }
    return SGB_OK;
}

}  // namespace sgb

using namespace sgb;

extern "C" int sgb_pack_request(sgb_grid* g, int64_t nboxes, const int64_t* boxes_host, int nprops, const int* props,
                                int64_t* bytes_host, sgb_stream stream) {
    if (!g || nboxes < 0 || (nboxes > 0 && (!boxes_host || !bytes_host))) return SGB_EINVAL;
    if (g->geo.dim != 3) return SGB_ENOTSUP;
    int es[kMaxProps];
    SGB_TRY(check_props(g, nprops, props, es));
    std::vector<uint32_t> rows;
    PackScratch ps{};
    SGB_TRY(pack_counts(g, nboxes, boxes_host, rows, ps, (cudaStream_t)stream));
    for (int64_t k = 0; k < nboxes; ++k)
        bytes_host[k] = layout_of(rows[2 * k + 3] - rows[2 * k + 1], rows[2 * k + 2] - rows[2 * k], nprops, es).bytes;
    return SGB_OK;
}

extern "C" int sgb_pack(sgb_grid* g, int64_t nboxes, const int64_t* boxes_host, int nprops, const int* props,
                        void* out_dev, int64_t capacity, int64_t* bytes_written, sgb_stream stream) {
    if (!g || nboxes < 0 || (nboxes > 0 && (!boxes_host || !out_dev)) || !bytes_written) return SGB_EINVAL;
    if (g->geo.dim != 3) return SGB_ENOTSUP;
    if ((uintptr_t)out_dev % 8 != 0) {
        set_error("the pack buffer must be 8-byte aligned");
        return SGB_EINVAL;
    }
    int es[kMaxProps];
    SGB_TRY(check_props(g, nprops, props, es));
    *bytes_written = 0;
    if (nboxes == 0) return SGB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    std::vector<uint32_t> rows;
    PackScratch ps{};
    SGB_TRY(pack_counts(g, nboxes, boxes_host, rows, ps, s));
    std::vector<PackBox> pb((size_t)nboxes);
    int64_t pos = 0;
    bool any_points = false;
    for (int64_t k = 0; k < nboxes; ++k) {
        PackBox& P = pb[k];
        std::memcpy(P.box.b, boxes_host + 6 * k, sizeof(P.box.b));
        P.pnt0 = rows[2 * k];
        P.cnk0 = rows[2 * k + 1];
        P.L = layout_of(rows[2 * k + 3] - rows[2 * k + 1], rows[2 * k + 2] - rows[2 * k], nprops, es);
        P.base = pos;
        pos += P.L.bytes;
        any_points |= P.L.n_pnt > 0;
    }
    if (pos > capacity) {
        set_error("the pack buffer is smaller than sgb_pack_request reported");
        return SGB_ERANGE;
    }
    SGB_TRY(g->scratch[5].ensure(pb.size() * sizeof(PackBox)));
    SGB_TRY(g->hscratch.ensure(pb.size() * sizeof(PackBox)));
    std::memcpy(g->hscratch.p, pb.data(), pb.size() * sizeof(PackBox));
    SGB_CUDA(cudaMemcpyAsync(g->scratch[5].p, g->hscratch.p, pb.size() * sizeof(PackBox), cudaMemcpyHostToDevice, s));
    unsigned char* out = (unsigned char*)out_dev;
    if (any_points) {
        PackProps pp{};
        pp.np = nprops;
        for (int p = 0; p < nprops; ++p) {
            pp.src[p] = g->data[props[p]].as<unsigned char>();
            pp.es[p] = es[p];
            // every box's block of property p starts at a multiple of es when the blocks before it do
            bool wide = true;
            for (const PackBox& P : pb) wide = wide && (P.base + P.L.off_data + P.L.prop_off[p]) % es[p] == 0;
            pp.wide[p] = wide;
        }
        int64_t cnks = 0;
        for (const PackBox& P : pb) cnks += P.L.n_cnk;
        k_pack_emit<<<wgrid(g, cnks), 256, 0, s>>>(ps.hits, ps.start + ps.len, g->keys.as<int64_t>(), g->geo,
                                                   g->mask.as<uint8_t>(), g->scratch[5].as<PackBox>(), ps.pre, ps.tiles, pp,
                                                   out);
        SGB_CUDA(cudaGetLastError());
    }
    k_pack_finish<<<(unsigned)nboxes, 32, 0, s>>>(g->scratch[5].as<PackBox>(), (int)nboxes, (int32_t)g->geo.size[0],
                                                 (int32_t)g->geo.size[1], (int32_t)g->geo.size[2], out);
    SGB_CUDA(cudaGetLastError());
    SGB_CUDA(cudaStreamSynchronize(s));  // the host staging of the box table is reused by the next call
    *bytes_written = pos;
    return SGB_OK;
}

extern "C" int sgb_unpack(sgb_grid* g, const void* buf_dev, int64_t nbytes, int nprops, const int* props,
                          const int64_t* start_host, int64_t* consumed, sgb_stream stream) {
    if (!g || !consumed || nbytes < 0 || (nbytes > 0 && !buf_dev)) return SGB_EINVAL;
    *consumed = 0;
    if (g->geo.dim != 3) return SGB_ENOTSUP;
    if ((uintptr_t)buf_dev % 8 != 0) {
        set_error("the pack buffer must be 8-byte aligned");
        return SGB_EINVAL;
    }
    int es[kMaxProps];
    SGB_TRY(check_props(g, nprops, props, es));
    for (int k = 0; k < nprops; ++k)
        for (int j = 0; j < k; ++j)
            if (props[j] == props[k]) return SGB_EINVAL;
    if (nbytes < 40) {  // the smallest packed box: header + one scan entry
        set_error("truncated pack buffer");
        return SGB_EINVAL;
    }
    cudaStream_t s = (cudaStream_t)stream;
    const unsigned char* buf = (const unsigned char*)buf_dev;
    SGB_TRY(g->hscratch.ensure(64));
    unsigned char* h = (unsigned char*)g->hscratch.p;
    SGB_CUDA(cudaMemcpyAsync(h, buf, 32, cudaMemcpyDeviceToHost, s));
    SGB_CUDA(cudaStreamSynchronize(s));
    uint64_t ncu;
    int32_t pst[3], psz[3];
    std::memcpy(&ncu, h, 8);
    std::memcpy(pst, h + 8, 12);
    std::memcpy(psz, h + 20, 12);
    if (ncu > (uint64_t)(nbytes - 36) / 12) {  // ids, scan and scan[n_cnk] must fit
        set_error("corrupt pack buffer (chunk count)");
        return SGB_EINVAL;
    }
    const int64_t nc_ = (int64_t)ncu;
    SGB_CUDA(cudaMemcpyAsync(h + 48, buf + 32 + 12 * nc_, 4, cudaMemcpyDeviceToHost, s));
    SGB_CUDA(cudaStreamSynchronize(s));
    uint32_t npu;
    std::memcpy(&npu, h + 48, 4);
    const PackLayout L = layout_of(nc_, npu, nprops, es);
    if (L.bytes > nbytes || (nc_ == 0 && npu != 0)) {
        set_error("corrupt pack buffer, or one packed with other properties");
        return SGB_EINVAL;
    }
    for (int d = 0; d < 3; ++d)
        if (psz[d] < 1) {
            set_error("corrupt pack buffer (grid size)");
            return SGB_EINVAL;
        }
    // the packing grid's chunk indexing: its size from the header, the same chunk edge
    Geometry src = g->geo;
    for (int d = 0; d < 3; ++d) {
        src.size[d] = psz[d];
        src.bsz[d] = (psz[d] + src.edge - 1) / src.edge;
    }
    int64_t sh[3] = {0, 0, 0};
    if (start_host)
        for (int d = 0; d < 3; ++d) sh[d] = start_host[d] - pst[d];
    const int64_t np_ = npu;
    if (np_ > 0) {
        SGB_TRY(g->pend_lin.reserve((size_t)(g->npend + np_) * 8));
        for (int p = 0; p < g->nprop; ++p)
            SGB_TRY(g->pend_val[p].reserve((size_t)(g->npend + np_) * elem_size(g->ptype[p])));
        // the properties that are not unpacked are staged with their background
        bool packed[kMaxProps] = {};
        for (int k = 0; k < nprops; ++k) packed[props[k]] = true;
        for (int p = 0; p < g->nprop; ++p) {
            const int pe = elem_size(g->ptype[p]);
            if (packed[p]) g->pend_has[p] = true;
            else SGB_TRY(fill(g->pend_val[p].as<unsigned char>() + (size_t)g->npend * pe, np_, pe, bck_pattern(g, p), s));
        }
        PackProps pp{};
        UnpackDst dst{};
        pp.np = nprops;
        for (int k = 0; k < nprops; ++k) {
            pp.es[k] = es[k];
            dst.p[k] = g->pend_val[props[k]].as<unsigned char>() + (size_t)g->npend * es[k];
        }
        k_unpack_stage<<<(unsigned)((np_ + 255) / 256), 256, 0, s>>>(buf, L, src, g->geo, sh[0], sh[1], sh[2],
                                                                     g->pend_lin.as<int64_t>() + g->npend, pp, dst,
                                                                     g->err.as<unsigned>());
        SGB_CUDA(cudaGetLastError());
        g->npend += np_;
    }
    *consumed = L.bytes;
    return SGB_OK;
}

extern "C" int sgb_unpack_boxes(sgb_grid* g, const void* buf_dev, int64_t nbytes, int nprops, const int* props,
                                int64_t nboxes, const int64_t* starts_host, int64_t* consumed, sgb_stream stream) {
    if (!g || !consumed || nbytes < 0 || nboxes < 0 || (nbytes > 0 && !buf_dev)) return SGB_EINVAL;
    *consumed = 0;
    if (g->geo.dim != 3) return SGB_ENOTSUP;
    if ((uintptr_t)buf_dev % 8 != 0) {
        set_error("the pack buffer must be 8-byte aligned");
        return SGB_EINVAL;
    }
    ElemSizes es{};
    SGB_TRY(check_props(g, nprops, props, es.es));
    es.np = nprops;
    for (int k = 0; k < nprops; ++k)
        for (int j = 0; j < k; ++j)
            if (props[j] == props[k]) return SGB_EINVAL;
    if (nboxes == 0) return SGB_OK;
    if (nboxes > (int64_t(1) << 20)) return SGB_EINVAL;
    cudaStream_t s = (cudaStream_t)stream;
    const size_t tb = (size_t)nboxes * sizeof(UnpackBox);
    SGB_TRY(g->scratch[0].ensure(tb));
    SGB_TRY(g->hscratch.ensure(tb));
    UnpackBox* dboxes = g->scratch[0].as<UnpackBox>();
    k_unpack_walk<<<1, 1, 0, s>>>((const unsigned char*)buf_dev, nbytes, (int)nboxes, es, dboxes);
    SGB_CUDA(cudaGetLastError());
    SGB_CUDA(cudaMemcpyAsync(g->hscratch.p, dboxes, tb, cudaMemcpyDeviceToHost, s));
    SGB_CUDA(cudaStreamSynchronize(s));
    std::vector<UnpackBox> hb((size_t)nboxes);
    std::memcpy(hb.data(), g->hscratch.p, tb);
    for (const UnpackBox& B : hb)
        if (B.bad) {
            set_error("corrupt or truncated pack buffer, or one packed with other properties");
            return SGB_EINVAL;
        }
    const int64_t total = hb.back().pnt0 + hb.back().n_pnt;
    for (int64_t k = 0; k < nboxes; ++k)
        for (int d = 0; d < 3; ++d) hb[k].shift[d] = starts_host ? starts_host[3 * k + d] - hb[k].start[d] : 0;
    if (total > 0) {
        std::memcpy(g->hscratch.p, hb.data(), tb);
        SGB_CUDA(cudaMemcpyAsync(dboxes, g->hscratch.p, tb, cudaMemcpyHostToDevice, s));
        SGB_TRY(g->pend_lin.reserve((size_t)(g->npend + total) * 8));
        for (int p = 0; p < g->nprop; ++p)
            SGB_TRY(g->pend_val[p].reserve((size_t)(g->npend + total) * elem_size(g->ptype[p])));
        bool packed[kMaxProps] = {};
        for (int k = 0; k < nprops; ++k) packed[props[k]] = true;
        for (int p = 0; p < g->nprop; ++p) {
            const int pe = elem_size(g->ptype[p]);
            if (packed[p]) g->pend_has[p] = true;
            else SGB_TRY(fill(g->pend_val[p].as<unsigned char>() + (size_t)g->npend * pe, total, pe, bck_pattern(g, p), s));
        }
        UnpackDst dst{};
        for (int k = 0; k < nprops; ++k) dst.p[k] = g->pend_val[props[k]].as<unsigned char>() + (size_t)g->npend * es.es[k];
        k_unpack_stage_all<<<(unsigned)((total + 255) / 256), 256, 0, s>>>(
            (const unsigned char*)buf_dev, dboxes, (int)nboxes, total, es, g->geo, g->pend_lin.as<int64_t>() + g->npend,
            dst, g->err.as<unsigned>());
        SGB_CUDA(cudaGetLastError());
        SGB_CUDA(cudaStreamSynchronize(s));  // the host staging of the box table is reused by the next call
        g->npend += total;
    }
    const PackLayout Ll = layout_of(hb.back().n_cnk, hb.back().n_pnt, nprops, es.es);
    *consumed = hb.back().pos + Ll.bytes;
    return SGB_OK;
}
