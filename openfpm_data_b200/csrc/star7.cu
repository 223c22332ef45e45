// 7-point stencils (HEAT7, GS7), for single grids and batches and for any
// chunk ids: first 8^3 chunks, 4^3 chunks below.
//
// Reference path: applyStencilInPlace (src/SparseGridGpu/SparseGridGpu.hpp:
// 954-1048) launches one 512-thread CTA per chunk; loadGhostBlock_impl<1>
// (src/SparseGridGpu/SparseGridGpu_ker_util.hpp:487-564) gathers the 10^3
// tile point by point and substitutes the background where a mask byte is 0.
//
// Work: 16 lanes take ZS (4 or 8) z slices of one chunk; lane l owns the x
// quad l % 2 of row l / 2 and marches z with z - 1 / z / z + 1 in registers.
// All of a group's loads are issued at once: its rows and the two y-face rows
// of every slice by cp.async into a tile in shared memory (80 floats per
// slice, so that the y neighbours of every lane are plain 16-byte shared
// loads), the outer x cells and the two z faces into registers.  The x
// neighbour of a chunk sits at the next or previous position under x-fastest
// ids, so most x cells are read from the neighbouring group's tile; the one
// block barrier is there for them.  Blocks do one round and leave: the
// latencies of one block are covered by the others on the SM, and every block
// pulls the masks and neighbour rows of a block one wave ahead into L2.
//
// Sparsity: a quad none of whose points exists is neither read nor written
// (points with mask byte 0 hold the background in HBM, which grid.cu and
// HEAT7's stores keep), so a step moves about the bytes of the existing rows
// and not of whole chunks.
//
// AGAIN: the source may hold anything at points that do not exist (a caller kept a pointer to it); each lane puts
// the background into what it has copied or loaded, by the mask bytes.  A kernel of its own, for the first step of a
// call: the tests in a uniform branch made the usual path a quarter slower (512^3 Gray-Scott, 50 steps, 1458 us,
// 1813 so).  Heat on 16,384 Morton chunks 15.0 us a step, 12.8 without.
//
// What bounds it: HBM for large grids, where the power cap is reached with
// it; latency and block turnover for one to four waves of blocks.  Measured
// on one B200 (us per step, the earlier kernel, a ring of bulk copies per
// warp over whole chunks, in brackets): Gray-Scott 512^3, 40 balls, 18,932
// chunks 29.3 (39.2); Gray-Scott 900^3, 200 balls 121-130 (189); heat 48
// grids of edge 32-384 199-215 = 5.7-6.1 TB/s (331); heat 509x301x211 6.2
// (9.8); heat 256^3 on Morton ids 5.3 (36.0, one CTA per chunk).  Tried and
// slower: rows read straight into registers through L1 without the tile
// (31.4 / heat 228-256), a persistent form with two tiles per group (27.9 for
// Gray-Scott, but heat 309-330), whole-chunk L2 prefetch (36.5-38.7: the
// absent rows are fetched too).
#include <algorithm>

#include "star7.cuh"

namespace sgb {

constexpr int kStarThreads = 128, kStarGroups = kStarThreads / 16;

// What only boxed launches need: the others have half as many bytes of parameters to copy on the host.
template <bool BOX>
struct BoxArgs {
    const int64_t* keys;
    Geometry geo;
    StencilParams prm;
};
template <>
struct BoxArgs<false> {};
template <bool BOX>
static BoxArgs<BOX> box_args(const LaunchDesc& L) {
    if constexpr (BOX) return {L.keys, L.geo, L.prm};
    else return {};
}

// A group's part of shared memory: rows -1 .. 8 of ZS slices, per field.
template <int NP, int ZS>
struct StarTile {
    float row[NP][ZS][80];
};

template <int KIND, int NP, bool BOX, bool BATCH, bool AGAIN, int ZS, int MINB>
__global__ void __launch_bounds__(kStarThreads, MINB)
    k_star7_e8(FieldSet fs, const uint8_t* __restrict__ mask, const int32_t* __restrict__ nn,
               BoxArgs<BOX> box, const int32_t* __restrict__ gid, const GridInfo* __restrict__ grids, GridInfo g0, int64_t n,
               int64_t t, int fill, int chained, int ahead) {
    constexpr int PARTS = 8 / ZS;
    // A batch holds clean copies and never fills.  (Heat compiled without the test took 1.3 % longer all the same.)
    constexpr bool CANFILL = !BATCH || KIND == SGB_HEAT7;
    extern __shared__ __align__(16) unsigned char star_smem[];
    StarTile<NP, ZS>* const tiles = reinterpret_cast<StarTile<NP, ZS>*>(star_smem);
    const int grp = threadIdx.x >> 4;
    StarTile<NP, ZS>& T = tiles[grp];
    // A chained launch follows one over the same map in the same call, so its masks and neighbours stand already.
    // The first launch of a call lets the next one begin only behind its own wait, which is what makes that true
    // whatever ran before it.  (One common trigger behind the branch made the compiler lose the overlap: heat
    // 256^3 Morton 5.40 us a step, 5.09 so.)
    if (chained) {
        grid_launch_dependents();
    } else {
        const int64_t first = grid_dependency_wait();
        mask += first;
        nn += first;
        grid_launch_dependents();
    }
    const int l16 = threadIdx.x & 15, y = l16 >> 1, xq = l16 & 1;
    const int o0 = y * 8 + xq * 4;
    const int64_t total = n * PARTS;
    const int64_t it = (int64_t)blockIdx.x * kStarGroups + grp;
    bool live = it < total;
    const int64_t c = live ? it / PARTS : 0;
    const int zb = PARTS == 1 ? 0 : (int)(it % PARTS) * ZS;
    GridInfo gb;
    int par = 0;
    if (BATCH) {
        gb = grids[gid[c]];
        live = live && t >= gb.start && t < gb.start + gb.nsteps;
        par = (int)((t - gb.start) & 1);
    }
    const GridInfo& gi = BATCH ? gb : g0;
    uint32_t m[ZS];  // mask bytes of the lane's quads
    const uint8_t* mp = mask + c * 512 + zb * 64 + o0;
#pragma unroll
    for (int z = 0; z < ZS; ++z) m[z] = live ? __ldg(reinterpret_cast<const uint32_t*>(mp + z * 64)) : 0u;
    const int4 na = __ldg(reinterpret_cast<const int4*>(nn + c * 8));
    const int2 nz = __ldg(reinterpret_cast<const int2*>(nn + c * 8 + 4));
    const int64_t dep = grid_dependency_wait();
    const float* src[NP];
    float bs[NP], bd[NP];  // backgrounds of the source and destination fields
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        src[p] = (par ? fs.in[1][p] : fs.in[0][p]) + dep;
        bs[p] = par ? gi.bck[1][p] : gi.bck[0][p];
        bd[p] = par ? gi.bck[0][p] : gi.bck[1][p];
    }
    const int64_t oc = c * 512 + zb * 64 + o0;
#pragma unroll
    for (int z = 0; z < ZS; ++z)
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            float* d = &T.row[p][z][8 + o0];
            if (m[z]) cp_async16(d, src[p] + oc + z * 64);
            else *reinterpret_cast<float4*>(d) = splat4(bs[p]);
        }
    // y faces: lanes 0..7 the -y side, 8..15 the +y side, quad xq of slice (l16 % 8) / 2 + 4 k
    const int side = l16 >> 3, zq = (l16 & 7) >> 1;
    uint32_t my[ZS / 4];  // AGAIN: their mask bytes
    {
        const int32_t ny = side ? na.w : na.z;
#pragma unroll
        for (int k = 0; k < ZS / 4; ++k) {
            const int z = zq + 4 * k;
            const int64_t oy = (int64_t)ny * 512 + (zb + z) * 64 + (side ? 0 : 56) + xq * 4;
            const bool there = live && ny >= 0;
            my[k] = AGAIN && there ? ldm4(mask + oy) : 0x01010101u;
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                float* d = &T.row[p][z][(side ? 72 : 0) + xq * 4];
                if (there) cp_async16(d, src[p] + oy);
                else *reinterpret_cast<float4*>(d) = splat4(bs[p]);
            }
        }
    }
    cp_async_commit();
    // the group `ahead` items on: its mask bytes and neighbour row on their way to L2 (3 % at 512^3)
    if (l16 < 2 && it + ahead < total) {
        const int64_t ai = it + ahead, ac = ai / PARTS;
        if (l16 == 0) {
            const uint8_t* q = mask + ac * 512 + (PARTS == 1 ? 0 : (int)(ai % PARTS) * ZS * 64);
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(q), "r"(ZS * 64) : "memory");
        } else {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(nn + ac * 8) : "memory");
        }
    }
    // an x neighbour at the next position is another tile of this block
    const int32_t nx = xq ? na.y : na.x;
    const int gq = grp / PARTS + (xq ? 1 : -1);
    const bool in_cta = live && nx >= 0 && nx == c + (xq ? 1 : -1) && gq >= 0 && gq < kStarGroups / PARTS;
    const float* xs = &tiles[grp + (in_cta ? (xq ? PARTS : -PARTS) : 0)].row[0][0][8 + y * 8 + (xq ? 0 : 7)];
    const int64_t ox = (int64_t)nx * 512 + zb * 64 + y * 8 + (xq ? 0 : 7);
    const int64_t ozm = zb > 0 ? oc - 64 : (nz.x >= 0 ? (int64_t)nz.x * 512 + 448 + o0 : -1);
    const int64_t ozp = zb + ZS < 8 ? oc + ZS * 64 : (nz.y >= 0 ? (int64_t)nz.y * 512 + o0 : -1);
    float4 zm[NP], zl[NP], cv[NP];
    float xh[ZS][NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        zm[p] = splat4(bs[p]);
        zl[p] = splat4(bs[p]);
        if (m[0] && ozm >= 0) {
            zm[p] = ldf4(src[p] + ozm);
            if constexpr (AGAIN) zm[p] = masked4(zm[p], ldm4(mask + ozm), bs[p]);
        }
        if (m[ZS - 1] && ozp >= 0) {
            zl[p] = ldf4(src[p] + ozp);
            if constexpr (AGAIN) zl[p] = masked4(zl[p], ldm4(mask + ozp), bs[p]);
        }
    }
#pragma unroll
    for (int z = 0; z < ZS; ++z)
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            xh[z][p] = bs[p];
            if (m[z] && nx >= 0 && !in_cta) {
                xh[z][p] = ldf1(src[p] + ox + z * 64);
                if constexpr (AGAIN)
                    if (!__ldg(mask + ox + z * 64)) xh[z][p] = bs[p];
            }
        }
    int32_t cx = 0, cy = 0, cz = 0;
    if constexpr (BOX) {
        int64_t o[3];
        chunk_origin(box.geo, box.keys[c], o);
        cx = (int32_t)o[0] + xq * 4;
        cy = (int32_t)o[1] + y;
        cz = (int32_t)o[2] + zb;
    }
    float* dst[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) dst[p] = (par ? fs.out[1][p] : fs.out[0][p]) + oc;
    cp_async_wait_all();
    if constexpr (AGAIN) {  // backgrounds into what this lane has copied
        auto mend = [&](float* d, uint32_t m4, float b) {
            if (m4 != 0x01010101u) *reinterpret_cast<float4*>(d) = masked4(*reinterpret_cast<const float4*>(d), m4, b);
        };
#pragma unroll
        for (int p = 0; p < NP; ++p) {
#pragma unroll
            for (int z = 0; z < ZS; ++z)
                if (m[z]) mend(&T.row[p][z][8 + o0], m[z], bs[p]);
#pragma unroll
            for (int k = 0; k < ZS / 4; ++k) mend(&T.row[p][zq + 4 * k][(side ? 72 : 0) + xq * 4], my[k], bs[p]);
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < NP; ++p) cv[p] = *reinterpret_cast<const float4*>(&T.row[p][0][8 + o0]);
#pragma unroll
    for (int z = 0; z < ZS; ++z) {
        Quad lap[NP];
        float4 zp[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            zp[p] = z + 1 < ZS ? *reinterpret_cast<const float4*>(&T.row[p][z + 1 < ZS ? z + 1 : 0][8 + o0]) : zl[p];
            const float4 ym = *reinterpret_cast<const float4*>(&T.row[p][z][o0]);
            const float4 yp = *reinterpret_cast<const float4*>(&T.row[p][z][16 + o0]);
            // the inner x cell is the partner quad's edge
            const float got = __shfl_xor_sync(0xffffffffu, xq ? cv[p].x : cv[p].w, 1);
            float xo = xh[z][p];
            if (in_cta) xo = xs[(p * ZS + z) * 80];
            lap[p] = lap_quad<KIND>(cv[p], xq ? got : xo, xq ? xo : got, ym, yp, zm[p], zp[p]);
        }
        if (m[z] || (CANFILL && fill && live)) {
            const uint32_t act = active_bits<BOX>(m[z], box, cx, cy, cz + z);
            star_store<KIND, NP>(cv, lap, m[z], act, gi, bd, dst[0] + z * 64, dst[NP - 1] + z * 64);
            if (KIND == SGB_GS7 && !BOX && !BATCH && fill > 1 && (m[z] & 0xfefefefeu)) star_rest<NP>(m[z], bd, dst[0] + z * 64, dst[NP - 1] + z * 64);
        }
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            zm[p] = cv[p];
            cv[p] = zp[p];
        }
    }
}

// 4^3 chunks: 16 lanes take one chunk, lane l the x row (y, z) = (l % 4, l / 4), all of whose neighbours are
// read straight from global memory (rows inside the chunk and of the chunks before and after it hit the lines
// that the block's other lanes load).  The one-CTA-per-chunk gather that served these chunks before kept 64 of
// 256 threads busy: Gray-Scott 250x190x131, 24,003 chunks and 1.33 M points, 65.7 us per step, now 6.46 (3.5
// TB/s of the points' bytes; 4 to 8 blocks per SM run the same).  Bound by latency: two waves of blocks.
template <int KIND, int NP, bool BOX, bool BATCH, bool AGAIN, int MINB>
__global__ void __launch_bounds__(kStarThreads, MINB)
    k_star7_e4(FieldSet fs, const uint8_t* __restrict__ mask, const int32_t* __restrict__ nn,
               BoxArgs<BOX> box, const int32_t* __restrict__ gid, const GridInfo* __restrict__ grids, GridInfo g0, int64_t n,
               int64_t t, int fill, int chained) {
    // A chained launch follows one over the same map in the same call, so its masks and neighbours stand already.
    // The first launch of a call lets the next one begin only behind its own wait, which is what makes that true
    // whatever ran before it.  (One common trigger behind the branch made the compiler lose the overlap: heat
    // 256^3 Morton 5.40 us a step, 5.09 so.)
    if (chained) {
        grid_launch_dependents();
    } else {
        const int64_t first = grid_dependency_wait();
        mask += first;
        nn += first;
        grid_launch_dependents();
    }
    constexpr bool CANFILL = !BATCH || KIND == SGB_HEAT7;  // as above
    const int l16 = threadIdx.x & 15, y = l16 & 3, z = l16 >> 2;
    const int64_t c = (int64_t)blockIdx.x * kStarGroups + (threadIdx.x >> 4);
    bool live = c < n;
    GridInfo gb;
    int par = 0;
    if (BATCH && live) {
        gb = grids[gid[c]];
        live = t >= gb.start && t < gb.start + gb.nsteps;
        par = (int)((t - gb.start) & 1);
    }
    const GridInfo& gi = BATCH ? gb : g0;
    const uint32_t m = live ? __ldg(reinterpret_cast<const uint32_t*>(mask + c * 64 + l16 * 4)) : 0u;
    if (!m && !(CANFILL && fill && live)) {
        // The row holds no point.  No thread leaves without the wait: a launch of idle rows only would be over
        // before the step ahead of it, and what follows in the stream waits for this launch alone.
        grid_dependency_wait();
        return;
    }
    const int4 na = __ldg(reinterpret_cast<const int4*>(nn + c * 8));
    const int2 nz = __ldg(reinterpret_cast<const int2*>(nn + c * 8 + 4));
    const int64_t oc = c * 64 + l16 * 4;
    const int64_t oxm = (int64_t)na.x * 64 + l16 * 4 + 3, oxp = (int64_t)na.y * 64 + l16 * 4;
    const int64_t oym = y > 0 ? oc - 4 : (na.z >= 0 ? (int64_t)na.z * 64 + z * 16 + 12 : -1);
    const int64_t oyp = y < 3 ? oc + 4 : (na.w >= 0 ? (int64_t)na.w * 64 + z * 16 : -1);
    const int64_t ozm = z > 0 ? oc - 16 : (nz.x >= 0 ? (int64_t)nz.x * 64 + 48 + y * 4 : -1);
    const int64_t ozp = z < 3 ? oc + 16 : (nz.y >= 0 ? (int64_t)nz.y * 64 + y * 4 : -1);
    const int64_t dep = grid_dependency_wait();
    float4 cv[NP];
    Quad lap[NP];
    float bd[NP];
    float* dst[NP];
    float4 ym[NP], yp[NP], zm[NP], zp[NP];
    float xm[NP], xp[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const float* src = (par ? fs.in[1][p] : fs.in[0][p]) + dep;
        const float bs = par ? gi.bck[1][p] : gi.bck[0][p];
        dst[p] = (par ? fs.out[1][p] : fs.out[0][p]) + oc;
        bd[p] = par ? gi.bck[0][p] : gi.bck[1][p];
        ym[p] = yp[p] = zm[p] = zp[p] = splat4(bs);
        xm[p] = xp[p] = bs;
        cv[p] = ldf4(src + oc);
        if (oym >= 0) ym[p] = ldf4(src + oym);
        if (oyp >= 0) yp[p] = ldf4(src + oyp);
        if (ozm >= 0) zm[p] = ldf4(src + ozm);
        if (ozp >= 0) zp[p] = ldf4(src + ozp);
        if (na.x >= 0) xm[p] = ldf1(src + oxm);
        if (na.y >= 0) xp[p] = ldf1(src + oxp);
        if constexpr (AGAIN) {
            cv[p] = masked4(cv[p], m, bs);
            ym[p] = masked4(ym[p], oym >= 0 ? ldm4(mask + oym) : 0u, bs);
            yp[p] = masked4(yp[p], oyp >= 0 ? ldm4(mask + oyp) : 0u, bs);
            zm[p] = masked4(zm[p], ozm >= 0 ? ldm4(mask + ozm) : 0u, bs);
            zp[p] = masked4(zp[p], ozp >= 0 ? ldm4(mask + ozp) : 0u, bs);
            if (na.x >= 0 && !__ldg(mask + oxm)) xm[p] = bs;
            if (na.y >= 0 && !__ldg(mask + oxp)) xp[p] = bs;
        }
    }
#pragma unroll
    for (int p = 0; p < NP; ++p) lap[p] = lap_quad<KIND>(cv[p], xm[p], xp[p], ym[p], yp[p], zm[p], zp[p]);
    int32_t cx = 0, cy = 0, cz = 0;
    if constexpr (BOX) {
        int64_t o[3];
        chunk_origin(box.geo, box.keys[c], o);
        cx = (int32_t)o[0];
        cy = (int32_t)o[1] + y;
        cz = (int32_t)o[2] + z;
    }
    star_store<KIND, NP>(cv, lap, m, active_bits<BOX>(m, box, cx, cy, cz), gi, bd, dst[0], dst[NP - 1]);
    if (KIND == SGB_GS7 && !BOX && !BATCH && fill > 1 && (m & 0xfefefefeu)) star_rest<NP>(m, bd, dst[0], dst[NP - 1]);
}

// Consecutive steps overlap one launch's ramp-up with the previous one's tail.
struct StarLaunch {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    StarLaunch(int64_t groups, size_t smem, cudaStream_t s) {
        cfg.gridDim = dim3((unsigned)((groups + kStarGroups - 1) / kStarGroups));
        cfg.blockDim = dim3(kStarThreads);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
    }
};

template <int KIND, int NP, bool BOX, bool BATCH, bool AGAIN, int ZS, int MINB>
static int launch_star(const LaunchDesc& L, cudaStream_t s) {
    auto kern = k_star7_e8<KIND, NP, BOX, BATCH, AGAIN, ZS, MINB>;
    const int64_t items = L.n * (8 / ZS);
    size_t smem = sizeof(StarTile<NP, ZS>) * kStarGroups;
    // a caller's limit on the CTAs per SM: each CTA takes its share of the SM's shared memory
    if (L.ctas_per_sm > 0) smem = std::max(smem, (size_t)(kMaxDynamicSmem / L.ctas_per_sm - 1024) & ~(size_t)127);
    if (smem > 48 * 1024) SGB_TRY(allow_max_smem(kern));
    StarLaunch l(items, smem, s);
    const int ahead = L.num_sms * 7 * kStarGroups;  // about the groups resident at a time
    SGB_CUDA(cudaLaunchKernelEx(&l.cfg, kern, L.fs, L.mask, L.nn, box_args<BOX>(L), L.gid, L.grids, L.g0, L.n, L.t,
                                L.fill, L.chained, ahead));
    return SGB_OK;
}

template <int KIND, int NP, int ZS, int MINB>
static int launch_star_kind(const LaunchDesc& L, cudaStream_t s) {
    constexpr int BATCHB = KIND == SGB_GS7 && ZS == 4 ? MINB - 1 : MINB;  // the grid entry takes registers
    if (L.grids) return launch_star<KIND, NP, false, true, false, ZS, BATCHB>(L, s);
    if (L.again) return L.prm.has_box ? launch_star<KIND, NP, true, false, true, ZS, MINB>(L, s)
                                      : launch_star<KIND, NP, false, false, true, ZS, MINB>(L, s);
    if (L.prm.has_box) return launch_star<KIND, NP, true, false, false, ZS, MINB>(L, s);
    return launch_star<KIND, NP, false, false, false, ZS, MINB>(L, s);
}

template <int KIND, int NP, bool BOX, bool BATCH, bool AGAIN>
static int launch_e4(const LaunchDesc& L, cudaStream_t s) {
    StarLaunch l(L.n, 0, s);
    // Gray-Scott held to 56 registers: 146.6 us for 20 steps on 24,003 chunks, 148.6 with the 64 it takes otherwise
    constexpr int MINB = KIND == SGB_HEAT7 ? 10 : AGAIN || BATCH || BOX ? 6 : 9;
    SGB_CUDA(cudaLaunchKernelEx(&l.cfg, k_star7_e4<KIND, NP, BOX, BATCH, AGAIN, MINB>, L.fs, L.mask, L.nn,
                                box_args<BOX>(L), L.gid, L.grids, L.g0, L.n, L.t, L.fill, L.chained));
    return SGB_OK;
}

template <int KIND, int NP>
static int launch_e4_kind(const LaunchDesc& L, cudaStream_t s) {
    if (L.grids) return launch_e4<KIND, NP, false, true, false>(L, s);
    if (L.again) return L.prm.has_box ? launch_e4<KIND, NP, true, false, true>(L, s) : launch_e4<KIND, NP, false, false, true>(L, s);
    if (L.prm.has_box) return launch_e4<KIND, NP, true, false, false>(L, s);
    return launch_e4<KIND, NP, false, false, false>(L, s);
}

// Slices per group.  Eight halve the z-face loads and the instructions per point, four fill the chip with half
// as many chunks.  Heat: eight from two full waves of such blocks on (us per step, 4 against 8: 5,637 chunks
// 5.3 / 8.0, 18,932 chunks 12.8 / 12.5, 33,000 chunks 33.3 / 31.7, 300,000 chunks 241 / 212).  Gray-Scott
// keeps four: the same time within 2 % at every size, and eight need 41 KB and 92 registers a block.  (Heat
// with eight slices fits 8 blocks of 128 threads on an SM, with four 10; Gray-Scott 7: no spills.)
int launch_star7(const LaunchDesc& L, cudaStream_t s) {
    if (L.edge == 4) return L.kind == SGB_GS7 ? launch_e4_kind<SGB_GS7, 2>(L, s) : launch_e4_kind<SGB_HEAT7, 1>(L, s);
    bool eight = L.kind == SGB_HEAT7 && L.n >= (int64_t)2 * L.num_sms * 8 * kStarGroups;
    if (L.stages > 0) eight = L.stages >= 4;
    if (L.kind == SGB_GS7)
        return eight ? launch_star_kind<SGB_GS7, 2, 8, 4>(L, s) : launch_star_kind<SGB_GS7, 2, 4, 7>(L, s);
    return eight ? launch_star_kind<SGB_HEAT7, 1, 8, 8>(L, s) : launch_star_kind<SGB_HEAT7, 1, 4, 10>(L, s);
}

}  // namespace sgb
