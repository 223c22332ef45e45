// All steps of a small grid's heat or Gray-Scott solve in one launch: first 8^3 chunks, 4^3 chunks below.
//
// A grid of a few hundred 8^3 chunks runs a step in less time than a launch
// costs.  Here one cluster of up to 16 CTAs keeps the whole solve in its
// shared memory: CTA r owns a contiguous range of chunk positions, both
// ping-pong buffers of their fields and their masks.  Rows inside a chunk are
// plain shared loads; the six faces come from the neighbouring chunks' tiles
// wherever they are in the cluster (distributed shared memory), by addresses
// worked out once.  One hardware cluster barrier per step orders the steps:
// there is no spin wait.  A unit of work is four z slices of a chunk on 16
// lanes, as in star7.cu, with the same arithmetic and stores.
//
// What bounds it: the barrier and one round of load and compute latency, about
// 0.9 us a step, then the throughput of the 16 SMs, about 190 cycles per chunk
// and SM (as star7.cu's).  It replaced a cooperative launch over all SMs with
// a software grid barrier: 3.9 us a step at 376 chunks.  Tried and slower: 768
// and 1024 threads (the registers spill), generic addresses for all faces.
#include <algorithm>

#include "star7.cuh"

namespace sgb {

constexpr int kSolveThreads = 512, kSolveGroups = kSolveThreads / 16, kSolveCtas = 16;

// Loads from the cluster's shared memory.  Not volatile, so that a unit's loads all go out before the first is
// waited for; their addresses carry a value made behind the step's barrier, which keeps them behind it.
__device__ __forceinline__ float4 ld_dsm4(uint32_t a) {
    float4 v;
    asm("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ float ld_dsm1(uint32_t a) {
    float v;
    asm("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t map_cluster(uint32_t a, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t opaque_zero() {
    uint32_t z;
    asm volatile("mov.u32 %0, 0;" : "=r"(z)::"memory");
    return z;
}

// Shared memory of a CTA that owns up to `cap` chunks.
template <int NP>
__host__ __device__ constexpr size_t solve_smem(int cap) {
    return (size_t)cap * (2 * NP * 2048 + 512 + 8 * 4) + 2 * NP * 16;
}

template <int KIND, int NP>
__global__ void __launch_bounds__(kSolveThreads, 1)
    k_solve_cluster(FieldSet fs, const uint8_t* __restrict__ mask, const int32_t* __restrict__ nn, int n, GridInfo gi,
                    int nsteps, int cap, int again) {
    extern __shared__ __align__(16) unsigned char solve_raw[];
    float* const F = reinterpret_cast<float*>(solve_raw);                   // [2][NP][cap][512]
    uint8_t* const mk = solve_raw + (size_t)cap * 2 * NP * 2048;            // [cap][512]
    uint32_t* const adr = reinterpret_cast<uint32_t*>(mk + (size_t)cap * 512);  // [cap][8]
    float4* const bq = reinterpret_cast<float4*>(adr + (size_t)cap * 8);        // [2][NP] backgrounds, absent neighbours
    uint32_t rank, nranks;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(nranks));
    const int P = (int)nranks;
    const int a = n * (int)rank / P, m = n * ((int)rank + 1) / P - a;
    const int fstride = cap * 512;  // floats between fields
    constexpr uint32_t kNone = 0xffffffffu;
    if (threadIdx.x < 2 * NP) {
        const int b = threadIdx.x / NP, p = threadIdx.x % NP;
        bq[threadIdx.x] = splat4(b ? (p ? gi.bck[1][NP - 1] : gi.bck[1][0]) : (p ? gi.bck[0][NP - 1] : gi.bck[0][0]));
    }
    const uint32_t bqa = map_cluster(smem_u32(bq), rank);
    for (int i = threadIdx.x; i < m * 128; i += kSolveThreads) {
        const uint32_t m4 = again ? reinterpret_cast<const uint32_t*>(mask + (int64_t)a * 512)[i] : 0x01010101u;
#pragma unroll
        for (int p = 0; p < NP; ++p)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                float4 v = reinterpret_cast<const float4*>(fs.in[b][p] + (int64_t)a * 512)[i];
                if (m4 != 0x01010101u) {
                    v.x = m4 & 0xffu ? v.x : gi.bck[b][p];
                    v.y = m4 & 0xff00u ? v.y : gi.bck[b][p];
                    v.z = m4 & 0xff0000u ? v.z : gi.bck[b][p];
                    v.w = m4 & 0xff000000u ? v.w : gi.bck[b][p];
                }
                reinterpret_cast<float4*>(F + (b * NP + p) * fstride)[i] = v;
            }
    }
    for (int i = threadIdx.x; i < m * 32; i += kSolveThreads)
        reinterpret_cast<uint4*>(mk)[i] = reinterpret_cast<const uint4*>(mask + (int64_t)a * 512)[i];
    // cluster addresses of the neighbours' tiles (field 0, buffer 0); the owner of position q is (P (q + 1) - 1) / n
    for (int i = threadIdx.x; i < m * 8; i += kSolveThreads) {
        const int q = (i & 7) < 6 ? nn[(int64_t)a * 8 + i] : -1;
        if (q >= 0) {
            const int r = (P * (q + 1) - 1) / n;
            adr[i] = map_cluster(smem_u32(F) + (uint32_t)(q - n * r / P) * 2048u, (uint32_t)r);
        } else {
            adr[i] = kNone;
        }
    }
    cluster_barrier();
    const int grp = threadIdx.x >> 4, l16 = threadIdx.x & 15, y = l16 >> 1, xq = l16 & 1;
    const int o0 = y * 8 + xq * 4;
    for (int t = 0; t < nsteps; ++t) {
        const int par = t & 1;
        float bd[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) bd[p] = par ? gi.bck[0][p] : gi.bck[1][p];
        const uint32_t step0 = opaque_zero();
        // both halves of a warp take the two halves of one chunk
        for (int u = grp; u < 2 * m; u += kSolveGroups) {
            const int c = u >> 1, zb = (u & 1) * 4;
            const float* S = F + par * NP * fstride + c * 512 + zb * 64 + o0;
            float* D = F + (par ^ 1) * NP * fstride + c * 512 + zb * 64 + o0;
            const uint32_t boff = (uint32_t)(par * NP * fstride) * 4u + step0, ba = bqa + (uint32_t)(par * NP) * 16u + step0;
            const uint32_t ax = adr[c * 8 + xq], ay = adr[c * 8 + (y == 0 ? 2 : 3)], az = adr[c * 8 + (zb ? 5 : 4)];
            const bool hy = (y == 0 || y == 7) && ay != kNone;
            uint32_t mz[4];
#pragma unroll
            for (int z = 0; z < 4; ++z) mz[z] = *reinterpret_cast<const uint32_t*>(mk + c * 512 + (zb + z) * 64 + o0);
            float4 cv[4][NP];
            Quad lap[4][NP];
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                // every load of the field, then its Laplacians: x cells and y rows outside the chunk (from a
                // background quad where there is no neighbour), the half's z face, the half's own rows
                const uint32_t po = boff + (uint32_t)(p * fstride) * 4u, bp = ba + p * 16u;
                float xh[4];
                float4 yf[4], ym[4], yp[4], zo;
                const uint32_t x0 = ax != kNone ? ax + po + (uint32_t)(zb * 64 + y * 8 + (xq ? 0 : 7)) * 4u : bp;
                const uint32_t y0 = hy ? ay + po + (uint32_t)(zb * 64 + (y ? 0 : 56) + xq * 4) * 4u : bp;
                const uint32_t xs = ax != kNone ? 256u : 0u, ys = hy ? 256u : 0u;
                const float4 zf = ld_dsm4(az != kNone ? az + po + (uint32_t)((zb ? 0 : 448) + o0) * 4u : bp);
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    xh[z] = ld_dsm1(x0 + z * xs);
                    yf[z] = ld_dsm4(y0 + z * ys);
                }
                const float* R = S + p * fstride;
                zo = *reinterpret_cast<const float4*>(zb ? R - 64 : R + 256);  // the other half's adjoining slice
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    cv[z][p] = *reinterpret_cast<const float4*>(R + z * 64);
                    ym[z] = *reinterpret_cast<const float4*>(R + z * 64 - (y > 0 ? 8 : 0));
                    yp[z] = *reinterpret_cast<const float4*>(R + z * 64 + (y < 7 ? 8 : 0));
                }
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    const float4 zm = z > 0 ? cv[z > 0 ? z - 1 : 0][p] : (zb ? zo : zf);
                    const float4 zp = z < 3 ? cv[z < 3 ? z + 1 : 3][p] : (zb ? zf : zo);
                    const float got = __shfl_xor_sync(0xffffffffu, xq ? cv[z][p].x : cv[z][p].w, 1);
                    lap[z][p] = lap_quad<KIND>(cv[z][p], xq ? got : xh[z], xq ? xh[z] : got, y > 0 ? ym[z] : yf[z],
                                               y < 7 ? yp[z] : yf[z], zm, zp);
                }
            }
#pragma unroll
            for (int z = 0; z < 4; ++z)
                if (mz[z])
                    star_store<KIND, NP>(cv[z], lap[z], mz[z], active_bits<false>(mz[z], 0, 0, 0, 0), gi, bd,
                                         D + z * 64, D + (NP - 1) * fstride + z * 64);
        }
        cluster_barrier();  // also: no CTA leaves while another may still read its tiles
    }
    for (int i = threadIdx.x; i < m * 128; i += kSolveThreads)
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            reinterpret_cast<float4*>(fs.out[1][p] + (int64_t)a * 512)[i] = reinterpret_cast<const float4*>(F + p * fstride)[i];
            reinterpret_cast<float4*>(fs.out[0][p] + (int64_t)a * 512)[i] =
                reinterpret_cast<const float4*>(F + (NP + p) * fstride)[i];
        }
}

template <int KIND, int NP>
static int launch_solve(const FieldSet& fs, const uint8_t* mask, const int32_t* nn, int n, const GridInfo& gi, int nsteps,
                        bool again, cudaStream_t s) {
    auto kern = k_solve_cluster<KIND, NP>;
    int ctas = 1;
    while (ctas < kSolveCtas && ctas < n) ctas *= 2;
    const int cap = (n + ctas - 1) / ctas;
    const size_t smem = solve_smem<NP>(cap);
    if (smem > kMaxDynamicSmem) return SGB_ENOTSUP;
    SGB_TRY(allow_max_smem(kern));
    SGB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(kSolveThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess || clusters < 1) {
        cudaGetLastError();  // the device has no room for such a cluster: one launch per step
        return SGB_ENOTSUP;
    }
    SGB_CUDA(cudaLaunchKernelEx(&cfg, kern, fs, mask, nn, n, gi, nsteps, cap, again ? 1 : 0));
    return SGB_OK;
}

// 4^3 chunks: all steps in one cooperative launch (all CTAs resident).  Each CTA takes chunks blockIdx.x + k *
// gridDim.x, a thread per cell of the 6^3 tile with the mask tested for each, and the CTAs meet at a grid barrier (an
// arrival counter, a bounded wait) before the next step reads what the last one wrote.  Field reads bypass L1 (other
// SMs wrote them during the launch).  Arithmetic and stores are those of k_stencil_tile.
template <int KIND>
__global__ void __launch_bounds__(256) k_steps_coop4(FieldSet fs, const uint8_t* __restrict__ mask,
                                                     const int32_t* __restrict__ nn, int64_t n, GridInfo gi, int nsteps,
                                                     unsigned* bar, unsigned* err) {
    constexpr int E = 4, T = E + 2, TT = T * T * T, BS = E * E * E;
    constexpr int NP = KIND == SGB_GS7 ? 2 : 1;
    __shared__ float tile[NP][TT];
    __shared__ int abort_run;
    if (threadIdx.x == 0) abort_run = 0;
    // the thread's cell of the tile: its neighbour slot (6: the chunk itself, -1: an edge, which 7 points do not use)
    // and its offset there
    const int tx = threadIdx.x % T, ty = threadIdx.x / T % T, tz = threadIdx.x / (T * T);
    const int dx = tx == 0 ? -1 : (tx == T - 1), dy = ty == 0 ? -1 : (ty == T - 1), dz = tz == 0 ? -1 : (tz == T - 1);
    const int out = (dx != 0) + (dy != 0) + (dz != 0);
    const int slot = threadIdx.x >= TT || out > 1 ? -1 : !out ? 6 : dx ? (dx > 0) : dy ? 2 + (dy > 0) : 4 + (dz > 0);
    const int off = (tx + E - 1) % E + E * ((ty + E - 1) % E + E * ((tz + E - 1) % E));
    for (int t = 0; t < nsteps; ++t) {
        const int par = t & 1;
        const float* src[2] = {par ? fs.in[1][0] : fs.in[0][0], par ? fs.in[1][NP - 1] : fs.in[0][NP - 1]};
        float* d0 = par ? fs.out[1][0] : fs.out[0][0];
        float* d1 = par ? fs.out[1][NP - 1] : fs.out[0][NP - 1];
        for (int64_t chunk = blockIdx.x; chunk < n; chunk += gridDim.x) {
            if (slot >= 0) {
                const int64_t sc = slot == 6 ? chunk : nn[chunk * 8 + slot];
                const int64_t idx = sc * BS + off;
                const bool ex = sc >= 0 && mask[idx] != 0;
#pragma unroll
                for (int p = 0; p < NP; ++p)
                    tile[p][threadIdx.x] = ex ? __ldcg(src[p] + idx) : (par ? gi.bck[1][p] : gi.bck[0][p]);
            }
            __syncthreads();
            if (threadIdx.x < BS) {
                const int x = threadIdx.x % E, y = threadIdx.x / E % E, z = threadIdx.x / (E * E);
                const int64_t gidx = chunk * BS + threadIdx.x;
                const uint8_t m = mask[gidx];
                const bool act = (m & 1) && !(m & 2);
                const int c = (x + 1) + T * ((y + 1) + T * (z + 1));
                auto lap_of = [&](const float* f) {
                    return lap7k<KIND>(f[c], f[c - 1], f[c + 1], f[c - T], f[c + T], f[c - T * T], f[c + T * T]);
                };
                if (KIND == SGB_HEAT7) {
                    const float cur = tile[0][c];
                    d0[gidx] = act ? __fmaf_rn(gi.dt, lap_of(tile[0]), cur) : (m ? cur : (par ? gi.bck[0][0] : gi.bck[1][0]));
                } else if (act) {
                    float un, vn;
                    gs_update(tile[0][c], tile[NP - 1][c], lap_of(tile[0]), lap_of(tile[NP - 1]), gi, un, vn);
                    d0[gidx] = un;
                    d1[gidx] = vn;
                }
            }
            __syncthreads();
        }
        if (t + 1 < nsteps) {
            // arrival t + 1 of every CTA; the counter only grows.  Every thread fences its stores of this step
            // before the CTA arrives.
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) {
                __threadfence();
                atomicAdd(bar, 1u);
                if (!counter_wait_bounded(bar, (unsigned)(t + 1) * gridDim.x, err)) abort_run = 1;
                __threadfence();
            }
            __syncthreads();
            if (abort_run) return;
        }
    }
}

static int run_steps_coop4(sgb_grid* g, int kind, const FieldSet& fields, const StencilParams& fwd, int nsteps, cudaStream_t s) {
    // Where it is the faster one (whole calls in us, here / a launch per step, heat; Gray-Scott within 10 %): 8 chunks
    // 100 steps 197 / 221, 12 chunks 232 / 221; 148 chunks 8 steps 24 / 24, 5 steps 17 / 18, 3 steps 11 / 14; 444 chunks
    // 3 steps 13 / 13, 592 chunks 15 / 14.
    const int64_t sms = g->num_sms;
    if (!(g->n <= 8 || (g->n <= sms && nsteps <= 8) || (g->n <= 3 * sms && nsteps <= 3))) return SGB_ENOTSUP;
    if ((int64_t)nsteps * g->n >= (int64_t(1) << 31)) return SGB_ENOTSUP;  // arrival counter range
    if (is_capturing(s)) return SGB_ENOTSUP;  // the counter is allocated by the first call
    FieldSet fs = fields;
    GridInfo gi = grid_info_of(fwd);
    const uint8_t* mask = g->mask.as<uint8_t>();
    const int32_t* nn = g->nn[SGB_NN_STAR].as<int32_t>();
    int64_t n = g->n;
    unsigned* err = g->err.as<unsigned>();
    SGB_TRY(g->scratch[11].ensure(64));
    unsigned* bar = g->scratch[11].as<unsigned>();
    const void* kern = kind == SGB_GS7 ? (const void*)k_steps_coop4<SGB_GS7> : (const void*)k_steps_coop4<SGB_HEAT7>;
    int per_sm = 0;
    SGB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, 0));
    if (per_sm < 1) return SGB_ENOTSUP;
    SGB_CUDA(cudaMemsetAsync(bar, 0, 4, s));
    const int64_t blocks = std::min<int64_t>(n, (int64_t)per_sm * g->num_sms);
    void* args[] = {&fs, &mask, &nn, &n, &gi, &nsteps, &bar, &err};
    SGB_CUDA(cudaLaunchCooperativeKernel(kern, dim3((unsigned)blocks), dim3(256), args, 0, s));
    return SGB_OK;
}

int run_steps_one_launch(sgb_grid* g, int kind, const int* src, const int* dst, const StencilParams& fwd, int nsteps,
                      bool again, cudaStream_t s) {
    if ((kind != SGB_HEAT7 && kind != SGB_GS7) || nsteps < 2) return SGB_ENOTSUP;
    const int np = kind == SGB_GS7 ? 2 : 1;
    FieldSet fs;
    for (int j = 0; j < 2; ++j) {
        fs.in[0][j] = g->data[src[j < np ? j : 0]].as<float>();
        fs.out[0][j] = g->data[dst[j < np ? j : 0]].as<float>();
        fs.in[1][j] = g->data[dst[j < np ? j : 0]].as<float>();
        fs.out[1][j] = g->data[src[j < np ? j : 0]].as<float>();
    }
    if (g->geo.edge == 4) return run_steps_coop4(g, kind, fs, fwd, nsteps, s);
    // Up to the chunks at which a launch per step is as fast, within 5 % for full and half-full chunks: heat while a
    // CTA's half chunks take one round of its 32 groups, Gray-Scott a little over half of that.  Whole calls in us, here /
    // a launch per step (which takes 2.2 to 2.6 us on the hosts measured), full chunks and half-full ones: heat 256
    // chunks 3 steps 13 / 14 and 13 / 14, 100 steps 215 / 229 and 240 / 242; 288 chunks 100 steps 267 / 240 and
    // 309 / 244.  Gray-Scott 144 chunks 3 steps 13 / 14 and 15 / 14, 100 steps 236 / 262 and 277 / 277; 160 chunks 3
    // steps 15 / 14 and 15 / 14, 100 steps 249 / 262 and 291 / 278; 192 chunks 100 steps 273 / 266 and 311 / 286.
    if (g->n > (np == 1 ? 16 : 10) * kSolveCtas || nsteps > (1 << 20)) return SGB_ENOTSUP;
    const GridInfo gi = grid_info_of(fwd);
    const uint8_t* mask = g->mask.as<uint8_t>();
    const int32_t* nn = g->nn[SGB_NN_STAR].as<int32_t>();
    return kind == SGB_GS7 ? launch_solve<SGB_GS7, 2>(fs, mask, nn, (int)g->n, gi, nsteps, again, s)
                           : launch_solve<SGB_HEAT7, 1>(fs, mask, nn, (int)g->n, gi, nsteps, again, s);
}

}  // namespace sgb
