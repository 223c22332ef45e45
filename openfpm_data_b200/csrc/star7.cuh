// Arithmetic and stores of the 7-point kernels: an x quad (four x-adjacent points) per lane.
#pragma once

#include "stencil.cuh"

namespace sgb {

// Plain (coherent) global loads: under programmatic dependent launch a block
// may start before the step that wrote these fields has finished, so the
// read-only path, which asks for data that is constant while the kernel runs,
// is not used for fields.
__device__ __forceinline__ float4 ldf4(const float* p) {
    float4 v;
    asm("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float ldf1(const float* p) {
    float v;
    asm("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 splat4(float b) { return make_float4(b, b, b, b); }
__device__ __forceinline__ uint32_t ldm4(const uint8_t* m) { return __ldg(reinterpret_cast<const uint32_t*>(m)); }
// The background b where a quad's mask byte is 0.
__device__ __forceinline__ float4 masked4(float4 v, uint32_t m4, float b) {
    v.x = m4 & 0xffu ? v.x : b;
    v.y = m4 & 0xff00u ? v.y : b;
    v.z = m4 & 0xff0000u ? v.z : b;
    v.w = m4 & 0xff000000u ? v.w : b;
    return v;
}

// Two float32 values in one 64-bit register pair and the packed arithmetic on them (each half rounds as the
// scalar instruction does).
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pk(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 upk(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
struct Quad {
    f32x2 a, b;  // points 0, 1 and 2, 3
};
__device__ __forceinline__ Quad quad(const float4& v) { return {pk(v.x, v.y), pk(v.z, v.w)}; }

// 7-point Laplacian of an x quad: lap7k of stencil.cuh point by point, the same operations in the same order.
template <int KIND>
__device__ __forceinline__ Quad lap_quad(const float4& c, float xm, float xp, const float4& ym, const float4& yp,
                                         const float4& zm, const float4& zp) {
    const Quad qym = quad(ym), qyp = quad(yp), qzm = quad(zm), qzp = quad(zp);
    // the x sums take unaligned pairs: scalar
    const f32x2 xa = pk(__fadd_rn(xm, c.y), __fadd_rn(c.x, c.z)), xb = pk(__fadd_rn(c.y, c.w), __fadd_rn(c.z, xp));
    Quad l;
    if (KIND == SGB_HEAT7) {
        const f32x2 m6 = pk(-6.0f, -6.0f);
        const Quad qc = quad(c);
        l.a = fma2(m6, qc.a, xa);
        l.b = fma2(m6, qc.b, xb);
    } else {
        // -6 c rounds on its own: scalar products, which the assembler leaves apart from the packed sum
        l.a = add2(pk(__fmul_rn(-6.0f, c.x), __fmul_rn(-6.0f, c.y)), xa);
        l.b = add2(pk(__fmul_rn(-6.0f, c.z), __fmul_rn(-6.0f, c.w)), xb);
    }
    l.a = add2(add2(l.a, add2(qym.a, qyp.a)), add2(qzm.a, qzp.a));
    l.b = add2(add2(l.b, add2(qym.b, qyp.b)), add2(qzm.b, qzp.b));
    return l;
}

// gs_update of two points.
__device__ __forceinline__ void gs_update2(f32x2 u, f32x2 v, f32x2 lu, f32x2 lv, const GridInfo& g, f32x2& un, f32x2& vn) {
    const f32x2 uvv = mul2(mul2(u, v), v);
    const f32x2 one = pk(1.0f, 1.0f), sgn = 0x8000000080000000ull;
    f32x2 du = fma2(pk(g.Du, g.Du), lu, uvv ^ sgn);
    du = fma2(pk(g.F, g.F), add2(one, u ^ sgn), du);
    f32x2 dv = fma2(pk(g.Dv, g.Dv), lv, uvv);
    dv = fma2(pk(g.nFK, g.nFK), v, dv);
    un = fma2(pk(g.dt, g.dt), du, u);
    vn = fma2(pk(g.dt, g.dt), dv, v);
}

// The update of one x quad and its stores.  m4: the quad's mask bytes; act bit k: point k takes the update.
template <int KIND, int NP>
__device__ __forceinline__ void star_store(const float4 (&c)[NP], const Quad (&lap)[NP], uint32_t m4, uint32_t act,
                                           const GridInfo& gi, const float (&bd)[NP], float* d0, float* d1) {
    Quad w[NP];
    const Quad c0 = quad(c[0]);
    if (KIND == SGB_HEAT7) {
        const f32x2 dt = pk(gi.dt, gi.dt);
        w[0].a = fma2(dt, lap[0].a, c0.a);
        w[0].b = fma2(dt, lap[0].b, c0.b);
    } else {
        const Quad c1 = quad(c[NP - 1]);
        gs_update2(c0.a, c1.a, lap[0].a, lap[NP - 1].a, gi, w[0].a, w[NP - 1].a);
        gs_update2(c0.b, c1.b, lap[0].b, lap[NP - 1].b, gi, w[0].b, w[NP - 1].b);
    }
    float4 o[NP];
#pragma unroll
    for (int p = 0; p < NP; ++p) {
        const float2 lo = upk(w[p].a), hi = upk(w[p].b);
        o[p] = make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    if (act != 0xfu) {
        const bool e0 = m4 & 0xffu, e1 = m4 & 0xff00u, e2 = m4 & 0xff0000u, e3 = m4 & 0xff000000u;
        if (KIND == SGB_HEAT7) {
            // inactive points: an existing one keeps its value, the others take the destination's background
            o[0].x = (act & 1u) ? o[0].x : (e0 ? c[0].x : bd[0]);
            o[0].y = (act & 2u) ? o[0].y : (e1 ? c[0].y : bd[0]);
            o[0].z = (act & 4u) ? o[0].z : (e2 ? c[0].z : bd[0]);
            o[0].w = (act & 8u) ? o[0].w : (e3 ? c[0].w : bd[0]);
        } else {
            const uint32_t ex = (e0 ? 1u : 0u) | (e1 ? 2u : 0u) | (e2 ? 4u : 0u) | (e3 ? 8u : 0u);
            if (ex & ~act) {  // existing inactive points (padding, outside the box) are left alone
                const float u4[4] = {o[0].x, o[0].y, o[0].z, o[0].w};
                const float v4[4] = {o[NP - 1].x, o[NP - 1].y, o[NP - 1].z, o[NP - 1].w};
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (act >> k & 1u) {
                        d0[k] = u4[k];
                        d1[k] = v4[k];
                    }
                return;
            }
            // points that do not exist take the destination's background, which no read can tell from
            // what they hold: one whole store
#pragma unroll
            for (int p = 0; p < NP; ++p) {
                o[p].x = (act & 1u) ? o[p].x : bd[p];
                o[p].y = (act & 2u) ? o[p].y : bd[p];
                o[p].z = (act & 4u) ? o[p].z : bd[p];
                o[p].w = (act & 8u) ? o[p].w : bd[p];
            }
        }
    }
    *reinterpret_cast<float4*>(d0) = o[0];
    if (NP > 1) *reinterpret_cast<float4*>(d1) = o[NP - 1];
}

// Backgrounds for a quad's points that do not exist beside existing ones that star_store leaves alone (mask bytes with
// more than EXIST; it has written all other quads whole).  Steps without a box only: solves.
template <int NP>
__device__ __forceinline__ void star_rest(uint32_t m4, const float (&bd)[NP], float* d0, float* d1) {
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (!(m4 >> 8 * k & 0xffu)) {
            d0[k] = bd[0];
            d1[k] = bd[NP - 1];
        }
}

// Bits of the quad's active points: EXIST and not PADDING, inside the box.
template <bool BOX, typename Args>
__device__ __forceinline__ uint32_t active_bits(uint32_t m4, const Args& box, int x, int y, int z) {
    // per byte: bit 0 set and bit 1 clear
    if (!BOX && m4 == 0x01010101u) return 0xfu;
    uint32_t a = m4 & ~(m4 >> 1) & 0x01010101u;
    a = (a | a >> 7 | a >> 14 | a >> 21) & 0xfu;
    if constexpr (BOX) {
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (!in_box(box.prm, x + k, y, z)) a &= ~(1u << k);
    }
    return a;
}

}  // namespace sgb
