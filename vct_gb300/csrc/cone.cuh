// Cone marching shared by the cone tracer (trace.cu) and the learned path
// (learned.cu): textureLod with GL_LINEAR_MIPMAP_LINEAR semantics over the
// radiance chain (shaders/phong.frag:135-180; sampler of
// src/Application.cpp:1088-1116) and the front-to-back cone march.
//
// Every fused multiply-add is written out (fmaf, __ffma2_rn); the including
// translation units are compiled without FMA contraction, so every
// instantiation rounds the same way.  The one exception is the warp map's lookup
// (warp.cuh), whose packed products and sums the compiler fuses all the same, in
// every instantiation: the tests compare them bit for bit.
#pragma once

#include "vct_device.cuh"

namespace vct {
namespace cone {

__device__ __forceinline__ f3 fnormalize(f3 v) { return mul(v, rsqrtf(dot(v, v))); }

// Texel (i, j, k) of level 0 from the bordered chain (0 outside the level).
__device__ __forceinline__ float4 texel0(const float4* __restrict__ pchain, int S, int i, int j, int k) {
    if ((unsigned)i >= (unsigned)S || (unsigned)j >= (unsigned)S || (unsigned)k >= (unsigned)S)
        return make_float4(0.f, 0.f, 0.f, 0.f);
    const int Pd = S + 2;
    return __ldg(pchain + (((k + 1) * Pd + (j + 1)) * Pd + (i + 1)));
}

// RGBA as two packed fp32 pairs: Blackwell issues one FFMA2/FMUL2 per pair.
struct rgba2 {
    float2 rg, ba;
};

__device__ __forceinline__ rgba2 from_float4(float4 v) { return {make_float2(v.x, v.y), make_float2(v.z, v.w)}; }

// The bordered chain holds each binary16 texel widened to fp32 (exactly), so
// a texel is one 16-byte read-only load with no conversion.
__device__ __forceinline__ rgba2 ld_texel(const float4* __restrict__ p) {
    return from_float4(__ldg(p));
}

// t*q + (p - t*p) on both pairs: two FFMA2 per pair.
__device__ __forceinline__ rgba2 lerp2(rgba2 p, rgba2 q, float t) {
    const float2 tt = make_float2(t, t), nt = make_float2(-t, -t);
    return {__ffma2_rn(tt, q.rg, __ffma2_rn(nt, p.rg, p.rg)), __ffma2_rn(tt, q.ba, __ffma2_rn(nt, p.ba, p.ba))};
}

__device__ __forceinline__ float4 to_float4(rgba2 v) { return make_float4(v.rg.x, v.rg.y, v.ba.x, v.ba.y); }

// The place of a lane in its warp's 2^wl x 2^(5-wl) pixels: eight lanes, which
// a 16-byte load serves at a time, take a 4 x 2 block (rather than a row of
// 8), whose footprints share more texels and lines.
__device__ __forceinline__ int lane_x(int lane, int wl) {
    return wl < 2 || wl > 4 ? lane & ((1 << wl) - 1) : (lane & 3) | (((lane >> 3) & ((1 << (wl - 2)) - 1)) << 2);
}
__device__ __forceinline__ int lane_y(int lane, int wl) {
    return wl < 2 || wl > 4 ? lane >> wl : ((lane >> 2) & 1) | ((lane >> (wl + 1)) << 1);
}

// What a sample needs to know of a level: the side S as a float, the row and
// slice strides of the bordered level, and the texel offset at which integers
// taken from the float trick below index it.
struct __align__(16) Level {
    float side;
    uint32_t row, slice, base;
};

// floor of a float by adding 1.5 x 2^23, rounding down: the sum's bits are the
// integer plus kRoundBits.
constexpr float kRound = 12582912.0f;
constexpr uint32_t kRoundBits = 0x4B400000u;

__device__ __forceinline__ Level level_of(int dim, int l) {
    Level v;
    v.side = (float)(dim >> l);
    v.row = (uint32_t)(dim >> l) + 2u;
    v.slice = v.row * v.row;
    // (the lower corner -1 of a footprint is texel 0)
    v.base = (uint32_t)padded_level_offset(dim, l) - (kRoundBits - 1u) * (1u + v.row + v.slice);
    return v;
}
__device__ __forceinline__ void fill_levels(const TraceParams& P, Level* lv) {
    if (threadIdx.x < VCT_MAX_LEVELS)
        lv[threadIdx.x] = level_of(P.dim, min((int)threadIdx.x, P.levels - 1));
}

// GL_LINEAR within level l with a (0,0,0,0) border, read from the bordered
// chain: for a position in [0,1]^3 the footprint's lower corner is in
// [-1, S-1]^3, i.e. [0, S]^3 of the (S+2)^3 bordered level, so the eight
// texels are plain loads at constant offsets with no bounds tests.
//
// The floors come from additions and the texel index from the sums' bits:
// no rounding or conversion instructions, which run at a quarter of the rate.
//
// With `guard` (warped positions: about an eye outside the volume, or
// projected by the perspective warp, they can leave [0,1]^3) the footprint is
// checked first: the bordered level holds texel indices -1..S, i.e. u = p S - 1/2 in [-1, S); outside that every texel of
// the footprint is border and the sample is (0,0,0,0).
__device__ __forceinline__ rgba2 trilinear2(const float4* __restrict__ pchain, const Level lv, f3 p, bool guard = false) {
    const float S = lv.side;
    const float u = fmaf(p.x, S, -0.5f), v = fmaf(p.y, S, -0.5f), w = fmaf(p.z, S, -0.5f);
    if (guard && !(u >= -1.0f && v >= -1.0f && w >= -1.0f && u < S && v < S && w < S))
        return {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    const float ru = __fadd_rd(u, kRound), rv = __fadd_rd(v, kRound), rw = __fadd_rd(w, kRound);
    const float a = u - (ru - kRound), b = v - (rv - kRound), c = w - (rw - kRound);
    const uint32_t at = lv.base + __float_as_uint(ru) + __float_as_uint(rv) * lv.row + __float_as_uint(rw) * lv.slice;
    const float4* q = pchain + at;
    const uint32_t sy = lv.row, sz = lv.slice;
    const rgba2 t0 = ld_texel(q), t1 = ld_texel(q + 1), t2 = ld_texel(q + sy), t3 = ld_texel(q + sy + 1);
    const rgba2 t4 = ld_texel(q + sz), t5 = ld_texel(q + sz + 1), t6 = ld_texel(q + sz + sy),
                t7 = ld_texel(q + sz + sy + 1);
    const rgba2 x00 = lerp2(t0, t1, a), x10 = lerp2(t2, t3, a);
    const rgba2 x01 = lerp2(t4, t5, a), x11 = lerp2(t6, t7, a);
    return lerp2(lerp2(x00, x10, b), lerp2(x01, x11, b), c);
}

__device__ __forceinline__ float4 trilinear(const float4* pchain, const Level lv, f3 p, bool guard = false) {
    return to_float4(trilinear2(pchain, lv, p, guard));
}

// The level choice of textureLod at `lambda`: level l and, with weight f, the
// next one; magnification (lambda <= 0) and the chain's last level (lambda >=
// its index) read one.
struct __align__(16) Lod {
    float h;       // the cone step's distance from the start, in voxels
    float lambda;
    float f;
    int l;         // level, or one of:
};
constexpr int kLodNearest = -1, kLodLast = -2, kLodStop = -3;  // kLodStop: the cone has no such step

__device__ __forceinline__ Lod choose_lod(float h, float lambda, int last) {
    Lod d = {h, lambda, 0.0f, kLodNearest};
    if (!(lambda <= 0.0f)) {
        const float fl = floorf(lambda);
        d.f = lambda - fl;
        d.l = lambda >= (float)last ? kLodLast : (int)fl;
    }
    return d;
}

template <int MODE>
__device__ __forceinline__ rgba2 sample_lod(const TraceParams& P, const Level* lv, f3 p, const Lod d, bool guard) {
    if (MODE == VCT_FILTER_HARDWARE) return from_float4(tex3DLod<float4>(P.tex, p.x, p.y, p.z, d.lambda));
    const int q = P.levels - 1;
    if (MODE == VCT_FILTER_HARDWARE_LEVELS) {
        // Texture units filter within each level; the two levels are blended
        // with the exact fp32 fraction (GL_LINEAR_MIPMAP_LINEAR level choice).
        if (d.l == kLodNearest) return from_float4(tex3DLod<float4>(P.tex, p.x, p.y, p.z, 0.0f));
        if (d.l == kLodLast) return from_float4(tex3DLod<float4>(P.tex, p.x, p.y, p.z, (float)q));
        return lerp2(from_float4(tex3DLod<float4>(P.tex, p.x, p.y, p.z, (float)d.l)),
                     from_float4(tex3DLod<float4>(P.tex, p.x, p.y, p.z, (float)(d.l + 1))), d.f);
    }
    if (MODE == VCT_FILTER_HYBRID && d.l >= 0) {
        // The level with the larger weight exactly, the other one by the
        // texture units at its integral level: the texture units' fixed-point
        // filter weights then enter the sample scaled by at most 1/2.  (The
        // step's level is the same in every lane, so the choice is uniform.)
        if (d.f <= 0.5f) {
            const rgba2 fine = trilinear2(P.pchain, lv[d.l], p, guard);
            return lerp2(fine, from_float4(tex3DLod<float4>(P.tex, p.x, p.y, p.z, (float)(d.l + 1))), d.f);
        }
        const float4 c = tex3DLod<float4>(P.tex, p.x, p.y, p.z, (float)d.l);
        return lerp2(from_float4(c), trilinear2(P.pchain, lv[d.l + 1], p, guard), d.f);
    }
    if (d.l == kLodNearest) {  // magnification: GL_NEAREST on level 0 (index S = border)
        const int S = P.dim;
        return from_float4(texel0(P.pchain + padded_level_offset(P.dim, 0), S, (int)floorf(p.x * S),
                                  (int)floorf(p.y * S), (int)floorf(p.z * S)));
    }
    if (d.l == kLodLast) return trilinear2(P.pchain, lv[q], p, guard);
    return lerp2(trilinear2(P.pchain, lv[d.l], p, guard), trilinear2(P.pchain, lv[d.l + 1], p, guard), d.f);
}

// A cone's steps do not depend on what it meets: their distances and levels
// are the same for every cone of a setting, so a CTA computes them once (by
// the recurrence, h += h tan(angle / 2)) and the march reads them.
constexpr int kConeSteps = kConeTableSteps;
struct ConeTable {
    Lod step[kConeSteps + 1];  // the step after the last one stops
};
// By threads first .. first + kConeSteps of the CTA.
__device__ __forceinline__ void fill_cone(const TraceParams& P, const vct_cone_settings& c, float maxd, ConeTable& T,
                                          int first) {
    const int i = (int)threadIdx.x - first;
    if (i < 0 || i >= kConeSteps || i > c.steps) return;  // (the step after the last one stops)
    const float scale = 1.0f / (float)P.dim, tanh = tanf(c.cone_angle * 0.5f);
    float h = c.cone_initial_height;
    for (int k = 0; k < i; ++k) h += h * tanh;
    Lod d = choose_lod(h, __log2f(fmaxf(1.0f, 2.0f * (h * tanh))) + c.lod_offset, P.levels - 1);
    if (i >= c.steps || h * scale > maxd) d.l = kLodStop;
    T.step[i] = d;
    if (i == 0) T.step[kConeSteps].l = kLodStop;
}

// KIND: no more steps than the table holds and no warp, the
// same with the warp map, or any.
//
// PAIRS (for kernels of few warps, with registers to spare; no warp): two
// steps at a time where both blend two levels, the second one's texels loaded
// before the first one's colour is added, and dropped where the march ends
// with the first.
template <int MODE, int KIND, bool PAIRS = false>
__device__ __forceinline__ float4 trace_cone(const TraceParams& P, const Level* lv, const ConeTable& T, f3 pos, f3 n,
                                             f3 dir, const vct_cone_settings& c, float maxd, unsigned& ns) {
    dir = fnormalize(dir);
    const float scale = 1.0f / (float)P.dim;
    const f3 start = add(pos, mul(mul(n, c.bias), scale));
    const bool guard = KIND == kConesAny && P.warp.mode != VCT_WARP_NONE;
    rgba2 acc = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};  // colour, and the opacity
    auto position = [&](const Lod d) {
        const f3 dh = mul(dir, d.h);
        return mk(fmaf(dh.x, scale, start.x), fmaf(dh.y, scale, start.y), fmaf(dh.z, scale, start.z));
    };
    // (not outside, nor NaN)
    auto inside = [](f3 p) { return p.x >= 0.f && p.y >= 0.f && p.z >= 0.f && p.x <= 1.f && p.y <= 1.f && p.z <= 1.f; };
    // Adds a sample: false when the cone is full.
    auto take = [&](const rgba2 s) {
        ++ns;
        const float a = 1.0f - acc.ba.y;
        const float2 aa = make_float2(a, a);
        acc = {__ffma2_rn(s.rg, aa, acc.rg), __ffma2_rn(s.ba, aa, acc.ba)};
        return acc.ba.y < 0.95f;
    };
    // One step: false when the cone leaves the volume or is full.
    auto march = [&](const Lod d) {
        const f3 sp = position(d);
        if (!inside(sp)) return false;
        f3 wp = sp;
        if (KIND == kConesMapped) {
            // saturated: a sample's footprint has to lie in the bordered level
            wp = warp_lookup<true>(P.warp.mapf, sp);
            wp = mk(__saturatef(wp.x), __saturatef(wp.y), __saturatef(wp.z));
        } else if (KIND == kConesAny) {
            wp = apply_warp(P.warp, sp);
        }
        return take(sample_lod<MODE>(P, lv, wp, d, guard));
    };
    bool on = true;
    const Lod* step = T.step;
    if (PAIRS) {
        static_assert(!PAIRS || (KIND == kConesPlain && MODE == VCT_FILTER_SOFTWARE), "pairs of plain software samples");
        while (on) {
            const Lod d0 = step[0];
            if (d0.l < 0) break;
            const Lod d1 = step[1];
            if (d1.l < 0) break;
            const f3 p0 = position(d0), q = position(d1);
            if (!inside(p0)) return to_float4(acc);
            const bool second = inside(q);
            const f3 p1 = second ? q : p0;
            const rgba2 a0 = trilinear2(P.pchain, lv[d0.l], p0), a1 = trilinear2(P.pchain, lv[d0.l + 1], p0);
            const rgba2 b0 = trilinear2(P.pchain, lv[d1.l], p1), b1 = trilinear2(P.pchain, lv[d1.l + 1], p1);
            on = take(lerp2(a0, a1, d0.f)) && second && take(lerp2(b0, b1, d1.f));
            step += 2;
        }
    }
    for (; on; ++step) {
        const Lod d = *step;
        if (d.l == kLodStop) break;
        on = march(d);
    }
    if (KIND == kConesAny && on && c.steps > kConeSteps && step == T.step + kConeSteps) {
        // the steps past the table
        const float tanh = tanf(c.cone_angle * 0.5f);
        float h = T.step[kConeSteps - 1].h;
        for (int i = kConeSteps; i < c.steps && on; ++i) {
            h += h * tanh;
            if (h * scale > maxd) break;
            on = march(choose_lod(h, __log2f(fmaxf(1.0f, 2.0f * (h * tanh))) + c.lod_offset, P.levels - 1));
        }
    }
    return to_float4(acc);
}

}  // namespace cone
}  // namespace vct
