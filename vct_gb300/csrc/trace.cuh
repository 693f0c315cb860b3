// What the cone tracer's two kernels share (trace.cu: a warp to 32 pixels;
// trace_split.cu: four): the cones of a pixel and its colour
// (shaders/phong.frag:455-520), pixel tiles, and the choice of a kernel by
// sampler and kind of march.
#pragma once

#include <type_traits>

#include "cone.cuh"

namespace vct {

// The split kernel, over the tiles of `S`.
template <class Scenes>
void launch_trace_split(const Scenes& S, int filter, int kind, long long tiles, int num_sms, bool overlap, cudaStream_t s);

namespace {

using namespace cone;

__constant__ float kConeDir[6][3] = {{0.f, 1.f, 0.f},
                                     {0.f, 0.5f, 0.866025f},
                                     {0.823639f, 0.5f, 0.267617f},
                                     {0.509037f, 0.5f, -0.700629f},
                                     {-0.5909037f, 0.5f, -0.700629f},  // sic, phong.frag:475
                                     {-0.823639f, 0.5f, 0.267617f}};
__constant__ float kConeWeight[6] = {0.25f, 0.15f, 0.15f, 0.15f, 0.15f, 0.15f};

__device__ __forceinline__ f3 volume_position(const TraceParams& P, float4 gp) {
    const f3 ext = sub(P.vmax, P.vmin);
    return mk(((gp.x - P.vcenter.x) - P.vmin.x) / ext.x, ((gp.y - P.vcenter.y) - P.vmin.y) / ext.y,
              ((gp.z - P.vcenter.z) - P.vmin.z) / ext.z);
}

// Orthonormal basis from N: Duff et al. 2017, "Building an Orthonormal Basis,
// Revisited" (JCGT 6(1)).
__device__ __forceinline__ void tangents(f3 N, f3& T, f3& B) {
    const float sgn = N.z >= 0.0f ? 1.0f : -1.0f;
    const float ca = -1.0f / (sgn + N.z);
    const float cb = N.x * N.y * ca;
    T = mk(1.0f + sgn * N.x * N.x * ca, sgn * cb, -sgn * N.x);
    B = mk(cb, sgn + N.y * N.y * ca, -N.y);
}

__device__ __forceinline__ f3 diffuse_direction(const TraceParams& P, int c, f3 N, f3 T, f3 B) {
    const float dx = kConeDir[c][0], dy = kConeDir[c][1], dz = kConeDir[c][2];
    return P.ref_tbn_quirk ? add(add(mul(T, dx), mul(B, dy)), mul(N, dz)) : sub(add(mul(T, dx), mul(N, dy)), mul(B, dz));
}

__device__ __forceinline__ f3 reflected(const TraceParams& P, float4 gp, f3 N) {
    const f3 I = sub(mk(gp.x, gp.y, gp.z), P.eye);
    return sub(I, mul(N, 2.0f * dot(N, I)));
}

__device__ __forceinline__ float4 add_cone(float4 ind, float w, float4 cr) {
    return make_float4(fmaf(w, cr.x, ind.x), fmaf(w, cr.y, ind.y), fmaf(w, cr.z, ind.z), fmaf(w, cr.w, ind.w));
}

// The pixel's colour from its gathered light (phong.frag:500-520).
__device__ __forceinline__ float4 composite(const TraceParams& P, long long pix, float4 ind, float4 spc) {
    f3 rgb;
    // the albedo is loaded after the cones: it is not live across them
    const float4 ga = __ldg(P.galb + pix);
    if (P.enable_indirect) {
        const float occ = 1.0f - clampf(ind.w, 0.0f, 1.0f);
        rgb = mk(ind.x, ind.y, ind.z);
        if (P.enable_reflections) rgb = add(rgb, mul(mk(spc.x, spc.y, spc.z), P.reflect_scale));
        const float as = P.ambient_scale;
        rgb = mk(rgb.x * (as * ga.x), rgb.y * (as * ga.y), rgb.z * (as * ga.z));
        if (P.draw_occlusion) rgb = mul(rgb, occ);
    } else {
        rgb = mk(P.ambient_scale * ga.x, P.ambient_scale * ga.y, P.ambient_scale * ga.z);
    }
    if (P.enable_postprocess) {
        const float g = 1.0f / 2.2f;
        rgb = mk(powf(rgb.x / (rgb.x + 1.0f), g), powf(rgb.y / (rgb.y + 1.0f), g), powf(rgb.z / (rgb.z + 1.0f), g));
    }
    return make_float4(rgb.x, rgb.y, rgb.z, 1.0f);
}

__device__ __forceinline__ void store_pixel(const TraceParams& P, long long pix, float4 irr, float4 spc, float4 out) {
    if (P.irradiance) P.irradiance[pix] = irr;
    if (P.specular) P.specular[pix] = spc;
    if (P.color) P.color[pix] = out;
}

// Pixel of lane `lane` of sub-tile `sub` of a tile of 2^tile_w_log2 x
// 2^tile_h_log2 = 256 pixels (a tuning setting); a sub-tile, a warp's share,
// is 2^warp_w_log2 x 32/2^warp_w_log2.
__device__ __forceinline__ void tile_pixel(const TraceParams& P, long long tile, int sub, int lane, int& x, int& y) {
    const int twl = P.tile_w_log2, thl = P.tile_h_log2, wwl = P.warp_w_log2;
    const int tiles_x = (P.width + (1 << twl) - 1) >> twl;
    const int tx = (int)(tile % tiles_x), ty = (int)(tile / tiles_x);
    const int wxl = twl - wwl;  // log2 of warps per tile row
    x = (tx << twl) + ((sub & ((1 << wxl) - 1)) << wwl) + lane_x(lane, wwl);
    y = (ty << thl) + ((sub >> wxl) << (5 - wwl)) + lane_y(lane, wwl);
}

__device__ __forceinline__ void count_samples(const TraceParams& P, unsigned ns) {
    if (P.samples) {
        unsigned tot = __reduce_add_sync(0xffffffffu, ns);
        if ((threadIdx.x & 31) == 0 && tot) atomicAdd(P.samples, (unsigned long long)tot);
    }
}

template <class Scenes>
void launch_tiles(void (*kernel)(Scenes), const Scenes& S, long long ctas, bool overlap, cudaStream_t s) {
    if (overlap) {
        launch_overlapped(kernel, dim3((unsigned)ctas), 256, 0, s, S);
    } else {
        kernel<<<(unsigned)ctas, 256, 0, s>>>(S);
        note_launches(1);
    }
}

// f(sampler, kind) with the two as integral constants.
template <class F>
void with_trace_mode(int filter, int kind, F f) {
    auto with_kind = [&](auto mode) {
        if (kind == kConesPlain)
            f(mode, std::integral_constant<int, kConesPlain>());
        else if (kind == kConesMapped)
            f(mode, std::integral_constant<int, kConesMapped>());
        else
            f(mode, std::integral_constant<int, kConesAny>());
    };
    if (filter == VCT_FILTER_HARDWARE)
        with_kind(std::integral_constant<int, VCT_FILTER_HARDWARE>());
    else if (filter == VCT_FILTER_HARDWARE_LEVELS)
        with_kind(std::integral_constant<int, VCT_FILTER_HARDWARE_LEVELS>());
    else if (filter == VCT_FILTER_HYBRID)
        with_kind(std::integral_constant<int, VCT_FILTER_HYBRID>());
    else
        with_kind(std::integral_constant<int, VCT_FILTER_SOFTWARE>());
}

}  // namespace
}  // namespace vct
