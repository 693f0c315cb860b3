// Device-side helpers shared by the VCT kernels.
//
// The voxelisation, normalisation, injection and mip kernels are compiled
// with --fmad=false: every a*b+c below is two IEEE-rounded operations and
// every division and square root is IEEE-rounded, so their results are
// reproducible bit for bit by any CPU that evaluates the same expressions in
// the same order.  The operation order used here is fixed: it follows the
// GLSL expression order of the reference shaders (left to right).
#pragma once

#include <cuda_fp16.h>
#include <stdint.h>

#include "vct_internal.h"
#include "warp.cuh"

namespace vct {

// ---- the carry table of exact accumulation (vct_internal.h, kCarrySlots)
__device__ __forceinline__ uint32_t carry_slot(uint32_t v, int probe) {
    return (((v * 2654435761u) >> (32 - kCarrySlotsLog2)) + (uint32_t)probe) & (uint32_t)(kCarrySlots - 1);
}
// Adds the crossings ev[] of voxel v to its entry (claimed on first use).
__device__ __forceinline__ void carry_add(uint32_t* table, uint32_t v, const uint32_t (&ev)[kCarryEvents],
                                          StatsDev* stats) {
    const uint32_t key = v + 1u;
    for (int i = 0; i < kCarryProbes; ++i) {
        uint32_t* e = table + 8 * carry_slot(v, i);
        const uint32_t k = atomicCAS(e, 0u, key);
        if (k == 0u || k == key) {
#pragma unroll
            for (int f = 0; f < kCarryEvents; ++f)
                if (ev[f]) atomicAdd(e + 1 + f, ev[f]);
            return;
        }
    }
    atomicOr(&stats->error_flags, VCT_STATS_COUNT_OVERFLOW);
}
// Whether adding `a` to the 64-bit word whose value was `o` carried out of
// the low 32-bit field, and whether the high field (with that carry) wrapped.
__device__ __forceinline__ uint32_t carry_lo(unsigned long long o, unsigned long long a) {
    return (uint32_t)(((o & 0xffffffffull) + (a & 0xffffffffull)) >> 32);
}
__device__ __forceinline__ uint32_t wrap_hi(unsigned long long o, unsigned long long a) {
    return (uint32_t)(((o >> 32) + (a >> 32) + carry_lo(o, a)) >> 32);
}

__device__ __forceinline__ f3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ f3 add(f3 a, f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 sub(f3 a, f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ f3 mul(f3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ f3 mulv(f3 a, f3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ float dot(f3 a, f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ f3 ld3(const float* p) { return {p[0], p[1], p[2]}; }
// a / b rounded to nearest, given y = RN(1 / b): the quotient a y is within 1.5
// units in the last place, its remainder is exact or off by one part in 2^24 in
// one fused multiply-add, and the corrected quotient is the rounded one (after
// P. Markstein, "Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34, 1990, which supposes a first quotient within
// one unit; the operands whose quotient lies near enough to a rounding boundary
// to matter are enumerated in tests/test_quotient.py), as long as nothing on
// the way overflows or underflows; a = 0 gives 0.  Cheaper than the division
// where y is at hand or shared, and above all for a = 0, which takes the
// division's slow path.
__device__ __forceinline__ float quotient(float a, float b, float y) {
    const float q = a * y;
    return fmaf(fmaf(-q, b, a), y, q);
}
// normalize(v) = v * (1 / sqrt(dot(v, v))), both operations IEEE-rounded (the
// rounded reciprocal is the rounded quotient of 1).
__device__ __forceinline__ f3 normalize(f3 v) {
    float inv = __frcp_rn(__fsqrt_rn(dot(v, v)));
    return mul(v, inv);
}
__device__ __forceinline__ float length(f3 v) { return __fsqrt_rn(dot(v, v)); }
__device__ __forceinline__ float clampf(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }
__device__ __forceinline__ float smoothstep(float e0, float e1, float x) {
    float t = clampf(__fdiv_rn(x - e0, e1 - e0), 0.0f, 1.0f);
    return t * t * (3.0f - 2.0f * t);
}

// glm mat4 (column-major) * vec4, columns summed in order.
__device__ __forceinline__ void mat_vec(const float* m, float x, float y, float z, float w, float out[4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r) out[r] = m[0 + r] * x + m[4 + r] * y + m[8 + r] * z + m[12 + r] * w;
}

// ---------------------------------------------------------------- binary16
__device__ __forceinline__ uint16_t f2h(float f) { return __half_as_ushort(__float2half_rn(f)); }
__device__ __forceinline__ float h2f(uint16_t h) { return __half2float(__ushort_as_half(h)); }
__device__ __forceinline__ uint2 pack_h4(float a, float b, float c, float d) {
    const __half2 lo = __floats2half2_rn(a, b), hi = __floats2half2_rn(c, d);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}
__device__ __forceinline__ float4 unpack_h4(uint2 v) {
    float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&v.x));
    float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}

// ------------------------------------------------------- rasterisation core
// Pixel-centre coverage on a 1/256 sub-pixel grid with a top-left tie rule,
// identical to the CPU oracle: window coordinates are snapped with
// rint(w * 256) after clamping to +-2^20 pixels, edge functions are exact
// 64-bit integers, and interpolation weights are e_k * (1 / area) in fp32.
constexpr int kSub = 256;

__device__ __forceinline__ int snap(float w) {
    w = clampf(w, -1048576.0f, 1048576.0f);
    return __float2int_rn(w * 256.0f);
}

// The fp32 value of 0 <= e < 2^46, rounded to nearest even as the conversion
// of a 64-bit integer is: two 23-bit halves become floats exactly (as the low
// bits of 2^23's significand), and one fused multiply-add rounds their sum.
// The conversion instruction for 64-bit integers runs on the FP64 pipe, which
// takes 16 cycles a warp on this chip: three of them per candidate pixel held
// that pipe at 64% and the 2048^2 shadow pass at 0.67 ms.
constexpr long long kHalvesLimit = 1LL << 46;
__device__ __forceinline__ float halves_to_float(long long e) {
    const uint32_t lo = (uint32_t)e, hi = (uint32_t)((unsigned long long)e >> 32);
    const float h = __uint_as_float(0x4B000000u | __funnelshift_l(lo, hi, 9)) - 8388608.0f;
    const float l = __uint_as_float(0x4B000000u | (lo & 0x7fffffu)) - 8388608.0f;
    return fmaf(h, 8388608.0f, l);
}
// `wide`: the triangle's area, which bounds its covered pixels' edge
// functions, is past that range (it reaches some 2^29 pixels).  A call, so
// that the conversion is branched around and not predicated.
static __device__ __noinline__ float wide_to_float(long long e) { return __ll2float_rn(e); }
__device__ __forceinline__ float edge_to_float(long long e, bool wide) {
    return wide ? wide_to_float(e) : halves_to_float(e);
}

struct RasterTri {
    int X[3], Y[3];  // snapped coordinates, within 2^28
    long long area;  // twice the area, positive
    int bias[3];     // -1 for an edge that is not top-left
    int px0, px1, py0, py1;
    int perm1;  // 1: vertices 1 and 2 were swapped to make the triangle CCW
    __device__ __forceinline__ bool wide() const { return area >= kHalvesLimit; }
    __device__ __forceinline__ float area_float() const { return edge_to_float(area, wide()); }
};

__device__ __forceinline__ bool raster_setup(const float wx[3], const float wy[3], int W, int H, RasterTri& t) {
    int X[3], Y[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        X[k] = snap(wx[k]);
        Y[k] = snap(wy[k]);
    }
    long long area = (long long)(X[1] - X[0]) * (long long)(Y[2] - Y[0]) -
                     (long long)(Y[1] - Y[0]) * (long long)(X[2] - X[0]);
    if (area == 0) return false;
    t.perm1 = area < 0;
    if (t.perm1) {
        area = -area;
        const int tx = X[1], ty = Y[1];
        X[1] = X[2];
        Y[1] = Y[2];
        X[2] = tx;
        Y[2] = ty;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        t.X[k] = X[k];
        t.Y[k] = Y[k];
    }
    t.area = area;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        int a = (k + 1) % 3, b = (k + 2) % 3;
        const int dx = X[b] - X[a], dy = Y[b] - Y[a];
        bool tl = (dy < 0) || (dy == 0 && dx < 0);
        t.bias[k] = tl ? 0 : -1;
    }
    const int minx = min(X[0], min(X[1], X[2])), maxx = max(X[0], max(X[1], X[2]));
    const int miny = min(Y[0], min(Y[1], Y[2])), maxy = max(Y[0], max(Y[1], Y[2]));
    // pixel centres within [min, max]: ceil((min - 128) / 256) .. floor((max - 128) / 256)
    t.px0 = max((minx - kSub / 2 + kSub - 1) >> 8, 0);
    t.py0 = max((miny - kSub / 2 + kSub - 1) >> 8, 0);
    t.px1 = min((maxx - kSub / 2) >> 8, W - 1);
    t.py1 = min((maxy - kSub / 2) >> 8, H - 1);
    return t.px0 <= t.px1 && t.py0 <= t.py1;
}

__device__ __forceinline__ float interp(const float l[3], float a, float b, float c) {
    return l[0] * a + l[1] * b + l[2] * c;
}

// ------------------------------------------- bilinear fetch, border 1.0
__device__ __forceinline__ float shadow_fetch(const float* __restrict__ sm, int W, int H, int i, int j) {
    if (i < 0 || j < 0 || i >= W || j >= H) return 1.0f;
    return __ldg(sm + (long long)j * W + i);
}
__device__ __forceinline__ float shadow_bilinear(const float* __restrict__ sm, int W, int H, float u, float v, int ox,
                                                 int oy) {
    float x = (u * (float)W + (float)ox) - 0.5f;
    float y = (v * (float)H + (float)oy) - 0.5f;
    float fx = floorf(x), fy = floorf(y);
    float a = x - fx, b = y - fy;
    int i = (int)fx, j = (int)fy;
    float t00, t10, t01, t11;
    if (i >= 0 && j >= 0 && i < W - 1 && j < H - 1) {
        const float* p = sm + (j * W + i);  // at most 2^30 texels
        t00 = __ldg(p);
        t10 = __ldg(p + 1);
        t01 = __ldg(p + W);
        t11 = __ldg(p + W + 1);
    } else {
        t00 = shadow_fetch(sm, W, H, i, j), t10 = shadow_fetch(sm, W, H, i + 1, j);
        t01 = shadow_fetch(sm, W, H, i, j + 1), t11 = shadow_fetch(sm, W, H, i + 1, j + 1);
    }
    float bot = t00 * (1.0f - a) + t10 * a;
    float top = t01 * (1.0f - a) + t11 * a;
    return bot * (1.0f - b) + top * b;
}

// calcShadowFactor (voxelize.frag:160-184 = phong.frag:183-207): 5-tap PCF of
// the bilinear light-space depth with bias 0.01; 0 beyond the far plane.
__device__ __forceinline__ float pcf5(const float* __restrict__ sm, int sw, int sh, const float* ls, f3 wp) {
    float c[4];
    mat_vec(ls, wp.x, wp.y, wp.z, 1.0f, c);
    // x / 1 == x exactly: skip the divide for an orthographic light.
    if (c[3] != 1.0f) {
        c[0] = __fdiv_rn(c[0], c[3]);
        c[1] = __fdiv_rn(c[1], c[3]);
        c[2] = __fdiv_rn(c[2], c[3]);
    }
    float sx = (c[0] + 1.0f) * 0.5f;
    float sy = (c[1] + 1.0f) * 0.5f;
    float sz = (c[2] + 1.0f) * 0.5f;
    float frag = sz - 0.01f;
    if (frag > 1.0f) return 0.0f;
    // The five taps' footprints share texels: when their corners are one texel
    // apart (they nearly always are; the offsets are added before rounding)
    // and inside the map, 12 loads from one address replace 20 with their
    // border tests.
    const float x[3] = {(sx * (float)sw + -1.0f) - 0.5f, (sx * (float)sw + 0.0f) - 0.5f, (sx * (float)sw + 1.0f) - 0.5f};
    const float y[3] = {(sy * (float)sh + -1.0f) - 0.5f, (sy * (float)sh + 0.0f) - 0.5f, (sy * (float)sh + 1.0f) - 0.5f};
    const float fx = floorf(x[1]), fy = floorf(y[1]);
    if (floorf(x[0]) == fx - 1.0f && floorf(x[2]) == fx + 1.0f && floorf(y[0]) == fy - 1.0f &&
        floorf(y[2]) == fy + 1.0f && fx >= 1.0f && fy >= 1.0f && fx < (float)(sw - 2) && fy < (float)(sh - 2)) {
        const float* p = sm + ((int)fy * sw + (int)fx);  // at most 2^30 texels
        const float *pu = p - sw, *pd = p + sw, *pd2 = pd + sw;
        const float t00 = __ldg(p), t10 = __ldg(p + 1), t01 = __ldg(pd), t11 = __ldg(pd + 1);
        const float l0 = __ldg(p - 1), l1 = __ldg(pd - 1), r0 = __ldg(p + 2), r1 = __ldg(pd + 2);
        const float u0 = __ldg(pu), u1 = __ldg(pu + 1), d0 = __ldg(pd2), d1 = __ldg(pd2 + 1);
        auto tap = [](float t00, float t10, float t01, float t11, float a, float b) {
            const float bot = t00 * (1.0f - a) + t10 * a, top = t01 * (1.0f - a) + t11 * a;
            return bot * (1.0f - b) + top * b;
        };
        const float a = x[1] - fx, b = y[1] - fy;
        const float al = x[0] - (fx - 1.0f), ar = x[2] - (fx + 1.0f), bu = y[0] - (fy - 1.0f), bd = y[2] - (fy + 1.0f);
        float n = 0.0f;
        n += frag > tap(t00, t10, t01, t11, a, b) ? 1.0f : 0.0f;
        n += frag > tap(t10, r0, t11, r1, ar, b) ? 1.0f : 0.0f;
        n += frag > tap(t01, t11, d0, d1, a, bd) ? 1.0f : 0.0f;
        n += frag > tap(l0, t00, l1, t01, al, b) ? 1.0f : 0.0f;
        n += frag > tap(u0, u1, t00, t10, a, bu) ? 1.0f : 0.0f;
        return quotient(n, 5.0f, 0.2f);
    }
    const int ox[5] = {0, 1, 0, -1, 0};
    const int oy[5] = {0, 0, 1, 0, -1};
    float f = 0.0f;
#pragma unroll
    for (int s = 0; s < 5; ++s)
        if (frag > shadow_bilinear(sm, sw, sh, sx, sy, ox[s], oy[s])) f += 1.0f;
    return quotient(f, 5.0f, 0.2f);
}

__device__ __forceinline__ uint32_t quant16(float x) { return __float2uint_rn(__saturatef(x) * 65535.0f); }

// ------------------------------------------------------------ scene sets
// Kernels are templated on a scene set: OneScene keeps the parameters in
// kernel-parameter space (the single-frame path), ManyScenes reads them from
// device memory and maps a global work index to (scene, local index).
template <class Params>
struct OneScene {
    Params p;
    __device__ __forceinline__ int count() const { return 1; }
    __device__ __forceinline__ const Params& get(int) const { return p; }
    __device__ __forceinline__ int find(long long w, long long& local) const {
        local = w;
        return 0;
    }
};

template <class Params>
struct ManyScenes {
    SceneBatch<Params> b;
    __device__ __forceinline__ int count() const { return b.n; }
    __device__ __forceinline__ const Params& get(int s) const { return b.p[s]; }
    __device__ __forceinline__ int find(long long w, long long& local) const {
        int lo = 0, hi = b.n - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(b.off + mid) <= w)
                lo = mid;
            else
                hi = mid - 1;
        }
        local = w - __ldg(b.off + lo);
        return lo;
    }
};

// Programmatic dependent launch: a kernel launched with launch_overlapped may
// start once every CTA of the kernel before it has called
// grid_launch_dependents (or ended), and waits in grid_wait for that kernel's
// end before it touches anything that other kernels read or write.  (Read-only
// loads may be moved before the wait by the compiler: use ordinary ones behind
// it, or addresses that a barrier behind it makes known.)  One exception: what
// was complete when an ordinary launch started, with only kernels that wait
// between that one and this, may be read before the wait: the triangles of the
// depth passes (before the fill of their keys) and the G-buffer of a frame's
// trace (before the resolve).
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... K, class... A>
inline void launch_overlapped(void (*kernel)(K...), dim3 grid, int threads, int smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, args...);
    note_launches(1);
}

// The viewpoints of a ViewSet (at most kMaxViews): found by a linear scan.
struct FewScenes {
    ViewSet v;
    __device__ __forceinline__ int count() const { return v.n; }
    __device__ __forceinline__ const TraceParams& get(int s) const { return v.p[s]; }
    __device__ __forceinline__ int find(long long w, long long& local) const {
        int s = 0;
        while (s + 1 < v.n && v.off[s + 1] <= w) ++s;
        local = w - v.off[s];
        return s;
    }
};

}  // namespace vct
