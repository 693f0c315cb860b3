// Frame set-up passes that the reference performs with the GL rasteriser:
// the depth-only shadow pass (src/Application.cpp:213-233) and a camera
// G-buffer (world position, normal, albedo) that replaces the depth prepass
// and the per-fragment inputs of phong.frag.
//
// Both use the pixel-centre integer rasteriser of vct_device.cuh.  Depth tests
// are atomicMin on keys: the shadow map keys are the bits of non-negative fp32
// depths (ordered like the floats), the G-buffer keys are (depth bits << 32 |
// triangle id), which also makes the nearest-triangle choice deterministic.
// Compiled with --fmad=false.
#include "lines.cuh"

namespace vct {

namespace {

using namespace lines;

// ------------------------------------------------- depth rasterisation
// One kernel for both passes, over the covered runs of the triangles' lines
// (lines.cuh).
//
// What bounds it is issue (70% of peak, 50% of the ALU pipe) at some 60
// instructions per 32 pixels and 250 per 32 lines.  262,144 triangles into a
// 2048^2 shadow map (71 M pixels, 3 M lines): 0.33 ms; into a 1920x1080
// G-buffer (33 M pixels, 5.5 M lines): 0.24 ms; 1,290 triangles, ten of them
// walls of a 500^2 / 641x359 image: 0.015 / 0.016 ms.  A warp per triangle over
// its whole bounding box, with 64-bit divisions and conversions per pixel, took
// 1.90, 11.1, 0.65 and 1.03 ms: it left one warp with a whole wall, and the
// columns' slivers with boxes of thousands of pixels around a few hundred.
// Launched with programmatic dependence, and the G-buffer's last pass too, the
// small scene's two passes take 41.5 us with their fills, 48 before.
// The CTA walk took 0.35, 0.27, 0.022 and 0.020 ms: at 60 instructions a step
// its warps spend a sixth to a quarter of their time at barriers.  Groups of
// 96 lines 0.34 and 0.24 ms (four views of 650,000 triangles 0.79 ms; 0.74 with
// 64, 0.77 with 32), long lines in pieces by the box's width instead of the
// line's 0.33 and 0.50, one step at a time 0.39 and 0.25, three 0.33 and 0.28.
// Runs of 8 neighbouring triangles to a CTA 0.34, 0.24, 0.017 and 0.021, of 2
// 0.33, 0.25, 0.013 and 0.017.

// Keys of two steps at a time: their loads are in flight together.  The keys
// only fall during the pass, so one that is not below the key it sees needs no
// atomic (a stale read costs a redundant one).
constexpr int kDepthSteps = 2;

template <class Pass>
struct DepthSink {
    const Pass& P;
    __device__ __forceinline__ void operator()(const LinePixel (&f)[kDepthSteps]) const {
        typename Pass::Key key[kDepthSteps], seen[kDepthSteps];
        typename Pass::Key* p[kDepthSteps];
#pragma unroll
        for (int h = 0; h < kDepthSteps; ++h) {
            p[h] = nullptr;
            if (f[h].on && f[h].z >= 0.0f && f[h].z <= 1.0f)  // GL clipping
                p[h] = P.place(f[h].px, f[h].py, f[h].z, f[h].rec->tri, key[h]);
        }
#pragma unroll
        for (int h = 0; h < kDepthSteps; ++h)
            if (p[h]) seen[h] = __ldcg(p[h]);
#pragma unroll
        for (int h = 0; h < kDepthSteps; ++h)
            if (p[h] && key[h] < seen[h]) atomicMin(p[h], key[h]);
    }
};

// `Pass`: setup(t, part, rt, z, more) sets up part `part` of triangle t (false:
// nothing to draw; more: there is another part, of kMaxParts at most), place
// gives a covered pixel's key and where it goes.
template <class Pass>
__global__ void __launch_bounds__(kLineThreads, 4) depth_raster_kernel(const Pass P, long long ntri) {
    __shared__ WarpLines S;
    const long long t = my_triangle<4>();
    bool more = t < ntri;
    const DepthSink<Pass> sink = {P};
    for (int part = 0; part < Pass::kMaxParts; ++part) {
        if (part > 0 && !__syncthreads_or(more)) return;
        int lines = 0;
        bool big = false;
        if (more) {
            RasterTri rt;
            float z[3];
            if (P.setup(t, part, rt, z, more)) {
                lines = store_rec<true>(S.recs[threadIdx.x], rt, z, (int)t);
                big = rt.area >= kBigArea;
            }
        }
        if (part == 0) grid_wait();  // (the triangles are older than the fill of the keys)
        walk_all<kDepthSteps>(S, lines, big, sink);
    }
}

struct ShadowPass : ShadowRasterParams {
    using Key = unsigned int;
    static constexpr int kMaxParts = 1;
    __device__ __forceinline__ bool setup(long long t, int, RasterTri& rt, float d[3], bool& more) const {
        more = false;
        const float* Pp = pos + t * 9;
        float wx[3], wy[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float c[4];
            mat_vec(ls, Pp[3 * k], Pp[3 * k + 1], Pp[3 * k + 2], 1.0f, c);
            float nx = c[0], ny = c[1], nz = c[2];
            if (c[3] != 1.0f) {  // x / 1 = x: no division for a directional light
                nx = __fdiv_rn(nx, c[3]);
                ny = __fdiv_rn(ny, c[3]);
                nz = __fdiv_rn(nz, c[3]);
            }
            wx[k] = (nx + 1.0f) * 0.5f * (float)w;
            wy[k] = (ny + 1.0f) * 0.5f * (float)h;
            d[k] = (nz + 1.0f) * 0.5f;
        }
        return raster_setup(wx, wy, w, h, rt);
    }
    __device__ __forceinline__ unsigned int* place(int px, int py, float z, int, unsigned int& key) const {
        key = __float_as_uint(z);
        return depth_bits + (py * w + px);  // at most 2^30 texels
    }
};

struct GbufferPass : GbufferRasterParams {
    using Key = unsigned long long;
    static constexpr int kMaxParts = 2;
    __device__ __forceinline__ void clip_space(long long t, float cv[3][4]) const {
        const float* Pp = pos + t * 9;
#pragma unroll
        for (int k = 0; k < 3; ++k) mat_vec(vp, Pp[3 * k], Pp[3 * k + 1], Pp[3 * k + 2], 1.0f, cv[k]);
    }
    // Two vertices in front of the near plane leave a quadrilateral: two parts.
    __device__ __forceinline__ bool setup(long long t, int part, RasterTri& rt, float d[3], bool& more) const {
        more = false;
        float cv[3][4];
        clip_space(t, cv);
        bool all_in = true;
#pragma unroll
        for (int k = 0; k < 3; ++k) all_in = all_in && cv[k][2] + cv[k][3] >= 0.0f;
        if (!all_in) {
            // Near-plane clip z >= -w (Sutherland-Hodgman), as the CPU oracle does.
            float poly[4][4];
            int np = 0;
            for (int k = 0; k < 3; ++k) {
                const float* a = cv[k];
                const float* b = cv[(k + 1) % 3];
                float da = a[2] + a[3], db = b[2] + b[3];
                if (da >= 0.0f) {
                    for (int c = 0; c < 4; ++c) poly[np][c] = a[c];
                    ++np;
                }
                if ((da >= 0.0f) != (db >= 0.0f)) {
                    float s = __fdiv_rn(da, da - db);
                    for (int c = 0; c < 4; ++c) poly[np][c] = a[c] + s * (b[c] - a[c]);
                    ++np;
                }
            }
            more = np > part + 3;
            if (np < part + 3) return false;
            for (int c = 0; c < 4; ++c) {
                const float v1 = poly[part + 1][c], v2 = poly[part + 2][c];
                cv[0][c] = poly[0][c];
                cv[1][c] = v1;
                cv[2][c] = v2;
            }
        } else if (part > 0) {
            return false;
        }
        float wx[3], wy[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            if (!(cv[k][3] > 0.0f)) return false;
            float nx = __fdiv_rn(cv[k][0], cv[k][3]), ny = __fdiv_rn(cv[k][1], cv[k][3]);
            float nz = __fdiv_rn(cv[k][2], cv[k][3]);
            wx[k] = (nx + 1.0f) * 0.5f * (float)w;
            wy[k] = (ny + 1.0f) * 0.5f * (float)h;
            d[k] = (nz + 1.0f) * 0.5f;
        }
        return raster_setup(wx, wy, w, h, rt);
    }
    __device__ __forceinline__ unsigned long long* place(int px, int py, float z, int tri,
                                                         unsigned long long& key) const {
        key = ((unsigned long long)__float_as_uint(z) << 32) | (unsigned long long)(unsigned)tri;
        return keys + (py * w + px);
    }
};

__device__ __forceinline__ f3 crossf(f3 a, f3 b) {
    return mk(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}

__global__ void gbuffer_resolve_kernel(const GbufferRasterParams P) {
    grid_wait();
    const unsigned n = (unsigned)P.w * (unsigned)P.h;  // at most 2^28
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const unsigned long long key = P.keys[i];
        if (key == ~0ull) {
            P.gpos[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            P.gnrm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            P.galb[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const int py = (int)(i / (unsigned)P.w), px = (int)(i - (unsigned)py * (unsigned)P.w);
        const long long t = (long long)(key & 0xffffffffull);
        const float* Pp = P.pos + t * 9;
        const float* Pn = P.nrm + t * 9;
        f3 p0 = ld3(Pp), p1 = ld3(Pp + 3), p2 = ld3(Pp + 6);
        float ndx = __fdiv_rn((float)px + 0.5f, (float)P.w) * 2.0f - 1.0f;
        float ndy = __fdiv_rn((float)py + 0.5f, (float)P.h) * 2.0f - 1.0f;
        float fw[4];
        mat_vec(P.ivp, ndx, ndy, 1.0f, 1.0f, fw);
        f3 dir = sub(mk(__fdiv_rn(fw[0], fw[3]), __fdiv_rn(fw[1], fw[3]), __fdiv_rn(fw[2], fw[3])), P.eye);
        f3 e1 = sub(p1, p0), e2 = sub(p2, p0);
        f3 pv = crossf(dir, e2);
        float det = dot(e1, pv);
        float u = __fdiv_rn(1.0f, 3.0f), v = u;
        if (det != 0.0f) {
            float inv = __fdiv_rn(1.0f, det);
            f3 tv = sub(P.eye, p0);
            u = dot(tv, pv) * inv;
            f3 qv = crossf(tv, e1);
            v = dot(dir, qv) * inv;
            u = clampf(u, 0.0f, 1.0f);
            v = clampf(v, 0.0f, 1.0f - u);
        }
        float w0 = 1.0f - u - v;
        f3 wp = add(add(mul(p0, w0), mul(p1, u)), mul(p2, v));
        f3 nn = normalize(add(add(mul(ld3(Pn), w0), mul(ld3(Pn + 3), u)), mul(ld3(Pn + 6), v)));
        P.gpos[i] = make_float4(wp.x, wp.y, wp.z, 1.0f);
        P.gnrm[i] = make_float4(nn.x, nn.y, nn.z, 0.0f);
        P.galb[i] = make_float4(P.albedo[3 * t], P.albedo[3 * t + 1], P.albedo[3 * t + 2], 1.0f);
    }
}

}  // namespace

namespace {
// Shares of about 2,048 pixels if the image is covered eight times over.
template <class Pass>
void launch_depth_raster(const Pass& P, cudaStream_t s) {
    const dim3 grid = line_grid(P.ntri, P.num_sms * 24LL, 8LL * P.w * P.h, 2048, P.num_sms, 2);
    launch_overlapped(depth_raster_kernel<Pass>, grid, kLineThreads, 0, s, P, P.ntri);
}
}  // namespace

void launch_shadow_raster(const ShadowRasterParams& P, cudaStream_t s) {
    launch_fill_u32(P.depth_bits, 0x3f800000u, (long long)P.w * P.h, s);  // 1.0f
    if (P.ntri > 0) launch_depth_raster(ShadowPass{P}, s);
}

void launch_gbuffer_raster(const GbufferRasterParams& P, cudaStream_t s) {
    long long n = (long long)P.w * P.h;
    launch_fill_u32(reinterpret_cast<uint32_t*>(P.keys), 0xffffffffu, 2 * n, s);
    if (P.ntri > 0) launch_depth_raster(GbufferPass{P}, s);
    long long rb = (n + 255) / 256;
    if (rb > 8192) rb = 8192;
    launch_overlapped(gbuffer_resolve_kernel, dim3((unsigned)rb), 256, 0, s, P);
}

}  // namespace vct
