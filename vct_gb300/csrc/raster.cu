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
#include <algorithm>

#include "vct_device.cuh"

namespace vct {

namespace {

// ------------------------------------------------- depth rasterisation
// One kernel for both passes.  A thread sets up one triangle; the triangle is
// then walked in lines: rows, or columns when its bounding box is more than
// twice as tall as wide, so that an upright sliver costs a few lines and not
// its whole height.  A line's covered pixels are contiguous and found from the
// triangle's crossings of it, with the edge functions at the first one.  A CTA
// walks the lines of its 256 triangles together: 256 lines at a time, a thread
// each, their pixel counts scanned; then every warp takes an equal share of
// the pixels, 32 a step, whichever lines and triangles they belong to.
//
// No scratch memory is asked of the caller, so work is not handed from one
// CTA to another: `slices` CTAs (gridDim.y) set up the same 256 triangles and
// share the pixels of the big ones, and `line_slices` of them the pixels of
// the others.
//
// What bounds it is issue (72% of peak; ALU pipe 50%) at some 60 instructions
// per 32 pixels and 300 per 32 lines.  262,144 triangles into a 2048^2 shadow
// map (71 M pixels, 3 M lines): 0.43 ms; into a 1920x1080 G-buffer (33 M
// pixels, 5.5 M lines): 0.33 ms; 1,290 triangles, ten of them walls of a
// 500^2 / 641x359 image: 0.036 / 0.032 ms.  The form before, a warp per
// triangle over its whole bounding box with 64-bit divisions and conversions
// per pixel, took 1.90, 11.1, 0.65 and 1.03 ms: it left one warp with a whole
// wall, and the columns' slivers with boxes of thousands of pixels around a
// few hundred.  256 threads beat 128 (0.42-0.51 and 0.40-0.41 ms).
constexpr int kRasterThreads = 256;
constexpr int kRasterWarps = kRasterThreads / 32;
// A set-up triangle in shared memory.  For its lines, counter-clockwise:
// {X0, Y0, X1, Y1}, {X2, Y2, x0 | y0 << 16, x1 | y1 << 16}, flags.  For its
// candidates, in the caller's vertex order: what a pixel along a line adds to
// each edge function (per sub-pixel unit) and 1 / area; the depths and the
// triangle.  (Five uint4: the odd stride spreads the banks.)
struct TriRec {
    uint4 v0, v1;
    int step[3];
    float inv;
    float z[3];
    int tri;
    uint32_t flags, unused[3];
};
static_assert(sizeof(TriRec) == 80, "a record's stride is five uint4");
// Flags: bits 0-2 the edges that are not top-left.
constexpr uint32_t kRecSwapped = 8u, kRecColumns = 16u;

// Stores the record of a set-up triangle; its lines.  Columns only for boxes
// four times as tall as wide: the pixels of a column are in as many sectors of
// the image.
__device__ __forceinline__ int store_rec(TriRec& r, const RasterTri& t, const float z[3], int tri) {
    const int w = t.px1 - t.px0 + 1, h = t.py1 - t.py0 + 1;
    const bool columns = 2 * w < h;
    r.v0 = make_uint4((uint32_t)t.X[0], (uint32_t)t.Y[0], (uint32_t)t.X[1], (uint32_t)t.Y[1]);
    r.v1 = make_uint4((uint32_t)t.X[2], (uint32_t)t.Y[2], (uint32_t)t.px0 | ((uint32_t)t.py0 << 16),
                      (uint32_t)t.px1 | ((uint32_t)t.py1 << 16));
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int a = (k + 1) % 3, b = (k + 2) % 3;
        const int s = columns ? t.X[b] - t.X[a] : t.Y[a] - t.Y[b];
        if (k == 0)
            r.step[0] = s;
        else
            r.step[t.perm1 ? 3 - k : k] = s;
        r.z[k] = z[k];
    }
    r.inv = __fdiv_rn(1.0f, t.area_float());
    r.tri = tri;
    r.flags = (t.bias[0] ? 1u : 0u) | (t.bias[1] ? 2u : 0u) | (t.bias[2] ? 4u : 0u) |
              (t.perm1 ? kRecSwapped : 0u) | (columns ? kRecColumns : 0u);
    return columns ? w : h;
}

// The covered pixels of line `k` of a triangle, which are contiguous: how
// many, the first one, and the edge functions there in the caller's vertex
// order (modulo 2^32 unless BIG).  The triangle's crossings of the line are
// computed in fp32, within 2^-21 of the coordinates' magnitude (the
// differences' conversion, the division, the product and the sum each round
// at 2^-24 or 2^-22).  Pixel centres further than 2^-20 of it and half a
// sub-pixel unit from a crossing are decided by it; the few nearer ones by the
// exact edge functions.
template <bool BIG>
__device__ __forceinline__ int line_pixels(const TriRec& r, int k, int& first, long long base[3]) {
    const uint4 v0 = r.v0, v1 = r.v1;
    const uint32_t flags = r.flags;
    const int X[3] = {(int)v0.x, (int)v0.z, (int)v1.x}, Y[3] = {(int)v0.y, (int)v0.w, (int)v1.y};
    const bool columns = (flags & kRecColumns) != 0u;
    const int x0 = (int)(v1.z & 0xffffu), y0 = (int)(v1.z >> 16), x1 = (int)(v1.w & 0xffffu), y1 = (int)(v1.w >> 16);
    const int at = ((columns ? x0 : y0) + k) * kSub + kSub / 2;
    int U[3], V[3];  // along the line, and across
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        U[i] = columns ? Y[i] : X[i];
        V[i] = columns ? X[i] : Y[i];
    }
    float lo = 3.0e38f, hi = -3.0e38f, big = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = i, b = (i + 1) % 3;
        const float ua = (float)U[a];
        big = fmaxf(big, fabsf(ua));
        if (min(V[a], V[b]) <= at && at <= max(V[a], V[b])) {
            const int dv = V[b] - V[a];
            // an edge along the line decides all of it
            if (dv == 0 && ((flags >> ((i + 2) % 3)) & 1u)) return 0;
            const float u = dv != 0 ? fmaf((float)(at - V[a]), __fdividef((float)(U[b] - U[a]), (float)dv), ua) : ua;
            const float v = dv != 0 ? u : (float)U[b];
            lo = fminf(lo, fminf(u, v));
            hi = fmaxf(hi, fmaxf(u, v));
        }
    }
    if (!(lo <= hi)) return 0;
    const float eps = fmaf(big, 9.5367431640625e-7f, 0.5f), half = 0.5f * (float)kSub, rs = 1.0f / (float)kSub;
    // the first and last pixel: certainly covered ones (in), possibly covered ones (out);
    // clamped to the image's part as floats, since the crossings may lie far outside
    const float p0 = (float)(columns ? y0 : x0), p1 = (float)(columns ? y1 : x1);
    const int in0 = (int)fminf(fmaxf(ceilf((lo + eps - half) * rs), p0), p1 + 1.0f);
    const int in1 = (int)fmaxf(fminf(floorf((hi - eps - half) * rs), p1), p0 - 1.0f);
    first = (int)fminf(fmaxf(ceilf((lo - eps - half) * rs), p0), p1 + 1.0f);
    int last = (int)fmaxf(fminf(floorf((hi + eps - half) * rs), p1), p0 - 1.0f);
    if (first != in0 || last != in1) {
        // (products of 32-bit factors, exact in 64)
        auto covered = [&](int p) {
            const int u = p * kSub + kSub / 2, sx = columns ? at : u, sy = columns ? u : at;
            bool in = true;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const int ia = (i + 1) % 3, ib = (i + 2) % 3;
                const long long e = (long long)(X[ib] - X[ia]) * (long long)(sy - Y[ia]) -
                                    (long long)(Y[ib] - Y[ia]) * (long long)(sx - X[ia]);
                in = in && e - (long long)((flags >> i) & 1u) >= 0;
            }
            return in;
        };
        while (last >= first && last != in1 && !covered(last)) --last;
        while (first <= last && first != in0 && !covered(first)) ++first;
    }
    if (first > last) return 0;
    const int u = first * kSub + kSub / 2, sx = columns ? at : u, sy = columns ? u : at;
    const bool sw = (flags & kRecSwapped) != 0u;
    long long e[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int ia = (i + 1) % 3, ib = (i + 2) % 3;
        if (BIG)
            e[i] = (long long)(X[ib] - X[ia]) * (long long)(sy - Y[ia]) -
                   (long long)(Y[ib] - Y[ia]) * (long long)(sx - X[ia]);
        else
            e[i] = (uint32_t)(X[ib] - X[ia]) * (uint32_t)(sy - Y[ia]) - (uint32_t)(Y[ib] - Y[ia]) * (uint32_t)(sx - X[ia]);
    }
    base[0] = e[0];
    base[1] = sw ? e[2] : e[1];
    base[2] = sw ? e[1] : e[2];
    return last - first + 1;
}

// Inclusive scans of `v` over the CTA, the totals in `total`; `s` holds a
// word per warp and value.  Callers put a barrier between two uses of one `s`.
template <int N>
__device__ __forceinline__ void cta_scan(int (&v)[N], int (*s)[kRasterWarps], int (&total)[N]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int u = __shfl_up_sync(0xffffffffu, v[n], o);
            if (lane >= o) v[n] += u;
        }
    }
    if (lane == 31)
        for (int n = 0; n < N; ++n) s[n][warp] = v[n];
    __syncthreads();
#pragma unroll
    for (int n = 0; n < N; ++n) {
        total[n] = 0;
#pragma unroll
        for (int w = 0; w < kRasterWarps; ++w) {
            if (w == warp) v[n] += total[n];
            total[n] += s[n][w];
        }
    }
}

struct RasterShared {
    TriRec recs[kRasterThreads];
    int line_off[kRasterThreads];  // first line of each triangle among the CTA's
    // lines with covered pixels, in order: the number of the first pixel among
    // the lines'; the edge functions there (64 bits each for big triangles) and
    // its place; the line's place | its triangle's record << 16
    int pix_off[kRasterThreads + 32];
    uint4 pix_base[2][kRasterThreads];
    uint32_t pix_line[kRasterThreads];
    int scan[3][kRasterWarps];
};

// Walks the CTA's triangles with `lines` lines each (a thread's own), handing
// this slice's share of every 256 lines' covered pixels to P.  BIG: triangles
// of any area; otherwise twice the area is below 2^31 square sub-pixel units,
// and so are the covered pixels' edge functions: 32 bits hold them, whatever
// the products on the way.
template <bool BIG, class Pass>
__device__ __forceinline__ void walk_triangles(const Pass& P, RasterShared& S, int lines, int slice, int slices) {
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int end[1] = {lines}, total[1];
    cta_scan(end, S.scan, total);
    S.line_off[tid] = end[0] - lines;
    __syncthreads();
    for (int l0 = 0; l0 < total[0]; l0 += kRasterThreads) {
        const int l = l0 + tid;
        int first = 0, cnt = 0, rec = 0, k = 0;
        long long base[3] = {0, 0, 0};
        if (l < total[0]) {
            // the last triangle whose lines start at or before l
#pragma unroll
            for (int st = kRasterThreads / 2; st > 0; st >>= 1)
                if (S.line_off[rec + st] <= l) rec += st;
            k = l - S.line_off[rec];
            cnt = line_pixels<BIG>(S.recs[rec], k, first, base);
        }
        int ends[2] = {cnt, cnt > 0 ? 1 : 0}, sums[2];  // covered pixels, lines that have any
        cta_scan(ends, S.scan + 1, sums);
        const int npix = sums[0], nline = sums[1], at = ends[1] - 1;
        if (cnt > 0) {
            S.pix_off[at] = ends[0] - cnt;
            if (BIG) {
                S.pix_base[0][at] = make_uint4((uint32_t)base[0], (uint32_t)(base[0] >> 32), (uint32_t)base[1],
                                               (uint32_t)(base[1] >> 32));
                S.pix_base[1][at] = make_uint4((uint32_t)base[2], (uint32_t)(base[2] >> 32), (uint32_t)first, 0u);
            } else {
                S.pix_base[0][at] = make_uint4((uint32_t)base[0], (uint32_t)base[1], (uint32_t)base[2], (uint32_t)first);
            }
            const uint32_t box = S.recs[rec].v1.z;
            const uint32_t place = ((S.recs[rec].flags & kRecColumns) ? (box & 0xffffu) : (box >> 16)) + (uint32_t)k;
            S.pix_line[at] = place | ((uint32_t)rec << 16);
        }
        if (tid < 32) S.pix_off[nline + tid] = 0x7fffffff;
        __syncthreads();
        const int steps = (npix + 31) / 32, me = slice * kRasterWarps + warp, all = slices * kRasterWarps;
        const int s0 = (int)((long long)steps * me / all), s1 = (int)((long long)steps * (me + 1) / all);
        int j = 0;  // the line of the step's first pixel
        if (s0 < s1) {
#pragma unroll
            for (int st = kRasterThreads / 2; st > 0; st >>= 1)
                if (j + st < nline && S.pix_off[j + st] <= s0 * 32) j += st;
        }
        for (int st = s0; st < s1; st += 2) {
            // two steps at a time: their key loads are in flight together
            typename Pass::Key key[2], seen[2];
            typename Pass::Key* p[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                // A step's 32 pixels lie in at most 32 lines, from line j on:
                // a bit where each of the later ones starts gives every
                // lane its line.
                const int c0 = (st + h) * 32, c = c0 + lane;
                const int off = S.pix_off[j + lane] - c0;
                const unsigned starts = __reduce_or_sync(FULL, off > 0 && off < 32 ? 1u << off : 0u);
                const int i = __popc(starts & (0xffffffffu >> (31 - lane)));
                p[h] = nullptr;
                if (st + h < s1 && c < npix) {
                    const uint32_t line = S.pix_line[j + i];
                    const TriRec& r = S.recs[line >> 16];
                    const int4 d = *reinterpret_cast<const int4*>(r.step);  // and 1 / area
                    const float4 zt = *reinterpret_cast<const float4*>(r.z);
                    const int n = c - S.pix_off[j + i];
                    const uint4 b0 = S.pix_base[0][j + i];
                    float e[3];
                    int u;
                    if (BIG) {
                        const uint4 b1 = S.pix_base[1][j + i];
                        const int m = n * kSub;
                        const long long e0 = (long long)(((unsigned long long)b0.y << 32) | b0.x) + (long long)d.x * m,
                                        e1 = (long long)(((unsigned long long)b0.w << 32) | b0.z) + (long long)d.y * m,
                                        e2 = (long long)(((unsigned long long)b1.y << 32) | b1.x) + (long long)d.z * m;
                        const bool wide = ((e0 | e1 | e2) >= kHalvesLimit);
                        e[0] = edge_to_float(e0, wide);
                        e[1] = edge_to_float(e1, wide);
                        e[2] = edge_to_float(e2, wide);
                        u = (int)b1.z + n;
                    } else {
                        const uint32_t m = (uint32_t)(n * kSub);
                        e[0] = __uint2float_rn(b0.x + (uint32_t)d.x * m);
                        e[1] = __uint2float_rn(b0.y + (uint32_t)d.y * m);
                        e[2] = __uint2float_rn(b0.z + (uint32_t)d.z * m);
                        u = (int)b0.w + n;
                    }
                    const float inv = __int_as_float(d.w);
                    const float l[3] = {e[0] * inv, e[1] * inv, e[2] * inv};
                    const float z = interp(l, zt.x, zt.y, zt.z);
                    if (z >= 0.0f && z <= 1.0f) {  // GL clipping
                        const int v = (int)(line & 0xffffu);
                        const bool columns = (r.flags & kRecColumns) != 0u;
                        p[h] = P.place(columns ? v : u, columns ? u : v, z, __float_as_int(zt.w), key[h]);
                    }
                }
                j += __popc(starts);
                if (S.pix_off[j + 1] <= c0 + 32) ++j;  // that line's last pixel was the step's last
            }
            // The keys only fall during the pass, so one that is not below the
            // key it sees needs no atomic (a stale read costs a redundant one).
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (p[h]) seen[h] = __ldcg(p[h]);
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (p[h] && key[h] < seen[h]) atomicMin(p[h], key[h]);
        }
        __syncthreads();
    }
}

// `Pass`: setup(t, part, rt, z) sets up part `part` of triangle t (false:
// nothing to draw), parts(t) counts them (at most kMaxParts), place gives a
// covered pixel's key and where it goes.
template <class Pass>
__global__ void __launch_bounds__(kRasterThreads, 4) depth_raster_kernel(const Pass P, long long ntri, int line_slices) {
    __shared__ RasterShared S;
    const int tid = threadIdx.x;
    // runs of eight triangles dealt out to the CTAs: neighbours in the array are
    // often alike in size
    const long long t = ((long long)(tid >> 3) * gridDim.x + blockIdx.x) * 8 + (tid & 7);
    const int slice = blockIdx.y, slices = gridDim.y;
    for (int part = 0; part < Pass::kMaxParts; ++part) {
        if (part > 0 && !__syncthreads_or(t < ntri && P.parts(t) > part)) return;
        int lines = 0;
        bool big = false;
        if (t < ntri) {
            RasterTri rt;
            float z[3];
            if (P.setup(t, part, rt, z)) {
                lines = store_rec(S.recs[tid], rt, z, (int)t);
                big = rt.area >= (1LL << 31);
            }
        }
        if (slice < line_slices) walk_triangles<false>(P, S, big ? 0 : lines, slice, line_slices);
        if (__syncthreads_or(big)) walk_triangles<true>(P, S, big ? lines : 0, slice, slices);
    }
}

struct ShadowPass : ShadowRasterParams {
    using Key = unsigned int;
    static constexpr int kMaxParts = 1;
    __device__ __forceinline__ int parts(long long) const { return 1; }
    __device__ __forceinline__ bool setup(long long t, int, RasterTri& rt, float d[3]) const {
        const float* Pp = pos + t * 9;
        float wx[3], wy[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            float c[4];
            mat_vec(ls, Pp[3 * k], Pp[3 * k + 1], Pp[3 * k + 2], 1.0f, c);
            float nx = __fdiv_rn(c[0], c[3]), ny = __fdiv_rn(c[1], c[3]), nz = __fdiv_rn(c[2], c[3]);
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
    __device__ __forceinline__ int parts(long long t) const {
        float cv[3][4];
        clip_space(t, cv);
        int in = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) in += cv[k][2] + cv[k][3] >= 0.0f ? 1 : 0;
        return in == 2 ? 2 : in == 0 ? 0 : 1;
    }
    __device__ __forceinline__ bool setup(long long t, int part, RasterTri& rt, float d[3]) const {
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
    const long long n = (long long)P.w * P.h;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long key = P.keys[i];
        if (key == ~0ull) {
            P.gpos[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            P.gnrm[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            P.galb[i] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        const int px = (int)(i % P.w), py = (int)(i / P.w);
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
// Slices: enough CTAs for six per SM (four are resident), up to 64, so that
// the triangles of small scenes fill the GPU; past 233,472 triangles there
// are enough with one, and setting the triangles up and narrowing their lines
// twice costs more than the better balance gives (G-buffer of 262,144
// triangles 0.39 against 0.33 ms; with 16 CTAs per SM 0.47).  At least four
// for the big triangles, so that a wall is shared by 32 warps.
template <class Pass>
void launch_depth_raster(const Pass& P, cudaStream_t s) {
    const long long ctas = (P.ntri + kRasterThreads - 1) / kRasterThreads;
    const long long want = ((long long)P.num_sms * 6 + ctas - 1) / ctas;
    const int slices = (int)std::max(4LL, std::min(want, 64LL));
    const int line_slices = (int)std::max(1LL, std::min(want, 64LL));
    depth_raster_kernel<Pass><<<dim3((unsigned)ctas, (unsigned)slices), kRasterThreads, 0, s>>>(P, P.ntri, line_slices);
    note_launches(1);
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
    gbuffer_resolve_kernel<<<(unsigned)rb, 256, 0, s>>>(P);
    note_launches(1);
}

}  // namespace vct
