// Triangle voxelisation: shaders/voxelize.geom:25-73 + voxelize.frag:75-280.
//
// One launch for one scene or for the concatenated triangles of a batch of
// scenes (voxelize_raster_kernel): a thread does the geometry-shader part of a
// triangle (dominant axis from the summed vertex normals, per-axis ortho
// projection, snapping to the 1/256 sub-pixel grid), the CTA walks the covered
// runs of its triangles' lines (lines.cuh), and each lane of a step lights one
// fragment (all enabled lights, 5-tap PCF for shadow casters) and adds it into
// the voxel's 32-byte accumulator record with fire-and-forget 64-bit
// reductions.
//
// What bounds it: issue (59% of peak at 3 CTAs, 24 warps, per SM; stalls on
// shared and global loads), some 700 instructions per 32 fragments, most of
// them the lighting's.  262,144 triangles, 5 lights, 6.7 M fragments into
// 256^3: 0.29 ms, 300 MB of records read and 167 MB written.  The form before
// had triangle set-up and a scan as kernels of their own, units of bounding-box
// rows taken by warps from a shared counter, an edge test per candidate pixel
// and a queue of the covered ones: 0.35 ms, and 0.10 against 0.016 ms for 1,290
// triangles in 64^3, where ten walls' units left most warps idle.  Runs of 32
// triangles to a CTA keep neighbouring triangles' records in the L2 together
// (0.29 ms; runs of 64: 0.31, 16: 0.32, 256: 0.35).
//
// Integer sums make the result independent of fragment order: it is
// bit-exact against the CPU oracle.  Compiled with --fmad=false (see
// vct_device.cuh).
#include "lines.cuh"

namespace vct {

namespace {

using namespace lines;

constexpr int kWarps = 8;
constexpr int kRasterBlocksPerSM = 3;  // register budget: up to 3 raster CTAs per SM
constexpr int kMaxBatchScenes = 256;   // per-scene fragment counters in shared memory

// Bit of a triangle's edge flags: its area is past halves_to_float's range.
constexpr int kWide = 8;

__device__ __forceinline__ float shadow_factor(const AccumParams& P, f3 wp) {
    return pcf5(P.shadowmap, P.sw, P.sh, P.ls, wp);
}

// ------------------------------------------------------------- set-up
// voxelize.geom:25-73 for triangle t of P: the dominant axis of the summed
// normals (strict >, ties to z, or the override), the projection through
// that axis' orthographic matrix into the N x N viewport, and the snapped
// raster set-up.  False when the triangle covers no pixel centre's bounding
// box (zero snapped area, or outside the viewport).
__device__ __forceinline__ bool project_triangle(const AccumParams& P, long long t, RasterTri& rt, float z[3],
                                                 int& axis) {
    const float* Pp = P.pos + t * 9;
    const float* Pn = P.nrm + t * 9;
    f3 n0 = ld3(Pn), n1 = ld3(Pn + 3), n2 = ld3(Pn + 6);
    f3 fn = normalize(add(add(n0, n1), n2));
    float ax = fabsf(fn.x), ay = fabsf(fn.y), az = fabsf(fn.z);
    axis = 2;
    if (ax > ay && ax > az)
        axis = 0;
    else if (ay > ax && ay > az)
        axis = 1;
    if (P.axis_override >= 0 && P.axis_override <= 2) axis = P.axis_override;
    const float* M = P.mvp + 16 * axis;
    const int N = P.dim;
    float wx[3], wy[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float c[4];
        mat_vec(M, Pp[3 * k], Pp[3 * k + 1], Pp[3 * k + 2], 1.0f, c);
        float nx = c[0], ny = c[1];
        z[k] = c[2];
        if (c[3] != 1.0f) {  // (x / 1 = x; the projections are orthographic)
            nx = __fdiv_rn(nx, c[3]);
            ny = __fdiv_rn(ny, c[3]);
            z[k] = __fdiv_rn(z[k], c[3]);
        }
        wx[k] = (nx + 1.0f) * 0.5f * (float)N;
        wy[k] = (ny + 1.0f) * 0.5f * (float)N;
    }
    return raster_setup(wx, wy, N, N, rt);
}

// ------------------------------------------------------------- raster
// Voxel of a fragment: voxelize.frag:79-108.  Without warping the axis
// swizzle resolves to integers: the projected coordinates are the pixel
// indices and the depth axis is trunc(N * (1 - u.z)).  With warping the
// fragment's volume coordinate (pixel centre (p + 0.5) / N, depth
// (z + 1) / 2, swizzled, z flipped) is warped and scaled, as the shader does.
__device__ __forceinline__ bool fragment_voxel(const AccumParams& P, int px, int py, int axis, float zf, int& vx,
                                               int& vy, int& vz) {
    const int N = P.dim;
    const float uz = (zf + 1.0f) * 0.5f;
    // voxelize.frag reads warpVoxels and warpTexture only: the perspective
    // warp (voxelizeTesselationWarp) leaves the rasterised grid linear.
    if (P.warp.mode == VCT_WARP_NONE || P.warp.mode == VCT_WARP_PERSPECTIVE) {
        const int iz = __float2int_rz((float)N * (1.0f - uz));
        if (axis == 0) {
            vx = iz;
            vy = py;
            vz = N - 1 - px;
        } else if (axis == 1) {
            vx = px;
            vy = iz;
            vz = N - 1 - py;
        } else {
            vx = px;
            vy = py;
            vz = iz;
        }
    } else {
        const float fN = (float)N, rN = __frcp_rn(fN);  // N is a power of two: the products are the quotients
        const float ux = ((float)px + 0.5f) * rN, uy = ((float)py + 0.5f) * rN;
        f3 u = axis == 0 ? mk(1.0f - uz, uy, ux) : axis == 1 ? mk(ux, 1.0f - uz, uy) : mk(ux, uy, uz);
        u.z = 1.0f - u.z;
        u = apply_warp(P.warp, u);
        vx = __float2int_rz(fN * u.x);
        vy = __float2int_rz(fN * u.y);
        vz = __float2int_rz(fN * u.z);
    }
    return !(vx < 0 || vy < 0 || vz < 0 || vx >= N || vy >= N || vz >= N);
}

// A warp's fragments on their way to the records: the four 64-bit words each
// adds, their halves in 16 bits, and where (null: nothing).  (What a CTA holds
// in shared memory, three CTAs an SM, is taken from the L1 that the shadow map
// and the triangles are read through: 45 KB a CTA leave 92 KB, 41 leave 124: eight scenes' kernel 1.01 and
// 0.95 ms, one 256^3 scene's 0.290 and 0.285; with the triangles in shared memory
// too, 70 KB a CTA, 1.58 and 0.338.)
struct RecordStage {
    uint4 words[32];
    unsigned long long* rec[32];
};

// Adds the staged fragments with fire-and-forget reductions (no result is
// waited for): four lanes take the four words of one record, so an
// instruction's 32 reductions fall into 8 sectors.  A lane adding all of its
// own record's words sends a sector per word (6.7 M fragments: 40 M requests to
// the L2 against 17 M).
__device__ __forceinline__ void flush_stage(const RecordStage& st, int lane) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(st.words);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        unsigned long long* rec = st.rec[8 * i + (lane >> 2)];
        const uint32_t x = w[32 * i + lane];
        if (rec) atomicAdd(rec + (lane & 3), (unsigned long long)(x & 0xffffu) | ((unsigned long long)(x >> 16) << 32));
    }
}

// The largest magnitude of three; NaN if one is, which fmaxf passes over and
// whose product with 0 is not 0.
__device__ __forceinline__ float largest(f3 v) {
    float m;
    asm("max.NaN.abs.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(v.x), "f"(v.y), "f"(v.z));
    return m;
}

// voxelize.frag:186-280 for one fragment: triangle t of the scene, pixel
// (px, py) of its dominant axis' view, weights l and depth z.
__device__ __forceinline__ void shade_fragment(const AccumParams& P, long long t, int axis, int px, int py,
                                               const float l[3], float z, RecordStage& st, int lane) {
    int vx, vy, vz;
    if (!fragment_voxel(P, px, py, axis, z, vx, vy, vz)) return;
    const int N = P.dim;
    const long long v = ((long long)vz * N + vy) * N + vx;
    const float* Pp = P.pos + t * 9;
    const float* Pn = P.nrm + t * 9;
    const f3 p0 = ld3(Pp), p1 = ld3(Pp + 3), p2 = ld3(Pp + 6);
    const f3 n0 = ld3(Pn), n1 = ld3(Pn + 3), n2 = ld3(Pn + 6);
    const f3 wp = mk(interp(l, p0.x, p1.x, p2.x), interp(l, p0.y, p1.y, p2.y), interp(l, p0.z, p1.z, p2.z));
    const f3 ni = mk(interp(l, n0.x, n1.x, n2.x), interp(l, n0.y, n1.y, n2.y), interp(l, n0.z, n1.z, n2.z));
    const f3 Nf = normalize(ni);
    f3 color = ld3(P.albedo + t * 3);
    if (P.lighting) {
        f3 fin = mk(0.0f, 0.0f, 0.0f);
        for (int li = 0; li < P.nlights; ++li) {
            const LightDev& L = P.lights[li];
            if (!L.enabled) continue;
            f3 lit = mk(0.0f, 0.0f, 0.0f);
            if (L.type == 0u) {
                f3 d = sub(L.position, wp);
                // Out of the light's range the attenuation is exactly 0, and
                // for a surface turned well away (by more than rounding) the
                // cosine is: the light then adds +-0, unless its product with
                // the albedo overflows.  Four point lights of range 0.3-0.8 in a
                // volume of side 2 leave one in nine fragments inside one.
                const f3 base = mulv(mul(color, L.intensity), L.color);
                const float d2 = dot(d, d), nd = dot(Nf, d);
                if ((d2 > L.beyond2 || (nd < 0.0f && nd * nd > 1e-6f * d2 && d2 > 1e-30f && L.beyond2 < 3.0e38f)) &&
                    largest(base) < 3.0e38f)
                    continue;
                float ndl = fmaxf(0.0f, dot(Nf, normalize(d)));
                lit = mul(base, ndl);
                float att = 1.0f - smoothstep(L.range075, L.range, length(d));
                lit = mul(lit, att);
            } else if (L.type == 1u) {
                float ndl = fmaxf(0.0f, dot(Nf, L.neg_dir_n));
                lit = mul(mul(mulv(color, L.color), L.intensity), ndl);
            }
            // lit *= 1 - shadow: when lit is exactly zero (the surface faces away, or the
            // light is out of range) the product is +-0 and adding it leaves `fin`
            // unchanged (1 - shadow is finite), so the PCF is not evaluated.
            if (L.shadow_caster && (lit.x != 0.0f || lit.y != 0.0f || lit.z != 0.0f))
                lit = mul(lit, 1.0f - shadow_factor(P, wp));
            fin = add(fin, lit);
        }
        color = mk(clampf(fin.x, 0.0f, 1.0f), clampf(fin.y, 0.0f, 1.0f), clampf(fin.z, 0.0f, 1.0f));
    }
    const f3 n01 = mk((Nf.x + 1.0f) * 0.5f, (Nf.y + 1.0f) * 0.5f, (Nf.z + 1.0f) * 0.5f);
    unsigned long long* rec = reinterpret_cast<unsigned long long*>(P.acc + kAccWords * record_slot(v, P.dim));
    st.words[lane] = make_uint4(1u | (quant16(color.x) << 16), quant16(color.y) | (quant16(color.z) << 16),
                                quant16(n01.x) | (quant16(n01.y) << 16), quant16(n01.z));
    st.rec[lane] = rec;
    // (Setting the occupancy bit only for the fragment that finds the count at
    // 0 waits for the first add's result and is slower.)
    atomicOr(P.occ + (v >> 5), 1u << (v & 31));
}

// Lights 32 fragments, one per lane, and counts them for
// VoxelizeInfo.totalVoxelFragments: covered and inside GL's depth clip.
template <class Scenes>
struct VoxelSink {
    const Scenes& S;
    RecordStage& stage;
    unsigned* frag_count;  // per scene, in shared memory
    int lane;
    __device__ __forceinline__ void operator()(const LinePixel (&f)[1]) {
        const unsigned FULL = 0xffffffffu;
        const bool on = f[0].on && f[0].z >= -1.0f && f[0].z <= 1.0f;
        const unsigned m = __ballot_sync(FULL, on);
        if (!m) return;
        const int scene = on ? (int)f[0].rec->user[1] : 0;
        if (S.count() == 1) {
            if (lane == 0) atomicAdd(frag_count, (unsigned)__popc(m));
        } else if (on) {
            atomicAdd(frag_count + scene, 1u);
        }
        stage.rec[lane] = nullptr;
        if (on)
            shade_fragment(S.get(scene), f[0].rec->tri, (int)f[0].rec->user[0], f[0].px, f[0].py, f[0].l, f[0].z, stage,
                           lane);
        __syncwarp();
        flush_stage(stage, lane);
        __syncwarp();
    }
};

template <class Scenes>
__global__ void __launch_bounds__(kLineThreads, kRasterBlocksPerSM)
    voxelize_raster_kernel(const Scenes S, long long ntri) {
    __shared__ CtaLines L;
    __shared__ RecordStage stages[kWarps];
    __shared__ unsigned frag_count[kMaxBatchScenes];
    const int nscenes = S.count();
    for (int i = threadIdx.x; i < nscenes; i += blockDim.x) frag_count[i] = 0;
    const long long g = my_triangle<32>();
    int lines = 0;
    bool big = false;
    if (g < ntri) {
        long long t;
        const int scene = S.find(g, t);
        RasterTri rt;
        float z[3];
        int axis;
        if (project_triangle(S.get(scene), t, rt, z, axis)) {
            TriRec& r = L.recs[threadIdx.x];
            lines = store_rec<false>(r, rt, z, (int)t);
            r.user[0] = (uint32_t)axis;
            r.user[1] = (uint32_t)scene;
            big = rt.area >= kBigArea;
        }
    }
    VoxelSink<Scenes> sink = {S, stages[threadIdx.x >> 5], frag_count, (int)(threadIdx.x & 31)};
    walk_all<1, 2>(L, lines, big, sink);
    __syncthreads();
    for (int i = threadIdx.x; i < nscenes; i += blockDim.x)
        if (frag_count[i]) atomicAdd(&S.get(i).stats->total_voxel_fragments, frag_count[i]);
}

// By default (units of 512 pixels, 3 CTAs per SM) 9 CTAs per SM, three times
// as many as are resident; smaller units share the lines out further.  Each
// CTA that sets the same triangles up again costs some 7 us of latency (loads,
// projection, scans), each CTA too few leaves SMs idle at the end: with 3, 6, 9,
// 12 and 24 per SM 38,040 triangles in 128^3 take 47, 46, 45, 45 and 46 us,
// 74,752 in 256^3 340, 294, 280, 269 and 275, 262,144 277, 278, 277, 276 and 285;
// past 300,000 triangles the least, two to each 256, is best (519,552: 0.497 ms
// with one, 0.460 with two).
//
// Where the triangles are few, what they cover is not known before they are set
// up: they get the CTAs that are resident, or in a large grid, whose walls have
// that many more pixels, one to 16,384 pixels if they covered its faces 64
// times.  255 triangles that cover a grid many times over take 0.108 ms in 256^3
// and 0.331 in 512^3; with no more than 64 CTAs to a set 0.293 and 1.451 (units
// handed to any CTA by a kernel before it, as once, 0.147 and 0.362), with 9 per
// SM 0.100 and 0.306; 255 that cover little 0.011 and 0.023, 0.010 and 0.018, 0.024
// and 0.027.
template <class Scenes>
void launch_voxelize(const Scenes& S, long long ntri, long long faces, int unit_log2, int num_sms, int blocks_per_sm,
                     cudaStream_t s) {
    if (ntri <= 0) return;
    const int bps = blocks_per_sm < 1 ? 1 : (blocks_per_sm > kRasterBlocksPerSM ? kRasterBlocksPerSM : blocks_per_sm);
    const long long resident = (long long)num_sms * bps, pixels = 64 * faces;
    const dim3 grid = line_grid(ntri, (3 * resident << 9) >> unit_log2, pixels, 2LL << unit_log2, num_sms, 2,
                                std::max(resident, pixels >> 14));
    voxelize_raster_kernel<Scenes><<<grid, kLineThreads, 0, s>>>(S, ntri);
    note_launches(1);
}

// ================================================ warp-map occupancy pass
// voxelize.frag:187-192: the occupancy voxelisation that the warp map is
// built from (Application.cpp:235-285), the same rasterisation rule as above
// at a 32^2 viewport, unwarped and unshaded.  Nearly every triangle of a
// scene covers a handful of pixels at that size, so that
// sharing out lines and pixels would cost far more than the pixels: one thread takes one triangle,
// sets it up and walks a bounding box of up to kOccLanePixels pixels itself;
// the warp walks the larger ones together, 32 pixels at a time.  The result
// is an OR of bits, so the order of the walks does not matter.
constexpr int kOccThreads = 256;
constexpr int kOccLanePixels = 32;

// Coverage of pixel (px, py) by a set-up triangle (snapped vertices X, Y; edge
// k runs from vertex a = k+1 to b = k+2 with deltas dX, dY; bit k of `bias`
// set for an edge that is not top-left, kWide for a triangle past
// halves_to_float's range) and the fragment's barycentrics and
// depth.  The edge function at the pixel centre is dX (sy - Ya) - dY (sx - Xa),
// every factor within 32 bits (|snapped coordinates| <= 2^28), each product
// exact in 64.  False outside the triangle or outside GL's depth clip.
__device__ __forceinline__ bool pixel_fragment(const int X[3], const int Y[3], const int dX[3], const int dY[3],
                                               int bias, int perm1, float inv, const float z[3], int px, int py,
                                               float l[3], float& zf) {
    const int sx = px * kSub + kSub / 2, sy = py * kSub + kSub / 2;
    long long e[3];
    bool cov = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int a = (k + 1) % 3;
        e[k] = (long long)dX[k] * (long long)(sy - Y[a]) - (long long)dY[k] * (long long)(sx - X[a]);
        cov = cov && (e[k] - ((bias >> k) & 1) >= 0);
    }
    if (!cov) return false;
    const bool wide = (bias & kWide) != 0;
    const float w0 = edge_to_float(e[0], wide) * inv, w1 = edge_to_float(e[1], wide) * inv,
                w2 = edge_to_float(e[2], wide) * inv;
    l[0] = w0;
    l[1] = perm1 ? w2 : w1;
    l[2] = perm1 ? w1 : w2;
    zf = interp(l, z[0], z[1], z[2]);
    return zf >= -1.0f && zf <= 1.0f;  // GL clipping
}

__device__ __forceinline__ void occupancy_fragment(const AccumParams& P, int axis, int px, int py, float zf) {
    int vx, vy, vz;
    if (!fragment_voxel(P, px, py, axis, zf, vx, vy, vz)) return;
    const long long v = ((long long)vz * P.dim + vy) * P.dim + vx;
    atomicOr(P.occ + (v >> 5), 1u << (v & 31));
}

template <class Scenes>
__global__ void __launch_bounds__(kOccThreads) occupancy_kernel(const Scenes S, long long ntri) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const long long g = (long long)blockIdx.x * kOccThreads + threadIdx.x;
    RasterTri rt;
    float z[3] = {0.f, 0.f, 0.f};
    int axis = 0, scene = 0;
    bool ok = false;
    if (g < ntri) {
        long long t;
        scene = S.find(g, t);
        const AccumParams& P = S.get(scene);
        ok = P.occ != nullptr && project_triangle(P, t, rt, z, axis);  // scenes without a map: no occupancy
    }
    int X[3] = {0, 0, 0}, Y[3] = {0, 0, 0}, dX[3], dY[3];
    int bias = 0, perm1 = 0, px0 = 0, py0 = 0, bw = 0, bh = 0;
    float inv = 0.f;
    if (ok) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            X[k] = rt.X[k];
            Y[k] = rt.Y[k];
        }
        bias = (rt.bias[0] ? 1 : 0) | (rt.bias[1] ? 2 : 0) | (rt.bias[2] ? 4 : 0) | (rt.wide() ? kWide : 0);
        perm1 = rt.perm1;
        inv = __fdiv_rn(1.0f, rt.area_float());
        px0 = rt.px0;
        py0 = rt.py0;
        bw = rt.px1 - rt.px0 + 1;
        bh = rt.py1 - rt.py0 + 1;
    }
    const int npix = bw * bh;
    if (npix <= kOccLanePixels) {
        const AccumParams& P = S.get(scene);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            dX[k] = X[(k + 2) % 3] - X[(k + 1) % 3];
            dY[k] = Y[(k + 2) % 3] - Y[(k + 1) % 3];
        }
        for (int py = py0; py < py0 + bh; ++py)
            for (int px = px0; px < px0 + bw; ++px) {
                float l[3], zf;
                if (pixel_fragment(X, Y, dX, dY, bias, perm1, inv, z, px, py, l, zf))
                    occupancy_fragment(P, axis, px, py, zf);
            }
    }
    unsigned big = __ballot_sync(FULL, npix > kOccLanePixels);
    while (big) {
        const int src = __ffs(big) - 1;
        big &= big - 1;
        int sX[3], sY[3], sdX[3], sdY[3];
        float sz[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            sX[k] = __shfl_sync(FULL, X[k], src);
            sY[k] = __shfl_sync(FULL, Y[k], src);
            sz[k] = __shfl_sync(FULL, z[k], src);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            sdX[k] = sX[(k + 2) % 3] - sX[(k + 1) % 3];
            sdY[k] = sY[(k + 2) % 3] - sY[(k + 1) % 3];
        }
        const int sbias = __shfl_sync(FULL, bias, src), sperm1 = __shfl_sync(FULL, perm1, src);
        const float sinv = __shfl_sync(FULL, inv, src);
        const int saxis = __shfl_sync(FULL, axis, src), sscene = __shfl_sync(FULL, scene, src);
        const int spx0 = __shfl_sync(FULL, px0, src), spy0 = __shfl_sync(FULL, py0, src);
        const int sbw = __shfl_sync(FULL, bw, src), sn = __shfl_sync(FULL, npix, src);
        const AccumParams& SP = S.get(sscene);
        for (int idx = lane; idx < sn; idx += 32) {
            const int row = idx / sbw;
            const int px = spx0 + (idx - row * sbw), py = spy0 + row;
            float l[3], zf;
            if (pixel_fragment(sX, sY, sdX, sdY, sbias, sperm1, sinv, sz, px, py, l, zf))
                occupancy_fragment(SP, saxis, px, py, zf);
        }
    }
}

// ====================================================== tessellation voxeliser
// testTesselation.tesc/.tese (Application.cpp:585-662) in four launches:
// per-triangle tessellation levels and unit counts (tess_setup_kernel), the
// scan of the block totals, and two persistent kernels of which one ends at
// once (tess_walks): single points, or the walk.
//
// Single points (tess_points_kernel): one to a lane, neighbours of a ring edge
// that fall into one voxel added together.  For triangles of ordinary shape,
// whose points are about a voxel apart in every direction: 24,576 box triangles
// (14.7 M points) in 256^3 take 0.37 ms, bound by the reductions.
//
// The walk (tess_walk_kernel).  The points of slivers fall into few voxels (on
// the 262,144-triangle scene, 14 points to each voxel that a triangle reaches),
// but not in the order of a patch's rings.  A lane therefore walks a sequence of
// points that is likely to stay in one voxel (TessItem) and sums it in registers
// while it does; a finished run goes to a queue in shared memory, and 32 queued
// runs are added to the records together.  Integer sums: any grouping gives the
// same record.  What bounds it is issue (82% of peak), some 300 instructions per
// 32 points: half of them the exact position, a tenth each the normal, the runs'
// queue and their additions, the rest each item's set-up.  53,248 column
// slivers and 24,576 box triangles (180 M points, 38 M runs) in 256^3: 1.85 ms,
// 4.46 as single points; lanes that walk whole ring edges, which finish a run
// every 1.6 points, 2.65.
//
// The walk's constants, by three scenes of column slivers and boxes (22,000 in
// 64^3, 30,000 in 128^3, 78,000 in 256^3; us): units taken at a time 2, 4, 8, 16, 32: 857, 788, 760,
// 764, 782; 934, 860, 832, 815, 870; 2,225, 2,006, 1,893, 1,852, 1,867 (16
// cost 16,000 slivers up to a tenth more).  Points of an edge to an item 4, 8, 16:
// 815, 760, 789; 888, 832, 858; 2,052, 1,893, 1,962.  Places in turn 1, 512, 2,048,
// 8,192, 32,768: 760, 763, 767, 760, 762; 828, 853, 852, 832, 828; 1,869, 1,950,
// 1,935, 1,893, 1,875, and 78,000 triangles in 16^3, whose units all add to
// the same few records, 311, 295, 289, 285, 286.  The inner level from which a sliver is
// walked across, 4 to 16: no difference.
//
// Tessellation levels after GL's equal_spacing rounding, packed 7 bits each:
// inner n | outer[0] << 7 | outer[1] << 14 | outer[2] << 21 (1..64 each) |
// 1 + the type of the edges that a sliver is walked along (0: none) << 28.
constexpr int kTessUnit = 32;  // items per work unit
constexpr int kTessBlocksPerSM = 3;
constexpr int kTessSliver = 8; // inner level from which slivers are walked across
constexpr float kTessThin = 12.0f;  // inner level, in lengths of the shortest edge, of the slivers that decide for the walk
constexpr int kTessRunLog2 = 3;     // log2 of the most points of an edge that one item holds
constexpr int kTessGrab = 8;  // units a warp takes at a time, when there are that many
constexpr int kTessSpread = 8192;  // places in the unit order that are worked on at a time
constexpr int kMaxTess = VCT_MAX_TESS_LEVEL;

// Work units, 32 items or 32 points of one triangle each.  A triangle's counts
// are in one word: its items' in the high half, its points' in the low one (at
// most 100, of 256 triangles 25,600).
__device__ __forceinline__ uint32_t item_units(uint32_t x) { return x >> 16; }
__device__ __forceinline__ uint32_t point_units(uint32_t x) { return x & 0xffffu; }

// Block-local exclusive scan of the per-triangle unit counts of one setup
// block into tri_scan, and the block's totals {items, points, points of
// slivers} into block_off[blockIdx.x].
__device__ __forceinline__ void block_scan_units(const VoxWork& W, long long g, uint32_t units, bool sliver) {
    __shared__ uint32_t warp_tot[kSetupThreads / 32], warp_slivers[kSetupThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t incl = units;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t slivers = __reduce_add_sync(0xffffffffu, sliver ? point_units(units) : 0u);
    if (lane == 31) {
        warp_tot[wid] = incl;
        warp_slivers[wid] = slivers;
    }
    __syncthreads();
    uint32_t before = 0, total = 0, total_slivers = 0;
#pragma unroll
    for (int w = 0; w < kSetupThreads / 32; ++w) {
        before += (w < wid) ? warp_tot[w] : 0u;
        total += warp_tot[w];
        total_slivers += warp_slivers[w];
    }
    if (g < W.ntri) W.tri_scan[g] = before + incl - units;
    if (threadIdx.x == 0) W.block_off[blockIdx.x] = make_uint4(item_units(total), point_units(total), total_slivers, 0u);
}

__global__ void __launch_bounds__(1024) voxelize_scan_kernel(uint4* block_off, int nblocks) {
    __shared__ uint4 warp_tot[32];
    __shared__ uint4 carry;
    auto add = [](uint4 a, uint4 b) { return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, 0u); };
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x == 0) carry = none;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int base = 0; base < nblocks; base += 1024) {
        const int i = base + threadIdx.x;
        const uint4 v = i < nblocks ? block_off[i] : none;
        uint4 incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint4 u = make_uint4(__shfl_up_sync(0xffffffffu, incl.x, o), __shfl_up_sync(0xffffffffu, incl.y, o),
                                       __shfl_up_sync(0xffffffffu, incl.z, o), 0u);
            if (lane >= o) incl = add(incl, u);
        }
        if (lane == 31) warp_tot[wid] = incl;
        __syncthreads();
        uint4 before = carry, total = none;
        for (int w = 0; w < 32; ++w) {
            if (w < wid) before = add(before, warp_tot[w]);
            total = add(total, warp_tot[w]);
        }
        if (i < nblocks)
            block_off[i] = make_uint4(before.x + incl.x - v.x, before.y + incl.y - v.y, before.z + incl.z - v.z, 0u);
        __syncthreads();
        if (threadIdx.x == 0) carry = add(carry, total);
        __syncthreads();
    }
    if (threadIdx.x == 0) block_off[nblocks] = carry;
}

// The triangle that a unit belongs to: its number, its first unit and how many
// it has, of the units of items or of points.
template <bool ITEMS>
struct UnitOwner {
    long long g;
    uint32_t start, units;
    static __device__ __forceinline__ uint32_t part(uint32_t x) { return ITEMS ? item_units(x) : point_units(x); }
    static __device__ __forceinline__ uint32_t block(const VoxWork& W, long long b) {
        return reinterpret_cast<const uint32_t*>(W.block_off + b)[ITEMS ? 0 : 1];
    }
    __device__ __forceinline__ void at(const VoxWork& W, long long t) {
        g = t;
        start = block(W, g / kSetupThreads) + part(W.tri_scan[g]);
        units = part(W.tri_units[g]);
    }
    __device__ __forceinline__ bool holds(uint32_t u) const { return u - start < units; }
    // By a search over the block offsets, then the block-local scan, 8 entries
    // per lane: the number of entries <= u is one past the last triangle starting
    // at or before u.
    __device__ __forceinline__ void find(const VoxWork& W, int nblocks, uint32_t u, int lane) {
        int lo = 0, hi = nblocks - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (block(W, mid) <= u)
                lo = mid;
            else
                hi = mid - 1;
        }
        const long long gbase = (long long)lo * kSetupThreads;
        const int in_block = (int)min((long long)kSetupThreads, W.ntri - gbase);
        const uint32_t rel = u - block(W, lo);
        int below = 0;
#pragma unroll
        for (int j = 0; j < kSetupThreads / 32; ++j) {
            const int k = lane * (kSetupThreads / 32) + j;
            below += (k < in_block && part(__ldg(W.tri_scan + gbase + k)) <= rel) ? 1 : 0;
        }
        below = __reduce_add_sync(0xffffffffu, below);
        at(W, gbase + max(below - 1, 0));
    }
    // The owner of the unit after one of this triangle's: often this one or the next.
    __device__ __forceinline__ void follow(const VoxWork& W, int nblocks, uint32_t u, int lane) {
        if (holds(u)) return;
        at(W, min(g + 1, W.ntri - 1));
        if (!holds(u)) find(W, nblocks, u, lane);
    }
};

// Float-to-int truncation of ivec3(): NaN -> 0, saturating (cvt.rzi.s32.f32).
__device__ __forceinline__ int trunc_sat(float x) { return __float2int_rz(x); }

// equal_spacing: clamp to [1, max], round up (OpenGL 4.6, 11.2.2).
__device__ __forceinline__ int tess_round(float level, float max_level) {
    return (int)ceilf(fminf(fmaxf(level, 1.0f), max_level));
}

// Points of the triangle primitive generator in point mode for inner level
// n and outer levels m0..m2: the outer ring (3 corners and m - 1 points per
// edge) plus the concentric inner rings k = 1.. of n - 2k segments each
// (3 (n - 2k) points, or the centre when n - 2k = 0).
__device__ __forceinline__ uint32_t tess_point_count(int n, int m0, int m1, int m2) {
    uint32_t c = (uint32_t)(m0 + m1 + m2);
    if (n >= 2) {
        const int K = (n & 1) ? (n - 1) / 2 : n / 2 - 1;
        c += 3u * (uint32_t)(K * n - K * (K + 1)) + ((n & 1) ? 0u : 1u);
    }
    return c;
}

// testTesselation.tesc:33-78: levels of one triangle; false if discarded
// (all three vertices truncate to one voxel: levels 0).
__device__ __forceinline__ bool tess_levels(const AccumParams& P, const float* Pp, uint32_t& packed, uint32_t& npts,
                                            bool& sliver) {
    const f3 a = ld3(Pp), b = ld3(Pp + 3), c = ld3(Pp + 6);
    const float fN = (float)P.dim;
    const f3 vtx[3] = {a, b, c};
    int vi[3][3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {  // ivec3(voxelDim * getVoxelPosition(p)), the shader's own linear mapping
        vi[k][0] = trunc_sat(fN * __fdiv_rn((vtx[k].x - P.vcenter.x) - P.vmin.x, P.ext.x));
        vi[k][1] = trunc_sat(fN * __fdiv_rn((vtx[k].y - P.vcenter.y) - P.vmin.y, P.ext.y));
        vi[k][2] = trunc_sat(fN * __fdiv_rn((vtx[k].z - P.vcenter.z) - P.vmin.z, P.ext.z));
    }
    if (vi[0][0] == vi[1][0] && vi[0][1] == vi[1][1] && vi[0][2] == vi[1][2] && vi[0][0] == vi[2][0] &&
        vi[0][1] == vi[2][1] && vi[0][2] == vi[2][2])
        return false;
    const f3 A = sub(c, b), B = sub(c, a), C = sub(b, a);
    const float lx = length(A), ly = length(B), lz = length(C);
    const float sp = ((lx + ly) + lz) * 0.5f;  // semiperimeter
    const float area = __fsqrt_rn(((sp * (sp - lx)) * (sp - ly)) * (sp - lz));  // Heron
    const float ax = __fdiv_rn(2.0f * area, lx), ay = __fdiv_rn(2.0f * area, ly), az = __fdiv_rn(2.0f * area, lz);
    const float max_alt = fmaxf(ax, fmaxf(ay, az));
    const f3 vs = mk(__fdiv_rn(P.ext.x, fN), __fdiv_rn(P.ext.y, fN), __fdiv_rn(P.ext.z, fN));
    const float dx = fabsf(length(mulv(normalize(A), vs))), dy = fabsf(length(mulv(normalize(B), vs))),
                dz = fabsf(length(mulv(normalize(C), vs)));
    const float ox = fmaxf(1.0f, __fdiv_rn(lx, dx)), oy = fmaxf(1.0f, __fdiv_rn(ly, dy)),
                oz = fmaxf(1.0f, __fdiv_rn(lz, dz));
    const float inner = fmaxf(1.0f, __fdiv_rn(max_alt, vs.x));
    // gl_TessLevelOuter[0] = outer.z, [1] = outer.x, [2] = outer.y
    const int m0 = tess_round(oz, P.max_tess_level), m1 = tess_round(ox, P.max_tess_level),
              m2 = tess_round(oy, P.max_tess_level);
    int n = tess_round(inner, P.max_tess_level);
    if (n == 1 && (m0 > 1 || m1 > 1 || m2 > 1)) n = 2;  // inner 1 + epsilon
    // A sliver (one edge under a quarter of the other two, which the levels cut
    // into steps of a voxel or more) is walked across, parallel to that edge:
    // type 0 from vertex 0 to 1, type 1 from 1 to 2, type 2 from 2 to 0.
    uint32_t across = 0;
    if (n >= kTessSliver) {
        if (4.0f * lz < fminf(lx, ly)) across = 1;
        if (4.0f * lx < fminf(ly, lz)) across = 2;
        if (4.0f * ly < fminf(lx, lz)) across = 3;
    }
    packed = (uint32_t)n | ((uint32_t)m0 << 7) | ((uint32_t)m1 << 14) | ((uint32_t)m2 << 21) | (across << 28);
    sliver = (float)n >= kTessThin * fminf(ox, fminf(oy, oz));  // (lengths in voxels, 1 at least)
    npts = tess_point_count(n, m0, m1, m2);
    return true;
}

// The work items of a patch.  Point (c, k, j) is j / q of the way along the
// edge of ring k from corner c to corner c + 1 (type c).  The outer edges
// (k = 0) are u = 0 (from vertex 1 to 2, outer[0] segments), v = 0 (2 to 0,
// outer[1]), w = 0 (0 to 1, outer[2]); the inner rings (inner level n >= 2)
// have q = n - 2k segments an edge, and their corners lie where the
// perpendiculars through the inner subdivision points nearest each corner
// meet: (h, t, t) and rotations, t = 2k / (3n), h = 1 - 2t.  An edge's last
// corner belongs to the next one.  An even inner level has a centre.
//
// An item is a sequence of points (c, k0 + dk i, j0 + dj i).  Edges are items
// of up to 2^run_log2 points.  The edges of ring k advance by 1 / n a point,
// whatever k, so in a sliver, where every such step of the two long types
// crosses a voxel or more, they are not walked along but across: parallel to
// the short type, that is (k + 3, j - 2) on the type after it and (k + 3,
// j - 4) on the one after that.  With w = 2k + 3j (4k + 3j) those diagonals
// are w = 2 .. 3n - 7 (4 .. 3n - 5), of up to n / 6 points; they are numbered so
// that neighbours are about as long (one from the side where the length rises
// by 1/6 of a point, two from the side where it falls by 1/12, or the other way
// round).
struct TessItem {
    int c, k, j, dk, dj, cnt;
};

// Runs 0 .. r of the inner edges of one type: run s has K - s h rings, as far as
// positive.
__device__ __forceinline__ int tess_rings_before(int K, int h, int r) {
    r = min(r + 1, (K + h - 1) / h);
    return r * K - h * (r * (r - 1) / 2);
}
__device__ __forceinline__ int tess_runs(int m, int rl) { return (m + (1 << rl) - 1) >> rl; }

__device__ __forceinline__ uint32_t tess_item_count(uint32_t packed, int rl) {
    const int n = (int)(packed & 127u);
    int c = tess_runs((int)((packed >> 7) & 127u), rl) + tess_runs((int)((packed >> 14) & 127u), rl) +
            tess_runs((int)((packed >> 21) & 127u), rl);
    if (n < 2) return (uint32_t)c;
    const int rings = tess_rings_before((n - 1) / 2, 1 << (rl - 1), n >> rl);
    return (uint32_t)(c + ((packed >> 28) ? rings + 2 * (3 * n - 8) : 3 * rings) + ((n & 1) ? 0 : 1));
}

__device__ __forceinline__ TessItem tess_item(uint32_t packed, int i, int rl) {
    const int n = (int)(packed & 127u), across = (int)(packed >> 28);
    TessItem t = {0, 0, 0, 0, 1, 1};
    // most of a sliver's items are diagonals: first, with nothing to search
    const int diagonals = across ? 3 * n - 8 : 0;
    if (i < 2 * diagonals) {
        const bool second = i >= diagonals;
        if (second) i -= diagonals;
        const int g = i / 3, r = i - 3 * g, f = second ? 4 : 2;
        const int w = second ? (r == 0 ? 3 * n - 5 - g : 3 + 2 * g + r) : (r == 0 ? 2 + g : 3 * n - 6 - 2 * g - r);
        const int last = (3 * n - w - 1) >> (second ? 1 : 2);  // j < q
        const int rest = (second ? w : 2 * w) % 3;             // w - f k a multiple of 3
        t.c = across - 1 + (second ? 2 : 1);
        if (t.c >= 3) t.c -= 3;
        t.k = rest ? rest : 3;
        t.j = (w - f * t.k) / 3;
        t.dk = 3;
        t.dj = -f;
        const int kmax = min(w >> (second ? 2 : 1), last);
        t.cnt = kmax >= t.k ? (kmax - t.k) / 3 + 1 : 0;
        return t;
    }
    i -= 2 * diagonals;
    // The inner edges, first runs first: run r has (n - 1) / 2 - r h rings (as far
    // as positive), h = 2^(rl - 1), so the ones before it have a quadratic in r.
    const int types = across ? 1 : 3, K = n > 1 ? (n - 1) / 2 : 0, h = 1 << (rl - 1), all = tess_rings_before(K, h, n >> rl);
    if (i < types * all) {
        const int ring = across ? i : i / 3;
        const float b = (float)K + 0.5f * (float)h;
        int r = (int)((b - sqrtf(fmaxf(b * b - 2.0f * (float)h * (float)ring, 0.0f))) / (float)h);
        while (r > 0 && tess_rings_before(K, h, r - 1) > ring) --r;
        while (tess_rings_before(K, h, r) <= ring) ++r;  // the runs up to r
        t.k = 1 + ring - tess_rings_before(K, h, r - 1);
        t.c = across ? across - 1 : i - 3 * ring;
        t.j = r << rl;
        t.cnt = min(n - 2 * t.k - t.j, 1 << rl);
        return t;
    }
    i -= types * all;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
        const int m = (int)((packed >> (7 + 7 * e)) & 127u), runs = tess_runs(m, rl);
        if (i >= 0 && i < runs) {
            t.c = e == 2 ? 0 : e + 1;
            t.j = i << rl;
            t.cnt = min(m - t.j, 1 << rl);
            return t;
        }
        i -= runs;
    }
    t.k = n / 2;  // the centre: q = 0
    return t;
}

// Point `i` of a patch in the order of tess_point_count: the corners, the
// outer edges' inner points, then ring by ring.
__device__ __forceinline__ f3 tess_coord(uint32_t packed, int i) {
    const int n = (int)(packed & 127u), m0 = (int)((packed >> 7) & 127u), m1 = (int)((packed >> 14) & 127u),
              m2 = (int)((packed >> 21) & 127u);
    if (i < 3) return i == 0 ? mk(1.0f, 0.0f, 0.0f) : i == 1 ? mk(0.0f, 1.0f, 0.0f) : mk(0.0f, 0.0f, 1.0f);
    i -= 3;
    if (i < m0 - 1) {
        const float s = __fdiv_rn((float)(i + 1), (float)m0);
        return mk(0.0f, 1.0f - s, s);
    }
    i -= m0 - 1;
    if (i < m1 - 1) {
        const float s = __fdiv_rn((float)(i + 1), (float)m1);
        return mk(s, 0.0f, 1.0f - s);
    }
    i -= m1 - 1;
    if (i < m2 - 1) {
        const float s = __fdiv_rn((float)(i + 1), (float)m2);
        return mk(1.0f - s, s, 0.0f);
    }
    i -= m2 - 1;
    int k = 1, q = n - 2;
    while (q > 0 && i >= 3 * q) {
        i -= 3 * q;
        ++k;
        q -= 2;
    }
    if (q <= 0) {  // the centre of an even inner level
        const float third = __fdiv_rn(1.0f, 3.0f);
        return mk(third, third, third);
    }
    const float t = __fdiv_rn((float)(2 * k), (float)(3 * n));
    const float h = 1.0f - 2.0f * t;
    const int e = i / q, j = i - e * q;
    const float s = __fdiv_rn((float)j, (float)q);
    // corners c_e and c_{e+1} of the ring: c0 = (h,t,t), c1 = (t,h,t), c2 = (t,t,h)
    const int e1 = e == 2 ? 0 : e + 1;
    const float a0 = e == 0 ? h : t, a1 = e == 1 ? h : t, a2 = e == 2 ? h : t;
    const float b0 = e1 == 0 ? h : t, b1 = e1 == 1 ? h : t, b2 = e1 == 2 ? h : t;
    return mk(a0 + s * (b0 - a0), a1 + s * (b1 - a1), a2 + s * (b2 - a2));
}

// Whether the items are walked: where thin slivers have most of the points, and
// at least some 1.3 M of them (totals: {items, points, points of slivers}, in
// units of 32).  Otherwise every point is taken singly.  A walk costs some 13 us
// before it gains, and on ordinary triangles it always loses.  Points against
// walk, with set-up and scan (us; slivers' points of all): columns of slivers and
// a few boxes in 16^3 (1.3 M of 1.3 M) 191 and 65, in 64^3 (1.4 of 1.6) 100 and
// 60, in 256^3 (1.7 of 3.6) 124 and 132; columns between 24,576 box
// triangles in 256^3 (26 of 40) 976 and 585; the boxes alone in 64^3 (0.1 of
// 1.2) 53 and 131, in 256^3 (1 of 15) 374 and 398; scattered slivers, which
// share no voxels, in 128^3 (1.2 of 1.2) 41 and 57, (12 of 12) 248 and 194, and
// where the rule loses, in 64^3 (3 of 3) 80 and 114.
__device__ __forceinline__ bool tess_walks(const uint4 total) {
    return total.z >= 40000u && (float)total.z >= 0.6f * (float)total.y;
}

// The walking warps' shared work counter: the 8 bytes after block_off[nblocks].
__device__ __forceinline__ unsigned long long* grab_counter(const VoxWork& W, int nblocks) {
    return reinterpret_cast<unsigned long long*>(W.block_off + nblocks + 1);
}

// Record of a triangle: {packed levels, items << 16 | points, scene, index within its scene}.
template <class Scenes>
__global__ void __launch_bounds__(kSetupThreads) tess_setup_kernel(const Scenes S, const VoxWork W) {
    const long long g = (long long)blockIdx.x * kSetupThreads + threadIdx.x;
    uint32_t units = 0;
    bool sliver = false;
    if (g < W.ntri) {
        long long t;
        const int scene = S.find(g, t);
        const AccumParams& P = S.get(scene);
        uint32_t packed = 0, npts = 0;
        if (!tess_levels(P, P.pos + t * 9, packed, npts, sliver)) npts = 0;
        const uint32_t items = npts ? tess_item_count(packed, kTessRunLog2) : 0u;
        W.tri_rec[g] = make_uint4(packed, items << 16 | npts, (uint32_t)scene, (uint32_t)t);
        units = ((items + kTessUnit - 1) / kTessUnit) << 16 | ((npts + kTessUnit - 1) / kTessUnit);
        W.tri_units[g] = units;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *grab_counter(W, gridDim.x) = 0ull;
    block_scan_units(W, g, units, sliver);
}

// A warp's queued items or points.
struct TessQueue {
    int tri[2 * kTessUnit];        // triangle index within its scene
    uint32_t item[2 * kTessUnit];  // item or point of the triangle | scene << 16
    uint32_t lev[2 * kTessUnit];   // packed levels
};
// Queues unit `unit` of a triangle's `n` items or points; `full` works on 32
// of them.  qn: the number queued (warp-uniform).
template <class F>
__device__ __forceinline__ void queue_unit(TessQueue& q, int& qn, const uint4 rec, uint32_t n, uint32_t unit, int lane,
                                           F full) {
    const int base = (int)unit * kTessUnit;
    const int cnt = min(kTessUnit, (int)n - base);
    if (lane < cnt) {
        q.tri[qn + lane] = (int)rec.w;
        q.item[qn + lane] = (uint32_t)(base + lane) | (rec.z << 16);
        q.lev[qn + lane] = rec.x;
    }
    __syncwarp();
    qn += cnt;
    if (qn >= kTessUnit) {
        full(kTessUnit);
        __syncwarp();
        if (lane < qn - kTessUnit) {
            q.tri[lane] = q.tri[kTessUnit + lane];
            q.item[lane] = q.item[kTessUnit + lane];
            q.lev[lane] = q.lev[kTessUnit + lane];
        }
        __syncwarp();
        qn -= kTessUnit;
    }
}

// A walking warp's queue, and its finished runs of points on their way to the
// records (a ring): the four 64-bit words of each, its voxel and scene.
struct TessStage {
    TessQueue q;
    ulonglong2 words[64][2];
    uint32_t vox[64], scene[64];
};

// Adds the `n` (at most 32) oldest queued runs to their records, four lanes to
// a record.
//
// Exact past 65,536 points: the old values show every crossing of 2^32 by r, g,
// b, nx and ny (the count itself never gets near one; nz's carries land in the
// last word's unused high half).  The add that takes the count past 65,536
// lists the voxel even without a crossing, so that the carry pass rewrites
// every voxel whose nz may have carried.  The voxel's occupancy bit is set by
// the add that found its count at 0.
template <class Scenes>
__device__ __forceinline__ void tess_flush(const Scenes& S, const TessStage& st, int head, int n, int lane) {
    const int w = lane & 3;
    unsigned long long add[4], was[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = 8 * i + (lane >> 2), e = (head + r) & 63;
        add[i] = was[i] = 0ull;
        if (r < n) {
            add[i] = reinterpret_cast<const unsigned long long*>(st.words)[4 * e + w];
            // (the record's place is found here and not where the run is queued: that is done every step)
            const AccumParams& P = S.get((int)st.scene[e]);
            was[i] = atomicAdd(reinterpret_cast<unsigned long long*>(P.acc + kAccWords * record_slot(st.vox[e], P.dim)) + w,
                               add[i]);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        // the sum carried out of the low field, out of the high one; the count
        // was 0, or passes 65,536
        const unsigned long long sum = was[i] + add[i];
        const uint32_t c0 = (uint32_t)was[i], c1 = (uint32_t)sum;
        const bool lo = c1 < c0, hi = sum < was[i];
        const bool first = w == 0 && c0 == 0u && add[i] != 0ull, listed = w == 0 && c0 <= 65536u && c1 > 65536u;
        if (w != 3 && (lo || hi || first || listed)) {
            const int e = (head + 8 * i + (lane >> 2)) & 63;
            const AccumParams& P = S.get((int)st.scene[e]);
            const uint32_t v = st.vox[e];
            if (first) atomicOr(P.occ + (v >> 5), 1u << (v & 31));
            if (P.carry && (lo || hi || listed)) {
                const uint32_t ev[kCarryEvents] = {w == 0 && hi, w == 1 && lo, w == 1 && hi, w == 2 && lo, w == 2 && hi};
                carry_add(P.carry, v, ev, P.stats);
            }
        }
    }
}

// The quotients of the points' places, IEEE-rounded: j / q, j < q, and 2k / (3n)
// for the rings k < n / 2 of inner level n.
struct TessTables {
    float quot[kMaxTess * (kMaxTess + 1) / 2];
    float ring[kMaxTess + 1][kMaxTess / 2];
};
__device__ __forceinline__ void fill_tables(TessTables& T) {
    for (int i = threadIdx.x; i < kMaxTess * kMaxTess; i += blockDim.x) {
        const int q = i / kMaxTess + 1, j = i % kMaxTess;
        if (j < q) T.quot[q * (q - 1) / 2 + j] = __fdiv_rn((float)j, (float)q);
        if (j < kMaxTess / 2) T.ring[q][j] = __fdiv_rn((float)(2 * j), (float)(3 * q));
    }
}

// testTesselation.tese:101-133: the voxel of a point at `pos`; false outside.
__device__ __forceinline__ bool tess_voxel(const AccumParams& P, f3 pos, uint32_t& v) {
    const int N = P.dim;
    const float fN = (float)N;
    f3 tc;  // times N
    if (P.warp.mode == VCT_WARP_PERSPECTIVE) {  // voxelTesselationWarpedPosition
        tc = mul(perspective_tc(P.warp, pos), fN);
    } else {  // voxelLinearPosition (the evaluation shader passes warpVoxels = false)
        tc = sub(sub(pos, P.vcenter), P.vmin);
        if (P.ext_rcp != 0.0f)  // the extents are a power of two, as N is: the product is the quotient's
            tc = mul(tc, P.ext_rcp * fN);
        else
            tc = mul(mk(__fdiv_rn(tc.x, P.ext.x), __fdiv_rn(tc.y, P.ext.y), __fdiv_rn(tc.z, P.ext.z)), fN);
    }
    const int vx = trunc_sat(tc.x), vy = trunc_sat(tc.y), vz = trunc_sat(tc.z);
    if ((uint32_t)(vx | vy | vz) >= (uint32_t)N) return false;  // not all in [0, N): N is a power of two
    v = (uint32_t)((vz * N + vy) * N + vx);
    return true;
}
// voxelStore: normalize(normal) * 0.5 + 0.5.
__device__ __forceinline__ void tess_normal(f3 nrm, uint32_t& qx, uint32_t& qy, uint32_t& qz) {
    const f3 Nf = normalize(nrm);
    qx = quant16(Nf.x * 0.5f + 0.5f);
    qy = quant16(Nf.y * 0.5f + 0.5f);
    qz = quant16(Nf.z * 0.5f + 0.5f);
}

// The queued points, one per lane (lanes >= nact idle), stored with 64-bit
// reductions.  Neighbouring points of a ring edge often share a voxel: an even
// lane takes its odd neighbour's sums when both hit the same voxel (one shuffle
// per word), so the pair costs one set of reductions.  Exact as tess_flush is.
template <class Scenes>
__device__ __forceinline__ void tess_store32(const Scenes& S, const TessQueue& q, int nact, int lane) {
    const unsigned FULL = 0xffffffffu;
    bool valid = false;
    uint32_t v = 0, qr = 0, qg = 0, qb = 0, qx = 0, qy = 0, qz = 0;
    const AccumParams& P = S.get(lane < nact ? (int)(q.item[lane] >> 16) : 0);
    if (lane < nact) {
        const long long t = q.tri[lane];
        const f3 bc = tess_coord(q.lev[lane], (int)(q.item[lane] & 0xffffu));
        const float* Pp = P.pos + t * 9;
        const float* Pn = P.nrm + t * 9;
        const f3 p0 = ld3(Pp), p1 = ld3(Pp + 3), p2 = ld3(Pp + 6);
        const f3 n0 = ld3(Pn), n1 = ld3(Pn + 3), n2 = ld3(Pn + 6);
        valid = tess_voxel(P, add(add(mul(p0, bc.x), mul(p1, bc.y)), mul(p2, bc.z)), v);
        if (valid) {
            const f3 col = ld3(P.albedo + t * 3);
            qr = quant16(col.x);
            qg = quant16(col.y);
            qb = quant16(col.z);
            tess_normal(add(add(mul(n0, bc.x), mul(n1, bc.y)), mul(n2, bc.z)), qx, qy, qz);
        }
    }
    const unsigned key = valid ? v : 0xffffffffu;
    const unsigned partner = __shfl_xor_sync(FULL, key, 1);  // every lane takes part
    const bool pair = valid && partner == key;
    const uint32_t pr = __shfl_xor_sync(FULL, qr, 1), pg = __shfl_xor_sync(FULL, qg, 1), pb = __shfl_xor_sync(FULL, qb, 1),
                   px = __shfl_xor_sync(FULL, qx, 1), py = __shfl_xor_sync(FULL, qy, 1), pz = __shfl_xor_sync(FULL, qz, 1);
    if (!valid || (pair && (lane & 1))) return;
    unsigned long long cnt = 1;
    if (pair) {
        cnt = 2;
        qr += pr;
        qg += pg;
        qb += pb;
        qx += px;
        qy += py;
        qz += pz;
    }
    unsigned long long* rec = reinterpret_cast<unsigned long long*>(P.acc + kAccWords * record_slot(v, P.dim));
    const unsigned long long a0 = cnt | ((unsigned long long)qr << 32);
    const unsigned long long a1 = (unsigned long long)qg | ((unsigned long long)qb << 32);
    const unsigned long long a2 = (unsigned long long)qx | ((unsigned long long)qy << 32);
    const unsigned long long was = atomicAdd(rec + 0, a0);
    const uint32_t c0 = (uint32_t)was;
    if (P.carry) {
        const unsigned long long w1 = atomicAdd(rec + 1, a1), w2 = atomicAdd(rec + 2, a2);
        atomicAdd(rec + 3, (unsigned long long)qz);
        const uint32_t ev[kCarryEvents] = {wrap_hi(was, a0), carry_lo(w1, a1), wrap_hi(w1, a1), carry_lo(w2, a2),
                                           wrap_hi(w2, a2)};
        if ((ev[0] | ev[1] | ev[2] | ev[3] | ev[4]) || (c0 <= 65536u && c0 + (uint32_t)cnt > 65536u))
            carry_add(P.carry, v, ev, P.stats);
    } else {
        atomicAdd(rec + 1, a1);
        atomicAdd(rec + 2, a2);
        atomicAdd(rec + 3, (unsigned long long)qz);
    }
    if (c0 == 0u) atomicOr(P.occ + (v >> 5), 1u << (v & 31));
}

// The queued items, one per lane (lanes >= nact idle).
template <class Scenes>
__device__ __forceinline__ uint32_t tess_walk32(const Scenes& S, TessStage& st, const TessTables& T, int nact, int lane,
                                                int& head, int& count) {
    const unsigned FULL = 0xffffffffu;
    constexpr uint32_t kNone = 0xffffffffu;
    f3 p0 = mk(0.f, 0.f, 0.f), p1 = p0, p2 = p0, n0 = p0, n1 = p0, n2 = p0;
    uint32_t qrg = 0, qb = 0;  // quantised albedo
    TessItem it = {0, 0, 0, 0, 0, 0};
    int scene = 0, at = 0, step = 0;  // the place in T.quot, what a point adds to it
    const float* ring = T.ring[1];
    float third = 0.0f;  // the centre's coordinates
    if (lane < nact) {
        scene = (int)(st.q.item[lane] >> 16);
        const AccumParams& P = S.get(scene);
        const long long t = st.q.tri[lane];
        const uint32_t packed = st.q.lev[lane];
        it = tess_item(packed, (int)(st.q.item[lane] & 0xffffu), kTessRunLog2);
        const int n = (int)(packed & 127u);
        ring = T.ring[n] + it.k;
        // (an outer edge's segments: outer[0] from corner 1, outer[1] from 2, outer[2] from 0)
        int q = it.k ? n - 2 * it.k : (int)((packed >> (it.c == 0 ? 21 : 7 * it.c)) & 127u);
        if (q == 0) {
            q = 1;
            ring = T.ring[1];
            third = __fdiv_rn(1.0f, 3.0f);
        }
        at = q * (q - 1) / 2 + it.j;
        step = it.dj - (it.dk ? 6 * q - 21 : 0);  // q falls by 6 with k + 3
        const float* Pp = P.pos + t * 9;
        const float* Pn = P.nrm + t * 9;
        p0 = ld3(Pp), p1 = ld3(Pp + 3), p2 = ld3(Pp + 6);
        n0 = ld3(Pn), n1 = ld3(Pn + 3), n2 = ld3(Pn + 6);
        const f3 col = ld3(P.albedo + t * 3);
        qrg = quant16(col.x) | (quant16(col.y) << 16);
        qb = quant16(col.z);
    }
    const int cnt = it.cnt;
    const AccumParams& P = S.get(scene);
    uint32_t cur = kNone, run = 0, sx = 0, sy = 0, sz = 0;
    // Queues the finished runs of the lanes with `push`; 32 queued ones go out.
    auto finish = [&](bool push) {
        const unsigned m = __ballot_sync(FULL, push);
        if (!m) return;
        if (push) {
            const int e = (head + count + __popc(m & ((1u << lane) - 1u))) & 63;
            st.words[e][0] = make_ulonglong2((unsigned long long)run | ((unsigned long long)((qrg & 0xffffu) * run) << 32),
                                             (unsigned long long)((qrg >> 16) * run) |
                                                 ((unsigned long long)(qb * run) << 32));
            st.words[e][1] = make_ulonglong2((unsigned long long)sx | ((unsigned long long)sy << 32), (unsigned long long)sz);
            st.vox[e] = cur;
            st.scene[e] = (uint32_t)scene;
        }
        count += __popc(m);
        __syncwarp();
        if (count >= 32) {
            tess_flush(S, st, head, 32, lane);
            head = (head + 32) & 63;
            count -= 32;
            __syncwarp();
        }
    };
    const int steps = __reduce_max_sync(FULL, cnt);
    for (int i = 0; i < steps; ++i) {
        uint32_t v = kNone, qx = 0, qy = 0, qz = 0;
        if (i < cnt) {
            // corner c's coordinate falls from h to t, the next one's rises from t to h, the third's is t
            const float s = T.quot[at], t = third != 0.0f ? third : *ring;
            const float h = third != 0.0f ? third : 1.0f - 2.0f * t, d = h - t;
            const float from = h + s * -d, to = t + s * d;
            const f3 bc = mk(it.c == 0 ? from : it.c == 2 ? to : t, it.c == 1 ? from : it.c == 0 ? to : t,
                             it.c == 2 ? from : it.c == 1 ? to : t);
            at += step;
            if (it.dk) step += 36;
            ring += it.dk;
            uint32_t at_voxel;
            if (tess_voxel(P, add(add(mul(p0, bc.x), mul(p1, bc.y)), mul(p2, bc.z)), at_voxel)) {
                v = at_voxel;
                tess_normal(add(add(mul(n0, bc.x), mul(n1, bc.y)), mul(n2, bc.z)), qx, qy, qz);
            }
        }
        const bool change = i < cnt && v != cur;
        finish(change && run > 0);
        if (change) {
            cur = v;
            run = sx = sy = sz = 0;
        }
        if (v != kNone) {
            ++run;
            sx += qx;
            sy += qy;
            sz += qz;
        }
    }
    finish(run > 0);
    return (uint32_t)cnt;
}

// The carry pass: every voxel listed in a scene's carry table gets its six
// 64-bit sums rebuilt from its record and its crossings of 2^32, its record
// rewritten with their float values (the resolve's dividend) and bit 31 of
// the count set, and its brick flagged for the resolve's exact pass.  One
// thread per table slot, blockIdx.y the scene.
template <class Scenes>
__global__ void __launch_bounds__(256) carry_fixup_kernel(const Scenes S) {
    const AccumParams& P = S.get(blockIdx.y);
    const int slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (!P.carry || slot >= kCarrySlots) return;
    const uint32_t* e = P.carry + 8 * slot;
    if (e[0] == 0u) return;
    const long long v = (long long)e[0] - 1;
    uint4* r = reinterpret_cast<uint4*>(P.acc + kAccWords * record_slot(v, P.dim));
    const uint4 r0 = r[0], r1 = r[1];
    const unsigned long long t = 1ull << 32;
    // {count | r}, {g | b}, {nx | ny}, {nz | nz's carries}: a high field holds
    // its own sum plus the low field's carries, modulo 2^32
    const unsigned long long sr = r0.y + t * e[1], sg = r0.z + t * e[2], sb = r0.w + t * e[3] - e[2],
                             sx = r1.x + t * e[4], sy = r1.y + t * e[5] - e[4], sz = r1.z + t * r1.w;
    r[0] = make_uint4(r0.x | 0x80000000u, __float_as_uint(__ull2float_rn(sr)), __float_as_uint(__ull2float_rn(sg)),
                      __float_as_uint(__ull2float_rn(sb)));
    r[1] = make_uint4(__float_as_uint(__ull2float_rn(sx)), __float_as_uint(__ull2float_rn(sy)),
                      __float_as_uint(__ull2float_rn(sz)), 0u);
    const long long N = P.dim, bpa = N / 16;  // the voxel's 16^3 brick, in the resolve's brick order
    const long long x = v % N, y = (v / N) % N, z = v / (N * N);
    P.brick_exact[((z / 16) * bpa + y / 16) * bpa + x / 16] = 1u;
}

// Adds a warp's counts of generated points (this lane's `points` of a single
// scene; or a scene's by point_count) to the scenes' statistics.
template <class Scenes>
__device__ __forceinline__ void add_points(const Scenes& S, unsigned* point_count, uint32_t points) {
    if (points) atomicAdd(&point_count[0], points);
    __syncthreads();
    for (int i = threadIdx.x; i < S.count(); i += blockDim.x)
        if (point_count[i] && S.get(i).stats) atomicAdd(&S.get(i).stats->total_voxel_fragments, point_count[i]);
}

// The walk.  Warps take units from a shared counter (their first by their own
// number), whose values are spread over the unit order (kTessSpread places in
// turn): neighbouring units, which belong to neighbouring triangles and add to
// the same records, are then not worked on at the same time.
template <class Scenes>
__global__ void __launch_bounds__(kWarps * 32, kTessBlocksPerSM) tess_walk_kernel(const Scenes S, const VoxWork W, int nblocks) {
    __shared__ TessStage stages[kWarps];
    __shared__ TessTables tables;
    __shared__ unsigned point_count[kMaxBatchScenes];  // generated points per scene
    grid_launch_dependents();  // the other kernel, of which one ends at once, reads nothing of this one
    const uint4 total = W.block_off[nblocks];
    if (!tess_walks(total)) return;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    TessStage& st = stages[threadIdx.x >> 5];
    const int nscenes = S.count();
    for (int i = threadIdx.x; i < nscenes; i += blockDim.x) point_count[i] = 0;
    fill_tables(tables);
    __syncthreads();
    const long long nw = (long long)gridDim.x * kWarps, warp = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    const int grab = (int)max(1LL, min((long long)kTessGrab, total.x / nw));
    const long long grabs = ((long long)total.x + grab - 1) / grab, spread = min((long long)kTessSpread, grabs),
                    stretch = (grabs + spread - 1) / spread;
    unsigned long long* counter = grab_counter(W, nblocks);
    int qn = 0;               // queued items (warp-uniform)
    int head = 0, count = 0;  // the ring of finished runs (warp-uniform)
    uint32_t points = 0;      // this lane's, of a single scene
    auto walk = [&](int nact) {
        const int scene = lane < nact ? (int)(st.q.item[lane] >> 16) : 0;
        const uint32_t pts = tess_walk32(S, st, tables, nact, lane, head, count);
        if (nscenes > 1) {
            if (pts) atomicAdd(&point_count[scene], pts);
        } else {
            points += pts;
        }
    };
    UnitOwner<true> o = {0, 0u, 0u};
    for (long long c = warp; c < stretch * spread;) {
        const long long u0 = ((c % spread) * stretch + c / spread) * grab;
        if (u0 < total.x) {
            const uint32_t u1 = (uint32_t)min(u0 + grab, (long long)total.x);
            o.find(W, nblocks, (uint32_t)u0, lane);
            for (uint32_t u = (uint32_t)u0; u < u1; ++u) {
                o.follow(W, nblocks, u, lane);
                const uint4 r = __ldg(W.tri_rec + o.g);
                queue_unit(st.q, qn, r, r.y >> 16, u - o.start, lane, walk);
            }
        }
        if (nw >= stretch * spread) break;
        unsigned long long next = 0;
        if (lane == 0) next = atomicAdd(counter, 1ull);
        c = nw + (long long)__shfl_sync(FULL, next, 0);
    }
    walk(qn);
    tess_flush(S, st, head, count, lane);
    add_points(S, point_count, points);
}

// The points, where nothing is walked: an equal range of units to each warp.
template <class Scenes>
__global__ void __launch_bounds__(kWarps * 32, 4) tess_points_kernel(const Scenes S, const VoxWork W, int nblocks) {
    __shared__ TessQueue queues[kWarps];
    __shared__ unsigned point_count[kMaxBatchScenes];
    const uint4 total = W.block_off[nblocks];
    if (tess_walks(total)) {
        grid_wait();  // (this kernel's end is the walk's for the ones behind it)
        return;
    }
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    TessQueue& q = queues[threadIdx.x >> 5];
    const int nscenes = S.count();
    for (int i = threadIdx.x; i < nscenes; i += blockDim.x) point_count[i] = 0;
    __syncthreads();
    const long long nw = (long long)gridDim.x * kWarps, warp = (long long)blockIdx.x * kWarps + (threadIdx.x >> 5);
    const uint32_t u0 = (uint32_t)((unsigned long long)total.y * warp / nw),
                   u1 = (uint32_t)((unsigned long long)total.y * (warp + 1) / nw);
    int qn = 0;
    uint32_t points = 0;
    auto store = [&](int nact) {
        tess_store32(S, q, nact, lane);
        if (nscenes > 1) {
            const int scene = lane < nact ? (int)(q.item[lane] >> 16) : -1;
            const unsigned same = __match_any_sync(FULL, scene);
            if (scene >= 0 && lane == __ffs(same) - 1) atomicAdd(&point_count[scene], (unsigned)__popc(same));
        } else {
            points += lane < nact ? 1u : 0u;
        }
    };
    UnitOwner<false> o = {0, 0u, 0u};
    if (u0 < u1) o.find(W, nblocks, u0, lane);
    for (uint32_t u = u0; u < u1; ++u) {
        o.follow(W, nblocks, u, lane);
        const uint4 r = __ldg(W.tri_rec + o.g);
        queue_unit(q, qn, r, r.y & 0xffffu, u - o.start, lane, store);
    }
    store(qn);
    add_points(S, point_count, points);
    grid_wait();
}

template <class Scenes>
void launch_tess(const Scenes& S, const VoxWork& W, int num_sms, cudaStream_t s) {
    if (W.ntri <= 0) return;
    const int nblocks = (int)((W.ntri + kSetupThreads - 1) / kSetupThreads);
    tess_setup_kernel<Scenes><<<nblocks, kSetupThreads, 0, s>>>(S, W);
    voxelize_scan_kernel<<<1, 1024, 0, s>>>(W.block_off, nblocks);
    tess_walk_kernel<Scenes><<<num_sms * kTessBlocksPerSM, kWarps * 32, 0, s>>>(S, W, nblocks);
    launch_overlapped(tess_points_kernel<Scenes>, dim3((unsigned)(num_sms * 4)), kWarps * 32, 0, s, S, W, nblocks);
    note_launches(3);
}

}  // namespace

// The tessellation voxeliser: setup, scan, the walk and the points.
void launch_tesselate(const AccumParams& P, cudaStream_t s) {
    const VoxWork W = {P.tri_rec, P.tri_units, P.tri_scan, P.block_off, P.ntri};
    launch_tess(OneScene<AccumParams>{P}, W, P.num_sms, s);
    if (P.carry) {
        carry_fixup_kernel<<<dim3(kCarrySlots / 256, 1), 256, 0, s>>>(OneScene<AccumParams>{P});
        note_launches(1);
    }
}

void launch_tesselate_batch(const SceneBatch<AccumParams>& B, const VoxWork& W, int num_sms, cudaStream_t s) {
    launch_tess(ManyScenes<AccumParams>{B}, W, num_sms, s);
    carry_fixup_kernel<<<dim3(kCarrySlots / 256, B.n), 256, 0, s>>>(ManyScenes<AccumParams>{B});
    note_launches(1);
}

void tess_bind_scratch(AccumParams& P, void* scratch) {
    char* p = static_cast<char*>(scratch);
    const long long ntri = P.ntri;
    P.tri_rec = reinterpret_cast<uint4*>(p);
    p += align256(ntri * 16);
    P.tri_units = reinterpret_cast<uint32_t*>(p);
    p += align256(ntri * 4);
    P.tri_scan = reinterpret_cast<uint32_t*>(p);
    p += align256(ntri * 4);
    P.block_off = reinterpret_cast<uint4*>(p);
}

void launch_occupancy(const AccumParams& P, cudaStream_t s) {
    if (P.ntri <= 0) return;
    occupancy_kernel<<<(unsigned)((P.ntri + kOccThreads - 1) / kOccThreads), kOccThreads, 0, s>>>(
        OneScene<AccumParams>{P}, P.ntri);
    note_launches(1);
}

void launch_occupancy_batch(const SceneBatch<AccumParams>& B, long long ntri, cudaStream_t s) {
    if (ntri <= 0) return;
    occupancy_kernel<<<(unsigned)((ntri + kOccThreads - 1) / kOccThreads), kOccThreads, 0, s>>>(
        ManyScenes<AccumParams>{B}, ntri);
    note_launches(1);
}

void launch_accumulate(const AccumParams& P, cudaStream_t s) {
    launch_voxelize(OneScene<AccumParams>{P}, P.ntri, (long long)P.dim * P.dim, P.unit_log2, P.num_sms, P.blocks_per_sm, s);
}

int accumulate_batch_max_scenes() { return kMaxBatchScenes; }

void launch_accumulate_batch(const SceneBatch<AccumParams>& B, long long ntri, long long faces, int unit_log2,
                             int num_sms, int blocks_per_sm, cudaStream_t s) {
    launch_voxelize(ManyScenes<AccumParams>{B}, ntri, faces, unit_log2, num_sms, blocks_per_sm, s);
}

}  // namespace vct
