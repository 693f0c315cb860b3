// Learned indirect light (the "learned" configuration): a cheap two-cone
// quarter-resolution trace plus G-buffer features feed a small BF16 MLP
// (42-64-64-64-4, FP32 accumulation) that predicts the 16-cone full-resolution
// irradiance and an estimate of its own error there.  Inference and training run on the fifth-generation tensor
// cores (tcgen05.mma, accumulators in TMEM; umma.cuh).
//
// Compiled with --fmad=false: the cone marching (cone.cuh) writes its fused
// multiply-adds out.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>

#include "cone.cuh"
#include "umma.cuh"

namespace vct {

namespace {

using namespace umma;

// ------------------------------------------------------------ GEMM check
// One 128 x N x K BF16 GEMM through the tensor core: A (128 x K) and B (N x K)
// row-major in global memory, D = A B^T (128 x N, FP32) back to global.
// `swap` exchanges the two descriptor strides (a diagnostic of the layout
// convention; both variants stay inside the zero-filled operand regions).
constexpr int kCheckSmemA = 32768, kCheckSmemB = 16384;

__global__ void __launch_bounds__(128) umma_check_kernel(const uint16_t* __restrict__ A,
                                                          const uint16_t* __restrict__ B, int K, int N, int swap,
                                                          float* __restrict__ D, uint32_t* __restrict__ status) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_base;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* sa = smem;
    uint8_t* sb = smem + kCheckSmemA;
    for (int i = threadIdx.x; i < (kCheckSmemA + kCheckSmemB) / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    for (int i = threadIdx.x; i < 128 * K; i += blockDim.x)
        *reinterpret_cast<uint16_t*>(sa + tile_offset(i / K, i % K, 128)) = A[i];
    for (int i = threadIdx.x; i < N * K; i += blockDim.x)
        *reinterpret_cast<uint16_t*>(sb + tile_offset(i / K, i % K, N)) = B[i];
    fence_async_smem();
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&mbar), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&tmem_base), 64);
        tmem_relinquish();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tbase = tmem_base;
    if (threadIdx.x == 0) {
        const uint32_t a0 = smem_u32(sa), b0 = smem_u32(sb);
        const uint32_t idesc = idesc_bf16_f32(128, N);
        for (int j = 0; j < K / 16; ++j) {
            const uint64_t da = swap ? smem_desc(a0 + j * 2 * 128 * 16, 128, 128 * 16) : tile_desc(a0, 128, j);
            const uint64_t db = swap ? smem_desc(b0 + j * 2 * N * 16, 128, N * 16) : tile_desc(b0, N, j);
            mma_bf16(tbase, da, db, idesc, j > 0 ? 1u : 0u);
        }
        commit(smem_u32(&mbar));
    }
    const int ok = __syncthreads_and(mbar_wait(smem_u32(&mbar), 0) ? 1 : 0);
    fence_after_sync();
    if (ok) {
        for (int c = 0; c < N; c += 16) {
            float v[16];
            tmem_ld16(tmem_addr(tbase, warp, c), v);
#pragma unroll
            for (int i = 0; i < 16; ++i) D[(32 * warp + lane) * N + c + i] = v[i];
        }
    } else if (threadIdx.x == 0) {
        atomicOr(status, 1u);
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, 64);
}

// -------------------------------------------------------------- helpers
__device__ __forceinline__ uint32_t bf16x2(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// max(a, 0) and max(b, 0) rounded to BF16 and packed (a low): one
// conversion with ReLU, which commutes with round-to-nearest.
__device__ __forceinline__ uint32_t bf16x2_relu(float a, float b) {
    uint32_t r;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(b), "f"(a));
    return r;
}
__device__ __forceinline__ uint16_t bf16(float a) { return __bfloat16_as_ushort(__float2bfloat16_rn(a)); }
__device__ __forceinline__ float bf16f(uint32_t bits16) { return __uint_as_float(bits16 << 16); }

__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

// Barrier that also orders tcgen05 operations across it.
__device__ __forceinline__ void tc_sync() {
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
}

// Orthonormal basis (T, B) around unit N: Duff et al. 2017, "Building an
// Orthonormal Basis, Revisited" (JCGT 6(1)), as the cone tracer uses it.
__device__ __forceinline__ void onb(f3 N, f3& T, f3& B) {
    const float sgn = N.z >= 0.0f ? 1.0f : -1.0f;
    const float ca = -1.0f / (sgn + N.z);
    const float cb = N.x * N.y * ca;
    T = mk(1.0f + sgn * N.x * N.x * ca, sgn * cb, -sgn * N.x);
    B = mk(cb, sgn + N.y * N.y * ca, -N.y);
}

// Position in [0,1]^3 volume texture coordinates (voxelLinearPosition).
__device__ __forceinline__ f3 volume_coord(const TraceParams& P, float4 gp) {
    const f3 ext = sub(P.vmax, P.vmin);
    return mk(((gp.x - P.vcenter.x) - P.vmin.x) / ext.x, ((gp.y - P.vcenter.y) - P.vmin.y) / ext.y,
              ((gp.z - P.vcenter.z) - P.vmin.z) / ext.z);
}

// ------------------------------------------------------- cheap trace
// Quarter-resolution features: for each 4x4 pixel block, at its first
// covered pixel (centre pixels first), two 90-degree cones along
// normalize(N + T) and normalize(N - T).  With a 90-degree aperture a cone's
// diameter doubles every step, so step s (distance 2^s voxels past the
// one-voxel normal bias) is one trilinear sample of mip level s + 1.  Each
// cone marches 8 steps (levels 1..8, clamped to the chain), compositing front
// to back as traceCone does; its accumulated RGBA after the samples of levels
// 2, 4, 6 and 8 are the cone's 4 x 4 features.  A cone that leaves the volume
// keeps its accumulated value.
__constant__ unsigned char kRepOrder[16] = {5, 10, 6, 9, 0, 1, 2, 3, 4, 7, 8, 11, 12, 13, 14, 15};

__global__ void __launch_bounds__(256) learned_features_kernel(const LearnedParams P) {
    __shared__ cone::Level s_lv[VCT_MAX_LEVELS];
    cone::fill_levels(P.T, s_lv);
    __syncthreads();
    const int qx = blockIdx.x * 16 + (threadIdx.x & 15), qy = blockIdx.y * 16 + (threadIdx.x >> 4);
    if (qx >= P.wq || qy >= P.hq) return;
    const TraceParams& T = P.T;
    float4 gp = make_float4(0.f, 0.f, 0.f, 0.f);
    long long pix = -1;
    for (int k = 0; k < 16 && pix < 0; ++k) {
        const int x = 4 * qx + (kRepOrder[k] & 3), y = 4 * qy + (kRepOrder[k] >> 2);
        if (x < T.width && y < T.height) {
            const long long p = (long long)y * T.width + x;
            gp = __ldg(T.gpos + p);
            if (gp.w != 0.0f) pix = p;
        }
    }
    uint32_t f[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) f[i] = 0u;
    if (pix >= 0) {
        const float4 gn = __ldg(T.gnrm + pix);
        const f3 N = cone::fnormalize(mk(gn.x, gn.y, gn.z));
        f3 Tg, Bg;
        onb(N, Tg, Bg);
        const f3 vp = volume_coord(T, gp);
        const float scale = 1.0f / (float)T.dim;
        const f3 start = add(vp, mul(N, scale));
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const f3 d = cone::fnormalize(c == 0 ? add(N, Tg) : sub(N, Tg));
            float h = 1.0f, alpha = 0.0f;
            f3 col = mk(0.f, 0.f, 0.f);
            bool inside = true;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const f3 sp = mk(fmaf(d.x, h * scale, start.x), fmaf(d.y, h * scale, start.y),
                                 fmaf(d.z, h * scale, start.z));
                inside = inside && sp.x >= 0.f && sp.y >= 0.f && sp.z >= 0.f && sp.x <= 1.f && sp.y <= 1.f &&
                         sp.z <= 1.f;
                if (inside) {
                    const f3 wp = T.warp.mode ? apply_warp(T.warp, sp) : sp;
                    const float4 smp =
                        cone::trilinear(T.pchain, s_lv[min(i + 1, T.levels - 1)], wp, T.warp.mode != VCT_WARP_NONE);
                    const float a = 1.0f - alpha;
                    col = mk(fmaf(smp.x, a, col.x), fmaf(smp.y, a, col.y), fmaf(smp.z, a, col.z));
                    alpha = fmaf(a, smp.w, alpha);
                }
                if (i & 1) {
                    const int k = c * 8 + (i >> 1) * 2;
                    f[k] = bf16x2(col.x, col.y);
                    f[k + 1] = bf16x2(col.z, alpha);
                }
                h *= 2.0f;
            }
        }
    }
    uint4* dst = reinterpret_cast<uint4*>(const_cast<uint16_t*>(P.qfeat) + ((long long)qy * P.wq + qx) * kCheapFeatures);
#pragma unroll
    for (int i = 0; i < 4; ++i) dst[i] = make_uint4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]);
}

// The 42 features of pixel `pix` (covered: gp.w != 0) as 24 packed BF16
// pairs (48 features, the last 6 zero): the quarter-resolution cone features
// of its 4x4 block, the unit normal N, the eye distance times depth_scale,
// the albedo, and the near-field radiance RGB: one trilinear sample of mip
// level 1 where the diffuse cones take their first sample along N (two
// voxels above the surface), zero outside the volume.
__device__ __forceinline__ void pixel_features(const LearnedParams& P, long long pix, float4 gp, uint32_t (&f)[24]) {
    const TraceParams& T = P.T;
    const int x = (int)(pix % T.width), y = (int)(pix / T.width);
    const uint4* q =
        reinterpret_cast<const uint4*>(P.qfeat + ((long long)(y >> 2) * P.wq + (x >> 2)) * kCheapFeatures);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint4 v = __ldg(q + i);
        f[4 * i] = v.x;
        f[4 * i + 1] = v.y;
        f[4 * i + 2] = v.z;
        f[4 * i + 3] = v.w;
    }
    const float4 gn = __ldg(T.gnrm + pix);
    const float4 ga = __ldg(T.galb + pix);
    const f3 N = cone::fnormalize(mk(gn.x, gn.y, gn.z));
    const f3 d = sub(mk(gp.x, gp.y, gp.z), T.eye);
    const float dist = sqrtf(dot(d, d));
    const f3 vp = volume_coord(T, gp);
    const float step = 2.0f / (float)T.dim;
    const f3 sp = mk(fmaf(N.x, step, vp.x), fmaf(N.y, step, vp.y), fmaf(N.z, step, vp.z));
    float4 near = make_float4(0.f, 0.f, 0.f, 0.f);
    if (sp.x >= 0.f && sp.y >= 0.f && sp.z >= 0.f && sp.x <= 1.f && sp.y <= 1.f && sp.z <= 1.f) {
        near = cone::trilinear(T.pchain, cone::level_of(T.dim, 1), T.warp.mode ? apply_warp(T.warp, sp) : sp,
                               T.warp.mode != VCT_WARP_NONE);
    }
    f[16] = bf16x2(N.x, N.y);
    f[17] = bf16x2(N.z, dist * P.depth_scale);
    f[18] = bf16x2(ga.x, ga.y);
    f[19] = bf16x2(ga.z, near.x);
    f[20] = bf16x2(near.y, near.z);
    f[21] = f[22] = f[23] = 0u;
}

// Training rows: the 42 features of listed pixels as fp32 (exactly the BF16
// values the inference kernel feeds the network).
__global__ void __launch_bounds__(256) learned_rows_kernel(const LearnedParams P) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    const long long pix = P.pixels[i];
    const float4 gp = __ldg(P.T.gpos + pix);
    float* row = P.rows_out + i * kMlpIn;
    if (gp.w == 0.0f) {
        for (int k = 0; k < kMlpIn; ++k) row[k] = 0.0f;
        return;
    }
    uint32_t f[24];
    pixel_features(P, pix, gp, f);
    for (int k = 0; k < kMlpIn; ++k) row[k] = bf16f((f[k >> 1] >> ((k & 1) * 16)) & 0xFFFFu);
}

// ------------------------------------------------------- 16-cone trace
// Irradiance of the 16-cone reference set: cones of the Fibonacci hemisphere
// set in the (T, B, N) frame, each weighted by its cosine, summed.
template <int KIND>
__device__ __forceinline__ float4 irradiance16(const LearnedParams& P, const cone::Level* lv, const cone::ConeTable& tab,
                                               const float (*dirs)[4], float4 gp, float4 gn, unsigned& ns) {
    const TraceParams& T = P.T;
    const f3 N = cone::fnormalize(mk(gn.x, gn.y, gn.z));
    f3 Tg, Bg;
    onb(N, Tg, Bg);
    const f3 vp = volume_coord(T, gp);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 1
    for (int c = 0; c < 16; ++c) {
        const f3 d = add(add(mul(Tg, dirs[c][0]), mul(Bg, dirs[c][1])), mul(N, dirs[c][2]));
        const float4 cr = cone::trace_cone<VCT_FILTER_SOFTWARE, KIND>(T, lv, tab, vp, N, d, P.ref_cone, T.max_distance, ns);
        const float w = dirs[c][3];
        acc = make_float4(fmaf(w, cr.x, acc.x), fmaf(w, cr.y, acc.y), fmaf(w, cr.z, acc.z), fmaf(w, cr.w, acc.w));
    }
    return acc;
}

__device__ __forceinline__ void load_dirs(const LearnedParams& P, float (*s_dirs)[4]) {
    if (threadIdx.x < 64) s_dirs[threadIdx.x >> 2][threadIdx.x & 3] = P.dirs16[threadIdx.x >> 2][threadIdx.x & 3];
}

// 16-cone irradiance of whole 16x16 tiles (every tile, or the listed ones), half
// a tile to a CTA and six of them to an SM, eight of the listed ones': an image of
// a few tiles to an SM otherwise ends with some SMs a heavy tile behind the others.
// 128^3 at 320x180, 640x360, 800x450 and 1920x1080: 142, 232, 379 and 1,673 us;
// whole tiles, four to an SM, 167, 294, 470 and 1,677, and before the cones' step
// tables, three to an SM, 185, 266, 401 and 1,754.
constexpr int kTile16Threads = 128;  // (the cones' table takes that many)
template <int KIND, bool LISTED>
__global__ void __launch_bounds__(kTile16Threads, LISTED ? 8 : 6) trace16_kernel(const LearnedParams P) {
    __shared__ cone::Level s_lv[VCT_MAX_LEVELS];
    __shared__ cone::ConeTable s_cone;
    __shared__ float s_dirs[16][4];
    const TraceParams& T = P.T;
    const int tiles_x = (T.width + kLearnTile - 1) / kLearnTile;
    const long long total = LISTED ? (long long)*P.count : (long long)tiles_x * ((T.height + kLearnTile - 1) / kLearnTile);
    if (blockIdx.x >= 2 * total) return;  // past the list
    cone::fill_levels(P.T, s_lv);
    cone::fill_cone(P.T, P.ref_cone, P.T.max_distance, s_cone, 64);
    load_dirs(P, s_dirs);
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned ns = 0;
    for (long long t = blockIdx.x; t < 2 * total; t += gridDim.x) {
        const long long tile = LISTED ? (long long)P.list[t >> 1] : t >> 1;
        const int x = (int)(tile % tiles_x) * kLearnTile + (wid & 1) * 8 + cone::lane_x(lane, 3);
        const int y = (int)(tile / tiles_x) * kLearnTile + (int)(t & 1) * 8 + (wid >> 1) * 4 + cone::lane_y(lane, 3);
        if (x >= T.width || y >= T.height) continue;
        const long long pix = (long long)y * T.width + x;
        const float4 gp = __ldg(T.gpos + pix);
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (gp.w != 0.0f) r = irradiance16<KIND>(P, s_lv, s_cone, s_dirs, gp, __ldg(T.gnrm + pix), ns);
        P.out[pix] = make_float4(r.x, r.y, r.z, 0.0f);
    }
}

// The per-pixel fallback's list: every covered pixel whose error estimate
// exceeds threshold x the frame's root-mean-square network irradiance over
// covered pixels.  A CTA scans a 16 x 16 pixel tile, each warp an 8 x 4
// part of it, and appends the tile's flagged pixels with one atomic, in
// warp order: the list holds them in 2D clusters whose cones march through
// neighbouring voxels when the fallback traces them.
__global__ void __launch_bounds__(256) learned_flag_kernel(const LearnedParams P) {
    const int W = P.T.width, H = P.T.height, tiles_x = (W + 15) / 16;
    const int tile = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int x = (tile % tiles_x) * 16 + (warp & 1) * 8 + cone::lane_x(lane, 3);
    const int y = (tile / tiles_x) * 16 + (warp >> 1) * 4 + cone::lane_y(lane, 3);
    const long long i = (long long)y * W + x;
    const float n = P.frame_sums[1];
    const float bound = P.threshold * sqrtf(n > 0.0f ? P.frame_sums[0] / n : 0.0f);
    const bool fb = x < W && y < H && P.est[i] >= 0.0f && P.est[i] > bound;
    const unsigned m = __ballot_sync(0xffffffffu, fb);
    __shared__ uint32_t s_off[8], s_base;
    if (lane == 0) s_off[warp] = (uint32_t)__popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t tot = 0;
        for (int w = 0; w < 8; ++w) {
            const uint32_t c = s_off[w];
            s_off[w] = tot;
            tot += c;
        }
        s_base = tot ? atomicAdd(P.count, tot) : 0u;
    }
    __syncthreads();
    if (fb) P.list[s_base + s_off[warp] + __popc(m & ((1u << lane) - 1u))] = (uint32_t)i;
}

// 16-cone irradiance of the listed pixels (the per-pixel fallback), one
// thread per list entry; the grid covers the longest possible list and
// threads past the list's length return at once.  CTAs of 128: the list is
// a few CTAs to an SM, and their last ones end sooner (128^3, 1080p: 10% of the
// covered pixels 0.416 ms, 3% 0.178; CTAs of 256 0.444 and 0.205, all pixels the same).
constexpr int kListThreads = 128;  // (the cones' table takes that many)
template <int KIND>
__global__ void __launch_bounds__(kListThreads, 8) trace16_pixels_kernel(const LearnedParams P) {
    __shared__ cone::Level s_lv[VCT_MAX_LEVELS];
    __shared__ cone::ConeTable s_cone;
    __shared__ float s_dirs[16][4];
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if ((long long)blockIdx.x * blockDim.x >= (long long)*P.count) return;  // the whole CTA is past the list
    cone::fill_levels(P.T, s_lv);
    cone::fill_cone(P.T, P.ref_cone, P.T.max_distance, s_cone, 64);
    load_dirs(P, s_dirs);
    __syncthreads();
    if (i >= (long long)*P.count) return;
    const long long pix = (long long)P.list[i];
    unsigned ns = 0;
    const float4 r = irradiance16<KIND>(P, s_lv, s_cone, s_dirs, __ldg(P.T.gpos + pix), __ldg(P.T.gnrm + pix), ns);
    P.out[pix] = make_float4(r.x, r.y, r.z, 0.0f);
}

// Per-tile error estimate of the network's output: the 16-cone irradiance at
// four probe pixels of each 16x16 tile (offsets 4 and 12 on each axis) against
// the network, relative L2 over the covered probes.  Tiles above the bound
// are listed for the 16-cone fallback.  One thread per (tile, probe, cone):
// a warp holds two probes' 16 cones, two warps a tile.
constexpr int kProbeThreads = 256;  // 4 tiles per CTA

template <int KIND>
__global__ void __launch_bounds__(kProbeThreads) learned_probe_kernel(const LearnedParams P) {
    __shared__ cone::Level s_lv[VCT_MAX_LEVELS];
    __shared__ cone::ConeTable s_cone;
    __shared__ float s_dirs[16][4];
    __shared__ float s_part[kProbeThreads / 32][2];
    cone::fill_levels(P.T, s_lv);
    cone::fill_cone(P.T, P.ref_cone, P.T.max_distance, s_cone, 64);
    load_dirs(P, s_dirs);
    __syncthreads();
    const TraceParams& T = P.T;
    const int tiles_x = (T.width + kLearnTile - 1) / kLearnTile;
    const long long ntiles = (long long)tiles_x * ((T.height + kLearnTile - 1) / kLearnTile);
    const long long tile = (long long)blockIdx.x * (kProbeThreads / 64) + (threadIdx.x >> 6);
    const int pr = (threadIdx.x >> 4) & 3, c = threadIdx.x & 15;
    float4 rc = make_float4(0.f, 0.f, 0.f, 0.f);
    long long pix = -1;
    unsigned ns = 0;
    if (tile < ntiles) {
        const int x = (int)(tile % tiles_x) * kLearnTile + ((pr & 1) ? 12 : 4);
        const int y = (int)(tile / tiles_x) * kLearnTile + ((pr & 2) ? 12 : 4);
        if (x < T.width && y < T.height) {
            const long long p = (long long)y * T.width + x;
            const float4 gp = __ldg(T.gpos + p);
            if (gp.w != 0.0f) {
                pix = p;
                const float4 gn = __ldg(T.gnrm + p);
                const f3 N = cone::fnormalize(mk(gn.x, gn.y, gn.z));
                f3 Tg, Bg;
                onb(N, Tg, Bg);
                const f3 vp = volume_coord(T, gp);
                const f3 d = add(add(mul(Tg, s_dirs[c][0]), mul(Bg, s_dirs[c][1])), mul(N, s_dirs[c][2]));
                const float4 cr = cone::trace_cone<VCT_FILTER_SOFTWARE, KIND>(T, s_lv, s_cone, vp, N, d, P.ref_cone, T.max_distance, ns);
                const float w = s_dirs[c][3];
                rc = make_float4(w * cr.x, w * cr.y, w * cr.z, 0.0f);
            }
        }
    }
    // irradiance of the probe: the sum over its 16 lanes (an estimate: the
    // order differs from the 16-cone trace's sequential accumulation)
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
        rc.x += __shfl_xor_sync(0xffffffffu, rc.x, o);
        rc.y += __shfl_xor_sync(0xffffffffu, rc.y, o);
        rc.z += __shfl_xor_sync(0xffffffffu, rc.z, o);
    }
    float se = 0.0f, st = 0.0f;
    if (c == 0 && pix >= 0) {
        const float4 o = P.out[pix];
        const float dx = o.x - rc.x, dy = o.y - rc.y, dz = o.z - rc.z;
        se = dx * dx + dy * dy + dz * dz;
        st = rc.x * rc.x + rc.y * rc.y + rc.z * rc.z;
    }
    se += __shfl_xor_sync(0xffffffffu, se, 16);
    st += __shfl_xor_sync(0xffffffffu, st, 16);
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) {
        s_part[w][0] = se;
        s_part[w][1] = st;
    }
    __syncthreads();
    if ((threadIdx.x & 63) == 0 && tile < ntiles) {
        se = s_part[w][0] + s_part[w + 1][0];
        st = s_part[w][1] + s_part[w + 1][1];
        const float err = st > 0.0f ? sqrtf(se / st) : (se > 0.0f ? 1.0e30f : 0.0f);
        P.tile_err[tile] = err;
        if (err > P.threshold) P.list[atomicAdd(P.count, 1u)] = (uint32_t)tile;
    }
}

// ------------------------------------------------------- MLP inference
// A CTA holds the forward weights once in shared memory and runs kInferGroups
// independent groups of four warps; a group owns kInferTiles 128-pixel tiles
// at a time (one pixel of each per thread and per TMEM lane), 64 TMEM columns
// and an A-operand tile per tile, an mbarrier, and its own named barrier, so
// the groups' MMA chains and epilogues interleave on the SM.  Per layer the
// group's elected thread issues the K/16 MMAs of every tile (A = the tile's
// BF16 activations, B = the layer's weights) into the tiles' FP32
// accumulators and commits once to the group's mbarrier; every thread then
// loads its rows, adds the bias, applies ReLU and writes the BF16 rows back as
// the next layer's A operands.  Each wait and barrier thus serves kInferTiles
// tiles: the chain of MMA, commit, wait, barrier, TMEM load and epilogue is
// mostly latency, and one group's tiles share it.  The features of the
// group's next tiles are gathered while its first MMAs run.
constexpr int kInferGroups = 2;
constexpr int kInferTiles = 2;
constexpr int kInferThreads = 128 * kInferGroups;
constexpr int kInferTile = 128 * kMlpHidden * 2;
constexpr int kInferSmem = kImgAll + kInferGroups * kInferTiles * kInferTile;
constexpr int kInferCols = 64 * kInferTiles * kInferGroups;  // TMEM columns per CTA
constexpr int kInferBlocksPerSM = 2;                        // 2 x 88 KB of shared memory, 2 x 256 TMEM columns

template <bool ROWS>
__device__ __forceinline__ bool gather_features(const LearnedParams& P, long long idx, uint32_t (&f)[24]) {
#pragma unroll
    for (int i = 0; i < 24; ++i) f[i] = 0u;
    if (idx >= P.n) return false;
    if (ROWS) {
        const float2* r = reinterpret_cast<const float2*>(P.rows + idx * kMlpIn);
#pragma unroll
        for (int i = 0; i < kMlpIn / 2; ++i) {
            const float2 v = __ldg(r + i);
            f[i] = bf16x2(v.x, v.y);
        }
        return true;
    }
    const float4 gp = __ldg(P.T.gpos + idx);
    if (gp.w == 0.0f) return false;
    pixel_features(P, idx, gp, f);
    return true;
}

template <bool ROWS>
__global__ void __launch_bounds__(kInferThreads, kInferBlocksPerSM) mlp_infer_kernel(const LearnedParams P) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(16) float s_bias[kBiasPad];
    __shared__ __align__(8) uint64_t mbar[kInferGroups];
    __shared__ uint32_t s_tmem;
    __shared__ int s_done[kInferGroups];
    const int tid = threadIdx.x, warp = tid >> 5, grp = warp >> 2, row = tid & 127;
    for (int i = tid; i < kImgAll / 16; i += kInferThreads)
        reinterpret_cast<uint4*>(smem)[i] = __ldg(reinterpret_cast<const uint4*>(P.img) + i);
    for (int i = tid; i < kBiasPad; i += kInferThreads) s_bias[i] = P.bias[i];
    if (tid < kInferGroups) mbar_init(smem_u32(&mbar[tid]), 1);
    if (tid == 0) fence_mbar_init();
    if (warp == 0) {
        tmem_alloc(smem_u32(&s_tmem), kInferCols);
        tmem_relinquish();  // lets the SM's other CTAs allocate
    }
    fence_async_smem();
    tc_sync();
    // tile k of the group: A operand at sa[k], accumulator at TMEM columns tm[k]
    uint8_t* sa[kInferTiles];
    uint32_t tm[kInferTiles], a0[kInferTiles];
#pragma unroll
    for (int k = 0; k < kInferTiles; ++k) {
        sa[k] = smem + kImgAll + (grp * kInferTiles + k) * kInferTile;
        a0[k] = smem_u32(sa[k]);
        tm[k] = s_tmem + 64u * (uint32_t)(grp * kInferTiles + k);
    }
    const uint32_t w0 = smem_u32(smem), mb = smem_u32(&mbar[grp]);
    const int bar = 1 + grp;
    const bool leader = row == 0;
    auto group_sync = [&]() {
        fence_before_sync();
        named_sync(bar, 128);
        fence_after_sync();
    };
    const long long ntiles = (P.n + 127) / 128;
    // the group's tiles: kInferTiles consecutive ones per step
    const long long stride = (long long)gridDim.x * kInferGroups * kInferTiles;
    uint32_t phase = 0;
    int ok = 1;
    long long t = ((long long)blockIdx.x * kInferGroups + grp) * kInferTiles;
    uint32_t f[kInferTiles][24];
    bool covered[kInferTiles];
#pragma unroll
    for (int k = 0; k < kInferTiles; ++k) covered[k] = gather_features<ROWS>(P, (t + k) * 128 + row, f[k]);
    float sum_sq = 0.0f, n_cov = 0.0f;
    for (; t < ntiles && ok; t += stride) {
        bool cov[kInferTiles];
#pragma unroll
        for (int k = 0; k < kInferTiles; ++k) {
            cov[k] = covered[k];
#pragma unroll
            for (int c = 0; c < 6; ++c)
                *reinterpret_cast<uint4*>(sa[k] + tile_offset(row, 8 * c, 128)) =
                    make_uint4(f[k][4 * c], f[k][4 * c + 1], f[k][4 * c + 2], f[k][4 * c + 3]);
        }
        fence_async_smem();
        group_sync();
        float o[kInferTiles][4];
#pragma unroll 1
        for (int layer = 0; layer < 4; ++layer) {
            const int K = layer == 0 ? kMlpInPad : kMlpHidden;
            const int N = layer == 3 ? kMlpOutPad : kMlpHidden;
            const uint32_t b = w0 + (layer == 0 ? kImgW1 : layer == 1 ? kImgW2 : layer == 2 ? kImgW3 : kImgW4);
            if (leader) {
                const uint32_t id = idesc_bf16_f32(128, N);
#pragma unroll
                for (int k = 0; k < kInferTiles; ++k)
                    for (int j = 0; j < K / 16; ++j)
                        mma_bf16(tm[k], tile_desc(a0[k], 128, j), tile_desc(b, N, j), id, j > 0);
                commit(mb);
            }
            // the next tiles' features load while the first layer runs
            if (layer == 0) {
#pragma unroll
                for (int k = 0; k < kInferTiles; ++k)
                    covered[k] = gather_features<ROWS>(P, (t + stride + k) * 128 + row, f[k]);
            }
            if (leader) s_done[grp] = mbar_wait(mb, phase) ? 1 : 0;
            phase ^= 1u;
            group_sync();
            ok = s_done[grp];
            if (!ok) break;
            if (layer < 3) {
                const float4* bb = reinterpret_cast<const float4*>(s_bias + kMlpHidden * layer);
#pragma unroll
                for (int k = 0; k < kInferTiles; ++k) {
#pragma unroll
                    for (int c = 0; c < kMlpHidden; c += 32) {
                        float v[32];
                        tmem_ld32(tmem_addr(tm[k], warp, c), v);
                        uint32_t pk[16];
                        // bias in packed FP32 pairs, then ReLU and rounding in one conversion
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const float4 b4 = bb[c / 4 + i];
                            const float2 z0 = __fadd2_rn(make_float2(v[4 * i], v[4 * i + 1]), make_float2(b4.x, b4.y));
                            const float2 z1 = __fadd2_rn(make_float2(v[4 * i + 2], v[4 * i + 3]), make_float2(b4.z, b4.w));
                            pk[2 * i] = bf16x2_relu(z0.x, z0.y);
                            pk[2 * i + 1] = bf16x2_relu(z1.x, z1.y);
                        }
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            *reinterpret_cast<uint4*>(sa[k] + tile_offset(row, c + 8 * q, 128)) =
                                make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
                    }
                }
                fence_async_smem();
                group_sync();
            } else {
#pragma unroll
                for (int k = 0; k < kInferTiles; ++k) {
                    float v[16];
                    tmem_ld16(tmem_addr(tm[k], warp, 0), v);
#pragma unroll
                    for (int q = 0; q < 4; ++q) o[k][q] = v[q] + s_bias[3 * kMlpHidden + q];
                }
            }
        }
        if (!ok) break;
#pragma unroll
        for (int k = 0; k < kInferTiles; ++k) {
            const long long idx = (t + k) * 128 + row;
            if (idx >= P.n) continue;
            if (ROWS) {
                *reinterpret_cast<float4*>(P.out_rows + idx * 4) = make_float4(o[k][0], o[k][1], o[k][2], o[k][3]);
            } else {
                P.out[idx] = cov[k] ? make_float4(o[k][0], o[k][1], o[k][2], 0.0f) : make_float4(0.f, 0.f, 0.f, 0.f);
                if (P.est) {
                    // the per-pixel fallback's inputs: the error estimate (-1 for
                    // background) and the frame's sum of squared irradiance
                    P.est[idx] = cov[k] ? o[k][3] : -1.0f;
                    if (cov[k]) {
                        sum_sq += o[k][0] * o[k][0] + o[k][1] * o[k][1] + o[k][2] * o[k][2];
                        n_cov += 1.0f;
                    }
                }
            }
        }
    }
    if (P.est) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sum_sq += __shfl_xor_sync(0xffffffffu, sum_sq, o);
            n_cov += __shfl_xor_sync(0xffffffffu, n_cov, o);
        }
        if ((tid & 31) == 0 && n_cov > 0.0f) {
            atomicAdd(P.frame_sums, sum_sq);
            atomicAdd(P.frame_sums + 1, n_cov);
        }
    }
    if (!ok && leader) atomicOr(P.status, 1u);
    tc_sync();
    if (warp == 0) tmem_dealloc(s_tmem, kInferCols);
}

// ------------------------------------------------------- MLP training
// A CTA of eight warps takes tiles of 128 samples: a thread a sample (a TMEM
// lane) and half of a layer's columns.  Forward as in inference, keeping each
// hidden layer's ReLU mask in registers and its BF16 activations in shared
// memory.  Backward, per layer l:
//   dZ_l = (dZ_{l+1} W_{l+1}) * mask_l           (MMA into the 64 scratch columns)
//   dW_l^T += H_{l-1}^T dZ_l                     (MMA, accumulated in TMEM over the CTA's tiles)
// Every operand is stored once, samples x features, and the weight-gradient
// MMAs read H and dZ transposed (as the backward ones read W).  A column of
// ones after an activation tile's features makes the same MMA accumulate the
// bias gradient; M = 128 rows also reads what follows the tile, into rows of
// the accumulator that nothing uses.  A layer's weight gradient is issued
// after the MMAs that the next layer waits for and runs beside its epilogue.
// At the end each CTA stores its TMEM gradients as its part, which the update
// kernel sums.
//
// What bounds it: the chain of eight MMAs, waits and epilogues that a tile is,
// and the launch.  A step of 16,384 rows takes 15 us with its update (a tile to
// a CTA; 10 us of them this kernel).  With 128 threads a CTA, transposed copies
// of every operand stored in 2-byte pieces over zeroed tiles, and atomics from
// 128 CTAs into one gradient (6 us of contention) it took 30 us, and 45 with the
// two memsets, the update and a copy of the loss.
// Loss: mean squared error over the
// n x 3 irradiance outputs, plus kMlpConfidenceWeight times the mean over the
// n samples of (e - |y - t|)^2, where e is the fourth output (the error
// estimate) and |y - t| the Euclidean error of the sample's irradiance, held
// constant (no gradient flows from this term into the irradiance outputs).
constexpr int kTrThreads = 256;
constexpr int kTrX = kImgAll;                      // input tile: 48 features, the ones' chunk
constexpr int kTrH = kTrX + 7 * 128 * 16;          // three activation tiles: 64 features, the ones' chunk
constexpr int kTrHTile = 9 * 128 * 16;
constexpr int kTrDZ = kTrH + 3 * kTrHTile;         // three dZ tiles, 128 x 64
constexpr int kTrDZTile = 128 * 64 * 2;
constexpr int kTrDY = kTrDZ + 3 * kTrDZTile;       // 128 x 16
constexpr int kTrSmem = kTrDY + 128 * 16 * 2;
static_assert(kTrSmem <= 227 * 1024 - 2048, "training tiles exceed shared memory");
// an M = 128 operand at the last activation tile reads 16 chunks
static_assert(kTrH + 2 * kTrHTile + 16 * 128 * 16 <= kTrSmem, "transposed operand exceeds shared memory");
// TMEM columns: scratch, dW1^T, dW2^T, dW3^T, dW4^T.
constexpr uint32_t kColFb = 0, kColW1 = 64, kColW2 = 128, kColW3 = 192, kColW4 = 256;
constexpr uint32_t kBf16One = 0x3F80u;

__global__ void __launch_bounds__(kTrThreads, 1) mlp_train_kernel(const TrainParams P) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(16) float s_bias[kBiasPad];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t s_tmem;
    __shared__ float s_loss[4], s_closs[4];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = tid & 127, half = tid >> 7;
    uint8_t* const xt = smem + kTrX;
    uint8_t* const dy = smem + kTrDY;
    // columns of ones: bias gradients
    const uint4 ones = make_uint4(kBf16One, 0u, 0u, 0u);
    if (half == 0) {
        *reinterpret_cast<uint4*>(xt + tile_offset(row, kMlpInPad, 128)) = ones;
        *reinterpret_cast<uint4*>(dy + tile_offset(row, 8, 128)) = make_uint4(0u, 0u, 0u, 0u);
    } else {
        for (int l = 0; l < 3; ++l)
            *reinterpret_cast<uint4*>(smem + kTrH + l * kTrHTile + tile_offset(row, kMlpHidden, 128)) = ones;
    }
    if (tid == 0) {
        mbar_init(smem_u32(&mbar), 1);
        fence_mbar_init();
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&s_tmem), 512);
        tmem_relinquish();
    }
    const uint32_t w0 = smem_u32(smem);
    grid_wait();  // nothing above reads what a kernel before this one writes
    for (int i = tid; i < kImgAll / 16; i += kTrThreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(w0 + 16u * (uint32_t)i),
                     "l"(P.mlp.img + 16 * (long long)i)
                     : "memory");
    const float bias = tid < kBiasPad ? __ldca(P.mlp.bias + tid) : 0.0f;  // stored with the first tile's input
    tc_sync();
    const uint32_t tm = s_tmem, mb = smem_u32(&mbar);
    const uint32_t x0 = w0 + kTrX, h0 = w0 + kTrH, dz0 = w0 + kTrDZ, dy0 = w0 + kTrDY;
    const uint32_t id64 = idesc_bf16_f32(128, 64), id16 = idesc_bf16_f32(128, 16);
    const long long ntiles = (P.n + 127) / 128;
    uint32_t phase = 0;
    int ok = 1;
    bool first = true;
    float loss = 0.0f, closs = 0.0f;

    // Waits for the MMAs committed by thread 0.  Every thread does, and after a
    // wait that gave up goes on without waiting (the barriers stay matched;
    // what it computes is not used).
    auto wait_mma = [&]() {
        if (ok) ok = mbar_wait(mb, phase) ? 1 : 0;
        phase ^= 1u;
        fence_after_sync();
    };

    for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const long long idx = t * 128 + row;
        const bool valid = idx < P.n;
        const long long src = valid ? (P.index ? (long long)__ldca(P.index + idx) : idx) : 0;
        // ---- input: 24 of the 48 features each
        float target[3] = {0.f, 0.f, 0.f};
        {
            uint32_t f[12];
            const float2* rp = reinterpret_cast<const float2*>(P.rows + src * kMlpIn) + 12 * half;
#pragma unroll
            for (int i = 0; i < 12; ++i) {
                f[i] = 0u;
                if (valid && (i < kMlpIn / 2 - 12 || half == 0)) {
                    const float2 v = __ldca(rp + i);  // (ordinary loads: they stay behind grid_wait)
                    f[i] = bf16x2(v.x, v.y);
                }
            }
            if (valid && half == 0) {
#pragma unroll
                for (int o = 0; o < 3; ++o) target[o] = __ldca(P.targets + src * 3 + o);
            }
#pragma unroll
            for (int c = 0; c < 3; ++c)
                *reinterpret_cast<uint4*>(xt + tile_offset(row, 24 * half + 8 * c, 128)) =
                    make_uint4(f[4 * c], f[4 * c + 1], f[4 * c + 2], f[4 * c + 3]);
        }
        if (first) {
            if (tid < kBiasPad) s_bias[tid] = bias;
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        fence_async_smem();
        tc_sync();
        // ---- forward, hidden layers
        uint32_t mask[3] = {0, 0, 0};
#pragma unroll
        for (int layer = 0; layer < 3; ++layer) {
            if (tid == 0) {
                const uint32_t a = layer == 0 ? x0 : h0 + (layer - 1) * kTrHTile;
                const uint32_t b = w0 + (layer == 0 ? kImgW1 : layer == 1 ? kImgW2 : kImgW3);
                for (int j = 0; j < (layer == 0 ? kMlpInPad : kMlpHidden) / 16; ++j)
                    mma_bf16(tm + kColFb, tile_desc(a, 128, j), tile_desc(b, 64, j), id64, j > 0);
                commit(mb);
            }
            wait_mma();
            const float* bb = s_bias + kMlpHidden * layer + 32 * half;
            uint8_t* h = smem + kTrH + layer * kTrHTile;
            float v[32];
            tmem_ld32(tmem_addr(tm + kColFb, warp, 32 * half), v);
            uint32_t m = 0;
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                v[i] = fmaxf(v[i] + bb[i], 0.0f);
                if (v[i] > 0.0f) m |= 1u << i;
            }
            mask[layer] = m;
#pragma unroll
            for (int c = 0; c < 4; ++c)
                *reinterpret_cast<uint4*>(h + tile_offset(row, 32 * half + 8 * c, 128)) =
                    make_uint4(bf16x2(v[8 * c], v[8 * c + 1]), bf16x2(v[8 * c + 2], v[8 * c + 3]),
                               bf16x2(v[8 * c + 4], v[8 * c + 5]), bf16x2(v[8 * c + 6], v[8 * c + 7]));
            fence_async_smem();
            tc_sync();
        }
        // ---- output layer, loss and dY
        if (tid == 0) {
            for (int j = 0; j < 4; ++j)
                mma_bf16(tm + kColFb, tile_desc(h0 + 2 * kTrHTile, 128, j), tile_desc(w0 + kImgW4, 16, j), id16, j > 0);
            commit(mb);
        }
        wait_mma();
        if (half == 0) {
            float v[16];
            tmem_ld16(tmem_addr(tm + kColFb, warp, 0), v);
            float d[4] = {0.f, 0.f, 0.f, 0.f};
            if (valid) {
                float e2 = 0.0f;
#pragma unroll
                for (int o = 0; o < 3; ++o) {
                    const float diff = (v[o] + s_bias[3 * kMlpHidden + o]) - target[o];
                    loss += diff * diff;
                    e2 += diff * diff;
                    d[o] = P.scale * diff;
                }
                // the error estimate's target |output - target| is a constant of the step
                const float dc = (v[3] + s_bias[3 * kMlpHidden + 3]) - sqrtf(e2);
                closs += dc * dc;
                d[3] = P.conf_scale * dc;
            }
            *reinterpret_cast<uint4*>(dy + tile_offset(row, 0, 128)) =
                make_uint4(bf16x2(d[0], d[1]), bf16x2(d[2], d[3]), 0u, 0u);
        }
        fence_async_smem();
        tc_sync();
        // ---- backward: dH3 = dY W4; dW4^T += H3^T dY
        if (tid == 0) {
            mma_bf16(tm + kColFb, tile_desc(dy0, 128, 0), tile_desc_t(w0 + kImgW4, 16, 0), id64 | kTransB, 0u);
            commit(mb);
            for (int j = 0; j < 8; ++j)
                mma_bf16(tm + kColW4, tile_desc_t(h0 + 2 * kTrHTile, 128, j), tile_desc_t(dy0, 128, j),
                         id16 | kTransA | kTransB, (!first || j > 0) ? 1u : 0u);
        }
        wait_mma();
#pragma unroll
        for (int layer = 2; layer >= 0; --layer) {
            // dZ_layer = dH * mask
            const uint32_t dz = dz0 + layer * kTrDZTile;
            {
                float v[32];
                tmem_ld32(tmem_addr(tm + kColFb, warp, 32 * half), v);
#pragma unroll
                for (int i = 0; i < 32; ++i) v[i] = (mask[layer] >> i) & 1u ? v[i] : 0.0f;
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    *reinterpret_cast<uint4*>(smem + kTrDZ + layer * kTrDZTile + tile_offset(row, 32 * half + 8 * c, 128)) =
                        make_uint4(bf16x2(v[8 * c], v[8 * c + 1]), bf16x2(v[8 * c + 2], v[8 * c + 3]),
                                   bf16x2(v[8 * c + 4], v[8 * c + 5]), bf16x2(v[8 * c + 6], v[8 * c + 7]));
            }
            fence_async_smem();
            tc_sync();
            if (tid == 0) {
                if (layer > 0) {
                    // dH_{layer-1} = dZ_layer W_layer
                    const uint32_t w = w0 + (layer == 2 ? kImgW3 : kImgW2);
                    for (int j = 0; j < 4; ++j)
                        mma_bf16(tm + kColFb, tile_desc(dz, 128, j), tile_desc_t(w, 64, j), id64 | kTransB, j > 0);
                    commit(mb);
                }
                // dW_layer^T += H_{layer-1}^T dZ_layer   (H_{-1} = X)
                const uint32_t h = layer == 0 ? x0 : h0 + (layer - 1) * kTrHTile;
                const uint32_t col = layer == 0 ? kColW1 : layer == 1 ? kColW2 : kColW3;
                for (int j = 0; j < 8; ++j)
                    mma_bf16(tm + col, tile_desc_t(h, 128, j), tile_desc_t(dz, 128, j), id64 | kTransA | kTransB,
                             (!first || j > 0) ? 1u : 0u);
                // the tile's last MMAs: nothing of it is read after them
                if (layer == 0) commit(mb);
            }
            wait_mma();
        }
        first = false;
    }
    // The update may start; it waits for this kernel's end before it reads anything.
    grid_launch_dependents();
    ok = __syncthreads_and(ok);
    // ---- gradients out: this CTA's part (zeros after a wait that gave up)
    float* const part = P.mlp.parts + (long long)blockIdx.x * kPartStride;
    {
        const int r = row;  // TMEM lane = row of dW^T = input feature (or the bias row)
#pragma unroll 1
        for (int layer = 0; layer < 4; ++layer) {
            const int in = layer == 0 ? kMlpIn : kMlpHidden;
            const int bias_row = layer == 0 ? kMlpInPad : kMlpHidden;
            const uint32_t col = layer == 0 ? kColW1 : layer == 1 ? kColW2 : layer == 2 ? kColW3 : kColW4;
            const int offw = layer == 0 ? kOffW1 : layer == 1 ? kOffW2 : layer == 2 ? kOffW3 : kOffW4;
            const int offb = layer == 0 ? kOffB1 : layer == 1 ? kOffB2 : layer == 2 ? kOffB3 : kOffB4;
            const int nout = layer == 3 ? (half == 0 ? kMlpOut : 0) : 32;
            float v[32];
            tmem_ld32(tmem_addr(tm + col, warp, layer == 3 ? 0 : 32 * half), v);
            float* p = r < in ? part + offw + r + 32 * half * in : part + offb + 32 * half;
            const int stride = r < in ? in : 1;
            if (r < in || r == bias_row) {
#pragma unroll
                for (int i = 0; i < 32; ++i)
                    if (i < nout) p[i * stride] = ok ? v[i] : 0.0f;
            }
        }
    }
    // ---- loss
    for (int o = 16; o > 0; o >>= 1) {
        loss += __shfl_xor_sync(0xffffffffu, loss, o);
        closs += __shfl_xor_sync(0xffffffffu, closs, o);
    }
    if (lane == 0 && half == 0) {
        s_loss[warp] = loss;
        s_closs[warp] = closs;
    }
    if (!ok && tid == 0) atomicOr(P.status, 1u);
    tc_sync();
    if (tid == 0)
        part[kMlpParams] = (s_loss[0] + s_loss[1] + s_loss[2] + s_loss[3]) * (0.5f * P.scale) +
                           (s_closs[0] + s_closs[1] + s_closs[2] + s_closs[3]) * (0.5f * P.conf_scale);
    if (warp == 0) tmem_dealloc(tm, 512);
}

// ------------------------------------------------------- optimiser
// The sum of the parts' gradients (eight threads a parameter, an eighth of the
// parts each), Adam on the fp32 master parameters, then the BF16 operand
// images and the padded bias vector the kernels read.
constexpr int kUpdateThreads = 512, kUpdateSlices = 8, kUpdateParams = kUpdateThreads / kUpdateSlices;

__global__ void __launch_bounds__(kUpdateThreads) mlp_update_kernel(const MlpDev M, int what, int nparts, float lr,
                                                                    float beta1, float beta2, float eps, float c1,
                                                                    float c2, float* loss_out) {
    __shared__ float s_sum[kUpdateSlices][kUpdateParams];
    const int slice = threadIdx.x / kUpdateParams, k = threadIdx.x % kUpdateParams;
    const int i = blockIdx.x * kUpdateParams + k;
    float w = 0.0f, m = 0.0f, v = 0.0f;
    const bool mine = slice == 0 && i < kMlpParams;
    grid_wait();
    grid_launch_dependents();
    if (mine && what == kUpdateAdam) {  // (in flight with the parts)
        w = M.params[i];
        m = M.m[i];
        v = M.v[i];
    }
    if (what != kUpdateImages) {
        float g = 0.0f;
        if (i < kMlpParams) {
#pragma unroll 16
            for (int p = slice; p < nparts; p += kUpdateSlices) g += __ldcg(M.parts + (long long)p * kPartStride + i);
        }
        s_sum[slice][k] = g;
        if (blockIdx.x == 0 && threadIdx.x < 32) {
            float l = 0.0f;
            for (int p = threadIdx.x; p < nparts; p += 32) l += __ldcg(M.parts + (long long)p * kPartStride + kMlpParams);
            for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            if (threadIdx.x == 0) {
                *M.loss = l;
                if (loss_out) *loss_out = l;
            }
        }
        __syncthreads();
    }
    if (!mine) return;
    if (what == kUpdateImages) {
        w = M.params[i];
    } else {
        const float g = ((s_sum[0][k] + s_sum[1][k]) + (s_sum[2][k] + s_sum[3][k])) +
                        ((s_sum[4][k] + s_sum[5][k]) + (s_sum[6][k] + s_sum[7][k]));
        if (what == kUpdateGradient) {
            M.grad[i] = g;
            return;
        }
        m = beta1 * m + (1.0f - beta1) * g;
        v = beta2 * v + (1.0f - beta2) * g * g;
        M.m[i] = m;
        M.v[i] = v;
        w = w - lr * (m * c1) / (sqrtf(v * c2) + eps);
        M.params[i] = w;
    }
    const uint16_t h = bf16(w);
    uint8_t* img = M.img;
    if (i < kOffB1) {
        const int o = i / kMlpIn, f = i % kMlpIn;
        *reinterpret_cast<uint16_t*>(img + kImgW1 + tile_offset(o, f, 64)) = h;
    } else if (i < kOffW2) {
        M.bias[i - kOffB1] = w;
    } else if (i < kOffB2) {
        const int o = (i - kOffW2) / kMlpHidden, f = (i - kOffW2) % kMlpHidden;
        *reinterpret_cast<uint16_t*>(img + kImgW2 + tile_offset(o, f, 64)) = h;
    } else if (i < kOffW3) {
        M.bias[kMlpHidden + i - kOffB2] = w;
    } else if (i < kOffB3) {
        const int o = (i - kOffW3) / kMlpHidden, f = (i - kOffW3) % kMlpHidden;
        *reinterpret_cast<uint16_t*>(img + kImgW3 + tile_offset(o, f, 64)) = h;
    } else if (i < kOffW4) {
        M.bias[2 * kMlpHidden + i - kOffB3] = w;
    } else if (i < kOffB4) {
        const int o = (i - kOffW4) / kMlpHidden, f = (i - kOffW4) % kMlpHidden;
        *reinterpret_cast<uint16_t*>(img + kImgW4 + tile_offset(o, f, 16)) = h;
    } else {
        M.bias[3 * kMlpHidden + i - kOffB4] = w;
    }
}

}  // namespace

// The timeout path of the bounded waits: one thread waits on an mbarrier that
// nothing arrives on, gives up after `limit_ns` and records it in `status`,
// exactly as the MLP kernels do when an MMA never completes.
__global__ void wait_probe_kernel(uint32_t* status, unsigned long long limit_ns) {
    __shared__ __align__(8) uint64_t mbar;
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&mbar), 1);
        fence_mbar_init();
        if (!mbar_wait_for(smem_u32(&mbar), 0u, limit_ns)) atomicOr(status, 1u);
    }
}

void launch_wait_probe(uint32_t* status, unsigned long long limit_ns, cudaStream_t s) {
    wait_probe_kernel<<<1, 32, 0, s>>>(status, limit_ns);
    note_launches(1);
}

void launch_umma_check(const uint16_t* A, const uint16_t* B, int K, int N, int swap, float* D, uint32_t* status,
                       cudaStream_t s) {
    cudaFuncSetAttribute(umma_check_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCheckSmemA + kCheckSmemB);
    umma_check_kernel<<<1, 128, kCheckSmemA + kCheckSmemB, s>>>(A, B, K, N, swap, D, status);
    note_launches(1);
}

void launch_learned_features(const LearnedParams& P, cudaStream_t s) {
    const dim3 grid((P.wq + 15) / 16, (P.hq + 15) / 16);
    learned_features_kernel<<<grid, 256, 0, s>>>(P);
    note_launches(1);
}

void launch_learned_rows(const LearnedParams& P, cudaStream_t s) {
    if (P.n <= 0) return;
    learned_rows_kernel<<<(unsigned)((P.n + 255) / 256), 256, 0, s>>>(P);
    note_launches(1);
}

void launch_mlp_infer(const LearnedParams& P, int num_sms, cudaStream_t s) {
    if (P.n <= 0) return;
    const long long tiles = (P.n + 127) / 128;
    // kInferBlocksPerSM resident CTAs per SM, each taking kInferGroups x kInferTiles tiles a step.
    const long long per_cta = (long long)kInferGroups * kInferTiles;
    const long long slots = (long long)num_sms * kInferBlocksPerSM * per_cta;
    const long long grid = (tiles < slots ? tiles + per_cta - 1 : slots) / per_cta;
    if (P.rows) {
        cudaFuncSetAttribute(mlp_infer_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kInferSmem);
        mlp_infer_kernel<true><<<(unsigned)grid, kInferThreads, kInferSmem, s>>>(P);
    } else {
        cudaFuncSetAttribute(mlp_infer_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kInferSmem);
        mlp_infer_kernel<false><<<(unsigned)grid, kInferThreads, kInferSmem, s>>>(P);
    }
    note_launches(1);
}

// f(integral constant) with the kind of the 16 cones' march.
template <class F>
static void with_kind(const LearnedParams& P, F f) {
    const int kind = cone_kind(P.T.warp, P.ref_cone.steps);
    if (kind == kConesPlain)
        f(std::integral_constant<int, kConesPlain>());
    else if (kind == kConesMapped)
        f(std::integral_constant<int, kConesMapped>());
    else
        f(std::integral_constant<int, kConesAny>());
}

void launch_learned_probe(const LearnedParams& P, cudaStream_t s) {
    const long long tiles = (long long)((P.T.width + kLearnTile - 1) / kLearnTile) *
                            ((P.T.height + kLearnTile - 1) / kLearnTile);
    const unsigned grid = (unsigned)((tiles + kProbeThreads / 64 - 1) / (kProbeThreads / 64));
    with_kind(P, [&](auto kind) { learned_probe_kernel<kind.value><<<grid, kProbeThreads, 0, s>>>(P); });
    note_launches(1);
}

void launch_trace16(const LearnedParams& P, bool listed, int num_sms, cudaStream_t s) {
    const long long tiles = (long long)((P.T.width + kLearnTile - 1) / kLearnTile) *
                            ((P.T.height + kLearnTile - 1) / kLearnTile);
    // Over all tiles a CTA to each half; over the listed ones, whose number is known
    // on the device, as many, or six times the CTAs that fit, which take halves in turn
    // (twice: 128^3, 1080p 1.76 ms, 1.74; a 256^3 scene of many small tiles 1.27, 1.17).
    with_kind(P, [&](auto kind) {
        if (listed)
            trace16_kernel<kind.value, true><<<(unsigned)std::min(num_sms * 48LL, 2 * tiles), kTile16Threads, 0, s>>>(P);
        else
            trace16_kernel<kind.value, false><<<(unsigned)(2 * tiles), kTile16Threads, 0, s>>>(P);
    });
    note_launches(1);
}

void launch_trace16_pixels(const LearnedParams& P, cudaStream_t s) {
    const long long n = (long long)P.T.width * P.T.height;
    const long long tiles = (long long)((P.T.width + 15) / 16) * ((P.T.height + 15) / 16);  // one CTA each
    learned_flag_kernel<<<(unsigned)tiles, 256, 0, s>>>(P);
    with_kind(P, [&](auto kind) {
        trace16_pixels_kernel<kind.value><<<(unsigned)((n + kListThreads - 1) / kListThreads), kListThreads, 0, s>>>(P);
    });
    note_launches(2);
}

int launch_mlp_train(const TrainParams& P, int num_sms, cudaStream_t s) {
    const long long tiles = (P.n + 127) / 128;
    const int grid = (int)(tiles < num_sms ? tiles : num_sms);
    cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrSmem);
    launch_overlapped(mlp_train_kernel, dim3((unsigned)grid), kTrThreads, kTrSmem, s, P);
    return grid;
}

void launch_mlp_update(const MlpDev& M, int what, int nparts, int step, float lr, float beta1, float beta2, float eps,
                       float* loss_out, cudaStream_t s) {
    const bool adam = what == kUpdateAdam;
    const double c1 = adam ? 1.0 / (1.0 - std::pow((double)beta1, (double)step)) : 1.0;
    const double c2 = adam ? 1.0 / (1.0 - std::pow((double)beta2, (double)step)) : 1.0;
    launch_overlapped(mlp_update_kernel, dim3((kMlpParams + kUpdateParams - 1) / kUpdateParams), kUpdateThreads, 0, s, M, what,
                      nparts, lr, beta1, beta2, eps, (float)c1, (float)c2, loss_out);
}

}  // namespace vct
