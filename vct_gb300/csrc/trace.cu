// Voxel cone tracing: shaders/phong.frag:135-180 (traceCone) and the
// indirect / specular / composite code of phong.frag:455-520.
//
// One thread per pixel; a 256-thread CTA shades a pixel tile (16x16 by
// default; the shape is a tuning setting) and each warp a sub-tile (8x4 by
// default), so the 32 lanes of a warp march neighbouring cones through
// neighbouring voxels at the same time (the cone step sequence depends only on
// the cone parameters, so every lane is at the same mip level each step).
// A lane leaves its cone at alpha >= 0.95 or on leaving the volume; the warp
// moves to the next cone once all lanes are done.
//
// Two samplers implement textureLod (cone.cuh): the software fp32 trilinear
// over a bordered fp32 copy of the chain (exact GL arithmetic), and the
// texture units (tex3DLod on a mip-mapped CUDA array, with their fixed-point
// filter weights).
//
// The file is compiled without FMA contraction: every fused multiply-add is
// written out (fmaf, __ffma2_rn; but for the warp map's lookup, see cone.cuh), so
// the single-scene and the batched instantiations of the kernel give bit-identical
// results.
#include <algorithm>

#include "trace.cuh"

namespace vct {

namespace {

// Bound by the L1 data pipe: a warp's 16-byte texel load takes four passes or
// more (5 on average), and the pipe is busy 78% of the time; the loads mostly
// hit L1 (96%), and instructions issue at 58% of peak.  Four resident CTAs
// per SM (64 registers) hide the loads' latency.  Distances, levels and level
// strides come from tables in shared memory, floors from additions, and a
// quarter warp's lanes are a 4 x 2 block of pixels: on a 256^3, 1920 x 1080
// frame the hybrid sampler's kernel takes 389 us (442 us without these), the
// software sampler's 565 us (602).
template <int MODE, int KIND, class Scenes>
__global__ void __launch_bounds__(256, 4) trace_kernel(const Scenes S) {
    // One CTA per tile (tiles of every scene of the launch in a row), one warp
    // per sub-tile.
    long long tile;
    const TraceParams& P = S.get(S.find(blockIdx.x, tile));
    int x, y;
    tile_pixel(P, tile, threadIdx.x >> 5, threadIdx.x & 31, x, y);
    __shared__ Level s_lv[VCT_MAX_LEVELS];
    __shared__ ConeTable s_cone[2];  // the diffuse and the specular cones' steps
    fill_levels(P, s_lv);
    fill_cone(P, P.diffuse, P.max_distance, s_cone[0], 64);
    fill_cone(P, P.specular_cone, P.max_distance, s_cone[1], 128);
    grid_wait();  // (the chain's addresses come from the tables behind the barrier)
    __syncthreads();
    unsigned ns = 0;
    if (x < P.width && y < P.height) {
        const long long pix = (long long)y * P.width + x;
        float4 irr = make_float4(0.f, 0.f, 0.f, 0.f), spc = irr, out = irr;
        const float4 gp = __ldg(P.gpos + pix);
        if (gp.w != 0.0f) {
            if (P.enable_indirect) {
                const float4 gn = __ldg(P.gnrm + pix);
                const f3 N = fnormalize(mk(gn.x, gn.y, gn.z));
                const f3 vp = volume_position(P, gp);
                f3 T, B;
                tangents(N, T, B);
#pragma unroll 1
                for (int c = 0; c < 6; ++c) {
                    const float4 cr = trace_cone<MODE, KIND>(P, s_lv, s_cone[0], vp, N, diffuse_direction(P, c, N, T, B),
                                                             P.diffuse, P.max_distance, ns);
                    irr = add_cone(irr, kConeWeight[c], cr);
                }
                // (the position is read again rather than kept live across the diffuse cones)
                if (P.enable_reflections)
                    spc = trace_cone<MODE, KIND>(P, s_lv, s_cone[1], vp, N, reflected(P, __ldg(P.gpos + pix), N),
                                                 P.specular_cone, P.max_distance, ns);
            }
            out = composite(P, pix, irr, spc);
        }
        store_pixel(P, pix, irr, spc, out);
    }
    count_samples(P, ns);
}

// Peak rate of textureLod samples (the denominator of the cone tracer's
// roofline): every thread takes `iters` samples with the tracer's sampler at
// positions inside one 8-voxel-wide region near the volume's centre, at the
// levels and fractions cone steps use, so the texels stay in L1 and nothing
// but sampling is timed.  The sum goes to `sink` so the work is kept.
template <int MODE>
__global__ void __launch_bounds__(256, 4) sampler_rate_kernel(const TraceParams P, int iters, float* sink) {
    __shared__ Level s_lv[VCT_MAX_LEVELS];
    fill_levels(P, s_lv);
    __syncthreads();
    const bool guard = P.warp.mode != VCT_WARP_NONE;
    const float span = 8.0f / (float)P.dim;
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    f3 p = mk(0.5f + span * (float)(t & 7) * 0.125f, 0.5f + span * (float)((t >> 3) & 7) * 0.125f,
              0.5f + span * (float)((t >> 6) & 7) * 0.125f);
    const f3 step = mk(span * 0.031f, span * 0.017f, span * 0.023f);
    const float top = (float)(P.levels - 1);
    float acc = 0.0f;
    for (int i = 0; i < iters; ++i) {
        const float lambda = fminf(0.1f + 0.37f * (float)(i & 7), top - 0.05f);
        const float4 v = to_float4(sample_lod<MODE>(P, s_lv, p, choose_lod(0.0f, lambda, P.levels - 1), guard));
        acc += v.x + v.y + v.z + v.w;
        p = add(p, step);
        if (p.x > 0.5f + span) p.x -= span;
        if (p.y > 0.5f + span) p.y -= span;
        if (p.z > 0.5f + span) p.z -= span;
    }
    sink[t] = acc;
}

}  // namespace

void launch_sampler_rate(const TraceParams& P, int filter, int blocks, int iters, float* sink, cudaStream_t s) {
    if (filter == VCT_FILTER_HARDWARE)
        sampler_rate_kernel<VCT_FILTER_HARDWARE><<<blocks, 256, 0, s>>>(P, iters, sink);
    else if (filter == VCT_FILTER_HARDWARE_LEVELS)
        sampler_rate_kernel<VCT_FILTER_HARDWARE_LEVELS><<<blocks, 256, 0, s>>>(P, iters, sink);
    else if (filter == VCT_FILTER_HYBRID)
        sampler_rate_kernel<VCT_FILTER_HYBRID><<<blocks, 256, 0, s>>>(P, iters, sink);
    else
        sampler_rate_kernel<VCT_FILTER_SOFTWARE><<<blocks, 256, 0, s>>>(P, iters, sink);
    note_launches(1);
}

namespace {

// Tiles per SM up to which a launch takes the split kernel: two rounds of the
// CTAs that an SM holds, fewer where a sample takes less time, so that the shorter
// chain gains less, and where the march checks every footprint.  The plain texture
// sampler's unsplit kernel holds five CTAs to an SM, which ends badly on few
// rounds: it splits up to 16.  Unsplit and split (us):
//   software, 64^3: 1,200 tiles 173 and 139, 1,450 166 and 127, 2,040 174 and 174;
//   hybrid, 256^3: 1,200 tiles 138 and 130, 1,450 110 and 121, 2,040 153 and 160;
//     any warp, 32^3: 1,040 tiles 73 and 70, 1,200 76 and 83;
//   texture by level, 32^3: 920 tiles 36 and 37, 1,200 43 and 52, 128^3 74 and 76;
//     any warp: 756 tiles 41 and 40, 128^3 56 and 51, 1,040 45 and 52, 60 and 68;
//   texture, 128^3: 1,250 tiles 69 and 50, 2,432 102 and 92, 3,600 124 and 134;
//     warp map, 32^3: 1,040 tiles 67 and 63, 1,200 68 and 76;
//     any warp, 32^3: 756 tiles 37 and 39, 128^3 51 and 49, 1,200 48 and 60, 73 and 80.
int split_tiles_per_sm(int filter, int kind) {
    if (filter == VCT_FILTER_SOFTWARE) return 8;
    if (filter == VCT_FILTER_HYBRID) return kind == kConesAny ? 7 : 8;
    if (filter == VCT_FILTER_HARDWARE && kind == kConesPlain) return 16;
    return kind == kConesAny ? 6 : 7;
}

template <class Scenes>
void launch_trace_set(const Scenes& S, int filter, int kind, long long tiles, int num_sms, bool overlap, cudaStream_t s) {
    if (tiles <= 0) return;
    if (tiles <= (long long)split_tiles_per_sm(filter, kind) * num_sms) {
        launch_trace_split(S, filter, kind, tiles, num_sms, overlap, s);
        return;
    }
    with_trace_mode(filter, kind, [&](auto mode, auto cones) {
        launch_tiles(trace_kernel<mode.value, cones.value, Scenes>, S, tiles, overlap, s);
    });
}

}  // namespace

int trace_kind(const TraceParams& P) {
    return cone_kind(P.warp, std::max(P.diffuse.steps, P.specular_cone.steps));
}

long long trace_tiles(int width, int height, int tile_w_log2, int tile_h_log2) {
    const long long tw = 1LL << tile_w_log2, th = 1LL << tile_h_log2;
    return ((width + tw - 1) / tw) * ((height + th - 1) / th);
}

void launch_trace(const TraceParams& P, bool overlap, cudaStream_t s) {
    launch_trace_set(OneScene<TraceParams>{P}, P.filter, trace_kind(P), trace_tiles(P.width, P.height, P.tile_w_log2, P.tile_h_log2),
                     P.num_sms, overlap, s);
}

void launch_trace_batch(const SceneBatch<TraceParams>& B, int filter, int kind, long long tiles, int num_sms,
                        cudaStream_t s) {
    launch_trace_set(ManyScenes<TraceParams>{B}, filter, kind, tiles, num_sms, false, s);
}

void launch_trace_views(const ViewSet& V, int filter, cudaStream_t s) {
    int kind = trace_kind(V.p[0]);
    for (int k = 1; k < V.n; ++k) kind = cone_kind_of(kind, trace_kind(V.p[k]));
    launch_trace_set(FewScenes{V}, filter, kind, V.off[V.n], V.p[0].num_sms, false, s);
}

}  // namespace vct
