// The cone tracer's kernel for launches of few pixels (see trace.cu, which
// chooses).  Compiled without FMA contraction, as trace.cu.
#include "trace.cuh"

namespace vct {

namespace {

// A launch of few pixels: four warps to 32 pixels instead of one, three of
// them with two diffuse cones each, the fourth with the specular one, which
// shortens the chain of samples that the launch waits for from all seven
// cones' to the specular one's.  The results are the same bits: the first warp
// adds the cones in the same order.
//
// Bound by that chain (32 samples of some 0.5 us) where the launch does not fill
// the GPU: 47 x 31 pixels over 16^3 voxels take 19 us (one warp to 32 pixels:
// 38), 320 x 180 over 64^3 36 (60), 640 x 360 88 (101).  Where it does, the three
// warps that wait for the fourth cost more than the shorter chain gains:
// 1920 x 1080 over 256^3 675 (560).
//
// PAIRS: the marches take two steps at a time.  For launches of a CTA to an SM
// at most, which have the registers: the 47 x 31 pixels' frame 37 us (43).  The
// software sampler without a warp only; the others have not been tried.
constexpr int kSplit = 4;
template <int MODE, int KIND, bool PAIRS, class Scenes>
__global__ void __launch_bounds__(256, PAIRS ? 1 : 4) trace_split_kernel(const Scenes S) {
    long long tile;
    const TraceParams& P = S.get(S.find(blockIdx.x / kSplit, tile));
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int group = warp >> 1, slot = threadIdx.x & 63;
    int x, y;
    tile_pixel(P, tile, (int)(blockIdx.x % kSplit) * 2 + (warp & 1), lane, x, y);
    __shared__ Level s_lv[VCT_MAX_LEVELS];
    __shared__ ConeTable s_cone[2];
    __shared__ float4 s_out[7][64];
    fill_levels(P, s_lv);
    fill_cone(P, P.diffuse, P.max_distance, s_cone[0], 64);
    fill_cone(P, P.specular_cone, P.max_distance, s_cone[1], 128);
    grid_wait();  // (the chain's addresses come from the tables behind the barrier)
    __syncthreads();
    unsigned ns = 0;
    const bool inside = x < P.width && y < P.height;
    const long long pix = (long long)y * P.width + x;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 gp = inside ? __ldg(P.gpos + pix) : zero;
    if (gp.w != 0.0f && P.enable_indirect) {
        const float4 gn = __ldg(P.gnrm + pix);
        const f3 N = fnormalize(mk(gn.x, gn.y, gn.z));
        const f3 vp = volume_position(P, gp);
        if (group < 3) {
            f3 T, B;
            tangents(N, T, B);
#pragma unroll 1
            for (int c = 2 * group; c < 2 * group + 2; ++c)
                s_out[c][slot] = trace_cone<MODE, KIND, PAIRS>(P, s_lv, s_cone[0], vp, N, diffuse_direction(P, c, N, T, B),
                                                        P.diffuse, P.max_distance, ns);
        } else if (P.enable_reflections) {
            s_out[6][slot] = trace_cone<MODE, KIND, PAIRS>(P, s_lv, s_cone[1], vp, N, reflected(P, gp, N), P.specular_cone,
                                                    P.max_distance, ns);
        }
    }
    __syncthreads();
    if (group == 0 && inside) {
        float4 irr = zero, spc = zero, out = zero;
        if (gp.w != 0.0f) {
            if (P.enable_indirect) {
                for (int c = 0; c < 6; ++c) irr = add_cone(irr, kConeWeight[c], s_out[c][slot]);
                if (P.enable_reflections) spc = s_out[6][slot];
            }
            out = composite(P, pix, irr, spc);
        }
        store_pixel(P, pix, irr, spc, out);
    }
    count_samples(P, ns);
}

}  // namespace

template <class Scenes>
void launch_trace_split(const Scenes& S, int filter, int kind, long long tiles, int num_sms, bool overlap, cudaStream_t s) {
    if (filter == VCT_FILTER_SOFTWARE && kind == kConesPlain && tiles * kSplit <= num_sms) {
        launch_tiles(trace_split_kernel<VCT_FILTER_SOFTWARE, kConesPlain, true, Scenes>, S, tiles * kSplit, overlap, s);
        return;
    }
    with_trace_mode(filter, kind, [&](auto mode, auto cones) {
        launch_tiles(trace_split_kernel<mode.value, cones.value, false, Scenes>, S, tiles * kSplit, overlap, s);
    });
}

template void launch_trace_split(const OneScene<TraceParams>&, int, int, long long, int, bool, cudaStream_t);
template void launch_trace_split(const ManyScenes<TraceParams>&, int, int, long long, int, bool, cudaStream_t);
template void launch_trace_split(const FewScenes&, int, int, long long, int, bool, cudaStream_t);

}  // namespace vct
