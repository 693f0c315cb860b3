// Line walking shared by the depth rasteriser (raster.cu) and the voxeliser
// (voxelize.cu): the covered pixels of 256 set-up triangles, dealt out to a
// CTA's warps 32 at a time.
//
// A triangle is walked in lines: rows, or columns when its bounding box is
// more than twice as tall as wide, so that an upright sliver costs a few lines
// and not its whole height.  A line's covered pixels are contiguous and found
// from the triangle's crossings of it, with the edge functions at the first
// one.  The lines of a CTA's 256 triangles are numbered through, a thread
// takes a line, the pixel counts are scanned, and the warps take the pixels, 32
// a step, whichever lines and triangles they belong to.  Two walks:
// - by warps, for passes whose pixels cost little: a warp takes 64 lines (long
//   ones in pieces) and walks their pixels itself; after the triangles'
//   set-up no warp waits for another.
// - by CTAs, for passes whose pixels cost much: the CTA takes 512 lines
//   together, and each warp takes pixels when it has done its last, so that
//   the warps end together and only the last step of 512 lines has idle lanes.
//
// No scratch memory is used, so work is not handed from one CTA to another:
// the CTAs of gridDim.y set up the same 256 triangles and share their lines.
#pragma once

#include <algorithm>

#include "vct_device.cuh"

namespace vct {
namespace lines {

constexpr int kLineThreads = 256;
constexpr int kChunkLines = 512;  // lines a CTA takes together (half as many of the big triangles')
constexpr int kGroup = 64;        // lines a warp takes at most (likewise)
constexpr int kLineWarps = kLineThreads / 32;
// A set-up triangle in shared memory.  For its lines, with U along the line
// and V across, counter-clockwise in (U, V): {U0, V0, U1, V1}, {U2, V2,
// u0 | u1 << 16, v0}, flags.  For its pixels, in the caller's vertex order:
// what a pixel along a line adds to each edge function (per sub-pixel unit)
// and 1 / area; the depths and the triangle; two words of the caller's.
// (Five uint4: the odd stride spreads the banks.)
struct TriRec {
    uint4 v0, v1;
    int step[3];
    float inv;
    float z[3];
    int tri;
    uint32_t flags, user[2], unused;
};
static_assert(sizeof(TriRec) == 80, "a record's stride is five uint4");
// Twice the area from which on 32 bits do not hold the edge functions.
constexpr long long kBigArea = 1LL << 31;
// Flags: bits 0-2 the edges that are not top-left; bits 8-10 the logarithm of a
// line's pieces, bits 16-31 their pixels (128 or less, as long as 64 suffice).
constexpr uint32_t kRecSwapped = 8u, kRecColumns = 16u;
constexpr int kRecPieces = 8, kRecPart = 16;

// Stores the record of a set-up triangle; its lines, or with PIECES the pieces
// of them.  Columns only for boxes
// more than twice as tall as wide: the pixels of a column are in as many
// sectors of the image.
template <bool PIECES>
__device__ __forceinline__ int store_rec(TriRec& r, const RasterTri& t, const float z[3], int tri) {
    const int w = t.px1 - t.px0 + 1, h = t.py1 - t.py0 + 1;
    const bool columns = 2 * w < h;
    // (exchanging the axes reverses the order of the vertices)
    int U[3], V[3], bias[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int m = k == 0 ? 0 : 3 - k;
        U[k] = columns ? t.Y[m] : t.X[k];
        V[k] = columns ? t.X[m] : t.Y[k];
        bias[k] = columns ? t.bias[m] : t.bias[k];
    }
    const bool swapped = (t.perm1 != 0) != columns;
    const int u0 = columns ? t.py0 : t.px0, u1 = columns ? t.py1 : t.px1, v0 = columns ? t.px0 : t.py0;
    int pieces = 0, part = 0;
    if (PIECES) {
        // the longest line, in pixels: area / extent across (rounded up amply)
        const int across = max(V[0], max(V[1], V[2])) - min(V[0], min(V[1], V[2]));
        const int longest = min((int)(t.area_float() / ((float)across * (float)kSub) * 1.001f) + 2, u1 - u0 + 1);
        pieces = min(32 - __clz((longest - 1) >> 7), 6);
        part = (longest + (1 << pieces) - 1) >> pieces;
    }
    r.v0 = make_uint4((uint32_t)U[0], (uint32_t)V[0], (uint32_t)U[1], (uint32_t)V[1]);
    r.v1 = make_uint4((uint32_t)U[2], (uint32_t)V[2], (uint32_t)u0 | ((uint32_t)u1 << 16), (uint32_t)v0);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int st = V[(k + 1) % 3] - V[(k + 2) % 3];
        if (k == 0)
            r.step[0] = st;
        else
            r.step[swapped ? 3 - k : k] = st;
        r.z[k] = z[k];
    }
    r.inv = __fdiv_rn(1.0f, t.area_float());
    r.tri = tri;
    r.flags = (bias[0] ? 1u : 0u) | (bias[1] ? 2u : 0u) | (bias[2] ? 4u : 0u) | (swapped ? kRecSwapped : 0u) |
              (columns ? kRecColumns : 0u) | ((uint32_t)pieces << kRecPieces) | ((uint32_t)part << kRecPart);
    return (columns ? w : h) << pieces;
}

// The covered pixels of piece `k` of a triangle's lines, which are contiguous:
// the line, how many, the first one, and the edge functions there in the caller's vertex
// order (modulo 2^32 unless BIG).  The triangle's crossings of the line are
// computed in fp32; pixel centres further than eps from one are decided by it,
// the few nearer ones by the exact edge functions.
//
// With M the largest coordinate along the line, at most 2^28 sub-pixel units: an edge's extent (up to 2M), its extent
// across and the line's distance convert within 2^-24 each and the quotient is
// within 2^-22 (two units in the last place), so their product is within 14 x
// 2^-24 M, and with the first end's conversion within 15 x 2^-24 M.  Where a crossing
// matters, within the image's 2^23 units, it, its sum with eps and that with half
// a pixel round within 1/4 each.  eps = 16 x 2^-24 M + 1/2 covers that from M = 2^23
// on; below, all but the quotient and the roundings (which shrink with M) is exact.
template <bool BIG>
__device__ __forceinline__ int line_pixels(const TriRec& r, int k, int& line, int& first, long long base[3]) {
    const uint4 v0 = r.v0, v1 = r.v1;
    const uint32_t flags = r.flags;
    const int U[3] = {(int)v0.x, (int)v0.z, (int)v1.x}, V[3] = {(int)v0.y, (int)v0.w, (int)v1.y};
    const int u0 = (int)(v1.z & 0xffffu), u1 = (int)(v1.z >> 16), pieces = (int)(flags >> kRecPieces) & 7;
    line = (int)v1.w + (k >> pieces);
    const int at = line * kSub + kSub / 2;
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
    const float p0 = (float)u0, p1 = (float)u1;
    const int in0 = (int)fminf(fmaxf(ceilf((lo + eps - half) * rs), p0), p1 + 1.0f);
    const int in1 = (int)fmaxf(fminf(floorf((hi - eps - half) * rs), p1), p0 - 1.0f);
    first = (int)fminf(fmaxf(ceilf((lo - eps - half) * rs), p0), p1 + 1.0f);
    int last = (int)fmaxf(fminf(floorf((hi + eps - half) * rs), p1), p0 - 1.0f);
    if (first != in0 || last != in1) {
        // (products of 32-bit factors, exact in 64)
        auto covered = [&](int p) {
            const int u = p * kSub + kSub / 2;
            bool in = true;
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const int ia = (i + 1) % 3, ib = (i + 2) % 3;
                const long long e = (long long)(U[ib] - U[ia]) * (long long)(at - V[ia]) -
                                    (long long)(V[ib] - V[ia]) * (long long)(u - U[ia]);
                in = in && e - (long long)((flags >> i) & 1u) >= 0;
            }
            return in;
        };
        while (last >= first && last != in1 && !covered(last)) --last;
        while (first <= last && first != in0 && !covered(first)) ++first;
    }
    if (pieces > 0) {  // this piece's part
        const int n = (int)(flags >> kRecPart), p = k & ((1 << pieces) - 1);
        first += p * n;
        if (p + 1 < (1 << pieces)) last = min(last, first + n - 1);
    }
    if (first > last) return 0;
    const int u = first * kSub + kSub / 2;
    const bool sw = (flags & kRecSwapped) != 0u;
    long long e[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int ia = (i + 1) % 3, ib = (i + 2) % 3;
        if (BIG)
            e[i] = (long long)(U[ib] - U[ia]) * (long long)(at - V[ia]) -
                   (long long)(V[ib] - V[ia]) * (long long)(u - U[ia]);
        else
            e[i] = (uint32_t)(U[ib] - U[ia]) * (uint32_t)(at - V[ia]) - (uint32_t)(V[ib] - V[ia]) * (uint32_t)(u - U[ia]);
    }
    base[0] = e[0];
    base[1] = sw ? e[2] : e[1];
    base[2] = sw ? e[1] : e[2];
    return last - first + 1;
}

// Inclusive scans of `v` over the CTA, the totals in `total`; `s` holds a
// word per warp and value.  Callers put a barrier between two uses of one `s`.
template <int N>
__device__ __forceinline__ void cta_scan(int (&v)[N], int (*s)[kLineWarps], int (&total)[N]) {
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
        for (int w = 0; w < kLineWarps; ++w) {
            if (w == warp) v[n] += total[n];
            total[n] += s[n][w];
        }
    }
}

// Lines with covered pixels, in order: the number of the first pixel among the
// lines'; the line | its triangle's record << 16; the edge functions at the
// first pixel (64 bits each for big triangles, in two halves of the array) and
// its place.
template <int N>
struct LineList {
    int pix_off[N + 32];
    uint32_t line[N];
    uint4 base[N];
};
struct CtaLines {
    TriRec recs[kLineThreads];
    int line_off[kLineThreads];  // first line of each triangle among the CTA's
    LineList<kChunkLines> list;
    int scan[5][kLineWarps];
    int next;  // the step that the next free warp takes
};
struct WarpLines {
    TriRec recs[kLineThreads];
    // the triangles with lines, in order: the number of the first one; the record
    int line_off[kLineThreads + 33];
    uint8_t order[kLineThreads + 32];
    LineList<kGroup> list[kLineWarps];
    int scan[2][kLineWarps];
    int next;  // the line that the next free warp takes
};

// One lane's share of a step: a covered pixel and its weights and depth.
struct LinePixel {
    bool on;
    int px, py;
    float l[3], z;
    const TriRec* rec;
};

// Appends a line's run: its first pixel's number, the line, the edge functions.
template <bool BIG, int N>
__device__ __forceinline__ void list_line(LineList<N>& L, int at, int pix, int line, int rec, int first,
                                          const long long base[3]) {
    L.pix_off[at] = pix;
    L.line[at] = (uint32_t)line | ((uint32_t)rec << 16);
    if (BIG) {
        L.base[at] = make_uint4((uint32_t)base[0], (uint32_t)(base[0] >> 32), (uint32_t)base[1], (uint32_t)(base[1] >> 32));
        L.base[N / 2 + at] = make_uint4((uint32_t)base[2], (uint32_t)(base[2] >> 32), (uint32_t)first, 0u);
    } else {
        L.base[at] = make_uint4((uint32_t)base[0], (uint32_t)base[1], (uint32_t)base[2], (uint32_t)first);
    }
}

// The 32 pixels from number c0 on, a lane each, before number `end`; j: the
// line of the first one, moved on to the next step's.
template <bool BIG, int N>
__device__ __forceinline__ void take_step(const LineList<N>& L, const TriRec* recs, int c0, int end, int& j, LinePixel& f) {
    const int lane = threadIdx.x & 31;
    // The pixels lie in at most 32 lines, from line j on: a bit where each of
    // the later ones starts gives every lane its line.
    const int c = c0 + lane;
    const int off = L.pix_off[j + lane] - c0;
    const unsigned starts = __reduce_or_sync(0xffffffffu, off > 0 && off < 32 ? 1u << off : 0u);
    const int i = __popc(starts & (0xffffffffu >> (31 - lane)));
    f.on = c < end;
    if (f.on) {
        const uint32_t line = L.line[j + i];
        const TriRec& r = recs[line >> 16];
        const int4 d = *reinterpret_cast<const int4*>(r.step);  // and 1 / area
        const int n = c - L.pix_off[j + i];
        const uint4 b0 = L.base[j + i];
        float e[3];
        int u;
        if (BIG) {
            const uint4 b1 = L.base[N / 2 + j + i];
            const int m = n * kSub;
            const long long e0 = (long long)(((unsigned long long)b0.y << 32) | b0.x) + (long long)d.x * m,
                            e1 = (long long)(((unsigned long long)b0.w << 32) | b0.z) + (long long)d.y * m,
                            e2 = (long long)(((unsigned long long)b1.y << 32) | b1.x) + (long long)d.z * m;
            const bool wide = (e0 | e1 | e2) >= kHalvesLimit;
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
#pragma unroll
        for (int q = 0; q < 3; ++q) f.l[q] = e[q] * inv;
        f.z = interp(f.l, r.z[0], r.z[1], r.z[2]);
        const int v = (int)(line & 0xffffu);
        const bool columns = (r.flags & kRecColumns) != 0u;
        f.px = columns ? v : u;
        f.py = columns ? u : v;
        f.rec = &r;
    }
    j += __popc(starts);
    if (L.pix_off[j + 1] <= c0 + 32) ++j;  // that line's last pixel was the step's last
}

// Walks this slice's share of the lines of the CTA's triangles (`lines` of a
// thread's own), handing their covered pixels to `sink`, STEPS times 32 at a
// time (every lane of the warp calls it).  BIG: triangles of any area;
// otherwise twice the area is below 2^31 square sub-pixel units, and so are
// the covered pixels' edge functions: 32 bits hold them, whatever the products
// on the way.
template <bool BIG, int STEPS, class Sink>
__device__ __forceinline__ void walk_by_warps(WarpLines& S, int lines, Sink& sink) {
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31;
    const unsigned upto = FULL >> (31 - lane);
    int ends[2] = {lines, lines > 0 ? 1 : 0}, total[2];
    cta_scan(ends, S.scan, total);
    const int l_begin = (int)((long long)total[0] * blockIdx.y / gridDim.y);
    const int l_end = (int)((long long)total[0] * (blockIdx.y + 1) / gridDim.y);
    if (lines > 0) {
        S.line_off[ends[1] - 1] = ends[0] - lines;
        S.order[ends[1] - 1] = (uint8_t)tid;
    }
    if (tid < 33) S.line_off[total[1] + tid] = 0x7fffffff;
    if (tid == 33) S.next = l_begin;
    __syncthreads();
    // four helpings for each warp, of up to kGroup lines
    const int helping = min(BIG ? kGroup / 2 : kGroup, max(4, (l_end - l_begin + 4 * kLineWarps - 1) / (4 * kLineWarps)));
    LineList<kGroup>& G = S.list[tid >> 5];
    for (;;) {
        int l0 = 0;
        if (lane == 0) l0 = atomicAdd(&S.next, helping);
        l0 = __shfl_sync(FULL, l0, 0);
        if (l0 >= l_end) break;
        const int l1 = min(l0 + helping, l_end);
        // the last triangle whose lines start at or before l0
        int c = 0;
        {
            const int n8 = __popc(__ballot_sync(FULL, 8 * lane < total[1] && S.line_off[min(8 * lane, total[1])] <= l0));
            c = 8 * (n8 - 1);
            c += __popc(__ballot_sync(FULL, lane < 8 && c + lane < total[1] && S.line_off[min(c + lane, total[1])] <= l0)) - 1;
        }
        int npix = 0, nline = 0;
#pragma unroll 1
        for (int lq = l0; lq < l1; lq += 32) {
            // 32 lines belong to at most 32 triangles, from the c-th on: a bit
            // where each of the later ones starts gives every lane its own.
            const int off = S.line_off[c + 1 + lane] - lq;
            const unsigned starts = __reduce_or_sync(FULL, off > 0 && off < 32 ? 1u << off : 0u);
            const int mine = c + __popc(starts & upto);
            int cnt = 0, first = 0, line = 0, rec = 0;
            long long base[3] = {0, 0, 0};
            if (lq + lane < l1) {
                rec = S.order[mine];
                cnt = line_pixels<BIG>(S.recs[rec], lq + lane - S.line_off[mine], line, first, base);
            }
            c += __popc(starts);
            if (S.line_off[c + 1] <= lq + 32) ++c;  // that triangle's last line was the 32nd
            int end = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int u = __shfl_up_sync(FULL, end, o);
                if (lane >= o) end += u;
            }
            const unsigned any = __ballot_sync(FULL, cnt > 0);
            if (cnt > 0)
                list_line<BIG>(G, nline + __popc(any & upto) - 1, npix + end - cnt, line, rec, first, base);
            npix += __shfl_sync(FULL, end, 31);
            nline += __popc(any);
        }
        G.pix_off[nline + lane] = 0x7fffffff;
        __syncwarp();
        const int steps = (npix + 31) / 32;
        int j = 0;  // the line of the step's first pixel
        for (int st = 0; st < steps; st += STEPS) {
            LinePixel f[STEPS];
#pragma unroll
            for (int h = 0; h < STEPS; ++h) take_step<BIG>(G, S.recs, (st + h) * 32, npix, j, f[h]);
            sink(f);
        }
        __syncwarp();
    }
    __syncthreads();
}

// The same by CTAs (lines in one piece); a warp takes GRAB steps when it has
// done its last.
template <bool BIG, int STEPS, int GRAB, class Sink>
__device__ __forceinline__ void walk_by_ctas(CtaLines& S, int lines, Sink& sink) {
    constexpr int kChunk = BIG ? kChunkLines / 2 : kChunkLines;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31;
    int end[1] = {lines}, total[1];
    cta_scan(end, S.scan, total);
    S.line_off[tid] = end[0] - lines;
    __syncthreads();
    const int l_end = (int)((long long)total[0] * (blockIdx.y + 1) / gridDim.y);
    for (int l0 = (int)((long long)total[0] * blockIdx.y / gridDim.y); l0 < l_end; l0 += kChunk) {
        int npix = 0, nline = 0;
#pragma unroll 1
        for (int q = 0; q < kChunk / kLineThreads; ++q) {
            const int l = l0 + q * kLineThreads + tid;
            int first = 0, cnt = 0, rec = 0, line = 0;
            long long base[3] = {0, 0, 0};
            if (l < l_end) {
                // the last triangle whose lines start at or before l
#pragma unroll
                for (int st = kLineThreads / 2; st > 0; st >>= 1)
                    if (S.line_off[rec + st] <= l) rec += st;
                cnt = line_pixels<BIG>(S.recs[rec], l - S.line_off[rec], line, first, base);
            }
            int ends[2] = {cnt, cnt > 0 ? 1 : 0}, sums[2];  // covered pixels, lines that have any
            cta_scan(ends, S.scan + 1 + 2 * (q & 1), sums);
            if (cnt > 0)
                list_line<BIG>(S.list, nline + ends[1] - 1, npix + ends[0] - cnt, line, rec, first, base);
            npix += sums[0];
            nline += sums[1];
        }
        const int steps = (npix + 31) / 32;
        if (tid < 32) S.list.pix_off[nline + tid] = 0x7fffffff;
        if (tid == 32) S.next = 0;
        __syncthreads();
        for (;;) {
            int s0 = 0;
            if (lane == 0) s0 = atomicAdd(&S.next, GRAB);
            s0 = __shfl_sync(FULL, s0, 0);
            if (s0 >= steps) break;
            const int s1 = min(s0 + GRAB, steps);
            int j = 0;  // the line of the step's first pixel
#pragma unroll
            for (int st = kChunk / 2; st > 0; st >>= 1)
                if (j + st < nline && S.list.pix_off[j + st] <= s0 * 32) j += st;
            for (int st = s0; st < s1; st += STEPS) {
                LinePixel f[STEPS];
#pragma unroll
                for (int h = 0; h < STEPS; ++h)
                    take_step<BIG>(S.list, S.recs, (st + h) * 32, min(npix, 32 * s1), j, f[h]);
                sink(f);
            }
        }
        __syncthreads();
    }
}

// Triangle of a thread: runs of RUN dealt out to the CTAs, since neighbours in
// the array are often alike in size.
template <int RUN>
__device__ __forceinline__ long long my_triangle() {
    return ((long long)(threadIdx.x / RUN) * gridDim.x + blockIdx.x) * RUN + (threadIdx.x % RUN);
}

// Every thread's set-up triangle: the small ones the 32-bit way, then the big
// ones.
template <int STEPS, class Sink>
__device__ __forceinline__ void walk_all(WarpLines& S, int lines, bool big, Sink& sink) {
    walk_by_warps<false, STEPS>(S, big ? 0 : lines, sink);
    if (__syncthreads_or(big)) walk_by_warps<true, STEPS>(S, big ? lines : 0, sink);
}
template <int STEPS, int GRAB, class Sink>
__device__ __forceinline__ void walk_all(CtaLines& S, int lines, bool big, Sink& sink) {
    walk_by_ctas<false, STEPS, GRAB>(S, big ? 0 : lines, sink);
    if (__syncthreads_or(big)) walk_by_ctas<true, STEPS, GRAB>(S, big ? lines : 0, sink);
}

// Grid of a kernel over `ntri` triangles: as many CTAs to each 256 of them (at
// most 64, or what gives `fill` in all) as give `want` in all, but no more than
// have some `share` pixels each if the triangles cover `pixels`, and at least
// `least` where there are more sets of 256 than SMs hold CTAs.
inline dim3 line_grid(long long ntri, long long want, long long pixels, long long share, int num_sms, long long least,
                      long long fill = 0) {
    const long long ctas = (ntri + kLineThreads - 1) / kLineThreads;
    const long long n = std::min((want + ctas - 1) / ctas, pixels / (ctas * share));
    return dim3((unsigned)ctas,
                (unsigned)std::max(ctas > 4LL * num_sms ? least : 1LL, std::min(n, std::max(64LL, fill / ctas))));
}

}  // namespace lines
}  // namespace vct
