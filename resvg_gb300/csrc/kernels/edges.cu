// Geometry kernels: per-draw setup, per-segment edge building, exclusive scans
// and row binning.
//
// Pipeline for one submission (all draws of all streams):
//   k_draw_setup   warp/draw:      transform points, bounds, scan ranges
//                                  (tiny-skia painter.rs fill_path + scan/path_aa.rs
//                                  fill_path), segment slots (path.rs PathEdgeIter)
//   k_edges<false> 1, 4 or 8 segments/warp: count line edges
//   scan           exclusive prefix sum -> edge offsets
//   k_edges<true>  1, 4 or 8 segments/warp: write line edges (edge_builder.rs)
//   k_draw_edges   thread/draw:    paths with < 2 edges are dropped
//   k_bin<false>   1 to 32 edges/warp: count (row, draw) bin sizes
//   scan           -> bin offsets
//   k_bin<true>    1 to 32 edges/warp: list the edge in its rows' bins
//   k_events       events.cu:      the coverage events of every (row, draw)
#include <cuda_runtime.h>
#include <stdint.h>
#include "edge_build.cuh"
#include "kernels.h"

namespace rgpu {
namespace {

using dev::Pt;

__device__ __forceinline__ bool nearly_zero(float v) { return fabsf(v) <= (1.0f / 4096.0f); }

// One warp per draw: points and verbs are taken 32 at a time, the verbs' points
// and segment slots by prefix counts.  (One thread per draw, walking its points
// and verbs twice, took 17 us on a 6-path icon and 78 us on 2,500 paths.)
constexpr int kSetupWarps = 4;
__global__ void __launch_bounds__(32 * kSetupWarps)
k_draw_setup(DrawRec *draws, uint32_t ndraws, const uint8_t *scene_verbs, const float *scene_pts,
             const uint8_t *stroke_verbs, const float *stroke_pts, Pt *tpts, SegRec *segs) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t d = blockIdx.x * kSetupWarps + (threadIdx.x >> 5);
    if (d >= ndraws) return;
    DrawRec dr = draws[d];  // every lane holds the record; lane 0 writes it back
    // a stroke outline built on the device lives in the stroke arrays
    const bool stroked = (dr.flags & DRAW_STROKED) != 0;
    const uint8_t *verbs = (stroked ? stroke_verbs : scene_verbs) + dr.verb_off;
    const float *pts = (stroked ? stroke_pts : scene_pts) + 2 * (size_t)dr.pt_off;
    dr.valid = 0;
    auto done = [&]() {
        if (lane == 0) draws[d] = dr;
    };
    // segment slots default to empty
    for (uint32_t i = lane; i <= dr.verb_cnt; i += 32u) segs[dr.seg_base + i] = SegRec{d, 0, 0, 0};
    __syncwarp();  // before other lanes write the segments to the same slots
    if (dr.flags & 0x80000000u) { done(); return; }  // host-side skip
    // ---- transform (tiny-skia Transform::map_points branches)
    const float sx = dr.ts[0], ky = dr.ts[1], kx = dr.ts[2], sy = dr.ts[3], tx = dr.ts[4], ty = dr.ts[5];
    const bool ident = sx == 1 && ky == 0 && kx == 0 && sy == 1 && tx == 0 && ty == 0;
    const bool skew = kx != 0 || ky != 0;
    const bool scale = sx != 1 || sy != 1;
    // bounds: fminf / fmaxf ignore NaN, so the order of the points does not matter
    const float nan = __int_as_float(0x7FC00000);
    float l = nan, t = nan, r = nan, b = nan;
    bool finite = true;
    for (uint32_t i = lane; i < dr.pt_cnt; i += 32u) {
        const float x = pts[2 * i], y = pts[2 * i + 1];
        float nx, ny;
        if (ident) { nx = x; ny = y; }
        else if (!skew && !scale) { nx = x + tx; ny = y + ty; }
        else if (!skew) { nx = x * sx + tx; ny = y * sy + ty; }
        else { nx = x * sx + y * kx + tx; ny = x * ky + y * sy + ty; }
        if (!ident && (!isfinite(nx) || !isfinite(ny))) finite = false;
        tpts[dr.tpt_base + i] = Pt{nx, ny};
        l = fminf(l, nx); r = fmaxf(r, nx);
        t = fminf(t, ny); b = fmaxf(b, ny);
    }
    for (int o = 16; o > 0; o >>= 1) {
        l = fminf(l, __shfl_xor_sync(0xffffffffu, l, o));
        t = fminf(t, __shfl_xor_sync(0xffffffffu, t, o));
        r = fmaxf(r, __shfl_xor_sync(0xffffffffu, r, o));
        b = fmaxf(b, __shfl_xor_sync(0xffffffffu, b, o));
    }
    finite = __all_sync(0xffffffffu, finite);
    if (!finite || dr.pt_cnt == 0) { done(); return; }
    if (nearly_zero(r - l) || nearly_zero(b - t)) { done(); return; }
    const float lim = 3.4028235e38f * 0.25f;
    if (!(l >= -lim && t >= -lim && r <= lim && b <= lim)) { done(); return; }
    const int32_t cw = dr.clip_w, ch = dr.clip_h;
    bool aa = (dr.flags & DRAW_AA) != 0;
    if (aa) {
        float fl = floorf(l), ft = floorf(t), fr = ceilf(r), fb = ceilf(b);
        int32_t ix = dev::sat_i32(fl), iy = dev::sat_i32(ft);
        int32_t iw = max(1, dev::sat_i32(fr - fl)), ih = max(1, dev::sat_i32(fb - ft));
        int32_t sl = max(ix, 0), st = max(iy, 0), sr = min(ix + iw, cw), sb = min(iy + ih, ch);
        if (sr <= sl || sb <= st) { done(); return; }
        bool ovf = sl > 8191 || st > 8191 || sr > 8191 || sb > 8191 || sl < -8192 || st < -8192;
        if (ovf) aa = false;  // supersampled coordinates would overflow i16: aliased fill
        else {
            if (cw > 32767 || ch > 32767) { done(); return; }
            bool contained = ix >= 0 && iy >= 0 && ix + iw <= cw && iy + ih <= ch;
            dr.shift = 2;
            dr.contained = contained;
            dr.sect_l = sl; dr.sect_t = st; dr.sect_r = sr; dr.sect_b = sb;
            int32_t sy0 = iy << 2, sy1 = (iy + ih) << 2;
            if (!contained) { sy0 = max(sy0, 0); sy1 = min(sy1, ch << 2); }
            dr.start_y = sy0; dr.stop_y = sy1;
            dr.valid = 1;
        }
    }
    if (!aa) {
        const double bias = 0.5 + 1.5 / 64.0;
        int32_t il = dev::sat_i32((float)ceil((double)l - bias));
        int32_t it = dev::sat_i32((float)ceil((double)t - bias));
        int32_t ir = dev::sat_i32((float)floor((double)r + bias));
        int32_t ib = dev::sat_i32((float)floor((double)b + bias));
        if (ir <= il || ib <= it) { done(); return; }
        bool contained = il >= 0 && it >= 0 && ir <= cw && ib <= ch;
        int32_t y0 = it, y1 = ib;
        if (!contained) { y0 = max(y0, 0); y1 = min(y1, ch); }
        if (y0 >= y1) { done(); return; }
        dr.shift = 0;
        dr.contained = contained;
        dr.sect_l = 0; dr.sect_t = 0; dr.sect_r = cw; dr.sect_b = ch;
        dr.start_y = y0; dr.stop_y = y1;
        dr.valid = 1;
    }
    // ---- segments (PathEdgeIter with implicit close lines), 32 verbs at a
    // time.  Every drawing verb needs a current point and its points must exist.
    // pi, ns: points and segments before the chunk; move_to: the last move's
    // point; open: a drawing verb since the last move or close.
    const uint32_t base = dr.tpt_base, below = (1u << lane) - 1u;
    uint32_t pi = 0, ns = 0, move_to = 0;
    bool open = false, have_cur = false, ok = true;
    for (uint32_t v0 = 0; v0 < dr.verb_cnt; v0 += 32u) {
        const bool in = v0 + lane < dr.verb_cnt;
        const uint32_t v = in ? verbs[v0 + lane] : 255u;
        const bool move = v == RGPU_MOVE, close = v == RGPU_CLOSE;
        const bool draw = v == RGPU_LINE || v == RGPU_QUAD || v == RGPU_CUBIC;
        const uint32_t moves = __ballot_sync(0xffffffffu, move), closes = __ballot_sync(0xffffffffu, close);
        const uint32_t drawn = __ballot_sync(0xffffffffu, draw);
        if (__any_sync(0xffffffffu, in && !move && !close && !draw)) ok = false;
        if (__any_sync(0xffffffffu, draw && !have_cur && (moves & below) == 0u)) ok = false;
        have_cur = have_cur || moves != 0u;
        const uint32_t np = move || v == RGPU_LINE ? 1u : v == RGPU_QUAD ? 2u : v == RGPU_CUBIC ? 3u : 0u;
        const uint32_t before = (uint32_t)dev::warp_prefix((int32_t)np) - np;
        // the contour's first point as of this verb, and whether a line is due to it
        const uint32_t prev_moves = moves & below, ends = (moves | closes) & below;
        const uint32_t mt = __shfl_sync(0xffffffffu, pi + before, prev_moves ? 31 - __clz(prev_moves) : 0);
        const uint32_t to = prev_moves ? mt : move_to;
        const uint32_t since = ends ? drawn & below & ~((2u << (31 - __clz(ends))) - 1u) : drawn & below;
        const bool due = since != 0u || (ends == 0u && open);
        const bool seg = draw || ((move || close) && due);
        const uint32_t segm = __ballot_sync(0xffffffffu, seg);
        if (seg) {
            const uint32_t p = base + pi + before - 1u;
            segs[dr.seg_base + ns + (uint32_t)__popc(segm & below)] =
                draw ? (v == RGPU_LINE ? SegRec{d, 1, p, p + 1u} : SegRec{d, v == RGPU_QUAD ? 2u : 3u, p, 0})
                     : SegRec{d, 1, p, base + to};
        }
        // carries
        const uint32_t all_ends = moves | closes;
        const uint32_t after = all_ends ? drawn & ~((2u << (31 - __clz(all_ends))) - 1u) : drawn;
        open = after != 0u || (all_ends == 0u && open);
        if (moves) move_to = __shfl_sync(0xffffffffu, pi + before, 31 - __clz(moves));
        pi += __shfl_sync(0xffffffffu, before + np, 31);
        ns += (uint32_t)__popc(segm);
    }
    if (!ok || pi > dr.pt_cnt) {
        // the path is not drawn: its slots are empty again
        __syncwarp();
        for (uint32_t i = lane; i <= dr.verb_cnt; i += 32u) segs[dr.seg_base + i] = SegRec{d, 0, 0, 0};
        dr.valid = 0;
        done();
        return;
    }
    if (open && lane == 0) segs[dr.seg_base + ns] = SegRec{d, 1, base + pi - 1, base + move_to};
    done();
}

// Eight segments per warp: a lane each for chopping and clipping, then the whole
// warp on each piece's lines.  One thread per segment, stepping up to 64 lines
// of a curve with a division each, took 18 + 23 us on a 6-path icon and 186 + 227
// us on 2,500 paths (count and emit), all of it one thread's latency.
// Few segments are spread thinner (per_warp), as their warps' latency is all
// that counts.  Count and emit, us, by 1 / 4 / 8 a warp: 4,200 curves 35 / 36 / 50,
// 4,200 straight lines 16 / 13 / 16, 2,000 lines 12 / 13 / 15; 12,000 curves 65 / 51 /
// 58, 16,600 curves 82 / 72 / 64 and lines 35 / 23 / 18.
constexpr int kEdgeWarps = 4;
constexpr int kEdgeSegs = 8;
inline uint32_t edge_segs_per_warp(uint32_t nsegs) {
    return nsegs <= 4096u ? 1u : nsegs <= 16384u ? 4u : (uint32_t)kEdgeSegs;
}
template <bool EMIT>
__global__ void __launch_bounds__(32 * kEdgeWarps)
k_edges(const SegRec *segs, uint32_t nsegs, const DrawRec *draws, const Pt *tpts, uint32_t *counts,
        const uint32_t *offsets, EdgeRec *edges, uint32_t *edge_draw, uint32_t edge_cap, uint32_t per_warp) {
    __shared__ dev::Piece pieces[kEdgeWarps][kEdgeSegs][dev::kMaxPieces];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t s0 = (blockIdx.x * kEdgeWarps + (uint32_t)warp) * per_warp;
    if (s0 >= nsegs) return;
    const uint32_t s = s0 + (uint32_t)lane;
    dev::PieceSink sink{pieces[warp][lane & (kEdgeSegs - 1)], 0};
    uint32_t draw = 0;
    int shift = 0;
    if ((uint32_t)lane < per_warp && s < nsegs) {
        const SegRec sg = segs[s];
        draw = sg.draw;
        if (sg.kind != 0) {
            const DrawRec &dr = draws[sg.draw];
            if (dr.valid) {
                Pt p[4];
                if (sg.kind == 1) { p[0] = tpts[sg.p0]; p[1] = tpts[sg.p1]; }
                else { for (uint32_t k = 0; k <= sg.kind; k++) p[k] = tpts[sg.p0 + k]; }
                const dev::ClipR clip{0.0f, 0.0f, (float)dr.clip_w, (float)dr.clip_h};
                shift = dr.shift;
                dev::build_segment(sink, (int)sg.kind, p, dr.contained != 0, clip);
            }
        }
    }
    __syncwarp();
    for (int i = 0; i < (int)per_warp && s0 + (uint32_t)i < nsegs; i++) {
        const uint32_t np = min(__shfl_sync(0xffffffffu, sink.n, i), (uint32_t)dev::kMaxPieces);
        const int sh = __shfl_sync(0xffffffffu, shift, i);
        const uint32_t d = __shfl_sync(0xffffffffu, draw, i);
        uint32_t off = 0, cap = 0, n = 0;
        if (EMIT) {
            off = offsets[s0 + (uint32_t)i];
            cap = min(off < edge_cap ? edge_cap - off : 0u, counts[s0 + (uint32_t)i]);
        }
        for (uint32_t k = 0; k < np; k++)
            dev::expand_piece(pieces[warp][i][k], sh, [&](const dev::LineE &e, int w, bool ok) {
                const uint32_t m = __ballot_sync(0xffffffffu, ok);
                const uint32_t at = n + (uint32_t)__popc(m & ((1u << lane) - 1u));
                if (EMIT && ok && at < cap) {
                    edges[off + at] = EdgeRec{e.x, e.dx, e.first_y, ((e.last_y - e.first_y) << 8) | (w & 0xff)};
                    edge_draw[off + at] = d;
                }
                n += (uint32_t)__popc(m);
            });
        if (!EMIT && lane == 0) counts[s0 + (uint32_t)i] = n;
    }
}

__global__ void k_draw_edges(DrawRec *draws, uint32_t ndraws, const uint32_t *seg_offsets) {
    uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
    if (d >= ndraws) return;
    DrawRec &dr = draws[d];
    uint32_t b = seg_offsets[dr.seg_base], e = seg_offsets[dr.seg_base + dr.verb_cnt + 1];
    if (dr.valid && e - b < 2) dr.valid = 0;
}

// The rows of a warp's edges (per_warp of them, at most 32) are shared out evenly
// over its lanes, whatever each edge's height: an edge walking its rows alone
// waits for one atomic after the other (494 us for the 1024^2 scene's 26 M entries).
constexpr int kBinThreads = 256;
template <bool SCATTER>
__global__ void __launch_bounds__(kBinThreads)
k_bin(const EdgeRec *edges, const uint32_t *edge_draw, uint32_t nedges, uint32_t per_warp, const DrawRec *draws,
      const StreamRec *streams, uint32_t *bin_counts, const uint32_t *bin_offsets, uint32_t bin_cap, uint32_t *err,
      uint32_t *bins) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t e0 = (blockIdx.x * (kBinThreads / 32) + (threadIdx.x >> 5)) * per_warp, e = e0 + lane;
    uint32_t rows = 0, slot = 0, step = 0;  // the edge's rows, the first one's slot, slots per row
    if (lane < per_warp && e < nedges) {
        const uint32_t d = edge_draw[e];
        const DrawRec &dr = draws[d];
        if (dr.valid) {
            const StreamRec &st = streams[dr.stream];
            const EdgeRec er = edges[e];
            const int32_t y0 = max(er.first_y, dr.start_y), y1 = min(er.first_y + (er.hw >> 8), dr.stop_y - 1);
            // every row of the pass the edge has a (sub)scanline in
            const int32_t b0 = max((y0 >> dr.shift) + dr.oy, st.row_lo), b1 = min((y1 >> dr.shift) + dr.oy, st.row_hi - 1);
            if (y1 >= y0 && b1 >= b0) {
                rows = (uint32_t)(b1 - b0 + 1);
                step = st.draw_cnt;
                slot = st.bin_off + (uint32_t)(b0 - st.row_lo) * step + (d - st.draw_off);
            }
        }
    }
    uint32_t upto = rows;  // rows of the edges up to this one
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= (uint32_t)o) upto += t;
    }
    const uint32_t total = __shfl_sync(0xffffffffu, upto, 31);
    for (uint32_t j0 = 0; j0 < total; j0 += 32u) {
        const uint32_t j = j0 + lane;
        // the edge that holds the j-th row: as many as end at or before it
        uint32_t k = 0;
#pragma unroll
        for (uint32_t o = 16; o > 0; o >>= 1) {
            const uint32_t t = __shfl_sync(0xffffffffu, upto, (int)(k + o - 1u));
            if (t <= j) k += o;
        }
        k = min(k, 31u);
        const uint32_t before = __shfl_sync(0xffffffffu, upto - rows, (int)k);
        const uint32_t first = __shfl_sync(0xffffffffu, slot, (int)k), per = __shfl_sync(0xffffffffu, step, (int)k);
        if (j < total) {
            const uint32_t at = first + (j - before) * per;
            const uint32_t n = atomicAdd(&bin_counts[at], 1u);
            if (SCATTER) {
                const uint32_t pos = bin_offsets[at] + n;
                if (pos < bin_cap) bins[pos] = e0 + k;
                else atomicOr(err, 1u);
            }
        }
    }
}

// Few edges are spread thinner, as a warp walks their rows 32 at a time.  Count and
// emit, us, by 1 / 4 / 8 / 32 edges a warp: 400 edges of 1,000 rows (rules across a
// 1024^2 canvas) 32 / 91 / 170 / 651, of 2 rows 9 / 9 / 9 / 10; 8,000 of 60 rows 16 /
// 17 / 22 / 57, of 2 rows 10 / 9 / 10 / 12; 16,000 of 60 rows 26 / 25 / 27 / 60, of 2
// rows 15 / 10 / 9 / 11; 64,000 of 10 rows 41 / 22 / 19 / 22; 130,000 of 60 rows 138 /
// 133 / 145 / 160, of 10 rows 72 / 36 / 31 / 30.
inline uint32_t bin_edges_per_warp(uint32_t nedges) {
    return nedges <= 8192u ? 1u : nedges <= 32768u ? 4u : nedges <= 131072u ? 8u : 32u;
}

// ---- exclusive scan (three passes, 1024-element tiles)
constexpr int SCAN_T = 256;
constexpr int SCAN_PER = 4;
constexpr int SCAN_TILE = SCAN_T * SCAN_PER;

template <class T>
__device__ __forceinline__ T block_exclusive(T v, T *sh, T *total) {
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T x = v;
    for (int o = 1; o < 32; o <<= 1) {
        T y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        T w = lane < (SCAN_T / 32) ? sh[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            T y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < (SCAN_T / 32)) sh[lane] = w;
    }
    __syncthreads();
    T warp_prefix = wid ? sh[wid - 1] : 0;
    *total = sh[SCAN_T / 32 - 1];
    __syncthreads();
    return warp_prefix + x - v;
}

// Sums that do not fit 32 bits are kept as 2^32 - 1, a tile's as well as the
// total, so that the caller sees a total that does not fit (the offsets are not
// used then); 64-bit sums in between.
__device__ __forceinline__ uint32_t sat_u32(unsigned long long v) { return (uint32_t)min(v, 0xFFFFFFFFull); }

__global__ void k_scan_reduce(const uint32_t *in, uint64_t n, uint32_t *block_sums) {
    __shared__ unsigned long long sh[32];
    uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    unsigned long long s = 0;
    for (int k = 0; k < SCAN_PER; k++) {
        uint64_t i = base + (uint64_t)threadIdx.x * SCAN_PER + k;
        if (i < n) s += in[i];
    }
    unsigned long long total;
    block_exclusive(s, sh, &total);
    if (threadIdx.x == 0) block_sums[blockIdx.x] = sat_u32(total);
}
__global__ void k_scan_blocks(uint32_t *block_sums, uint32_t nblocks, uint32_t *total_out) {
    __shared__ unsigned long long sh[32];
    unsigned long long carry = 0;
    for (uint32_t base = 0; base < nblocks; base += SCAN_T) {
        uint32_t i = base + threadIdx.x;
        unsigned long long v = i < nblocks ? block_sums[i] : 0, tot;
        unsigned long long ex = block_exclusive(v, sh, &tot);
        if (i < nblocks) block_sums[i] = (uint32_t)(carry + ex);
        carry += tot;
    }
    if (threadIdx.x == 0) *total_out = sat_u32(carry);
}
__global__ void k_scan_down(const uint32_t *in, uint64_t n, const uint32_t *block_sums, uint32_t *out) {
    __shared__ uint32_t sh[32];
    uint64_t base = (uint64_t)blockIdx.x * SCAN_TILE;
    uint32_t v[SCAN_PER];
    uint32_t s = 0;
    for (int k = 0; k < SCAN_PER; k++) {
        uint64_t i = base + (uint64_t)threadIdx.x * SCAN_PER + k;
        v[k] = i < n ? in[i] : 0;
        s += v[k];
    }
    uint32_t total;
    uint32_t ex = block_exclusive(s, sh, &total) + block_sums[blockIdx.x];
    for (int k = 0; k < SCAN_PER; k++) {
        uint64_t i = base + (uint64_t)threadIdx.x * SCAN_PER + k;
        if (i < n) out[i] = ex;
        ex += v[k];
    }
}

// The whole scan in one block, bound by launch and load latency.  The three
// launches above take 8.3 us and the gaps between them however little they do;
// this one 4.0 us for 1,001 words, 4.7 for 4,096.  Threads read neighbouring runs,
// so longer runs cost more transactions (16,381 words by 16 each: 15.1 us), and
// the line is at 4 words per thread.  Sums are 64-bit up to the total; offsets past
// a total that does not fit are not read.
constexpr int SCAN_ONE_T = 1024;
constexpr int SCAN_ONE_PER = 4;
__global__ void __launch_bounds__(SCAN_ONE_T)
k_scan_one(const uint32_t *in, uint32_t n, uint32_t per, uint32_t *out, uint32_t *total_out) {
    __shared__ unsigned long long warp_sums[32];
    const uint32_t lane = threadIdx.x & 31u, wid = threadIdx.x >> 5, base = threadIdx.x * per;
    uint32_t v[SCAN_ONE_PER];
    unsigned long long sum = 0;
#pragma unroll
    for (uint32_t k = 0; k < (uint32_t)SCAN_ONE_PER; k++) {
        v[k] = k < per && base + k < n ? in[base + k] : 0u;
        sum += v[k];
    }
    unsigned long long x = sum;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= (uint32_t)o) x += y;
    }
    if (lane == 31u) warp_sums[wid] = x;
    __syncthreads();
    const unsigned long long w = warp_sums[lane];
    unsigned long long before = lane < wid ? w : 0ull, all = w;
    for (int o = 16; o; o >>= 1) {
        before += __shfl_xor_sync(0xffffffffu, before, o);
        all += __shfl_xor_sync(0xffffffffu, all, o);
    }
    unsigned long long at = before + x - sum;
#pragma unroll
    for (uint32_t k = 0; k < (uint32_t)SCAN_ONE_PER; k++) {
        if (k < per && base + k < n) out[base + k] = (uint32_t)at;
        at += v[k];
    }
    if (threadIdx.x == 0) *total_out = sat_u32(all);
}

inline uint32_t blocks_for(uint64_t n, uint32_t t) { return (uint32_t)((n + t - 1) / t); }

}  // namespace

// ---------------------------------------------------------------- host launchers
cudaError_t launch_draw_setup(DrawRec *draws, uint32_t ndraws, const uint8_t *verbs, const float *pts,
                              const uint8_t *stroke_verbs, const float *stroke_pts, void *tpts, SegRec *segs,
                              cudaStream_t s) {
    if (!ndraws) return cudaSuccess;
    k_draw_setup<<<blocks_for(ndraws, kSetupWarps), 32 * kSetupWarps, 0, s>>>(draws, ndraws, verbs, pts, stroke_verbs, stroke_pts,
                                                         (Pt *)tpts, segs);
    return cudaGetLastError();
}
cudaError_t launch_edges(bool emit, const SegRec *segs, uint32_t nsegs, const DrawRec *draws, const void *tpts,
                         uint32_t *counts, const uint32_t *offsets, EdgeRec *edges, uint32_t *edge_draw,
                         uint32_t edge_cap, cudaStream_t s) {
    if (!nsegs) return cudaSuccess;
    const uint32_t per = edge_segs_per_warp(nsegs);
    const uint32_t blocks = blocks_for(nsegs, kEdgeWarps * per);
    if (emit)
        k_edges<true><<<blocks, 32 * kEdgeWarps, 0, s>>>(segs, nsegs, draws, (const Pt *)tpts, counts, offsets, edges,
                                                         edge_draw, edge_cap, per);
    else
        k_edges<false><<<blocks, 32 * kEdgeWarps, 0, s>>>(segs, nsegs, draws, (const Pt *)tpts, counts, offsets, edges,
                                                          edge_draw, edge_cap, per);
    return cudaGetLastError();
}
cudaError_t launch_draw_edges(DrawRec *draws, uint32_t ndraws, const uint32_t *seg_offsets, cudaStream_t s) {
    if (!ndraws) return cudaSuccess;
    k_draw_edges<<<blocks_for(ndraws, 256), 256, 0, s>>>(draws, ndraws, seg_offsets);
    return cudaGetLastError();
}
cudaError_t launch_bin(bool scatter, const EdgeRec *edges, const uint32_t *edge_draw, uint32_t nedges,
                       const DrawRec *draws, const StreamRec *streams, uint32_t *bin_counts,
                       const uint32_t *bin_offsets, uint32_t bin_cap, uint32_t *err, uint32_t *bins, cudaStream_t s) {
    if (!nedges) return cudaSuccess;
    const uint32_t per = bin_edges_per_warp(nedges), blocks = blocks_for(nedges, kBinThreads / 32 * per);
    if (scatter)
        k_bin<true><<<blocks, kBinThreads, 0, s>>>(edges, edge_draw, nedges, per, draws, streams, bin_counts,
                                                   bin_offsets, bin_cap, err, bins);
    else
        k_bin<false><<<blocks, kBinThreads, 0, s>>>(edges, edge_draw, nedges, per, draws, streams, bin_counts,
                                                    bin_offsets, bin_cap, err, bins);
    return cudaGetLastError();
}
uint32_t scan_launches(uint64_t n) { return n <= (uint64_t)SCAN_ONE_T * SCAN_ONE_PER ? 1u : 3u; }
size_t scan_scratch_words(uint64_t n) { return (size_t)blocks_for(n ? n : 1, SCAN_TILE) + 1; }
// out[i] = sum(in[0..i)), *total = sum(in); `scratch` holds scan_scratch_words(n) words.
cudaError_t launch_exclusive_scan(const uint32_t *in, uint32_t *out, uint64_t n, uint32_t *scratch, uint32_t *total,
                                  cudaStream_t s) {
    if (n == 0) return cudaMemsetAsync(total, 0, 4, s);
    if (scan_launches(n) == 1) {
        k_scan_one<<<1, SCAN_ONE_T, 0, s>>>(in, (uint32_t)n, blocks_for(n, SCAN_ONE_T), out, total);
        return cudaGetLastError();
    }
    uint32_t nb = blocks_for(n, SCAN_TILE);
    k_scan_reduce<<<nb, SCAN_T, 0, s>>>(in, n, scratch);
    k_scan_blocks<<<1, SCAN_T, 0, s>>>(scratch, nb, total);
    k_scan_down<<<nb, SCAN_T, 0, s>>>(in, n, scratch, out);
    return cudaGetLastError();
}

}  // namespace rgpu
