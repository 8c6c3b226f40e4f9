// The event kernel: for every (row, draw) of every stream, the ends of the spans
// that the draw's binned edges make on the row's sub-scanlines (events.cuh).
//
// One warp takes 32 draws of one row.  The draws with edges in the row are
// picked out by ballots, so rows that few draws touch cost little, and eight of
// them are worked on at a time, one lane per (draw, sub-scanline): gather the
// crossings into the lane's column of shared memory, sort it in registers (a
// network), walk it and overwrite it with events, and write each row's list as
// one coalesced run.
//
// A kernel of its own, because the work splits evenly over (row, draw) while
// shading splits over pixels: rows cut into pieces for the raster kernel share
// the events instead of making them again, and neither kernel's code evicts the
// other's from the instruction caches (one kernel doing both, a warp per row
// piece, had 9.9 of 13 stalled warps waiting for instructions).
//
// What bounds it: issue, at 70% of the slots and 45% of the warps, and the latency
// of the edge gathers on small scenes: 0.60 ms for 14.2 M binned edges on 1024^2
// pixels, 4.8 ms for 114.6 M of 128 mixed scenes.  64 registers, as the compiler has
// it: 80 (3 CTAs per SM) took 2% more of the 1024^2 frame, 95 took 5%.  The gather
// is free of branches: with one per edge for crossings left of the row a 512^2
// drawing took 60 us in this kernel for 45.
#include <cuda_runtime.h>
#include <stdint.h>
#include "events.cuh"
#include "kernels.h"

namespace rgpu {
namespace {

using dev::event_diffs;

constexpr int kWarps = 8;
constexpr int kCol = 32;         // events of a lane
constexpr int kMaxSort = kCol - 2;  // crossings it sorts: the row's start and end may add an event each
constexpr int kColStride = 33;   // words between a column's entries
constexpr uint32_t kOver = 0xFFFFFFFFu;

// A crossing's sort key: the x of an edge on the sub-scanline relative to the
// row's first pixel (16.16 sub-columns, below 2^31: anti-aliased rows end below
// pixel 8192, aliased ones hold kMaxStrip pixels at most), and the winding in the lowest bit (-1
// first among equal x, as the reference's sort has it; crossings of equal x and
// winding commute).  Only crossings inside the row have one: of those left of it
// the sum of the windings matters alone, `before`, and of those right of it
// nothing.  (A view into a drawing has many of both: its clipped contours run
// along the clip's sides.)
__device__ __forceinline__ bool crossing_key(const int4 &e, int32_t y, int32_t base, uint32_t xmax, uint32_t *key,
                                             int32_t *before) {
    const int32_t dy = y - e.z;
    const bool hit = (uint32_t)dy <= (uint32_t)(e.w >> 8);
    const int32_t X = (int32_t)((uint32_t)e.x + (uint32_t)dy * (uint32_t)e.y);
    const uint32_t up = (e.w & 0x80) ? 0u : 1u, d = (uint32_t)X - (uint32_t)base;
    const bool left = X <= base;
    *before += hit && left ? (int32_t)(up << 1) - 1 : 0;
    *key = hit && !left ? (d << 1) | up : 0u;
    return hit && !left && d < xmax;
}
// the key's x rounded to a sub-column: ((key >> 1) + 0x8000) >> 16
__device__ __forceinline__ uint32_t key_sub(uint32_t key) { return (key + 0x10000u) >> 17; }
__device__ __forceinline__ int32_t key_winding(uint32_t key) { return (int32_t)((key & 1u) << 1) - 1; }

// The differences of an end depend on few cases, so they come from a table:
// kind (0: M = 64, 1: M = 63, 2: aliased) x 16 + closing x 4 + span inside the
// pixel x 8 + l.
__device__ __forceinline__ uint32_t end_entry(int idx) {
    const int kind = idx >> 4, l = idx & 3, M = kind == 0 ? 64 : 63;
    if (kind == 2) return event_diffs((idx & 4) ? -255 : 255, 0);
    if (!(idx & 4)) {
        const int d0 = l ? 64 - 16 * l : M;
        return event_diffs(d0, M - d0);
    }
    const int c = (idx & 8) ? 64 - M : 0;
    return event_diffs(16 * l - M - c, c - 16 * l);
}

// A crossing right of pixel 32767.5 rounds, in 32 bits, to -32768: it comes last
// but its end lies at the row's start (an opening one) or closes a span of no
// length (a closing one).  Only layers wider than 32767 pixels have such.
constexpr uint32_t kWide = 3;
constexpr int32_t kRoundsOver = 0x7FFF8000;

// One sub-scanline of one row of one draw, as its lane sees it.
struct RowScan {
    const uint32_t *list;  // the draw's binned edges (indices)
    uint32_t nb;           // their number; 0: nothing to draw on this sub-scanline
    int32_t y, base;       // (sub)scanline; the row's first pixel in 16.16 (sub)columns
    uint32_t xmax;         // the row's width in 16.16 (sub)columns
    uint32_t off;          // the row's first pixel among the pass's columns
    uint32_t kind;         // end_entry's; kWide: 2, on a layer wider than 16.16 coordinates reach
    int32_t fill_mask;     // 1 even-odd, -1 non-zero
};

// Sorts v[0 .. n) by a whole warp: bitonic, every exchange towards ascending
// order (each merge starts with mirrored pairs), so entries past n need not exist.
__device__ __forceinline__ void sort_list(uint32_t *v, uint32_t n) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k = 2; (k >> 1) < n; k <<= 1)
        for (uint32_t j = k >> 1; j; j >>= 1) {
            for (uint32_t q = lane;; q += 32u) {
                const uint32_t lo = ((q & ~(j - 1u)) << 1) | (q & (j - 1u));
                const uint32_t hi = j == k >> 1 ? lo ^ (k - 1u) : lo + j;
                if (lo >= n) break;
                if (hi >= n) continue;
                const uint32_t a = v[lo], b = v[hi];
                if (a > b) {
                    v[lo] = b;
                    v[hi] = a;
                }
            }
            __syncwarp();
        }
}

// A sub-scanline with more crossings than a column holds, by a whole warp in
// global memory: `v` holds nb + 1 words, the most events the sub-scanline can
// have.  The keys go to v[1 ..], are sorted there, and are walked 32 at a time
// into events from v[0] on (never past the keys read).  Returns their number.
// n log^2 n / 32 steps, whatever the crossings: ties and shared pixels are usual
// where contours are clipped.
__device__ __noinline__ uint32_t crowded(const RowScan &r, const int4 *edges, const uint32_t *ends, uint32_t *v) {
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const uint32_t psh = r.kind >= 2u ? 0u : 2u, lm = r.kind >= 2u ? 0u : 3u;
    const uint32_t *tab = ends + 16 * min(r.kind, 2u);
    uint32_t n = 0;
    int32_t w = 0;
    for (uint32_t i0 = 0; i0 < r.nb; i0 += 32u) {
        uint32_t key = 0;
        bool in = i0 + lane < r.nb &&
                  crossing_key(__ldg(edges + __ldg(r.list + i0 + lane)), r.y, r.base, r.xmax, &key, &w);
        // rounds over (key: its distance from the row's start, or 0): last of all
        if (r.kind == kWide && (key >> 1) >= (uint32_t)kRoundsOver - (uint32_t)r.base && key != 0u) {
            key = ((r.xmax + 1u) << 1) | (key & 1u);
            in = true;
        }
        const uint32_t who = __ballot_sync(0xffffffffu, in);
        if (in) v[1u + n + (uint32_t)__popc(who & below)] = key;
        n += (uint32_t)__popc(who);
    }
    w = __reduce_add_sync(0xffffffffu, w);
    __syncwarp();
    sort_list(v + 1, n);
    uint32_t m = 0, left = 0;  // events, and where the last span opened
    if ((w & r.fill_mask) != 0) {  // open at the row's start
        if (lane == 0) v[0] = r.off + tab[0];
        m = 1;
    }
    for (uint32_t i0 = 0; i0 < n; i0 += 32u) {
        const bool valid = i0 + lane < n;
        const uint32_t key = valid ? v[1u + i0 + lane] : 0u;
        int32_t upto = valid ? key_winding(key) : 0;
        const int32_t own = upto;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t t = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= (uint32_t)o) upto += t;
        }
        upto += w;
        const bool in = ((upto - own) & r.fill_mask) != 0, now = (upto & r.fill_mask) != 0, end = valid && in != now;
        const uint32_t who = __ballot_sync(0xffffffffu, end), opens = __ballot_sync(0xffffffffu, end && now);
        const uint32_t mine = opens & below;
        const bool over = (key >> 1) > r.xmax;  // rounds over
        uint32_t x = over ? 0u : key_sub(key);
        const uint32_t opened = __shfl_sync(0xffffffffu, x, mine ? 31 - __clz(mine) : 0), from = mine ? opened : left;
        if (over && in) x = from;
        const uint32_t p = x >> psh;
        uint32_t t = x & lm;
        if (in) t += ((from & lm) != 0u && (from >> psh) == p) ? 12u : 4u;
        __syncwarp();  // these 32 keys have been read
        if (end) v[m + (uint32_t)__popc(who & below)] = (r.off + p) + tab[t];
        m += (uint32_t)__popc(who);
        w = __shfl_sync(0xffffffffu, upto, 31);
        if (opens) left = __shfl_sync(0xffffffffu, x, 31 - __clz(opens));
    }
    if ((w & r.fill_mask) != 0) {  // unclosed: the span runs to the row's end
        if (lane == 0) v[m] = (r.off + (r.xmax >> (16 + psh))) + tab[4];
        m++;
    }
    __syncwarp();
    return m;
}

__device__ __forceinline__ void cmp_swap(uint32_t &a, uint32_t &b) {
    const uint32_t lo = min(a, b), hi = max(a, b);
    a = lo;
    b = hi;
}
// Batcher's odd-even merge sort, from the stage that merges runs of P at distance K.
template <int N, int P, int K>
__device__ __forceinline__ void merge_stages(uint32_t (&v)[N]) {
#pragma unroll
    for (int i = 0; i + K < N; i++)
        if (i >= K % P && (i - K % P) % (2 * K) < K && i / (2 * P) == (i + K) / (2 * P)) cmp_swap(v[i], v[i + K]);
    if constexpr (K > 1) merge_stages<N, P, K / 2>(v);
    else if constexpr (2 * P < N) merge_stages<N, 2 * P, 2 * P>(v);
}
// Sorts the first n entries of a lane's column in N registers (absent entries
// sort last): every lane takes the same steps, and none waits for shared memory.
template <int N>
__device__ __forceinline__ void sort_column(uint32_t *col, uint32_t n) {
    uint32_t v[N];
#pragma unroll
    for (int i = 0; i < N; i++) v[i] = (uint32_t)i < n ? col[i * kColStride] : 0xFFFFFFFFu;
    merge_stages<N, 1, 1>(v);
#pragma unroll
    for (int i = 0; i < N; i++)
        if ((uint32_t)i < n) col[i * kColStride] = v[i];
}

// The events of one lane's sub-scanline, over its column; returns their number
// (kOver: more crossings than the column holds) and widens [first, last], the
// pixels its coverage may touch.  All lanes of the warp call it.
__device__ __forceinline__ uint32_t lane_events(uint32_t *col, const RowScan &r, const int4 *edges, const uint32_t *ends,
                                                uint32_t *first, uint32_t *last) {
    uint32_t n = 0;
    int32_t w = 0;
    uint32_t *keys = col + kColStride;  // from the second entry on: the walk writes one event ahead
#pragma unroll 4
    for (uint32_t i = 0; i < r.nb; i++) {
        const int4 e = __ldg(edges + __ldg(r.list + i));
        uint32_t key;
        if (crossing_key(e, r.y, r.base, r.xmax, &key, &w)) {
            if (n < (uint32_t)kMaxSort) keys[n * kColStride] = key;
            n++;
        }
    }
    const bool over = n > (uint32_t)kMaxSort || r.kind == kWide;
    if (over) n = 0;
    const uint32_t most = __reduce_max_sync(0xffffffffu, n);
    if (most > 16) sort_column<kMaxSort>(keys, n);
    else if (most > 8) sort_column<16>(keys, n);
    else if (most > 4) sort_column<8>(keys, n);
    else if (most > 1) sort_column<4>(keys, n);
    // walk: each end of a span overwrites the column from its start (never past
    // the crossings read)
    const uint32_t psh = r.kind >= 2u ? 0u : 2u, lm = r.kind >= 2u ? 0u : 3u;
    const uint32_t *tab = ends + 16 * min(r.kind, 2u);
    uint32_t m = 0, left = 0, f = 0;
    bool in = (w & r.fill_mask) != 0;  // inside a span
    if (in) {  // open at the row's start
        col[0] = r.off + tab[0];
        m = 1;
    }
    for (uint32_t i = 0; i < n; i++) {
        const uint32_t key = keys[i * kColStride];
        w += key_winding(key);
        const bool now = (w & r.fill_mask) != 0;
        if (now != in) {
            const uint32_t x = key_sub(key), p = x >> psh;
            uint32_t t = x & lm;
            if (in) t += ((left & lm) != 0u && (left >> psh) == p) ? 12u : 4u;
            if (m == 0u) f = p;
            col[m * kColStride] = (r.off + p) + tab[t];
            m++;
            left = x;
            in = now;
        }
    }
    if (m) {
        *first = r.off + f;
        *last = r.off + (left >> psh);
    }
    if (in) {  // unclosed: the span runs to the row's end
        *last = r.off + (r.xmax >> (16 + psh));
        col[m * kColStride] = *last + tab[4];
        m++;
    }
    return over ? kOver : m;
}

__global__ void __launch_bounds__(32 * kWarps)
k_events(const StreamRec *streams, uint32_t nstreams, uint32_t ntasks, const DrawRec *draws, const EdgeRec *edge_recs,
         const uint32_t *bins, const uint32_t *bin_offsets, const uint32_t *bin_counts, uint32_t *headers,
         uint32_t *events, uint32_t *err) {
    __shared__ uint32_t ends[48];
    __shared__ uint32_t cols[kWarps][kCol * kColStride];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (threadIdx.x < 48) ends[threadIdx.x] = end_entry((int)threadIdx.x);
    __syncthreads();
    const int4 *edges = reinterpret_cast<const int4 *>(edge_recs);
    uint32_t *col = cols[warp] + lane;
    for (uint32_t task = blockIdx.x * kWarps + warp; task < ntasks; task += gridDim.x * kWarps) {
        // the stream: the last whose first task is not after this one
        uint32_t lo = 0, hi = nstreams;
        while (hi - lo > 1u) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(&streams[mid].task_off) <= task) lo = mid;
            else hi = mid;
        }
        const StreamRec &st = streams[lo];
        const uint32_t per_row = (st.draw_cnt + 31u) >> 5, t = task - st.task_off;
        const uint32_t r0 = t / per_row, d0 = (t - r0 * per_row) << 5;  // the row, from the pass's first
        const uint32_t slot0 = st.bin_off + r0 * st.draw_cnt + d0, nd = min(32u, st.draw_cnt - d0);
        uint32_t work = __ballot_sync(0xffffffffu, lane < nd && __ldg(bin_counts + slot0 + lane) != 0u);
        if (lane < nd && !(work >> lane & 1u)) headers[slot0 + lane] = 0u;  // no edges here
        while (work) {
            // lane group q takes the q-th of the next eight draws
            const uint32_t q = lane >> 2, sub = lane & 3u;
            uint32_t w = work;
#pragma unroll
            for (uint32_t k = 0; k < 8u; k++) {
                if (k < q) w &= w - 1u;
                work &= work - 1u;
            }
            const bool have = w != 0u;
            const uint32_t slot = slot0 + (have ? (uint32_t)__ffs(w) - 1u : 0u);
            RowScan r;
            r.list = nullptr;
            r.nb = 0;
            r.y = r.base = 0;
            r.xmax = r.off = r.kind = 0;
            r.fill_mask = -1;
            uint32_t boff = 0;
            if (have) {
                const DrawRec &dr = draws[st.draw_off + (slot - st.bin_off - r0 * st.draw_cnt)];
                const int32_t ox = dr.ox, ly = st.row_lo + (int32_t)r0 - dr.oy;
                const int32_t xl = max(dr.sect_l, st.x_lo - ox), xr = min(dr.sect_r, st.x_hi - ox);
                const bool aa = dr.shift != 0;
                boff = __ldg(bin_offsets + slot);
                r.y = aa ? ly * 4 + (int32_t)sub : ly;
                if (dr.valid && xl < xr && ly >= dr.sect_t && ly < dr.sect_b && r.y >= dr.start_y && r.y < dr.stop_y &&
                    (aa || sub == 0u)) {
                    r.list = bins + boff;
                    r.nb = __ldg(bin_counts + slot);
                    // past pixel 32767 every crossing lies left of the row
                    r.base = aa ? xl << 18 : xl > 32767 ? INT32_MAX : xl << 16;
                    r.xmax = (uint32_t)(xr - xl) << (aa ? 18 : 16);
                    r.off = (uint32_t)(xl + ox - st.x_lo);
                    r.kind = !aa ? (dr.sect_r > 32767 ? kWide : 2u) : (sub == 3u ? 1u : 0u);
                    r.fill_mask = (dr.flags & DRAW_EVENODD) ? 1 : -1;
                }
            }
            uint32_t first = 0x7FFFu, last = 0u;
            uint32_t m = lane_events(col, r, edges, ends, &first, &last);
            __syncwarp();
            const uint32_t overs = __ballot_sync(0xffffffffu, m == kOver);
            if (m == kOver) {
                first = r.off;
                last = r.off + (r.xmax >> (r.kind >= 2u ? 16 : 18));
            }
            auto scan_of = [&](int src) {
                RowScan s;
                s.list = reinterpret_cast<const uint32_t *>(
                    __shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)r.list, src));
                s.nb = __shfl_sync(0xffffffffu, r.nb, src);
                s.y = __shfl_sync(0xffffffffu, r.y, src);
                s.base = __shfl_sync(0xffffffffu, r.base, src);
                s.xmax = __shfl_sync(0xffffffffu, r.xmax, src);
                s.off = __shfl_sync(0xffffffffu, r.off, src);
                s.kind = __shfl_sync(0xffffffffu, r.kind, src);
                s.fill_mask = __shfl_sync(0xffffffffu, r.fill_mask, src);
                return s;
            };
            // each sub-scanline of a row has a quarter of the row's room in the list,
            // where a crowded one makes its events
            uint32_t *list = events + 4ull * ((unsigned long long)boff + slot);
            auto list_of = [&](int src) {
                return reinterpret_cast<uint32_t *>(__shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)list, src));
            };
            for (uint32_t o = overs; o; o &= o - 1u) {
                const int src = __ffs(o) - 1;
                const RowScan s = scan_of(src);
                const uint32_t c = crowded(s, edges, ends, list_of(src) + (size_t)(src & 3) * (s.nb + 1u));
                if ((int)lane == src) m = c;
            }
            // the row's header and the lanes' places in its list
            uint32_t before = 0, all = m;
            const uint32_t m1 = __shfl_xor_sync(0xffffffffu, m, 1);
            const uint32_t pair = m + m1, other = __shfl_xor_sync(0xffffffffu, pair, 2);
            before = (sub & 1u ? m1 : 0u) + (sub & 2u ? other : 0u);
            all = pair + other;
            first = min(first, __shfl_xor_sync(0xffffffffu, first, 1));
            first = min(first, __shfl_xor_sync(0xffffffffu, first, 2));
            last = max(last, __shfl_xor_sync(0xffffffffu, last, 1));
            last = max(last, __shfl_xor_sync(0xffffffffu, last, 2));
            if (have && sub == 0u) {
                uint32_t h = 0u;
                if (all > dev::kMaxEvents) atomicOr(err, 2u);
                else if (all >= dev::kManyEvents) h = dev::kManyEvents << 20 | all;
                else if (all) h = all << 20 | (first >> 5) << 10 | last >> 5;
                headers[slot] = h;
            }
            // each row's list as a run: entry k is entry k - before of the lane
            // whose share holds it
            for (int g = 0; g < 32; g += 4) {
                const uint32_t n = __shfl_sync(0xffffffffu, all, g);
                if (!n) continue;
                const uint32_t s1 = __shfl_sync(0xffffffffu, before, g + 1), s2 = __shfl_sync(0xffffffffu, before, g + 2),
                               s3 = __shfl_sync(0xffffffffu, before, g + 3);
                uint32_t *dst = list_of(g);
                const uint32_t og = overs >> g & 0xFu;
                if (og == 0u) {
                    for (uint32_t k = lane; k < n; k += 32u) {
                        const uint32_t s = (uint32_t)(k >= s1) + (uint32_t)(k >= s2) + (uint32_t)(k >= s3);
                        const uint32_t i = k - (s == 0u ? 0u : s == 1u ? s1 : s == 2u ? s2 : s3);
                        dst[k] = cols[warp][i * kColStride + (uint32_t)g + s];
                    }
                    continue;
                }
                // sub-scanlines in order: a share never starts after its own
                // quarter, so it overwrites no later one
                for (int s = 0; s < 4; s++) {
                    const uint32_t from = s == 0 ? 0u : s == 1 ? s1 : s == 2 ? s2 : s3;
                    const uint32_t c = (s == 0 ? s1 : s == 1 ? s2 : s == 2 ? s3 : n) - from;
                    const uint32_t room = __shfl_sync(0xffffffffu, r.nb, g + s) + 1u;
                    const uint32_t *src = dst + (size_t)s * room;
                    for (uint32_t k0 = 0; k0 < c; k0 += 32u) {
                        const uint32_t k = k0 + lane;
                        uint32_t e = 0;
                        if (k < c) e = (og >> s & 1u) ? src[k] : cols[warp][k * kColStride + (uint32_t)(g + s)];
                        __syncwarp();
                        if (k < c) dst[from + k] = e;
                        __syncwarp();
                    }
                }
            }
            __syncwarp();  // the columns have been read
        }
    }
}

}  // namespace

cudaError_t launch_events(const StreamRec *streams, uint32_t nstreams, uint32_t ntasks, const DrawRec *draws,
                          const EdgeRec *edges, const uint32_t *bins, const uint32_t *bin_offsets,
                          const uint32_t *bin_counts, uint32_t *headers, uint32_t *events, uint32_t *err,
                          cudaStream_t s) {
    if (!ntasks) return cudaSuccess;
    const uint32_t blocks = (ntasks + kWarps - 1) / kWarps;
    k_events<<<blocks, 32 * kWarps, 0, s>>>(streams, nstreams, ntasks, draws, edges, bins, bin_offsets, bin_counts,
                                            headers, events, err);
    return cudaGetLastError();
}

}  // namespace rgpu
