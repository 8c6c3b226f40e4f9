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
#include <cuda_runtime.h>
#include <stdint.h>
#include "events.cuh"
#include "kernels.h"

namespace rgpu {
namespace {

using dev::event_diffs;

constexpr int kWarps = 8;
constexpr int kCol = 32;         // events of a lane (one more than the crossings it sorts)
constexpr int kColStride = 33;   // words between a column's entries
constexpr uint32_t kOver = 0xFFFFFFFFu;

// A crossing's sort key: the x of an edge on the sub-scanline relative to the
// row's first pixel, clamped to the row's pixels (16.16 sub-columns, below 2^31:
// anti-aliased rows end below pixel 8192, aliased ones below 32768), and the
// winding in the lowest bit (-1 first among equal x, as the reference's sort has
// it; crossings of equal x and winding commute).  Where clamping merges
// crossings left (right) of the row, only the winding at the row's first pixel
// matters (nothing does), so their order is free.
__device__ __forceinline__ bool crossing_key(const int4 &e, int32_t y, int32_t base, uint32_t xmax, uint32_t *key) {
    const int32_t dy = y - e.z;
    if ((uint32_t)dy > (uint32_t)(e.w >> 8)) return false;
    const int32_t X = (int32_t)((uint32_t)e.x + (uint32_t)dy * (uint32_t)e.y);
    const uint32_t d = X > base ? min((uint32_t)X - (uint32_t)base, xmax) : 0u;
    *key = (d << 1) | ((e.w & 0x80) ? 0u : 1u);
    return true;
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

// One sub-scanline of one row of one draw, as its lane sees it.
struct RowScan {
    const uint32_t *list;  // the draw's binned edges (indices)
    uint32_t nb;           // their number; 0: nothing to draw on this sub-scanline
    int32_t y, base;       // (sub)scanline; the row's first pixel in 16.16 (sub)columns
    uint32_t xmax;         // the row's width in 16.16 (sub)columns
    uint32_t off;          // the row's first pixel in the stream's row
    uint32_t kind;         // end_entry's
    int32_t fill_mask;     // 1 even-odd, -1 non-zero
};

// A sub-scanline with more crossings than a column holds, by a whole warp:
// each lane takes an edge and sums the windings of the crossings before its own
// (32 crossings ranked at a time, no limit on their number).  Counts the events,
// or writes them to `out` (EMIT).
template <bool EMIT>
__device__ __noinline__ uint32_t crowded(const RowScan &r, const int4 *edges, const uint32_t *ends, uint32_t *out) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t psh = r.kind == 2u ? 0u : 2u, lm = r.kind == 2u ? 0u : 3u;
    const uint32_t *tab = ends + 16 * r.kind;
    auto key_at = [&](uint32_t j, uint32_t *key) {
        return crossing_key(__ldg(edges + __ldg(r.list + j)), r.y, r.base, r.xmax, key);
    };
    auto winding_before = [&](uint32_t key, uint32_t i) {
        int32_t w = 0;
        for (uint32_t j = 0; j < r.nb; j++) {
            uint32_t kj;
            if (key_at(j, &kj) && (kj < key || (kj == key && j < i))) w += key_winding(kj);
        }
        return w;
    };
    uint32_t count = 0;
    for (uint32_t i0 = 0; i0 < r.nb; i0 += 32) {
        const uint32_t i = i0 + lane;
        uint32_t key = 0;
        bool end = false, in = false;
        if (i < r.nb && key_at(i, &key)) {
            const int32_t w = winding_before(key, i);
            in = (w & r.fill_mask) != 0;
            end = in != (((w + key_winding(key)) & r.fill_mask) != 0);
        }
        const uint32_t who = __ballot_sync(0xffffffffu, end);
        if (EMIT && end) {
            const uint32_t x = key_sub(key), p = x >> psh;
            uint32_t t = x & lm;
            if (in) {
                // the span's opening end, if it lies in the same pixel: the last
                // opening crossing before this one there
                bool found = false;
                uint32_t best = 0, best_j = 0;
                if (r.kind == 1u)
                    for (uint32_t j = 0; j < r.nb; j++) {
                        uint32_t kj;
                        if (!key_at(j, &kj) || !(kj < key || (kj == key && j < i)) || (key_sub(kj) >> 2) != p) continue;
                        if (found && (kj < best || (kj == best && j < best_j))) continue;
                        const int32_t wj = winding_before(kj, j);
                        if ((wj & r.fill_mask) != 0 || ((wj + key_winding(kj)) & r.fill_mask) == 0) continue;
                        found = true;
                        best = kj;
                        best_j = j;
                    }
                t += found && (key_sub(best) & 3u) != 0u ? 12u : 4u;
            }
            out[count + (uint32_t)__popc(who & ((1u << lane) - 1u))] = (r.off + p) + tab[t];
        }
        count += (uint32_t)__popc(who);
    }
    __syncwarp();
    if ((winding_before(0xFFFFFFFFu, 0) & r.fill_mask) != 0) {  // unclosed: the span runs to the row's end
        if (EMIT && lane == 0) out[count] = (r.off + (r.xmax >> (16 + psh))) + tab[4];
        count++;
    }
    return count;
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
#pragma unroll 4
    for (uint32_t i = 0; i < r.nb; i++) {
        const int4 e = __ldg(edges + __ldg(r.list + i));
        uint32_t key;
        if (crossing_key(e, r.y, r.base, r.xmax, &key)) {
            if (n < (uint32_t)kCol - 1) col[n * kColStride] = key;
            n++;
        }
    }
    const bool over = n > (uint32_t)kCol - 1;
    if (over) n = 0;
    const uint32_t most = __reduce_max_sync(0xffffffffu, n);
    if (most > 16) sort_column<32>(col, n);
    else if (most > 8) sort_column<16>(col, n);
    else if (most > 4) sort_column<8>(col, n);
    else if (most > 1) sort_column<4>(col, n);
    // walk: each end of a span overwrites the column from its start (never past
    // the crossings read)
    const uint32_t psh = r.kind == 2u ? 0u : 2u, lm = r.kind == 2u ? 0u : 3u;
    const uint32_t *tab = ends + 16 * r.kind;
    uint32_t m = 0, left = 0, f = 0;
    int32_t w = 0;
    bool in = false;  // inside a span
    for (uint32_t i = 0; i < n; i++) {
        const uint32_t key = col[i * kColStride];
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
        const uint32_t row = t / per_row, d0 = (t - row * per_row) << 5;
        const uint32_t slot0 = st.bin_off + row * st.draw_cnt + d0, nd = min(32u, st.draw_cnt - d0);
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
                const DrawRec &dr = draws[st.draw_off + (slot - st.bin_off - row * st.draw_cnt)];
                const int32_t ox = dr.ox, ly = (int32_t)row - dr.oy;
                const int32_t xl = max(dr.sect_l, -ox), xr = min(dr.sect_r, st.out_w - ox);
                const bool aa = dr.shift != 0;
                boff = __ldg(bin_offsets + slot);
                r.y = aa ? ly * 4 + (int32_t)sub : ly;
                if (dr.valid && xl < xr && ly >= dr.sect_t && ly < dr.sect_b && r.y >= dr.start_y && r.y < dr.stop_y &&
                    (aa || sub == 0u)) {
                    r.list = bins + boff;
                    r.nb = __ldg(bin_counts + slot);
                    r.base = xl << (aa ? 18 : 16);
                    r.xmax = (uint32_t)(xr - xl) << (aa ? 18 : 16);
                    r.off = (uint32_t)(xl + ox);
                    r.kind = !aa ? 2u : (sub == 3u ? 1u : 0u);
                    r.fill_mask = (dr.flags & DRAW_EVENODD) ? 1 : -1;
                }
            }
            uint32_t first = 0x7FFFu, last = 0u;
            uint32_t m = lane_events(col, r, edges, ends, &first, &last);
            __syncwarp();
            const uint32_t overs = __ballot_sync(0xffffffffu, m == kOver);
            if (m == kOver) {
                first = r.off;
                last = r.off + (r.xmax >> (r.kind == 2u ? 16 : 18));
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
            for (uint32_t o = overs; o; o &= o - 1u) {
                const int src = __ffs(o) - 1;
                const uint32_t c = crowded<false>(scan_of(src), edges, ends, nullptr);
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
            uint32_t *list = events + 4ull * ((unsigned long long)boff + slot);
            // each row's list as a run: entry k is entry k - before of the lane
            // whose share holds it
            for (int g = 0; g < 32; g += 4) {
                const uint32_t n = __shfl_sync(0xffffffffu, all, g);
                if (!n) continue;
                const uint32_t s1 = __shfl_sync(0xffffffffu, before, g + 1), s2 = __shfl_sync(0xffffffffu, before, g + 2),
                               s3 = __shfl_sync(0xffffffffu, before, g + 3);
                uint32_t *dst = reinterpret_cast<uint32_t *>(
                    __shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)list, g));
                const uint32_t og = overs >> g & 0xFu;
                for (uint32_t k = lane; k < n; k += 32u) {
                    const uint32_t s = (uint32_t)(k >= s1) + (uint32_t)(k >= s2) + (uint32_t)(k >= s3);
                    const uint32_t i = k - (s == 0u ? 0u : s == 1u ? s1 : s == 2u ? s2 : s3);
                    if (!(og >> s & 1u)) dst[k] = cols[warp][i * kColStride + (uint32_t)g + s];
                }
                for (uint32_t o = og; o; o &= o - 1u) {
                    const int s = __ffs(o) - 1;
                    crowded<true>(scan_of(g + s), edges, ends, dst + (s == 0 ? 0u : s == 1 ? s1 : s == 2 ? s2 : s3));
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
