// The raster kernel: one persistent kernel renders every work item (a row of a stream,
// or a piece of it) by executing the stream's command list, one warp per item.
//
// Per draw, the warp adds the row's coverage events (events.cuh) to a difference
// array in shared memory, scans it into one coverage byte per pixel and a mask
// of the 32-pixel groups with any coverage, and shades the groups the mask
// names, two at a time, 32 neighbouring pixels per step.  Draws whose header
// says they do not touch the piece are never visited.
//
// Warps share nothing, so none waits for another; the only wait is for the
// next commands, copied ahead into shared memory (bounded, see wait_chunk).
//
// What bounds it: instruction issue while enough warps are resident, and a
// warp's own dependent chain while they are not.  Measured on 1024^2 pixels with
// 2,000 gradient fills and 500 strokes: 6.8 ms, 3.6 G instructions, 0.42 of the
// issue slots (9 warps per SM on average: the rows' costs differ and the last
// ones run alone).  The kernel before it, with four producer warps per CTA that
// rasterised spans and eight consumer warps that walked run lists pixel by
// pixel, took 12.2 ms and issued 6 G; on 256 mixed scenes 29.5 against 84.7 ms
// (beside the event kernel: 4.8 ms of it to 17.6 here on 128 of them).
#include <cuda_runtime.h>
#include <stdint.h>
#include "events.cuh"
#include "kernels.h"
#include "pipeline.cuh"

namespace rgpu {
namespace {

constexpr int kWarps = 4;               // warps per CTA
constexpr int kThreads = 32 * kWarps;
// 20 warps per SM at 96 registers: at 80 (24 warps) the row's state spills,
// 10.3 against 9.1 ms on the 1024^2 scene, 53.4 against 52.0 ms on the mixed ones
constexpr int kMinBlocks = 5;
constexpr int kMaxDepth = 48;    // layer stack depth
constexpr int kChunk = 32;       // commands copied at a time
constexpr uint32_t kNone = 0xFFFFFFFFu;

// What drawing a fill reads, copied ahead (cp.async) while the fill before it is
// drawn: no registers hold it and no load waits for another.
struct FillSlot {
    uint4 rows[2 * kMaxGradStops];   // the gradient's colour rows
    uint4 paint[3];                  // the PaintRec
    float4 stops[3];                 // the gradient's stop positions
    uint32_t events[32];             // the first events
    int2 org;                        // layer origin
    int2 _pad;
};

struct WarpShared {
    unsigned long long mb;           // mbarrier of the command copies
    int32_t first, _pad;             // the piece's first pixel among the row's event pixels (no register held)
    Cmd chunk[2][kChunk];            // the current commands and the next
    uint32_t rect[kMaxDepth];        // layer-stack layers by depth
    PaintRec hair_paint;             // the current hairline's paint
    FillSlot fill[2];                // the current fill and the next
    // followed (per warp) by the difference array (row width / 2 + 4 words, two
    // 16-bit differences each), the coverage bytes and the top layer's pixels
};
static_assert(sizeof(WarpShared) % 16 == 0 && sizeof(FillSlot) % 16 == 0 && sizeof(Cmd) == 16 && sizeof(PaintRec) == 48,
              "16-byte copies");
static_assert(offsetof(DrawRec, ox) % 8 == 0 && offsetof(DrawRec, oy) == offsetof(DrawRec, ox) + 4 && sizeof(DrawRec) % 8 == 0 &&
              2 * kMaxGradStops == 24, "copies of a fill");
__host__ __device__ constexpr size_t warp_bytes(uint32_t row_w) {
    return sizeof(WarpShared) + (row_w / 2 + 4) * 4 + row_w + row_w * 4;
}

// ---- the command copies (cp.async.bulk into shared memory, mbarrier, bounded waits)
__device__ __forceinline__ uint32_t smem_addr(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void mb_init(unsigned long long *mb, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(mb)), "r"(count) : "memory");
}
// copies `n` commands (16 bytes each, 16-byte aligned on both sides); one lane
__device__ __forceinline__ void copy_chunk(WarpShared &ws, uint32_t buf, const Cmd *src, uint32_t n) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&ws.mb)), "r"(16u * n) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(smem_addr(ws.chunk[buf])), "l"(src), "r"(16u * n), "r"(smem_addr(&ws.mb)) : "memory");
}
// asynchronous copies of 4, 8 or 16 bytes into shared memory
template <int N>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(smem_addr(dst)), "l"(src), "n"(N) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Waits, as a whole warp, for the copy of parity `parity`; false (for every
// lane) when it does not land within `limit` try_wait rounds
// (rgpu_set_wait_limit).
__device__ __forceinline__ bool wait_chunk(WarpShared &ws, uint32_t parity, uint32_t limit) {
    const uint32_t a = smem_addr(&ws.mb);
    for (uint32_t it = 0; it < limit; it++) {
        uint32_t ok;
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (__any_sync(0xffffffffu, ok)) return true;
    }
    return false;
}

// adds an event at pixel p of the row to a difference array of 16-bit pairs
// (sums of packed 32-bit words: exact whatever the order, as the final
// differences fit 16 bits)
__device__ __forceinline__ void add_event(uint32_t *diff, uint32_t p, int32_t e0, int32_t e1) {
    const uint32_t d0 = (uint32_t)e0, d1 = (uint32_t)e1;
    const bool odd = (p & 1u) != 0u;
    atomicAdd(diff + (p >> 1), odd ? d0 << 16 : d0 + (d1 << 16));
    if (odd && d1) atomicAdd(diff + (p >> 1) + 1, d1);
}

// Scans a row's differences (two per word, WPL words per lane) into coverage
// bytes and zeroes them; `left` is the coverage just left of the row.  Returns
// the lanes whose pixels have any coverage.
// The prefix sums run on two 16-bit pixels per register, biased so that a half
// never borrows from the other: pair (a, b) times 0x10001 is (a, a + b), and
// the previous pair's upper half is added to both.
template <int WPL>
__device__ __forceinline__ uint32_t scan_row(uint32_t *diff, uint8_t *cov, int32_t left) {
    const int lane = threadIdx.x & 31;
    uint32_t v[WPL];
    uint32_t *d = diff + WPL * lane;
    if constexpr (WPL >= 4) {
#pragma unroll
        for (int k = 0; k < WPL; k += 4) {
            uint4 *q = reinterpret_cast<uint4 *>(d + k);
            const uint4 t = *q;
            *q = make_uint4(0, 0, 0, 0);
            v[k] = t.x; v[k + 1] = t.y; v[k + 2] = t.z; v[k + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < WPL; k++) {
            v[k] = d[k];
            d[k] = 0;
        }
    }
    if (lane == 0) diff[32 * WPL] = 0;
    constexpr uint32_t kBias = 0x4000u;
    uint32_t run = kBias * 0x10001u;
#pragma unroll
    for (int k = 0; k < WPL; k++) {
        v[k] = v[k] * 0x10001u + run;
        run = __byte_perm(v[k], 0u, 0x3232);
    }
    int32_t s = (int32_t)(run & 0xFFFFu) - (int32_t)kBias;
    const int32_t own = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += t;
    }
    const uint32_t add = (uint32_t)((s - own + left - (int32_t)kBias) & 0xFFFF) * 0x10001u;
    uint32_t any = 0;
#pragma unroll
    for (int k = 0; k < WPL; k++) {
        v[k] = __viaddmin_s16x2(v[k], add, 0x00FF00FFu);
        any |= v[k];
    }
    if constexpr (WPL >= 2) {
        uint32_t b[WPL / 2];
#pragma unroll
        for (int k = 0; k < WPL / 2; k++) b[k] = __byte_perm(v[2 * k], v[2 * k + 1], 0x6420);
        if constexpr (WPL == 2) reinterpret_cast<uint32_t *>(cov)[lane] = b[0];
        else if constexpr (WPL == 4) reinterpret_cast<uint2 *>(cov)[lane] = make_uint2(b[0], b[1]);
        else {
#pragma unroll
            for (int k = 0; k < WPL / 2; k += 4)
                reinterpret_cast<uint4 *>(cov)[(WPL / 8) * lane + k / 4] = make_uint4(b[k], b[k + 1], b[k + 2], b[k + 3]);
        }
    } else {
        reinterpret_cast<uint16_t *>(cov)[lane] = (uint16_t)(v[0] | v[0] >> 8);
    }
    return __ballot_sync(0xffffffffu, any != 0u);
}

// shade_groups for the paints and blend modes off its fast paths, one group a step
__device__ __forceinline__ void shade_groups_slow(uint32_t mask, int bits_sh, const PaintRec *paint, const GradRec *gr,
                                               uint32_t *px, const uint8_t *cov, int32_t lx0, int32_t ly) {
#pragma unroll 1
    for (; mask; mask &= mask - 1u) {
        const int g = (__ffs(mask) - 1) >> bits_sh;
        const uint32_t cv = cov[32 * g];
        if (cv) px[32 * g] = dev::shade_pixel(*paint, gr, lx0 + 32 * g, ly, cv, px[32 * g]);
    }
}

// Shades the groups `mask` of a row (bit g << bits_sh for group g: 32 pixels
// from 32 g on) with one fill, whose paint, stop positions and colour rows are in
// shared memory.  The common lowp paints (a solid or gradient colour, drawn source-over or, where
// opaque, source) run in loops of their own, two groups a step and without
// branches on the coverage (0 and 255 need none: the arithmetic leaves the
// pixel, or takes the colour, exactly); every other paint goes through
// shade_pixel.
__device__ __forceinline__ void shade_groups(uint32_t mask, int bits_sh, const uint4 *paint, const float4 *tv,
                                             const uint4 *rows, const GradRec *grads, uint32_t *px,
                                             const uint8_t *cov, int32_t lx0, int32_t ly) {
    const uint4 p0 = paint[0];
    const uint32_t kind = p0.x, blend = p0.y, flags = p0.z;
    if (flags & PAINT_SKIP) return;
    const bool source = blend == RGPU_BLEND_SOURCE;
    if (!(flags & PAINT_LOWP) || !(source || blend == RGPU_BLEND_SOURCE_OVER) || kind > 1) {
        shade_groups_slow(mask, bits_sh, reinterpret_cast<const PaintRec *>(paint), grads + p0.w, px, cov, lx0, ly);
        return;
    }
    const uint4 p1 = paint[1], p2 = paint[2];
    // the next two groups of the mask: their first pixels, and whether there are two
    int o[2];
    bool two;
    auto next = [&]() {
        o[0] = ((__ffs(mask) - 1) >> bits_sh) << 5;
        mask &= mask - 1u;
        two = mask != 0u;
        o[1] = two ? ((__ffs(mask) - 1) >> bits_sh) << 5 : o[0];
        mask &= mask - 1u;
    };
    uint32_t cv[2], d[2];
    // a clear of an aliased path is a source of its memset colour, whatever the
    // paint (its coverage is 0 or 255 only)
    if (kind == 0 || (flags & PAINT_MEMSET)) {
        uint32_t rb = __byte_perm(p1.x, p1.y, 0x5410), ga = __byte_perm(p1.x, p1.y, 0x7632);
        if (flags & PAINT_MEMSET) {  // the colour where the pixel is fully covered (the same, or a clear)
            rb = dev::pair_rb(p2.z);
            ga = dev::pair_ga(p2.z);
        }
#pragma unroll 1
        while (mask) {
            next();
#pragma unroll
            for (int u = 0; u < 2; u++) {
                cv[u] = cov[o[u]];
                d[u] = px[o[u]];
            }
            if (source) {
#pragma unroll
                for (int u = 0; u < 2; u++) d[u] = dev::lowp_source(rb, ga, cv[u], d[u]);
            } else {
#pragma unroll
                for (int u = 0; u < 2; u++) d[u] = dev::lowp_over(rb, ga, cv[u], d[u]);
            }
            px[o[0]] = d[0];
            if (two) px[o[1]] = d[1];
        }
        return;
    }
    // gradients: the transform, spread and stop positions in registers
    const uint32_t meta = p2.w, gflags = meta & 0xFFu, spread = (meta >> 8) & 0xFFu, gn = meta >> 16;
    const float g0 = __uint_as_float(p1.x), g1 = __uint_as_float(p1.y);
    const float g4 = __uint_as_float(p2.x), g5 = __uint_as_float(p2.y);
    const float y = (float)ly + 0.5f, yg2 = y * __uint_as_float(p1.z), yg3 = y * __uint_as_float(p1.w);
    const bool radial = (gflags & GRAD_RADIAL_SIMPLE) != 0, premul = (gflags & GRAD_PREMUL) != 0;
    const bool clamp = spread != RGPU_SPREAD_PAD || (gflags & GRAD_PAD_CLAMP) != 0;
    // stop positions (absent ones are NaN: no t is >= NaN) for the bisection;
    // nq quarters of them are in use
    const int nq = (gflags & GRAD_TWO_STOP) ? 0 : (gn > 8u ? 3 : (gn > 4u ? 2 : 1));
    float4 ta = make_float4(0.f, 0.f, 0.f, 0.f), tb = ta;
    if (nq >= 1) ta = tv[0];
    if (nq >= 2) tb = tv[1];
    const float xc = (float)lx0 + 0.5f;
#pragma unroll 1
    while (mask) {
        next();
        float t[2];
        uint32_t idx[2] = {0u, 0u};
#pragma unroll
        for (int u = 0; u < 2; u++) {
            cv[u] = cov[o[u]];
            d[u] = px[o[u]];
            t[u] = xc + (float)o[u];  // exact: integers and a half
        }
        if (radial) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const float tx = t[u] * g0 + yg2 + g4, ty = t[u] * g1 + yg3 + g5;
                t[u] = __fsqrt_rn(tx * tx + ty * ty);
            }
        } else {
#pragma unroll
            for (int u = 0; u < 2; u++) t[u] = t[u] * g0 + yg2 + g4;
        }
        if (spread == RGPU_SPREAD_REFLECT) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const float v = t[u] - 1.0f;
                t[u] = fabsf(v - 2.0f * floorf(v * 0.5f) - 1.0f);
            }
        } else if (spread == RGPU_SPREAD_REPEAT) {
#pragma unroll
            for (int u = 0; u < 2; u++) t[u] = t[u] - floorf(t[u]);
        }
        if (clamp) {
#pragma unroll
            for (int u = 0; u < 2; u++) t[u] = fminf(fmaxf(t[u], 0.0f), 1.0f);
        }
        // the interval: how many of the stop positions 1 .. are <= t, by
        // bisection (the positions are non-decreasing)
        if (nq == 1) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const bool c1 = t[u] >= ta.z;
                idx[u] = (c1 ? 2u : 0u) + (uint32_t)(t[u] >= (c1 ? ta.w : ta.y));
            }
        } else if (nq >= 2) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const bool c1 = t[u] >= tb.x;
                const bool c2 = t[u] >= (c1 ? tb.z : ta.z);
                const float q = c1 ? (c2 ? tb.w : tb.y) : (c2 ? ta.w : ta.y);
                idx[u] = (c1 ? 4u : 0u) + (c2 ? 2u : 0u) + (uint32_t)(t[u] >= q);
            }
            if (nq == 3) {
                const float4 tc = tv[2];
#pragma unroll
                for (int u = 0; u < 2; u++)
                    if (t[u] >= tc.x) {
                        const bool c3 = t[u] >= tc.z;
                        idx[u] = 8u + (c3 ? 2u : 0u) + (uint32_t)(t[u] >= (c3 ? tc.w : tc.y));
                    }
            }
        }
        uint32_t rb[2], ga[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const float4 *row = reinterpret_cast<const float4 *>(rows) + 2 * idx[u];
            const float4 f = row[0], b = row[1];
            const uint4 c = dev::lowp_bits(t[u] * f.x + b.x, t[u] * f.y + b.y, t[u] * f.z + b.z, t[u] * f.w + b.w);
            rb[u] = __byte_perm(c.x, c.z, 0x1410);
            ga[u] = __byte_perm(c.y, c.w & 0xFFu, 0x1410);
        }
        if (premul) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const uint32_t a = ga[u] >> 16;
                rb[u] = dev::div255_2(rb[u] * a);
                ga[u] = __byte_perm(ga[u] * a + 0xFFu, a, 0x5451);
            }
        }
        if (source) {
#pragma unroll
            for (int u = 0; u < 2; u++) d[u] = dev::lowp_source(rb[u], ga[u], cv[u], d[u]);
        } else {
#pragma unroll
            for (int u = 0; u < 2; u++) d[u] = dev::lowp_over(rb[u], ga[u], cv[u], d[u]);
        }
        px[o[0]] = d[0];
        if (two) px[o[1]] = d[1];
    }
}

// Coverage of layer pixel (px, py) from one hairline span (tiny-skia
// scan/hairline_aa.rs: the step k on the pixel's major coordinate, the two
// pixels its blitter touches, alpha scaled by the end-cap fraction); 0 = no
// blit.  A vline whose two columns coincide (x in [0, 1)) blits each pixel
// twice: the host emits it as two spans, the second (HAIR_SECOND) carrying
// only the second blit.
static_assert(sizeof(HairSpan) == 32, "a hairline span is two int4: setup, then its pixel rect");

// A read-only 16-byte load the compiler keeps in place: hoisting a span's
// fields out of the per-pixel loop would hold eight more registers across it.
__device__ __forceinline__ int4 ld_span(const int4 *p) {
    int4 r;
    asm volatile("ld.global.nc.v4.s32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w)
                 : "l"(p));
    return r;
}

__device__ __forceinline__ uint32_t hair_cov(const HairSpan *hsp, int32_t px, int32_t py) {
    const int4 r = ld_span(reinterpret_cast<const int4 *>(hsp) + 1);
    if (px < r.x || py < r.y || px >= r.z || py >= r.w) return 0u;
    const int4 q = ld_span(reinterpret_cast<const int4 *>(hsp));
    const int32_t istart = q.x, f0 = q.y, slope = q.z;
    const uint32_t pack = (uint32_t)q.w, kind = pack & 3u;
    const int32_t n = (int32_t)(pack >> 16);
    const int32_t k = (kind < 2 ? px : py) - istart, minor = kind < 2 ? py : px;
    const int32_t cv = slope >= 0 ? max(f0, 0) + k * slope : max(f0 + k * slope, 0);
    const int32_t hi = cv >> 16;
    const uint32_t a = (uint32_t)(cv >> 8) & 0xFFu;
    const uint32_t stop = (pack >> 9) & 127u;
    const uint32_t mod = k == 0 ? ((pack >> 2) & 127u) : ((k == n - 1 && stop > 0) ? stop : 64u);
    const uint32_t sa = (a * mod) >> 6, sna = ((255u - a) * mod) >> 6;
    const int32_t lo = max(hi, 1) - 1;
    if (kind == 0) {  // hline: row hi, then row hi - 1 (when hi >= 1)
        if (minor == hi) return sa;
        return (hi >= 1 && minor == hi - 1) ? sna : 0u;
    }
    if (kind == 2) {  // vline: column hi, then column max(hi, 1) - 1
        if (pack & HAIR_SECOND) return minor == lo ? sna : 0u;
        if (minor == hi) return sa;
        return (minor == lo && lo != hi) ? sna : 0u;
    }
    // horish / vertish: lo then lo + 1
    return minor == lo ? sna : (minor == lo + 1 ? sa : 0u);
}

// A hairline stroke on the item's row: its spans in order, each lane on its own
// pixels, so blits to one pixel keep their order.  The warp tests 32 span rects
// at a time against the row.
__device__ __forceinline__ void hairline(const HairRec &hr, const PaintRec &pr, const HairSpan *spans, const GradRec *grads,
                                      uint32_t *px, int32_t x0, int32_t x1, int32_t cy) {
    const int lane = threadIdx.x & 31;
    const int32_t lx0 = x0 - hr.ox, lx1 = x1 - hr.ox, ly = cy - hr.oy;
    if (hr.x1 <= lx0 || hr.x0 >= lx1 || hr.y1 <= ly || hr.y0 > ly) return;
    const GradRec *gr = grads + pr.grad;
    for (uint32_t base = 0; base < hr.span_cnt; base += 32) {
        const uint32_t s = base + (uint32_t)lane;
        bool meets = false;
        if (s < hr.span_cnt) {
            const int4 r = __ldg(reinterpret_cast<const int4 *>(spans + hr.span_off + s) + 1);
            meets = !(r.z <= lx0 || r.x >= lx1 || r.w <= ly || r.y > ly);
        }
        for (uint32_t hm = __ballot_sync(0xffffffffu, meets); hm; hm &= hm - 1) {
            const HairSpan *hs = spans + hr.span_off + base + (uint32_t)(__ffs(hm) - 1);
#pragma unroll 1
            for (int32_t lx = lx0 + lane; lx < lx1; lx += 32) {
                const uint32_t cv = hair_cov(hs, lx, ly);
                uint32_t &dst = px[lx - lx0 - lane];
                if (cv) dst = dev::shade_pixel(pr, gr, lx, ly, cv, dst);
            }
        }
    }
}

// One draw's coverage of the row piece from event pixel x0 on, from its n events (the first
// 32 in shared memory, all of them at `list`): the coverage bytes, and the mask
// of covered groups (bit g << bits of a group's lanes).
__device__ __forceinline__ uint32_t make_row(const uint32_t *firsts32, const uint32_t *list, uint32_t n, int32_t x0,
                                             uint32_t row_w, uint32_t *diff, uint8_t *cov) {
    const uint32_t lane = threadIdx.x & 31u;
    int32_t left = 0;
    for (uint32_t k = lane; k < n; k += 32u) {
        const uint32_t e = k < 32u ? firsts32[k] : __ldg(list + k);
        const int32_t p = dev::event_pixel(e) - x0, d0 = dev::event_d0(e), d1 = dev::event_d1(e);
        if (p < 0) left += d0 + d1;
        else if (p < (int32_t)row_w) add_event(diff, (uint32_t)p, d0, d1);
    }
    left = __reduce_add_sync(0xffffffffu, left);
    __syncwarp();
    uint32_t groups;
    switch (row_w) {
    case 64: groups = scan_row<1>(diff, cov, left); break;
    case 128: groups = scan_row<2>(diff, cov, left); break;
    case 256: groups = scan_row<4>(diff, cov, left); break;
    default: groups = scan_row<8>(diff, cov, left); break;
    }
    __syncwarp();
    // one bit per group: the lowest of its lanes' bits
    groups |= groups >> 1;
    if (row_w <= 256) groups |= groups >> 2;
    if (row_w <= 128) groups |= groups >> 4;
    if (row_w <= 64) groups |= groups >> 8;
    const uint32_t firsts = row_w == 512 ? 0x55555555u : row_w == 256 ? 0x11111111u
                          : row_w == 128 ? 0x01010101u : 0x00010001u;
    return groups & firsts;
}

__global__ void __launch_bounds__(kThreads, kMinBlocks)
k_raster(uint32_t max_row_w, const StreamRec *streams, const WorkItem *items, uint32_t nitems, uint32_t *item_counter,
         const Cmd *cmds, const DrawRec *draws, const PaintRec *paints, const GradRec *grads, const LayerRec *layers,
         const uint32_t *bin_offsets, const uint32_t *headers, const uint32_t *events, uint32_t *stack_scratch,
         uint32_t stack_depth, const HairRec *hairs, const HairSpan *hair_spans, uint32_t *err, uint32_t wait_limit,
         uint32_t withhold) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    unsigned char *mem = smem_raw + (size_t)warp * warp_bytes(max_row_w);
    WarpShared &ws = *reinterpret_cast<WarpShared *>(mem);
    uint32_t *diff = reinterpret_cast<uint32_t *>(mem + sizeof(WarpShared));
    uint32_t *px = diff + max_row_w / 2 + 4 + lane;          // this lane's pixel of each group
    uint8_t *cov = reinterpret_cast<uint8_t *>(px - lane + max_row_w);
    // neighbouring items go to different CTAs, so that few items spread over all SMs
    const uint32_t gwarp = (uint32_t)warp * gridDim.x + blockIdx.x, nwarps = gridDim.x * kWarps;
    uint32_t *stack = stack_scratch + (size_t)gwarp * stack_depth * max_row_w + lane;
    for (uint32_t k = (uint32_t)lane; k < max_row_w / 2 + 4; k += 32) diff[k] = 0;
    if (lane == 0) {
        mb_init(&ws.mb, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");  // the copies see it initialised
    }
    uint32_t copies = 0;  // command copies waited for so far
    __syncthreads();
    for (uint32_t idx = gwarp; idx < nitems;) {
        // the next item, taken ahead of time
        uint32_t fetched = 0;
        if (lane == 0) fetched = nwarps + atomicAdd(item_counter, 1u);
        const WorkItem wi = items[idx];
        const StreamRec &st = streams[wi.stream];
        const Cmd *scmds = cmds + st.cmd_off;
        const uint32_t ncmd = st.cmd_cnt;
        // the first commands (failure-detection test hook: CTA 0 never asks for
        // its first ones, so the bounded wait for them must run out)
        if (lane == 0 && ncmd && !(withhold && blockIdx.x == 0 && copies == 0))
            copy_chunk(ws, 0, scmds, min(ncmd, (uint32_t)kChunk));
        const uint32_t row_w = st.row_w;
        const int bits_sh = 10 - (31 - __clz(row_w));       // lanes per group of the scan, log2
        const int ngroup = (wi.x1 - wi.x0 + 31) >> 5;
        const uint32_t in_piece = 0xFFFFFFFFu >> (32 - (ngroup << bits_sh));
        const int32_t cy = (int32_t)wi.row, x0 = wi.x0, x1 = wi.x1;
        if (lane == 0) ws.first = x0 - st.x_lo;
        auto out_row = [&]() {
            return reinterpret_cast<uint32_t *>(reinterpret_cast<uint8_t *>((uintptr_t)st.out_ptr) +
                                                (size_t)cy * st.out_stride) + x0 + lane;
        };
        // f(first pixel of the group, the lane's pixel, its x) over the row's groups
        auto each_group = [&](auto f) {
#pragma unroll 2
            for (int g = 0; g < ngroup; g++) f(32 * g, px[32 * g], x0 + 32 * g + lane);
        };
        {
            const uint32_t *out = out_row();
            each_group([&](int o, uint32_t &p, int32_t x) { p = x < x1 ? out[o] : 0u; });
        }
        auto rect_at = [&](int32_t d) {
            if (d == 0) return make_int4(0, 0, st.out_w, st.out_h);
            const LayerRec &L = layers[st.layer_off + ws.rect[d]];
            return make_int4(L.x, L.y, L.w, L.h);
        };
        int32_t depth = 0;
        const uint32_t slot0 = st.bin_off + (wi.row - (uint32_t)st.row_lo) * st.draw_cnt;
        const uint32_t row_slot = slot0 - st.draw_off;  // + draw: its slot
        // the row's lists start here (offsets and slots each fit 32 bits, their sum may not)
        const uint32_t off0 = __ldg(bin_offsets + slot0);
        const uint32_t row_loc = off0 + slot0;
        const uint32_t *row_events = events + 4ull * ((unsigned long long)off0 + slot0);
        bool stop = false, failed = false;
        for (uint32_t ci = 0, buf = 0; ci < ncmd && !stop; ci += kChunk, buf ^= 1u) {
            if (!wait_chunk(ws, copies & 1u, wait_limit)) {
                // Nothing of this warp's copies may land after it has gone: wait
                // once more, then leave the item unfinished.  Other warps do not
                // depend on this one.
                if (lane == 0) atomicOr(err, 16u);
                wait_chunk(ws, copies & 1u, wait_limit);
                return;
            }
            copies++;
            __syncwarp();  // every lane is past the other buffer's commands
            if (lane == 0 && ci + kChunk < ncmd) copy_chunk(ws, buf ^ 1u, scmds + ci + kChunk, min(ncmd - ci - kChunk, (uint32_t)kChunk));
            // 32 commands at a time, one per lane; fills that do not touch the
            // piece are never visited
            const Cmd *chunk = ws.chunk[buf];
            uint32_t my_op = kNone, n = 0, loc = 0;  // command, number of events, place of their list
            if (ci + (uint32_t)lane < ncmd) {
                my_op = chunk[lane].op;
                if (my_op == CMD_FILL || my_op == CMD_APPLY_REGION) {
                    const uint32_t slot = row_slot + chunk[lane].a, h = __ldg(headers + slot);
                    n = h >> 20;
                    if (n == dev::kManyEvents) n = h & dev::kMaxEvents;
                    else if ((int32_t)(h >> 10 & 0x3FFu) > (ws.first + (x1 - x0) - 1) >> 5 || (int32_t)(h & 0x3FFu) < ws.first >> 5) n = 0;
                    if (n) loc = __ldg(bin_offsets + slot) + slot - row_loc;
                }
            }
            auto list_of = [&](int s) { return row_events + 4ull * __shfl_sync(0xffffffffu, loc, s); };
            uint32_t todo = __ballot_sync(0xffffffffu, my_op != kNone && (my_op != CMD_FILL || n != 0u));
            const uint32_t with_events = __ballot_sync(0xffffffffu, n != 0u);
            // copies what the first fill of `from` needs into slot `par`
            uint32_t par = 0;
            auto load_fill = [&](uint32_t from) {
                const int s = __ffs(from & with_events) - 1;
                if (s >= 0) {
                    FillSlot &f = ws.fill[par];
                    const Cmd &c = chunk[s];
                    const uint32_t g = __float_as_uint(c.f);  // the gradient, if any
                    const uint32_t *list = list_of(s);
                    if ((uint32_t)lane < __shfl_sync(0xffffffffu, n, s)) cp_async<4>(&f.events[lane], list + lane);
                    if (lane < 24) {
                        if (g != kNone) cp_async<16>(&f.rows[lane], reinterpret_cast<const uint4 *>(grads[g].iv) + lane);
                    } else if (lane < 27) {
                        if (g != kNone) cp_async<16>(&f.stops[lane - 24], reinterpret_cast<const float4 *>(grads[g].t) + (lane - 24));
                    } else if (lane < 30) {
                        cp_async<16>(&f.paint[lane - 27], reinterpret_cast<const uint4 *>(paints + c.b) + (lane - 27));
                    } else if (lane == 30) {
                        cp_async<8>(&f.org, &draws[c.a].ox);
                    }
                }
                cp_commit();
            };
            load_fill(todo);
            while (todo) {
                const int cl = __ffs(todo) - 1;
                const uint32_t op = __shfl_sync(0xffffffffu, my_op, cl);
                if (op == CMD_FILL || op == CMD_APPLY_REGION) {
                    todo &= todo - 1u;
                    const uint32_t cnt = __shfl_sync(0xffffffffu, n, cl);
                    const FillSlot &f = ws.fill[par];
                    uint32_t groups = 0;
                    if (cnt) {
                        const uint32_t *list = list_of(cl);
                        par ^= 1u;
                        load_fill(todo);
                        cp_wait<1>();  // all but the copies just asked for
                        __syncwarp();
                        groups = make_row(f.events, list, cnt, ws.first, row_w, diff, cov) & in_piece;
                    }
                    if (op == CMD_FILL) {
                        if (groups)
                            shade_groups(groups, bits_sh, f.paint, f.stops, f.rows, grads, px, cov + lane,
                                         x0 + lane - f.org.x, cy - f.org.y);
                    } else {
                        // region mask: Mask::fill_path coverage (lerp 0 -> 255), then apply_mask
                        const int4 t = rect_at(depth);
                        const bool row_in = cy >= t.y && cy < t.y + t.w;
                        each_group([&](int off, uint32_t &p, int32_t x) {
                            if (!(row_in && x < x1 && x >= t.x && x < t.x + t.z)) return;
                            const uint32_t cv = groups ? cov[off + lane] : 0u;
                            const uint32_t mv = cv == 255 ? 255u
                                                          : (uint32_t)dev::div255((uint32_t)dev::sat_u16(((float)cv * dev::kInv255) * 255.0f + 0.5f) * 255u);
                            p = dev::mask_pixel(p, mv);
                        });
                    }
                    __syncwarp();  // the coverage bytes and the slot have been read
                    continue;
                }
                todo &= todo - 1u;
                if (op == CMD_END) {
                    stop = true;
                    break;
                }
                const uint32_t ca = chunk[cl].a, cb = chunk[cl].b;
                if (op == CMD_HAIR) {
                    const HairRec &hr = hairs[ca];
                    __syncwarp();  // the previous hairline's pixels are done with the paint
                    if (lane < (int)(sizeof(PaintRec) / 4))
                        reinterpret_cast<uint32_t *>(&ws.hair_paint)[lane] =
                            __ldg(reinterpret_cast<const uint32_t *>(&paints[hr.paint]) + lane);
                    __syncwarp();
                    if (!(ws.hair_paint.flags & PAINT_SKIP)) hairline(hr, ws.hair_paint, hair_spans, grads, px, x0, x1, cy);
                } else if (op == CMD_PUSH) {
                    if (depth + 1 >= kMaxDepth || (uint32_t)depth >= stack_depth) {
                        if (lane == 0) atomicOr(err, 4u);
                        stop = failed = true;
                        break;
                    }
                    uint32_t *lvl = stack + (size_t)depth * max_row_w;
                    depth++;
                    __syncwarp();
                    if (lane == 0) ws.rect[depth] = ca;
                    __syncwarp();
                    const LayerRec &L = layers[st.layer_off + ca];
                    const uint32_t init = cb == 1 ? 0xFF000000u : 0u;
                    const int32_t Lx = L.x, Ly = L.y, Lw = L.w;
                    const bool row_in = cy >= Ly && cy < Ly + L.h;
                    const uint32_t *src = (cb == 2 && L.buf) ? (const uint32_t *)(uintptr_t)L.buf : nullptr;
                    each_group([&](int off, uint32_t &p, int32_t x) {
                        lvl[off] = p;
                        uint32_t v = 0u;
                        if (row_in && x >= Lx && x < Lx + Lw) v = src ? src[(size_t)(cy - Ly) * Lw + (x - Lx)] : init;
                        p = v;
                    });
                } else if (op == CMD_POP_COMPOSITE || op == CMD_POP_CLIP || op == CMD_POP_MASK) {
                    if (depth == 0) {
                        if (lane == 0) atomicOr(err, 4u);
                        stop = failed = true;
                        break;
                    }
                    const float cf = chunk[cl].f;
                    const int4 t = rect_at(depth);
                    depth--;
                    const uint32_t *lvl = stack + (size_t)depth * max_row_w;
                    const int4 p4 = rect_at(depth);
                    const bool in_rows = cy >= t.y && cy < t.y + t.w && cy >= p4.y && cy < p4.y + p4.w;
                    each_group([&](int off, uint32_t &p, int32_t x) {
                        uint32_t parent = lvl[off];
                        const uint32_t child = p;
                        if (in_rows && x >= t.x && x < t.x + t.z && x >= p4.x && x < p4.x + p4.z) {
                            if (op == CMD_POP_COMPOSITE) parent = dev::composite_pixel(child, parent, cf, cb);
                            else if (op == CMD_POP_CLIP) parent = dev::mask_pixel(parent, 255u - dev::ch(child, 3));
                            else parent = dev::mask_pixel(parent, dev::mask_value(child, cb == 0));
                        }
                        p = parent;
                    });
                } else if (op == CMD_CLEAR) {
                    const int4 t = rect_at(depth);
                    const bool row_in = cy >= t.y && cy < t.y + t.w;
                    each_group([&](int, uint32_t &p, int32_t x) {
                        if (row_in && x >= t.x && x < t.x + t.z) p = 0u;
                    });
                }
            }
            cp_wait<0>();
            // a chunk asked for after the last command read is waited for, so
            // that the buffers are the next item's
            if (stop && ci + kChunk < ncmd) {
                if (!wait_chunk(ws, copies & 1u, wait_limit)) {
                    if (lane == 0) atomicOr(err, 16u);
                    return;
                }
                copies++;
            }
            __syncwarp();  // the commands have been read
        }
        if (depth != 0 && !failed && lane == 0) atomicOr(err, 8u);
        if (!failed) {
            uint32_t *out = out_row();
            each_group([&](int o, uint32_t &p, int32_t x) {
                if (x < x1) out[o] = p;
            });
        }
        idx = __shfl_sync(0xffffffffu, fetched, 0);
    }
}

// launch arguments of the failure-detection controls (read at launch time; a
// captured graph keeps the values it was captured with)
constexpr uint32_t kDefaultWaitLimit = 1u << 22;
uint32_t g_wait_limit = kDefaultWaitLimit;
uint32_t g_withhold = 0;

}  // namespace

size_t raster_smem_bytes(uint32_t row_w) { return kWarps * warp_bytes(row_w); }
int raster_warps() { return kWarps; }

cudaError_t raster_init() {
    return cudaFuncSetAttribute(k_raster, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)raster_smem_bytes(kRasterMaxRow));
}

cudaError_t launch_raster(uint32_t row_w, uint32_t grid, uint32_t stack_depth, const StreamRec *streams,
                          const WorkItem *items, uint32_t nitems, uint32_t *item_counter, const Cmd *cmds,
                          const DrawRec *draws, const PaintRec *paints, const GradRec *grads, const LayerRec *layers,
                          const uint32_t *bin_offsets, const uint32_t *headers, const uint32_t *events,
                          uint32_t *stack, const HairRec *hairs, const HairSpan *hair_spans, uint32_t *err,
                          cudaStream_t s) {
    k_raster<<<grid, kThreads, raster_smem_bytes(row_w), s>>>(
        row_w, streams, items, nitems, item_counter, cmds, draws, paints, grads, layers, bin_offsets, headers, events,
        stack, stack_depth, hairs, hair_spans, err, g_wait_limit, g_withhold);
    return cudaGetLastError();
}

void raster_set_wait_limit(uint32_t rounds) { g_wait_limit = rounds ? rounds : kDefaultWaitLimit; }
uint32_t raster_wait_limit() { return g_wait_limit; }
void raster_set_withhold(bool on) { g_withhold = on ? 1u : 0u; }

int raster_max_blocks_per_sm(uint32_t row_w) {
    int n = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_raster, kThreads, raster_smem_bytes(row_w));
    if (e != cudaSuccess || n < 1) { cudaGetLastError(); n = 1; }
    return n;
}

}  // namespace rgpu
