// Differentiable soft-coverage renderer: a forward pass and a hand-written
// adjoint for batches of scenes of closed cubic paths (no counterpart in the
// reference; resvg renders hard-edged, non-differentiable coverage).
//
// Forward, per scene (premultiplied RGBA in FP32):
//   * a path of n cubics is closed by construction: its 3n points are the
//     start S, then (control 1, control 2, end) per cubic, where the last
//     cubic ends at S; every cubic is flattened into kFlat lines at uniform t
//     (vertex list: P_c(i/kFlat), i = 0..kFlat-1, for each cubic c; the line
//     from the last vertex back to the first closes the loop);
//   * soft coverage of pixel (px, py) by a path is c = min(|A|, 1), where A is
//     the winding-weighted area of the pixel: for every line, the integral over
//     y in [py, py+1] of the part of the pixel row right of the line, signed by
//     the line's y direction; for a line clipped to the row, from (xl, yl) to
//     (xh, yh) with sdy = +-(yh - yl), the pixel gets sdy * G(xl - px, xh - px)
//     with G(a, b) the mean of clamp(1 - x, 0, 1) over x from a to b, written
//     in closed, well-conditioned form per case;
//   * paints (at pixel centres): a straight RGBA colour or a linear gradient of
//     4 stops (pad spread, offsets ascending), its alpha multiplied by the
//     path's opacity, premultiplied after interpolation; paths composite
//     source-over in order from transparent;
//   * a Gaussian blur of the composite, separable, radius kRadius, weights
//     exp(-j^2 / 2 sigma^2) normalised over [-kRadius, kRadius], zero outside
//     the canvas.
// Adjoint: given dL/d(blurred), the blur is transposed (the same symmetric
// filter) and d sigma is accumulated from the derivative weights; then the areas
// are computed again, the composite is run and reversed path by path,
// paint-parameter gradients are reduced per warp, and each crossing line's
// gradient is the sum over its pixels of the area function's derivatives in the
// clipped ends, chained to the line's ends by dual numbers; vertex gradients are
// chained to control points with the Bernstein weights of the flattening.
#include <cuda_runtime.h>
#include <stdint.h>
#include <algorithm>
#include <cmath>
#include <mutex>
#include <type_traits>
#include "kernels.h"
#include "resvg_gpu.h"

namespace rgpu {
void set_last_error_message(const char *msg);  // render.cpp
bool forced_alloc_failure();                   // render.cpp

namespace soft {
namespace {

constexpr int kFlat = 16;      // lines per cubic
constexpr int kMaxWidth = 1024;
constexpr int kRadius = 12;    // blur radius (3 x the largest sigma of the workload)
constexpr int kMaxCross = 512; // crossing lines per (path, row): as many are reported as RGPU_ERR_CAPACITY

// ---- forward-mode dual numbers over the 4 endpoint coordinates of a line
struct D4 {
    float v, d[4];
};
__device__ __forceinline__ float val(float x) { return x; }
__device__ __forceinline__ float val(const D4 &x) { return x.v; }
__device__ __forceinline__ D4 mk(float v) { D4 r; r.v = v; r.d[0] = r.d[1] = r.d[2] = r.d[3] = 0.f; return r; }
__device__ __forceinline__ D4 operator+(const D4 &a, const D4 &b) {
    D4 r; r.v = a.v + b.v;
#pragma unroll
    for (int i = 0; i < 4; i++) r.d[i] = a.d[i] + b.d[i];
    return r;
}
__device__ __forceinline__ D4 operator-(const D4 &a, const D4 &b) {
    D4 r; r.v = a.v - b.v;
#pragma unroll
    for (int i = 0; i < 4; i++) r.d[i] = a.d[i] - b.d[i];
    return r;
}
__device__ __forceinline__ D4 operator*(const D4 &a, const D4 &b) {
    D4 r; r.v = a.v * b.v;
#pragma unroll
    for (int i = 0; i < 4; i++) r.d[i] = a.d[i] * b.v + a.v * b.d[i];
    return r;
}
__device__ __forceinline__ D4 operator/(const D4 &a, const D4 &b) {
    D4 r; r.v = a.v / b.v;
    const float ib2 = 1.0f / (b.v * b.v);
#pragma unroll
    for (int i = 0; i < 4; i++) r.d[i] = (a.d[i] * b.v - a.v * b.d[i]) * ib2;
    return r;
}
__device__ __forceinline__ D4 operator-(float a, const D4 &b) {
    D4 r; r.v = a - b.v;
#pragma unroll
    for (int i = 0; i < 4; i++) r.d[i] = -b.d[i];
    return r;
}
__device__ __forceinline__ D4 operator*(const D4 &a, float b) {
    D4 r; r.v = a.v * b;
#pragma unroll
    for (int i = 0; i < 4; i++) r.d[i] = a.d[i] * b;
    return r;
}

template <class T> __device__ __forceinline__ T cst(float v);
template <> __device__ __forceinline__ float cst<float>(float v) { return v; }
template <> __device__ __forceinline__ D4 cst<D4>(float v) { return mk(v); }

// Mean of clamp(1 - x, 0, 1) over x running linearly from a to b.
__device__ __forceinline__ float mean_right(float a, float b) {
    if (a > b) { float t = a; a = b; b = t; }
    if (b <= 0.0f) return 1.0f;
    if (a >= 1.0f) return 0.0f;
    if (a >= 0.0f && b <= 1.0f) return 1.0f - (a + b) * 0.5f;
    if (a < 0.0f && b <= 1.0f) return 1.0f - (b * b) / ((b - a) * 2.0f);
    if (a >= 0.0f) return ((1.0f - a) * (1.0f - a)) / ((b - a) * 2.0f);
    return (0.5f - a) / (b - a);
}

// A line from (x0, y0) to (x1, y1) clipped to the row [py, py + 1]:
// (xl, xh) the x at the clipped ends and sdy the signed clipped height.
// Returns false when nothing of the line lies in the row.
template <class T>
__device__ __forceinline__ bool clip_row(T x0, T y0, T x1, T y1, float py, T *xl, T *xh, T *sdy) {
    if (val(y0) == val(y1)) return false;
    const float dir = val(y1) > val(y0) ? 1.0f : -1.0f;
    T xa = x0, ya = y0, xb = x1, yb = y1;
    if (dir < 0.0f) { xa = x1; ya = y1; xb = x0; yb = y0; }
    if (!(val(ya) < py + 1.0f && val(yb) > py)) return false;
    T ylo, yhi;
    if (val(ya) >= py) { ylo = ya; *xl = xa; }
    else { ylo = cst<T>(py); *xl = xa + (xb - xa) * ((py - ya) / (yb - ya)); }
    if (val(yb) <= py + 1.0f) { yhi = yb; *xh = xb; }
    else { yhi = cst<T>(py + 1.0f); *xh = xa + (xb - xa) * (((py + 1.0f) - ya) / (yb - ya)); }
    if (!(val(yhi) > val(ylo))) return false;
    *sdy = (yhi - ylo) * dir;
    return true;
}

// ---- paints
struct PaintOut {
    float r, g, b, a;  // straight colour at the pixel, alpha times the path's opacity
    float raw_a;       // the paint's alpha before the opacity
    float op;          // the path's opacity
    int seg;           // gradient: stop interval (-1: below first, 3: at/above last), solid: -2
    float w, t;        // interpolation weight and gradient parameter
};

__device__ __forceinline__ PaintOut eval_paint_raw(const rgpu_soft_batch &B, uint32_t j, float x, float y);

__device__ __forceinline__ PaintOut eval_paint(const rgpu_soft_batch &B, uint32_t j, float x, float y) {
    PaintOut o = eval_paint_raw(B, j, x, y);
    o.op = B.opacity ? B.opacity[j] : 1.0f;
    o.raw_a = o.a;
    o.a = o.a * o.op;
    return o;
}

__device__ __forceinline__ PaintOut eval_paint_raw(const rgpu_soft_batch &B, uint32_t j, float x, float y) {
    PaintOut o;
    o.w = 0.0f; o.t = 0.0f;
    if (B.paint_kind[j] == 0) {
        const float4 c = reinterpret_cast<const float4 *>(B.colors)[j];
        o.r = c.x; o.g = c.y; o.b = c.z; o.a = c.w; o.seg = -2;
        return o;
    }
    const float4 ln = reinterpret_cast<const float4 *>(B.grad_line)[j];
    const float dx = ln.z - ln.x, dy = ln.w - ln.y;
    const float len2 = dx * dx + dy * dy;
    float t = len2 > 0.0f ? ((x - ln.x) * dx + (y - ln.y) * dy) / len2 : 0.0f;
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    o.t = t;
    const float *off = B.stop_offsets + 4 * (size_t)j;
    const float4 *sc = reinterpret_cast<const float4 *>(B.stop_colors) + 4 * (size_t)j;
    if (t < off[0]) { const float4 c = sc[0]; o.r = c.x; o.g = c.y; o.b = c.z; o.a = c.w; o.seg = -1; return o; }
    if (t >= off[3]) { const float4 c = sc[3]; o.r = c.x; o.g = c.y; o.b = c.z; o.a = c.w; o.seg = 3; return o; }
    int i = 0;
    if (t >= off[1]) i = 1;
    if (t >= off[2]) i = 2;
    const float span = off[i + 1] - off[i];
    const float w = span > 0.0f ? (t - off[i]) / span : 1.0f;
    const float4 c0 = sc[i], c1 = sc[i + 1];
    o.r = c0.x + w * (c1.x - c0.x);
    o.g = c0.y + w * (c1.y - c0.y);
    o.b = c0.z + w * (c1.z - c0.z);
    o.a = c0.w + w * (c1.w - c0.w);
    o.seg = i; o.w = w;
    return o;
}

__device__ __forceinline__ uint32_t path_vbase(const rgpu_soft_batch &B, uint32_t j) { return kFlat * B.seg_offset[j]; }
__device__ __forceinline__ uint32_t path_nverts(const rgpu_soft_batch &B, uint32_t j) {
    return kFlat * (B.seg_offset[j + 1] - B.seg_offset[j]);
}

// ---- work split
// Areas and line gradients are independent per (row, path): a warp each.  The
// composite is a chain over the paths but independent per pixel: a warp per few
// groups of 32 pixels of a row.  Between them go, per (row, path), the areas (in
// the adjoint later dL/dA), the colours under the path, and a mask of the
// groups the path covers.  The scenes, and the rows of a scene that is too large
// by itself, are taken in slices of bounded scratch.
// On 16 scenes of 64 paths on 256^2 pixels: areas 0.32 ms, composite 0.15 ms, its
// reverse 0.56 ms, line gradients 0.32 ms.  (One CTA per row doing all of it in
// turn, with a block barrier for every step of every path, took 1.10 ms forward
// and 5.42 ms for the adjoint.)
struct Slice {
    uint32_t s0, scenes;  // scenes of the batch,
    uint32_t row0, rows;  // these rows of each
    uint32_t ng;          // 32-pixel groups per row
    float *area;          // [scene, row][path][32 ng]
    float4 *under;        // adjoint: the colours under each path, likewise
    uint32_t *mask;       // [scene, row][path]
};

constexpr int kRowWarps = 8;  // warps per CTA of the row kernels, at most

// shared memory of a warp of the row kernels: two words per pixel (padded, see
// at()) and the crossing lines being collected
struct RowMem {
    uint32_t *a, *b;
    float4 *list;  // (xl, xh, sdy, line index as float bits)
    int esh;       // log2 of the pixels a lane scans
    // a word per run of 2^esh pixels is skipped, so that the lanes' runs start in different banks
    __device__ __forceinline__ int at(int x) const { return x + (x >> esh); }
};
__host__ __device__ constexpr int row_esh(uint32_t ng) {
    int e = 0;
    while ((1u << e) < ng) e++;
    return e;
}
__host__ __device__ constexpr size_t row_words(uint32_t ng) { return ((size_t)(32u << row_esh(ng)) + 36) & ~(size_t)3; }
__host__ __device__ constexpr size_t row_bytes(uint32_t ng) { return 2 * row_words(ng) * 4 + 64 * sizeof(float4); }
__device__ __forceinline__ RowMem row_mem(unsigned char *smem, uint32_t ng) {
    unsigned char *m = smem + (threadIdx.x >> 5) * row_bytes(ng);
    RowMem r;
    r.list = reinterpret_cast<float4 *>(m);
    r.a = reinterpret_cast<uint32_t *>(m + 64 * sizeof(float4));
    r.b = r.a + row_words(ng);
    r.esh = row_esh(ng);
    return r;
}

// Calls f(xl, xh, sdy, line) for the lines of path j that cross row py, up to 32
// at a time, one per lane (every lane calls; `valid` tells).  Returns their number.
template <class F>
__device__ __forceinline__ uint32_t for_crossings(const RowMem &rm, const float2 *verts, uint32_t nv, float py, F f) {
    const int lane = threadIdx.x & 31;
    uint32_t n = 0, total = 0;
    for (uint32_t base = 0; base < nv; base += 32) {
        const uint32_t s = base + (uint32_t)lane;
        float xl = 0.f, xh = 0.f, sdy = 0.f;
        bool hit = false;
        if (s < nv) {
            const float2 a = verts[s], b = verts[s + 1 < nv ? s + 1 : 0];
            hit = clip_row<float>(a.x, a.y, b.x, b.y, py, &xl, &xh, &sdy);
        }
        const uint32_t m = __ballot_sync(0xffffffffu, hit);
        if (hit) rm.list[n + (uint32_t)__popc(m & ((1u << lane) - 1u))] = make_float4(xl, xh, sdy, __uint_as_float(s));
        n += (uint32_t)__popc(m);
        total += (uint32_t)__popc(m);
        __syncwarp();
        if (n >= 32u) {
            const float4 c = rm.list[lane], rest = rm.list[32 + lane];
            __syncwarp();
            rm.list[lane] = rest;
            n -= 32u;
            f(c, true);
        }
        __syncwarp();
    }
    if (n) f(rm.list[lane], (uint32_t)lane < n);
    __syncwarp();
    return total;
}

// the first pixel wholly right of a line with x range up to xmax, and the first
// its range touches
__device__ __forceinline__ int first_full(float xmax, int W) { return max((int)ceilf(fminf(fmaxf(xmax, -1.0f), (float)W)), 0); }
__device__ __forceinline__ int first_touched(float xmin, int W) { return max((int)floorf(fminf(fmaxf(xmin, -1.0f), (float)W)), 0); }

// v in 2^-40 fixed point, as v = hi 2^-20 + lo 2^-40 (0 <= lo <= 2^20): two
// 32-bit shared atomics instead of a 64-bit one, sums exact whatever the order
struct Fix {
    int32_t hi, lo;
};
__device__ __forceinline__ Fix fix40(float v) {
    const float s = v * 1048576.0f, f = floorf(s);
    return Fix{(int32_t)f, __float2int_rn((s - f) * 1048576.0f)};
}

// The area A(x) of every pixel x of the row: the sum over the crossing lines of
// sdy * mean_right(xl - x, xh - x), by line instead of by pixel.  A line adds
// sdy in full to every pixel from first_full on and evaluates mean_right over
// the pixels its x range touches; both go into a difference array (a lane walks
// its line's pixels, so each difference takes the previous pixel's value off),
// which the warp then scans.
__global__ void __launch_bounds__(32 * kRowWarps)
k_area(rgpu_soft_batch B, Slice sl, const float2 *verts, uint32_t *overflow) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t H = sl.rows, P = B.paths_per_scene;
    const int W = (int)B.width, lane = threadIdx.x & 31;
    const RowMem rm = row_mem(smem, sl.ng);
    const uint32_t id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (id >= sl.scenes * P * H) return;
    // neighbouring warps: neighbouring rows of one path
    const uint32_t r = id % H, row = sl.row0 + r, sp = id / H, p = sp % P, sc = sp / P, j = (sl.s0 + sc) * P + p;
    const int E = 1 << rm.esh;
    for (int x = lane; x < 32 * E + 33; x += 32) rm.a[x] = rm.b[x] = 0;
    __syncwarp();
    auto add = [&](int x, Fix v, Fix &prev) {
        const int i = rm.at(x);
        atomicAdd(&rm.a[i], (uint32_t)(v.hi - prev.hi));
        atomicAdd(&rm.b[i], (uint32_t)(v.lo - prev.lo));
        prev = v;
    };
    const uint32_t total = for_crossings(rm, verts + path_vbase(B, j), path_nverts(B, j), (float)row, [&](float4 c, bool valid) {
        if (!valid) return;
        const float lo = fminf(c.x, c.y), hi = fmaxf(c.x, c.y);
        const int xr = first_full(hi, W), xe = min(xr, W);
        Fix prev{0, 0};
        for (int x = first_touched(lo, W); x < xe; x++)
            add(x, fix40(c.z * mean_right(c.x - (float)x, c.y - (float)x)), prev);
        if (xr < W) add(xr, fix40(c.z), prev);
    });
    if (lane == 0 && total >= (uint32_t)kMaxCross) atomicOr(overflow, 1u);
    const size_t at = ((size_t)(sc * H + r) * P + p);
    uint32_t mask = 0;
    if (total) {
        // scan: each lane a run of E pixels
        int32_t rh = 0, rl = 0;
        const int x0 = lane << rm.esh, i0 = rm.at(x0);
        for (int k = 0; k < E; k++) {
            rh += (int32_t)rm.a[i0 + k];
            rl += (int32_t)rm.b[i0 + k];
        }
        int32_t sh = rh, sl2 = rl;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t th = __shfl_up_sync(0xffffffffu, sh, o), tl = __shfl_up_sync(0xffffffffu, sl2, o);
            if (lane >= o) { sh += th; sl2 += tl; }
        }
        sh -= rh;
        sl2 -= rl;
        for (int k = 0; k < E; k++) {
            sh += (int32_t)rm.a[i0 + k];
            sl2 += (int32_t)rm.b[i0 + k];
            rm.a[i0 + k] = __float_as_uint(__ll2float_rn((long long)sh * 1048576 + sl2) * (1.0f / 1099511627776.0f));
        }
        __syncwarp();
        float *out = sl.area + at * (32 * sl.ng);
        for (uint32_t g = 0; g < sl.ng; g++) {
            const int x = (int)(32 * g) + lane;
            const float A = x < W ? __uint_as_float(rm.a[rm.at(x)]) : 0.0f;
            if (__any_sync(0xffffffffu, A != 0.0f)) {
                out[x] = A;
                mask |= 1u << g;
            }
        }
    }
    if (lane == 0) sl.mask[at] = mask;
}

// C = c P + (1 - c a) C for one pixel and path; a pixel without coverage keeps its
// colour whatever the paint (an infinite one would make it NaN)
__device__ __forceinline__ void composite(float4 &C, float A, const PaintOut &po) {
    const float c = fminf(fabsf(A), 1.0f);
    const bool on = c != 0.0f;  // selects: a branch per group took 5% more of a small step
    const float ca = c * po.a, keep = 1.0f - ca;
    C.x = on ? c * (po.r * po.a) + keep * C.x : C.x;
    C.y = on ? c * (po.g * po.a) + keep * C.y : C.y;
    C.z = on ? c * (po.b * po.a) + keep * C.z : C.z;
    C.w = on ? ca + keep * C.w : C.w;
}

// the warp's row and groups: G neighbouring groups of one row
template <int G>
struct Strip {
    uint32_t sc, row, g0;  // scene of the slice, row of the scene, first group
    uint32_t r;            // row of the slice
    bool ok;
    __device__ __forceinline__ Strip(const rgpu_soft_batch &B, const Slice &sl) {
        const uint32_t per_row = (sl.ng + G - 1) / G;
        const uint32_t id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
        r = id / per_row;
        g0 = (id - r * per_row) * G;
        sc = r / sl.rows;
        row = sl.row0 + r - sc * sl.rows;
        ok = r < sl.scenes * sl.rows;
    }
};

// ---- forward composite: one group per warp (see wide_strips)
__global__ void __launch_bounds__(128) k_composite(rgpu_soft_batch B, Slice sl, float4 *image) {
    const Strip<1> st(B, sl);
    if (!st.ok) return;
    const int lane = threadIdx.x & 31, W = (int)B.width, x = (int)(32 * st.g0) + lane;
    const uint32_t P = B.paths_per_scene;
    float4 C = make_float4(0.f, 0.f, 0.f, 0.f);
    const size_t r = st.r;
    for (uint32_t p0 = 0; p0 < P; p0 += 32) {
        // 32 paths' masks at a time; those without coverage here are skipped
        const bool m = p0 + (uint32_t)lane < P && (sl.mask[r * P + p0 + (uint32_t)lane] >> st.g0 & 1u) != 0u;
        for (uint32_t todo = __ballot_sync(0xffffffffu, m); todo; todo &= todo - 1u) {
            const uint32_t p = p0 + (uint32_t)__ffs(todo) - 1u, j = (sl.s0 + st.sc) * P + p;
            composite(C, sl.area[(r * P + p) * (32 * sl.ng) + 32 * st.g0 + (uint32_t)lane],
                      eval_paint(B, j, (float)x + 0.5f, (float)st.row + 0.5f));
        }
    }
    if (x < W) image[((size_t)(sl.s0 + st.sc) * B.height + st.row) * W + x] = C;
}

// ---- flattening: one thread per (path, vertex)
// Control points of cubic c of an n-cubic path (points base 3 * seg_offset):
// start pts[3c] (the previous cubic's end; pts[0] for c = 0), controls
// pts[3c+1], pts[3c+2], end pts[3c+3], or pts[0] for the last cubic.
__device__ __forceinline__ float bern(int role, float t) {
    const float u = 1.0f - t;
    return role == 0 ? u * u * u : role == 1 ? 3.0f * u * u * t : role == 2 ? 3.0f * u * t * t : t * t * t;
}

__global__ void k_flatten(rgpu_soft_batch B, uint32_t npaths, float2 *verts) {
    const uint32_t j = blockIdx.y;
    if (j >= npaths) return;
    const uint32_t s0 = B.seg_offset[j], ns = B.seg_offset[j + 1] - s0;
    const float2 *pts = reinterpret_cast<const float2 *>(B.points) + 3 * s0;
    float2 *v = verts + kFlat * s0;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < kFlat * ns; q += gridDim.x * blockDim.x) {
        const uint32_t c = q / kFlat, i = q % kFlat;
        const float t = (float)i / (float)kFlat;
        const float b0 = bern(0, t), b1 = bern(1, t), b2 = bern(2, t), b3 = bern(3, t);
        const float2 P0 = pts[3 * c], P1 = pts[3 * c + 1], P2 = pts[3 * c + 2];
        const float2 P3 = c + 1 < ns ? pts[3 * c + 3] : pts[0];
        v[q] = make_float2(b0 * P0.x + b1 * P1.x + b2 * P2.x + b3 * P3.x, b0 * P0.y + b1 * P1.y + b2 * P2.y + b3 * P3.y);
    }
}

// vertex gradients -> control-point gradients (the transpose of k_flatten)
__global__ void k_unflatten(rgpu_soft_batch B, uint32_t npaths, const float2 *vgrad, float *pgrad) {
    const uint32_t j = blockIdx.y;
    if (j >= npaths) return;
    const uint32_t s0 = B.seg_offset[j], ns = B.seg_offset[j + 1] - s0;
    const float2 *vg = vgrad + kFlat * s0;
    float2 *pg = reinterpret_cast<float2 *>(pgrad) + 3 * s0;
    for (uint32_t m = blockIdx.x * blockDim.x + threadIdx.x; m < 3 * ns; m += gridDim.x * blockDim.x) {
        float gx = 0.f, gy = 0.f;
        auto add = [&](uint32_t c, int role) {
            for (int i = 0; i < kFlat; i++) {
                const float b = bern(role, (float)i / (float)kFlat);
                const float2 g = vg[kFlat * c + i];
                gx += b * g.x;
                gy += b * g.y;
            }
        };
        const uint32_t c = m / 3, r = m % 3;
        if (r == 0) {
            add(c, 0);                          // start of cubic c
            add(c == 0 ? ns - 1 : c - 1, 3);    // end of the previous cubic (of the last one for c = 0)
        } else {
            add(c, (int)r);
        }
        pg[m] = make_float2(gx, gy);
    }
}

// ---- blur
// w_j = exp(-j^2 / 2s^2) / Z and, for `deriv`, d w_j / d sigma, by the block's
// first threads (the sums in the order of j)
__device__ __forceinline__ void blur_weights(float sigma, bool deriv, float *w, int tid) {
    __shared__ float e[2 * kRadius + 1], zm[2];
    const int n = 2 * kRadius + 1, j = tid - kRadius;
    if (tid < n) e[tid] = expf(-(float)(j * j) / (2.0f * sigma * sigma));
    __syncthreads();
    if (tid == 0) {
        float z = 0.0f, m = 0.0f;
        for (int i = 0; i < n; i++) {
            z += e[i];
            m += e[i] * (float)((i - kRadius) * (i - kRadius));
        }
        zm[0] = z;
        zm[1] = m;
    }
    __syncthreads();
    if (tid < n) {
        const float wj = e[tid] / zm[0];
        w[tid] = deriv ? wj * ((float)(j * j) - zm[1] / zm[0]) / (sigma * sigma * sigma) : wj;
    }
    __syncthreads();
}

// The filter of one block: f(x, y, filtered pixel) for 32 x 32 pixels of the scene,
// taps outside the canvas skipped as zeros.  A block is 32 x 8 threads.
// Horizontally the rows with their halo go through shared memory, two by two;
// vertically each thread keeps a column's taps in flight for four pixels in turn.
constexpr int kTile = 32;
template <bool HORIZ, class F>
__device__ __forceinline__ void filter_tile(const float4 *img, const float *k, int W, int H, F f) {
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int x0 = blockIdx.x * kTile, y0 = blockIdx.y * kTile;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [](float4 &a, float q, float4 v) {
        a.x += q * v.x; a.y += q * v.y; a.z += q * v.z; a.w += q * v.w;
    };
    if (HORIZ) {
        __shared__ float4 line[8][kTile + 2 * kRadius];
        for (int r = 0; r < kTile; r += 8) {
            const int y = y0 + r + ty;
            for (int i = tx; i < kTile + 2 * kRadius; i += 32) {
                const int x = x0 + i - kRadius;
                line[ty][i] = (y < H && x >= 0 && x < W) ? img[(size_t)y * W + x] : zero;
            }
            __syncwarp();  // a warp reads the row it wrote
            float4 acc = zero;
#pragma unroll
            for (int j = 0; j <= 2 * kRadius; j++) add(acc, k[j], line[ty][tx + j]);
            __syncwarp();
            if (x0 + tx < W && y < H) f(x0 + tx, y, acc);
        }
    } else {
        const int x = x0 + tx, y = y0 + 4 * ty;
        float4 acc[4] = {zero, zero, zero, zero};
        if (x < W)
#pragma unroll 4
            for (int i = 0; i < 2 * kRadius + 4; i++) {
                const int yy = y + i - kRadius;
                const float4 v = (yy >= 0 && yy < H) ? img[(size_t)yy * W + x] : zero;
#pragma unroll
                for (int o = 0; o < 4; o++)
                    if (i - o >= 0 && i - o <= 2 * kRadius) add(acc[o], k[i - o], v);
            }
#pragma unroll
        for (int o = 0; o < 4; o++)
            if (x < W && y + o < H) f(x, y + o, acc[o]);
    }
}

// out = K applied along x (HORIZ) or y
template <bool HORIZ>
__global__ void __launch_bounds__(256) k_blur(const float4 *in, float4 *out, const float *sigma, int W, int H) {
    __shared__ float w[2 * kRadius + 1];
    const uint32_t s = blockIdx.z;
    blur_weights(sigma[s], false, w, (int)(threadIdx.y * 32 + threadIdx.x));
    float4 *o = out + (size_t)s * W * H;
    filter_tile<HORIZ>(in + (size_t)s * W * H, w, W, H, [&](int x, int y, float4 v) { o[(size_t)y * W + x] = v; });
}

// dsigma[s] += sum over pixels of a . (dK applied to b) along x or y
template <bool HORIZ>
__global__ void __launch_bounds__(256) k_dsigma(const float4 *a, const float4 *b, const float *sigma, int W, int H,
                                                float *dsigma) {
    __shared__ float w[2 * kRadius + 1], red[8];
    const uint32_t s = blockIdx.z;
    const int tid = (int)(threadIdx.y * 32 + threadIdx.x);
    blur_weights(sigma[s], true, w, tid);
    const float4 *g = a + (size_t)s * W * H;
    float sum = 0.0f;
    filter_tile<HORIZ>(b + (size_t)s * W * H, w, W, H, [&](int x, int y, float4 v) {
        const float4 q = g[(size_t)y * W + x];
        sum += q.x * v.x + q.y * v.y + q.z * v.z + q.w * v.w;
    });
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((tid & 31) == 0) red[tid >> 5] = sum;
    __syncthreads();
    if (tid == 0) {
        float t = 0.0f;
        for (int i = 0; i < 8; i++) t += red[i];
        atomicAdd(&dsigma[s], t);
    }
}

// ---- adjoint of the rows
// per path: 16 stop colours + 4 stop offsets (gradient) or 4 colour
// channels (solid), then the opacity at index 20
constexpr int kAcc = 21;

__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Lane q gets the warp's sum of v[q]: at each step a lane keeps one half of the
// values and adds the other lane's share of it (31 exchanges for up to 32
// values, instead of five per value).
template <int H>
__device__ __forceinline__ void sum_step(float (&v)[32]) {
    const bool up = (threadIdx.x & H) != 0;
#pragma unroll
    for (int q = 0; q < H; q++) {
        const float keep = up ? v[q + H] : v[q], give = up ? v[q] : v[q + H];
        v[q] = keep + __shfl_xor_sync(0xffffffffu, give, H);
    }
    if constexpr (H > 1) sum_step<H / 2>(v);
}
template <int N>
__device__ __forceinline__ float warp_sums(const float (&acc)[N]) {
    float v[32];
#pragma unroll
    for (int q = 0; q < 32; q++) v[q] = q < N ? acc[q] : 0.0f;
    sum_step<16>(v);
    return v[0];
}

// The composite forwards (keeping the colours under each path), then in reverse:
// paint gradients, reduced over the warp's pixels, and dL/dA in place of the
// areas.
template <int G>
__global__ void __launch_bounds__(128) k_reverse(rgpu_soft_batch B, Slice sl, rgpu_soft_grads Gr, const float4 *grad_image) {
    const Strip<G> st(B, sl);
    if (!st.ok) return;
    const int lane = threadIdx.x & 31, W = (int)B.width;
    const uint32_t P = B.paths_per_scene;
    const size_t r = st.r, stride = 32 * (size_t)sl.ng;
    const size_t first = r * P * stride + 32 * st.g0 + (uint32_t)lane;
    const float py = (float)st.row + 0.5f;
    float4 C[G], gC[G];
#pragma unroll
    for (int k = 0; k < G; k++) {
        const int x = (int)(32 * (st.g0 + k)) + lane;
        C[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        gC[k] = x < W ? grad_image[((size_t)(sl.s0 + st.sc) * B.height + st.row) * W + x] : C[k];
    }
    auto masks = [&](uint32_t p0) {
        return p0 + (uint32_t)lane < P ? (sl.mask[r * P + p0 + (uint32_t)lane] >> st.g0) & ((1u << G) - 1u) : 0u;
    };
    for (uint32_t p0 = 0; p0 < P; p0 += 32) {
        const uint32_t m = masks(p0);
        for (uint32_t todo = __ballot_sync(0xffffffffu, m != 0u); todo; todo &= todo - 1u) {
            const int l = __ffs(todo) - 1;
            const uint32_t p = p0 + (uint32_t)l, mp = __shfl_sync(0xffffffffu, m, l), j = (sl.s0 + st.sc) * P + p;
            const size_t at = first + p * stride;
#pragma unroll
            for (int k = 0; k < G; k++)
                if (mp >> k & 1u) {
                    sl.under[at + 32 * k] = C[k];
                    composite(C[k], sl.area[at + 32 * k], eval_paint(B, j, (float)(32 * (st.g0 + k) + lane) + 0.5f, py));
                }
        }
    }
    for (int32_t p0 = (int32_t)((P - 1) & ~31u); p0 >= 0; p0 -= 32) {
        const uint32_t m = masks((uint32_t)p0);
        for (uint32_t todo = __ballot_sync(0xffffffffu, m != 0u); todo;) {
            const int l = 31 - __clz(todo);
            todo &= ~(1u << l);
            const uint32_t p = (uint32_t)p0 + (uint32_t)l, mp = __shfl_sync(0xffffffffu, m, l), j = (sl.s0 + st.sc) * P + p;
            const size_t at = first + p * stride;
            const bool is_grad = B.paint_kind[j] != 0;
            float acc[kAcc];
#pragma unroll
            for (int q = 0; q < kAcc; q++) acc[q] = 0.0f;
#pragma unroll
            for (int k = 0; k < G; k++) {
                if (!(mp >> k & 1u)) continue;
                const float A = sl.area[at + 32 * k];
                const float c = fminf(fabsf(A), 1.0f);
                float dA = 0.0f;
                if (c != 0.0f) {
                    const float4 Cp = sl.under[at + 32 * k];
                    const PaintOut po = eval_paint(B, j, (float)(32 * (st.g0 + k) + lane) + 0.5f, py);
                    const float4 g = gC[k];
                    const float Pr = po.r * po.a, Pg = po.g * po.a, Pb = po.b * po.a, Pa = po.a;
                    // C = c P + (1 - c a) Cp
                    const float dc = g.x * (Pr - po.a * Cp.x) + g.y * (Pg - po.a * Cp.y) + g.z * (Pb - po.a * Cp.z) +
                                     g.w * (Pa - po.a * Cp.w);
                    const float da_keep = -c * (g.x * Cp.x + g.y * Cp.y + g.z * Cp.z + g.w * Cp.w);
                    const float dPr = c * g.x, dPg = c * g.y, dPb = c * g.z, dPa = c * g.w;
                    // straight colour; `da` is d/d(alpha times opacity): the
                    // paint's own alpha gets da * opacity, the opacity da * alpha
                    const float dr = dPr * po.a, dg = dPg * po.a, db = dPb * po.a;
                    const float da_eff = dPr * po.r + dPg * po.g + dPb * po.b + dPa + da_keep;
                    const float da = da_eff * po.op;
                    acc[20] += da_eff * po.raw_a;
                    if (!is_grad) {
                        acc[0] += dr; acc[1] += dg; acc[2] += db; acc[3] += da;
                    } else {
                        // acc[0..15]: stop colours (4 x RGBA), acc[16..19]: stop offsets;
                        // flat below the first / above the last stop: that stop's colour
                        const bool flat = po.seg < 0 || po.seg == 3;
                        const int i = po.seg < 0 ? 0 : po.seg;
                        const float w = flat ? 0.0f : po.w, u = 1.0f - w;
                        float dlo = 0.0f, dhi = 0.0f;
                        if (!flat) {
                            // w = (t - o_i) / (o_{i+1} - o_i)
                            const float *off = B.stop_offsets + 4 * (size_t)j;
                            const float span = off[i + 1] - off[i];
                            if (span > 0.0f) {
                                const float4 *scol = reinterpret_cast<const float4 *>(B.stop_colors) + 4 * (size_t)j;
                                const float4 c0 = scol[i], c1 = scol[i + 1];
                                const float dw = dr * (c1.x - c0.x) + dg * (c1.y - c0.y) + db * (c1.z - c0.z) + da * (c1.w - c0.w);
                                const float inv2 = 1.0f / (span * span);
                                dlo = dw * (po.t - off[i + 1]) * inv2;
                                dhi = -dw * (po.t - off[i]) * inv2;
                            }
                        }
#pragma unroll
                        for (int q = 0; q < 4; q++) {  // constant indexes keep acc in registers
                            const float f = q == i ? u : (q == i + 1 ? w : 0.0f);
                            if (q == i || q == i + 1) {
                                acc[4 * q] += f * dr; acc[4 * q + 1] += f * dg; acc[4 * q + 2] += f * db; acc[4 * q + 3] += f * da;
                                acc[16 + q] += q == i ? dlo : dhi;
                            }
                        }
                    }
                    const float keep = 1.0f - c * po.a;
                    gC[k].x *= keep;
                    gC[k].y *= keep;
                    gC[k].z *= keep;
                    gC[k].w *= keep;
                    const float dcA = (fabsf(A) < 1.0f) ? (A > 0.0f ? 1.0f : (A < 0.0f ? -1.0f : 0.0f)) : 0.0f;
                    dA = dc * dcA;
                }
                sl.area[at + 32 * k] = dA;
            }
            // the paint gradients of this path over the warp's pixels
            float mine = 0.0f;  // lane q: the sum of acc[q]
            if (is_grad) mine = warp_sums(acc);
            else {
#pragma unroll
                for (int q = 0; q < 5; q++) {
                    const float v = warp_sum(acc[q < 4 ? q : 20]);
                    if (lane == (q < 4 ? q : 20)) mine = v;
                }
            }
            if (lane < kAcc && mine != 0.0f) {
                if (lane == 20) { if (Gr.opacity) atomicAdd(&Gr.opacity[j], mine); }
                else if (!is_grad) atomicAdd(&Gr.colors[4 * (size_t)j + lane], mine);
                else if (lane < 16) atomicAdd(&Gr.stop_colors[16 * (size_t)j + lane], mine);
                else atomicAdd(&Gr.stop_offsets[4 * (size_t)j + (lane - 16)], mine);
            }
        }
    }
}

// mean_right with its derivatives in both ends
__device__ __forceinline__ float mean_right_d(float a, float b, float *da, float *db) {
    const bool swap = a > b;
    const float lo = swap ? b : a, hi = swap ? a : b;
    float v, dl, dh;
    if (hi <= 0.0f) { v = 1.0f; dl = dh = 0.0f; }
    else if (lo >= 1.0f) { v = dl = dh = 0.0f; }
    else if (lo >= 0.0f && hi <= 1.0f) { v = 1.0f - (lo + hi) * 0.5f; dl = dh = -0.5f; }
    else {
        const float inv = 1.0f / (hi - lo), h = 0.5f * inv * inv;
        if (hi <= 1.0f) {         // lo < 0
            v = 1.0f - hi * hi * (0.5f * inv);
            dl = -hi * hi * h;
            dh = hi * (lo + lo - hi) * h;
        } else if (lo >= 0.0f) {  // hi > 1
            const float q = 1.0f - lo;
            v = q * q * (0.5f * inv);
            dl = q * (q - 2.0f * (hi - lo)) * h;
            dh = -q * q * h;
        } else {
            v = (0.5f - lo) * inv;
            dl = (0.5f - hi) * inv * inv;
            dh = (lo - 0.5f) * inv * inv;
        }
    }
    *da = swap ? dh : dl;
    *db = swap ? dl : dh;
    return v;
}

// Line gradients of one (row, path): a lane per crossing line sums dL/dA times
// the area and its derivatives in the clipped ends over the pixels the line
// touches, plus the suffix sum of dL/dA over the pixels right of it; the clipped
// ends' derivatives in the line's end coordinates (dual numbers) are the same
// for all of them.
__global__ void __launch_bounds__(32 * kRowWarps)
k_lines(rgpu_soft_batch B, Slice sl, const float2 *verts, float2 *vgrad) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t H = sl.rows, P = B.paths_per_scene;
    const int W = (int)B.width, lane = threadIdx.x & 31;
    const RowMem rm = row_mem(smem, sl.ng);
    const uint32_t id = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (id >= sl.scenes * P * H) return;
    const uint32_t r = id % H, row = sl.row0 + r, sp = id / H, p = sp % P, sc = sp / P, j = (sl.s0 + sc) * P + p;
    const size_t at = ((size_t)(sc * H + r) * P + p);
    const uint32_t mask = sl.mask[at];
    if (!mask) return;
    const int E = 1 << rm.esh;
    float *d = reinterpret_cast<float *>(rm.a), *S = reinterpret_cast<float *>(rm.b);
    bool any = false;
    for (uint32_t g = 0; g < (uint32_t)E; g++) {
        const int x = (int)(32 * g) + lane;
        const float v = (g < sl.ng && (mask >> g & 1u) && x < W) ? sl.area[at * (32 * sl.ng) + x] : 0.0f;
        d[rm.at(x)] = v;
        any = any || v != 0.0f;
    }
    if (!__any_sync(0xffffffffu, any)) return;
    __syncwarp();
    // suffix sums: each lane a run of E pixels from the right
    {
        const int i0 = rm.at(lane << rm.esh);
        float run = 0.0f;
        for (int k = E - 1; k >= 0; k--) run += d[i0 + k];
        float sum = run;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float t = __shfl_down_sync(0xffffffffu, sum, o);
            if (lane + o < 32) sum += t;
        }
        // the sum right of the run
        const float right = __shfl_down_sync(0xffffffffu, sum, 1);
        float acc = lane == 31 ? 0.0f : right;
        for (int k = E - 1; k >= 0; k--) {
            acc += d[i0 + k];
            S[i0 + k] = acc;
        }
    }
    __syncwarp();
    const float2 *v = verts + path_vbase(B, j);
    const uint32_t nv = path_nverts(B, j), vb = path_vbase(B, j);
    for_crossings(rm, v, nv, (float)row, [&](float4 cr, bool valid) {
        if (!valid) return;
        const uint32_t ia = __float_as_uint(cr.w), ib = ia + 1 < nv ? ia + 1 : 0;
        const float lo = fminf(cr.x, cr.y), hi = fmaxf(cr.x, cr.y);
        const int xr = first_full(hi, W), xe = min(xr, W);
        float sv = 0.0f, sa = 0.0f, sb = 0.0f;  // dL/dA times the area's mean, and its derivatives in xl and xh
        for (int x = first_touched(lo, W); x < xe; x++) {
            const float dx = d[rm.at(x)];
            if (dx == 0.0f) continue;
            float da, db;
            sv += dx * mean_right_d(cr.x - (float)x, cr.y - (float)x, &da, &db);
            sa += dx * da;
            sb += dx * db;
        }
        if (xr < W) sv += S[rm.at(xr)];
        if (sv == 0.0f && sa == 0.0f && sb == 0.0f) return;
        const float2 a = v[ia], b = v[ib];
        D4 X0 = mk(a.x), Y0 = mk(a.y), X1 = mk(b.x), Y1 = mk(b.y);
        X0.d[0] = 1.f; Y0.d[1] = 1.f; X1.d[2] = 1.f; Y1.d[3] = 1.f;
        D4 xl, xh, sdy;
        if (!clip_row<D4>(X0, Y0, X1, Y1, (float)row, &xl, &xh, &sdy)) return;
        float g[4];
#pragma unroll
        for (int q = 0; q < 4; q++) g[q] = sv * sdy.d[q] + sdy.v * (sa * xl.d[q] + sb * xh.d[q]);
        if (g[0] != 0.0f) atomicAdd(&vgrad[vb + ia].x, g[0]);
        if (g[1] != 0.0f) atomicAdd(&vgrad[vb + ia].y, g[1]);
        if (g[2] != 0.0f) atomicAdd(&vgrad[vb + ib].x, g[2]);
        if (g[3] != 0.0f) atomicAdd(&vgrad[vb + ib].y, g[3]);
    });
}

// The loss: every block's share in 64 bits, and the sum of the shares, in their
// order, by the block that finishes last (`done` counts them and is zero again
// after it).  Added up in 32 bits in the order of arrival it differed by 2e-6 from
// run to run.
constexpr int kMseBlocks = 1024, kMseThreads = 256;
struct MseScratch {
    double share[kMseBlocks];
    uint32_t done;
};
__device__ __forceinline__ double block_sum(double v, double *red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.0;
    for (int i = 0; i < kMseThreads / 32; i++) v += red[i];
    return v;
}
__global__ void __launch_bounds__(kMseThreads)
k_mse(const float *a, const float *b, size_t n, float scale, float *loss, float *grad, MseScratch *scratch) {
    __shared__ double red[kMseThreads / 32];
    __shared__ bool last;
    float sum = 0.0f;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const float d = a[i] - b[i];
        sum += d * d;
        if (grad) grad[i] = 2.0f * d * scale;
    }
    const double share = block_sum((double)sum, red);
    if (threadIdx.x == 0) {
        scratch->share[blockIdx.x] = share;
        __threadfence();
        last = atomicAdd(&scratch->done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double all = 0.0;
    for (int i = (int)threadIdx.x; i < kMseBlocks; i += kMseThreads) all += __ldcg(&scratch->share[i]);
    all = block_sum(all, red);
    if (threadIdx.x == 0) {
        *loss = (float)(all * (double)scale);
        scratch->done = 0u;
    }
}

// ---- host side: cached work buffers
struct Buf {
    void *p = nullptr;
    size_t cap = 0;
    cudaError_t ensure(size_t bytes) {
        if (bytes <= cap) return cudaSuccess;
        release();
        cudaError_t e = forced_alloc_failure() ? cudaErrorMemoryAllocation : cudaMalloc(&p, bytes);
        if (e == cudaSuccess) cap = bytes;
        else {
            p = nullptr;
            cudaGetLastError();  // reported here, not by the next launch
        }
        return e;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
    }
};
std::mutex g_mu;
Buf g_verts, g_vgrad, g_tmp0, g_tmp1, g_tmp2, g_slice, g_flags, g_mse;

bool valid(const rgpu_soft_batch *b) {
    return b && b->scenes && b->width && b->height && b->paths_per_scene && b->seg_offset && b->points &&
           b->paint_kind && b->colors && b->stop_offsets && b->stop_colors && b->grad_line && b->sigma &&
           b->width <= (uint32_t)kMaxWidth && b->total_segments;
}

int fail(cudaError_t e) {
    set_last_error_message(cudaGetErrorString(e));
    return RGPU_ERR_CUDA;
}

// The scratch of a slice of scenes, one buffer for both passes: areas (4 bytes per
// pixel and path), for the adjoint the colours under each path (16), and masks;
// at least one row of one scene.  Slices that fit the L2 cache instead (96 MB, one
// scene of 64 paths on 256^2 pixels each) leave the SMs short of warps: the four
// kernels took 3.25 ms against 1.84.  Where memory is short, slices are halved.
constexpr size_t kSliceBytes = (size_t)1536 << 20;
cudaError_t make_slice(const rgpu_soft_batch &b, bool adjoint, Slice *sl) {
    sl->ng = (b.width + 31) / 32;
    const size_t P = b.paths_per_scene, row_px = P * 32 * sl->ng, row_bytes = row_px * (adjoint ? 20 : 4) + P * 4;
    for (size_t most = kSliceBytes;;) {
        // rows that fit; warps, one per (row, path) or group of a row, are counted in 32 bits
        const size_t fit = std::min<size_t>(most / row_bytes, 0x7FFFFFFFull / (P + sl->ng));
        sl->rows = (uint32_t)std::min<size_t>(b.height, std::max<size_t>(1, fit));
        sl->scenes = (uint32_t)std::min<size_t>(b.scenes, std::max<size_t>(1, fit / b.height));
        const size_t rows = (size_t)sl->scenes * sl->rows;
        cudaError_t e = g_slice.ensure(rows * row_bytes);
        if (e == cudaErrorMemoryAllocation && rows > 1) {
            most = rows * row_bytes / 2;
            continue;
        }
        sl->area = (float *)g_slice.p;
        sl->under = (float4 *)(sl->area + rows * row_px);
        sl->mask = (uint32_t *)(sl->area + rows * row_px * (adjoint ? 5 : 1));
        return e;
    }
}
// CTA size and shared memory of the row kernels for the slice's width
uint32_t row_warps(const Slice &sl) {
    return (uint32_t)std::min<size_t>(kRowWarps, std::max<size_t>(1, (48u << 10) / row_bytes(sl.ng)));
}
uint32_t blocks(uint64_t n, uint32_t per) { return (uint32_t)((n + per - 1) / per); }

// Groups per warp of the reverse composite.  Every warp adds its share of a path's
// paint gradients to the same words, so where many groups of a scene do that and
// a warp's chain over the paths is short, two groups per warp halve the adds.  One
// / two groups, us: 500^2 pixels x 4 paths 15.8 / 11.9, x 64 paths 185 / 188; 16
// scenes of 256 x 512 x 16 385 / 309; but 16 of 256^2 x 64 558 / 757, 1 of 256^2 x 4
// 9.5 / 11.9.  The lines lie at 160 groups per path and 6,000 in all (640^2 x 64, 200
// per path, 0.91 .. 1.01; 13 of 117 x 544 x 12, 181 per path, the step 0.98; 256^2 x
// 16, 128 per path, 0.91 .. 1.39; 256 x 512 x 4, 4,096 in all, 1.05; 500^2 x 4, 8,000,
// 0.75).  The forward composite adds nothing up: one group is never slower there by
// more than 7%, and up to a third faster.
bool wide_strips(const rgpu_soft_batch &b, const Slice &sl) {
    const uint64_t per_scene = (uint64_t)b.height * sl.ng, all = (uint64_t)sl.scenes * sl.rows * sl.ng;
    return sl.ng >= 2 && per_scene >= 160ull * b.paths_per_scene && all >= 6000;
}
template <class F>
void with_groups(bool wide, F f) {
    if (wide) f(std::integral_constant<int, 2>());
    else f(std::integral_constant<int, 1>());
}
// f(slice) over the batch's scenes; launch errors are left for the caller's check
template <class F>
void each_slice(const rgpu_soft_batch &b, Slice sl, F f) {
    const uint32_t most = sl.scenes, most_rows = sl.rows;
    for (uint64_t s0 = 0; s0 < b.scenes; s0 += most)
        for (uint64_t r0 = 0; r0 < b.height; r0 += most_rows) {
            sl.s0 = (uint32_t)s0;
            sl.scenes = (uint32_t)std::min<uint64_t>(most, b.scenes - s0);
            sl.row0 = (uint32_t)r0;
            sl.rows = (uint32_t)std::min<uint64_t>(most_rows, b.height - r0);
            f(sl);
        }
}
void launch_area(const rgpu_soft_batch &b, const Slice &sl, cudaStream_t s) {
    const uint32_t nw = row_warps(sl);
    k_area<<<blocks((uint64_t)sl.scenes * b.paths_per_scene * sl.rows, nw), 32 * nw, nw * row_bytes(sl.ng), s>>>(
        b, sl, (const float2 *)g_verts.p, (uint32_t *)g_flags.p);
}

cudaError_t flatten(const rgpu_soft_batch &b, cudaStream_t s) {
    const uint32_t npaths = b.scenes * b.paths_per_scene;
    const size_t nverts = (size_t)kFlat * b.total_segments;
    cudaError_t e = g_verts.ensure(nverts * sizeof(float2));
    if (e != cudaSuccess) return e;
    dim3 grid(1, npaths);
    k_flatten<<<grid, 256, 0, s>>>(b, npaths, (float2 *)g_verts.p);
    return cudaGetLastError();
}

cudaError_t blur(const float4 *in, float4 *out, float4 *tmp, const rgpu_soft_batch &b, cudaStream_t s) {
    const dim3 blk(32, 8), grid((b.width + kTile - 1) / kTile, (b.height + kTile - 1) / kTile, b.scenes);
    k_blur<true><<<grid, blk, 0, s>>>(in, tmp, b.sigma, (int)b.width, (int)b.height);
    k_blur<false><<<grid, blk, 0, s>>>(tmp, out, b.sigma, (int)b.width, (int)b.height);
    return cudaGetLastError();
}

}  // namespace

// rgpu_trim's share: the work buffers are empty again
void release_buffers() {
    std::lock_guard<std::mutex> lock(g_mu);  // every call ends with its stream synchronised
    for (Buf *b : {&g_verts, &g_vgrad, &g_tmp0, &g_tmp1, &g_tmp2, &g_slice, &g_flags, &g_mse}) b->release();
}

}  // namespace soft
}  // namespace rgpu

using namespace rgpu::soft;

extern "C" int rgpu_soft_forward(const rgpu_soft_batch *b, float *image, float *blurred, void *stream) {
    rgpu::set_last_error_message("");
    if (!valid(b) || !image || !blurred) {
        rgpu::set_last_error_message("invalid arguments (canvas width is limited to 1024)");
        return RGPU_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = flatten(*b, s);
    if (e == cudaSuccess) e = g_flags.ensure(16);
    if (e == cudaSuccess) e = g_tmp0.ensure((size_t)b->scenes * b->width * b->height * sizeof(float4));
    if (e != cudaSuccess) return fail(e);
    Slice slice;
    e = make_slice(*b, false, &slice);
    if (e != cudaSuccess) return fail(e);
    cudaMemsetAsync(g_flags.p, 0, 16, s);
    each_slice(*b, slice, [&](const Slice &sl) {
        launch_area(*b, sl, s);
        k_composite<<<blocks((uint64_t)sl.scenes * sl.rows * sl.ng, 4), 128, 0, s>>>(*b, sl, (float4 *)image);
    });
    e = blur((const float4 *)image, (float4 *)blurred, (float4 *)g_tmp0.p, *b, s);
    uint32_t ovf = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&ovf, g_flags.p, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(e);
    if (ovf) {
        rgpu::set_last_error_message("more than 512 lines of one path cross a pixel row");
        return RGPU_ERR_CAPACITY;
    }
    return RGPU_OK;
}

extern "C" int rgpu_soft_backward(const rgpu_soft_batch *b, const float *image, const float *grad_blurred,
                                  rgpu_soft_grads *g, void *stream) {
    rgpu::set_last_error_message("");
    if (!valid(b) || !image || !grad_blurred || !g || !g->points || !g->colors || !g->stop_offsets ||
        !g->stop_colors || !g->sigma) {
        rgpu::set_last_error_message("invalid arguments");
        return RGPU_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t npaths = b->scenes * b->paths_per_scene;
    const size_t npx = (size_t)b->scenes * b->width * b->height;
    const size_t nverts = (size_t)kFlat * b->total_segments;
    const size_t npts = 3 * (size_t)b->total_segments;
    cudaError_t e = flatten(*b, s);
    if (e == cudaSuccess) e = g_vgrad.ensure(nverts * sizeof(float2));
    if (e == cudaSuccess) e = g_tmp0.ensure(npx * sizeof(float4));
    if (e == cudaSuccess) e = g_tmp1.ensure(npx * sizeof(float4));
    if (e == cudaSuccess) e = g_tmp2.ensure(npx * sizeof(float4));
    Slice slice;
    if (e == cudaSuccess) e = make_slice(*b, true, &slice);
    if (e == cudaSuccess) e = g_flags.ensure(16);
    if (e != cudaSuccess) return fail(e);
    // gradients are overwritten
    cudaMemsetAsync(g->points, 0, npts * sizeof(float2), s);
    cudaMemsetAsync(g->colors, 0, (size_t)npaths * 16, s);
    cudaMemsetAsync(g->stop_offsets, 0, (size_t)npaths * 16, s);
    cudaMemsetAsync(g->stop_colors, 0, (size_t)npaths * 64, s);
    cudaMemsetAsync(g->sigma, 0, (size_t)b->scenes * 4, s);
    if (g->opacity) cudaMemsetAsync(g->opacity, 0, (size_t)npaths * 4, s);
    cudaMemsetAsync(g_vgrad.p, 0, nverts * sizeof(float2), s);
    cudaMemsetAsync(g_flags.p, 0, 16, s);
    const dim3 blk(32, 8), grid((b->width + kTile - 1) / kTile, (b->height + kTile - 1) / kTile, b->scenes);
    const int W = (int)b->width, Hh = (int)b->height;
    float4 *gI = (float4 *)g_tmp0.p, *H = (float4 *)g_tmp1.p, *T = (float4 *)g_tmp2.p;
    const float4 *gB = (const float4 *)grad_blurred, *I = (const float4 *)image;
    // blurred = Kv(Kh I): dsigma = <gB, dKv (Kh I)> + <Kv gB, dKh I>; gI = Kh(Kv gB)
    k_blur<true><<<grid, blk, 0, s>>>(I, H, b->sigma, W, Hh);
    k_dsigma<false><<<grid, blk, 0, s>>>(gB, H, b->sigma, W, Hh, g->sigma);
    k_blur<false><<<grid, blk, 0, s>>>(gB, T, b->sigma, W, Hh);
    k_dsigma<true><<<grid, blk, 0, s>>>(T, I, b->sigma, W, Hh, g->sigma);
    k_blur<true><<<grid, blk, 0, s>>>(T, gI, b->sigma, W, Hh);
    each_slice(*b, slice, [&](const Slice &sl) {
        launch_area(*b, sl, s);
        with_groups(wide_strips(*b, sl), [&](auto G) {
            constexpr int kG = decltype(G)::value;
            const uint64_t warps = (uint64_t)sl.scenes * sl.rows * ((sl.ng + kG - 1) / kG);
            k_reverse<kG><<<blocks(warps, 4), 128, 0, s>>>(*b, sl, *g, gI);
        });
        const uint32_t nw = row_warps(sl);
        k_lines<<<blocks((uint64_t)sl.scenes * b->paths_per_scene * sl.rows, nw), 32 * nw, nw * row_bytes(sl.ng), s>>>(
            *b, sl, (const float2 *)g_verts.p, (float2 *)g_vgrad.p);
    });
    dim3 ug(1, npaths);
    k_unflatten<<<ug, 256, 0, s>>>(*b, npaths, (const float2 *)g_vgrad.p, g->points);
    uint32_t ovf = 0;
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaMemcpyAsync(&ovf, g_flags.p, 4, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return fail(e);
    if (ovf) {
        rgpu::set_last_error_message("more than 512 lines of one path cross a pixel row");
        return RGPU_ERR_CAPACITY;
    }
    return RGPU_OK;
}

extern "C" int rgpu_soft_mse(const float *blurred, const float *target, size_t count, float *loss,
                             float *grad_blurred, void *stream) {
    rgpu::set_last_error_message("");
    if (!blurred || !target || !loss || !count) {
        rgpu::set_last_error_message("invalid arguments");
        return RGPU_ERR_INVALID_ARG;
    }
    std::lock_guard<std::mutex> lock(g_mu);
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaSuccess;
    if (!g_mse.p) {
        e = g_mse.ensure(sizeof(MseScratch));
        if (e == cudaSuccess) e = cudaMemsetAsync(g_mse.p, 0, sizeof(MseScratch), s);
        if (e != cudaSuccess) return fail(e);
    }
    k_mse<<<kMseBlocks, kMseThreads, 0, s>>>(blurred, target, count, 1.0f / (float)count, loss, grad_blurred,
                                             (MseScratch *)g_mse.p);
    e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    return e == cudaSuccess ? RGPU_OK : fail(e);
}
