// Coverage events: what the event kernel (events.cu) writes for every (row, draw)
// of a stream and the raster kernel (raster.cu) reads.
//
// Coverage follows tiny-skia's supersampling scan converter (scan/path_aa.rs:
// SHIFT = 2, 4 sub-scanlines x 4 sub-columns per pixel; SkScan_AntiPath).  A
// sub-scanline's crossings, sorted by x and walked with the fill rule
// (scan/path.rs walk_edges), open and close spans of sub-columns; a span adds
// 16 per covered sub-column to a pixel, or M where it covers the whole pixel (64;
// 63 on the 4th sub-scanline: SuperBlitter::blit_h's max_value), and the row's
// sum is capped at 255 (SkAlphaRuns catch-overflow).
//
// Both ends of a span change the coverage of two neighbouring pixels only: an
// event is a pixel and the two differences, and a pixel's coverage is the prefix
// sum of the differences up to it.  With l = x & 3, an opening end adds
// 64 - 16 l (M for l = 0), then M less that; a closing end takes M - 16 l, then
// 16 l.  Ends are independent of each other except for a span inside one pixel
// that starts after its left edge: opening and closing then differ by 64 - M
// too much, which the closing end takes back.  Aliased fills add and take 255
// per whole pixel.
//
// The events of a (row, draw) are unordered, at 4 x (bin offset + slot) words
// of the event array: a row's bin of nb edges makes at most nb + 1 events on
// each of 4 sub-scanlines, so the bins' offsets place the lists too.  A header
// word per slot: events (12 bits, from bit 20), first and last 32-pixel group
// that coverage may touch (10 bits each, from bits 10 and 0); kManyEvents in
// the upper 12 bits: the lower 20 hold the number of events.
#pragma once
#include <stdint.h>

namespace rgpu {
namespace dev {

constexpr uint32_t kManyEvents = 0xFFFu;
constexpr uint32_t kMaxEvents = (1u << 20) - 1u;

// an event: pixel of the row from the pass's first column on (15 bits), first
// difference (9 bits), second (7 bits)
__host__ __device__ __forceinline__ uint32_t event_diffs(int d0, int d1) {
    return ((uint32_t)(d0 & 0x1FF) << 15) | ((uint32_t)(d1 & 0x7F) << 24);
}
__device__ __forceinline__ int32_t event_pixel(uint32_t e) { return (int32_t)(e & 0x7FFFu); }
__device__ __forceinline__ int32_t event_d0(uint32_t e) { return (int32_t)(e << 8) >> 23; }
__device__ __forceinline__ int32_t event_d1(uint32_t e) { return (int32_t)(e << 1) >> 25; }

}  // namespace dev
}  // namespace rgpu
