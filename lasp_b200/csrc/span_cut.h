// How the sequences of a launch are cut into spans of tiles and which CTA walks which span, kept free of CUDA types so
// that the same functions run in the kernels and in the host-side simulation of the test-suite.
#pragma once
#include <stdint.h>

#include "exchange_layout.h"   // LASP_HD

namespace lasp {
namespace tc {

LASP_HD int least(int a, int b) {
#if defined(__CUDA_ARCH__)
  return min(a, b);
#else
  return a < b ? a : b;
#endif
}

// An item is one span of consecutive tiles of one (batch, head) sequence; CTA b takes items b, b + grid, ...  `base`, `extra` and `magic` are what the
// kernels would otherwise divide for at every item (three integer divisions, inlined wherever a role steps through its
// tiles, were a third of a walk kernel's code).
struct SpanCut {
  int items, nspans, span, tiles;
  int base, extra;   // tiles / nspans and the remainder
  uint32_t magic;    // it / nspans = (it * magic) >> 32 with 64-bit arithmetic while items * nspans < 2^32
};
inline SpanCut make_span_cut(int items, int nspans, int span, int tiles) {
  return {items, nspans, span, tiles, tiles / nspans, tiles % nspans, nspans > 1 ? (uint32_t)(0x100000000ull / nspans) + 1 : 0};
}
LASP_HD int sequence_of_item(const SpanCut& c, int it) {
  return c.nspans == 1 ? it : (int)(((uint64_t)(uint32_t)it * c.magic) >> 32);
}

// first tile of span `s` of a sequence (s = nspans: one past the last tile).  `span` tiles each, the last one of a
// sequence whatever is left (even = false), or - for a kernel whose CTAs wait for one another - the tiles shared out
// evenly, spans differing by one tile at most, with the longer spans where the walk starts: there nobody has to wait
// for anybody's total, and the spans with the longest look-back get the fewest tiles (even = true).
template <bool BACKWARDS>
LASP_HD int span_first_tile(const SpanCut& c, bool even, int s) {
  if (!even) return least(s * c.span, c.tiles);
  // `extra` spans have base + 1 tiles
  return s * c.base + (BACKWARDS ? -least(0, c.nspans - c.extra - s) : least(s, c.extra));
}

// The span of its sequence that place `r` among the sequence's CTAs stands for.  Where CTAs wait for one another
// (`even`), one that walks backwards waits for the totals of the later spans: those come first, so that every CTA waits
// for lower block indexes only, which have started before it - another stream's kernel may hold the SMs that the higher
// ones still need.
template <bool BACKWARDS>
LASP_HD int span_of_place(const SpanCut& c, bool even, int r) {
  return BACKWARDS && even ? c.nspans - 1 - r : r;
}

}  // namespace tc
}  // namespace lasp
