// The cut of a launch into spans and their assignment to CTAs (lasp_b200/csrc/span_cut.h), for every number of sequences
// and tiles that a launch whose CTAs wait for one another can have on `sms` multiprocessors: every tile is walked once,
// and no CTA waits for the span total of a CTA with a higher block index.
#include <stdio.h>
#include <stdlib.h>

#include <vector>

#include "span_cut.h"

using namespace lasp::tc;

static int fail(const char* what, const SpanCut& c, int block) {
  printf("%s: items %d, spans %d, tiles %d, block %d\n", what, c.items, c.nspans, c.tiles, block);
  return 1;
}

template <bool BACKWARDS>
int check(const SpanCut& c, bool even, int grid) {
  std::vector<int> block_of(c.items, -1);
  std::vector<int> walked((size_t)(c.items / c.nspans) * c.tiles, 0);
  for (int b = 0; b < grid; ++b)
    for (int it = b; it < c.items; it += grid) {
      const int bh = sequence_of_item(c, it), sp = span_of_place<BACKWARDS>(c, even, it - bh * c.nspans);
      if (bh != it / c.nspans) return fail("wrong sequence", c, b);
      int& owner = block_of[bh * c.nspans + sp];
      if (owner >= 0) return fail("an item twice", c, b);
      owner = b;
      for (int t = span_first_tile<BACKWARDS>(c, even, sp); t < span_first_tile<BACKWARDS>(c, even, sp + 1); ++t)
        ++walked[(size_t)bh * c.tiles + t];
    }
  for (int w : walked)
    if (w != 1) return fail("a tile not walked once", c, -1);
  if (even)   // the CTAs wait: forwards for the earlier spans of their sequence, backwards for the later ones
    for (int it = 0; it < c.items; ++it)
      for (int other = it; other / c.nspans == it / c.nspans && other >= 0 && other < c.items; other += BACKWARDS ? 1 : -1)
        if (other != it && block_of[other] >= block_of[it]) return fail("a CTA waits for a later one", c, block_of[it]);
  return 0;
}

int main(int argc, char** argv) {
  const int sms = argc > 1 ? atoi(argv[1]) : 148;
  for (int seqs = 1; seqs <= 2 * sms; seqs = seqs < 20 ? seqs + 1 : seqs + 7)
    for (int tiles = 1; tiles <= 300; tiles = tiles < 40 ? tiles + 1 : tiles + 13) {
      const int per_seq = sms / seqs;
      const int span = per_seq >= 1 ? (tiles + per_seq - 1) / per_seq : tiles;
      const int nspans = (tiles + span - 1) / span, items = seqs * nspans, grid = items < sms ? items : sms;
      const SpanCut c = make_span_cut(items, nspans, span, tiles);
      if (check<false>(c, false, grid) || check<true>(c, false, grid)) return 1;
      if (items <= sms && (check<false>(c, true, grid) || check<true>(c, true, grid))) return 1;
    }
  printf("ok\n");
  return 0;
}
