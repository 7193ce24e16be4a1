// Host walk over the even-share schedule (balanced_schedule.cuh), for tests without a GPU.
#include "balanced_schedule.cuh"

#include <vector>

// Writes every segment of every unit, in order, as (unit, row, stream, first tile, end tile, slot, partials).  `tail`,
// `min_tiles`, `segment_tiles` and `stream_tiles` are what the kernels hand to the schedule; `capacity` = partial slots of a
// stream.  *num_segments = segments there are, of which the first max_segments are written.
extern "C" int anna_kv_selftest_even_shares(const int64_t* lengths, int batch, int streams_per_row, int units, int capacity,
                                            int tail, int min_tiles, int segment_tiles, int stream_tiles, int32_t* segments,
                                            int max_segments, int* num_segments) {
  using namespace anna;
  ANNA_REQUIRE(lengths != nullptr && segments != nullptr && num_segments != nullptr,
               "anna_kv_selftest_even_shares: null pointer argument");
  int64_t longest = 0;
  for (int b = 0; b < batch; ++b) longest = longest < lengths[b] ? lengths[b] : longest;
  ANNA_REQUIRE(batch > 0 && streams_per_row > 0 && units > 0 && min_tiles > 0 && segment_tiles >= 0 && stream_tiles >= 0 &&
                   tail >= 0 && balanced_schedule_fits(batch, streams_per_row, longest, capacity, stream_tiles),
               "anna_kv_selftest_even_shares: sizes out of range");
  std::vector<int> tiles(batch), prefix(batch + 1);
  int max_tiles = 0, streams = 0;
  for (int b = 0; b < batch; ++b) {
    const int64_t len = lengths[b] - tail;
    tiles[b] = len > 0 ? (int)((len + kBalancedTileTokens - 1) / kBalancedTileTokens) : 0;
    max_tiles = max_tiles < tiles[b] ? tiles[b] : max_tiles;
    streams += tiles[b] > 0 ? streams_per_row : 0;
  }
  auto scan = [&](int piece_tiles) {
    for (int b = 0; b < batch; ++b)
      prefix[b + 1] = prefix[b] + streams_per_row * balanced_line_length(tiles[b], stream_tiles, piece_tiles);
    return prefix[batch];
  };
  *num_segments = 0;
  const int line = scan(0);
  if (line == 0) return ANNA_OK;
  const BalancedCut cut = balanced_cut(line, streams, max_tiles, units, capacity, min_tiles, segment_tiles, stream_tiles);
  const int total = cut.piece_tiles > 0 ? scan(cut.piece_tiles) : line;
  for (int unit = 0, b = 0; unit < units; ++unit) {
    int64_t pos = (int64_t)unit * cut.share;
    const int64_t end = pos + cut.share < total ? pos + cut.share : total;
    while (pos < end) {
      while (prefix[b + 1] <= pos) ++b;
      const BalancedSegment seg = balanced_segment(cut, unit, (int)pos, (int)end, prefix[b], tiles[b], stream_tiles);
      if (seg.last > seg.first) {
        if (*num_segments < max_segments) {
          const int32_t record[7] = {unit, b, seg.stream, seg.first, seg.last, seg.slot, seg.partials};
          for (int i = 0; i < 7; ++i) segments[(int64_t)*num_segments * 7 + i] = record[i];
        }
        ++*num_segments;
      }
      pos += seg.positions;
    }
  }
  return ANNA_OK;
}
