// Even-share schedule for a persistent split pass.
//
// The 16-token tiles of all (row, stream) pairs form one line in (row, stream-in-row, tile) order, where a "stream" is
// one (kv head, group of up to 8 query heads) of a row.  The grid is one resident wave and CTA c owns tiles
// [c * tpc, (c + 1) * tpc).  A CTA walks its range stream by stream and emits one split-K partial per stream it
// touches, so every CTA moves the same number of bytes whatever the mix of context lengths, and a long context costs
// one pipeline start per CTA instead of one per fixed-size chunk.  Every CTA recomputes the partition from the
// device-side lengths (a block-wide scan), so no host round trip is needed; the slot of each partial and the number
// of partials per stream (for the arrival counter of the fused merge) follow from the same arithmetic, which is host code
// as well (anna_kv_selftest_even_shares walks it).
#pragma once

#include "common.cuh"

namespace anna {

constexpr int kBalancedMaxRows = 1024;
constexpr int kBalancedMinTiles = 4;   // per CTA: one tile per warp
constexpr int kBalancedTileTokens = 16;

// Positions on the line that a stream of `tiles` tiles takes: its tiles, in front of them what a segment costs beside them
// (`stream_tiles`, in tiles), or its pieces of at most `piece_tiles` tiles.
__host__ __device__ __forceinline__ int balanced_line_length(int tiles, int stream_tiles, int piece_tiles) {
  if (tiles == 0) return 0;
  return piece_tiles > 0 ? (tiles + piece_tiles - 1) / piece_tiles : tiles + stream_tiles;
}

// Rows of a thread: batch <= kBalancedMaxRows rows dealt in runs of ceil(batch / THREADS).
template <int THREADS>
constexpr int kBalancedRowsPerThread = (kBalancedMaxRows + THREADS - 1) / THREADS;

// Tiles of each stream of this thread's rows; the newest `tail` tokens of a row have no tile.
template <int THREADS>
__device__ __forceinline__ void balanced_load_tiles(const int64_t* visible_lengths, int64_t max_len, int batch, int tail,
                                                    int (&tiles)[kBalancedRowsPerThread<THREADS>]) {
  const int rpt = (batch + THREADS - 1) / THREADS;
#pragma unroll
  for (int i = 0; i < kBalancedRowsPerThread<THREADS>; ++i) {
    const int b = threadIdx.x * rpt + i;
    tiles[i] = 0;
    if (i < rpt && b < batch) {
      int64_t len = visible_lengths ? visible_lengths[b] : max_len;
      len = max((int64_t)0, min(len, max_len) - tail);
      tiles[i] = (int)((len + kBalancedTileTokens - 1) / kBalancedTileTokens);
    }
  }
}

// Block-wide exclusive scan of the line: s_prefix[b] = positions (over all streams) of the rows before row b,
// s_prefix[batch] = all positions.  Returns the largest number of tiles of any single stream.  Ends with a barrier.
// THREADS = blockDim.x (a multiple of 32).  *streams = streams with a tile.
template <int THREADS>
__device__ __forceinline__ int balanced_scan(const int (&tiles)[kBalancedRowsPerThread<THREADS>], int batch,
                                             int streams_per_row, int* s_prefix, int stream_tiles, int piece_tiles,
                                             int* streams) {
  constexpr int kWarps = THREADS / 32;
  constexpr int kRowsPerThread = kBalancedRowsPerThread<THREADS>;
  __shared__ int s_warp_sum[kWarps];
  __shared__ int s_warp_max[kWarps];
  __shared__ int s_warp_rows[kWarps];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int rpt = (batch + THREADS - 1) / THREADS;
  int local[kRowsPerThread];
  int sum = 0, mx = 0, rows = 0;
#pragma unroll
  for (int i = 0; i < kRowsPerThread; ++i) {
    local[i] = 0;
    if (i < rpt) {
      local[i] = balanced_line_length(tiles[i], stream_tiles, piece_tiles);
      mx = max(mx, tiles[i]);
      rows += tiles[i] > 0 ? 1 : 0;
      sum += local[i];
    }
  }
  int incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += v;
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, d));
  }
  rows = __reduce_add_sync(0xffffffffu, rows);
  if (lane == 31) s_warp_sum[warp] = incl;
  if (lane == 0) {
    s_warp_max[warp] = mx;
    s_warp_rows[warp] = rows;
  }
  __syncthreads();
  int excl = incl - sum;
  int total = 0, max_tiles = 0, filled = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) excl += s_warp_sum[w];
    total += s_warp_sum[w];
    max_tiles = max(max_tiles, s_warp_max[w]);
    filled += s_warp_rows[w];
  }
  *streams = filled * streams_per_row;
#pragma unroll
  for (int i = 0; i < kRowsPerThread; ++i) {
    const int b = threadIdx.x * rpt + i;
    if (i < rpt && b < batch) s_prefix[b] = excl * streams_per_row;
    excl += local[i];
  }
  if (threadIdx.x == 0) s_prefix[batch] = total * streams_per_row;
  __syncthreads();
  return max_tiles;
}

// How the line is cut among `units` CTAs: `share` positions each, which may cross from one stream into the next; or, when
// piece_tiles > 0, one piece of a single stream each (share = 1 position of the line of pieces).
struct BalancedCut {
  int share;
  int piece_tiles;
};

// line = positions of all streams, max_tiles = tiles of the longest stream, capacity = partial slots of a stream.
// A share is even, at least `min_tiles`, and long enough that no stream needs more partial slots than there are (a stream of
// n tiles touches at most ceil(n / share) + 1 units).
//
// Every segment costs about as much as `segment_tiles` tiles beside its own (first copies, merge), which is most of a short
// one.  `stream_tiles` puts the first segment of every stream on the line, so that a CTA that comes upon many short streams
// takes fewer of them (96 quantized rows of 129-1000 tokens with 8 KV heads: 127 us when a share counted tiles only, 54
// now); a CTA then spends `share` and, when it begins inside a stream, one segment more.
//
// Pieces have no crossing: with t = tiles / (units - streams) tiles at most in each, the streams have no more than
// tiles / t + streams = units pieces, and t beyond the longest stream is one piece per stream.  They are taken when a piece
// costs no more than a share with its further segment (half of a stream's first one is left out of that: 64 quantized rows
// of 1000 tokens at head_dim 256 39.0 us in pieces, 41.7 in shares no longer than a piece).
__host__ __device__ __forceinline__ BalancedCut balanced_cut(int line, int streams, int max_tiles, int units, int capacity,
                                                             int min_tiles, int segment_tiles, int stream_tiles) {
  const auto ceil_div = [](int a, int b) { return (a + b - 1) / b; };
  const auto larger = [](int a, int b) { return a > b ? a : b; };
  BalancedCut cut{larger(larger(ceil_div(line, units), min_tiles), ceil_div(max_tiles, capacity - 1)), 0};
  if (segment_tiles > 0 && streams < units) {
    const int tiles = line - streams * stream_tiles;
    int t = larger(larger(ceil_div(tiles, units - streams), min_tiles), ceil_div(max_tiles, capacity));
    if (t > max_tiles) t = max_tiles;
    if (t - cut.share <= segment_tiles - stream_tiles / 2) cut = BalancedCut{1, t};
  }
  return cut;
}

// One stream's part of the positions [pos, end) of a CTA, pos inside row b, whose streams have `tiles` tiles each.
struct BalancedSegment {
  int stream;
  int first, last;  // tiles [first, last) of the stream; none when the part holds nothing but the cost of the segment
  int slot;         // of the partial
  int partials;     // of the stream
  int positions;    // how far this part goes
};

__host__ __device__ __forceinline__ BalancedSegment balanced_segment(const BalancedCut& cut, int unit, int pos, int end,
                                                                     int row_first, int tiles, int stream_tiles) {
  BalancedSegment seg;
  const int n = balanced_line_length(tiles, stream_tiles, cut.piece_tiles);
  seg.stream = (pos - row_first) / n;
  const int at = (pos - row_first) - seg.stream * n;  // position inside the stream
  seg.positions = n - at < end - pos ? n - at : end - pos;
  if (cut.piece_tiles > 0) {
    seg.slot = at;
    seg.partials = n;
    seg.first = (int)((int64_t)tiles * at / n);
    seg.last = (int)((int64_t)tiles * (at + 1) / n);
  } else {
    const int stream_first = row_first + seg.stream * n;
    const int first_unit = (stream_first + stream_tiles) / cut.share;  // the CTA that has the first tile
    seg.slot = unit - first_unit;
    seg.partials = (stream_first + n - 1) / cut.share - first_unit + 1;
    seg.first = at > stream_tiles ? at - stream_tiles : 0;
    seg.last = at + seg.positions - stream_tiles;
  }
  return seg;
}

// The line of a batch of at most 32 rows, worked out by every warp for itself, a row per lane: no barriers and no shared
// memory between the load of the lengths and the first tile.
struct WarpLine {
  int len;          // of this lane's row, without its tail
  int tiles;        // of each of the row's streams
  int first, next;  // positions of the row's streams: [first, next)

  __device__ __forceinline__ void load(const int64_t* visible_lengths, int64_t max_len, int batch, int tail) {
    const int b = threadIdx.x & 31;
    int64_t n = 0;
    if (b < batch) n = max((int64_t)0, min(visible_lengths ? visible_lengths[b] : max_len, max_len) - tail);
    len = (int)n;
    tiles = (len + kBalancedTileTokens - 1) / kBalancedTileTokens;
  }
  // returns all positions
  __device__ __forceinline__ int scan(int streams_per_row, int stream_tiles, int piece_tiles) {
    const int lane = threadIdx.x & 31;
    const int n = balanced_line_length(tiles, stream_tiles, piece_tiles) * streams_per_row;
    next = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, next, d);
      if (lane >= d) next += v;
    }
    first = next - n;
    return __shfl_sync(0xffffffffu, next, 31);
  }
};

// Calls zero_row(b) for this CTA's share of the rows without any visible key, then
// segment(b, stream, t0, t1, slot, partials_of_stream) for each piece of this CTA's tile range, in order.
// THREADS = blockDim.x (a multiple of 32, at most 1024 / 8 rows per thread); all threads of the CTA must call it and
// `segment` may synchronise the CTA.  `tail`: the newest tokens of every row that the line leaves out; the rest: see
// balanced_cut.  kWarpLine: batches of at most 32 rows are lined up in registers (WarpLine), which a kernel has to have room
// for: un-quantized decode of 4 rows of 60-900 tokens 12.3 -> 10.8 us, but one
// packed row of 4000 tokens 18.6 -> 20.2, where the row's state went to local memory and back around every segment.
template <int THREADS, bool kWarpLine, typename ZeroFn, typename SegmentFn>
__device__ __forceinline__ void balanced_for_each_segment(const int64_t* visible_lengths, int64_t max_len, int batch,
                                                          int streams_per_row, int chunk_capacity, ZeroFn&& zero_row,
                                                          SegmentFn&& segment, int tail, int min_tiles, int segment_tiles,
                                                          int stream_tiles) {
  __shared__ int s_prefix[kBalancedMaxRows + 1];
  const bool small = kWarpLine && batch <= 32;
  WarpLine line{};
  int tiles_of_rows[kBalancedRowsPerThread<THREADS>];
  if (small) line.load(visible_lengths, max_len, batch, tail);
  else balanced_load_tiles<THREADS>(visible_lengths, max_len, batch, tail, tiles_of_rows);
  int streams = 0, max_tiles, total;
  if (small) {
    total = line.scan(streams_per_row, stream_tiles, 0);
    max_tiles = __reduce_max_sync(0xffffffffu, line.tiles);
    const unsigned filled = __ballot_sync(0xffffffffu, line.tiles > 0);
    streams = __popc(filled) * streams_per_row;
    for (int b = blockIdx.x; b < batch; b += gridDim.x)
      if (!((filled >> b) & 1u)) zero_row(b);
  } else {
    max_tiles = balanced_scan<THREADS>(tiles_of_rows, batch, streams_per_row, s_prefix, stream_tiles, 0, &streams);
    total = s_prefix[batch];
    // rows without a visible key have no tile: their zero outputs are dealt round-robin
    for (int b = blockIdx.x; b < batch; b += gridDim.x)
      if (s_prefix[b + 1] == s_prefix[b]) zero_row(b);
  }
  if (total == 0) return;

  const BalancedCut cut = balanced_cut(total, streams, max_tiles, (int)gridDim.x, chunk_capacity, min_tiles, segment_tiles,
                                       stream_tiles);
  if (cut.piece_tiles > 0) {  // the line of pieces instead of tiles
    if (small) {
      total = line.scan(streams_per_row, 0, cut.piece_tiles);
    } else {
      __syncthreads();  // s_prefix is written again
      balanced_scan<THREADS>(tiles_of_rows, batch, streams_per_row, s_prefix, 0, cut.piece_tiles, &streams);
      total = s_prefix[batch];
    }
  }
  int pos = (int)min((int64_t)blockIdx.x * cut.share, (int64_t)total);
  const int end = (int)min((int64_t)pos + cut.share, (int64_t)total);
  if (pos >= end) return;

  int b = 0;
  if (!small) {  // row that holds position `pos`: the last b with s_prefix[b] <= pos (rows without tiles are skipped)
    int lo = 0, hi = batch;  // invariant: s_prefix[lo] <= pos < s_prefix[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_prefix[mid] <= pos) lo = mid; else hi = mid;
    }
    b = lo;
  }
  while (pos < end) {
    int len, row_first;
    if (small) {
      b = __popc(__ballot_sync(0xffffffffu, line.next <= pos));  // rows that end at or before it (never all: pos < total)
      len = __shfl_sync(0xffffffffu, line.len, b);
      row_first = __shfl_sync(0xffffffffu, line.first, b);
    } else {
      while (s_prefix[b + 1] <= pos) ++b;
      const int64_t n = visible_lengths ? visible_lengths[b] : max_len;
      len = (int)max((int64_t)0, min(n, max_len) - tail);
      row_first = s_prefix[b];
    }
    const int tiles = (len + kBalancedTileTokens - 1) / kBalancedTileTokens;
    const BalancedSegment seg = balanced_segment(cut, (int)blockIdx.x, pos, end, row_first, tiles, stream_tiles);
    if (seg.last > seg.first)
      segment(b, seg.stream, seg.first * kBalancedTileTokens, min(len, seg.last * kBalancedTileTokens), seg.slot,
              seg.partials);
    pos += seg.positions;
  }
}

// Whether the schedule can be used for this problem (host side).
inline bool balanced_schedule_fits(int batch, int64_t streams_per_row, int64_t max_len, int chunk_capacity,
                                   int stream_tiles) {
  if (batch > kBalancedMaxRows || chunk_capacity < 2) return false;
  return (int64_t)batch * streams_per_row * ((max_len + kBalancedTileTokens - 1) / kBalancedTileTokens + stream_tiles) <
         ((int64_t)1 << 30);
}

}  // namespace anna
