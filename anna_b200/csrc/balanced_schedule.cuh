// Even-share schedule for a persistent split pass.
//
// The 16-token tiles of all (row, stream) pairs form one line in (row, stream-in-row, tile) order, where a "stream" is
// one (kv head, group of up to 8 query heads) of a row.  The grid is one resident wave and CTA c owns tiles
// [c * tpc, (c + 1) * tpc).  A CTA walks its range stream by stream and emits one split-K partial per stream it
// touches, so every CTA moves the same number of bytes whatever the mix of context lengths, and a long context costs
// one pipeline start per CTA instead of one per fixed-size chunk.  Every CTA recomputes the partition from the
// device-side lengths (a block-wide scan), so no host round trip is needed; the slot of each partial and the number
// of partials per stream (for the arrival counter of the fused merge) follow from the same arithmetic.
#pragma once

#include "common.cuh"

namespace anna {

constexpr int kBalancedMaxRows = 1024;
constexpr int kBalancedMinTiles = 4;   // per CTA: one tile per warp
constexpr int kBalancedTileTokens = 16;

// Block-wide exclusive scan of the tiles per row: s_prefix[b] = tiles (over all streams) of the rows before row b,
// s_prefix[batch] = all tiles.  Returns the largest number of tiles of any single stream.  Ends with a barrier.
// THREADS = blockDim.x (a multiple of 32); batch <= kBalancedMaxRows.  The newest `tail` tokens of a row have no tile here.
// tiles_per_piece > 0 counts pieces of at most that many tiles instead of tiles.  *streams = streams with a tile.
template <int THREADS>
__device__ __forceinline__ int balanced_scan(const int64_t* visible_lengths, int64_t max_len, int batch,
                                             int streams_per_row, int* s_prefix, int tail, int tiles_per_piece,
                                             int* streams) {
  constexpr int kWarps = THREADS / 32;
  constexpr int kRowsPerThread = (kBalancedMaxRows + THREADS - 1) / THREADS;
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
    const int b = threadIdx.x * rpt + i;
    int tiles = 0;
    if (i < rpt && b < batch) {
      int64_t len = visible_lengths ? visible_lengths[b] : max_len;
      len = max((int64_t)0, min(len, max_len) - tail);
      tiles = (int)((len + kBalancedTileTokens - 1) / kBalancedTileTokens);
    }
    mx = max(mx, tiles);
    rows += tiles > 0 ? 1 : 0;
    if (tiles_per_piece > 0) tiles = (tiles + tiles_per_piece - 1) / tiles_per_piece;
    local[i] = tiles;
    sum += tiles;
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

// Share of tiles per work unit: even, at least `min_tiles`, and long enough that no stream needs more partial slots
// than the caller's scratch holds (a stream of n tiles touches at most ceil(n / share) + 1 units).
__device__ __forceinline__ int balanced_share(int total, int units, int max_tiles, int chunk_capacity, int min_tiles) {
  int share = (total + units - 1) / units;
  share = max(share, min_tiles);
  return max(share, (max_tiles + chunk_capacity - 2) / (chunk_capacity - 1));
}

// Calls zero_row(b) for this CTA's share of the rows without any visible key, then
// segment(b, stream, t0, t1, slot, partials_of_stream) for each piece of this CTA's tile range, in order.
// THREADS = blockDim.x (a multiple of 32, at most 1024 / 8 rows per thread); all threads of the CTA must call it and
// `segment` may synchronise the CTA.  `tail`: the newest tokens of every row that the line leaves out; `min_tiles`: the
// smallest share of a CTA; `segment_tiles`: the cost of a segment beyond its tiles, in tiles (0: shares always cross).
template <int THREADS, typename ZeroFn, typename SegmentFn>
__device__ __forceinline__ void balanced_for_each_segment(const int64_t* visible_lengths, int64_t max_len, int batch,
                                                          int streams_per_row, int chunk_capacity, ZeroFn&& zero_row,
                                                          SegmentFn&& segment, int tail = 0,
                                                          int min_tiles = kBalancedMinTiles, int segment_tiles = 0) {
  __shared__ int s_prefix[kBalancedMaxRows + 1];
  int streams = 0;
  const int max_tiles = balanced_scan<THREADS>(visible_lengths, max_len, batch, streams_per_row, s_prefix, tail, 0, &streams);
  const int total = s_prefix[batch];
  auto row_len = [&](int b) -> int {
    int64_t len = visible_lengths ? visible_lengths[b] : max_len;
    return (int)max((int64_t)0, min(len, max_len) - tail);
  };

  // rows without a visible key have no tile: their zero outputs are dealt round-robin
  for (int b = blockIdx.x; b < batch; b += gridDim.x)
    if (s_prefix[b + 1] == s_prefix[b]) zero_row(b);
  if (total == 0) return;

  const int tpc = balanced_share(total, (int)gridDim.x, max_tiles, chunk_capacity, min_tiles);
  // Short shares: a CTA whose share crosses from one stream into the next pays for two segments, which is most of its
  // time.  Pieces of single streams, one per CTA: with t = total / (CTAs - streams) tiles at most in each, the streams
  // have no more than total / t + streams = CTAs pieces.  Taken when such a piece is less than a segment's cost longer
  // than the even share: 16 quantized rows of 0.4-4 K tokens 49 -> 36 us, 4 un-quantized rows of 60-900 tokens
  // 14.4 -> 12.4 us.
  int piece_tiles = 0;
  if (segment_tiles > 0 && streams < (int)gridDim.x) {
    const int spare = (int)gridDim.x - streams;
    const int t = max(max((total + spare - 1) / spare, min_tiles), (max_tiles + chunk_capacity - 1) / chunk_capacity);
    if (t - tpc < segment_tiles) piece_tiles = t;
  }
  int pos = (int)min((int64_t)blockIdx.x * tpc, (int64_t)total);
  int end = (int)min((int64_t)pos + tpc, (int64_t)total);
  if (piece_tiles > 0) {
    __syncthreads();  // s_prefix is written again: pieces instead of tiles
    balanced_scan<THREADS>(visible_lengths, max_len, batch, streams_per_row, s_prefix, tail, piece_tiles, &streams);
    pos = (int)blockIdx.x;
    end = min(pos + 1, s_prefix[batch]);
  }
  if (pos >= end) return;

  // row that holds position `pos`: the last b with s_prefix[b] <= pos (rows without tiles are skipped by construction)
  int lo = 0, hi = batch;  // invariant: s_prefix[lo] <= pos < s_prefix[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (s_prefix[mid] <= pos) lo = mid; else hi = mid;
  }
  int b = lo;
  while (pos < end) {
    while (s_prefix[b + 1] <= pos) ++b;
    const int row_first = s_prefix[b];
    const int n = (s_prefix[b + 1] - row_first) / streams_per_row;  // tiles (or pieces) of each stream of this row
    const int stream = (pos - row_first) / n;
    int first = (pos - row_first) - stream * n;  // tile (or piece) of the stream
    const int seg = min(n - first, end - pos);
    const int len = row_len(b);
    int slot, partials, last;
    if (piece_tiles > 0) {
      const int tiles = (len + kBalancedTileTokens - 1) / kBalancedTileTokens;
      slot = first;
      partials = n;
      last = (int)((int64_t)tiles * (slot + 1) / n);
      first = (int)((int64_t)tiles * slot / n);
    } else {
      const int stream_first = row_first + stream * n;
      const int first_cta = stream_first / tpc;
      slot = (int)blockIdx.x - first_cta;
      partials = (stream_first + n - 1) / tpc - first_cta + 1;
      last = first + seg;
    }
    segment(b, stream, first * kBalancedTileTokens, min(len, last * kBalancedTileTokens), slot, partials);
    pos += seg;
  }
}

// Whether the schedule can be used for this problem (host side).
inline bool balanced_schedule_fits(int batch, int64_t streams_per_row, int64_t max_len, int chunk_capacity) {
  if (batch > kBalancedMaxRows || chunk_capacity < 2) return false;
  return (int64_t)batch * streams_per_row * ((max_len + kBalancedTileTokens - 1) / kBalancedTileTokens) <
         ((int64_t)1 << 30);
}

}  // namespace anna
