// Split-K merge done by the last CTA that finishes a (row, kv-head group): no second launch, no waiting.
//
// Every CTA of the split pass publishes its partial and bumps a per-(row, group) counter (an acquire-release).  The CTA that
// observes the final count owns the merge: it re-reads the partials (L2 resident), applies the optional sigmoid(gate)
// epilogue and stores the output row.  Nobody spins: a CTA either is last or leaves.  The counter is reset by the
// merging CTA, so the caller's buffer stays all-zero between launches.
#pragma once

#include <type_traits>

#include "common.cuh"

namespace anna {

struct FusedCombine {
  int32_t* counters;   // [batch, kv heads x groups-of-8] zero on entry; nullptr selects the two-pass path
  void* out;
  int64_t out_stride_b, out_stride_h;
  const void* gate;
  int64_t gate_stride_b, gate_stride_h;
  // KV-head-sharded decode: the same rows of the output tensors of the other ranks (peer memory mapped into this
  // process).  Every merged output row is stored to all of them at the offset it has in `out`.
  void* peers[kMaxPeerOutputs];
  int num_peers;
};

constexpr int kFusedMaxChunks = 512;  // weights of one head are staged in shared memory

// ---- what both forms of the merge below are made of ----------------------------------------------------------------------

// Counts this CTA's partial; true in all threads of the CTA that is the last of `arrivals`.
__device__ __forceinline__ bool merge_arrive(const FusedCombine& fc, int64_t counter_index, int arrivals) {
  __shared__ int s_is_last;
  __syncthreads();  // all partial stores of this CTA are ordered before the arrival below
  if (threadIdx.x == 0) {
    // releases this CTA's partial and acquires those of the CTAs counted before; the barriers on both sides extend that to
    // the other threads (4 un-quantized rows of 60-900 tokens: 10.8 us with a full fence on either side, 10.3 so)
    int32_t* counter = fc.counters + counter_index;
    int prev;
    asm volatile("atom.acq_rel.gpu.global.add.s32 %0, [%1], 1;\n" : "=r"(prev) : "l"(counter) : "memory");
    s_is_last = (prev == arrivals - 1) ? 1 : 0;
    if (s_is_last) *counter = 0;
  }
  __syncthreads();
  return s_is_last != 0;
}

// A warp works out the weights of one head: max, denominator, normalised weights.
__device__ __forceinline__ void merge_weigh_head(const float* stats, int chunk_capacity, int active_chunks, float* smem_weights, int g,
                                                 int lane) {
  const float* st = stats + (int64_t)g * chunk_capacity * 2;
  float m = -INFINITY;
  for (int c = lane; c < active_chunks; c += 32) m = fmaxf(m, __ldcg(st + 2 * c));
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
  const float m_ref = m == -INFINITY ? 0.0f : m;
  float den = 0.0f;
  for (int c = lane; c < active_chunks; c += 32) {
    const float w = __expf(__ldcg(st + 2 * c) - m_ref);
    den += __ldcg(st + 2 * c + 1) * w;
    smem_weights[g * kFusedMaxChunks + c] = w;
  }
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) den += __shfl_xor_sync(0xffffffffu, den, d);
  const float inv = den > 0.0f ? 1.0f / den : 0.0f;
  for (int c = lane; c < active_chunks; c += 32) smem_weights[g * kFusedMaxChunks + c] *= inv;
}

__device__ __forceinline__ void merge_add(float4& acc, const float4& v, float w) {
  acc.x = fmaf(v.x, w, acc.x);
  acc.y = fmaf(v.y, w, acc.y);
  acc.z = fmaf(v.z, w, acc.z);
  acc.w = fmaf(v.w, w, acc.w);
}

// Four dims of a query head, gated, to this GPU's output and the peers'.
template <typename T>
__device__ __forceinline__ void merge_store4(const FusedCombine& fc, int b, int hq, int d, const float4& o) {
  const float acc[4] = {o.x, o.y, o.z, o.w};
  const T* gate = fc.gate == nullptr ? nullptr
                                     : reinterpret_cast<const T*>(fc.gate) + (int64_t)b * fc.gate_stride_b +
                                           (int64_t)hq * fc.gate_stride_h + d;
  const int64_t offset = (int64_t)b * fc.out_stride_b + (int64_t)hq * fc.out_stride_h + d;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const T result = ElemTraits<T>::from_float(gate ? acc[i] * sigmoidf_fast(ElemTraits<T>::to_float(gate[i])) : acc[i]);
    reinterpret_cast<T*>(fc.out)[offset + i] = result;
    for (int peer = 0; peer < fc.num_peers; ++peer) reinterpret_cast<T*>(fc.peers[peer])[offset + i] = result;
  }
}

// The whole sum, one dim per thread, where the values are not aligned for four; then the fence behind the peers' stores.
template <typename T, int D, int THREADS>
__device__ __forceinline__ void merge_finish(const FusedCombine& fc, int b, int hq0, int g_count, int active_chunks, int chunk_capacity,
                                             const float* values, const float* smem_weights, bool aligned) {
  for (int item = threadIdx.x; !aligned && item < g_count * D; item += THREADS) {
    const int g = item / D;
    const int d = item % D;
    const float* vals = values + (int64_t)g * chunk_capacity * D + d;
    const float* w = smem_weights + g * kFusedMaxChunks;
    float acc = 0.0f;
    for (int c = 0; c < active_chunks; ++c) acc = fmaf(__ldcg(vals + (int64_t)c * D), w[c], acc);
    if (fc.gate) {
      const T* gate = reinterpret_cast<const T*>(fc.gate) + (int64_t)b * fc.gate_stride_b +
                      (int64_t)(hq0 + g) * fc.gate_stride_h;
      acc *= sigmoidf_fast(ElemTraits<T>::to_float(gate[d]));
    }
    const int64_t offset = (int64_t)b * fc.out_stride_b + (int64_t)(hq0 + g) * fc.out_stride_h + d;
    const T result = ElemTraits<T>::from_float(acc);
    reinterpret_cast<T*>(fc.out)[offset] = result;
    for (int peer = 0; peer < fc.num_peers; ++peer) reinterpret_cast<T*>(fc.peers[peer])[offset] = result;
  }
  // stores to other GPUs are ordered before whatever this stream signals to them after the kernel
  if (fc.num_peers > 0) __threadfence_system();
}

// Called by all threads of the CTA after they wrote their partial.  `active_chunks` = partials that contribute to this
// (row, group); `arrivals` of them (0 = all; the others are known to be complete before any arrival) are counted in
// counters[counter_index]; stats / values point at chunk 0 of query head hq0.  Natural-log stats.  THREADS = blockDim.x,
// HEADS = most query heads of a group, MERGE: how the values are read, see below.
enum class MergeLoads { kOneColumn, kAllColumns, kAllOrTwoColumns };
template <typename T, int D, int THREADS, int HEADS = 8, MergeLoads MERGE = MergeLoads::kAllOrTwoColumns>
__device__ __forceinline__ void fused_combine_tail(const FusedCombine& fc, int b, int hq0, int g_count,
                                                   int active_chunks, int chunk_capacity, const float* stats,
                                                   const float* values, float* smem_weights /* [8][kFusedMaxChunks] */,
                                                   int64_t counter_index, int arrivals = 0) {
  if (!merge_arrive(fc, counter_index, arrivals > 0 ? arrivals : active_chunks)) return;

  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  constexpr int kWarps = THREADS / 32;
  for (int g = warp; g < g_count; g += kWarps) merge_weigh_head(stats, chunk_capacity, active_chunks, smem_weights, g, lane);
  __syncthreads();
  auto store = [&](int g, int d, const float4& o) { merge_store4<T>(fc, b, hq0 + g, d, o); };
  // Four dims per thread and load.  What this part takes is the latency of its loads: a head group with more columns of four
  // dims than the CTA has threads reads all of a thread's columns side by side, kInFlight loads at a time, instead of one
  // column after the other (16 rows of 0.4-4 K packed tokens, 16/2 heads of 256: 37.1 -> 34.9 us; 64 rows of 4-32 K 170 ->
  // 168.4).  With 16 loads in flight the even-share kernels lost more to spilled registers than the merge gained, and with one
  // column per thread eight at a time are no faster than a plain loop (one packed row of 4000 tokens: 20.6 us and 18.5).
  const bool aligned = (reinterpret_cast<uintptr_t>(values) & 15u) == 0;
  constexpr int kCols = D / 4;
  constexpr int kRounds = (HEADS * kCols + THREADS - 1) / THREADS;
  constexpr int kInFlight = 8;
  const int items = g_count * kCols;
  auto side_by_side = [&](auto columns) {
    constexpr int kColumns = decltype(columns)::value;  // of a thread
    constexpr int kAtOnce = kInFlight / kColumns;       // partials
    float4 acc[kColumns];
    const float* vals[kColumns];
#pragma unroll
    for (int r = 0; r < kColumns; ++r) {
      const int item = min((int)threadIdx.x + r * THREADS, items - 1);  // past the end: the last column again, not stored
      acc[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      vals[r] = values + (int64_t)(item / kCols) * chunk_capacity * D + 4 * (item % kCols);
    }
    for (int c0 = 0; c0 < active_chunks; c0 += kAtOnce) {
      float4 v[kAtOnce][kColumns];
#pragma unroll
      for (int k = 0; k < kAtOnce; ++k)
#pragma unroll
        for (int r = 0; r < kColumns; ++r)
          v[k][r] = __ldcg(reinterpret_cast<const float4*>(vals[r] + (int64_t)min(c0 + k, active_chunks - 1) * D));
#pragma unroll
      for (int r = 0; r < kColumns; ++r) {
        const float* w = smem_weights + min(((int)threadIdx.x + r * THREADS) / kCols, g_count - 1) * kFusedMaxChunks;
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k)
          if (c0 + k < active_chunks) merge_add(acc[r], v[k][r], w[c0 + k]);
      }
    }
#pragma unroll
    for (int r = 0; r < kColumns; ++r) {
      const int item = (int)threadIdx.x + r * THREADS;
      if (item < items) store(item / kCols, 4 * (item % kCols), acc[r]);
    }
  };
  // No more columns than the group has: with four of them for two (four heads of 256) every second load is in vain (one packed
  // row of 20000 tokens, 8/2 heads: 42.4 us, 31.0 so, 38.6 one column after the other; 4 un-quantized rows of 3-6 K 14.6, 12.9
  // and 15.9).  Kernels that know HEADS have one form of the loop, which costs fewer registers than two.
  constexpr bool kTwo = kRounds > 2 && MERGE == MergeLoads::kAllOrTwoColumns;
  if (MERGE != MergeLoads::kOneColumn && kRounds > 1 && aligned && items > (kTwo ? 2 : 1) * THREADS) {
    side_by_side(std::integral_constant<int, kRounds>{});
  } else if (kTwo && aligned && items > THREADS) {
    side_by_side(std::integral_constant<int, 2>{});
  } else if (aligned) {
    auto column = [&](int item) {
      const int g = item / kCols, d = 4 * (item % kCols);
      const float* vals = values + (int64_t)g * chunk_capacity * D + d;
      const float* w = smem_weights + g * kFusedMaxChunks;
      float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
      for (int c = 0; c < active_chunks; ++c)
        merge_add(acc, __ldcg(reinterpret_cast<const float4*>(vals + (int64_t)c * D)), w[c]);
      store(g, d, acc);
    };
    // a loop also where no thread has a second column: the compiler makes the better code of it at head_dim 256 (16 packed rows of 201
    // tokens, 4/2 heads: 11.7 us, 12.4 without), and the worse one at 128 (one of 4000, 32/8 heads: 14.1 and 13.6)
    if constexpr (MERGE == MergeLoads::kOneColumn || D == 256) {
      for (int item = threadIdx.x; item < items; item += THREADS) column(item);
    } else {
      if ((int)threadIdx.x < items) column(threadIdx.x);
    }
  }
  merge_finish<T, D, THREADS>(fc, b, hq0, g_count, active_chunks, chunk_capacity, values, smem_weights, aligned);
}

// The same with the first values read beside the statistics, and these once.  The merge is a chain of reads from L2 (counter,
// statistics twice, values a few at a time), so each one taken out of it is 0.6 us of a call that waits for its last CTA (GPU time: 4
// un-quantized rows of 0.7-5.7 K tokens, 32/4 heads 15.6 -> 13.4 us; 16 packed rows of 0.4-4 K, 16/2 heads of 256 32.1 -> 30.3;
// 240 calls of 1-60 rows by 4 % in the mean).  Kernels that have no registers to spare for it keep the other one (12 packed rows of
// 17000, 8/8 heads, 4 bits 74.4 and 75.8 with this one; two fp32 rows of 300-600, 8/2 heads, CUDA cores 13.9 and 15.8).
template <typename T, int D, int THREADS, int HEADS = 8, MergeLoads MERGE = MergeLoads::kAllOrTwoColumns>
__device__ __forceinline__ void fused_combine_ahead(const FusedCombine& fc, int b, int hq0, int g_count,
                                                    int active_chunks, int chunk_capacity, const float* stats,
                                                   const float* values, float* smem_weights /* [8][kFusedMaxChunks] */,
                                                   int64_t counter_index, int arrivals = 0) {
  if (!merge_arrive(fc, counter_index, arrivals > 0 ? arrivals : active_chunks)) return;

  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  constexpr int kWarps = THREADS / 32;
  auto weigh = [&] {
    // one warp per head: max, denominator, normalised weights.  Where a lane has at most kHeld partials of a head their statistics are
    // read once, and those of the warp's next head beside them.
    constexpr int kHeld = 2;
    if (active_chunks <= 32 * kHeld && (reinterpret_cast<uintptr_t>(stats) & 7u) == 0) {
      for (int g0 = warp; g0 < g_count; g0 += 2 * kWarps) {
        float2 s[2][kHeld];
#pragma unroll
        for (int k = 0; k < 2; ++k)
#pragma unroll
          for (int i = 0; i < kHeld; ++i) {
            const int g = g0 + k * kWarps, c = lane + 32 * i;
            s[k][i] = g < g_count && c < active_chunks
                          ? __ldcg(reinterpret_cast<const float2*>(stats + ((int64_t)g * chunk_capacity + c) * 2))
                          : make_float2(-INFINITY, 0.0f);
          }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const int g = g0 + k * kWarps;
          if (g >= g_count) break;
          float m = s[k][0].x;
#pragma unroll
          for (int i = 1; i < kHeld; ++i) m = fmaxf(m, s[k][i].x);
#pragma unroll
          for (int d = 16; d >= 1; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
          const float m_ref = m == -INFINITY ? 0.0f : m;
          float den = 0.0f;
#pragma unroll
          for (int i = 0; i < kHeld; ++i) {
            const float w = __expf(s[k][i].x - m_ref);
            den += s[k][i].y * w;
            s[k][i].x = w;
          }
#pragma unroll
          for (int d = 16; d >= 1; d >>= 1) den += __shfl_xor_sync(0xffffffffu, den, d);
          const float inv = den > 0.0f ? 1.0f / den : 0.0f;
#pragma unroll
          for (int i = 0; i < kHeld; ++i)
            if (lane + 32 * i < active_chunks) smem_weights[g * kFusedMaxChunks + lane + 32 * i] = s[k][i].x * inv;
        }
      }
    } else {
      for (int g = warp; g < g_count; g += kWarps) merge_weigh_head(stats, chunk_capacity, active_chunks, smem_weights, g, lane);
    }
    __syncthreads();
  };
  auto store = [&](int g, int d, const float4& o) { merge_store4<T>(fc, b, hq0 + g, d, o); };
  const bool aligned = (reinterpret_cast<uintptr_t>(values) & 15u) == 0;
  constexpr int kCols = D / 4;
  constexpr int kRounds = (HEADS * kCols + THREADS - 1) / THREADS;
  constexpr int kInFlight = 8, kAhead = 4;
  const int items = g_count * kCols;
  auto side_by_side = [&](auto columns) {
    constexpr int kColumns = decltype(columns)::value;  // of a thread
    constexpr int kAtOnce = kInFlight / kColumns;       // partials
    float4 acc[kColumns];
    const float* vals[kColumns];
#pragma unroll
    for (int r = 0; r < kColumns; ++r) {
      const int item = min((int)threadIdx.x + r * THREADS, items - 1);  // past the end: the last column again, not stored
      acc[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      vals[r] = values + (int64_t)(item / kCols) * chunk_capacity * D + 4 * (item % kCols);
    }
    float4 v[kAtOnce][kColumns];
    auto load = [&](int c0) {
#pragma unroll
      for (int k = 0; k < kAtOnce; ++k)
#pragma unroll
        for (int r = 0; r < kColumns; ++r)
          v[k][r] = __ldcg(reinterpret_cast<const float4*>(vals[r] + (int64_t)min(c0 + k, active_chunks - 1) * D));
    };
    load(0);
    weigh();
    for (int c0 = 0;;) {
#pragma unroll
      for (int r = 0; r < kColumns; ++r) {
        const float* w = smem_weights + min(((int)threadIdx.x + r * THREADS) / kCols, g_count - 1) * kFusedMaxChunks;
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k)
          if (c0 + k < active_chunks) merge_add(acc[r], v[k][r], w[c0 + k]);
      }
      c0 += kAtOnce;
      if (c0 >= active_chunks) break;
      load(c0);
    }
#pragma unroll
    for (int r = 0; r < kColumns; ++r) {
      const int item = (int)threadIdx.x + r * THREADS;
      if (item < items) store(item / kCols, 4 * (item % kCols), acc[r]);
    }
  };
  constexpr bool kTwo = kRounds > 2 && MERGE == MergeLoads::kAllOrTwoColumns;
  if (MERGE != MergeLoads::kOneColumn && kRounds > 1 && aligned && items > (kTwo ? 2 : 1) * THREADS) {
    side_by_side(std::integral_constant<int, kRounds>{});
  } else if (kTwo && aligned && items > THREADS) {
    side_by_side(std::integral_constant<int, 2>{});
  } else if (aligned) {
    float4 first[kAhead];  // of this thread's first column
    {
      const int item = min((int)threadIdx.x, items - 1);
      const float* vals = values + (int64_t)(item / kCols) * chunk_capacity * D + 4 * (item % kCols);
#pragma unroll
      for (int k = 0; k < kAhead; ++k)
        first[k] = __ldcg(reinterpret_cast<const float4*>(vals + (int64_t)min(k, active_chunks - 1) * D));
    }
    weigh();
    for (int item = threadIdx.x; item < items; item += THREADS) {
      const int g = item / kCols, d = 4 * (item % kCols);
      const float* vals = values + (int64_t)g * chunk_capacity * D + d;
      const float* w = smem_weights + g * kFusedMaxChunks;
      float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      int c = 0;
      if (item < THREADS) {
#pragma unroll
        for (int k = 0; k < kAhead; ++k)
          if (k < active_chunks) merge_add(acc, first[k], w[k]);
        c = kAhead;
      }
#pragma unroll 4
      for (; c < active_chunks; ++c) merge_add(acc, __ldcg(reinterpret_cast<const float4*>(vals + (int64_t)c * D)), w[c]);
      store(g, d, acc);
    }
  } else {
    weigh();
  }
  merge_finish<T, D, THREADS>(fc, b, hq0, g_count, active_chunks, chunk_capacity, values, smem_weights, aligned);
}

// A row with no visible key has no contributing CTA; the CTA of chunk 0 writes its zeros.
template <typename T, int D, int THREADS>
__device__ __forceinline__ void fused_write_zero_row(const FusedCombine& fc, int b, int hq0, int g_count) {
  for (int item = threadIdx.x; item < g_count * D; item += THREADS) {
    const int g = item / D;
    const int d = item % D;
    const int64_t offset = (int64_t)b * fc.out_stride_b + (int64_t)(hq0 + g) * fc.out_stride_h + d;
    reinterpret_cast<T*>(fc.out)[offset] = ElemTraits<T>::from_float(0.0f);
    for (int peer = 0; peer < fc.num_peers; ++peer)
      reinterpret_cast<T*>(fc.peers[peer])[offset] = ElemTraits<T>::from_float(0.0f);
  }
  if (fc.num_peers > 0) __threadfence_system();
}

}  // namespace anna
