// Building blocks of the kernels that work on several tokens per warp (appends of chunks, dense views): a lane holds 16
// coordinates of a token (D/16 lanes per token, so 8, 4 or 2 tokens per warp at head_dim 64, 128, 256) as pairs (i, i + 8)
// that the packed fp32 instructions work on together.
#pragma once

#include "tq_common.cuh"

#include <type_traits>

namespace anna {

__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
  uint64_t v;
  asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
  return v;
}
__device__ __forceinline__ void halves_of(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add_pair(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// A packed product that goes into a packed sum is contracted with it, explicit rounding or not (one in twenty residual norms was
// off by its last bit), so this one is for products that are exact or go elsewhere.
__device__ __forceinline__ uint64_t mul_pair(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// The product with rounding of its own, whatever becomes of it.
__device__ __forceinline__ uint64_t mul_pair_rounded(uint64_t a, uint64_t b) {
  float a_lo, a_hi, b_lo, b_hi;
  halves_of(a, a_lo, a_hi);
  halves_of(b, b_lo, b_hi);
  return pair_of(__fmul_rn(a_lo, b_lo), __fmul_rn(a_hi, b_hi));
}

constexpr int kBulkCoords = 16;              // coordinates of a token per lane
constexpr int kBulkPairs = kBulkCoords / 2;  // pair i = coordinates i and i + 8 of the lane's run
constexpr int kBulkWarps = 4;

// The same butterflies as warp_fwht (strides 1, 2, 4, ... D/2, every sum and difference rounded once).
template <int LANES>
__device__ __forceinline__ void bulk_fwht(uint64_t (&w)[kBulkPairs], int lane) {
  const uint64_t minus = pair_of(-1.0f, -1.0f);
#pragma unroll
  for (int h = 1; h < kBulkPairs; h <<= 1) {
#pragma unroll
    for (int i = 0; i < kBulkPairs; ++i) {
      if ((i & h) == 0) {
        const uint64_t a = w[i], b = w[i + h];
        w[i] = add_pair(a, b);
        w[i + h] = fma_pair(b, minus, a);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kBulkPairs; ++i) {
    float lo, hi;
    halves_of(w[i], lo, hi);
    w[i] = pair_of(__fadd_rn(lo, hi), __fsub_rn(lo, hi));
  }
#pragma unroll
  for (int dl = 1; dl < LANES; dl <<= 1) {
    const float sgn = (lane & dl) != 0 ? -1.0f : 1.0f;
    const uint64_t sgn2 = pair_of(sgn, sgn);
#pragma unroll
    for (int i = 0; i < kBulkPairs; ++i) {
      float lo, hi;
      halves_of(w[i], lo, hi);
      lo = __shfl_xor_sync(0xffffffffu, lo, dl);
      hi = __shfl_xor_sync(0xffffffffu, hi, dl);
      w[i] = fma_pair(w[i], sgn2, pair_of(lo, hi));
    }
  }
}

// Sum of the squares of a token's coordinates in the order of warp_tree_sum; every lane of the token gets it.
template <int LANES>
__device__ __forceinline__ float bulk_square_sum(const uint64_t (&w)[kBulkPairs]) {
  uint64_t t[kBulkPairs];
#pragma unroll
  for (int i = 0; i < kBulkPairs; ++i) t[i] = mul_pair_rounded(w[i], w[i]);
#pragma unroll
  for (int h = 1; h < kBulkPairs; h <<= 1)
#pragma unroll
    for (int i = 0; i < kBulkPairs; i += 2 * h) t[i] = add_pair(t[i], t[i + h]);
  float lo, hi;
  halves_of(t[0], lo, hi);
  float s = __fadd_rn(lo, hi);
#pragma unroll
  for (int dl = 1; dl < LANES; dl <<= 1) s = __fadd_rn(s, __shfl_xor_sync(0xffffffffu, s, dl));
  return s;
}

// A lane's 16 elements as loaded: 16 bytes at a time.
template <typename T>
struct BulkRaw {
  static constexpr int kWords = kBulkCoords * (int)sizeof(T) / 4;
  uint32_t w[kWords];
  __device__ __forceinline__ void load(const T* ptr) {
#pragma unroll
    for (int c = 0; c < kWords / 4; ++c) {
      const uint4 v = reinterpret_cast<const uint4*>(ptr)[c];
      w[4 * c] = v.x; w[4 * c + 1] = v.y; w[4 * c + 2] = v.z; w[4 * c + 3] = v.w;
    }
  }
  __device__ __forceinline__ void store(T* ptr) const {
#pragma unroll
    for (int c = 0; c < kWords / 4; ++c)
      reinterpret_cast<uint4*>(ptr)[c] = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
  }
  __device__ __forceinline__ float value(int j) const {
    if constexpr (sizeof(T) == 4) {
      return __uint_as_float(w[j]);
    } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      return __uint_as_float(j % 2 == 0 ? w[j / 2] << 16 : w[j / 2] & 0xffff0000u);
    } else {
      const __half2 h = *reinterpret_cast<const __half2*>(&w[j / 2]);
      return j % 2 == 0 ? __low2float(h) : __high2float(h);
    }
  }
  __device__ __forceinline__ void set(int j, float lo, float hi) {  // elements j, j + 1 (j even)
    if constexpr (sizeof(T) == 4) {
      w[j] = __float_as_uint(lo);
      w[j + 1] = __float_as_uint(hi);
    } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
      w[j / 2] = *reinterpret_cast<const uint32_t*>(&v);
    } else {
      const __half2 v = __floats2half2_rn(lo, hi);
      w[j / 2] = *reinterpret_cast<const uint32_t*>(&v);
    }
  }
  __device__ __forceinline__ uint64_t pair(int i) const { return pair_of(value(i), value(i + kBulkPairs)); }
  // Smallest and largest element; NaNs lose against numbers, as in fminf / fmaxf.
  __device__ __forceinline__ void extremes(float& lo, float& hi) const {
    if constexpr (sizeof(T) == 4) {
      lo = hi = value(0);
#pragma unroll
      for (int j = 1; j < kBulkCoords; ++j) {
        lo = fminf(lo, value(j));
        hi = fmaxf(hi, value(j));
      }
    } else {
      using T2 = typename std::conditional<std::is_same<T, __nv_bfloat16>::value, __nv_bfloat162, __half2>::type;
      T2 lo2 = *reinterpret_cast<const T2*>(&w[0]), hi2 = lo2;
#pragma unroll
      for (int k = 1; k < kWords; ++k) {
        const T2 v = *reinterpret_cast<const T2*>(&w[k]);
        lo2 = __hmin2(lo2, v);
        hi2 = __hmax2(hi2, v);
      }
      lo = fminf(ElemTraits<T>::to_float(lo2.x), ElemTraits<T>::to_float(lo2.y));
      hi = fmaxf(ElemTraits<T>::to_float(hi2.x), ElemTraits<T>::to_float(hi2.y));
    }
  }
};

// BITS_PER-bit fields of a lane's 16 coordinates as words of its packed row: coordinate j at bit BITS_PER * j.
template <int BITS_PER>
struct BulkFields {
  static constexpr int kWords = kBulkCoords * BITS_PER >= 32 ? kBulkCoords * BITS_PER / 32 : 1;
  static __device__ __forceinline__ void store(uint8_t* row, int token_lane, const uint32_t (&f)[kWords]) {
    if constexpr (BITS_PER == 4) reinterpret_cast<uint2*>(row)[token_lane] = make_uint2(f[0], f[1]);
    else if constexpr (BITS_PER == 2) reinterpret_cast<uint32_t*>(row)[token_lane] = f[0];
    else reinterpret_cast<uint16_t*>(row)[token_lane] = (uint16_t)f[0];
  }
  static __device__ __forceinline__ void load(const uint8_t* row, int token_lane, uint32_t (&f)[kWords]) {
    if constexpr (BITS_PER == 4) {
      const uint2 v = reinterpret_cast<const uint2*>(row)[token_lane];
      f[0] = v.x;
      f[kWords - 1] = v.y;
    } else if constexpr (BITS_PER == 2) {
      f[0] = reinterpret_cast<const uint32_t*>(row)[token_lane];
    } else {
      f[0] = reinterpret_cast<const uint16_t*>(row)[token_lane];
    }
  }
};

// CTAs of a kernel that fit the whole GPU at once, worked out at its first launch on a device.
template <typename Kernel>
static int bulk_resident_ctas(Kernel kernel, int threads, int (&known)[64], int device, int* ctas) {
  *ctas = (device >= 0 && device < 64) ? known[device] : 0;
  if (*ctas != 0) return ANNA_OK;
  int sms = 0, per_sm = 0;
  ANNA_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  ANNA_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, 0));
  *ctas = sms * (per_sm > 0 ? per_sm : 1);
  if (device >= 0 && device < 64) known[device] = *ctas;
  return ANNA_OK;
}

// Pieces that the tokens of each (row, kv head) are cut into: what fills one to four resident waves of CTAs, whichever has the fewest
// trips one after the other (waves x trips of a CTA), a wave's start counted as one more trip.
inline int bulk_chunks(int64_t heads_total, int64_t trips, int resident) {
  int64_t best = 1, best_cost = INT64_MAX;
  for (int64_t waves = 1; waves <= 4; ++waves) {
    int64_t chunks = waves * resident / heads_total;
    if (chunks > trips) chunks = trips;
    if (chunks < 1) chunks = 1;
    const int64_t cost = ((heads_total * chunks + resident - 1) / resident) * ((trips + chunks - 1) / chunks + 1);
    if (cost < best_cost) { best_cost = cost; best = chunks; }
  }
  return (int)(best < (1 << 30) ? best : (1 << 30));
}

}  // namespace anna
