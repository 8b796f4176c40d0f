// Device steps of kyto's per-cell maps (normalize_total, log1p), shared by the map
// entry points and the PCA's pack kernel.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace kg {

// A stored value as kyto's KernelValue reads it (crates/kyto-exec/src/kernels.rs:48-90).
__device__ __forceinline__ double value_wide(const uint32_t* v, uint64_t i, bool round32) {
  return round32 ? (double)__uint2float_rn(v[i]) : (double)v[i];
}
__device__ __forceinline__ double value_wide(const float* v, uint64_t i, bool) {
  return (double)v[i];
}

// The normalize divisor of one row, computed by the 8 threads of an aligned group of 8
// lanes (lane class c = lane % 8 sums values c, c+8, ... of the row in order, as kyto's
// SUM_LANES accumulators; the classes combine in kyto's fixed tree
// ((a0+a4)+(a2+a6))+((a1+a5)+(a3+a7)), kernels.rs:281-292). Every thread of the group
// gets the divisor: f32(total) / f32(target), 0 -> 1 (elementwise.rs:262-269).
// All 32 lanes of the warp must call it together.
// round32: the block holds a u32 count that is not a float32 (elementwise.rs:241-257).
template <class V>
__device__ __forceinline__ float row_divisor(const V* values, uint64_t s, uint64_t e,
                                             float target32, bool round32) {
  const unsigned lane = threadIdx.x & 31u;
  const unsigned c = lane & 7u;
  double acc = 0.0;
  for (uint64_t i = s + c; i < e; i += 8) acc = __dadd_rn(acc, value_wide(values, i, round32));
  const unsigned mask = 0xFFFFFFFFu;  // the whole warp calls this (rows past the end
                                      // pass s == e)
  // h_c = a_c + a_{c+4} (c < 4); q_c = h_c + h_{c+2} (c < 2); total = q_0 + q_1.
  double other = __shfl_down_sync(mask, acc, 4, 8);
  double h = __dadd_rn(acc, other);
  other = __shfl_down_sync(mask, h, 2, 8);
  double q = __dadd_rn(h, other);
  other = __shfl_down_sync(mask, q, 1, 8);
  double total = __dadd_rn(q, other);
  total = __shfl_sync(mask, total, 0, 8);
  float divisor = __fdiv_rn((float)total, target32);
  return divisor == 0.0f ? 1.0f : divisor;
}

// kyto's log1p (crates/kyto-exec/src/kernels/log1p.rs:49-75): ln(1 + x) evaluated in f64
// and rounded once to f32. CUDA's f64 log1p is within an ulp of f64, so the f32
// rounding is the correctly rounded one except within ~1e-16 of a halfway point.
__device__ __forceinline__ float log1p_f32(float x) { return (float)log1p((double)x); }

// One stored value after the maps: f32(v) / divisor (IEEE division), then log1p.
__device__ __forceinline__ float mapped_f32(float v, bool normalize, float divisor, bool do_log1p) {
  if (normalize) v = __fdiv_rn(v, divisor);
  if (do_log1p) v = log1p_f32(v);
  return v;
}
// Rust's `as f32`: round to nearest even.
__device__ __forceinline__ float to_f32(uint32_t v) { return __uint2float_rn(v); }
__device__ __forceinline__ float to_f32(float v) { return v; }

// Counts are mostly small whole numbers and a row's values share one divisor, so a row's
// maps are a table of its first kMapTable counts, one f64 log1p an entry instead of one a
// stored value (a block of 8,192 x 1,900 counts: 264 us with a log1p a value, bound by the
// FP64 pipe). Whether v is in the table (f32 -0 is not: its maps keep the sign).
constexpr uint32_t kMapTable = 64;
__device__ __forceinline__ bool map_tabled(uint32_t v, uint32_t& c) {
  c = v;
  return v < kMapTable;
}
__device__ __forceinline__ bool map_tabled(float v, uint32_t& c) {
  c = (uint32_t)v;
  return v < (float)kMapTable && (float)c == v && __float_as_uint(v) != 0x80000000u;
}

// A whole value's place in an exact sum (false for a value that is not a whole number up to
// 2^24); u32 counts above 2^24 as kyto sums them, rounded to f32 (elementwise.rs:241-257
// rounds a block's values when one of them is not an f32; the others do not change).
__device__ __forceinline__ bool whole_value(uint32_t v, unsigned long long& out) {
  out = v <= (1u << 24) ? v : (unsigned long long)__uint2float_rn(v);
  return true;
}
__device__ __forceinline__ bool whole_value(float v, unsigned long long& out) {
  out = (uint32_t)v;
  return v >= 0.0f && v <= 16777216.0f && (float)(uint32_t)v == v;
}

// Whether the row [s, e) looks like counts, by its first values: if not, the integer sum and the
// table would be for nothing. (For the whole warp.)
__device__ __forceinline__ bool row_of_counts(const uint32_t*, uint64_t, uint64_t) { return true; }
__device__ __forceinline__ bool row_of_counts(const float* values, uint64_t s, uint64_t e) {
  const uint64_t i = s + (threadIdx.x & 31u);
  unsigned long long w;
  return __all_sync(0xFFFFFFFFu, i >= e || whole_value(values[i], w));
}

// The normalize divisor of the row [s, e), by a whole warp (every lane gets it). Whole
// numbers whose sum stays below 2^53 add up exactly in any order, so the lanes sum integers (a
// row of `counts`: row_of_counts); any other row takes kyto's order (row_divisor: eight chains of
// dependent f64 additions).
template <class V>
__device__ __forceinline__ float warp_row_divisor(const V* values, uint64_t s, uint64_t e,
                                                  float target32, bool counts) {
  if (!counts) return row_divisor(values, s, e, target32, true);
  const unsigned lane = threadIdx.x & 31u;
  unsigned long long sum = 0;
  bool whole = true;
  auto add = [&](V v) {
    unsigned long long w;
    whole &= whole_value(v, w);
    sum += w;
  };
  uint64_t i = s + lane;
  for (; i + 96 < e; i += 128) {
    const V a = values[i], b = values[i + 32], c = values[i + 64], d = values[i + 96];
    add(a), add(b), add(c), add(d);
  }
  for (; i < e; i += 32) add(values[i]);
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
  if (!__all_sync(0xFFFFFFFFu, whole) || sum >= (1ull << 53))
    return row_divisor(values, s, e, target32, true);
  const float divisor = __fdiv_rn((float)(double)sum, target32);
  return divisor == 0.0f ? 1.0f : divisor;
}

// A row's maps by a warp: fill() makes the table (kMapTable floats of the warp's own) for a row of
// counts (row_of_counts) of more values than the table has, at() maps a value. (A lane makes two of
// the table's entries: a shorter row's lanes have two values at most.)
struct RowMap {
  float* table;
  float divisor;
  bool normalize, do_log1p;
  __device__ __forceinline__ static bool tabled(uint64_t n, bool counts) {
    return counts && n > kMapTable;
  }
  __device__ __forceinline__ void fill(uint64_t n, bool counts) {
    if (!tabled(n, counts)) {
      table = nullptr;
      return;
    }
    __syncwarp();
    for (uint32_t c = threadIdx.x & 31u; c < kMapTable; c += 32)
      table[c] = mapped_f32((float)c, normalize, divisor, do_log1p);
    __syncwarp();
  }
  template <class V>
  __device__ __forceinline__ float at(V v) const {
    uint32_t c;
    return table && map_tabled(v, c) ? table[c] : mapped_f32(to_f32(v), normalize, divisor, do_log1p);
  }
};

}  // namespace kg
