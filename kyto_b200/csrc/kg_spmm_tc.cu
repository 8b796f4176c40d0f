// The PCA's sparse x dense products on the 5th-generation tensor cores.
//
//   C (rows x 64) = S (rows x K, sparse) . D (K x 64)
//
// S is the held input X (rows = cells, K = genes) for X Q and the embedding pass, or X^T
// (rows = genes, K = cells) for X^T W, the sketch and the gene statistics; both are kept
// in the pair-entry layout of kg_spmm_tc.cuh (128 rows x 32 columns a block: a header of
// (mask, base) words per row quarter and column pair, then one 8-byte entry per row and
// pair holding the fp16 hi/lo parts of both columns' scaled values). D comes as D^T in the
// same two fp16 parts (the dense layout of kg_spmm_tc.cuh). Each 128 x 32 block of S is
// expanded straight into tensor memory as a 128 x 32 hi tile and a lo tile (a lane per
// row; a lane without an entry for a pair writes the absent value, so the loads have no
// branches), and multiplied by three kind::f16 MMAs per 16 K that read A from TMEM and
// D^T from shared memory (hi.hi + hi.lo + lo.hi: both operands to about 2^-22, as three
// tf32 products give, at twice their rate), accumulated in TMEM over at most
// kFlushChunks chunks and then added into f64 registers (no f32 sum runs over more than
// 512 terms); the scales come off in f64 at the end (powers of two, exact).
//
// Per CTA (persistent, 576 threads) and per K-chunk of a work item (tile, K segment):
//   warp 16     loads: the chunk's D^T tile (64 x (32 hi + 32 lo) fp16, one TMA box) and
//               the block (one bulk copy) into one of kLoadStages stages;
//   warps 0-7   expand: the 128 x 32 block in row quarters and column pairs, from the
//               block's header words and entries into TMEM lanes of one of kABufs A
//               buffers (16 hi and 16 lo words a row, two fp16 a word);
//   warp 17     MMA: 6 tcgen05.mma (kind::f16, A from TMEM, M=128 N=64 K=16) into one of
//               two TMEM accumulators;
//   warps 8-15  drain: TMEM -> f64 registers per flush group, 32 columns a warp; at the
//               end of the item the rows (C - offsets, as the next product's D^T, f32 rows
//               and column sums) or the segment's f64 partial.
// HBM sees each block once per product (512 header bytes and 8 bytes an entry) and D^T
// about once per pass over it (L2 serves the other tiles of a segment).
#include <cuda_fp16.h>
#include <cudaTypedefs.h>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstring>

#include "kg_internal.cuh"
#include "kg_sm100.cuh"
#include "kg_spmm_tc.cuh"
#include "kg_tma.cuh"

namespace kg {

using namespace sm100;

int part_scale(double bound) {
  if (!(bound > 0.0) || !std::isfinite(bound)) return 0;
  int e = 0;
  std::frexp(bound, &e);  // bound in [2^(e-1), 2^e)
  return 15 - e;
}

namespace {

constexpr int kRows = 128;              // rows per tile (M)
constexpr int kChunk = 32;              // K per chunk (a block's columns)
constexpr int kN = 64;                  // output columns (N)
constexpr int kLoadStages = 8;
constexpr int kFlushChunks = 16;        // K-chunks summed in f32 before the f64 flush
constexpr uint32_t kBBytes = kN * 128;  // 8 KB: 64 rows x (32 hi + 32 lo) fp16
constexpr uint32_t kHeaderBytes = 64 * 8;  // (mask, base) per row quarter and column pair
constexpr uint32_t kBlockMaxBytes = kHeaderBytes + kRows * (kChunk / 2) * 8;
constexpr uint32_t kAbsentHi = 0x8000u;  // fp16 -0: the high part of a column without a value
// Two expand warps per sub-partition (rows 32 q.. of a block, half of its column pairs
// each) and two drain warps (rows 32 q.., half of the 64 output columns each).
constexpr int kExpandWarps = 8;
constexpr int kDrainWarps = 8;
constexpr int kSpThreads = (kExpandWarps + kDrainWarps + 2) * 32;
constexpr int kABufs = 4;
// TMEM columns: two 64-column f32 accumulators (0..127), then kABufs A buffers of 32
// columns (16 words of hi parts, then 16 of lo parts; lane = row of the tile).
constexpr uint32_t kTmemColsS = 256;
constexpr uint32_t kAccCols = 64, kABase = 128, kACols = 32;
static_assert(kABase + kABufs * kACols <= kTmemColsS, "TMEM columns");

struct LoadStage {
  uint8_t b[kBBytes];
  uint8_t blk[(kBlockMaxBytes + 1023) / 1024 * 1024];  // header, then the entries
};
// The expansion may read one entry past a full block's last.
static_assert(sizeof(LoadStage::blk) >= kBlockMaxBytes + 8, "stage room past the entries");
// Swizzled tiles (TMA destinations, MMA operands) start on 1024-byte boundaries.
static_assert(sizeof(LoadStage) % 1024 == 0, "load stage size");

struct SpSmem {
  LoadStage st[kLoadStages];
  double colsum[2][4][kN];  // per item parity, per 32-row quarter of the tile
  uint64_t ld_full[kLoadStages], ld_empty[kLoadStages];
  uint64_t a_full[kABufs], a_empty[kABufs];
  uint64_t cs_ready;
  uint64_t acc_full[2], acc_empty[2];
  uint64_t drained;
  uint32_t present[kLoadStages];
  uint32_t tmem_base;
  int abort;
};
constexpr size_t kSpSmemBytes = sizeof(SpSmem) + 1024;
static_assert(kSpSmemBytes <= 227 * 1024, "SpMM shared memory");
static_assert(offsetof(SpSmem, st) % 1024 == 0, "tile alignment");

// A 1D bulk copy global -> shared, counted in bytes on `bar` (16-byte aligned, size a
// multiple of 16).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes,
                                          uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
          "r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}


// The two fp16 parts of x (hi = fp16(x), lo = fp16(x - hi)) in one word, hi low.
__device__ __forceinline__ uint32_t split_pair(float x) {
  const __half hi = __float2half_rn(x);
  const __half lo = __float2half_rn(x - __half2float(hi));
  return (uint32_t)__half_as_ushort(hi) | ((uint32_t)__half_as_ushort(lo) << 16);
}

struct ValueMap;
__device__ __forceinline__ uint2 map_entry(uint2 e, const ValueMap& vm, float mean_r);

struct Geometry {
  uint32_t n_tiles, n_chunks, seg_chunks, n_segs;
  __device__ __forceinline__ uint64_t items() const { return (uint64_t)n_tiles * n_segs; }
  // Consecutive items share a K segment (its D^T tiles stay in L2 for the next tile).
  __device__ __forceinline__ void item(uint64_t w, uint32_t& tile, uint32_t& seg) const {
    tile = (uint32_t)(w % n_tiles);
    seg = (uint32_t)(w / n_tiles);
  }
  __device__ __forceinline__ uint32_t chunks(uint32_t seg) const {
    uint32_t c0 = seg * seg_chunks;
    return min(seg_chunks, n_chunks - c0);
  }
  __device__ __forceinline__ uint64_t first_block(uint32_t tile, uint32_t seg) const {
    return (uint64_t)tile * n_chunks + (uint64_t)seg * seg_chunks;
  }
};

// How the expansion maps each stored value: the mode, and for centred squares the factor
// that undoes S's scale and the one that scales the squares.
struct ValueMap {
  int mode;
  float unscale, sq_scale;
};

// An entry's two columns mapped by the value mode: kValueOne gives 1 where a column holds
// a value, kValueCentredSquare (v - mean_r)^2 scaled; a column without a value gives 0. Both
// columns together, by packed conversions and without branches: the expanding warps bound the
// product of centred squares (a column at a time: 6.2 ms for 1M x 2,000 with 570M values, the
// plain product 2.4).
__device__ __forceinline__ uint2 map_entry(uint2 e, const ValueMap& vm, float mean_r) {
  const bool h0 = (e.x & 0xFFFFu) != kAbsentHi, h1 = (e.x >> 16) != kAbsentHi;
  const uint32_t held = (h0 ? 0xFFFFu : 0u) | (h1 ? 0xFFFF0000u : 0u);
  if (vm.mode == kValueOne) return make_uint2(0x3C003C00u & held, 0u);  // fp16 1.0, low part 0
  const float2 hi = __half22float2(*reinterpret_cast<const __half2*>(&e.x));
  const float2 lo = __half22float2(*reinterpret_cast<const __half2*>(&e.y));
  const float d0 = (hi.x + lo.x) * vm.unscale - mean_r, d1 = (hi.y + lo.y) * vm.unscale - mean_r;
  const float s0 = d0 * d0 * vm.sq_scale, s1 = d1 * d1 * vm.sq_scale;
  // split_pair of both.
  const __half2 sh = __floats2half2_rn(s0, s1);
  const float2 back = __half22float2(sh);
  const __half2 sl = __floats2half2_rn(s0 - back.x, s1 - back.y);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&sh) & held,
                    *reinterpret_cast<const uint32_t*>(&sl) & held);
}

// C's value `c` at (row, column j): less the column's offset into the outputs that are wanted
// (fp16 parts of the next product's D^T, f32 rows); the value as the next product sees it.
__device__ __forceinline__ double row_output(const SpmmOut& out, uint64_t row, bool live, int j,
                                             double c, double t_mul, double t_inv) {
  const double cval = live && j < (int)out.width ? c - out.offsets[j] : 0.0;
  double seen = cval;
  if (out.t) {
    const double y = cval * t_mul;
    const __half hi = __double2half(y);
    const __half lo = __double2half(y - (double)__half2float(hi));
    seen = ((double)__half2float(hi) + (double)__half2float(lo)) * t_inv;
    if (live) {
      uint16_t* t = out.t + (row / 32) * 64 + (row % 32) + (uint64_t)j * out.ld_t;
      t[0] = __half_as_ushort(hi);
      t[32] = __half_as_ushort(lo);
    }
  }
  if (live && out.rows_f32 && j < (int)out.width)
    out.rows_f32[row * (uint64_t)out.width + j] = (float)cval;
  return seen;
}

// One CTA per SM, 18 warps: the register file is split over the SM's four sub-partitions
// (five warps on two of them), so 96 registers a thread; each drain warp keeps 32 f64
// sums, and two expand warps per sub-partition hide each other's latency.
__global__ void __launch_bounds__(kSpThreads, 1)
spmm_tc_kernel(const __grid_constant__ CUtensorMap tmap_dt, const uint64_t* __restrict__ off,
               const uint8_t* __restrict__ data, uint64_t rows, Geometry geo, ValueMap vmap,
               const double* __restrict__ row_means, double out_scale, SpmmOut out,
               int* error) {
  extern __shared__ uint8_t smem_raw[];
  // Aligned to 1024 bytes by an offset into the __shared__ array itself, so the compiler
  // keeps every access in the shared state space (no generic loads and stores).
  SpSmem& sm = *reinterpret_cast<SpSmem*>(smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u));
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint64_t n_items = geo.items();
  volatile int* abort = &sm.abort;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kLoadStages; ++s) {
      mbar_init(&sm.ld_full[s], 1);
      mbar_init(&sm.ld_empty[s], kExpandWarps + 1);  // the expanders and the MMA commit
    }
    for (int b = 0; b < kABufs; ++b) {
      mbar_init(&sm.a_full[b], kExpandWarps);
      mbar_init(&sm.a_empty[b], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sm.acc_full[b], 1);
      mbar_init(&sm.acc_empty[b], kDrainWarps);
    }
    mbar_init(&sm.cs_ready, kDrainWarps);
    mbar_init(&sm.drained, 1);
    sm.abort = 0;
    fence_mbar_init();
  }
  if (warp == 0) tmem_alloc(&sm.tmem_base, kTmemColsS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sm.tmem_base;

  if (warp < kExpandWarps) {
    // ----------------------------------------------------------- expand -------------
    const uint32_t q = (uint32_t)warp & 3u;   // rows 32 q .. 32 q + 31 of each block
    const int hh = warp >> 2;                 // column pairs 8 hh .. 8 hh + 7
    const uint32_t lt = (1u << lane) - 1u;    // the lanes (rows) before this one
    const uint32_t lb = 1u << lane;
    uint64_t it = 0;
    bool ok = true;
    for (uint64_t w = blockIdx.x; w < n_items && ok; w += gridDim.x) {
      uint32_t tile, seg;
      geo.item(w, tile, seg);
      const uint32_t nc = geo.chunks(seg);
      float mean_r = 0.0f;
      if (vmap.mode == kValueCentredSquare) {
        const uint64_t row = (uint64_t)tile * kRows + q * 32u + lane;
        mean_r = row < rows ? (float)row_means[row] : 0.0f;
      }
      for (uint32_t c = 0; c < nc; ++c, ++it) {
        const int ls = (int)(it % kLoadStages);
        const uint32_t lph = (uint32_t)((it / kLoadStages) & 1);
        const uint32_t ab = (uint32_t)(it % kABufs), aph = (uint32_t)((it / kABufs) & 1);
        if (!mbar_wait(&sm.ld_full[ls], lph, abort) || !mbar_wait(&sm.a_empty[ab], aph ^ 1, abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const LoadStage& st = sm.st[ls];
        // This quarter's 16 (mask, base) words, two pairs a 16-byte load, and the entries.
        const uint4* hdr = reinterpret_cast<const uint4*>(st.blk) + q * 8;
        const uint2* ent = reinterpret_cast<const uint2*>(st.blk + kHeaderBytes);
        const bool present = sm.present[ls] != 0;
        // Row (32 q + lane) of the A tiles: pair p's high-part word to column p, its
        // low-part word to column 16 + p (a row without an entry for the pair: zeros).
        const uint32_t arow = tmem + ((q * 32u) << 16) + kABase + ab * kACols;
        {
          uint32_t hw[8], lw[8];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            // Every lane loads (no divergence): a lane without an entry reads the next
            // lane's, or one past the block's last entry (inside the stage buffer), and
            // drops it.
            const uint4 m = present ? hdr[4 * hh + i] : make_uint4(0u, 0u, 0u, 0u);
            uint2 e0 = ent[m.y + __popc(m.x & lt)];
            uint2 e1 = ent[m.w + __popc(m.z & lt)];
            if (vmap.mode != kValuePlain) {
              e0 = map_entry(e0, vmap, mean_r);
              e1 = map_entry(e1, vmap, mean_r);
            }
            const bool h0 = (m.x & lb) != 0, h1 = (m.z & lb) != 0;
            hw[2 * i] = h0 ? e0.x : 0u;
            lw[2 * i] = h0 ? e0.y : 0u;
            hw[2 * i + 1] = h1 ? e1.x : 0u;
            lw[2 * i + 1] = h1 ? e1.y : 0u;
          }
          tmem_st_8(arow + 8u * hh, hw);
          tmem_st_8(arow + 16u + 8u * hh, lw);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();  // every lane has read the stage
        if (lane == 0) {
          mbar_arrive(&sm.a_full[ab]);
          mbar_arrive(&sm.ld_empty[ls]);
        }
      }
    }
  } else if (warp < kExpandWarps + kDrainWarps) {
    // ----------------------------------------------------------- drain TMEM ---------
    const uint32_t quad = (uint32_t)warp & 3u;  // TMEM lanes 32 quad .. (rows of the tile)
    const uint32_t half = (uint32_t)(warp - kExpandWarps) >> 2;  // columns 32 half ..
    constexpr int kH = kN / 2;
    const uint32_t i = quad * 32u + lane;
    uint64_t fg = 0, item_no = 0;
    bool ok = true;
    for (uint64_t w = blockIdx.x; w < n_items && ok; w += gridDim.x, ++item_no) {
      uint32_t tile, seg;
      geo.item(w, tile, seg);
      const uint64_t row = (uint64_t)tile * kRows + i;
      double acc[kH];
#pragma unroll
      for (int j = 0; j < kH; ++j) acc[j] = 0.0;
      const uint32_t nc = geo.chunks(seg);
      const uint32_t groups = (nc + kFlushChunks - 1) / kFlushChunks;
      for (uint32_t gr = 0; gr < groups; ++gr, ++fg) {
        const uint32_t b = (uint32_t)(fg & 1), bph = (uint32_t)((fg >> 1) & 1);
        if (!mbar_wait(&sm.acc_full[b], bph, abort)) {
          ok = false;
          break;
        }
        tc_fence_after();
        __syncwarp();
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          uint32_t rr[16];
          tmem_ld_16(tmem + ((quad * 32u) << 16) + b * kAccCols + half * kH + hf * 16u, rr);
          tmem_wait_ld();
          if (out.mode == kOutGroups) {
            const uint64_t group = (uint64_t)seg * (geo.seg_chunks / kFlushChunks) + gr;
            uint4* dst = reinterpret_cast<uint4*>(out.groups + (group * rows + row) * kN + half * kH +
                                                  hf * 16);
            if (row < rows) {
#pragma unroll
              for (int j = 0; j < 4; ++j)
                dst[j] = make_uint4(rr[4 * j], rr[4 * j + 1], rr[4 * j + 2], rr[4 * j + 3]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[hf * 16 + j] += (double)__uint_as_float(rr[j]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&sm.acc_empty[b]);
      }
      if (!ok) break;
      if (out.mode == kOutRows) {
        // C = S D - offsets: the next product's D^T (fp16 parts), the f32 rows, and this
        // tile's column sums (fixed tree: warp shuffles, then the 4 quarters in order).
        const bool live = row < rows;
        const double t_mul = ldexp(1.0, out.t_scale), t_inv = ldexp(1.0, -out.t_scale);
#pragma unroll
        for (int jj = 0; jj < kH; ++jj) {
          const int j = (int)half * kH + jj;
          const double seen = row_output(out, row, live, j, acc[jj] * out_scale, t_mul, t_inv);
          if (out.colsum_partial) {
            double sv = seen;
            for (int o = 16; o; o >>= 1) sv += __shfl_xor_sync(0xFFFFFFFFu, sv, o);
            if (lane == 0) sm.colsum[item_no & 1][quad][j] = sv;
          }
        }
        if (out.colsum_partial) {
          // The four quarters' sums in a fixed order (double-buffered by item, so a warp
          // running one item ahead cannot overwrite what the quarter-0 warps still read).
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm.cs_ready);
          if (!mbar_wait(&sm.cs_ready, (uint32_t)(item_no & 1), abort)) break;
          if (quad == 0) {
            const double(*cs)[kN] = sm.colsum[item_no & 1];
            const int j = (int)half * kH + lane;
            const double tsum = ((cs[0][j] + cs[1][j]) + cs[2][j]) + cs[3][j];
            out.colsum_partial[(uint64_t)tile * kN + j] = tsum;
          }
        }
      } else if (out.mode == kOutPartial && row < rows) {
        double* dst = out.partial + ((uint64_t)seg * rows + row) * kN + half * kH;
#pragma unroll
        for (int j = 0; j < kH; ++j) dst[j] = acc[j] * out_scale;
      }
    }
  } else if (warp == kExpandWarps + kDrainWarps) {
    // ----------------------------------------------------------- loads --------------
    // Lane 0 issues; the warp reads the item's block offsets 32 at a time ahead of it.
    // (Prefetching the next 32 blocks into L2 ahead of their copies made the products 9%
    // slower on the 1M benchmark: part of it was evicted before use and read twice.)
    if (lane == 0) prefetch_tmap(&tmap_dt);
    uint64_t it = 0;
    int issued_phase[kLoadStages];
    for (int s = 0; s < kLoadStages; ++s) issued_phase[s] = -1;
    bool ok = true;
    for (uint64_t w = blockIdx.x; w < n_items && ok; w += gridDim.x) {
      uint32_t tile, seg;
      geo.item(w, tile, seg);
      const uint32_t nc = geo.chunks(seg);
      const uint64_t b0 = geo.first_block(tile, seg);
      uint64_t win = 0, win_end = 0;
      for (uint32_t c = 0; c < nc; ++c, ++it) {
        const uint32_t at = c & 31u;
        if (at == 0) {
          // off[b0 + c + lane] and, in lane 0, off[b0 + c + 32] (indices <= nc: the
          // offsets array holds one entry past every block).
          win = c + lane <= nc ? off[b0 + c + lane] : 0;
          win_end = lane == 0 && c + 32 <= nc ? off[b0 + c + 32] : 0;
        }
        const uint64_t e0 = __shfl_sync(0xFFFFFFFFu, win, at);
        const uint64_t e1n = __shfl_sync(0xFFFFFFFFu, win, (at + 1) & 31u);
        const uint64_t e1w = __shfl_sync(0xFFFFFFFFu, win_end, 0);
        const uint64_t e1 = at == 31 ? e1w : e1n;
        if (lane == 0) {
          const int s = (int)(it % kLoadStages);
          const uint32_t ph = (uint32_t)((it / kLoadStages) & 1);
          if (!mbar_wait(&sm.ld_empty[s], ph ^ 1, abort)) {
            ok = false;
          } else {
            const uint32_t chunk = seg * geo.seg_chunks + c;
            const uint32_t bytes = (uint32_t)((e1 - e0) * 16);
            sm.present[s] = bytes ? 1u : 0u;
            mbar_arrive_expect_tx(&sm.ld_full[s], kBBytes + bytes);
            tma_load_2d(sm.st[s].b, &tmap_dt, &sm.ld_full[s], (int32_t)(chunk * 64), 0);
            if (bytes) bulk_load(sm.st[s].blk, data + e0 * 16, bytes, &sm.ld_full[s]);
            issued_phase[s] = (int)ph;
          }
        }
        ok = __shfl_sync(0xFFFFFFFFu, ok, 0);
        if (!ok) break;
      }
    }
    if (lane == 0) {
      for (int s = 0; s < kLoadStages; ++s) {
        if (issued_phase[s] < 0) continue;
        for (uint32_t q = 0; q < kWaitPolls && !mbar_try_wait(&sm.ld_full[s], issued_phase[s]); ++q)
          ;
      }
    }
  } else {
    // ----------------------------------------------------------- MMA ----------------
    if (lane == 0) {
      const uint32_t idesc = idesc_f32acc(0u, kRows, kN);  // f16 x f16 -> f32
      uint64_t it = 0, fg = 0;
      bool ok = true;
      for (uint64_t w = blockIdx.x; w < n_items && ok; w += gridDim.x) {
        uint32_t tile, seg;
        geo.item(w, tile, seg);
        const uint32_t nc = geo.chunks(seg);
        for (uint32_t c = 0; c < nc && ok; ++c, ++it) {
          const uint32_t in_group = c % kFlushChunks;
          const uint32_t b = (uint32_t)(fg & 1), bph = (uint32_t)((fg >> 1) & 1);
          if (in_group == 0 && !mbar_wait(&sm.acc_empty[b], bph ^ 1, abort)) {
            ok = false;
            break;
          }
          const int ls = (int)(it % kLoadStages);
          const uint32_t lph = (uint32_t)((it / kLoadStages) & 1);
          const uint32_t ab = (uint32_t)(it % kABufs), aph = (uint32_t)((it / kABufs) & 1);
          if (!mbar_wait(&sm.ld_full[ls], lph, abort) || !mbar_wait(&sm.a_full[ab], aph, abort)) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t d = tmem + b * kAccCols;
          const uint32_t ah = tmem + kABase + ab * kACols, al = ah + 16u;
          const uint32_t bs = smem_addr(sm.st[ls].b);
#pragma unroll
          for (int kk = 0; kk < kChunk / 16; ++kk) {
            // 16 K: 8 A columns (pairs), 32 bytes of a B row; B's lo parts 64 bytes on.
            const uint32_t o = kk * 32;
            mma_f16_ts(d, ah + kk * 8, desc_k_sw128(bs + o), idesc, (in_group | kk) != 0);
            mma_f16_ts(d, ah + kk * 8, desc_k_sw128(bs + 64 + o), idesc, 1);
            mma_f16_ts(d, al + kk * 8, desc_k_sw128(bs + o), idesc, 1);
          }
          mma_commit(&sm.ld_empty[ls]);
          mma_commit(&sm.a_empty[ab]);
          if (in_group == kFlushChunks - 1 || c == nc - 1) {
            mma_commit(&sm.acc_full[b]);
            ++fg;
          }
        }
      }
      mma_commit(&sm.drained);
      for (uint32_t q = 0; q < kWaitPolls && !mbar_try_wait(&sm.drained, 0); ++q)
        ;
    }
  }
  __syncwarp();
  __syncthreads();
  if (sm.abort && threadIdx.x == 0) atomicExch(error, 1);
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, kTmemColsS);
  }
}

// ------------------------------------------------------------------ builders -------

// Per row: the sum of squared values (f64) into the largest so far, and the largest and
// smallest nonzero |value| (non-negative doubles compare as their bit patterns). Reading the
// values once bounds it: a warp takes row after row, four reads a lane on their way, and only
// its own largest and smallest reach the three totals (three atomics a row: 2.9 ms for 1M rows
// of 570 values, now 0.64).
constexpr int kStatsAhead = 4;

__global__ void __launch_bounds__(256)
csr_stats_kernel(const uint64_t* __restrict__ ptr, const float* __restrict__ val, uint64_t n_rows,
                 unsigned long long* max_sq, unsigned long long* max_abs,
                 unsigned long long* min_abs) {
  const unsigned lane = threadIdx.x & 31u;
  const uint64_t warps = gridDim.x * (uint64_t)(blockDim.x / 32);
  double best_sq = 0.0;
  float hi = 0.0f, lo = INFINITY;
  bool nan = false;
  for (uint64_t r = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5; r < n_rows; r += warps) {
    const uint64_t end = ptr[r + 1];
    double sq = 0.0;
    for (uint64_t i = ptr[r] + lane; i < end; i += 32 * kStatsAhead) {
      float v[kStatsAhead];
#pragma unroll
      for (int k = 0; k < kStatsAhead; ++k) v[k] = i + 32 * k < end ? fabsf(val[i + 32 * k]) : 0.0f;
#pragma unroll
      for (int k = 0; k < kStatsAhead; ++k) {
        const double w = (double)v[k];
        sq += w * w;  // (zeros past the row's end change nothing)
        hi = fmaxf(hi, v[k]);
        if (v[k] > 0.0f) lo = fminf(lo, v[k]);
        nan = nan || v[k] != v[k];
      }
    }
    for (int o = 16; o; o >>= 1) sq += __shfl_xor_sync(0xFFFFFFFFu, sq, o);
    // As the totals compare: by bit pattern (a NaN above everything).
    if (__double_as_longlong(sq) > __double_as_longlong(best_sq)) best_sq = sq;
  }
  for (int o = 16; o; o >>= 1) {
    hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
    lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
  }
  nan = __any_sync(0xFFFFFFFFu, nan);
  if (lane == 0) {
    atomicMax(max_sq, (unsigned long long)__double_as_longlong(best_sq));
    atomicMax(max_abs, nan ? 0x7FF8000000000000ull
                           : (unsigned long long)__double_as_longlong((double)hi));
    atomicMin(min_abs, (unsigned long long)__double_as_longlong((double)lo));
  }
}

// A value's two fp16 parts (hi in bits 0-15, lo in 16-31) of x = v * 2^scale; a stored
// -0 becomes +0 (-0 marks a column without a value).
__device__ __forceinline__ uint32_t stored_parts(float v, int scale) {
  const float x = ldexpf(v, scale);
  return split_pair(x == 0.0f ? 0.0f : x);
}

// An entry from its two columns' parts words (kAbsentHi for a column without a value).
__device__ __forceinline__ uint2 make_entry(uint32_t w0, uint32_t w1) {
  return make_uint2((w0 & 0xFFFFu) | (w1 << 16), (w0 >> 16) | (w1 & 0xFFFF0000u));
}

// The layouts of a CSR matrix (X: rows = CSR rows) and of its transpose (rows = CSR columns) are
// filled from one reading: a CTA takes 32 CSR rows, which are a row quarter of X's tile and one
// chunk of X^T's columns, through a window of columns at a time in shared memory, a warp four
// rows, the lanes over each row's entries. Reading the entries and writing both layouts bounds
// it. (Each layout by itself, a lane writing where its entry goes, every entry a sector:
// masks 3.8 and values 11.0 ms for 1M rows of 570 entries, now 1.8 and 3.8.)
constexpr int kLayWarps = 8;                // a CTA
constexpr int kLayRows = 32 / kLayWarps;    // CSR rows a warp
constexpr uint32_t kMaskCols = 512;         // columns a window of masks_kernel
constexpr uint32_t kValueCols = 256;        // and of values_kernel

// This warp's rows: each row's entries still to come.
struct WalkRows {
  uint64_t at[kLayRows], end[kLayRows];
};

__device__ __forceinline__ WalkRows walk_start(const uint64_t* __restrict__ ptr, uint64_t n_rows) {
  WalkRows w;
#pragma unroll
  for (int k = 0; k < kLayRows; ++k) {
    const uint64_t r = blockIdx.x * 32ull + (threadIdx.x >> 5) * kLayRows + k;
    w.at[k] = r < n_rows ? ptr[r] : 0;
    w.end[k] = r < n_rows ? ptr[r + 1] : 0;
  }
  return w;
}

// Calls f(row, column - c0, value) for the entries of this warp's rows in columns [c0, c0 + Cols)
// that it has not passed yet. The value is 0 without `Values`. With `Checked`, f's columns lie inside
// the window whatever the rows hold, and *jumped becomes not 0 when an entry stands behind one of
// a later run of kValueCols columns: where that is so for no window, each entry is passed once, in
// its own window, in windows of Cols and of kValueCols columns alike (within a run the order does
// not matter: the tiles are filled by column). Rows without a jump need no check of the window's
// lower end (0.5 ms of values_kernel's 3.8 for the check; masks_kernel's checks take 0.4 of 1.8).
template <bool Values, bool Checked, uint32_t Cols, class F>
__device__ __forceinline__ void walk_window(const uint32_t* __restrict__ col,
                                            const float* __restrict__ val, WalkRows& w, uint32_t c0,
                                            uint32_t* jumped, F&& f) {
  static_assert(Cols == kValueCols || Cols == 2 * kValueCols, "a window is one or two runs");
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint64_t(&at)[kLayRows] = w.at;
  const uint64_t(&end)[kLayRows] = w.end;
  uint32_t second = 0;  // bit k: row k is in the window's second run
  for (;;) {
    uint32_t c[kLayRows];
    float v[kLayRows];
#pragma unroll
    for (int k = 0; k < kLayRows; ++k) {
      const uint64_t i = at[k] + lane;
      c[k] = i < end[k] ? col[i] : 0xFFFFFFFFu;
      v[k] = Values && i < end[k] ? val[i] : 0.0f;
    }
    bool more = false;
#pragma unroll
    for (int k = 0; k < kLayRows; ++k) {
      const bool in = Checked ? c[k] - c0 < Cols : c[k] < c0 + Cols;
      if (in) f(warp * kLayRows + k, c[k] - c0, v[k]);
      const uint32_t held = __ballot_sync(0xFFFFFFFFu, in);  // in order: the first n
      const uint32_t n = __popc(held);
      if (Checked) {
        const uint32_t run = __ballot_sync(0xFFFFFFFFu, c[k] - c0 < kValueCols);
        *jumped |= (held & (held + 1u)) | (run & (run + 1u)) | (run & (0u - (second >> k & 1u)));
        second |= (held != run ? 1u : 0u) << k;
      }
      at[k] += n;
      more = more || n == 32;
    }
    if (!more) break;
  }
}

// Whether every entry of this warp's rows was passed: one that comes behind an entry of a later
// window holds its row up before its end.
__device__ __forceinline__ bool walk_ended(const WalkRows& w) {
  bool all = true;
#pragma unroll
  for (int k = 0; k < kLayRows; ++k) all = all && w.at[k] == w.end[k];
  return all;
}

// Header masks of X (masks, words of 64 a block) and, if masks_t, of X^T: a byte an entry in
// shared memory, gathered into words by ballots. Every word of both layouts is written. `groups`:
// groups of 32 columns to pass, at least X's chunks and four times X^T's tiles. With X^T each
// column's entries are counted too (counts, if given: whole numbers, so any order; a column twice
// in a row counts once). *unsorted is set when a row's entries do not come run by run of kValueCols
// columns, and without `counts` when a row holds a column twice: the masks are then of no use.
__global__ void __launch_bounds__(kLayWarps * 32, 5)
masks_kernel(const uint64_t* __restrict__ ptr, const uint32_t* __restrict__ col, uint64_t n_rows,
             uint32_t n_chunks, uint32_t n_tiles_t, uint32_t n_chunks_t, uint32_t groups,
             uint32_t* masks, uint32_t* masks_t, unsigned long long* counts,
             unsigned long long* unsorted) {
  constexpr uint32_t kLd = kMaskCols / 4 + 1;  // words a row: an odd stride
  __shared__ uint32_t flags[32][kLd];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t rb = blockIdx.x, tile = rb / 4, q = rb % 4;
  WalkRows rows = walk_start(ptr, n_rows);
  uint32_t held_x = 0, jumped = 0;
  for (uint32_t g0 = 0; g0 < groups; g0 += kMaskCols / 32) {
    for (uint32_t i = threadIdx.x; i < 32 * kLd; i += kLayWarps * 32) (&flags[0][0])[i] = 0;
    __syncthreads();
    const uint32_t c0 = g0 * 32;
    walk_window<false, true, kMaskCols>(col, nullptr, rows, c0, &jumped,
                                        [&](uint32_t row, uint32_t c, float) {
                                          reinterpret_cast<unsigned char*>(flags[row])[c] = 1;
                                        });
    __syncthreads();
    for (uint32_t g = warp; g < kMaskCols / 32 && g0 + g < groups; g += kLayWarps) {
      if (g0 + g < n_chunks) {  // lane = row
        uint32_t mine = 0;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
          const uint32_t w = flags[lane][g * 8 + k];
          const uint32_t even = __ballot_sync(0xFFFFFFFFu, w & 0xFFFFu);
          const uint32_t odd = __ballot_sync(0xFFFFFFFFu, w >> 16);
          if (lane == 2 * k) mine = even;
          if (lane == 2 * k + 1) mine = odd;
          if (!counts) held_x += __popc(w);  // (a byte an entry, 0 or 1)
        }
        if (lane < 16) masks[(tile * n_chunks + g0 + g) * 64 + q * 16 + lane] = mine;
      }
      if (masks_t && g0 + g < 4 * n_tiles_t && rb < n_chunks_t) {  // lane = column
        uint32_t mine = 0, held = 0;
#pragma unroll
        for (uint32_t p = 0; p < 16; ++p) {
          const uint32_t w =
              (uint32_t)reinterpret_cast<const unsigned char*>(flags[2 * p])[g * 32 + lane] +
              reinterpret_cast<const unsigned char*>(flags[2 * p + 1])[g * 32 + lane];
          const uint32_t any = __ballot_sync(0xFFFFFFFFu, w);
          if (lane == p) mine = any;
          held += w;
        }
        if (counts && held) atomicAdd(&counts[(g0 + g) * 32 + lane], (unsigned long long)held);
        if (lane < 16)
          masks_t[((uint64_t)((g0 + g) / 4) * n_chunks_t + rb) * 64 + (g0 + g) % 4 * 16 + lane] = mine;
      }
    }
    __syncthreads();
  }
  if (jumped || !walk_ended(rows)) *unsorted = 1;
  if (!counts) {
    __shared__ uint32_t held_all;
    if (threadIdx.x == 0) held_all = 0;
    __syncthreads();
    atomicAdd(&held_all, held_x);
    __syncthreads();
    const uint64_t first = min(rb * 32, n_rows), past = min(rb * 32 + 32, n_rows);
    if (threadIdx.x == 0 && held_all != ptr[past] - ptr[first]) *unsorted = 1;
  }
}

// A layout as values_kernel writes it.
struct LayoutOut {
  const uint32_t* masks;  // null: not wanted
  const uint16_t* bases;
  const uint64_t* off;
  uint8_t* data;
  uint32_t n_chunks;
};

// Quarter q of block b: its header words and entries, pair p's parts words as parts(p, 0) and
// parts(p, 1) in lane = row.
template <class P>
__device__ __forceinline__ void write_quarter(const LayoutOut& o, uint64_t b, uint32_t q, P&& parts) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t start = o.off[b];
  if (o.off[b + 1] == start) return;
  uint8_t* block = o.data + start * 16;
  uint32_t mask = 0, base = 0;
  if (lane < 16) {
    mask = o.masks[b * 64 + q * 16 + lane];
    base = o.bases[b * 64 + q * 16 + lane];
    reinterpret_cast<uint2*>(block)[q * 16 + lane] = make_uint2(mask, base);
  }
  uint2* entries = reinterpret_cast<uint2*>(block + kHeaderBytes);
#pragma unroll 4
  for (uint32_t p = 0; p < 16; ++p) {
    const uint32_t m = __shfl_sync(0xFFFFFFFFu, mask, p), first = __shfl_sync(0xFFFFFFFFu, base, p);
    const uint2 e = make_entry(parts(p, 0), parts(p, 1));
    if ((m >> lane) & 1u) entries[first + __popc(m & ((1u << lane) - 1u))] = e;
  }
}

// Headers and entries of X and, if wanted, of X^T, of rows that masks_kernel has passed. `groups` as
// there.
__global__ void __launch_bounds__(kLayWarps * 32)
values_kernel(const uint64_t* __restrict__ ptr, const uint32_t* __restrict__ col,
              const float* __restrict__ val, uint64_t n_rows, uint32_t n_tiles_t, uint32_t groups,
              int scale, LayoutOut x, LayoutOut t) {
  __shared__ uint32_t tile[32][kValueCols + 1];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t rb = blockIdx.x;
  WalkRows rows = walk_start(ptr, n_rows);
  for (uint32_t g0 = 0; g0 < groups; g0 += kValueCols / 32) {
    for (uint32_t i = threadIdx.x; i < 32 * (kValueCols + 1); i += kLayWarps * 32)
      (&tile[0][0])[i] = kAbsentHi;
    __syncthreads();
    walk_window<true, false, kValueCols>(
        col, val, rows, g0 * 32, nullptr,
        [&](uint32_t row, uint32_t c, float v) { tile[row][c] = stored_parts(v, scale); });
    __syncthreads();
    for (uint32_t g = warp; g < kValueCols / 32 && g0 + g < groups; g += kLayWarps) {
      if (g0 + g < x.n_chunks)
        write_quarter(x, rb / 4 * x.n_chunks + g0 + g, rb % 4, [&](uint32_t p, uint32_t odd) {
          return tile[lane][g * 32 + 2 * p + odd];
        });
      if (t.masks && g0 + g < 4 * n_tiles_t && rb < t.n_chunks)
        write_quarter(t, (uint64_t)((g0 + g) / 4) * t.n_chunks + rb, (g0 + g) % 4,
                      [&](uint32_t p, uint32_t odd) { return tile[2 * p + odd][g * 32 + lane]; });
    }
    __syncthreads();
  }
}

// Per block (warp): each header word's base (the entries of the words before it) and the
// block's size in 16-byte units (0 for a block without entries).
__global__ void pair_base_kernel(const uint32_t* masks, uint64_t n_blocks, uint16_t* bases,
                                 uint64_t* units) {
  const uint64_t b = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  if (b > n_blocks) return;
  if (b == n_blocks) {
    if (lane == 0) units[b] = 0;
    return;
  }
  const uint32_t c0 = __popc(masks[b * 64 + 2 * lane]), c1 = __popc(masks[b * 64 + 2 * lane + 1]);
  uint32_t incl = c0 + c1;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if ((int)lane >= o) incl += t;
  }
  const uint32_t excl = incl - c0 - c1;
  bases[b * 64 + 2 * lane] = (uint16_t)excl;
  bases[b * 64 + 2 * lane + 1] = (uint16_t)(excl + c0);
  const uint32_t total = __shfl_sync(0xFFFFFFFFu, incl, 31);
  if (lane == 0) units[b] = total ? (kHeaderBytes + 8ull * total + 15) / 16 : 0;
}

// A layout on its way: its masks, then its bases and offsets.
struct Building {
  Blocked* out = nullptr;
  DeviceBuffer<uint32_t> masks;
  DeviceBuffer<uint16_t> bases;
  DeviceBuffer<unsigned char> scratch;
  uint64_t units = 0;
  uint64_t blocks() const { return (uint64_t)out->n_tiles * out->n_chunks; }
  void start(Blocked& b, uint64_t rows, uint64_t K, cudaStream_t s) {
    out = &b;
    b.rows = rows;
    b.K = K;
    b.n_tiles = (uint32_t)((rows + kRows - 1) / kRows);
    b.n_chunks = (uint32_t)((K + kChunk - 1) / kChunk);
    masks.alloc(blocks() * 64, s);
  }
  // (`units` is read back on the stream.)
  void offsets(cudaStream_t s) {
    const uint64_t nb = blocks();
    bases.alloc(nb * 64, s);
    out->off.alloc(nb + 1, s);
    pair_base_kernel<<<blocks_for((nb + 1) * 32, 256), 256, 0, s>>>(masks.ptr, nb, bases.ptr,
                                                                    out->off.ptr);
    KG_LAUNCH_CHECK();
    size_t temp = 0;
    KG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, temp, out->off.ptr, out->off.ptr, nb + 1, s));
    scratch.alloc(temp, s);
    KG_CUDA(cub::DeviceScan::ExclusiveSum(scratch.ptr, temp, out->off.ptr, out->off.ptr, nb + 1, s));
    KG_CUDA(cudaMemcpyAsync(&units, out->off.ptr + nb, 8, cudaMemcpyDeviceToHost, s));
  }
  LayoutOut layout(cudaStream_t s) {
    out->bytes = units * 16;
    out->data.alloc(std::max<uint64_t>(out->bytes, 16), s);
    return {masks.ptr, bases.ptr, out->off.ptr, out->data.ptr, out->n_chunks};
  }
};

}  // namespace

bool build_blocked(const uint64_t* ptr, const uint32_t* col, const float* val, uint64_t n_rows,
                   uint64_t n_cols, uint64_t nnz, Blocked& out, Blocked* twin,
                   unsigned long long* col_counts, cudaStream_t s) {
  if (col_counts) KG_CUDA(cudaMemsetAsync(col_counts, 0, n_cols * sizeof *col_counts, s));
  // The values' range (the scale of their fp16 parts) and the largest row norm.
  // And the masks' verdict on the rows' order.
  DeviceBuffer<unsigned long long> st(4, s);
  const unsigned long long init[4] = {0ull, 0ull, 0x7FF0000000000000ull, 0ull};  // 0, 0, +inf, 0
  KG_CUDA(cudaMemcpyAsync(st.ptr, init, sizeof init, cudaMemcpyHostToDevice, s));
  if (nnz) {
    csr_stats_kernel<<<std::min<unsigned>(blocks_for(n_rows * 32, 256), 2048), 256, 0, s>>>(
        ptr, val, n_rows, st.ptr, st.ptr + 1, st.ptr + 2);
    KG_LAUNCH_CHECK();
  }
  Building x, t;
  x.start(out, n_rows, n_cols, s);
  if (twin) t.start(*twin, n_cols, n_rows, s);
  const uint32_t tiles_t = twin ? twin->n_tiles : 0, chunks_t = twin ? twin->n_chunks : 0;
  const uint32_t groups = std::max(out.n_chunks, 4 * tiles_t);
  const unsigned grid = out.n_tiles * 4;
  if (grid) {
    masks_kernel<<<grid, kLayWarps * 32, 0, s>>>(ptr, col, n_rows, out.n_chunks, tiles_t, chunks_t,
                                                 groups, x.masks.ptr, t.masks.ptr, col_counts,
                                                 st.ptr + 3);
    KG_LAUNCH_CHECK();
  }
  x.offsets(s);
  if (twin) t.offsets(s);
  unsigned long long h_st[4];
  KG_CUDA(cudaMemcpyAsync(h_st, st.ptr, sizeof h_st, cudaMemcpyDeviceToHost, s));
  KG_CUDA(cudaStreamSynchronize(s));
  if (h_st[3]) return false;
  double d[3];
  std::memcpy(d, h_st, sizeof d);
  out.max_row_norm = std::sqrt(d[0]);
  out.max_abs = d[1];
  out.min_abs = std::isinf(d[2]) ? 0.0 : d[2];
  out.scale = part_scale(out.max_abs);
  if (twin) {
    twin->scale = out.scale;
    twin->max_abs = out.max_abs;
    twin->min_abs = out.min_abs;
    twin->max_row_norm = 0.0;  // not tracked for the transpose
  }
  const LayoutOut xo = x.layout(s);
  const LayoutOut to = twin ? t.layout(s) : LayoutOut{nullptr, nullptr, nullptr, nullptr, 0};
  if (!x.units) return true;
  values_kernel<<<grid, kLayWarps * 32, 0, s>>>(ptr, col, val, n_rows, tiles_t, groups, out.scale, xo,
                                                to);
  KG_LAUNCH_CHECK();
  return true;
}

namespace {

// partial[seg][row][j] = the segment's groups (per groups of the product's f32 sums) added in
// f64 in order, times the scale: what the product itself writes for a whole segment.
__global__ void __launch_bounds__(256)
sum_groups_kernel(const float* __restrict__ groups, uint32_t n_groups, uint32_t per, uint64_t rows,
                  double out_scale, double* partial) {
  const uint64_t at = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, plane = rows * kN;
  if (at >= plane) return;
  const uint32_t g0 = blockIdx.y * per, g1 = min(g0 + per, n_groups);
  double acc = 0.0;
#pragma unroll 8
  for (uint32_t g = g0; g < g1; ++g) acc += (double)groups[g * plane + at];
  partial[blockIdx.y * plane + at] = acc * out_scale;
}

// kOutRows from the groups of the product's f32 sums: each value's groups added in f64 in order,
// then the product's own epilogue (column sums: lanes, then the tile's quarters in order). A CTA a
// tile, a warp 32 rows and 16 columns, a lane a row.
__global__ void __launch_bounds__(512)
rows_of_groups_kernel(const float* __restrict__ groups, uint32_t n_groups, uint64_t rows,
                      double out_scale, SpmmOut out) {
  __shared__ double colsum[4][kN];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t quad = warp & 3u, j0 = (warp >> 2) * 16;
  const uint64_t row = blockIdx.x * (uint64_t)kRows + quad * 32 + lane;
  const bool live = row < rows;
  double acc[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) acc[j] = 0.0;
  for (uint32_t g = 0; g < n_groups && live; ++g) {
    const float4* from = reinterpret_cast<const float4*>(groups + (g * rows + row) * kN + j0);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float4 v = from[k];
      acc[4 * k] += (double)v.x;
      acc[4 * k + 1] += (double)v.y;
      acc[4 * k + 2] += (double)v.z;
      acc[4 * k + 3] += (double)v.w;
    }
  }
  const double t_mul = ldexp(1.0, out.t_scale), t_inv = ldexp(1.0, -out.t_scale);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    double sv = row_output(out, row, live, (int)j0 + j, acc[j] * out_scale, t_mul, t_inv);
    if (out.colsum_partial) {
      for (int o = 16; o; o >>= 1) sv += __shfl_xor_sync(0xFFFFFFFFu, sv, o);
      if (lane == 0) colsum[quad][j0 + j] = sv;
    }
  }
  if (!out.colsum_partial) return;
  __syncthreads();
  if (threadIdx.x < kN) {
    const uint32_t j = threadIdx.x;
    out.colsum_partial[blockIdx.x * (uint64_t)kN + j] =
        ((colsum[0][j] + colsum[1][j]) + colsum[2][j]) + colsum[3][j];
  }
}

// Whether `items` whole segments leave too much of the chip idle: up to three rounds of one item
// an SM with a fifth or more of them empty. X^T of 50,000 cells x 2,000 genes has 64 segments: 340
// us whole, 158 and 11 us for the sums in groups; X of 2,700 cells has 22 tiles: 57 us, 20 and 12.
// (Where the last of many rounds is the ragged one, the groups, 256 bytes a row and 512 columns,
// cost more than it does.)
bool split_groups(uint64_t items, int sm_count) {
  const uint64_t rounds = (items + sm_count - 1) / sm_count;
  return rounds <= 3 && items * 5 < rounds * sm_count * 4;
}

}  // namespace

void spmm_tc(const SpmmArgs& a, cudaStream_t s) {
  const Blocked& b = *a.s;
  if (b.K == 0 || b.rows == 0) return;
  allow_dynamic_smem(spmm_tc_kernel, kSpSmemBytes);
  if (a.ld_t != dense_ld(b.K)) fail(KG_ERR_INVALID, "spmm: D^T row length must be dense_ld(K)");
  if (a.out.mode == kOutRows && a.out.t && a.out.ld_t != dense_ld(b.rows))
    fail(KG_ERR_INVALID, "spmm: the output D^T row length must be dense_ld(rows)");
  if (!a.error) fail(KG_ERR_INVALID, "spmm: no error flag");
  Geometry geo;
  geo.n_tiles = b.n_tiles;
  geo.n_chunks = b.n_chunks;
  geo.seg_chunks = (uint32_t)std::min<uint64_t>(a.seg_chunks ? a.seg_chunks : b.n_chunks, b.n_chunks);
  geo.n_segs = (geo.n_chunks + geo.seg_chunks - 1) / geo.seg_chunks;
  if (a.out.mode == kOutRows && geo.n_segs != 1)
    fail(KG_ERR_INVALID, "spmm: row output needs one K segment");
  // A chip that one segment a tile leaves idle: shorter work items whose f32 groups are added
  // afterwards in the segments' order. (Whole segments give the same bits, and take no memory.)
  const uint64_t seg_chunks = geo.seg_chunks;
  SpmmOut to = a.out;
  DeviceBuffer<float> groups;
  const uint32_t n_groups = (geo.n_chunks + kFlushChunks - 1) / kFlushChunks;
  auto room = [&] {
    try {
      groups.alloc((uint64_t)n_groups * b.rows * kN, s);
      return true;
    } catch (const Error& e) {
      if (e.status != KG_ERR_OOM) throw;
      return false;
    }
  };
  if (n_groups > geo.n_segs && (seg_chunks % kFlushChunks == 0 || geo.n_segs == 1) &&
      split_groups((uint64_t)geo.n_tiles * geo.n_segs, a.sm_count) && room()) {
    uint32_t part = kFlushChunks;
    while (part * 2 < seg_chunks &&
           (uint64_t)geo.n_tiles * (geo.n_chunks / (part * 2)) >= 4ull * a.sm_count)
      part *= 2;
    geo.seg_chunks = part;
    geo.n_segs = (geo.n_chunks + part - 1) / part;
    to.mode = kOutGroups;
    to.groups = groups.ptr;
  }
  // S's stored values enter the MMA times 2^a_scale (the stored scale, 0 for the ones,
  // a square's own scale for the centred squares), D^T times 2^dt_scale.
  ValueMap vm;
  vm.mode = a.value_mode;
  vm.unscale = ldexpf(1.0f, -b.scale);
  int a_scale = b.scale;
  vm.sq_scale = 1.0f;
  if (a.value_mode == kValueOne) {
    a_scale = 0;
  } else if (a.value_mode == kValueCentredSquare) {
    // (v - mean)^2 <= (|v| + |mean|)^2 <= (2 max|v|)^2.
    a_scale = part_scale(4.0 * b.max_abs * b.max_abs);
    vm.sq_scale = ldexpf(1.0f, a_scale);
  }
  const double out_scale = std::ldexp(1.0, -(a_scale + a.dt_scale));
  CUtensorMap m = tma_map_2d_16bit(a.dt, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, a.ld_t, kN,
                                   a.ld_t * 2, 64, kN);
  uint64_t items = (uint64_t)geo.n_tiles * geo.n_segs;
  unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(items, (uint64_t)a.sm_count));
  spmm_tc_kernel<<<grid, kSpThreads, kSpSmemBytes, s>>>(m, b.off.ptr, b.data.ptr, b.rows, geo, vm,
                                                        a.row_means, out_scale, to, a.error);
  KG_LAUNCH_CHECK();
  if (to.mode == kOutGroups && a.out.mode == kOutRows) {
    rows_of_groups_kernel<<<b.n_tiles, 512, 0, s>>>(groups.ptr, n_groups, b.rows, out_scale, a.out);
    KG_LAUNCH_CHECK();
  } else if (to.mode == kOutGroups) {
    const uint32_t segs = (uint32_t)((geo.n_chunks + seg_chunks - 1) / seg_chunks);
    sum_groups_kernel<<<dim3(blocks_for(b.rows * kN, 256), segs), 256, 0, s>>>(
        groups.ptr, n_groups, (uint32_t)((seg_chunks + kFlushChunks - 1) / kFlushChunks), b.rows, out_scale,
        a.out.partial);
    KG_LAUNCH_CHECK();
  }
}

}  // namespace kg
