// normalize_total / log1p and the seurat HVG statistics pass on the device, and the
// seurat flags on the host (kyto computes them on the host too).
#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>
#include <limits>
#include <vector>

#include "kg_internal.cuh"
#include "kg_maps.cuh"

namespace kg {

// The largest gene index of a block (a block's indices must be below its genes).
__global__ void max_index_kernel(const uint32_t* idx, uint64_t nnz, unsigned int* out) {
  unsigned int m = 0;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nnz;
       i += (uint64_t)gridDim.x * blockDim.x)
    m = max(m, idx[i]);
  for (int o = 16; o; o >>= 1) m = max(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  if ((threadIdx.x & 31u) == 0) atomicMax(out, m);
}

// Refuses a block whose largest gene index is `worst`.
void check_worst_index(uint32_t worst, uint32_t n_genes) {
  if (worst >= n_genes)
    fail(KG_ERR_INVALID, "a block holds gene index " + std::to_string(worst) + " but has " +
                             std::to_string(n_genes) + " genes");
}

void check_indices(const uint32_t* d_idx, uint64_t nnz, uint32_t n_genes, cudaStream_t s) {
  if (!nnz) return;
  DeviceBuffer<unsigned int> m(1, s);
  m.zero();
  unsigned blocks = std::min<unsigned>(blocks_for(nnz, 256), 4096);
  max_index_kernel<<<blocks, 256, 0, s>>>(d_idx, nnz, m.ptr);
  KG_LAUNCH_CHECK();
  unsigned int h = 0;
  KG_CUDA(cudaMemcpyAsync(&h, m.ptr, 4, cudaMemcpyDeviceToHost, s));
  KG_CUDA(cudaStreamSynchronize(s));
  check_worst_index(h, n_genes);
}

// A warp per row: the row's divisor, its table (kg_maps.cuh), then its mapped values, four
// loads in flight a lane. HBM-bound: 8 bytes a value (the second read of a row comes from
// L2); 8,192 rows of 1,900 counts: 39 us, 3.2 TB/s (eight threads a row with a log1p a value
// and a rounding pass before: 296 us).
// Short rows leave a warp's lanes idle, and the instructions bound it. Where a block of kShortRows
// or more holds kShortRow values a row or fewer, eight lanes take a row and map value by value (the
// offsets tell, so no host waits for them): 1M rows of 30 counts 200 us, a warp a row 400; with
// 8,000 rows of 30 both take 16. So they do where a block of kManyRows or more holds f32 values that
// are no counts: a row's divisor is then eight chains of additions, which a warp a row computes
// four times over (100,000 rows of 200: 105 us, a warp a row 139; with fewer rows the warps are
// what is short).
constexpr int kMapWarps = 8;
constexpr unsigned kMapBlocks = 8192;  // at most: warps go on to further rows
constexpr uint64_t kShortRow = 64, kShortRows = 16384, kManyRows = 32768;
template <class V>
__global__ void __launch_bounds__(kMapWarps * 32)
normalize_log1p_kernel(const uint64_t* indptr, const V* __restrict__ values, uint64_t n_rows,
                       float target32, int normalize, int do_log1p, float* __restrict__ out) {
  __shared__ float tables[kMapWarps][kMapTable];
  const unsigned lane = threadIdx.x & 31u;
  const uint64_t first = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const uint64_t warps = gridDim.x * (uint64_t)kMapWarps;
  bool eight = false;
  if (n_rows >= kShortRows) {
    const uint64_t s0 = indptr[0], end = indptr[n_rows];
    eight = end - s0 <= kShortRow * n_rows;
    if (!eight && normalize && n_rows >= kManyRows) eight = !row_of_counts(values, s0, end);
  }
  if (eight) {
    for (uint64_t row4 = 4 * first; row4 < n_rows; row4 += 4 * warps) {  // whole warps
      const uint64_t row = row4 + lane / 8;
      const uint64_t s = row < n_rows ? indptr[row] : 0, e = row < n_rows ? indptr[row + 1] : 0;
      // (A u32 count that is not an f32 enters its row's sum rounded: whole_value.)
      const float divisor = normalize ? row_divisor(values, s, e, target32, true) : 1.0f;
      for (uint64_t i = s + (lane & 7u); i < e; i += 8)
        out[i] = mapped_f32(to_f32(values[i]), normalize != 0, divisor, do_log1p != 0);
    }
    return;
  }
  for (uint64_t row = first; row < n_rows; row += warps) {
    const uint64_t s = indptr[row], e = indptr[row + 1];
    RowMap map{tables[threadIdx.x >> 5], 1.0f, normalize != 0, do_log1p != 0};
    const bool counts = row_of_counts(values, s, e);
    if (normalize) map.divisor = warp_row_divisor(values, s, e, target32, counts);
    map.fill(e - s, counts);
    uint64_t i = s + lane;
    for (; i + 96 < e; i += 128) {
      const V a = values[i], b = values[i + 32], c = values[i + 64], d = values[i + 96];
      out[i] = map.at(a);
      out[i + 32] = map.at(b);
      out[i + 64] = map.at(c);
      out[i + 96] = map.at(d);
    }
    for (; i < e; i += 32) out[i] = map.at(values[i]);
  }
}

// Device f32 map outputs of a (device) CSR block.
void map_block(const uint64_t* d_indptr, const void* d_values, kg_dtype dtype,
               uint64_t n_rows, double target_sum, int do_log1p, float* d_out,
               cudaStream_t stream) {
  if (!n_rows) return;
  const int normalize = std::isnan(target_sum) ? 0 : 1;
  const unsigned blocks = std::min(blocks_for(n_rows, kMapWarps), kMapBlocks);
  if (dtype == KG_U32)
    normalize_log1p_kernel<uint32_t><<<blocks, kMapWarps * 32, 0, stream>>>(
        d_indptr, (const uint32_t*)d_values, n_rows, (float)target_sum, normalize, do_log1p,
        d_out);
  else
    normalize_log1p_kernel<float><<<blocks, kMapWarps * 32, 0, stream>>>(
        d_indptr, (const float*)d_values, n_rows, (float)target_sum, normalize, do_log1p, d_out);
  KG_LAUNCH_CHECK();
}

// seurat's transformed value and its f32 square (hvg_pass.rs:189-206).
__global__ void expm1_kernel(const float* v, uint64_t nnz, float* t) {
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < nnz;
       i += (uint64_t)gridDim.x * blockDim.x)
    t[i] = (float)expm1((double)v[i]);
}

// colptr[g] = first sorted entry of gene >= g.
__global__ void column_starts_kernel(const uint32_t* sorted_genes, uint64_t nnz,
                                     uint32_t n_genes, uint64_t* colptr) {
  uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (g > n_genes) return;
  uint64_t lo = 0, hi = nnz;
  while (lo < hi) {
    uint64_t mid = (lo + hi) >> 1;
    if (sorted_genes[mid] < g) lo = mid + 1; else hi = mid;
  }
  colptr[g] = lo;
}

// ----- The moments without a sort. seurat_rows_kernel maps the rows once (and notes where
// each crosses from one group of genes to the next); group_moments_kernel then gives every
// group of genes a CTA that walks all rows in order. A radix sort of (gene, value) pairs and
// one chain a gene over the sorted values, behind separate map, expm1, range and rounding
// passes, took 5.4 ms for 95M values of 20,000 genes; placing the values gene by gene with
// scattered writes instead of the sort, 2.7 ms (23 four-byte writes a clock, all SMs); this,
// 1.6 ms.

enum : int { kFlagWorst = 0, kFlagUnsorted = 1, kFlagWide = 2, kFlags = 3 };
constexpr int kSeuratThreads = 256;       // 32 rows, four a warp
constexpr uint32_t kGroupsMax = 1024;     // groups of genes (their bounds a shared-memory tile)

__device__ __forceinline__ float seurat_value(float mapped) { return (float)expm1((double)mapped); }

// t[i] = seurat's f32(expm1(f64(mapped value))) of every stored value; bounds[(k - 1) * n_rows
// + row] = the row's first entry of a gene in group k >= 1 (group_genes genes each) or later;
// flags: [kFlagWorst] the largest gene index at or past n_genes (0: none), [kFlagUnsorted]
// set by a row whose genes do not increase strictly, [kFlagWide] set by a seurat value that
// is not 0 nor of a magnitude in [least, 2^60). HBM-bound: 8 bytes a value in, 4 out.
template <class V>
__global__ void __launch_bounds__(kSeuratThreads, 5)
seurat_rows_kernel(const uint64_t* indptr, const uint32_t* __restrict__ idx,
                   const V* __restrict__ values, uint64_t n_rows, uint32_t n_genes,
                   uint32_t magic, uint32_t groups, int normalize,
                   float target32, int do_log1p, float least, float* __restrict__ t,
                   uint32_t* bounds, unsigned int* flags) {
  __shared__ float tables[kSeuratThreads / 32][kMapTable];
  extern __shared__ uint32_t crossing[];  // [groups - 1][33]
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t rb = blockIdx.x * 32ull;
  // The block will be sorted: nothing here is used any more.
  if (__syncthreads_or(threadIdx.x == 0 && *(volatile unsigned int*)(flags + kFlagUnsorted))) return;
  for (uint32_t rr = warp; rr < 32 && rb + rr < n_rows; rr += kSeuratThreads / 32) {
    const uint64_t r = rb + rr;
    const uint64_t s = indptr[r], e = max(indptr[r + 1], s);  // (a row that ends before it starts)
    RowMap map{tables[warp], 1.0f, normalize != 0, do_log1p != 0};
    const bool counts = row_of_counts(values, s, e);
    if (normalize) map.divisor = warp_row_divisor(values, s, e, target32, counts);
    const bool tabled = RowMap::tabled(e - s, counts);
    if (tabled) {
      __syncwarp();
      for (uint32_t c = lane; c < kMapTable; c += 32)
        map.table[c] = seurat_value(mapped_f32((float)c, map.normalize, map.divisor, map.do_log1p));
      __syncwarp();
    }
    // gene / group_genes: exact for genes below 2^24 (magic = ceil(2^32 / group_genes), a
    // divisor of at most 2^8); a gene out of range may land in any group.
    auto group_of = [&](uint32_t gene) { return min(__umulhi(gene, magic), groups - 1); };
    const uint32_t* row_idx = idx + s;
    const V* row_values = values + s;
    float* row_t = t + s;
    const uint32_t len = (uint32_t)(e - s), at = (uint32_t)s;
    bool unsorted = indptr[r + 1] < s, wide = false;
    uint32_t worst = 0, carry = 0;  // carry: the gene before the chunk's first
    for (uint32_t j0 = 0; j0 < len; j0 += 128) {
      uint32_t gene[4];
      V v[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint32_t j = j0 + 32 * m + lane;
        gene[m] = j < len ? row_idx[j] : 0;
        v[m] = j < len ? row_values[j] : V(0);
      }
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint32_t j = j0 + 32 * m + lane;
        uint32_t before = __shfl_up_sync(0xFFFFFFFFu, gene[m], 1);
        if (lane == 0) before = carry;
        carry = __shfl_sync(0xFFFFFFFFu, gene[m], 31);
        if (j >= len) continue;
        unsorted |= j > 0 && before >= gene[m];
        worst = max(worst, gene[m]);
        // The groups whose first entry this is: those after the previous entry's.
        const uint32_t to = group_of(gene[m]);
        for (uint32_t k = j > 0 ? group_of(before) : 0; k < to; ++k) crossing[k * 33 + rr] = at + j;
        uint32_t c;
        const float x = tabled && map_tabled(v[m], c)
                            ? map.table[c]
                            : seurat_value(mapped_f32(to_f32(v[m]), map.normalize, map.divisor,
                                                      map.do_log1p));
        wide |= x != 0.0f && !(fabsf(x) >= least && fabsf(x) < 0x1p60f);
        row_t[j] = x;
      }
    }
    for (uint32_t k = (len ? group_of(row_idx[len - 1]) : 0) + lane; k + 1 < groups; k += 32)
      crossing[k * 33 + rr] = at + len;
    if (worst >= n_genes) atomicMax(flags + kFlagWorst, worst);
    if (__any_sync(0xFFFFFFFFu, unsorted) && lane == 0) flags[kFlagUnsorted] = 1;
    if (__any_sync(0xFFFFFFFFu, wide) && lane == 0) flags[kFlagWide] = 1;
  }
  __syncthreads();
  for (uint32_t k = 1 + warp; k < groups; k += kSeuratThreads / 32)
    if (rb + lane < n_rows) bounds[(uint64_t)(k - 1) * n_rows + rb + lane] = crossing[(k - 1) * 33 + lane];
}

// The moments of group blockIdx.x's genes: the bits of kyto's single-leaf fold (per gene two
// f64 sums, each in cell order). Rows come through a ring of kRing dense tiles of kTileRows
// rows x the group's genes in shared memory (f32, zeros where a row holds nothing: adding
// them changes no sum). kRing teams of loading warps fill every kRing-th tile each: zeros,
// the rows' entries, so their loads' latency spreads over as many tiles' time. The chain warps, a
// gene a lane, then add a tile's rows in order.
// The chains' instructions bound it: per row and lane two dependent f64 additions and the
// conversions before them, one through the conversion unit (16 lanes a clock an SM), the
// square's by shifting its bits. That shift reads an f32 zero as 2^-127. A gene's zeros before its
// first real square add up to less than n_rows of those, which that square swallows while it is
// large enough (least_value; a gene of no nonzero value is put right at the end); a block with
// other values converts both.
constexpr int kTileRows = 32;
constexpr int kRing = 7;               // two named barriers a slot, 15 in all
constexpr int kTeamWarps = 2;
constexpr int kLoadWarps = kRing * kTeamWarps;
constexpr uint32_t kGroupGenes = 192;  // at most (6 chain warps)
constexpr int kRowsAWarp = kTileRows / kTeamWarps;

__device__ __forceinline__ double widen_square(float v) {
  const uint32_t b = __float_as_uint(v);
  return __hiloint2double((int)((b >> 3) + 0x38000000u), (int)(b << 29));
}

__global__ void __launch_bounds__(kLoadWarps * 32 + kGroupGenes, 1)
group_moments_kernel(const uint64_t* indptr, const uint32_t* __restrict__ idx,
                     const float* __restrict__ t, uint64_t n_rows, uint32_t n_genes,
                     uint32_t group_genes, uint32_t groups, const uint32_t* __restrict__ bounds,
                     const unsigned int* flags, double* sums, double* squares,
                     uint64_t* positives) {
  extern __shared__ float tiles[];  // [kRing][kTileRows][group_genes], then two counts a gene
  if (flags[kFlagUnsorted]) return;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t k = blockIdx.x, g0 = k * group_genes;
  const uint32_t genes = min(group_genes, n_genes - g0);
  const uint64_t n_tiles = (n_rows + kTileRows - 1) / kTileRows;
  const uint32_t tile_floats = kTileRows * group_genes;
  uint32_t* n_positive = reinterpret_cast<uint32_t*>(tiles + kRing * tile_floats);
  uint32_t* n_other = n_positive + group_genes;
  for (uint32_t x = threadIdx.x; x < 2 * group_genes; x += blockDim.x) n_positive[x] = 0;
  __syncthreads();
  // Barrier 1 + slot: a filled tile (its team arrives, the chain warps wait); barrier 1 +
  // kRing + slot: an emptied one (the other way round).
  const uint32_t both = kTeamWarps * 32 + group_genes;
  if (warp < kLoadWarps) {
    const uint32_t slot = warp / kTeamWarps, member = warp % kTeamWarps;
    const uint32_t half = lane >> 4, l = lane & 15u;  // two rows at a time
    float* rows = tiles + slot * tile_floats + member * kRowsAWarp * group_genes;
    auto put = [&](uint32_t row, uint32_t gene, float v) {
      if (gene >= genes) return;
      rows[row * group_genes + gene] = v;
      // t > 0 exactly when the log1p value > 0.
      if (v != 0.0f) atomicAdd((v > 0.0f ? n_positive : n_other) + gene, 1u);
    };
    // A row's range: lane j the warp's row j of tile b.
    auto ranges = [&](uint64_t b, uint32_t& from, uint32_t& to) {
      const uint64_t r = b * kTileRows + member * kRowsAWarp + lane;
      from = to = 0;
      if (lane < kRowsAWarp && r < n_rows) {
        from = k == 0 ? (uint32_t)indptr[r] : bounds[(uint64_t)(k - 1) * n_rows + r];
        to = k + 1 == groups ? (uint32_t)indptr[r + 1] : bounds[(uint64_t)k * n_rows + r];
      }
    };
    uint32_t next_lo = 0, next_hi = 0;
    ranges(slot, next_lo, next_hi);
    for (uint64_t b = slot; b < n_tiles; b += kRing) {
      // The warp's rows' entries (and the next tile's ranges), before the tile is free.
      const uint32_t lo = next_lo, hi = next_hi;
      uint32_t gene[kRowsAWarp / 2][2];
      float v[kRowsAWarp / 2][2];
      bool more = false;
#pragma unroll
      for (int j = 0; j < kRowsAWarp / 2; ++j) {
        const uint32_t a = __shfl_sync(0xFFFFFFFFu, lo, 2 * j + half) + l;
        const uint32_t e = __shfl_sync(0xFFFFFFFFu, hi, 2 * j + half);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          const bool in = a < e && e - a > 16u * m;
          gene[j][m] = in ? idx[a + 16 * m] - g0 : 0xFFFFFFFFu;
          v[j][m] = in ? t[a + 16 * m] : 0.0f;
        }
        more |= a < e && e - a > 32;
      }
      ranges(b + kRing, next_lo, next_hi);
      if (b >= kRing) asm volatile("bar.sync %0, %1;" ::"r"(1 + kRing + slot), "r"(both) : "memory");
      for (uint32_t x = lane * 4; x < kRowsAWarp * group_genes; x += 128)
        *reinterpret_cast<float4*>(rows + x) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < kRowsAWarp / 2; ++j)
#pragma unroll
        for (int m = 0; m < 2; ++m) put(2 * j + half, gene[j][m], v[j][m]);
      if (__any_sync(0xFFFFFFFFu, more)) {  // a row of over 32 values in the group
        for (int j = 0; j < kRowsAWarp / 2; ++j) {
          const uint32_t a = __shfl_sync(0xFFFFFFFFu, lo, 2 * j + half) + 32 + l;
          const uint32_t e = __shfl_sync(0xFFFFFFFFu, hi, 2 * j + half);
          for (uint32_t i = a; i < e; i += 16) put(2 * j + half, idx[i] - g0, t[i]);
        }
      }
      asm volatile("bar.arrive %0, %1;" ::"r"(1 + slot), "r"(both) : "memory");
    }
    __syncthreads();
  } else {
    const uint32_t c = threadIdx.x - kLoadWarps * 32;  // < group_genes (the block's size)
    const bool wide = flags[kFlagWide] != 0;
    double s = 0.0, q = 0.0;
    for (uint64_t b = 0; b < n_tiles; ++b) {
      const uint32_t slot = (uint32_t)(b % kRing);
      asm volatile("bar.sync %0, %1;" ::"r"(1 + slot), "r"(both) : "memory");
      const float* at = tiles + slot * tile_floats + c;
      for (int r0 = 0; r0 < kTileRows; r0 += 16) {
        float x[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) x[r] = at[(r0 + r) * group_genes];
        if (!wide) {
#pragma unroll
          for (int r = 0; r < 16; ++r) {
            s = __dadd_rn(s, (double)x[r]);
            q = __dadd_rn(q, widen_square(__fmul_rn(x[r], x[r])));
          }
        } else {
#pragma unroll
          for (int r = 0; r < 16; ++r) {
            s = __dadd_rn(s, (double)x[r]);
            q = __dadd_rn(q, (double)__fmul_rn(x[r], x[r]));
          }
        }
      }
      if (b + kRing < n_tiles)
        asm volatile("bar.arrive %0, %1;" ::"r"(1 + kRing + slot), "r"(both) : "memory");
    }
    __syncthreads();
    if (c < genes) {
      sums[g0 + c] = s;
      squares[g0 + c] = n_positive[c] + n_other[c] ? q : 0.0;
      positives[g0 + c] = n_positive[c];
    }
  }
}

// ----- The moments of values already sorted by gene.

// A warp per four genes, their cells in cell order: the bits of kyto's single-leaf fold (two
// f64 sums a gene, each in one fixed sequential order). The lanes bring the next 64 values
// of each gene and leave them, and their squares, in shared memory as f64 while the eight
// sums (lane modulo 8) run over the 64 before: a chain of dependent additions each, with the
// conversions between them. The longest gene's chain bounds it (8.5 cycles an addition; one
// lane converting, squaring and adding both sums took 94 cycles a value, 2.45 ms for genes of
// 50,000 cells).
constexpr int kMomentWarps = 4;
constexpr int kMomentGenes = 4;
constexpr int kMomentChunk = 64;

__global__ void __launch_bounds__(kMomentWarps * 32)
gene_moments_kernel(const uint64_t* colptr, const float* __restrict__ t, uint32_t n_genes,
                    double* sums, double* squares, uint64_t* positives) {
  constexpr int kParts = kMomentChunk / 32;
  // Rows of 16-byte multiples whose starts fall on different banks.
  __shared__ __align__(16) double buf[kMomentWarps][2][2 * kMomentGenes][kMomentChunk + 2];
  const unsigned lane = threadIdx.x & 31u, wi = threadIdx.x >> 5;
  const uint32_t g0 = (blockIdx.x * kMomentWarps + wi) * kMomentGenes;
  if (g0 >= n_genes) return;
  uint64_t at[kMomentGenes], end[kMomentGenes], longest = 0;
  uint32_t p[kMomentGenes];
#pragma unroll
  for (int k = 0; k < kMomentGenes; ++k) {
    const bool in = g0 + k < n_genes;
    at[k] = in ? colptr[g0 + k] : 0;
    end[k] = in ? colptr[g0 + k + 1] : 0;
    longest = max(longest, end[k] - at[k]);
    p[k] = 0;
  }
  float x[kMomentGenes * kParts];
  auto load = [&]() {
#pragma unroll
    for (int k = 0; k < kMomentGenes; ++k) {
#pragma unroll
      for (int m = 0; m < kParts; ++m) {
        const uint64_t i = at[k] + m * 32 + lane;
        x[k * kParts + m] = i < end[k] ? t[i] : 0.0f;  // past the gene: adds nothing
      }
      at[k] += kMomentChunk;
    }
  };
  auto stash = [&](int half, int q) {  // value q of x
    const int k = q / kParts, m = q % kParts;
    const float v = x[q];
    buf[wi][half][2 * k][m * 32 + lane] = (double)v;
    buf[wi][half][2 * k + 1][m * 32 + lane] = (double)__fmul_rn(v, v);
    p[k] += v > 0.0f ? 1u : 0u;  // t > 0 exactly when the log1p value > 0
  };
  constexpr int kHeld = kMomentGenes * kParts;
  const unsigned chain = lane % (2 * kMomentGenes);  // gene chain / 2, its sum or its squares
  double acc = 0.0;
  load();
#pragma unroll
  for (int q = 0; q < kHeld; ++q) stash(0, q);
  load();
  __syncwarp();
  int half = 0;
  for (uint64_t done = 0; done < longest; done += kMomentChunk, half ^= 1) {
    const double2* row = reinterpret_cast<const double2*>(buf[wi][half][chain]);
#pragma unroll
    for (int q = 0; q < kHeld; ++q) {
#pragma unroll
      for (int j = 0; j < kMomentChunk / 2 / kHeld; ++j) {
        const double2 d = lane < 2 * kMomentGenes ? row[q * (kMomentChunk / 2 / kHeld) + j]
                                                  : make_double2(0.0, 0.0);
        acc = __dadd_rn(acc, d.x);
        acc = __dadd_rn(acc, d.y);
      }
      stash(half ^ 1, q);
    }
    load();
    __syncwarp();
  }
#pragma unroll
  for (int k = 0; k < kMomentGenes; ++k) {
    uint32_t c = p[k];
    for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(0xFFFFFFFFu, c, o);
    if (lane == 0 && g0 + k < n_genes) positives[g0 + k] = c;
  }
  const uint32_t g = g0 + chain / 2;
  if (lane < 2 * kMomentGenes && g < n_genes) ((chain & 1u) ? squares : sums)[g] = acc;
}

void gene_moments(const uint64_t* colptr, const float* t, uint32_t n_genes, double* sums,
                  double* squares, uint64_t* positives, cudaStream_t s) {
  if (!n_genes) return;
  const uint32_t per = kMomentWarps * kMomentGenes;
  gene_moments_kernel<<<(n_genes + per - 1) / per, kMomentWarps * 32, 0, s>>>(
      colptr, t, n_genes, sums, squares, positives);
  KG_LAUNCH_CHECK();
}

// The least magnitude, a power of two 2^b, of the nonzero values whose squares may be widened by their
// bits: n_rows 2^-127 has to be below half an ulp of the smallest square, 2^(2 b - 53).
float least_value(uint64_t n_rows) {
  int b = -28;
  while (std::ldexp((double)n_rows, -(2 * b + 74)) >= 1.0) ++b;
  return (float)std::ldexp(1.0, b);
}

// Whether `groups` groups of `group_genes` genes suit a block. A group's CTA passes every row of the
// block, stored values or none, so its time goes by the rows (16 ns a row for groups of 32 genes, 21
// for 160; as often as the groups go over the SMs); the sort's goes by the values, after some 30
// us more of launches. Measured, group / sort: 60,000 rows of 285 values of 2,000 genes 1.21 /
// 1.20 ms, of 95 values 1.02 / 0.64; 16,000 rows of 427 of 20,000 genes 0.44 / 0.52, of 285 0.43 /
// 0.35; 250,000 rows of 95 of 20,000 genes 5.3 / 1.9; 4,000 rows of 190 of 2,000 genes 0.14 / 0.18;
// 60,000 rows of 380 of 32,000 genes (two rounds of groups) 2.7 / 1.3. The rule also keeps the groups'
// bounds, 4 bytes a row and group, below the sort's own scratch.
bool groups_suit(uint64_t n_rows, uint64_t nnz, uint32_t group_genes, uint32_t groups, int sm_count) {
  const uint64_t passes = n_rows * ((groups + sm_count - 1) / sm_count);
  return passes <= 4096 || nnz / passes >= 220 + group_genes * 5 / 4;
}

// The moments of a block whose rows hold their genes in strictly increasing order, without a
// sort; false (and nothing queued) for a shape outside the kernels' (more groups of genes than
// their bounds' tile holds) or that the sort suits better. The flags are read by the caller once
// its work is queued: a block with an index out of range or an unsorted row leaves the moments
// meaningless (every access stays inside the arrays).
template <class V>
bool moments_by_group(const uint64_t* indptr, const uint32_t* idx, const V* values,
                      uint64_t n_rows, uint64_t nnz, uint32_t n_genes, double target_sum,
                      int do_log1p, int sm_count, double* sums, double* squares,
                      uint64_t* positives, unsigned int* flags, cudaStream_t s) {
  // About a group an SM, in whole warps of genes.
  const uint32_t gg =
      std::min(kGroupGenes, ((n_genes + sm_count - 1) / sm_count + 31) / 32 * 32);
  const uint32_t groups = (n_genes + gg - 1) / gg;
  if (groups > kGroupsMax || !groups_suit(n_rows, nnz, gg, groups, sm_count)) return false;
  allow_dynamic_smem(seurat_rows_kernel<V>, kGroupsMax * 33 * 4);
  allow_dynamic_smem(group_moments_kernel, (kRing * kTileRows + 2) * kGroupGenes * 4);
  DeviceBuffer<float> t(nnz, s);
  DeviceBuffer<uint32_t> bounds((uint64_t)(groups - 1) * n_rows, s);
  seurat_rows_kernel<V><<<blocks_for(n_rows, 32), kSeuratThreads, (groups - 1) * 33 * 4, s>>>(
      indptr, idx, values, n_rows, n_genes, (uint32_t)(((1ull << 32) + gg - 1) / gg), groups,
      std::isnan(target_sum) ? 0 : 1, (float)target_sum, do_log1p, least_value(n_rows), t.ptr,
      bounds.ptr, flags);
  KG_LAUNCH_CHECK();
  group_moments_kernel<<<groups, kLoadWarps * 32 + gg, (kRing * kTileRows + 2) * gg * 4, s>>>(
      indptr, idx, t.ptr, n_rows, n_genes, gg, groups, bounds.ptr, flags, sums, squares,
      positives);
  KG_LAUNCH_CHECK();
  return true;
}

int bits_for(uint32_t n) {
  int b = 1;
  while (b < 32 && (1ull << b) < (uint64_t)n) ++b;
  return b;
}

// Stable sort of (gene, payload) by gene: each gene's payloads stay in cell order.
template <class P>
void sort_by_gene(const uint32_t* genes, const P* payload, uint64_t nnz, uint32_t n_genes,
                  DeviceBuffer<uint32_t>& genes_out, DeviceBuffer<P>& payload_out,
                  cudaStream_t stream) {
  if (nnz > (uint64_t)std::numeric_limits<int>::max())
    fail(KG_ERR_INVALID, "a block of more than 2^31 stored values");
  genes_out.alloc(nnz, stream);
  payload_out.alloc(nnz, stream);
  size_t temp = 0;
  int end_bit = bits_for(n_genes + 1);
  KG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, temp, genes, genes_out.ptr, payload,
                                          payload_out.ptr, (int)nnz, 0, end_bit, stream));
  DeviceBuffer<unsigned char> scratch(temp, stream);
  KG_CUDA(cub::DeviceRadixSort::SortPairs(scratch.ptr, temp, genes, genes_out.ptr, payload,
                                          payload_out.ptr, (int)nnz, 0, end_bit, stream));
}

template void sort_by_gene<uint32_t>(const uint32_t*, const uint32_t*, uint64_t, uint32_t,
                                     DeviceBuffer<uint32_t>&, DeviceBuffer<uint32_t>&,
                                     cudaStream_t);
template void sort_by_gene<uint64_t>(const uint32_t*, const uint64_t*, uint64_t, uint32_t,
                                     DeviceBuffer<uint32_t>&, DeviceBuffer<uint64_t>&,
                                     cudaStream_t);

void column_starts(const uint32_t* sorted_genes, uint64_t nnz, uint32_t n_genes,
                   uint64_t* colptr, cudaStream_t stream) {
  column_starts_kernel<<<blocks_for((uint64_t)n_genes + 1, 256), 256, 0, stream>>>(
      sorted_genes, nnz, n_genes, colptr);
  KG_LAUNCH_CHECK();
}

// ------------------------------------------------------------------ seurat (host) ----

double kahan_mean(const std::vector<double>& values) {
  double sum = 0.0, comp = 0.0;
  uint64_t count = 0;
  for (double v : values) {
    if (std::isnan(v)) continue;
    ++count;
    double y = v - comp;
    double t = sum + y;
    comp = t - sum - y;
    if (std::isnan(comp)) comp = 0.0;
    sum = t;
  }
  return count == 0 ? NAN : sum / (double)count;
}

double welford_std(const std::vector<double>& values) {
  uint64_t count = 0;
  double mean = 0.0, squared = 0.0;
  for (double v : values) {
    if (std::isnan(v)) continue;
    ++count;
    double prev = mean;
    mean += (v - prev) / (double)count;
    squared += (v - mean) * (v - prev);
  }
  return count <= 1 ? NAN : std::sqrt(squared / (double)(count - 1));
}

}  // namespace kg

using namespace kg;

extern "C" {

kg_status kg_normalize_log1p(kg_ctx* ctx, const uint64_t* indptr, const void* values,
                             kg_dtype dtype, uint64_t n_rows, double target_sum,
                             int32_t log1p, float* out) {
  return guarded([&] {
    if (!ctx || !indptr || (!values && n_rows) || !out)
      fail(KG_ERR_INVALID, "kg_normalize_log1p: NULL argument");
    if (dtype != KG_U32 && dtype != KG_F32) fail(KG_ERR_INVALID, "unknown dtype");
    use_device(ctx);
    cudaStream_t s = ctx->stream;
    DeviceBuffer<uint64_t> hp;
    const uint64_t* d_indptr = device_view(indptr, n_rows + 1, hp, s);
    // The stored values' count is needed for host arrays only (the kernel reads the offsets).
    const bool out_dev = is_device_pointer(out);
    uint64_t nnz = 0;
    if (!out_dev || (values && !is_device_pointer(values))) {
      KG_CUDA(cudaMemcpyAsync(&nnz, indptr + n_rows, 8, cudaMemcpyDefault, s));
      KG_CUDA(cudaStreamSynchronize(s));
    }
    DeviceBuffer<uint32_t> hv;
    const void* d_values = device_view((const uint32_t*)values, nnz, hv, s);
    DeviceBuffer<float> ho;
    float* d_out = out;
    if (!out_dev) {
      ho.alloc(nnz, s);
      d_out = ho.ptr;
    }
    map_block(d_indptr, d_values, dtype, n_rows, target_sum, log1p, d_out, s);
    if (!out_dev && nnz)
      KG_CUDA(cudaMemcpyAsync(out, d_out, nnz * 4, cudaMemcpyDeviceToHost, s));
    wait_stream(ctx, s);
  });
}

kg_status kg_hvg_moments(kg_ctx* ctx, const uint64_t* indptr, const uint32_t* indices,
                         const void* values, kg_dtype dtype, uint64_t n_rows,
                         uint32_t n_genes, double target_sum, int32_t log1p,
                         double* sums, double* sums_of_squares, uint64_t* positives) {
  return guarded([&] {
    if (!ctx || !indptr || !sums || !sums_of_squares || !positives)
      fail(KG_ERR_INVALID, "kg_hvg_moments: NULL argument");
    if (dtype != KG_U32 && dtype != KG_F32) fail(KG_ERR_INVALID, "unknown dtype");
    use_device(ctx);
    cudaStream_t s = ctx->stream;
    DeviceBuffer<uint64_t> hp;
    const uint64_t* d_indptr = device_view(indptr, n_rows + 1, hp, s);
    uint64_t nnz = 0;
    KG_CUDA(cudaMemcpyAsync(&nnz, d_indptr + n_rows, 8, cudaMemcpyDefault, s));
    KG_CUDA(cudaStreamSynchronize(s));
    DeviceBuffer<uint32_t> hi, hv;
    const uint32_t* d_idx = device_view(indices, nnz, hi, s);
    const void* d_values = device_view((const uint32_t*)values, nnz, hv, s);
    DeviceBuffer<double> dsum(n_genes, s), dsq(n_genes, s);
    DeviceBuffer<uint64_t> dpos(n_genes, s);
    // Rows of strictly increasing genes (kyto's) need no sort; a block with any other row,
    // found on the way, is sorted: what is left of the rows' pass then ends at once.
    bool sorted = nnz > 0 && n_genes > 0 && nnz <= (uint64_t)std::numeric_limits<int>::max();
    if (sorted) {
      DeviceBuffer<unsigned int> flags(kFlags, s);
      flags.zero();
      if (dtype == KG_U32)
        sorted = moments_by_group(d_indptr, d_idx, (const uint32_t*)d_values, n_rows, nnz,
                                  n_genes, target_sum, log1p, ctx->sm_count, dsum.ptr, dsq.ptr,
                                  dpos.ptr, flags.ptr, s);
      else
        sorted = moments_by_group(d_indptr, d_idx, (const float*)d_values, n_rows, nnz, n_genes,
                                  target_sum, log1p, ctx->sm_count, dsum.ptr, dsq.ptr, dpos.ptr,
                                  flags.ptr, s);
      if (sorted) {
        unsigned int h[kFlags] = {};
        KG_CUDA(cudaMemcpyAsync(h, flags.ptr, sizeof h, cudaMemcpyDeviceToHost, s));
        wait_stream(ctx, s);
        sorted = h[kFlagUnsorted] == 0;
        if (sorted) check_worst_index(h[kFlagWorst], n_genes);  // (else not every row was read)
      }
    }
    if (!sorted) {
      check_indices(d_idx, nnz, n_genes, s);
      DeviceBuffer<float> t(nnz, s);
      map_block(d_indptr, d_values, dtype, n_rows, target_sum, log1p, t.ptr, s);
      if (nnz) {
        unsigned blocks = std::min<unsigned>(blocks_for(nnz, 256), 8192);
        expm1_kernel<<<blocks, 256, 0, s>>>(t.ptr, nnz, t.ptr);
        KG_LAUNCH_CHECK();
      }
      DeviceBuffer<uint32_t> genes_sorted, t_sorted;
      sort_by_gene<uint32_t>(d_idx, (const uint32_t*)t.ptr, nnz, n_genes, genes_sorted,
                             t_sorted, s);
      DeviceBuffer<uint64_t> colptr((uint64_t)n_genes + 1, s);
      column_starts(genes_sorted.ptr, nnz, n_genes, colptr.ptr, s);
      gene_moments(colptr.ptr, (const float*)t_sorted.ptr, n_genes, dsum.ptr, dsq.ptr, dpos.ptr,
                   s);
    }
    KG_CUDA(cudaMemcpyAsync(sums, dsum.ptr, n_genes * 8ull, cudaMemcpyDefault, s));
    KG_CUDA(cudaMemcpyAsync(sums_of_squares, dsq.ptr, n_genes * 8ull, cudaMemcpyDefault, s));
    KG_CUDA(cudaMemcpyAsync(positives, dpos.ptr, n_genes * 8ull, cudaMemcpyDefault, s));
    wait_stream(ctx, s);
  });
}

kg_status kg_hvg_seurat(const double* sums, const double* sums_of_squares,
                        const uint64_t* positives, uint64_t n_cells, uint32_t n_genes,
                        int64_t n_top_genes, double* means_out, double* dispersions_out,
                        double* normalized_out, uint8_t* flags_out) {
  (void)positives;  // seurat without batches keeps every gene (hvg.rs:290-293)
  return guarded([&] {
    if (!sums || !sums_of_squares || !means_out || !dispersions_out || !normalized_out ||
        !flags_out)
      fail(KG_ERR_INVALID, "kg_hvg_seurat: NULL argument");
    const int kBins = 20;  // hvg.rs:34
    double n = (double)n_cells;
    std::vector<double> mean(n_genes), disp(n_genes), norm(n_genes, NAN);
    for (uint32_t g = 0; g < n_genes; ++g) {
      // statistics.rs:153-168 (variances with ddof=1), hvg.rs:295-308.
      double m = sums[g] / n;
      double var = sums_of_squares[g] / n - m * m;
      if (n_cells != 1) var = var * (n / (n - 1.0));
      if (m == 0.0) m = 1e-12;
      double d = var / m;
      if (d == 0.0) d = NAN;
      d = std::log(d);
      mean[g] = std::log1p(m);
      disp[g] = d;
    }
    // hvg.rs:393-425: 20 equal-width bins (pd.cut).
    double lo = INFINITY, hi = -INFINITY;
    bool any = false;
    for (double m : mean)
      if (!std::isnan(m)) {
        lo = std::min(lo, m);
        hi = std::max(hi, m);
        any = true;
      }
    std::vector<int> bins(n_genes, -1);
    if (any) {
      std::vector<double> edges(kBins + 1);
      auto linspace = [&](double a, double b) {
        double step = (b - a) / (double)kBins;
        for (int i = 0; i <= kBins; ++i) edges[i] = (double)i * step + a;
        edges[kBins] = b;
      };
      if (lo == hi) {
        linspace(lo - (lo == 0.0 ? 0.001 : 0.001 * std::fabs(lo)),
                 hi + (hi == 0.0 ? 0.001 : 0.001 * std::fabs(hi)));
      } else {
        linspace(lo, hi);
        edges[0] -= (hi - lo) * 0.001;
      }
      for (uint32_t g = 0; g < n_genes; ++g) {
        if (std::isnan(mean[g])) continue;
        int index = (int)(std::lower_bound(edges.begin(), edges.end(), mean[g]) -
                          edges.begin());
        index = std::max(index, 1);
        if (index < (int)edges.size()) bins[g] = index - 1;
      }
    }
    // hvg.rs:501-535: z-score of the dispersion in its bin.
    std::vector<std::vector<double>> members(kBins);
    for (uint32_t g = 0; g < n_genes; ++g)
      if (bins[g] >= 0) members[bins[g]].push_back(disp[g]);
    std::vector<std::pair<double, double>> stats(kBins);
    for (int b = 0; b < kBins; ++b) {
      double avg = kahan_mean(members[b]);
      double dev = welford_std(members[b]);
      stats[b] = std::isnan(dev) ? std::make_pair(0.0, avg) : std::make_pair(avg, dev);
    }
    for (uint32_t g = 0; g < n_genes; ++g)
      if (bins[g] >= 0) norm[g] = (disp[g] - stats[bins[g]].first) / stats[bins[g]].second;
    // hvg.rs:320-349: top n by >= cutoff, or scanpy's cutoffs.
    auto nan_to_num = [](double v, double nan) {
      if (std::isnan(v)) return nan;
      if (v == INFINITY) return std::numeric_limits<double>::max();
      if (v == -INFINITY) return std::numeric_limits<double>::lowest();
      return v;
    };
    if (n_top_genes >= 0) {
      std::vector<double> finite;
      for (double v : norm)
        if (!std::isnan(v)) finite.push_back(v);
      uint64_t count = std::min<uint64_t>((uint64_t)n_top_genes,
                                          std::min<uint64_t>(n_genes, finite.size()));
      if (count == 0) {
        for (uint32_t g = 0; g < n_genes; ++g) flags_out[g] = 0;
      } else {
        std::sort(finite.begin(), finite.end(), [](double a, double b) { return a > b; });
        double cutoff = finite[count - 1];
        for (uint32_t g = 0; g < n_genes; ++g)
          flags_out[g] = nan_to_num(norm[g], -INFINITY) >= cutoff ? 1 : 0;
      }
    } else {
      for (uint32_t g = 0; g < n_genes; ++g) {
        double z = nan_to_num(norm[g], 0.0);
        flags_out[g] = (mean[g] > 0.0125 && mean[g] < 3.0 && z > 0.5 && z < INFINITY) ? 1 : 0;
      }
    }
    for (uint32_t g = 0; g < n_genes; ++g) {
      means_out[g] = mean[g];
      dispersions_out[g] = disp[g];
      normalized_out[g] = norm[g];
    }
  });
}

}  // extern "C"

// ------------------------------------------ seurat moments in fixed scratch ----------

namespace kg {

constexpr size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// The limits of kg_hvg_moments_noalloc and the layout of its scratch (byte offsets):
// the largest index, the sort's key and payload double buffers, the per-gene arrays, the radix
// sort's temporary storage. 22.1 MB in all.
constexpr uint64_t kNoAllocMaxValues = 1ull << 20;  // stored values of one block
constexpr uint32_t kNoAllocMaxGenes = 1u << 16;
constexpr size_t kNoAllocValues = align256(kNoAllocMaxValues * 4);
constexpr size_t kNoAllocGenes = align256(((size_t)kNoAllocMaxGenes + 1) * 8);
constexpr size_t kNoAllocKeys0 = 256;
constexpr size_t kNoAllocKeys1 = kNoAllocKeys0 + kNoAllocValues;
constexpr size_t kNoAllocVals0 = kNoAllocKeys1 + kNoAllocValues;
constexpr size_t kNoAllocVals1 = kNoAllocVals0 + kNoAllocValues;
constexpr size_t kNoAllocColptr = kNoAllocVals1 + kNoAllocValues;
constexpr size_t kNoAllocSums = kNoAllocColptr + kNoAllocGenes;
constexpr size_t kNoAllocSquares = kNoAllocSums + kNoAllocGenes;
constexpr size_t kNoAllocPositives = kNoAllocSquares + kNoAllocGenes;
constexpr size_t kNoAllocSort = kNoAllocPositives + kNoAllocGenes;
constexpr size_t kNoAllocSortBytes = 4u << 20;
constexpr size_t kNoAllocBytes = kNoAllocSort + kNoAllocSortBytes;

// One array per device (this module's static device memory), shared by every call on
// that device.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

constexpr int kNoAllocDevices = 64;

// The scratch's device address on `device` (which must be current). The first call on
// a device resolves it with cudaGetSymbolAddress, which loads this module there, and
// checks that the radix sort's storage for the largest block fits its slot.
unsigned char* noalloc_scratch(int device) {
  static std::mutex mu;
  static unsigned char* resolved[kNoAllocDevices] = {};
  if (device < 0 || device >= kNoAllocDevices)
    fail(KG_ERR_INVALID, "kg_hvg_moments_noalloc: device ordinal above 63");
  std::lock_guard<std::mutex> lock(mu);
  if (resolved[device]) return resolved[device];
  void* p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
  if (e != cudaSuccess) fail_cuda(e, "cudaGetSymbolAddress (fixed scratch)", __FILE__, __LINE__);
  size_t temp = 0;
  cub::DoubleBuffer<uint32_t> keys(nullptr, nullptr), vals(nullptr, nullptr);
  KG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, temp, keys, vals, (int)kNoAllocMaxValues, 0,
                                          bits_for(kNoAllocMaxGenes + 1)));
  if (temp > kNoAllocSortBytes)
    fail(KG_ERR_DEVICE, "kg_hvg_moments_noalloc: the radix sort wants " +
                            std::to_string(temp) + " bytes, above its fixed slot");
  resolved[device] = (unsigned char*)p;
  return resolved[device];
}

}  // namespace kg

extern "C" {

kg_status kg_hvg_moments_noalloc(kg_ctx* ctx, const uint64_t* indptr, const uint32_t* indices,
                                 const void* values, kg_dtype dtype, uint64_t n_rows,
                                 uint32_t n_genes, double target_sum, int32_t log1p,
                                 double* sums, double* sums_of_squares, uint64_t* positives) {
  return guarded([&] {
    if (!ctx || !indptr || !sums || !sums_of_squares || !positives)
      fail(KG_ERR_INVALID, "kg_hvg_moments_noalloc: NULL argument");
    if (dtype != KG_U32 && dtype != KG_F32) fail(KG_ERR_INVALID, "unknown dtype");
    if (n_genes > kNoAllocMaxGenes)
      fail(KG_ERR_INVALID, "kg_hvg_moments_noalloc: " + std::to_string(n_genes) +
                               " genes, above its limit of " +
                               std::to_string(kNoAllocMaxGenes) + " (use kg_hvg_moments)");
    use_device(ctx);
    if (!is_device_pointer(indptr))
      fail(KG_ERR_INVALID, "kg_hvg_moments_noalloc: indptr must be device memory");
    unsigned char* base = noalloc_scratch(ctx->device);
    cudaStream_t s = ctx->stream;
    uint64_t nnz = 0;
    KG_CUDA(cudaMemcpyAsync(&nnz, indptr + n_rows, 8, cudaMemcpyDeviceToHost, s));
    KG_CUDA(cudaStreamSynchronize(s));
    if (nnz > kNoAllocMaxValues)
      fail(KG_ERR_INVALID, "kg_hvg_moments_noalloc: a block of " + std::to_string(nnz) +
                               " stored values, above its limit of " +
                               std::to_string(kNoAllocMaxValues) + " (use kg_hvg_moments)");
    if (nnz && (!is_device_pointer(indices) || !is_device_pointer(values)))
      fail(KG_ERR_INVALID, "kg_hvg_moments_noalloc: indices and values must be device memory");
    unsigned int* max_index = (unsigned int*)base;
    uint32_t* keys0 = (uint32_t*)(base + kNoAllocKeys0);
    uint32_t* keys1 = (uint32_t*)(base + kNoAllocKeys1);
    float* vals0 = (float*)(base + kNoAllocVals0);
    float* vals1 = (float*)(base + kNoAllocVals1);
    uint64_t* colptr = (uint64_t*)(base + kNoAllocColptr);
    double* dsum = (double*)(base + kNoAllocSums);
    double* dsq = (double*)(base + kNoAllocSquares);
    uint64_t* dpos = (uint64_t*)(base + kNoAllocPositives);
    KG_CUDA(cudaMemsetAsync(base, 0, 8, s));
    cub::DoubleBuffer<uint32_t> keys(keys0, keys1), vals((uint32_t*)vals0, (uint32_t*)vals1);
    if (nnz) {
      unsigned blocks = std::min<unsigned>(blocks_for(nnz, 256), 4096);
      max_index_kernel<<<blocks, 256, 0, s>>>(indices, nnz, max_index);
      KG_LAUNCH_CHECK();
      unsigned int h = 0;
      KG_CUDA(cudaMemcpyAsync(&h, max_index, 4, cudaMemcpyDeviceToHost, s));
      KG_CUDA(cudaStreamSynchronize(s));
      check_worst_index(h, n_genes);
      map_block(indptr, values, dtype, n_rows, target_sum, log1p, vals0, s);
      expm1_kernel<<<std::min<unsigned>(blocks_for(nnz, 256), 8192), 256, 0, s>>>(vals0, nnz,
                                                                                 vals0);
      KG_LAUNCH_CHECK();
      // The sort may write either half of each double buffer: the keys start as a copy.
      KG_CUDA(cudaMemcpyAsync(keys0, indices, nnz * 4, cudaMemcpyDeviceToDevice, s));
      size_t temp = 0;
      int end_bit = bits_for(n_genes + 1);
      KG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, temp, keys, vals, (int)nnz, 0, end_bit,
                                              s));
      if (temp > kNoAllocSortBytes)
        fail(KG_ERR_DEVICE, "kg_hvg_moments_noalloc: the radix sort wants " +
                                std::to_string(temp) + " bytes, above its fixed slot");
      temp = kNoAllocSortBytes;
      KG_CUDA(cub::DeviceRadixSort::SortPairs(base + kNoAllocSort, temp, keys, vals, (int)nnz,
                                              0, end_bit, s));
    }
    if (n_genes) {
      column_starts(keys.Current(), nnz, n_genes, colptr, s);
      gene_moments(colptr, (const float*)vals.Current(), n_genes, dsum, dsq, dpos, s);
      KG_CUDA(cudaMemcpyAsync(sums, dsum, n_genes * 8ull, cudaMemcpyDefault, s));
      KG_CUDA(cudaMemcpyAsync(sums_of_squares, dsq, n_genes * 8ull, cudaMemcpyDefault, s));
      KG_CUDA(cudaMemcpyAsync(positives, dpos, n_genes * 8ull, cudaMemcpyDefault, s));
    }
    wait_stream(ctx, s);
  });
}

}  // extern "C"
