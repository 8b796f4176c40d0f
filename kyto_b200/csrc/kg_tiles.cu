// One cell block of kyto's tiled sparse layers (docs/format.md 4.1-4.3) joined into CSR
// rows on the device: kyto-store's decode_cell_block and its checks
// (crates/kyto-store/src/tile_decode.rs:74-196), which kyto runs on the host before
// kyto-exec rebuilds the rows once more for its GPU path (pca/gpu.rs:73-115).
//
// Two kernels, each a pass over bytes (no arithmetic to speak of; latency and launches bound
// a block's few MB):
//   1. tile_check_kernel: a thread per value of the block's indptr shard checks kyto's four
//      indptr rules (starts at 0, ends at the tile's nnz, never decreases, flat over padding
//      rows); a warp per row and tile checks that the row's local indices strictly increase
//      below the block width, its range cut to the tile (a tile whose indptr breaks a rule is
//      reported for that rule first, whatever its rows hold);
//   2. tile_join_kernel: a warp per row and tile copies its segment, adding the block's first
//      gene to the local indices, unless the checks found a problem (then it writes nothing).
//      A tile's indptr counts its entries in the rows before, so a segment's place is a sum
//      over the tiles' indptrs (row r, and row r + 1 of the tiles before it): no scan.
// Every problem found becomes one 64-bit key ordered as kyto reports problems (gene
// block, then the check in kyto's order, then the row, then which of a row's two checks
// fails), and the smallest key wins (atomicMin). Both kernels are queued at once; the host
// reads the key once, after the join, and words a problem as kyto does (KG_ERR_CORRUPT,
// kyto's KY-E107). A call waits once (twice with host outputs, three times with
// device-resident tile_offsets).
// A block of 4,096 x 627 entries in two tiles: 48 us a call, 20 us in the kernels; checking and summing the rows,
// scanning their lengths and joining a row a warp took 81 us (the join alone 33 us).

#include <algorithm>
#include <cstring>
#include <string>

#include "kg_tiles.cuh"

namespace kg {
namespace {

constexpr unsigned long long kNoProblem = ~0ull;
// The checks in kyto's order: check_tile_indptr's four, then check_tile_rows.
enum : uint64_t { kStart = 0, kEnd = 1, kDecrease = 2, kFlat = 3, kRow = 4 };
// Gene blocks a key can name (26 bits); the row takes 34 bits (C <= 2^32 - 1).
constexpr uint64_t kMaxGeneBlocks = 1ull << 26;

__host__ __device__ __forceinline__ unsigned long long problem_key(uint64_t g, uint64_t check,
                                                                   uint64_t row, uint64_t sub) {
  return (g << 38) | (check << 35) | (row << 1) | sub;
}

// Where each tile starts among the block's entries, and their end: as a kernel argument for
// up to kStartsInline tiles, else in device memory.
constexpr uint32_t kStartsInline = 64;
struct TileStarts {
  uint64_t v[kStartsInline + 1];
  const uint64_t* more;
  __device__ __forceinline__ uint64_t operator[](uint32_t g) const { return more ? more[g] : v[g]; }
};

constexpr unsigned kTileThreads = 256;

// Past kOneByOne tiles a row's segments are short and a warp takes 32 tiles of a row, a lane a
// tile's offsets, then the segments' entries as one run. (A warp a tile sums every tile's offsets
// for each: 4,096 rows x 512 tiles of 2 entries 1.15 ms and 0.49 for the checks, in runs 75 us and 49; one
// warp for the whole row, its tiles one after another, had taken 0.69 for both. Up to 32 tiles that
// sum is one read a lane, and a warp a tile has the more warps: 39 and 36 us for 32 tiles of 37.)
constexpr uint32_t kOneByOne = 32;

// Segments of up to 32 tiles, a lane a tile: this lane's length and where it starts in the run.
struct SegmentRun {
  uint64_t end, total;  // this lane's segment's end in the run; the run's length
  __device__ __forceinline__ explicit SegmentRun(uint64_t len) : end(len) {
    const unsigned lane = threadIdx.x & 31u;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const uint64_t v = __shfl_up_sync(0xFFFFFFFFu, end, o);
      if (lane >= (unsigned)o) end += v;
    }
    total = __shfl_sync(0xFFFFFFFFu, end, 31);
  }
  // The lane whose segment holds entry x (< total) of the run: the first whose end is past it.
  __device__ __forceinline__ unsigned find(uint64_t x) const {
    unsigned at = 0;
#pragma unroll
    for (unsigned step = 16; step; step /= 2)
      if (__shfl_sync(0xFFFFFFFFu, end, at + step - 1) <= x) at += step;
    return at;
  }
};

// Blocks [0, shard_blocks): a thread per value i of the shard (tile g = i / (C + 1), row r =
// i % (C + 1)). The others: a warp per (tile, row).
template <bool Runs>
__global__ void __launch_bounds__(kTileThreads)
tile_check_kernel(const uint32_t* __restrict__ shard, uint32_t n_gb, uint64_t row_len,
                  uint32_t rows, const __grid_constant__ TileStarts start,
                  const uint32_t* __restrict__ idx, uint64_t gene_block, uint64_t n_genes,
                  uint64_t shard_blocks, unsigned long long* problem) {
  if (blockIdx.x < shard_blocks) {
    const uint64_t i = blockIdx.x * (uint64_t)kTileThreads + threadIdx.x;
    if (i >= (uint64_t)n_gb * row_len) return;
    const uint64_t g = i / row_len, r = i % row_len;
    const uint32_t v = shard[i];
    unsigned long long key = kNoProblem;
    if (r == 0 && v != 0) key = problem_key(g, kStart, 0, 0);
    if (r + 1 == row_len && (uint64_t)v != start[g + 1] - start[g])
      key = min(key, problem_key(g, kEnd, 0, 0));
    if (r + 1 < row_len && shard[i + 1] < v) key = min(key, problem_key(g, kDecrease, r, 0));
    if (r > rows && v != shard[g * row_len + rows]) key = min(key, problem_key(g, kFlat, 0, 0));
    if (key != kNoProblem) atomicMin(problem, key);
    return;
  }
  const unsigned lane = threadIdx.x & 31u;
  const uint64_t warps = (gridDim.x - shard_blocks) * (kTileThreads / 32);
  uint64_t wq = ((blockIdx.x - shard_blocks) * (uint64_t)kTileThreads + threadIdx.x) >> 5;
  if (Runs) {  // a warp per (32 tiles, row)
    for (; wq < (uint64_t)((n_gb + 31) / 32) * rows; wq += warps) {
      const uint32_t g = (uint32_t)(wq / rows) * 32 + lane, r = (uint32_t)(wq % rows);
      uint64_t from = 0, len = 0;
      if (g < n_gb) {
        const uint64_t nnz = start[g + 1] - start[g];
        const uint64_t a = min((uint64_t)shard[g * row_len + r], nnz);
        const uint64_t e = min((uint64_t)shard[g * row_len + r + 1], nnz);
        from = start[g] + a;
        len = e > a ? e - a : 0;
      }
      const SegmentRun run(len);
      for (uint64_t x0 = 0; x0 < run.total; x0 += 32) {
        const uint64_t x = min(x0 + lane, run.total - 1);  // (the last again: the same verdict)
        const unsigned at = run.find(x);
        const uint64_t in = x - (__shfl_sync(0xFFFFFFFFu, run.end, at) - __shfl_sync(0xFFFFFFFFu, len, at));
        const uint32_t* t = idx + __shfl_sync(0xFFFFFFFFu, from, at) + in;
        const uint32_t tile = g - lane + at, v = *t;
        if (v >= min(gene_block, n_genes - tile * gene_block))
          atomicMin(problem, problem_key(tile, kRow, r, 0));
        else if (in && v <= t[-1])
          atomicMin(problem, problem_key(tile, kRow, r, 1));
      }
    }
    return;
  }
  for (; wq < (uint64_t)n_gb * rows; wq += warps) {
    const uint32_t g = (uint32_t)(wq / rows), r = (uint32_t)(wq % rows);
    const uint64_t nnz = start[g + 1] - start[g];
    const uint64_t a = min((uint64_t)shard[g * row_len + r], nnz);
    const uint64_t e = min((uint64_t)shard[g * row_len + r + 1], nnz);
    const uint32_t* t = idx + start[g];
    const uint64_t width = min(gene_block, n_genes - g * gene_block);
    bool wide = false, unsorted = false;
    uint32_t carry = 0;  // the index before the chunk's first
    for (uint64_t x0 = a; x0 < e; x0 += 128) {
      uint32_t v[4];
#pragma unroll
      for (int m = 0; m < 4; ++m) v[m] = x0 + 32 * m + lane < e ? t[x0 + 32 * m + lane] : 0;
#pragma unroll
      for (int m = 0; m < 4; ++m) {
        const uint64_t x = x0 + 32 * m + lane;
        uint32_t before = __shfl_up_sync(0xFFFFFFFFu, v[m], 1);
        if (lane == 0) before = carry;
        carry = __shfl_sync(0xFFFFFFFFu, v[m], 31);
        if (x >= e) continue;
        wide |= v[m] >= width;
        unsorted |= x > a && v[m] <= before;
      }
    }
    const unsigned w = __ballot_sync(0xFFFFFFFFu, wide);
    const unsigned u = __ballot_sync(0xFFFFFFFFu, unsorted);
    if (lane == 0 && (w | u)) atomicMin(problem, problem_key(g, kRow, r, w ? 0 : 1));
  }
}

// A warp per (row, tile) or (row, 32 tiles). Writes nothing when the checks found a problem (the caller's
// outputs stay as they were): every thread reads the verdict, final once the checks ran
// before it on the stream.
template <bool Runs>
__global__ void __launch_bounds__(kTileThreads)
tile_join_kernel(const uint32_t* __restrict__ shard, uint32_t n_gb, uint64_t row_len,
                 uint32_t rows, const __grid_constant__ TileStarts start,
                 const uint32_t* __restrict__ idx, const uint32_t* __restrict__ val,
                 uint64_t gene_block, const unsigned long long* problem, uint64_t* out_ptr,
                 uint32_t* __restrict__ out_idx, uint32_t* __restrict__ out_val) {
  const unsigned lane = threadIdx.x & 31u;
  const uint64_t warps = gridDim.x * (uint64_t)(kTileThreads / 32);
  uint64_t wq = (blockIdx.x * (uint64_t)kTileThreads + threadIdx.x) >> 5;
  if (*problem != kNoProblem) return;
  if (n_gb == 0) {  // a layer without genes: empty rows
    for (; wq <= rows; wq += warps)
      if (lane == 0) out_ptr[wq] = 0;
    return;
  }
  if (Runs) {  // a warp per (32 tiles, row)
    for (; wq < (uint64_t)((n_gb + 31) / 32) * rows; wq += warps) {
      const uint32_t g0 = (uint32_t)(wq / rows) * 32, g = g0 + lane, r = (uint32_t)(wq % rows);
      uint64_t dst = 0, from = 0, len = 0;
      for (uint32_t h = lane; h < n_gb; h += 32) dst += shard[h * row_len + r + (h < g0 ? 1 : 0)];
      for (int o = 16; o; o >>= 1) dst += __shfl_xor_sync(0xFFFFFFFFu, dst, o);
      if (g < n_gb) {
        const uint64_t a = shard[g * row_len + r];
        len = shard[g * row_len + r + 1] - a;
        from = start[g] + a;
      }
      const SegmentRun run(len);
      if (lane == 0) {
        if (g0 + 32 >= n_gb) out_ptr[r + 1] = dst + run.total;
        if (r == 0 && g0 == 0) out_ptr[0] = 0;
      }
      for (uint64_t x0 = 0; x0 < run.total; x0 += 32) {
        const uint64_t x = min(x0 + lane, run.total - 1);
        const unsigned at = run.find(x);
        const uint64_t in = x - (__shfl_sync(0xFFFFFFFFu, run.end, at) - __shfl_sync(0xFFFFFFFFu, len, at));
        const uint64_t src = __shfl_sync(0xFFFFFFFFu, from, at) + in;
        if (x0 + lane >= run.total) continue;
        out_idx[dst + x] = (uint32_t)((g0 + at) * gene_block) + idx[src];
        out_val[dst + x] = val[src];
      }
    }
    return;
  }
  for (; wq < (uint64_t)n_gb * rows; wq += warps) {
    const uint32_t r = (uint32_t)(wq / n_gb), g = (uint32_t)(wq % n_gb);
    uint64_t dst = 0;
    for (uint32_t h = lane; h < n_gb; h += 32) dst += shard[h * row_len + r + (h < g ? 1 : 0)];
    for (int o = 16; o; o >>= 1) dst += __shfl_xor_sync(0xFFFFFFFFu, dst, o);
    const uint64_t a = shard[g * row_len + r], len = shard[g * row_len + r + 1] - a;
    if (lane == 0) {
      if (g + 1 == n_gb) out_ptr[r + 1] = dst + len;
      if (r == 0 && g == 0) out_ptr[0] = 0;
    }
    // g G + local < n_genes <= 2^32 - 1 (the checks passed).
    const uint32_t first_gene = (uint32_t)(g * gene_block);
    const uint32_t* ti = idx + start[g] + a;
    const uint32_t* tv = val + start[g] + a;
    uint32_t* oi = out_idx + dst;
    uint32_t* ov = out_val + dst;
    uint64_t x = lane;
    for (; x + 96 < len; x += 128) {
      const uint32_t i0 = ti[x], i1 = ti[x + 32], i2 = ti[x + 64], i3 = ti[x + 96];
      const uint32_t v0 = tv[x], v1 = tv[x + 32], v2 = tv[x + 64], v3 = tv[x + 96];
      oi[x] = first_gene + i0, oi[x + 32] = first_gene + i1;
      oi[x + 64] = first_gene + i2, oi[x + 96] = first_gene + i3;
      ov[x] = v0, ov[x + 32] = v1, ov[x + 64] = v2, ov[x + 96] = v3;
    }
    for (; x < len; x += 32) {
      oi[x] = first_gene + ti[x];
      ov[x] = tv[x];
    }
  }
}

// Blocks of a warp per (tile, row) or (32 tiles, row), the warps going on from the grid's end past
// 2^25 of them.
unsigned row_blocks_for(uint64_t tiles, uint64_t rows) {
  const uint64_t pairs = (tiles > kOneByOne ? (tiles + 31) / 32 : std::max<uint64_t>(tiles, 1)) * rows;
  return (unsigned)std::min<uint64_t>((pairs + kTileThreads / 32 - 1) / (kTileThreads / 32), 1u << 22);
}

template <class T>
T read_one(const T* p, cudaStream_t s) {
  T v{};
  KG_CUDA(cudaMemcpyAsync(&v, p, sizeof(T), cudaMemcpyDefault, s));
  KG_CUDA(cudaStreamSynchronize(s));
  return v;
}

}  // namespace

TileShape tile_shape(const kg_tile_block* tb, cudaStream_t s) {
  if (!tb || !tb->indptr || !tb->tile_offsets) fail(KG_ERR_INVALID, "tiles: NULL argument");
  if (tb->dtype != KG_U32 && tb->dtype != KG_F32) fail(KG_ERR_INVALID, "tiles: unknown dtype");
  const uint64_t c = tb->cell_block_size, gs = tb->gene_block_size;
  if (c == 0 || gs == 0) fail(KG_ERR_INVALID, "tiles: a tile size is 0");
  if (tb->rows == 0 || tb->rows > c || tb->rows > 0x7FFFFFFFu)
    fail(KG_ERR_INVALID, "tiles: rows must be 1..cell_block_size (" + std::to_string(tb->rows) +
                             " rows, cell_block_size " + std::to_string(c) + ")");
  if (tb->n_genes > 0xFFFFFFFFull) fail(KG_ERR_INVALID, "tiles: n_genes above 2^32 - 1");
  if ((unsigned __int128)c * gs > 0xFFFFFFFFull)
    fail(KG_ERR_INVALID, "tiles: cell_block_size * gene_block_size above 2^32 - 1");
  const uint64_t n_gb = (tb->n_genes + gs - 1) / gs;
  if (n_gb >= kMaxGeneBlocks) fail(KG_ERR_INVALID, "tiles: more than 2^26 gene blocks");
  TileShape sh;
  sh.n_gene_blocks = (uint32_t)n_gb;
  sh.start.resize(n_gb + 1);
  if (is_device_pointer(tb->tile_offsets)) {
    KG_CUDA(cudaMemcpyAsync(sh.start.data(), tb->tile_offsets, (n_gb + 1) * 8,
                            cudaMemcpyDeviceToHost, s));
    KG_CUDA(cudaStreamSynchronize(s));
  } else {
    std::memcpy(sh.start.data(), tb->tile_offsets, (n_gb + 1) * 8);
  }
  // check_tile_offsets (tile_decode.rs:29-66) over the block's slice.
  for (uint64_t g = 0; g < n_gb; ++g)
    if (sh.start[g + 1] < sh.start[g])
      fail(KG_ERR_CORRUPT, "the layer is corrupt: tile_offsets decreases after tile " +
                               std::to_string(tb->block * n_gb + g));
  sh.first = sh.start[0];
  for (auto& v : sh.start) v -= sh.first;
  sh.nnz = sh.start[n_gb];
  if (sh.nnz && (!tb->indices || !tb->data)) fail(KG_ERR_INVALID, "tiles: NULL entries");
  return sh;
}

void join_tiles(kg_ctx* ctx, cudaStream_t s, const kg_tile_block* tb, const TileShape& sh,
                uint64_t* d_indptr, uint32_t* d_indices, uint32_t* d_values) {
  const uint32_t n_gb = sh.n_gene_blocks, rows = tb->rows;
  const uint64_t row_len = (uint64_t)tb->cell_block_size + 1;
  DeviceBuffer<uint32_t> hs, hi, hv;
  const uint32_t* shard = device_view(tb->indptr, (size_t)n_gb * row_len, hs, s);
  const uint32_t* idx = device_view(tb->indices, sh.nnz, hi, s);
  const uint32_t* val = device_view(static_cast<const uint32_t*>(tb->data), sh.nnz, hv, s);
  TileStarts start{};
  DeviceBuffer<uint64_t> more;
  if (n_gb <= kStartsInline) {
    std::copy(sh.start.begin(), sh.start.end(), start.v);
  } else {
    more.alloc(n_gb + 1, s);
    KG_CUDA(cudaMemcpyAsync(more.ptr, sh.start.data(), (n_gb + 1) * 8ull, cudaMemcpyHostToDevice, s));
    start.more = more.ptr;
  }
  DeviceBuffer<unsigned long long> problem(1, s);
  KG_CUDA(cudaMemsetAsync(problem.ptr, 0xFF, 8, s));
  const bool runs = n_gb > kOneByOne;
  const unsigned row_blocks = row_blocks_for(n_gb, rows);
  if (n_gb) {
    const uint64_t shard_blocks = blocks_for((uint64_t)n_gb * row_len, kTileThreads);
    (runs ? tile_check_kernel<true> : tile_check_kernel<false>)
        <<<(unsigned)(shard_blocks + row_blocks), kTileThreads, 0, s>>>(
            shard, n_gb, row_len, rows, start, idx, tb->gene_block_size, tb->n_genes, shard_blocks,
            problem.ptr);
    KG_LAUNCH_CHECK();
  }
  // The join is queued before the verdict is read (one wait a call); it writes only when the
  // checks passed.
  (runs ? tile_join_kernel<true> : tile_join_kernel<false>)<<<row_blocks, kTileThreads, 0, s>>>(
      shard, n_gb, row_len, rows, start, idx, val, tb->gene_block_size, problem.ptr, d_indptr,
      d_indices, d_values);
  KG_LAUNCH_CHECK();
  unsigned long long key = kNoProblem;
  KG_CUDA(cudaMemcpyAsync(&key, problem.ptr, 8, cudaMemcpyDeviceToHost, s));
  wait_stream(ctx, s);
  if (key == kNoProblem) return;
  // kyto's wording (tile_decode.rs:129-196), the details read back from the inputs.
  const uint64_t g = key >> 38, check = (key >> 35) & 7u, r = (key >> 1) & ((1ull << 34) - 1);
  std::string what;
  if (check == kStart) {
    what = "indptr does not start at 0";
  } else if (check == kEnd) {
    const uint32_t end = read_one(shard + g * row_len + row_len - 1, s);
    what = "indptr ends at Some(" + std::to_string(end) + ") but tile_offsets gives " +
           std::to_string(sh.start[g + 1] - sh.start[g]) + " entries";
  } else if (check == kDecrease) {
    what = "indptr decreases after row " + std::to_string(r);
  } else if (check == kFlat) {
    what = "indptr is not flat after the last row " + std::to_string(rows);
  } else if (key & 1u) {
    what = "row " + std::to_string(r) + ": gene indices are not strictly increasing";
  } else {
    const uint64_t width = std::min(tb->gene_block_size, tb->n_genes - g * tb->gene_block_size);
    const uint32_t a = read_one(shard + g * row_len + r, s);
    const uint32_t e = read_one(shard + g * row_len + r + 1, s);
    std::vector<uint32_t> row(e - a);
    if (e > a) {
      KG_CUDA(cudaMemcpyAsync(row.data(), idx + sh.start[g] + a, (e - a) * 4ull,
                              cudaMemcpyDeviceToHost, s));
      KG_CUDA(cudaStreamSynchronize(s));
    }
    uint32_t local = 0;
    for (uint32_t v : row)
      if (v >= width) {
        local = v;
        break;
      }
    what = "row " + std::to_string(r) + ": local gene index " + std::to_string(local) +
           " is not below the block width " + std::to_string(width);
  }
  fail(KG_ERR_CORRUPT, "the layer is corrupt: tile (" + std::to_string(tb->block) + ", " +
                           std::to_string(g) + "): " + what);
}

}  // namespace kg

using namespace kg;

extern "C" {

kg_status kg_tiles_to_csr(kg_ctx* ctx, const kg_tile_block* block, uint64_t* indptr,
                          uint32_t* indices, void* values) {
  return guarded([&] {
    if (!ctx || !block || !indptr) fail(KG_ERR_INVALID, "kg_tiles_to_csr: NULL argument");
    use_device(ctx);
    cudaStream_t s = ctx->stream;
    const TileShape sh = tile_shape(block, s);
    if (sh.nnz && (!indices || !values)) fail(KG_ERR_INVALID, "kg_tiles_to_csr: NULL output");
    const uint64_t rows = block->rows;
    DeviceBuffer<uint64_t> op;
    DeviceBuffer<uint32_t> oi, ov;
    const bool dp = is_device_pointer(indptr), di = is_device_pointer(indices),
               dv = is_device_pointer(values);
    if (!dp) op.alloc(rows + 1, s);
    if (!di) oi.alloc(sh.nnz, s);
    if (!dv) ov.alloc(sh.nnz, s);
    uint64_t* d_ptr = dp ? indptr : op.ptr;
    uint32_t* d_idx = di ? indices : oi.ptr;
    uint32_t* d_val = dv ? static_cast<uint32_t*>(values) : ov.ptr;
    join_tiles(ctx, s, block, sh, d_ptr, d_idx, d_val);
    if (dp && di && dv) return;  // join_tiles waited for the join
    if (!dp) KG_CUDA(cudaMemcpyAsync(indptr, d_ptr, (rows + 1) * 8, cudaMemcpyDeviceToHost, s));
    if (!di && sh.nnz)
      KG_CUDA(cudaMemcpyAsync(indices, d_idx, sh.nnz * 4, cudaMemcpyDeviceToHost, s));
    if (!dv && sh.nnz)
      KG_CUDA(cudaMemcpyAsync(values, d_val, sh.nnz * 4, cudaMemcpyDeviceToHost, s));
    wait_stream(ctx, s);
  });
}

}  // extern "C"
