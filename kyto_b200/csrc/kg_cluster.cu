// k-means on the device (kg_cluster.cuh). Every sum runs in a fixed order; ties go to
// the lower index: the same clusters on every run.
#include "kg_cluster.cuh"

#include <cub/device/device_radix_sort.cuh>

#include <algorithm>
#include <cmath>

namespace kg {

namespace {

constexpr int kNcRows = 128;  // rows per nearest-centre block
constexpr int kNcChunk = 64;  // centres per shared-memory chunk

struct NcShared {
  float x[kClusterDim][kNcRows + 4];   // 16-byte aligned runs of rows
  float c[kClusterDim][kNcChunk + 4];  // and of centres
  float cb[kNcChunk];
};

// 256 threads: thread (ty, tx) holds rows ty*8.. and centres tx*4.. of each chunk: three
// 16-byte shared-memory reads for 32 multiply-adds a component (four by four with 4-byte
// reads: eight for 16, bound by shared memory at half the rate). Every dot product runs over
// the components in order.
__global__ void __launch_bounds__(256)
nearest_centres_kernel(const float* __restrict__ x, uint64_t n, uint32_t width, uint32_t d,
                       const float* __restrict__ centres, const float* __restrict__ cn,
                       uint32_t K, uint32_t* labels) {
  extern __shared__ __align__(16) unsigned char nc_smem[];
  NcShared& sh = *reinterpret_cast<NcShared*>(nc_smem);
  const uint32_t tx = threadIdx.x & 15u, ty = threadIdx.x >> 4;
  const uint64_t r0 = blockIdx.x * (uint64_t)kNcRows;
  for (uint32_t e = threadIdx.x; e < d * kNcRows; e += 256) {
    const uint32_t j = e / kNcRows, rr = e % kNcRows;  // a lane a row: no bank conflicts
    sh.x[j][rr] = r0 + rr < n ? x[(r0 + rr) * width + j] : 0.0f;
  }
  float best[8];
  uint32_t arg[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    best[i] = INFINITY;
    arg[i] = 0xFFFFFFFFu;
  }
  for (uint32_t c0 = 0; c0 < K; c0 += kNcChunk) {
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < (d + 3) / 4 * kNcChunk; e += 256) {
      const uint32_t cc = e % kNcChunk, j = e / kNcChunk * 4;
      const float4 v = c0 + cc < K ? *reinterpret_cast<const float4*>(
                                         centres + (uint64_t)(c0 + cc) * kClusterDim + j)
                                   : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      sh.c[j][cc] = v.x, sh.c[j + 1][cc] = v.y, sh.c[j + 2][cc] = v.z, sh.c[j + 3][cc] = v.w;
    }
    if (threadIdx.x < kNcChunk) {
      const uint32_t c = c0 + threadIdx.x;
      sh.cb[threadIdx.x] = c < K ? cn[c] : INFINITY;
    }
    __syncthreads();
    float dot[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) dot[i][j] = 0.0f;
#pragma unroll 2
    for (uint32_t j = 0; j < d; ++j) {
      float a[8], b[4];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&sh.x[j][ty * 8]);
      *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&sh.x[j][ty * 8 + 4]);
      *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(&sh.c[j][tx * 4]);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) dot[i][jj] = fmaf(a[i], b[jj], dot[i][jj]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const uint32_t c = c0 + tx * 4 + jj;
        const float dist = sh.cb[tx * 4 + jj] - 2.0f * dot[i][jj];
        if (c < K && (dist < best[i] || (dist == best[i] && c < arg[i]))) {
          best[i] = dist;
          arg[i] = c;
        }
      }
  }
  // The 16 threads of a row group (lanes sharing ty) combine.
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float bv = best[i];
    uint32_t ba = arg[i];
    for (int o = 8; o; o >>= 1) {
      const float ov = __shfl_xor_sync(0xFFFFFFFFu, bv, o);
      const uint32_t oa = __shfl_xor_sync(0xFFFFFFFFu, ba, o);
      if (ov < bv || (ov == bv && oa < ba)) {
        bv = ov;
        ba = oa;
      }
    }
    const uint64_t row = r0 + ty * 8 + i;
    if (tx == 0 && row < n) labels[row] = ba;
  }
}

__global__ void gather_rows_kernel(const float* x, uint64_t n, uint32_t width, uint32_t d,
                                   uint64_t m, float* out) {
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= m * d) return;
  const uint64_t r = i / d, j = i % d;
  const uint64_t row = r * n / m;  // evenly strided
  out[r * d + j] = x[row * width + j];
}

// centre[c] = row (c * m / K) of the sample (d columns, padded with zeros).
__global__ void seed_centres_kernel(const float* sample, uint64_t m, uint32_t d, uint32_t K,
                                    double* centre) {
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= (uint64_t)K * kClusterDim) return;
  const uint64_t c = i / kClusterDim, j = i % kClusterDim;
  centre[i] = j < d ? (double)sample[(c * m / K) * d + j] : 0.0;
}

// A centre's f32 components and their squared norm (summed in order by one lane; the components
// are read by kClusterDim lanes, since a lane reading them all waits 13 us).
constexpr uint32_t kCentresABlock = 4;

__global__ void __launch_bounds__(kCentresABlock * kClusterDim)
centres_f32_kernel(const double* centre, uint32_t K, float* cf, float* cn) {
  __shared__ float v[kCentresABlock][kClusterDim];
  const uint32_t i = threadIdx.x / kClusterDim, j = threadIdx.x % kClusterDim;
  const uint32_t c = blockIdx.x * kCentresABlock + i;
  if (c < K) {
    v[i][j] = (float)centre[(uint64_t)c * kClusterDim + j];
    cf[(uint64_t)c * kClusterDim + j] = v[i][j];
  }
  __syncthreads();
  if (c < K && j == 0) {
    float s = 0.0f;
    for (uint32_t k = 0; k < kClusterDim; ++k) s = fmaf(v[i][k], v[i][k], s);
    cn[c] = s;
  }
}

// key = (label << 32) | the first component's f32 bits mapped to an unsigned order.
__global__ void order_key_kernel(const float* x, uint64_t n, uint32_t width, const uint32_t* label,
                                 unsigned long long* key, uint32_t* iota) {
  uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (r >= n) return;
  uint32_t b = __float_as_uint(x[r * width]);
  b = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  key[r] = ((unsigned long long)label[r] << 32) | b;
  iota[r] = (uint32_t)r;
}

// key = the first component's f32 bits mapped to an unsigned order.
__global__ void component_key_kernel(const float* x, uint64_t n, uint32_t width, uint32_t* key,
                                     uint32_t* iota) {
  uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (r >= n) return;
  uint32_t b = __float_as_uint(x[r * width]);
  key[r] = (b & 0x80000000u) ? ~b : (b | 0x80000000u);
  iota[r] = (uint32_t)r;
}

// out row i = row order[i] of x (d components each).
__global__ void permute_rows_kernel(const float* x, uint64_t n, uint32_t d, const uint32_t* order,
                                    float* out) {
  uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n * d) return;
  out[i] = x[(uint64_t)order[i / d] * d + i % d];
}

__device__ __forceinline__ uint32_t label_of(unsigned long long key) { return (uint32_t)(key >> 32); }
__device__ __forceinline__ uint32_t label_of(uint32_t label) { return label; }

// starts[c] = the first position whose key's label is >= c (c = 0..K).
template <class Key>
__global__ void key_starts_kernel(const Key* sorted, uint64_t n, uint32_t K, uint32_t* starts) {
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c > K) return;
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (label_of(sorted[mid]) < c) lo = mid + 1; else hi = mid;
  }
  starts[c] = (uint32_t)lo;
}

// centre[c] = the mean (f64, members in slot order) of cluster c's rows; an empty
// cluster keeps its centre. One block per cluster: thread j < d adds component j over a tile
// of kUcRows members in shared memory while every thread has the next tile's loads (and the
// members after it) on their way, so the chain of additions (8.5 cycles each) sets the pace.
// A thread a component gathering row after row took 340 us a pass for clusters of 1,000 to
// 8,000 rows, one dependent pair of loads behind every few additions; now 51 us.
constexpr uint32_t kUcRows = 128;
constexpr uint32_t kUcThreads = 256;
constexpr uint32_t kUcRowsAWarp = kUcRows / (kUcThreads / 32);

__global__ void __launch_bounds__(kUcThreads)
update_centres_kernel(const float* __restrict__ x, uint32_t width, uint32_t d,
                      const uint32_t* __restrict__ order, const uint32_t* __restrict__ starts,
                      double* centre, double* partial) {
  __shared__ float tile[kUcRows][kClusterDim];
  __shared__ uint32_t member[2][kUcRows];
  const uint32_t c = blockIdx.x, tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  uint32_t b = starts[c], e = starts[c + 1];
  if (b == e) return;
  if (gridDim.y > 1) {  // this part's share of the members
    const uint64_t members = e - b;
    const uint32_t first = b;
    b = first + (uint32_t)(members * blockIdx.y / gridDim.y);
    e = first + (uint32_t)(members * (blockIdx.y + 1) / gridDim.y);
  }
  float v[kUcRowsAWarp][2];
  auto load = [&](uint32_t i0, const uint32_t* rows) {
#pragma unroll
    for (uint32_t u = 0; u < kUcRowsAWarp; ++u) {
      const uint32_t r = warp + u * (kUcThreads / 32);
      const float* xr = x + (uint64_t)rows[r] * width;
      v[u][0] = i0 + r < e && lane < d ? xr[lane] : 0.0f;
      v[u][1] = i0 + r < e && lane + 32 < d ? xr[lane + 32] : 0.0f;
    }
  };
  auto next_member = [&](uint32_t i0) { return tid < kUcRows && i0 + tid < e ? order[i0 + tid] : 0u; };
  if (tid < kUcRows) {
    member[0][tid] = next_member(b);
    member[1][tid] = next_member(b + kUcRows);
  }
  __syncthreads();
  load(b, member[0]);
  double s = 0.0;
  uint32_t half = 0;  // member[half]: the tile in v
  for (uint32_t i0 = b; i0 < e; i0 += kUcRows, half ^= 1) {
#pragma unroll
    for (uint32_t u = 0; u < kUcRowsAWarp; ++u) {
      tile[warp + u * (kUcThreads / 32)][lane] = v[u][0];
      tile[warp + u * (kUcThreads / 32)][lane + 32] = v[u][1];
    }
    __syncthreads();
    if (i0 + kUcRows < e) load(i0 + kUcRows, member[half ^ 1]);
    const uint32_t after = next_member(i0 + 2 * kUcRows);
    if (tid < d) {
      const uint32_t n = min(kUcRows, e - i0);
      if (n == kUcRows) {
#pragma unroll 16
        for (uint32_t r = 0; r < kUcRows; ++r) s += (double)tile[r][tid];
      } else {
        for (uint32_t r = 0; r < n; ++r) s += (double)tile[r][tid];
      }
    }
    __syncthreads();
    if (tid < kUcRows) member[half][tid] = after;
  }
  if (tid >= d) return;
  if (gridDim.y > 1)
    partial[((uint64_t)c * gridDim.y + blockIdx.y) * kClusterDim + tid] = s;
  else
    centre[(uint64_t)c * kClusterDim + tid] = s / (double)(e - b);
}

// centre[c] from its parts' sums, in order.
__global__ void __launch_bounds__(kClusterDim)
join_centres_kernel(const double* partial, uint32_t parts, const uint32_t* starts, uint32_t d,
                    double* centre) {
  const uint32_t c = blockIdx.x, j = threadIdx.x;
  const uint32_t members = starts[c + 1] - starts[c];
  if (j >= d || !members) return;
  double s = 0.0;
  for (uint32_t p = 0; p < parts; ++p) s += partial[((uint64_t)c * parts + p) * kClusterDim + j];
  centre[(uint64_t)c * kClusterDim + j] = s / (double)members;
}

// The centres of the clusters' rows. A large cluster's chain of additions is what a call waits
// for (8,000 rows: 36 us), so unless the sums are to be in slot order throughout (`ordered`) a
// cluster is cut into up to 16 parts while there are fewer than four an SM: 50 us a round of
// 58 clusters of 60,000 rows, in parts 11 and 5 to join them.
void update_centres(const float* x, uint32_t width, uint32_t d, const uint32_t* order,
                    const uint32_t* starts, uint32_t K, bool ordered, int sm_count, double* centre,
                    cudaStream_t s) {
  const uint32_t parts = ordered ? 1 : std::min(16u, std::max(1u, 4u * (uint32_t)sm_count / K));
  DeviceBuffer<double> partial(parts > 1 ? (uint64_t)K * parts * kClusterDim : 0, s);
  update_centres_kernel<<<dim3(K, parts), kUcThreads, 0, s>>>(x, width, d, order, starts, centre,
                                                              partial.ptr);
  KG_LAUNCH_CHECK();
  if (parts > 1) {
    join_centres_kernel<<<K, kClusterDim, 0, s>>>(partial.ptr, parts, starts, d, centre);
    KG_LAUNCH_CHECK();
  }
}

// Sorts (key, value) pairs by the key's low `bits` (stable).
template <class Key>
void sort_pairs(const Key* key, Key* key_out, const uint32_t* val, uint32_t* val_out, uint64_t n,
                int bits, cudaStream_t s) {
  size_t temp = 0;
  KG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, temp, key, key_out, val, val_out, (int)n, 0, bits,
                                          s));
  DeviceBuffer<unsigned char> scratch(temp, s);
  KG_CUDA(cub::DeviceRadixSort::SortPairs(scratch.ptr, temp, key, key_out, val, val_out, (int)n, 0,
                                          bits, s));
}

int label_bits(uint32_t K) {
  int bits = 1;
  while (bits < 32 && (1ull << bits) <= (uint64_t)K) ++bits;
  return bits;
}

// The rows by (cluster, first component): perm and the clusters' starts.
void order_by_cluster(const float* x, uint64_t n, uint32_t width, const uint32_t* label,
                      uint32_t K, DeviceBuffer<uint32_t>& perm, DeviceBuffer<uint32_t>& start,
                      cudaStream_t s) {
  DeviceBuffer<unsigned long long> key(n, s), key_sorted(n, s);
  DeviceBuffer<uint32_t> iota(n, s);
  order_key_kernel<<<blocks_for(n, 256), 256, 0, s>>>(x, n, width, label, key.ptr, iota.ptr);
  KG_LAUNCH_CHECK();
  perm.alloc(n, s);
  sort_pairs(key.ptr, key_sorted.ptr, iota.ptr, perm.ptr, n, 32 + label_bits(K), s);
  start.alloc((uint64_t)K + 1, s);
  key_starts_kernel<<<blocks_for((uint64_t)K + 1, 256), 256, 0, s>>>(key_sorted.ptr, n, K,
                                                                    start.ptr);
  KG_LAUNCH_CHECK();
}

}  // namespace

void nearest_centres(const float* x, uint64_t n, uint32_t width, uint32_t d,
                     const float* centres, const float* cn, uint32_t K, uint32_t* labels,
                     cudaStream_t s) {
  if (!n) return;
  if (d > kClusterDim) fail(KG_ERR_INVALID, "clusters: more than 64 components");
  allow_dynamic_smem(nearest_centres_kernel, sizeof(NcShared));
  nearest_centres_kernel<<<(unsigned)((n + kNcRows - 1) / kNcRows), 256, sizeof(NcShared), s>>>(
      x, n, width, d, centres, cn, K, labels);
  KG_LAUNCH_CHECK();
}

void cluster_rows(const float* x, uint64_t n, uint32_t width, uint32_t d, uint32_t K,
                  uint32_t iters, uint64_t sample, bool ordered, int sm_count, Clusters& out,
                  cudaStream_t s) {
  if (d > kClusterDim) fail(KG_ERR_INVALID, "clusters: more than 64 components");
  K = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(K, n));
  out.K = K;
  const uint64_t m = std::max<uint64_t>(std::min<uint64_t>(sample, n), K);
  DeviceBuffer<float> xs(m * d, s), cf((uint64_t)K * kClusterDim, s), cn(K, s);
  gather_rows_kernel<<<blocks_for(m * d, 256), 256, 0, s>>>(x, n, width, d, m, xs.ptr);
  KG_LAUNCH_CHECK();
  out.centre.alloc((uint64_t)K * kClusterDim, s);
  seed_centres_kernel<<<blocks_for((uint64_t)K * kClusterDim, 256), 256, 0, s>>>(
      xs.ptr, m, d, K, out.centre.ptr);
  KG_LAUNCH_CHECK();
  // The sample by its first component, once: a round then sorts by the cluster alone, one or two
  // passes that keep each cluster's rows in that order (by both, five passes a round, 45 us).
  DeviceBuffer<uint32_t> key(m, s), key_sorted(m, s), iota(m, s), order(m, s), starts(K + 1ull, s);
  DeviceBuffer<float> sorted(m * d, s);
  component_key_kernel<<<blocks_for(m, 256), 256, 0, s>>>(xs.ptr, m, d, key.ptr, iota.ptr);
  KG_LAUNCH_CHECK();
  sort_pairs(key.ptr, key_sorted.ptr, iota.ptr, order.ptr, m, 32, s);
  permute_rows_kernel<<<blocks_for(m * d, 256), 256, 0, s>>>(xs.ptr, m, d, order.ptr, sorted.ptr);
  KG_LAUNCH_CHECK();
  for (uint32_t it = 0; it < iters; ++it) {
    centres_f32_kernel<<<(K + kCentresABlock - 1) / kCentresABlock, kCentresABlock * kClusterDim, 0,
                       s>>>(out.centre.ptr, K, cf.ptr, cn.ptr);
    KG_LAUNCH_CHECK();
    nearest_centres(sorted.ptr, m, d, d, cf.ptr, cn.ptr, K, key.ptr, s);
    sort_pairs(key.ptr, key_sorted.ptr, iota.ptr, order.ptr, m, label_bits(K), s);
    key_starts_kernel<<<blocks_for((uint64_t)K + 1, 256), 256, 0, s>>>(key_sorted.ptr, m, K,
                                                                       starts.ptr);
    KG_LAUNCH_CHECK();
    update_centres(sorted.ptr, d, d, order.ptr, starts.ptr, K, ordered, sm_count, out.centre.ptr, s);
  }
  centres_f32_kernel<<<(K + kCentresABlock - 1) / kCentresABlock, kCentresABlock * kClusterDim, 0,
                       s>>>(out.centre.ptr, K, cf.ptr, cn.ptr);
  KG_LAUNCH_CHECK();
  out.label.alloc(n, s);
  nearest_centres(x, n, width, d, cf.ptr, cn.ptr, K, out.label.ptr, s);
  order_by_cluster(x, n, width, out.label.ptr, K, out.perm, out.start, s);
  update_centres(x, width, d, out.perm.ptr, out.start.ptr, K, ordered, sm_count, out.centre.ptr, s);
}

}  // namespace kg
