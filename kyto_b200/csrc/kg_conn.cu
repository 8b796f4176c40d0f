// UMAP connectivities of a kNN graph on the device: kyto's `connectivities`
// (crates/kyto-exec/src/connectivities.rs:84-131, scanpy's pp.neighbors(method="umap")
// weights). One thread per row ranks the row's distances in shared memory and bisects its
// sigma; the row's entries are weighed in f32; the fuzzy union w + w^T - w o w^T pairs each
// row's own entries with the transposed ones (a radix sort of the columns), a warp a row,
// and a last pass closes the rows up, columns increasing, no stored zeros. The f32
// arithmetic is IEEE without contraction (explicit _rn intrinsics), the sums run in kyto's
// order, and the one f32 exponential is evaluated in f64 and rounded once. The host waits
// once, for the verdict on the graph and the entry count.
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include <cfloat>
#include <cmath>
#include <vector>

#include "kg_internal.cuh"

namespace kg {

namespace {

constexpr int kConnIterations = 64;        // SMOOTH_K_ITERATIONS (connectivities.rs:26)
constexpr double kConnTolerance = 1e-5;    // SMOOTH_K_TOLERANCE (:28)
constexpr double kMinKDistScale = 1e-3;    // MIN_K_DIST_SCALE (:30)
constexpr uint32_t kConnMaxK = 255;        // stored neighbours a row, at most

// f32 bits as an int in IEEE total order (Rust's f32::total_cmp).
__device__ __forceinline__ int32_t total_order(float v) {
  const int32_t b = __float_as_int(v);
  return b ^ (int32_t)((uint32_t)(b >> 31) >> 1);
}

// exp2(x), f32, about 2^-22 relative.
__device__ __forceinline__ float exp2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The rows' checks, sigmas and memberships, a CTA's blockDim.x rows at a time (their entries
// are one run). Sets *bad on a violation of the graph's shape: 1 when row r does not hold
// entries [r k, (r + 1) k), 2 when its columns do not increase strictly below n. A CTA reads its
// rows' entries only after all its rows' indptr has passed (a graph of another k may hold fewer),
// and the kernels after this one return on *bad: what a CTA left out is not written, and a column
// out of range would take a merge past its rows.
//
// A thread a row (connectivities.rs:90-104, 133-176): the distances ranked by (distance,
// column), a stable insertion sort in shared memory (equal distances keep the input order,
// which is the order of their increasing columns); rho = the first ranked distance above 0;
// sigma by the 64-step bisection on sum_j [d_j > 0 ? exp(-(d_j / mid)) : 1] = target (d_j =
// f32(ranked_j - rho) widened), floored at 1e-3 of the row's mean (a sequential f32 sum over
// n_neighbors) when rho > 0. (Rows with rho == 0 have kyto's floor from the mean of every
// distance; none of their distances exceeds rho, so their memberships are 1 whatever sigma
// is, and it is left out.)
// A step needs the sum's side of the target and whether it is within 1e-5: an f32 sum tells
// both unless it comes within `margin` of the target (its error bound and the tolerance),
// and only then are the f64 exponentials taken: 4 or 5 of about 20 steps. With f64
// exponentials in every step FP64 bounded the kernel (200,000 rows of 14: 224 us; this form
// with the memberships, 130 us).
//
// Then an entry a thread (connectivities.rs:189-198): its membership, and (column, entry)
// for the transpose.
__global__ void graph_rows_kernel(const uint64_t* indptr, const uint32_t* __restrict__ indices,
                                  const float* __restrict__ distances, uint64_t n, uint32_t k,
                                  uint32_t n_neighbors, double target, float* __restrict__ w,
                                  uint32_t* __restrict__ tcol, uint32_t* __restrict__ tentry,
                                  int* bad) {
  extern __shared__ float conn_smem[];
  const uint32_t ld = k | 1u;  // odd: a step of every thread's row is free of bank conflicts
  float* sorted = conn_smem;
  float* sigma_s = conn_smem + blockDim.x * ld;
  float* rho_s = sigma_s + blockDim.x;
  const uint64_t r0 = blockIdx.x * (uint64_t)blockDim.x;
  const uint32_t rows = (uint32_t)min((uint64_t)blockDim.x, n - r0);
  const uint32_t entries = rows * k;
  const uint64_t e0 = r0 * k;
  const uint64_t r = r0 + threadIdx.x;
  if (__syncthreads_or(threadIdx.x < rows && (indptr[r] != r * k || indptr[r + 1] != (r + 1) * k))) {
    if (threadIdx.x == 0) atomicExch(bad, 1);
    return;
  }
  for (uint32_t x = threadIdx.x; x < entries; x += blockDim.x)
    sorted[(x / k) * ld + x % k] = distances[e0 + x];
  __syncthreads();
  if (threadIdx.x < rows) {
    float* row = sorted + threadIdx.x * ld;
    for (uint32_t j = 1; j < k; ++j) {
      const float v = row[j];
      const int32_t kv = total_order(v);
      uint32_t at = j;
      while (at > 0 && total_order(row[at - 1]) > kv) {
        row[at] = row[at - 1];
        --at;
      }
      row[at] = v;
    }
    float rho = 0.0f;
    for (uint32_t j = 0; j < k; ++j)
      if (row[j] > 0.0f) {
        rho = row[j];
        break;
      }
    // |f32 sum - exact sum| <= k (the terms' approximations, under 1e-6 each) + k^2 2^-24
    // (the additions), doubled.
    const double margin = kConnTolerance + 2e-6 * k + 1.2e-7 * (double)k * k;
    const double ceiling = (double)FLT_MAX;
    double lo = 0.0, hi = ceiling, mid = 1.0;
    auto step = [&](double sum) {
      if (sum > target) {
        hi = mid;
        mid = __dmul_rn(__dadd_rn(lo, hi), 0.5);
      } else {
        lo = mid;
        mid = hi >= ceiling ? __dmul_rn(mid, 2.0) : __dmul_rn(__dadd_rn(lo, hi), 0.5);
      }
    };
    // Each row takes f32 steps until one is too close to tell; the warp's rows then take
    // their f64 step together.
    int it = 0;
    const unsigned active = __activemask();
    bool done = false;
    while (__any_sync(active, !done)) {
      while (!done && it < kConnIterations) {
        const float scale = -1.44269504f / (float)mid;
        float est = 0.0f;
        for (uint32_t j = 0; j < k; ++j) {
          const float d = __fsub_rn(row[j], rho);
          est += d > 0.0f ? exp2_approx(d * scale) : 1.0f;
        }
        if (!(fabs((double)est - target) > margin)) break;
        step((double)est);
        ++it;
      }
      __syncwarp(active);
      if (it >= kConnIterations) done = true;
      if (!done) {
        double sum = 0.0;
        for (uint32_t j = 0; j < k; ++j) {
          const double dj = (double)__fsub_rn(row[j], rho);
          sum = __dadd_rn(sum, dj > 0.0 ? exp(-__ddiv_rn(dj, mid)) : 1.0);
        }
        done = fabs(sum - target) < kConnTolerance;
        if (!done) step(sum);
        ++it;
      }
      __syncwarp(active);
    }
    float sigma = __double2float_rn(mid);
    if (rho > 0.0f) {
      float s = 0.0f;
      for (uint32_t j = 0; j < k; ++j) s = __fadd_rn(s, row[j]);
      const double floor_v = kMinKDistScale * ((double)s / (double)n_neighbors);
      if ((double)sigma < floor_v) sigma = __double2float_rn(floor_v);
    }
    sigma_s[threadIdx.x] = sigma;
    rho_s[threadIdx.x] = rho;
  }
  __syncthreads();
  for (uint32_t x = threadIdx.x; x < entries; x += blockDim.x) {
    const uint64_t e = e0 + x;
    const uint32_t lr = x / k, c = indices[e];
    if (c >= n || (x % k > 0 && c <= indices[e - 1])) atomicExch(bad, 2);
    const float s = sigma_s[lr], t = __fsub_rn(distances[e], rho_s[lr]);
    float v;
    if (c == r0 + lr)
      v = 0.0f;
    else if (t <= 0.0f || s == 0.0f)
      v = 1.0f;
    else
      v = __double2float_rn(exp(-(double)__fdiv_rn(t, s)));
    w[e] = v;
    tcol[e] = c < n ? c : (uint32_t)(n - 1);
    tentry[e] = (uint32_t)e;
  }
}

// tstart[c] = the first sorted transposed entry of column (= transposed row) c.
__global__ void transposed_starts_kernel(const uint32_t* __restrict__ sorted, uint64_t m,
                                         uint64_t n, uint32_t* tstart) {
  const uint64_t c = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (c > n) return;
  uint64_t lo = 0, hi = m;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (sorted[mid] < c) lo = mid + 1; else hi = mid;
  }
  tstart[c] = (uint32_t)lo;
}

__device__ __forceinline__ float union_weight(float wf, float wt) {
  return __fsub_rn(__fadd_rn(wf, wt), __fmul_rn(wf, wt));
}

// The union of row r (connectivities.rs:221-255): its own entries (increasing columns) and
// its transposed ones (the entries naming it, in increasing order of their rows); weight (w +
// wT) - w wT in f32, zeros dropped. Row r's entries go to place r k + tstart[r] on (the rows
// before it have at most that many), its count to counts[r].
// k <= 32: a warp a row, a lane one of its own entries; the transposed ones pass 32 at a
// time, first to meet the own entries, then to be placed between them (200,000 rows of 14:
// 106 us and 35 us to close them up; a thread a row merging twice, to count and to write,
// 137 us and two copies).
__global__ void union_rows_kernel(const uint32_t* __restrict__ indices,
                                  const float* __restrict__ w, uint64_t n, uint32_t k,
                                  const uint32_t* __restrict__ tentry,
                                  const uint32_t* __restrict__ tstart, const int* bad,
                                  uint64_t* counts, uint32_t* __restrict__ out_idx,
                                  float* __restrict__ out_w) {
  const uint64_t r = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  if (r >= n || *bad) return;
  const bool own = lane < k;
  const uint32_t col = own ? indices[r * k + lane] : 0xFFFFFFFFu;
  const float wf = own ? w[r * k + lane] : 0.0f;
  const uint32_t b0 = tstart[r], deg = tstart[r + 1] - b0;
  // Chunks of the transposed entries, 32 at a time: `eq` those naming an own column, and for
  // each own column the entries below it.
  float wt = 0.0f;
  uint32_t src = 0xFFFFFFFFu, met = 0, less = 0, before = 0;
  float wr = 0.0f;
  auto chunk = [&](uint32_t i0) {
    src = 0xFFFFFFFFu;
    wr = 0.0f;
    if (i0 + lane < deg) {
      const uint32_t e = tentry[b0 + i0 + lane];
      src = e / k;
      wr = w[e];
    }
    met = less = before = 0;
    for (uint32_t j = 0; j < k; ++j) {
      const uint32_t c = __shfl_sync(0xFFFFFFFFu, col, j);
      const uint32_t eq = __ballot_sync(0xFFFFFFFFu, src == c);
      const uint32_t lt = __ballot_sync(0xFFFFFFFFu, src < c);
      if (eq) {
        const float v = __shfl_sync(0xFFFFFFFFu, wr, __ffs(eq) - 1);
        if (lane == j) wt = v;
        met |= eq;
      }
      if (lane == j) less = lt;
      before += c < src ? 1u : 0u;
    }
  };
  for (uint32_t i0 = 0; i0 < deg; i0 += 32) chunk(i0);
  const float weight = union_weight(wf, wt);
  const unsigned kept = __ballot_sync(0xFFFFFFFFu, own && weight != 0.0f);
  const uint64_t base = r * k + b0;
  uint32_t between = 0, placed = 0;  // other rows' entries before the own one; so far
  for (uint32_t i0 = 0; i0 < deg; i0 += 32) {
    if (deg > 32) chunk(i0);
    const float v = union_weight(0.0f, wr);
    const bool in = i0 + lane < deg && !((met >> lane) & 1u) && v != 0.0f;
    const unsigned others = __ballot_sync(0xFFFFFFFFu, in);
    between += __popc(less & others);
    if (in) {
      const uint64_t at = base + placed + __popc(others & below) +
                          __popc(kept & (before >= 32 ? 0xFFFFFFFFu : (1u << before) - 1u));
      out_idx[at] = src;
      out_w[at] = v;
    }
    placed += __popc(others);
  }
  if ((kept >> lane) & 1u) {
    const uint64_t at = base + __popc(kept & below) + between;
    out_idx[at] = col;
    out_w[at] = weight;
  }
  if (lane == 0) counts[r] = __popc(kept) + placed;
}

// Any k: a thread a row, the two runs merged.
__global__ void union_merge_kernel(const uint32_t* indices, const float* w, uint64_t n, uint32_t k,
                                   const uint32_t* tentry, const uint32_t* tstart,
                                   const int* bad, uint64_t* counts, uint32_t* out_idx,
                                   float* out_w) {
  const uint64_t r = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (r >= n || *bad) return;
  uint64_t f = r * k;
  const uint64_t f_end = f + k;
  uint32_t b = tstart[r];
  const uint32_t b_end = tstart[r + 1];
  const uint64_t base = f + b;
  uint64_t count = 0;
  while (f < f_end || b < b_end) {
    const uint32_t fc = f < f_end ? indices[f] : 0xFFFFFFFFu;
    const uint32_t bc = b < b_end ? tentry[b] / k : 0xFFFFFFFFu;
    const uint32_t col = min(fc, bc);
    const float wf = fc == col ? w[f++] : 0.0f;
    const float wt = bc == col ? w[tentry[b++]] : 0.0f;
    const float weight = union_weight(wf, wt);
    if (weight != 0.0f) {
      out_idx[base + count] = col;
      out_w[base + count] = weight;
      ++count;
    }
  }
  counts[r] = count;
}

// The rows closed up, a warp each (nothing when the graph was bad).
__global__ void close_rows_kernel(const uint32_t* __restrict__ idx, const float* __restrict__ w,
                                  uint64_t n, uint32_t k, const uint32_t* __restrict__ tstart,
                                  const uint64_t* __restrict__ ptr, const int* bad,
                                  uint64_t* out_ptr, uint32_t* __restrict__ out_idx,
                                  float* __restrict__ out_w) {
  const uint64_t r = (blockIdx.x * (uint64_t)blockDim.x + threadIdx.x) >> 5;
  const unsigned lane = threadIdx.x & 31u;
  if (r >= n || *bad) return;
  const uint64_t to = ptr[r], from = r * k + tstart[r];
  const uint32_t count = (uint32_t)(ptr[r + 1] - to);
  if (lane == 0) {
    out_ptr[r] = to;
    if (r + 1 == n) out_ptr[n] = ptr[n];
  }
  for (uint32_t i = lane; i < count; i += 32) {
    out_idx[to + i] = idx[from + i];
    out_w[to + i] = w[from + i];
  }
}

}  // namespace

}  // namespace kg

using namespace kg;

extern "C" kg_status kg_connectivities(kg_ctx* ctx, const uint64_t* indptr,
                                       const uint32_t* indices, const float* distances,
                                       uint64_t n_rows, uint32_t n_neighbors,
                                       uint64_t* out_indptr, uint32_t* out_indices,
                                       float* out_weights, uint64_t* out_nnz) {
  return guarded([&] {
    if (!ctx || !indptr || !indices || !distances || !out_indptr || !out_indices ||
        !out_weights || !out_nnz)
      fail(KG_ERR_INVALID, "kg_connectivities: NULL argument");
    if (n_neighbors < 2 || n_neighbors - 1 > kConnMaxK)
      fail(KG_ERR_INVALID, "kg_connectivities: n_neighbors must be 2.." +
                               std::to_string(kConnMaxK + 1));
    if (n_rows == 0 || n_rows >= 0xFFFFFFFFull ||
        n_rows * (uint64_t)(n_neighbors - 1) > (uint64_t)INT32_MAX)
      fail(KG_ERR_INVALID,
           "kg_connectivities: n_rows must be at least 1 and n_rows x (n_neighbors - 1) below 2^31");
    use_device(ctx);
    cudaStream_t s = ctx->stream;
    Trace trace(s, "connectivities");
    const uint32_t k = n_neighbors - 1;
    const uint64_t m = n_rows * k;
    DeviceBuffer<uint64_t> hp;
    DeviceBuffer<uint32_t> hi;
    DeviceBuffer<float> hd;
    // (Host arrays are copied whole: their offsets are looked at first.)
    if (!is_device_pointer(indptr) && indptr[n_rows] != m)
      fail(KG_ERR_INVALID, "kg_connectivities: every row must hold n_neighbors - 1 entries");
    const uint64_t* d_ptr = device_view(indptr, n_rows + 1, hp, s);
    const uint32_t* d_idx = device_view(indices, m, hi, s);
    const float* d_dist = device_view(distances, m, hd, s);
    struct Verdict {
      uint64_t nnz;
      int bad;
    };
    DeviceBuffer<int> bad(1, s);
    bad.zero();
    // Rows: checks, sigma, memberships.
    DeviceBuffer<float> w(m, s);
    DeviceBuffer<uint32_t> tcol(m, s), tentry(m, s), tcol_sorted(m, s), tentry_sorted(m, s);
    const unsigned threads = k <= 192 ? 128 : 64;
    const size_t smem = threads * ((k | 1u) + 2) * sizeof(float);
    allow_dynamic_smem(graph_rows_kernel, 128 * 195 * sizeof(float));
    graph_rows_kernel<<<blocks_for(n_rows, threads), threads, smem, s>>>(
        d_ptr, d_idx, d_dist, n_rows, k, n_neighbors, std::log2((double)n_neighbors), w.ptr,
        tcol.ptr, tentry.ptr, bad.ptr);
    KG_LAUNCH_CHECK();
    trace.mark("memberships");
    // The transpose: the entries sorted by column (stable: their rows stay in order).
    int bits = 1;
    while (bits < 32 && (1ull << bits) < n_rows) ++bits;
    size_t temp = 0;
    KG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, temp, tcol.ptr, tcol_sorted.ptr, tentry.ptr,
                                            tentry_sorted.ptr, (int)m, 0, bits, s));
    DeviceBuffer<unsigned char> scratch(temp, s);
    KG_CUDA(cub::DeviceRadixSort::SortPairs(scratch.ptr, temp, tcol.ptr, tcol_sorted.ptr,
                                            tentry.ptr, tentry_sorted.ptr, (int)m, 0, bits, s));
    DeviceBuffer<uint32_t> tstart(n_rows + 1, s);
    transposed_starts_kernel<<<blocks_for(n_rows + 1, 256), 256, 0, s>>>(tcol_sorted.ptr, m,
                                                                         n_rows, tstart.ptr);
    KG_LAUNCH_CHECK();
    trace.mark("transpose");
    // The union, then its rows closed up.
    DeviceBuffer<uint64_t> ptr(n_rows + 1, s);
    DeviceBuffer<uint32_t> oi(2 * m, s);
    DeviceBuffer<float> ow(2 * m, s);
    KG_CUDA(cudaMemsetAsync(ptr.ptr + n_rows, 0, 8, s));
    if (k <= 32)
      union_rows_kernel<<<blocks_for(n_rows * 32, 256), 256, 0, s>>>(
          d_idx, w.ptr, n_rows, k, tentry_sorted.ptr, tstart.ptr, bad.ptr, ptr.ptr, oi.ptr,
          ow.ptr);
    else
      union_merge_kernel<<<blocks_for(n_rows, 128), 128, 0, s>>>(
          d_idx, w.ptr, n_rows, k, tentry_sorted.ptr, tstart.ptr, bad.ptr, ptr.ptr, oi.ptr,
          ow.ptr);
    KG_LAUNCH_CHECK();
    size_t temp2 = 0;
    KG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, temp2, ptr.ptr, ptr.ptr, n_rows + 1, s));
    DeviceBuffer<unsigned char> scratch2(temp2, s);
    KG_CUDA(cub::DeviceScan::ExclusiveSum(scratch2.ptr, temp2, ptr.ptr, ptr.ptr, n_rows + 1, s));
    const bool dev_out = is_writable_here(out_indptr, ctx->device) &&
                         is_writable_here(out_indices, ctx->device) &&
                         is_writable_here(out_weights, ctx->device);
    DeviceBuffer<uint64_t> hp_out;
    DeviceBuffer<uint32_t> hi_out;
    DeviceBuffer<float> hw_out;
    if (!dev_out) {
      hp_out.alloc(n_rows + 1, s);
      hi_out.alloc(2 * m, s);
      hw_out.alloc(2 * m, s);
    }
    close_rows_kernel<<<blocks_for(n_rows * 32, 256), 256, 0, s>>>(
        oi.ptr, ow.ptr, n_rows, k, tstart.ptr, ptr.ptr, bad.ptr, dev_out ? out_indptr : hp_out.ptr,
        dev_out ? out_indices : hi_out.ptr, dev_out ? out_weights : hw_out.ptr);
    KG_LAUNCH_CHECK();
    trace.mark("union");
    Verdict v{};
    KG_CUDA(cudaMemcpyAsync(&v.nnz, ptr.ptr + n_rows, 8, cudaMemcpyDeviceToHost, s));
    KG_CUDA(cudaMemcpyAsync(&v.bad, bad.ptr, 4, cudaMemcpyDeviceToHost, s));
    wait_stream(ctx, s);
    if (v.bad == 1)
      fail(KG_ERR_INVALID, "kg_connectivities: every row must hold n_neighbors - 1 entries");
    if (v.bad == 2)
      fail(KG_ERR_INVALID,
           "kg_connectivities: a row's columns must increase strictly and be below n_rows");
    const uint64_t nnz = v.nnz;
    if (!dev_out) {
      KG_CUDA(cudaMemcpyAsync(out_indptr, hp_out.ptr, (n_rows + 1) * 8, cudaMemcpyDefault, s));
      if (nnz) {
        KG_CUDA(cudaMemcpyAsync(out_indices, hi_out.ptr, nnz * 4, cudaMemcpyDefault, s));
        KG_CUDA(cudaMemcpyAsync(out_weights, hw_out.ptr, nnz * 4, cudaMemcpyDefault, s));
      }
      wait_stream(ctx, s);
    }
    *out_nnz = nnz;
  });
}
