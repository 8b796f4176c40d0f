// The leading eigenpairs of a dense symmetric f64 matrix of up to 544 rows (kg_dense.cuh):
// Householder tridiagonalisation in one cluster, the wanted eigenvalues by Sturm counts, their
// vectors by inverse iteration, and a check of the residuals and of orthonormality.
#include <cooperative_groups.h>
#include <cuda_pipeline_primitives.h>

#include <cfloat>
#include <cmath>

#include "kg_dense.cuh"
#include "kg_internal.cuh"

namespace cg = cooperative_groups;

namespace kg {

namespace {

constexpr uint32_t kTriCtas = 16;                 // CTAs of the cluster
constexpr uint32_t kTriWarps = 8;                 // a CTA
constexpr uint32_t kTriThreads = 32 * kTriWarps;
constexpr uint32_t kTriRows = 17;                 // rows of a column a lane holds
constexpr uint32_t kTriCols = 5;                  // columns a warp holds
constexpr uint32_t kMaxM = 32 * kTriRows;         // 544
constexpr uint32_t kTriKept = kMaxM / kTriCtas;   // reflectors a CTA keeps
constexpr uint32_t kTriSlots = kTriWarps * kTriCols;  // columns a CTA holds
static_assert(kTriCtas * kTriSlots >= kMaxM, "every column has a slot");

// Where column c's value is in a gathered vector: CTA c % 16's slots in a row (one store of up
// to 32 lanes a sender), an odd stride apart (no bank conflicts where consecutive columns are
// read).
constexpr uint32_t kGatherLd = kTriSlots + 1;
__device__ __forceinline__ uint32_t gathered(uint32_t c) {
  return (c % kTriCtas) * kGatherLd + c / kTriCtas;
}

// A gathered vector's barrier: a phase completes when every CTA's slots have arrived.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t cta) {
  uint32_t a;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(cta));
  return a;
}
__device__ __forceinline__ void store_async(uint32_t to, double v, uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(to),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}

// Slot `lane` (low) and 32 + lane (high) of this CTA into every CTA's `to`, two CTAs a warp,
// counted on that CTA's `bar`.
__device__ __forceinline__ void gather(double* to, uint64_t* bar, uint32_t rank, double low,
                                       double high) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
  for (uint32_t k = 0; k < kTriCtas / kTriWarps; ++k) {
    const uint32_t peer = warp * (kTriCtas / kTriWarps) + k;
    const uint32_t at = cluster_addr(to + rank * kGatherLd, peer), b = cluster_addr(bar, peer);
    store_async(at + lane * 8, low, b);
    if (lane < kTriSlots - 32) store_async(at + (32 + lane) * 8, high, b);
  }
}

// Waits for phase `phase` of a gathered vector (thread 0 says how many bytes make it up). A wait
// that runs out sets *stuck, after which no wait waits: the kernel ends with d[0] a NaN.
constexpr uint32_t kGatherPolls = 1u << 22;
__device__ __forceinline__ void await(uint64_t* bar, uint32_t phase, volatile int* stuck) {
  const uint32_t b = (uint32_t)__cvta_generic_to_shared(bar);
  if (threadIdx.x == 0)
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(b),
                 "r"(kTriCtas * kTriSlots * 8u)
                 : "memory");
  for (uint32_t n = 0; n < kGatherPolls && !*stuck; ++n) {
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(done)
        : "r"(b), "r"(phase)
        : "memory");
    if (done) return;
  }
  *stuck = 1;
}

// The sum of one value a thread, the same bits in every thread and in every CTA that adds the
// same values. `red`: kTriWarps values, not in use by an earlier call without a barrier between.
__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double t[kTriWarps];
#pragma unroll
  for (uint32_t i = 0; i < kTriWarps; ++i) t[i] = red[i];
#pragma unroll
  for (uint32_t o = kTriWarps / 2; o; o >>= 1)
#pragma unroll
    for (uint32_t i = 0; i < o; ++i) t[i] += t[i + o];
  return t[0];
}

// tridiagonalise_kernel's pass of step j over the held columns: the last step's update, then the
// product with this step's reflector into `dots`; row j + 1 goes to `next` as it passes by. The
// first Q slots of columns and 4 Q row blocks are done with (a copy of the code each: a branch a
// row block and column cost 0.4 ms of 2.5 for 540 columns).
template <uint32_t Q>
__device__ __forceinline__ void pass_over(double (&h)[kTriCols][kTriRows], const double* old_v,
                                          const double* wv, const double* new_v, double* next,
                                          double* dots, uint32_t m, uint32_t j, uint32_t rank) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  double acc[kTriCols], cw[kTriCols], cv[kTriCols];
#pragma unroll
  for (uint32_t q = Q; q < kTriCols; ++q) {
    const uint32_t c = min((q * kTriWarps + warp) * kTriCtas + rank, kMaxM - 1);
    acc[q] = 0.0;
    cw[q] = wv[c];
    cv[q] = old_v[c];
  }
#pragma unroll
  for (uint32_t r = 4 * Q; r < kTriRows; ++r) {
    const uint32_t i = 32 * r + lane;
    const double vi = old_v[i], wi = wv[i], ni = new_v[i];
#pragma unroll
    for (uint32_t q = Q; q < kTriCols; ++q) {
      h[q][r] = fma(-vi, cw[q], fma(-wi, cv[q], h[q][r]));
      acc[q] = fma(h[q][r], ni, acc[q]);
      if (r < 4 * Q + 5 && i == j + 1) next[q * kTriWarps + warp] = h[q][r];
    }
  }
  // The columns' sums over the lanes, four columns together: the first two steps halve how many
  // columns a lane adds up, so that lane 8 i ends with column Q + i's.
  constexpr uint32_t kFour = kTriCols - Q < 4 ? kTriCols - Q : 4;
  double v[4];
#pragma unroll
  for (uint32_t i = 0; i < 4; ++i) v[i] = i < kFour ? acc[(Q + i) % kTriCols] : 0.0;
  const bool up = lane & 16u, upper = lane & 8u;
  double a = up ? v[2] : v[0], b = up ? v[3] : v[1];
  a += __shfl_xor_sync(0xFFFFFFFFu, up ? v[0] : v[2], 16);
  b += __shfl_xor_sync(0xFFFFFFFFu, up ? v[1] : v[3], 16);
  double t = upper ? b : a;
  t += __shfl_xor_sync(0xFFFFFFFFu, upper ? a : b, 8);
#pragma unroll
  for (int o = 4; o; o >>= 1) t += __shfl_xor_sync(0xFFFFFFFFu, t, o);
  const uint32_t mine = (up ? 2u : 0u) + (upper ? 1u : 0u);
  if (lane % 8 == 0 && mine < kFour) dots[(Q + mine) * kTriWarps + warp] = t;
  if (Q + 4 < kTriCols) {
    double last = acc[kTriCols - 1];
#pragma unroll
    for (int o = 16; o; o >>= 1) last += __shfl_xor_sync(0xFFFFFFFFu, last, o);
    if (lane == 0) dots[(kTriCols - 1) * kTriWarps + warp] = last;
  }
}

// a (m x m, column-major, symmetric) = H_0 .. H_{m-2} T (..)^T with H_j = I - tau[j] v_j v_j^T
// (v_j: column j of `reflect`, zero up to row j, one at j + 1) and T of diagonal d and
// off-diagonal e. The textbook's column by column reduction (Golub and Van Loan, Matrix
// Computations, 8.3), with the rank-two update of a step and the product of the next made in
// one pass.
//
// One cluster of 16 CTAs holds the matrix in registers: column c in CTA c % 16, warp and slot
// (c / 16) % 8 and c / 128, a lane every 32nd row. A step's two vectors, the column (which is
// the row by symmetry: every CTA holds the entries of its own columns) and A v, are gathered
// into every CTA's shared memory by asynchronous stores counted on its barrier; the reflector is
// then computed in every CTA alike. A CTA sends its part of a step's vector only when it has read
// the vector before, and none can be a step ahead without every other's part, so one buffer a
// vector does. Latency bounds it: two exchanges, two block sums and the pass over the held columns
// a step, 5,900 cycles in all, 1.65 ms for 540 columns (with plain distributed stores, a cluster
// barrier behind each, 2.1 ms; cuSOLVER's reduction takes 4.4).
__global__ void __cluster_dims__(kTriCtas, 1, 1) __launch_bounds__(kTriThreads, 1)
tridiagonalise_kernel(const double* __restrict__ a, uint32_t m, double* d, double* e, double* tau,
                      double* reflect) {
  cg::cluster_group cluster = cg::this_cluster();
  const uint32_t rank = cluster.block_rank();
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  __shared__ double row[kTriCtas * kGatherLd];   // row j of the matrix, gathered
  __shared__ double prod[kTriCtas * kGatherLd];  // A v, gathered
  __shared__ double vec[2][kMaxM];  // the reflector of the step and of the last one
  __shared__ double wv[kMaxM];     // the last step's w: the update is A - v w^T - w v^T
  __shared__ double next[kTriSlots];  // this CTA's entries of the next row
  __shared__ double dots[kTriSlots];  // and of A v
  __shared__ double red[2][kTriWarps];
  __shared__ uint64_t row_bar, prod_bar;
  __shared__ int stuck;
  // Step j's reflector in CTA j % 16, and d, e and tau in CTA 0: written out at the end (a store
  // to global memory inside a step is one more trip that its barriers wait for).
  extern __shared__ double kept[];
  __shared__ double out_d[kMaxM], out_e[kMaxM], out_tau[kMaxM];
  double h[kTriCols][kTriRows];
#pragma unroll
  for (uint32_t q = 0; q < kTriCols; ++q) {
    const uint32_t c = (q * kTriWarps + warp) * kTriCtas + rank;
#pragma unroll
    for (uint32_t t = 0; t < kTriRows; ++t) {
      const uint32_t i = 32 * t + lane;
      h[q][t] = i < m && c < m ? a[(uint64_t)c * m + i] : 0.0;
    }
    if (lane == 0) next[q * kTriWarps + warp] = h[q][0];  // row 0
  }
  for (uint32_t i = tid; i < kMaxM; i += kTriThreads) {
    vec[0][i] = 0.0;
    vec[1][i] = 0.0;
    wv[i] = 0.0;  // (rows past m stay zero in all three)
  }
  if (tid < kTriSlots) dots[tid] = 0.0;
  if (tid == 0) {
    stuck = 0;
    for (uint64_t* bar : {&row_bar, &prod_bar})
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((uint32_t)__cvta_generic_to_shared(bar))
                   : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  cluster.sync();
  for (uint32_t j = 0; j < m; ++j) {
    const double* old_v = vec[(j + 1) & 1u];
    double* new_v = vec[j & 1u];
    // Row j with the last step's update, to every CTA.
    {
      const double vj = old_v[j], wj = wv[j];
      const uint32_t c0 = lane * kTriCtas + rank, c1 = (32 + lane) * kTriCtas + rank;
      double low = 0.0, high = 0.0;
      if (c0 < m) low = next[lane] - vj * wv[c0] - wj * old_v[c0];
      if (c1 < m && lane < kTriSlots - 32) high = next[32 + lane] - vj * wv[c1] - wj * old_v[c1];
      gather(row, &row_bar, rank, low, high);
    }
    await(&row_bar, j & 1u, &stuck);
    if (tid == 0) out_d[j] = row[gathered(j)];
    if (j + 1 == m) break;
    // The reflector of row[j + 1 ..): every CTA computes it, CTA 0 writes it.
    const double alpha = row[gathered(j + 1)];
    double part = 0.0;
    for (uint32_t i = tid; i < m; i += kTriThreads)
      if (i > j + 1) {
        const double r = row[gathered(i)];
        part += r * r;
      }
    const double sigma = block_sum(part, red[0]);
    double beta = alpha, t = 0.0, scale = 0.0;
    if (sigma > 0.0) {
      beta = -copysign(sqrt(alpha * alpha + sigma), alpha);
      t = (beta - alpha) / beta;
      scale = 1.0 / (alpha - beta);
    }
    for (uint32_t i = tid; i < m; i += kTriThreads) {
      const double v = i <= j ? 0.0 : i == j + 1 ? 1.0 : row[gathered(i)] * scale;
      new_v[i] = v;
      if (j % kTriCtas == rank) kept[j / kTriCtas * m + i] = v;
    }
    if (tid == 0) {
      out_e[j] = beta;
      out_tau[j] = t;
    }
    __syncthreads();
    // (j + 1) / 128 whole slots of columns and four times as many row blocks are done with.
    switch ((j + 1) / (kTriWarps * kTriCtas)) {
      case 0: pass_over<0>(h, old_v, wv, new_v, next, dots, m, j, rank); break;
      case 1: pass_over<1>(h, old_v, wv, new_v, next, dots, m, j, rank); break;
      case 2: pass_over<2>(h, old_v, wv, new_v, next, dots, m, j, rank); break;
      case 3: pass_over<3>(h, old_v, wv, new_v, next, dots, m, j, rank); break;
      default: pass_over<4>(h, old_v, wv, new_v, next, dots, m, j, rank); break;
    }
    __syncthreads();
    gather(prod, &prod_bar, rank, dots[lane], lane < kTriSlots - 32 ? dots[32 + lane] : 0.0);
    await(&prod_bar, j & 1u, &stuck);
    part = 0.0;
    for (uint32_t i = tid; i < m; i += kTriThreads)
      if (i > j) part += prod[gathered(i)] * new_v[i];
    const double pv = block_sum(part, red[1]);
    const double half = 0.5 * t * t * pv;
    for (uint32_t i = tid; i < m; i += kTriThreads)
      wv[i] = i > j ? t * prod[gathered(i)] - half * new_v[i] : 0.0;
    __syncthreads();
  }
  __syncthreads();
  if (stuck) {
    if (tid == 0) out_d[0] = NAN;
    for (int n = 0; n < 1000; ++n) __nanosleep(1000);  // for what is still on its way
  }
  cluster.sync();  // no CTA leaves while another may still write to it
  for (uint32_t j = rank; j + 1 < m; j += kTriCtas)
    for (uint32_t i = tid; i < m; i += kTriThreads)
      reflect[(uint64_t)j * m + i] = kept[j / kTriCtas * m + i];
  if (rank == 0)
    for (uint32_t i = tid; i < m; i += kTriThreads) {
      d[i] = out_d[i];
      if (i + 1 < m) {
        e[i] = out_e[i];
        tau[i] = out_tau[i];
      }
    }
}

constexpr uint32_t kBisectThreads = 256;
constexpr int kBisectRounds = 7;  // 257^7 > 2^56: the last interval is below rounding

// bounds[0], bounds[1]: an interval with every eigenvalue of T; values[r]: its r-th largest. A
// CTA an eigenvalue and a point a thread: the Sturm count of each (the sign changes of the
// leading minors of T - x I, by their three-term recurrence; Givens) tells how many eigenvalues
// lie below it. T is scaled to norm 1, and every eight steps the last two minors are by a power of
// two, so neither leaves the range; a vanishing e^2 is kept at 2^-120, 2^-60 of the norm. The
// chain is one multiply-add a step (with the quotients of the minors instead it is a division:
// 319 us for 50 of 540).
__global__ void __launch_bounds__(kBisectThreads)
bisect_kernel(const double* d, const double* e, uint32_t m, double* values, double* bounds) {
  __shared__ double sd[kMaxM], se2[kMaxM];  // (a multiple of eight: T continued by eigenvalues of 4)
  __shared__ double lows[kBisectThreads / 32], highs[kBisectThreads / 32];
  const uint32_t tid = threadIdx.x;
  double lo = INFINITY, hi = -INFINITY;
  for (uint32_t i = tid; i < m; i += kBisectThreads) {
    const double l = i ? fabs(e[i - 1]) : 0.0, r = i + 1 < m ? fabs(e[i]) : 0.0;
    sd[i] = d[i];
    se2[i] = i ? e[i - 1] : 0.0;
    lo = fmin(lo, d[i] - (l + r));
    hi = fmax(hi, d[i] + (l + r));
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
  }
  if ((tid & 31u) == 0) {
    lows[tid >> 5] = lo;
    highs[tid >> 5] = hi;
  }
  __syncthreads();
  for (uint32_t i = 0; i < kBisectThreads / 32; ++i) {
    lo = fmin(lo, lows[i]);
    hi = fmax(hi, highs[i]);
  }
  const double norm = fmax(fmax(fabs(lo), fabs(hi)), DBL_MIN);
  const double slack = 4.0 * m * DBL_EPSILON * norm;
  lo -= slack;
  hi += slack;
  if (blockIdx.x == 0 && tid == 0) {
    bounds[0] = lo;
    bounds[1] = hi;
  }
  const double to_one = 1.0 / norm;
  for (uint32_t i = tid; i < kMaxM; i += kBisectThreads) {
    const double t = i < m ? se2[i] * to_one : 0.0;
    sd[i] = i < m ? sd[i] * to_one : 4.0;
    se2[i] = fmax(t * t, 0x1p-120);
  }
  __syncthreads();
  const uint32_t index = m - 1 - blockIdx.x;  // ascending: `index` eigenvalues lie below
  for (int round = 0; round < kBisectRounds; ++round) {
    const double step = (hi - lo) / (kBisectThreads + 1);
    const double x = (lo + step * (tid + 1)) * to_one;
    double p1 = 1.0, p2 = 0.0;  // the last two minors
    uint32_t below = 0, sign = 0;
    for (uint32_t i0 = 0; i0 < m; i0 += 8) {
#pragma unroll
      for (uint32_t k = 0; k < 8; ++k) {
        const uint32_t i = i0 + k;
        const double p = fma(sd[i] - x, p1, -(se2[i] * p2));
        p2 = p1;
        p1 = p;
        // (A zero counts as a change: the next minor then has its sign.)
        const uint32_t now = p == 0.0 ? sign ^ 1u : (uint32_t)__double2hiint(p) >> 31;
        below += now ^ sign;
        sign = now;
      }
      const uint32_t exponent =
          max((uint32_t)__double2hiint(p1) >> 20 & 0x7FFu, (uint32_t)__double2hiint(p2) >> 20 & 0x7FFu);
      const double scale = __hiloint2double((int)((2046u - min(exponent, 2045u)) << 20), 0);
      p1 *= scale;
      p2 *= scale;
    }
    const int left = __syncthreads_count(below <= index);  // points at or below the eigenvalue
    const double base = lo;
    lo = base + step * left;
    if (left < (int)kBisectThreads) hi = base + step * (left + 1);
  }
  if (tid == 0) values[blockIdx.x] = 0.5 * (lo + hi);
}

__device__ __forceinline__ double start_value(uint32_t r, uint32_t i) {  // in (-1, 1), never 0
  uint64_t z = ((uint64_t)r << 32 | i) + 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return ((double)(z >> 11) + 0.5) * 0x1p-52 - 1.0;
}

// Column r of x (m x take): the vector of T's r-th largest eigenvalue, by inverse iteration
// with T - value I factored by Gaussian elimination with row exchanges (Wilkinson; as LAPACK's
// dstein: random starts, close shifts set apart, tiny pivots replaced). One lane a vector
// solves, a chain of m steps a solve (a division each in the factorisation); the vectors run
// side by side.
constexpr int kInverseIterations = 3;

__global__ void __launch_bounds__(32)
inverse_iteration_kernel(const double* d, const double* e, uint32_t m, const double* values,
                         const double* bounds, double* x) {
  __shared__ double sd[kMaxM], se[kMaxM], mult[kMaxM], inv[kMaxM], up1[kMaxM], up2[kMaxM],
      v[kMaxM];
  __shared__ unsigned char swapped[kMaxM];
  const uint32_t lane = threadIdx.x, r = blockIdx.x;
  const double norm = fmax(fmax(fabs(bounds[0]), fabs(bounds[1])), DBL_MIN);
  for (uint32_t i = lane; i < m; i += 32) {
    sd[i] = d[i];
    se[i] = i + 1 < m ? e[i] : 0.0;
    v[i] = start_value(r, i);
  }
  __syncwarp();
  if (lane == 0) {
    double shift = values[0];
    for (uint32_t i = 1; i <= r; ++i) shift = fmin(values[i], shift - 8.0 * DBL_EPSILON * norm);
    const double tiny = DBL_EPSILON * norm;
    double p = sd[0] - shift, q = se[0];
    for (uint32_t i = 0; i + 1 < m; ++i) {
      const double s = se[i], t = sd[i + 1] - shift, u = se[i + 1];
      const bool swap = fabs(p) < fabs(s);
      double pivot = swap ? s : p;
      if (fabs(pivot) < tiny) pivot = copysign(tiny, pivot);
      const double r1 = 1.0 / pivot;
      const double l = (swap ? p : s) * r1;
      up1[i] = swap ? t : q;
      up2[i] = swap ? u : 0.0;
      inv[i] = r1;
      mult[i] = l;
      swapped[i] = swap;
      p = swap ? q - l * t : t - l * q;
      q = swap ? -l * u : u;
    }
    if (fabs(p) < tiny) p = copysign(tiny, p);
    inv[m - 1] = 1.0 / p;
    up1[m - 1] = up2[m - 1] = 0.0;
  }
  __syncwarp();
  for (int it = 0; it < kInverseIterations; ++it) {
    if (lane == 0) {
      if (it) {  // (the first start stands for a vector already forward-solved)
        double cur = v[0];
        for (uint32_t i = 0; i + 1 < m; ++i) {
          const double nx = v[i + 1];
          const bool swap = swapped[i];
          const double first = swap ? nx : cur, second = swap ? cur : nx;
          v[i] = first;
          cur = second - mult[i] * first;
        }
        v[m - 1] = cur;
      }
      double b1 = 0.0, b2 = 0.0;
      for (uint32_t i = m; i-- > 0;) {
        const double b0 = (v[i] - up1[i] * b1 - up2[i] * b2) * inv[i];
        v[i] = b0;
        b2 = b1;
        b1 = b0;
      }
    }
    __syncwarp();
    double most = 0.0;
    for (uint32_t i = lane; i < m; i += 32) most = fmax(most, fabs(v[i]));
#pragma unroll
    for (int o = 16; o; o >>= 1) most = fmax(most, __shfl_xor_sync(0xFFFFFFFFu, most, o));
    const double down = most > 0.0 ? 1.0 / most : 1.0;
    for (uint32_t i = lane; i < m; i += 32) v[i] *= down;
    __syncwarp();
  }
  for (uint32_t i = lane; i < m; i += 32) x[(uint64_t)r * m + i] = v[i];
}

// x (m x take) made orthonormal by modified Gram-Schmidt in the order of
// the columns, in shared memory: the part along the current column is taken out of all later
// ones at once, a warp a column. (Inverse iteration leaves close to orthonormal vectors but for
// close eigenvalues, and those independent; what is off all the same fails the check.)
constexpr uint32_t kMgsThreads = 1024;
constexpr uint32_t kMaxTake = 50;

__global__ void __launch_bounds__(kMgsThreads, 1)
orthonormalise_kernel(double* x, uint32_t m, uint32_t take) {
  extern __shared__ double s[];  // columns of kMaxM, zeros past m
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  for (uint32_t i = tid; i < kMaxM * take; i += kMgsThreads) {
    const uint32_t r = i % kMaxM, c = i / kMaxM;
    s[i] = r < m ? x[(uint64_t)c * m + r] : 0.0;
  }
  __syncthreads();
  for (uint32_t r = 0; r < take; ++r) {
    double* cr = s + r * kMaxM;
    // (Each warp computes the norm; the scaled column is written after all have read it, and
    // not read again before the end.)
    double pivot[kTriRows], n[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (uint32_t t = 0; t < kTriRows; ++t) {
      pivot[t] = cr[32 * t + lane];
      n[t & 3] = fma(pivot[t], pivot[t], n[t & 3]);
    }
    double n2 = (n[0] + n[1]) + (n[2] + n[3]);
#pragma unroll
    for (int o = 16; o; o >>= 1) n2 += __shfl_xor_sync(0xFFFFFFFFu, n2, o);
    const double inv2 = 1.0 / n2;
    for (uint32_t c = r + 1 + warp; c < take; c += kMgsThreads / 32) {
      double* cc = s + c * kMaxM;
      double d[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (uint32_t t = 0; t < kTriRows; ++t) d[t & 3] = fma(pivot[t], cc[32 * t + lane], d[t & 3]);
      double dot = (d[0] + d[1]) + (d[2] + d[3]);
#pragma unroll
      for (int o = 16; o; o >>= 1) dot += __shfl_xor_sync(0xFFFFFFFFu, dot, o);
      dot *= inv2;
#pragma unroll
      for (uint32_t t = 0; t < kTriRows; ++t) cc[32 * t + lane] = fma(-dot, pivot[t], cc[32 * t + lane]);
    }
    __syncthreads();
    for (uint32_t i = tid; i < m; i += kMgsThreads) x[(uint64_t)r * m + i] = cr[i] * (1.0 / sqrt(n2));
  }
}

// z -= tau (v . z) v over the row blocks from T0 on (v is zero before).
template <uint32_t T0>
__device__ __forceinline__ void reflect_column(double (&z)[kTriRows], const double* v, double tau) {
  const uint32_t lane = threadIdx.x;
  double r[kTriRows], a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (uint32_t t = T0; t < kTriRows; ++t) {
    r[t] = v[32 * t + lane];
    a[t & 3] = fma(r[t], z[t], a[t & 3]);
  }
  double dot = (a[0] + a[1]) + (a[2] + a[3]);
#pragma unroll
  for (int o = 16; o; o >>= 1) dot += __shfl_xor_sync(0xFFFFFFFFu, dot, o);
  dot *= tau;
#pragma unroll
  for (uint32_t t = T0; t < kTriRows; ++t) z[t] = fma(-dot, r[t], z[t]);
}

// x's column (one warp a column) = H_0 .. H_{m-2} of it. The reflectors stream through shared
// memory kBackAhead steps ahead (read when they are needed, the L2's latency a step: 333 us).
constexpr uint32_t kBackAhead = 8;

__global__ void __launch_bounds__(32)
back_transform_kernel(const double* __restrict__ reflect, const double* __restrict__ tau,
                      uint32_t m, double* x) {
  __shared__ double ring[kBackAhead][kMaxM];
  __shared__ double st[kMaxM];
  const uint32_t lane = threadIdx.x;
  double* col = x + (uint64_t)blockIdx.x * m;
  double z[kTriRows];
#pragma unroll
  for (uint32_t t = 0; t < kTriRows; ++t) {
    const uint32_t i = 32 * t + lane;
    z[t] = i < m ? col[i] : 0.0;
    if (i + 1 < m) st[i] = tau[i];
#pragma unroll
    for (uint32_t b = 0; b < kBackAhead; ++b) ring[b][i] = 0.0;  // rows past m stay zero
  }
  __syncwarp();
  // Reflector j is zero up to row j; rows are read from the first row block in use on.
  auto fetch = [&](uint32_t j) {
    double* to = ring[j % kBackAhead];
    const double* from = reflect + (uint64_t)j * m;
    for (uint32_t i = (j + 1) / 128 * 128 + lane; i < m; i += 32)
      __pipeline_memcpy_async(to + i, from + i, 8);
  };
  const uint32_t last = m - 2;
  for (uint32_t b = 0; b + 1 < kBackAhead; ++b) {
    if (b <= last) fetch(last - b);
    __pipeline_commit();
  }
  for (uint32_t step = 0; step <= last; ++step) {
    const uint32_t j = last - step;
    __syncwarp();  // the slot of step - 1 has been read
    if (step + kBackAhead - 1 <= last) fetch(j - (kBackAhead - 1));
    __pipeline_commit();
    __pipeline_wait_prior(kBackAhead - 1);
    __syncwarp();
    const double* v = ring[j % kBackAhead];
    const double tj = st[j];
    switch ((j + 1) / 128) {  // (a copy of the code for every four row blocks done with)
      case 0: reflect_column<0>(z, v, tj); break;
      case 1: reflect_column<4>(z, v, tj); break;
      case 2: reflect_column<8>(z, v, tj); break;
      case 3: reflect_column<12>(z, v, tj); break;
      default: reflect_column<16>(z, v, tj); break;
    }
  }
#pragma unroll
  for (uint32_t t = 0; t < kTriRows; ++t) {
    const uint32_t i = 32 * t + lane;
    if (i < m) col[i] = z[t];
  }
}

// *good = 0 where a pair's residual (of the norm) or the vectors' orthonormality is off: az = a x,
// gram = x^T x, a warp a column. The line is about six times what the method reaches: measured,
// in units of 2^-52, residuals to 9 and products to 6 for 11 columns, 11 and 11 for 63 with three
// eigenvalues many times each, 4 and 8 for 192, 4 and 7 for 270, 3 and 14 for 540.
__global__ void __launch_bounds__(32)
check_pairs_kernel(const double* az, const double* x, const double* gram, const double* values,
                   const double* bounds, uint32_t m, uint32_t take, int* good) {
  const uint32_t lane = threadIdx.x, r = blockIdx.x;
  const double norm = fmax(fabs(bounds[0]), fabs(bounds[1]));
  const double tol = (16.0 + 0.125 * m) * DBL_EPSILON;
  double sum = 0.0;
  for (uint32_t i = lane; i < m; i += 32) {
    const double t = az[(uint64_t)r * m + i] - values[r] * x[(uint64_t)r * m + i];
    sum += t * t;
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
  bool ok = sqrt(sum) <= tol * norm;
  for (uint32_t c = lane; c < take; c += 32)
    ok = ok && fabs(gram[(uint64_t)r * take + c] - (c == r ? 1.0 : 0.0)) <= tol;
  if (!__all_sync(0xFFFFFFFFu, ok) && lane == 0) *good = 0;
}

cudaLaunchConfig_t tri_config(cudaLaunchAttribute* at, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kTriCtas);
  cfg.blockDim = dim3(kTriThreads);
  cfg.dynamicSmemBytes = kTriKept * kMaxM * sizeof(double);
  cfg.stream = s;
  at->id = cudaLaunchAttributeClusterDimension;
  at->val.clusterDim.x = kTriCtas;
  at->val.clusterDim.y = 1;
  at->val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cfg;
}

}  // namespace

bool leading_eigenpairs(cublasHandle_t cublas, const double* a, uint32_t m, uint32_t take,
                        double* vectors, std::vector<double>& values, cudaStream_t s) {
  if (m < 2 || m > kMaxM || take < 1 || take > m || take > kMaxTake) return false;
  // A cluster of 16 CTAs is past the portable size: asked for, and used only where it fits.
  KG_CUDA(cudaFuncSetAttribute(tridiagonalise_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed,
                               1));
  allow_dynamic_smem(tridiagonalise_kernel, kTriKept * kMaxM * sizeof(double));
  allow_dynamic_smem(orthonormalise_kernel, kMaxTake * kMaxM * sizeof(double));
  cudaLaunchAttribute at;
  cudaLaunchConfig_t cfg = tri_config(&at, s);
  int fit = 0;
  if (cudaOccupancyMaxActiveClusters(&fit, tridiagonalise_kernel, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  if (fit < 1) return false;
  DeviceBuffer<double> work((uint64_t)m * m + 3ull * m + 2 * take + 2 + 2ull * m * take, s);
  double* reflect = work.ptr;
  double* d = reflect + (uint64_t)m * m;
  double* e = d + m;
  double* tau = e + m;
  double* vals = tau + m;
  double* bounds = vals + take;
  double* az = bounds + 2;
  DeviceBuffer<double> gram((uint64_t)take * take, s);
  DeviceBuffer<int> good(1, s);
  KG_CUDA(cudaLaunchKernelEx(&cfg, tridiagonalise_kernel, a, m, d, e, tau, reflect));
  KG_LAUNCH_CHECK();
  bisect_kernel<<<take, kBisectThreads, 0, s>>>(d, e, m, vals, bounds);
  KG_LAUNCH_CHECK();
  inverse_iteration_kernel<<<take, 32, 0, s>>>(d, e, m, vals, bounds, vectors);
  KG_LAUNCH_CHECK();
  orthonormalise_kernel<<<1, kMgsThreads, (size_t)kMaxM * take * sizeof(double), s>>>(vectors, m,
                                                                                             take);
  KG_LAUNCH_CHECK();
  back_transform_kernel<<<take, 32, 0, s>>>(reflect, tau, m, vectors);
  KG_LAUNCH_CHECK();
  const double one = 1.0, zero = 0.0;
  KG_CUBLAS(cublasDgemm(cublas, CUBLAS_OP_N, CUBLAS_OP_N, m, take, m, &one, a, m, vectors, m, &zero,
                        az, m));
  KG_CUBLAS(cublasDgemm(cublas, CUBLAS_OP_T, CUBLAS_OP_N, take, take, m, &one, vectors, m, vectors,
                        m, &zero, gram.ptr, take));
  KG_CUDA(cudaMemsetAsync(good.ptr, 1, sizeof(int), s));
  check_pairs_kernel<<<take, 32, 0, s>>>(az, vectors, gram.ptr, vals, bounds, m, take, good.ptr);
  KG_LAUNCH_CHECK();
  values.resize(take);
  int h_good = 0;
  KG_CUDA(cudaMemcpyAsync(values.data(), vals, take * 8ull, cudaMemcpyDeviceToHost, s));
  KG_CUDA(cudaMemcpyAsync(&h_good, good.ptr, sizeof(int), cudaMemcpyDeviceToHost, s));
  KG_CUDA(cudaStreamSynchronize(s));
  return h_good != 0;
}

}  // namespace kg
