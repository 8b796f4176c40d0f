// The PCA's dense FP64 steps on narrow blocks (kg_dense.cuh). Every sum runs in a fixed
// order: the same bits on every run, whatever the thread layout.
#include <cmath>

#include "kg_dense.cuh"
#include "kg_internal.cuh"
#include "kg_order.cuh"

namespace kg {

namespace {

constexpr uint32_t kW = kQrMaxCols;

// ------------------------------------------------ Cholesky --------------------------

constexpr int kCholHold = 256;                // threads holding the matrix
constexpr int kCholThreads = kCholHold + 64;  // and those dividing the pivots' rows

// Right-looking Cholesky of a matrix of up to 64 columns, one CTA: a thread holds the 4 x 4
// entries (ty + 16 i, tx + 16 j) in registers; the pivot's row goes to shared memory, 64
// more threads divide it by the pivot's root (one entry each), and every thread subtracts
// its products. Entry by entry the operations and their order are those of the textbook
// loop. Latency bounds it: a step is a square root, a division, two shared-memory round
// trips and two barriers. With 1,024 threads on the matrix in shared memory and four
// barriers a step a block of 60 columns took 53 us; this form 30 us.
__global__ void __launch_bounds__(kCholThreads, 1)
cholesky_step_kernel(const double* gram, uint32_t w, double shift, double* r, int* status) {
  __shared__ double a[kW][kW + 1];  // R by row
  __shared__ double raw[kW];        // the pivot's row before its division
  __shared__ double trace;
  __shared__ int bad;
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t tx = tid & 15u, ty = (tid >> 4) & 15u;
  double m[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint32_t row = ty + 16 * i, c = tx + 16 * j;
      m[i][j] = row < w && c < w ? gram[(uint64_t)c * w + row] : 0.0;
      if (row == c) a[row][c] = m[i][j];
    }
  if (tid == 0) bad = 0;
  __syncthreads();
  if (tid == 0) {
    double tr = 0.0;
    for (uint32_t j = 0; j < w; ++j) tr += a[j][j];
    trace = tr;
  }
  __syncthreads();
  if (tx == ty) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (ty + 16 * i < w) m[i][i] += shift * trace;
  }
  // Warps 8 and 9 divide; the others hold the matrix. Barrier 1: the pivot's row (its warp
  // and the dividers); barrier 0: the divided row (everyone). The next pivot's row is
  // updated and handed over before the rest of a step's products.
  if (warp >= kCholHold / 32) {
    const uint32_t c = tid - kCholHold;
    for (uint32_t j = 0; j < w; ++j) {
      asm volatile("bar.sync 1, 96;" ::: "memory");
      const double d = raw[j];
      if (!(d > 0.0)) bad = 1;
      const double piv = sqrt(d);
      a[j][c] = c == j ? piv : raw[c] / piv;
      __syncthreads();
    }
  } else {
    auto hand_over = [&](uint32_t j, const double(&row)[4]) {
      if (j < w && warp == (j & 15u) / 2) {
        if (ty == (j & 15u)) {
#pragma unroll
          for (int c = 0; c < 4; ++c) raw[tx + 16 * c] = row[c];
        }
        __syncwarp();
        asm volatile("bar.arrive 1, 96;" ::: "memory");
      }
    };
    hand_over(0, m[0]);
#pragma unroll
    for (int jb = 0; jb < 4; ++jb) {
      for (uint32_t jj = 0; jj < 16; ++jj) {
        const uint32_t j = jb * 16 + jj;
        if (j >= w) break;  // the same for every thread
        __syncthreads();
        double x[4], y[4];
#pragma unroll
        for (int i = jb; i < 4; ++i) x[i] = a[j][ty + 16 * i];
#pragma unroll
        for (int i = jb; i < 4; ++i) y[i] = a[j][tx + 16 * i];
#pragma unroll
        for (int i = jb; i < 4; ++i) {
#pragma unroll
          for (int c = jb; c < 4; ++c) m[i][c] = fma(-x[i], y[c], m[i][c]);
          if (i == jb && jj < 15) hand_over(j + 1, m[i]);
          if (i == jb + 1 && jj == 15) hand_over(j + 1, m[i]);
        }
      }
    }
  }
  __syncthreads();
  if (bad) {
    if (tid == 0) *status = 1;
    return;
  }
  for (uint32_t x = tid; x < w * w; x += kCholThreads) {
    const uint32_t c = x / w, i = x % w;
    r[x] = i <= c ? a[i][c] : 0.0;
  }
}

// ------------------------------------------------ one-sided Jacobi (square) ---------

constexpr int kJacobiThreads = 256;  // 32 pairs of 8 lanes

struct JacobiShared {
  double a[kW][kW + 2];  // by column (rows at jacobi_row): the matrix, then U diag(sigma)
  double norms[kW];
  uint32_t order[kW];
};

// Where row r of a column lies: a lane of the column's 8 (lane r % 8) finds its rows r and
// r + 8 side by side, one 16-byte access, and the 8 lanes of an access cover 128 bytes: no
// bank conflicts, whatever columns a warp's four pairs hold.
__device__ __forceinline__ uint32_t jacobi_row(uint32_t r) {
  return (r >> 4) * 16 + (r & 7u) * 2 + ((r >> 3) & 1u);
}

// A lane's 8 rows of a column: v[m] = row lane + 8 m.
__device__ __forceinline__ void jacobi_load(const double* col, uint32_t lane, double (&v)[8]) {
#pragma unroll
  for (int x = 0; x < 4; ++x) {
    const double2 p = *reinterpret_cast<const double2*>(col + 16 * x + 2 * lane);
    v[2 * x] = p.x;
    v[2 * x + 1] = p.y;
  }
}
__device__ __forceinline__ void jacobi_store(double* col, uint32_t lane, const double (&v)[8]) {
#pragma unroll
  for (int x = 0; x < 4; ++x)
    *reinterpret_cast<double2*>(col + 16 * x + 2 * lane) = make_double2(v[2 * x], v[2 * x + 1]);
}

// The dot product over 8 lanes in the order of a 32-lane warp's: partial sums of rows L and
// L + 32, then a butterfly over 16, 8, 4, 2, 1 (the first two inside a lane).
__device__ __forceinline__ double jacobi_dot(const double (&u)[8], const double (&v)[8]) {
  double p[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) p[k] = fma(u[k + 4], v[k + 4], fma(u[k], v[k], 0.0));
  double s = (p[0] + p[2]) + (p[1] + p[3]);
#pragma unroll
  for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
  return s;
}

// Whether |ga| > 1e-15 sqrt(al) sqrt(be), as those operations round it: the squares decide
// except within rounding of the line (and where they leave the range).
__device__ __forceinline__ bool jacobi_above(double ga, double al, double be) {
  const double g2 = ga * ga, line = 1e-30 * (al * be);
  if (g2 > line * (1.0 + 1e-12) && g2 < 1e300) return true;
  if (g2 < line * (1.0 - 1e-12) && line < 1e300) return false;
  return fabs(ga) > 1e-15 * sqrt(al) * sqrt(be);
}

// Hestenes' one-sided Jacobi on the w columns of the w x w matrix in sh.a (everything past
// them zero; round-robin tournament, pairs orthogonal to 1e-15 of their norms): sh.a becomes
// U diag(sigma), sh.norms its column norms, sh.order the columns by descending norm (ties to
// the lower column), sigma[] the singular values in that order. Returns 0, or 1 if 60 sweeps
// did not converge. All threads of the CTA (at least 256) call it; the first 256 work.
//
// A block's 60 columns take about 11 sweeps of 59 rounds, so a round is everything, and it
// is latency: both columns read, three dot products, the angle (three divisions, two square
// roots and hypot in turn), the update, a barrier. Eight lanes a pair keep the round to
// eight warps, so that its FP64 instructions (two issue cycles a warp) and its shared-memory
// passes stay short: 1,270 cycles a round, 0.43 ms a block of 60; a warp a pair took 30
// warps and 3,900 cycles a round, 1.28 ms a block.
// The arithmetic is that form's, bit for bit: the Krylov blocks enter the products as fp16
// parts, and a last-bit change there moves the variances by 1e-9 of their size.
__device__ __forceinline__ int jacobi_square(JacobiShared& sh, uint32_t w, double* sigma) {
  const uint32_t lane = threadIdx.x & 7u, pair = threadIdx.x >> 3;
  const bool work = threadIdx.x < kJacobiThreads;
  const uint32_t players = (w + 1) & ~1u, turns = players - 1;
  const bool mine = work && pair < players / 2;
  int sweep = 0;
  for (; sweep < 60; ++sweep) {
    int rotated = 0;
    // Position 0 stays, the others turn; pair p meets positions p and players - 1 - p.
    uint32_t pi = mine && pair ? pair - 1 : 0, pj = players - 2 - (mine ? pair : 0);
    for (uint32_t r = 0; r < turns; ++r) {
      if (work) {  // whole warps
        uint32_t i = pair == 0 ? 0 : pi + 1, j = pj + 1;
        if (i > j) {
          const uint32_t t = i;
          i = j;
          j = t;
        }
        const bool live = mine && j < w;
        double* ci = sh.a[live ? i : 0];
        double* cj = sh.a[live ? j : 0];
        double u[8], v[8];
        jacobi_load(ci, lane, u);
        jacobi_load(cj, lane, v);
        const double al = jacobi_dot(u, u), be = jacobi_dot(v, v), ga = jacobi_dot(u, v);
        if (live && al > 0.0 && be > 0.0 && jacobi_above(ga, al, be)) {
          const double zeta = (be - al) / (2.0 * ga);
          const double tn = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + hypot(1.0, zeta));
          const double cs = 1.0 / sqrt(1.0 + tn * tn), sn = cs * tn;
#pragma unroll
          for (int x = 0; x < 8; ++x) {
            const double p = u[x], q = v[x];
            u[x] = cs * p - sn * q;
            v[x] = sn * p + cs * q;
          }
          jacobi_store(ci, lane, u);
          jacobi_store(cj, lane, v);
          rotated = 1;
        }
        if (++pi == turns) pi = 0;
        if (++pj == turns) pj = 0;
      }
      __syncthreads();
    }
    if (!__syncthreads_or(rotated)) break;
  }
  if (work) {
    for (uint32_t c = pair; c < kW; c += kJacobiThreads / 8) {
      double u[8];
      jacobi_load(sh.a[c], lane, u);
      const double ss = jacobi_dot(u, u);
      if (lane == 0) sh.norms[c] = sqrt(ss);
    }
  }
  __syncthreads();
  if (threadIdx.x < w) {
    const uint32_t c = threadIdx.x;
    const double n = sh.norms[c];
    uint32_t rank = 0;
    for (uint32_t o = 0; o < w; ++o) {
      rank += column_before(sh.norms[o], o, n, c) ? 1u : 0u;
    }
    sh.order[rank] = c;  // the ranks are a permutation of 0 .. w - 1
    sigma[rank] = n;
  }
  __syncthreads();
  return sweep >= 60 ? 1 : 0;
}

// A part's sum of squares: values [n part / parts, n (part + 1) / parts) of m, to thread 0 (a fixed
// order). Waiting for the reads is what it does: eight are on their way a thread, and the parts
// spread over the chip. (One CTA, a read at a time, behind a block of 60,000 genes x 40: 4.1 ms; now
// the parts end long before the SVD beside them.)
__device__ double squares_part(const double* m, uint64_t n, uint32_t part, uint32_t parts,
                               double* warp_sums) {
  constexpr int kAhead = 8;
  const uint64_t end = n * (part + 1) / parts;
  double ss = 0.0;
  for (uint64_t i = n * part / parts + threadIdx.x; i < end; i += kAhead * (uint64_t)blockDim.x) {
    double v[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      v[k] = i + k * (uint64_t)blockDim.x < end ? m[i + k * (uint64_t)blockDim.x] : 0.0;
#pragma unroll
    for (int k = 0; k < kAhead; ++k) ss = fma(v[k], v[k], ss);
  }
  for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
  if ((threadIdx.x & 31u) == 0) warp_sums[threadIdx.x >> 5] = ss;
  __syncthreads();
  double t = 0.0;
  for (uint32_t i = 0; i < blockDim.x / 32; ++i) t += warp_sums[i];
  return t;
}

struct SvdShared {
  JacobiShared jac;
  double f[2][kW][kW + 1];  // two factors by row
};

// CTA 0: the SVD of R = R_3 R_2 R_1. The others meanwhile: the block's sums of squares (the host
// needs both at once).
__global__ void __launch_bounds__(kJacobiThreads, 1)
small_svd_kernel(const double* r, uint32_t w, const double* block, uint64_t n, const int* status,
                 double* u_r, double* out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SvdShared& sm = *reinterpret_cast<SvdShared*>(smem_raw);
  JacobiShared& sh = sm.jac;
  if (blockIdx.x > 0) {
    const double t = squares_part(block, n, blockIdx.x - 1, gridDim.x - 1, sh.norms);
    if (threadIdx.x == 0) out[w + blockIdx.x] = t;
    return;
  }
  if (*status) {  // a factor was not written (the same for every thread)
    if (threadIdx.x == 0) out[w] = 1.0;
    return;
  }
  const uint32_t tid = threadIdx.x, tx = tid & 15u, ty = tid >> 4;
  auto load = [&](const double* from, double(*to)[kW + 1]) {
    for (uint32_t x = tid; x < kW * kW; x += blockDim.x) {
      const uint32_t c = x / kW, i = x % kW;
      to[i][c] = c < w && i < w ? from[(uint64_t)c * w + i] : 0.0;
    }
  };
  load(r, sm.f[0]);
  for (int step = 1; step < 3; ++step) {
    // f[0] = R_{step + 1} f[0], sums in index order (the zeros below the diagonals add
    // nothing).
    load(r + (uint64_t)step * w * w, sm.f[1]);
    __syncthreads();
    double t[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) t[i][c] = 0.0;
    for (uint32_t k = 0; k < w; ++k) {
      double x[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = sm.f[1][ty + 16 * i][k];
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] = sm.f[0][k][tx + 16 * i];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) t[i][c] = fma(x[i], y[c], t[i][c]);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) sm.f[0][ty + 16 * i][tx + 16 * c] = t[i][c];
  }
  __syncthreads();
  for (uint32_t x = tid; x < kW * kW; x += blockDim.x) {
    const uint32_t c = x / kW, i = x % kW;
    sh.a[c][jacobi_row(i)] = i <= c ? sm.f[0][i][c] : 0.0;
  }
  __syncthreads();
  const int failed = jacobi_square(sh, w, out);
  for (uint32_t x = tid; x < w * w; x += blockDim.x) {
    const uint32_t c = x / w, i = x % w;
    const double nv = sh.norms[sh.order[c]];
    u_r[x] = nv > 0.0 ? sh.a[sh.order[c]][jacobi_row(i)] / nv : 0.0;
  }
  if (tid == 0) out[w] = failed ? 1.0 : 0.0;
}

__global__ void __launch_bounds__(kJacobiThreads)
squares_kernel(const double* m, uint64_t n, double* out) {
  __shared__ double warp_sums[kJacobiThreads / 32];
  const double t = squares_part(m, n, blockIdx.x, gridDim.x, warp_sums);
  if (threadIdx.x == 0) out[blockIdx.x] = t;
}

// ------------------------------------------------ Householder QR + Jacobi -----------

// The thin SVD's left singular vectors of the g x w column-major block `b` (w <= 64,
// overwritten), one CTA of 32 warps: Householder QR in place (b = Q R, the reflectors
// below the diagonal, LAPACK's dlarfg convention v_j = 1), then Hestenes' one-sided
// Jacobi on R in shared memory (R V = U_R diag(sigma); pairs orthogonal to 1e-15 of
// their norms), then U = Q [U_R; 0] by applying the reflectors backwards. QR is
// backward stable, so sigma carries an absolute error of about 1e-16 |b|: the drop rule
// (sigma > 1e-10 |b|_F) sees rank deficiency as an SVD of b would.
__global__ void __launch_bounds__(1024)
qr_svd_kernel(double* b, uint32_t g, uint32_t w, double* u, double* out) {
  __shared__ JacobiShared sh;  // R, then U_R diag(sigma), by column
  __shared__ double tau[kW], beta_inv[kW];
  const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const unsigned warps = blockDim.x >> 5;
  auto colp = [&](uint32_t c) { return b + (uint64_t)c * g; };

  // Householder QR.
  for (uint32_t j = 0; j < w; ++j) {
    if (warp == 0) {
      const double* bj = colp(j);
      double ss = 0.0;
      for (uint32_t i = j + 1 + lane; i < g; i += 32) ss = fma(bj[i], bj[i], ss);
      for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
      if (lane == 0) {
        double alpha = bj[j];
        double normx = sqrt(fma(alpha, alpha, ss));
        if (ss == 0.0) {
          tau[j] = 0.0;  // already upper triangular in this column
        } else {
          double beta = alpha >= 0.0 ? -normx : normx;
          tau[j] = (beta - alpha) / beta;
          beta_inv[j] = 1.0 / (alpha - beta);  // scale of v below the diagonal
          colp(j)[j] = beta;
        }
      }
    }
    __syncthreads();
    const double t = tau[j];
    if (t != 0.0) {
      double* bj = colp(j);
      const double sc = beta_inv[j];
      for (uint32_t i = j + 1 + threadIdx.x; i < g; i += blockDim.x) bj[i] *= sc;
      __syncthreads();
      for (uint32_t c = j + 1 + warp; c < w; c += warps) {
        double* bc = colp(c);
        double d = (lane == 0) ? bc[j] : 0.0;
        for (uint32_t i = j + 1 + lane; i < g; i += 32) d = fma(bj[i], bc[i], d);
        for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xFFFFFFFFu, d, o);
        const double f = t * d;
        if (lane == 0) bc[j] -= f;
        for (uint32_t i = j + 1 + lane; i < g; i += 32) bc[i] = fma(-f, bj[i], bc[i]);
      }
    }
    __syncthreads();
  }
  // R into shared memory.
  for (uint32_t x = threadIdx.x; x < kW * kW; x += blockDim.x) {
    uint32_t c = x / kW, r = x % kW;
    sh.a[c][jacobi_row(r)] = c < w && r <= c ? colp(c)[r] : 0.0;
  }
  __syncthreads();
  const int failed = jacobi_square(sh, w, out);
  if (threadIdx.x == 0) out[w] = failed ? 1.0 : 0.0;
  // U = Q [U_R; 0]: start from U_R's unit columns, apply H_{w-1}, ..., H_0.
  for (uint64_t x = threadIdx.x; x < (uint64_t)g * w; x += blockDim.x) {
    uint32_t c = (uint32_t)(x / g), r = (uint32_t)(x % g);
    double nv = sh.norms[sh.order[c]];
    u[x] = (r < w && nv > 0.0) ? sh.a[sh.order[c]][jacobi_row(r)] / nv : 0.0;
  }
  __syncthreads();
  for (int j = (int)w - 1; j >= 0; --j) {
    const double t = tau[j];
    if (t == 0.0) continue;
    const double* v = colp(j);
    for (uint32_t c = warp; c < w; c += warps) {
      double* uc = u + (uint64_t)c * g;
      double d = (lane == 0) ? uc[j] : 0.0;
      for (uint32_t i = j + 1 + lane; i < g; i += 32) d = fma(v[i], uc[i], d);
      for (int o = 16; o; o >>= 1) d += __shfl_xor_sync(0xFFFFFFFFu, d, o);
      const double f = t * d;
      if (lane == 0) uc[j] -= f;
      for (uint32_t i = j + 1 + lane; i < g; i += 32) uc[i] = fma(-f, v[i], uc[i]);
    }
    __syncthreads();
  }
}

}  // namespace

void cholesky_step(const double* gram, uint32_t w, double shift, double* r, int* status,
                   cudaStream_t s) {
  cholesky_step_kernel<<<1, kCholThreads, 0, s>>>(gram, w, shift, r, status);
  KG_LAUNCH_CHECK();
}

void small_svd(const double* r, uint32_t w, const double* block, uint64_t n, const int* status,
               double* u_r, double* out, cudaStream_t s) {
  allow_dynamic_smem(small_svd_kernel, sizeof(SvdShared));
  small_svd_kernel<<<1 + squares_parts(n), kJacobiThreads, sizeof(SvdShared), s>>>(r, w, block, n, status, u_r, out);
  KG_LAUNCH_CHECK();
}

void qr_svd(double* b, uint32_t g, uint32_t w, double* u, double* out, cudaStream_t s) {
  qr_svd_kernel<<<1, 1024, 0, s>>>(b, g, w, u, out);
  KG_LAUNCH_CHECK();
}

void squares(const double* m, uint64_t n, double* out, cudaStream_t s) {
  squares_kernel<<<squares_parts(n), kJacobiThreads, 0, s>>>(m, n, out);
  KG_LAUNCH_CHECK();
}

}  // namespace kg
