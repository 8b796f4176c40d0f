// The PCA's dense FP64 steps on narrow blocks (kg_dense.cuh). Every sum runs in a fixed
// order: the same bits on every run.
#include <cooperative_groups.h>

#include <cmath>

#include "kg_dense.cuh"
#include "kg_internal.cuh"

namespace cg = cooperative_groups;

namespace kg {

namespace {

constexpr uint32_t kW = kQrMaxCols;

// ------------------------------------------------ one-sided Jacobi (square) ---------

// Approximations for a rotation's angle (about 20 bits).
__device__ __forceinline__ double rcp_approx(double v) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(v));
  return r;
}

__device__ __forceinline__ float rcp_approx(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float sqrt_approx(float v) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// 1/sqrt(x) for x in [1, 2] to f64: an f32 start and two Newton steps.
__device__ __forceinline__ double rsqrt_12(double x) {
  double y = (double)rsqrtf((float)x);
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const double e = fma(-x * y, y, 1.0);
    y = fma(0.5 * y, e, y);
  }
  return y;
}

constexpr int kJacobiThreads = 256;  // 32 pairs of 8 lanes

struct JacobiShared {
  double a[kW][kW + 1];  // by column: the matrix, then U diag(sigma)
  double norms[kW];
  double red[32];
  uint32_t order[kW];
};

// Hestenes' one-sided Jacobi on the w columns of the w x w matrix sh.a (rows w .. 63 zero,
// w <= 64): a round-robin tournament, pairs orthogonal to 1e-15 of their norms; sh.a
// becomes U diag(sigma) / 2^e, sh.norms its column norms, sh.order the columns by
// descending norm (ties to the lower column), sigma[] the singular values in that order.
// Returns 0, or 1 if 60 sweeps did not converge. All threads of the CTA (at least 256)
// call it; the first 256 work.
//
// A block's 60 columns take about 10 sweeps of 59 rounds, so the round is everything: a
// pair is 8 lanes of 8 rows (three dot products, three shuffle steps), the rotation's
// angle comes from 20-bit approximations (the pair's remaining product is a 2^-20th of
// it, which the next sweeps take; c and s keep c^2 + s^2 = 1 to f64), and a round is one
// barrier of 8 warps. One warp a pair with IEEE division, square root and hypot took 1.27
// ms a block of 60 columns (about 3,900 cycles a round).
__device__ int jacobi_square(JacobiShared& sh, uint32_t w, double* sigma) {
  const uint32_t lane = threadIdx.x & 7u, pair = threadIdx.x >> 3;
  const bool work = threadIdx.x < kJacobiThreads;
  // Scaled by a power of two (exact) so that the squares and their products stay in range.
  double top = 0.0;
  if (work)
    for (uint32_t x = threadIdx.x; x < kW * kW; x += kJacobiThreads)
      top = fmax(top, fabs(sh.a[x / kW][x % kW]));
  for (int o = 16; o; o >>= 1) top = fmax(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
  if ((threadIdx.x & 31u) == 0) sh.red[threadIdx.x >> 5] = top;
  __syncthreads();
  top = 0.0;
  for (uint32_t i = 0; i < blockDim.x / 32; ++i) top = fmax(top, sh.red[i]);
  const int e = top > 0.0 && isfinite(top) ? ilogb(top) : 0;
  if (work && e != 0)
    for (uint32_t x = threadIdx.x; x < kW * kW; x += kJacobiThreads)
      sh.a[x / kW][x % kW] = ldexp(sh.a[x / kW][x % kW], -e);
  __syncthreads();

  const uint32_t players = (w + 1) & ~1u, turns = players - 1;
  const bool mine = work && pair < players / 2;
  int sweep = 0;
  for (; sweep < 60; ++sweep) {
    int rotated = 0;
    // Positions 1 .. players - 1 turn; player 0 stays. Pair p meets positions p and
    // players - 1 - p.
    uint32_t pi = pair == 0 ? 0 : pair - 1, pj = players - 2 - (mine ? pair : 0);
    for (uint32_t r = 0; r < turns; ++r) {
      if (work) {  // whole warps
        uint32_t i = pair == 0 ? 0 : pi + 1, j = pj + 1;
        if (i > j) {
          const uint32_t t = i;
          i = j;
          j = t;
        }
        const bool live = mine && j < w;
        double* ai = sh.a[live ? i : 0];
        double* aj = sh.a[live ? j : 0];
        double u[kW / 8], v[kW / 8];
        double al = 0.0, be = 0.0, ga = 0.0;
#pragma unroll
        for (int x = 0; x < (int)kW / 8; ++x) {
          u[x] = ai[lane + 8 * x];
          v[x] = aj[lane + 8 * x];
          al = fma(u[x], u[x], al);
          be = fma(v[x], v[x], be);
          ga = fma(u[x], v[x], ga);
        }
#pragma unroll
        for (int o = 4; o; o >>= 1) {
          al += __shfl_xor_sync(0xFFFFFFFFu, al, o);
          be += __shfl_xor_sync(0xFFFFFFFFu, be, o);
          ga += __shfl_xor_sync(0xFFFFFFFFu, ga, o);
        }
        if (live && al > 0.0 && be > 0.0 && ga * ga > 1e-30 * (al * be)) {
          const double zeta = 0.5 * (be - al) * rcp_approx(ga);
          // t = sign(zeta) / (|zeta| + sqrt(1 + zeta^2)), and 1 / (2 zeta) far out (columns
          // of very different norms: past f32's range).
          const float z = (float)zeta;
          const float tf = rcp_approx(fabsf(z) + sqrt_approx(fmaf(z, z, 1.0f)));
          const double t = fabs(zeta) > 1e8 ? rcp_approx(2.0 * zeta)
                                            : (double)(z >= 0.0f ? tf : -tf);
          const double c = rsqrt_12(fma(t, t, 1.0)), s = c * t;
#pragma unroll
          for (int x = 0; x < (int)kW / 8; ++x) {
            ai[lane + 8 * x] = fma(c, u[x], -(s * v[x]));
            aj[lane + 8 * x] = fma(s, u[x], c * v[x]);
          }
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
      double ss = 0.0;
#pragma unroll
      for (int x = 0; x < (int)kW / 8; ++x) ss = fma(sh.a[c][lane + 8 * x], sh.a[c][lane + 8 * x], ss);
#pragma unroll
      for (int o = 4; o; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
      if (lane == 0) sh.norms[c] = sqrt(ss);
    }
  }
  __syncthreads();
  if (threadIdx.x < w) {
    const uint32_t c = threadIdx.x;
    const double n = sh.norms[c];
    uint32_t rank = 0;
    for (uint32_t o = 0; o < w; ++o) {
      const double m = sh.norms[o];
      rank += (m > n || (!(m < n) && o < c)) ? 1u : 0u;
    }
    if (rank < w) {
      sh.order[rank] = c;
      sigma[rank] = ldexp(n, e);
    }
  }
  __syncthreads();
  return sweep >= 60 ? 1 : 0;
}

// ------------------------------------------------ the block's SVD, one cluster ------

constexpr int kXbThreads = 256;
constexpr uint32_t kXbCluster = 16;    // CTAs (non-portable; 8 where 16 do not fit)
constexpr uint32_t kXbRows = 64;       // rows a staged chunk
constexpr uint32_t kXbSolve = 128;     // rows a triangular solve's pass

struct XbShared {
  union {
    struct {
      double part[kW * kW];  // this CTA's rows' share of the Gram matrix
      double full[kW * kW];  // the whole Gram matrix
    } g;
    double x[kW][kXbSolve];  // rows under the triangular solve
  };
  double r[kW][kW];          // the round's R by row
  double rtot[2][kW][kW];    // the running product of the rounds' R (rank 0)
  union {
    double rows[kXbRows][kW + 1];  // a staged chunk
    JacobiShared jac;
  };
  double dinv[kW];           // 1 / R[j][j]
  double red[kXbThreads / 32];
  double norm;
  int bad;
};

// Stage rows [r0, r0 + 64) of a (g x w column-major; rows at or past r1 and columns past w
// as zeros) into sh.rows.
__device__ __forceinline__ void stage_rows(XbShared& sh, const double* a, uint32_t g, uint32_t w,
                                           uint32_t r0, uint32_t r1) {
  for (uint32_t x = threadIdx.x; x < kXbRows * kW; x += kXbThreads) {
    const uint32_t r = x % kXbRows, c = x / kXbRows;
    sh.rows[r][c] = r0 + r < r1 && c < w ? a[(uint64_t)c * g + r0 + r] : 0.0;
  }
}

// The orthonormalisation of a Krylov block in one launch: shifted CholeskyQR3 (Fukaya,
// Kannan, Nakatsukasa, Yamamoto and Yanagisawa, "Shifted Cholesky QR for computing the QR
// factorization of ill-conditioned matrices", SIAM J. Sci. Comput. 2020), the Jacobi SVD
// of R, U = Q U_R. A cluster of 16 CTAs splits the rows; each round is: the rows' share of
// the Gram matrix (four 64-thread groups of 8 x 8 outputs a thread), the shares summed
// through distributed shared memory (a slice of the entries a CTA, handed to all), the
// Cholesky factor in every CTA (the same bits everywhere: 4 x 4 entries a thread in
// registers, rows published through shared memory, LDL^T so that a step waits for one
// reciprocal), and the rows' triangular solve (a thread a row, 8-column blocks). Rank 0
// runs the Jacobi while the others wait.
// Latency bounds it (a 2,000 x 60 block is 1 MB, 3 x 7 Mflop): the same steps as separate
// launches (three Gram GEMMs, factors and solves of cuBLAS and one-CTA kernels, the SVD,
// the last GEMM, two norms read by the host) took 2.02 ms a block.
__global__ void __launch_bounds__(kXbThreads, 1)
extend_svd_kernel(const double* __restrict__ block, const double* __restrict__ rest, uint32_t g,
                  uint32_t w, double shift, double* q, double* __restrict__ u, double* out) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  XbShared& sh = *reinterpret_cast<XbShared*>(smem_raw);
  cg::cluster_group cl = cg::this_cluster();
  const uint32_t rank = cl.block_rank(), ranks = cl.num_blocks();
  const uint32_t per = (g + ranks - 1) / ranks;
  const uint32_t row0 = min(g, rank * per), row1 = min(g, row0 + per);
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t tx = tid & 15u, ty = tid >> 4;
  if (tid == 0) sh.bad = 0;

  // |block|_F over this CTA's rows (summed over the cluster below).
  {
    double ss = 0.0;
    for (uint32_t c = warp; c < w; c += kXbThreads / 32)
      for (uint32_t r = row0 + (tid & 31u); r < row1; r += 32) {
        const double v = block[(uint64_t)c * g + r];
        ss = fma(v, v, ss);
      }
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xFFFFFFFFu, ss, o);
    if ((tid & 31u) == 0) sh.red[warp] = ss;
    __syncthreads();
    if (tid == 0) {
      double t = 0.0;
      for (int i = 0; i < kXbThreads / 32; ++i) t += sh.red[i];
      sh.norm = t;
    }
  }

  for (int round = 0; round < 3; ++round) {
    const double* a = round == 0 ? rest : q;
    // The Gram matrix over this CTA's rows: group `grp` takes every fourth staged row.
    const uint32_t grp = tid >> 6, gx = tid & 7u, gy = (tid >> 3) & 7u;
    double acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.0;
    for (uint32_t r0 = row0; r0 < row1; r0 += kXbRows) {
      __syncthreads();
      stage_rows(sh, a, g, w, r0, row1);
      __syncthreads();
      const uint32_t n = min(kXbRows, row1 - r0);
      for (uint32_t r = grp; r < n; r += 4) {
        double x[8], y[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = sh.rows[r][gy + 8 * i];
#pragma unroll
        for (int i = 0; i < 8; ++i) y[i] = sh.rows[r][gx + 8 * i];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i][j] = fma(x[i], y[j], acc[i][j]);
      }
    }
    __syncthreads();
    for (uint32_t t = 0; t < 4; ++t) {
      if (grp == t) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            double* at = &sh.g.part[(gy + 8 * i) * kW + gx + 8 * j];
            *at = t == 0 ? acc[i][j] : *at + acc[i][j];
          }
      }
      __syncthreads();
    }
    cl.sync();
    // The cluster's sum, a slice of the entries a CTA, handed to every CTA.
    for (uint32_t x = rank * kXbThreads + tid; x < kW * kW; x += ranks * kXbThreads) {
      double s = 0.0;
      for (uint32_t p = 0; p < ranks; ++p) s += *cl.map_shared_rank(&sh.g.part[x], p);
      for (uint32_t p = 0; p < ranks; ++p) *cl.map_shared_rank(&sh.g.full[x], p) = s;
    }
    if (round == 0 && rank == 0 && tid == 0) {
      double t = 0.0;
      for (uint32_t p = 0; p < ranks; ++p) t += *cl.map_shared_rank(&sh.norm, p);
      out[w] = sqrt(t);
    }
    cl.sync();

    // R^T R = G (+ shift * trace(G) in the first round; columns past w the identity). Each
    // thread holds the entries (ty + 16 i, tx + 16 j); a step publishes the pivot's row.
    double diag = 0.0;
    if (round == 0) {
      for (uint32_t j = 0; j < w; ++j) diag += sh.g.full[j * kW + j];
      diag *= shift;
    }
    double m[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t r = ty + 16 * i, c = tx + 16 * j;
        double v = r < w && c < w ? sh.g.full[r * kW + c] : 0.0;
        if (r == c) v = r < w ? v + diag : 1.0;
        m[i][j] = v;
      }
    bool ok = true;
#pragma unroll
    for (int jb = 0; jb < 4; ++jb) {
      for (uint32_t jj = 0; jj < 16; ++jj) {
        const uint32_t j = jb * 16 + jj;
        if (ty == jj) {
#pragma unroll
          for (int c = 0; c < 4; ++c) sh.r[j][tx + 16 * c] = m[jb][c];
        }
        __syncthreads();
        const double d = sh.r[j][j];
        ok = ok && d > 0.0;
        const double inv = 1.0 / d;
        double x[4], y[4];
#pragma unroll
        for (int i = jb; i < 4; ++i) x[i] = sh.r[j][ty + 16 * i];
#pragma unroll
        for (int i = jb; i < 4; ++i) y[i] = sh.r[j][tx + 16 * i] * inv;
#pragma unroll
        for (int i = jb; i < 4; ++i)
#pragma unroll
          for (int c = jb; c < 4; ++c) m[i][c] = fma(-x[i], y[c], m[i][c]);
      }
    }
    __syncthreads();
    if (!ok) sh.bad = 1;  // the same for every thread
    // Row j of R = row j of the trailing matrix / sqrt(d_j), zeros below the diagonal.
    if (tid < kW) sh.dinv[tid] = 1.0 / sqrt(sh.r[tid][tid]);
    __syncthreads();
    for (uint32_t x = tid; x < kW * kW; x += kXbThreads) {
      const uint32_t j = x / kW, c = x % kW;
      sh.r[j][c] = c >= j ? sh.r[j][c] * sh.dinv[j] : 0.0;
    }
    __syncthreads();
    // rtot = R rtot (rank 0; R itself in the first round).
    if (rank == 0) {
      double(*dst)[kW] = sh.rtot[round & 1];
      const double(*src)[kW] = sh.rtot[(round & 1) ^ 1];
      if (round == 0) {
        for (uint32_t x = tid; x < kW * kW; x += kXbThreads) dst[x / kW][x % kW] = sh.r[x / kW][x % kW];
      } else {
        double t[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) t[i][c] = 0.0;
        for (uint32_t k = 0; k < w; ++k) {
          double x[4], y[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) x[i] = sh.r[ty + 16 * i][k];
#pragma unroll
          for (int i = 0; i < 4; ++i) y[i] = src[k][tx + 16 * i];
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) t[i][c] = fma(x[i], y[c], t[i][c]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) dst[ty + 16 * i][tx + 16 * c] = t[i][c];
      }
    }
    __syncthreads();
    // Q = A R^-1 on this CTA's rows, a thread a row, 128 rows a pass.
    for (uint32_t r0 = row0; r0 < row1; r0 += kXbSolve) {
      if (tid < kXbSolve && r0 + tid < row1) {
        const uint32_t row = r0 + tid;
        for (uint32_t jb = 0; jb < w; jb += 8) {
          double b[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) b[i] = jb + i < w ? a[(uint64_t)(jb + i) * g + row] : 0.0;
          for (uint32_t k = 0; k < jb; ++k) {
            const double xk = sh.x[k][tid];
#pragma unroll
            for (int i = 0; i < 8; ++i) b[i] = fma(-xk, sh.r[k][jb + i], b[i]);
          }
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            b[i] *= sh.dinv[jb + i];
#pragma unroll
            for (int k = i + 1; k < 8; ++k) b[k] = fma(-b[i], sh.r[jb + i][jb + k], b[k]);
            sh.x[jb + i][tid] = b[i];
            if (jb + i < w) q[(uint64_t)(jb + i) * g + row] = b[i];
          }
        }
      }
    }
    __syncthreads();
  }

  // The SVD of R (rank 0), then U = Q U_R on this CTA's rows.
  if (rank == 0) {
    const double(*r)[kW] = sh.rtot[0];
    for (uint32_t x = tid; x < kW * kW; x += kXbThreads) {
      const uint32_t c = x / kW, i = x % kW;
      sh.jac.a[c][i] = c < w && i < w ? r[i][c] : 0.0;
    }
    __syncthreads();
    const int failed = jacobi_square(sh.jac, w, out);
    for (uint32_t x = tid; x < kW * kW; x += kXbThreads) {
      const uint32_t i = x / kW, c = x % kW;
      double v = 0.0;
      if (c < w && i < w) {
        const uint32_t o = sh.jac.order[c];
        const double nv = sh.jac.norms[o];
        v = nv > 0.0 ? sh.jac.a[o][i] / nv : 0.0;
      }
      sh.rtot[1][i][c] = v;
    }
    if (tid == 0) out[w + 1] = failed || sh.bad ? 1.0 : 0.0;
  }
  cl.sync();
  for (uint32_t x = tid; x < kW * kW; x += kXbThreads)
    sh.r[x / kW][x % kW] = *cl.map_shared_rank(&sh.rtot[1][x / kW][x % kW], 0);
  cl.sync();  // rank 0's shared memory is read until here
  for (uint32_t r0 = row0; r0 < row1; r0 += kXbRows) {
    __syncthreads();
    stage_rows(sh, q, g, w, r0, row1);
    __syncthreads();
    double t[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int c = 0; c < 4; ++c) t[i][c] = 0.0;
    // Rows along tx (the writes of a column are consecutive).
    for (uint32_t k = 0; k < w; ++k) {
      double x[4], y[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = sh.rows[tx + 16 * i][k];
#pragma unroll
      for (int i = 0; i < 4; ++i) y[i] = sh.r[k][ty + 16 * i];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) t[i][c] = fma(x[i], y[c], t[i][c]);
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t r = r0 + tx + 16 * i, col = ty + 16 * c;
        if (r < row1 && col < w) u[(uint64_t)col * g + r] = t[i][c];
      }
  }
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
    sh.a[c][r] = c < w && r <= c ? colp(c)[r] : 0.0;
  }
  __syncthreads();
  const int failed = jacobi_square(sh, w, out);
  if (threadIdx.x == 0) out[w + 1] = failed ? 1.0 : 0.0;
  // U = Q [U_R; 0]: start from U_R's unit columns, apply H_{w-1}, ..., H_0.
  for (uint64_t x = threadIdx.x; x < (uint64_t)g * w; x += blockDim.x) {
    uint32_t c = (uint32_t)(x / g), r = (uint32_t)(x % g);
    double nv = sh.norms[sh.order[c]];
    u[x] = (r < w && nv > 0.0) ? sh.a[sh.order[c]][r] / nv : 0.0;
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

// The CTAs of a cluster launch of extend_svd_kernel on the current device: 16 where the
// device can hold such a cluster, else the portable 8.
uint32_t xb_cluster(int device) {
  static std::mutex mu;
  static std::vector<uint32_t> known;
  std::lock_guard<std::mutex> lock(mu);
  if ((size_t)device >= known.size()) known.resize((size_t)device + 1, 0);
  if (!known[device]) {
    KG_CUDA(cudaFuncSetAttribute(extend_svd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(XbShared)));
    KG_CUDA(cudaFuncSetAttribute(extend_svd_kernel,
                                 cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(kXbCluster);
    cfg.blockDim = dim3(kXbThreads);
    cfg.dynamicSmemBytes = sizeof(XbShared);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = kXbCluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, extend_svd_kernel, &cfg) != cudaSuccess) {
      cudaGetLastError();
      fit = 0;
    }
    known[device] = fit > 0 ? kXbCluster : 8;
  }
  return known[device];
}

}  // namespace

void extend_svd(const double* block, const double* rest, uint32_t g, uint32_t w, double* q,
                double* u, double* out, cudaStream_t s) {
  static_assert(sizeof(XbShared) <= 227 * 1024, "extend_svd shared memory");
  int device = 0;
  KG_CUDA(cudaGetDevice(&device));
  const uint32_t ctas = xb_cluster(device);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(ctas);
  cfg.blockDim = dim3(kXbThreads);
  cfg.dynamicSmemBytes = sizeof(XbShared);
  cfg.stream = s;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = ctas;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  const double shift = 11.0 * ((double)g * w + (double)w * (w + 1)) * 0x1p-53;
  KG_CUDA(cudaLaunchKernelEx(&cfg, extend_svd_kernel, block, rest, g, w, shift, q, u, out));
  KG_LAUNCH_CHECK();
}

void qr_svd(double* b, uint32_t g, uint32_t w, double* u, double* out, cudaStream_t s) {
  qr_svd_kernel<<<1, 1024, 0, s>>>(b, g, w, u, out);
  KG_LAUNCH_CHECK();
}

}  // namespace kg
