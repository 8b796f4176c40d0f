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
__device__ __forceinline__ float rsqrt_approx(float v) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
// t = sign(z) / (|z| + sqrt(1 + z^2)).
__device__ __forceinline__ float small_tangent(float z) {
  const float t = rcp_approx(fabsf(z) + sqrt_approx(fmaf(z, z, 1.0f)));
  return z >= 0.0f ? t : -t;
}

constexpr int kJacobiThreads = 256;  // 32 pairs of 8 lanes
constexpr int kJacobiLd = kW + 2;    // a column's stride: 16-byte aligned

struct JacobiShared {
  double a[kW][kJacobiLd];  // by column: the matrix, then U diag(sigma)
  double norms[kW];         // squared norms while rotating, then norms
  double red[32];
  uint32_t order[kW];
};

// A column's rows of one of its 8 lanes: 16 x + 2 lane and the row after it (a 16-byte
// access whose 8 lanes cover 128 bytes: free of bank conflicts whatever the columns).
struct JacobiRows {
  double2 v[kW / 16];
  __device__ __forceinline__ void load(const double* col, uint32_t lane) {
#pragma unroll
    for (int x = 0; x < (int)kW / 16; ++x)
      v[x] = *reinterpret_cast<const double2*>(col + 16 * x + 2 * lane);
  }
  __device__ __forceinline__ void store(double* col, uint32_t lane) const {
#pragma unroll
    for (int x = 0; x < (int)kW / 16; ++x)
      *reinterpret_cast<double2*>(col + 16 * x + 2 * lane) = v[x];
  }
  __device__ __forceinline__ double dot(const JacobiRows& o) const {
    double p = 0.0, q = 0.0;
#pragma unroll
    for (int x = 0; x < (int)kW / 16; ++x) {
      p = fma(v[x].x, o.v[x].x, p);
      q = fma(v[x].y, o.v[x].y, q);
    }
    p += q;
#pragma unroll
    for (int o8 = 4; o8; o8 >>= 1) p += __shfl_xor_sync(0xFFFFFFFFu, p, o8);
    return p;
  }
};

// Hestenes' one-sided Jacobi on the w columns of the w x w matrix sh.a (everything past
// them zero, w <= 64): pairs orthogonal to 1e-15 of their norms; sh.a becomes U diag(sigma)
// / 2^e, sh.norms its column norms, sh.order the columns by descending norm (ties to the
// lower column), sigma[] the singular values in that order. Returns 0, or 1 if 60 sweeps
// did not converge. All threads of the CTA (at least 256) call it; the first 256 work.
//
// A block's 60 columns take 10 to 12 sweeps, so a round of 32 disjoint pairs is
// everything. A pair is 8 lanes of 8 rows. The sweep's order halves the columns again and
// again: at span h, column i of the lower half of each 2h columns meets the h columns of
// the upper half in turn, staying in registers while those pass through shared memory (one
// column read and written a round instead of two). The squared norms follow the rotations
// (al - t ga, be + t ga; summed afresh every sweep), so a round has one dot product. The
// angle comes from f32 approximations (the pair keeps a 2^-20th of its product, which the
// next sweep takes); c = 1 / sqrt(1 + t^2) and s = c t hold c^2 + s^2 = 1 to f64.
// Latency bounds it: a round is a chain of a shared-memory read, the dot product and three
// shuffles, the angle, the update and a barrier, about 880 cycles (a warp a pair with
// three dot products and IEEE division, square root and hypot: 3,900; eight lanes a pair
// with both columns passing through shared memory: 1,400).
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

  const uint32_t span = w <= 16 ? 16 : w <= 32 ? 32 : 64;  // columns taking part
  const bool mine = work && pair < span / 2;
  int sweep = 0;
  for (; sweep < 60; ++sweep) {
    if (work) {
      for (uint32_t c = pair; c < span; c += kJacobiThreads / 8) {
        JacobiRows r;
        r.load(sh.a[c], lane);
        const double n = r.dot(r);
        if (lane == 0) sh.norms[c] = n;
      }
    }
    __syncthreads();
    int rotated = 0;
    for (uint32_t h = span / 2; h; h >>= 1) {
      const uint32_t i = pair & (h - 1), base = mine ? (pair & ~(h - 1)) * 2 : 0;
      JacobiRows u;
      double al = 0.0;
      if (work) {
        u.load(sh.a[base + i], lane);
        al = sh.norms[base + i];
      }
      for (uint32_t t = 0; t < h; ++t) {
        if (work) {  // whole warps
          const uint32_t j = base + h + ((i + t) & (h - 1));
          JacobiRows v;
          v.load(sh.a[j], lane);
          const double be = sh.norms[j];
          const double ga = u.dot(v);
          if (mine && al > 0.0 && be > 0.0 && ga * ga > 1e-30 * (al * be)) {
            const double gap = be - al;
            const float z = 0.5f * (float)gap * rcp_approx((float)ga);
            float tf = small_tangent(z);
            double tn = (double)tf;
            double y = (double)rsqrt_approx(fmaf(tf, tf, 1.0f));
            if (!(fabsf(z) < 1e8f)) {
              // Columns of very different norms, or products past f32's range:
              // t = 1 / (2 zeta).
              const double zeta = 0.5 * gap * rcp_approx(ga);
              tn = fabs(zeta) > 1e8 ? rcp_approx(2.0 * zeta) : (double)small_tangent((float)zeta);
              y = (double)rsqrt_approx(fmaf((float)tn, (float)tn, 1.0f));
            }
            // 1 / sqrt(1 + t^2) from its f32 approximation by one third-order step.
            const double x1 = fma(tn, tn, 1.0);
            const double er = fma(-x1 * y, y, 1.0);
            const double c = fma(y * er, fma(er, 0.375, 0.5), y), s = c * tn;
#pragma unroll
            for (int x = 0; x < (int)kW / 16; ++x) {
              const double2 p = u.v[x], q = v.v[x];
              u.v[x].x = fma(c, p.x, -(s * q.x));
              u.v[x].y = fma(c, p.y, -(s * q.y));
              v.v[x].x = fma(s, p.x, c * q.x);
              v.v[x].y = fma(s, p.y, c * q.y);
            }
            v.store(sh.a[j], lane);
            if (lane == 0) sh.norms[j] = fma(tn, ga, be);
            al = fma(-tn, ga, al);
            rotated = 1;
          }
        }
        // Spans of up to four pairs pass their columns inside one warp.
        if (h > 4)
          __syncthreads();
        else
          __syncwarp();
      }
      if (mine) {
        u.store(sh.a[base + i], lane);
        if (lane == 0) sh.norms[base + i] = al;
      }
      __syncthreads();
    }
    if (!__syncthreads_or(rotated)) break;
  }
  if (work) {
    for (uint32_t c = pair; c < kW; c += kJacobiThreads / 8) {
      JacobiRows r;
      r.load(sh.a[c], lane);
      const double n = r.dot(r);
      if (lane == 0) sh.norms[c] = sqrt(n);
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
  const uint32_t r = threadIdx.x % kXbRows, c0 = threadIdx.x / kXbRows;
  double v[kW * kXbRows / kXbThreads];
#pragma unroll
  for (int i = 0; i < (int)(kW * kXbRows / kXbThreads); ++i) {
    const uint32_t c = c0 + i * (kXbThreads / kXbRows);
    v[i] = r0 + r < r1 && c < w ? a[(uint64_t)c * g + r0 + r] : 0.0;
  }
#pragma unroll
  for (int i = 0; i < (int)(kW * kXbRows / kXbThreads); ++i)
    sh.rows[r][c0 + i * (kXbThreads / kXbRows)] = v[i];
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
// Latency bounds it (a 2,000 x 60 block is 1 MB, 3 x 7 Mflop): 0.43 ms on 2,000 x 60, of
// it 0.32 ms in the Jacobi. The same steps as separate launches (three Gram GEMMs, factors
// and solves of cuBLAS and one-CTA kernels, the SVD, the last GEMM, two norms read by the
// host) took 2.02 ms a block.
__global__ void __launch_bounds__(kXbThreads, 1)
extend_svd_kernel(const double* __restrict__ block, const double* __restrict__ rest, uint32_t g,
                  uint32_t w, double shift, double* q, double* __restrict__ u, double* ur,
                  double* out) {
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
    // Q = A R^-1 on this CTA's rows, a thread a row, 128 rows a pass, the next columns'
    // loads ahead of the current ones' arithmetic. Rank 0's other 128 threads make
    // rtot = R rtot meanwhile (R itself in the first round).
    if (tid < kXbSolve) {
      for (uint32_t row = row0 + tid; row < row1; row += kXbSolve) {
        double nb[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) nb[i] = (uint32_t)i < w ? a[(uint64_t)i * g + row] : 0.0;
        for (uint32_t jb = 0; jb < w; jb += 8) {
          double b[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            b[i] = nb[i];
            const uint32_t c = jb + 8 + i;
            nb[i] = c < w ? a[(uint64_t)c * g + row] : 0.0;
          }
          for (uint32_t k0 = 0; k0 < jb; k0 += 8) {
            double xk[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) xk[k] = sh.x[k0 + k][tid];
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
              for (int i = 0; i < 8; ++i) b[i] = fma(-xk[k], sh.r[k0 + k][jb + i], b[i]);
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
    } else if (rank == 0) {
      double(*dst)[kW] = sh.rtot[round & 1];
      const double(*src)[kW] = sh.rtot[(round & 1) ^ 1];
      const uint32_t t2 = tid - kXbSolve;
      if (round == 0) {
        for (uint32_t x = t2; x < kW * kW; x += kXbThreads - kXbSolve)
          dst[x / kW][x % kW] = sh.r[x / kW][x % kW];
      } else {
        const uint32_t ry = t2 >> 4;
        double t[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) t[i][c] = 0.0;
        for (uint32_t k = 0; k < w; ++k) {
          double x[8], y[4];
#pragma unroll
          for (int i = 0; i < 8; ++i) x[i] = sh.r[ry + 8 * i][k];
#pragma unroll
          for (int i = 0; i < 4; ++i) y[i] = src[k][tx + 16 * i];
#pragma unroll
          for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) t[i][c] = fma(x[i], y[c], t[i][c]);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int c = 0; c < 4; ++c) dst[ry + 8 * i][tx + 16 * c] = t[i][c];
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
      ur[x] = v;
    }
    if (tid == 0) out[w + 1] = failed || sh.bad ? 1.0 : 0.0;
  }
  // U_R goes through global memory (16 CTAs reading rank 0's shared memory queue there).
  cl.sync();
  for (uint32_t x = tid; x < kW * kW; x += kXbThreads) sh.r[x / kW][x % kW] = ur[x];
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
  // The first round's shift (times the trace): 11 (g w + w (w + 1)) u.
  const double shift = 11.0 * ((double)g * w + (double)w * (w + 1)) * 0x1p-53;
  KG_CUDA(cudaLaunchKernelEx(&cfg, extend_svd_kernel, block, rest, g, w, shift, q,
                             u, q + (uint64_t)g * w, out));
  KG_LAUNCH_CHECK();
}

void qr_svd(double* b, uint32_t g, uint32_t w, double* u, double* out, cudaStream_t s) {
  qr_svd_kernel<<<1, 1024, 0, s>>>(b, g, w, u, out);
  KG_LAUNCH_CHECK();
}

}  // namespace kg
