/*
 * lgb_factor.cu -- batched per-patch collocation assembly, Cholesky and solve in FP64 precision.
 *
 * Replaces the lazy patch set-up and solve of LagRBF_PartitionsSetUp (src/partitions/partition.c:
 * 384-478): PartitionAssembleRBFMatrix (partition_solve.c:47-95, partition_asmb_avx512.c:119-198),
 * MatCholeskyFactor / KSP preonly+PCCHOLESKY (partition_factor.c:37-55, partition_ksp.c:115-172) and
 * the RHS gather + MatMatSolve (partition_factor.c:57-135).
 *
 * Patches are queued by size class (LGB_NCLS classes of sizes up to 32, 64, ..., 2048 and beyond);
 * each class is one launch of a persistent grid over its work list (graph-capturable with a
 * device-side count).  Patches of up to 64 points run k_factor<NT> (CTA size from the measured table
 * lgb_factor_tune.h): the matrix is assembled column-major into a per-CTA workspace slot, factored in
 * FP64 in panels of CHOL_NB columns, and solved.  Larger patches run k_factor_blk, whose updates are
 * formed on the tensor cores and the integer pipe (below), and k_solve_blk where only the field values
 * changed and the factor is kept (A_FACTOR / A_KSP).  The collocation systems are ill-conditioned: the
 * error of the coefficients against extended precision is that of an FP64 factorisation or smaller
 * (0.5-1.0 of it over patches of 196-343 points and kappa up to 1e9).  A non-positive pivot sets
 * ctrl->factor_error (1-based row) and leaves the patch not set up; no trap, no abort.  Factors are
 * "prepared" for the solves (reciprocal diagonal and scaled diagonal blocks, below); the first solve
 * and re-solves run the same code on the same values.
 *
 * Roofline: GB300 issues 2 DFMA per clock per SM, which bounds an FP64 factorisation at m^3 / 6 / 2
 * clocks per patch.  Measured: 1,728 patches of up to 729 points 148.9 ms in FP64 throughout, 24.9 ms
 * with k_factor_blk (bound by the tensor cores' 21 digit products, then by the latency of the pivots);
 * re-solve of 4,096 patches with kept factors 7.7 ms, then 3.7 ms (bound by reading the factor).
 */
#include "lgb_common.cuh"
#include "lgb_fx.cuh"
#include "lgb_optin.cuh"

#define CHOL_NB 16 /* columns per Cholesky panel */

struct FactorParams {
  lgb_geom g;
  int F, keep;
  const int *cstart;
  const double *xs, *fs;
  const int *pm, *slot, *work;  /* work: the nodes of one patch-size class, *nwork of them */
  const int *nwork;
  const long long *coff, *foff;
  int *setup, *solved;
  double *c64, *fac, *ws;
  float *c32;
  int *cexp;
  long long ws_stride;
  lgb_ctrl *ctrl;
  int fixed;       /* blocked kernel: kernel values in fixed point */
  double *kappa;   /* non-NULL: 1-norm condition estimate of every factored patch, by node */
};


/* Column j of the lower factor from its diagonal element down: packed column-major (m(m+1)/2,
   the kept factors) or the full column-major workspace.  L(i, j) = L[lbase(j) + (i - j)]. */
template <bool PACKED>
__device__ __forceinline__ long long lbase(int m, int j)
{
  return PACKED ? (long long)j * m - ((long long)j * (j - 1)) / 2 : (long long)j * m + j;
}
template <bool PACKED>
__device__ __forceinline__ long long lstep(int m, int j)
{
  return PACKED ? (long long)(m - j) : (long long)m + 1; /* base(j + 1) - base(j) */
}

/* The factor as the solves read it ("prepared"): the 32 x 32 diagonal blocks hold the reciprocal
   1 / L(j, j) on the diagonal and M(i, j) = L(i, j) / L(j, j) below it; every other entry is
   L(i, j).  With M the substitutions inside a diagonal block are fused multiply-adds only:
     forward   u_i = b_i - sum_{k<i} M(i,k) u_k,              y_i = u_i / L(i,i)
     backward  w_i = y_i / L(i,i) - sum_{k>i} M(k,i) x_k,      x_i = w_i
   (L(i,k) y_k = M(i,k) u_k and L(k,i) x_k / L(i,i) = M(k,i) x_k), which halves the FP64
   instructions of the block substitutions, the serial part of the solve. */
template <bool PACKED>
__device__ void prepare_diag_blocks(double *L, int m)
{
  for (int j = threadIdx.x; j < m; j += blockDim.x) {
    const long long b = lbase<PACKED>(m, j);
    const double d = L[b];
    const int iend = min((j / 32 + 1) * 32, m);
    for (int i = j + 1; i < iend; i++) L[b + (i - j)] /= d;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < m; j += blockDim.x) {
    const long long b = lbase<PACKED>(m, j);
    L[b] = 1.0 / L[b];
  }
  __syncthreads();
}

/* D[r * 33 + c] = prepared diagonal block entry (j0 + r, j0 + c), r >= c; column-wise reads. */
template <bool PACKED>
__device__ __forceinline__ void stage_diag(const double *L, int m, int j0, int nb, double *D)
{
  for (int t = threadIdx.x; t < nb * nb; t += blockDim.x) {
    const int c = t / nb, r = t - c * nb;
    if (r >= c) D[r * 33 + c] = L[lbase<PACKED>(m, j0 + c) + (r - c)];
  }
}

/* Solves L L^T X = B in place for FC (1..4) columns of B (B[q*m + i]) with the prepared factor,
   in blocks of 32 rows.  Each diagonal block is staged in shared memory (D, 32 x 33) and
   substituted by one warp with shuffles, every lane issuing the same fused multiply-add (zero
   multiplier where a lane has nothing to subtract); the block's solution is kept in shared memory
   (Y, 4 x 32) and the other rows are updated by all threads, each factor element read once per
   block for all FC right-hand sides.  Forward: rows below the block, L(i, j) read down columns
   (coalesced).  Backward: rows above the block, x_i -= sum_r L(i0 + r, i) x_r, each thread
   reading 32 consecutive entries of its own column.  Only FP64 fused multiply-adds and one
   multiplication per block and right-hand side; no reductions. */
template <bool PACKED, int FC>
__device__ void chol_solve_group(const double *__restrict__ L, int m, double *B0, double *D, double *Y)
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (m + 31) / 32;
  for (int kb = 0; kb < nblk; kb++) {
    const int j0 = kb * 32, nb = min(32, m - j0);
    stage_diag<PACKED>(L, m, j0, nb, D);
    __syncthreads();
    if (warp == 0) {
      double u[FC];
#pragma unroll
      for (int q = 0; q < FC; q++) u[q] = (lane < nb) ? B0[(size_t)q * m + j0 + lane] : 0.0;
      for (int jj = 0; jj < nb - 1; jj++) {
        const double mij = (lane > jj && lane < nb) ? D[lane * 33 + jj] : 0.0;
#pragma unroll
        for (int q = 0; q < FC; q++) u[q] = fma(-mij, __shfl_sync(0xffffffffu, u[q], jj), u[q]);
      }
      const double rl = (lane < nb) ? D[lane * 33 + lane] : 0.0;
#pragma unroll
      for (int q = 0; q < FC; q++) {
        const double y = u[q] * rl;
        Y[q * 32 + lane] = y;
        if (lane < nb) B0[(size_t)q * m + j0 + lane] = y;
      }
    }
    __syncthreads();
    const long long b0 = lbase<PACKED>(m, j0);
    for (int i = j0 + nb + tid; i < m; i += blockDim.x) {
      double acc[FC];
#pragma unroll
      for (int q = 0; q < FC; q++) acc[q] = B0[(size_t)q * m + i];
      long long cb = b0 - j0; /* element (i, j) of column j at cb + i */
#pragma unroll 8
      for (int jj = 0; jj < nb; jj++) {
        const double l = L[cb + i - jj];
#pragma unroll
        for (int q = 0; q < FC; q++) acc[q] = fma(-l, Y[q * 32 + jj], acc[q]);
        cb += lstep<PACKED>(m, j0 + jj);
      }
#pragma unroll
      for (int q = 0; q < FC; q++) B0[(size_t)q * m + i] = acc[q];
    }
    __syncthreads();
  }
  for (int kb = nblk - 1; kb >= 0; kb--) {
    const int i0 = kb * 32, nb = min(32, m - i0);
    stage_diag<PACKED>(L, m, i0, nb, D);
    __syncthreads();
    if (warp == 0) {
      const double rl = (lane < nb) ? D[lane * 33 + lane] : 0.0;
      double w[FC];
#pragma unroll
      for (int q = 0; q < FC; q++) w[q] = ((lane < nb) ? B0[(size_t)q * m + i0 + lane] : 0.0) * rl;
      for (int ii = nb - 1; ii >= 1; ii--) {
        const double mi = (lane < ii) ? D[ii * 33 + lane] : 0.0;
#pragma unroll
        for (int q = 0; q < FC; q++) w[q] = fma(-mi, __shfl_sync(0xffffffffu, w[q], ii), w[q]);
      }
#pragma unroll
      for (int q = 0; q < FC; q++) {
        Y[q * 32 + lane] = w[q];
        if (lane < nb) B0[(size_t)q * m + i0 + lane] = w[q];
      }
    }
    __syncthreads();
    for (int i = tid; i < i0; i += blockDim.x) {
      double acc[FC];
#pragma unroll
      for (int q = 0; q < FC; q++) acc[q] = B0[(size_t)q * m + i];
      const double *ci = L + lbase<PACKED>(m, i) + (i0 - i); /* L(i0 + r, i) = ci[r] */
#pragma unroll 8
      for (int r = 0; r < nb; r++) {
        const double l = ci[r];
#pragma unroll
        for (int q = 0; q < FC; q++) acc[q] = fma(-l, Y[q * 32 + r], acc[q]);
      }
#pragma unroll
      for (int q = 0; q < FC; q++) B0[(size_t)q * m + i] = acc[q];
    }
    __syncthreads();
  }
}

/* All F right-hand sides of B (B[f*m + i]), four at a time. */
template <bool PACKED>
__device__ void chol_solve(const double *L, int m, int F, double *B, double *D, double *Y)
{
  for (int f0 = 0; f0 < F; f0 += 4) {
    double *B0 = B + (size_t)f0 * m;
    switch (min(4, F - f0)) {
    case 1: chol_solve_group<PACKED, 1>(L, m, B0, D, Y); break;
    case 2: chol_solve_group<PACKED, 2>(L, m, B0, D, Y); break;
    case 3: chol_solve_group<PACKED, 3>(L, m, B0, D, Y); break;
    default: chol_solve_group<PACKED, 4>(L, m, B0, D, Y); break;
    }
  }
}

/* ---- block reductions (blockDim.x threads; red: 32 doubles of shared memory) ---- */
__device__ double blk_reduce(double v, double *red, bool is_max)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int o = 16; o > 0; o >>= 1) {
    const double u = __shfl_xor_sync(0xffffffffu, v, o);
    v = is_max ? fmax(v, u) : v + u;
  }
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double r = red[0];
  for (int w = 1; w < nw; w++) r = is_max ? fmax(r, red[w]) : r + red[w];
  return r;
}
/* Largest |z_i| and its first index. */
__device__ double blk_argmax_abs(const double *z, int m, int *idx, double *red, int *ired)
{
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  double best = -1.0;
  int bi = 0;
  for (int i = threadIdx.x; i < m; i += blockDim.x)
    if (fabs(z[i]) > best) { best = fabs(z[i]); bi = i; }
  for (int o = 16; o > 0; o >>= 1) {
    const double u = __shfl_xor_sync(0xffffffffu, best, o);
    const int ui = __shfl_xor_sync(0xffffffffu, bi, o);
    if (u > best || (u == best && ui < bi)) { best = u; bi = ui; }
  }
  __syncthreads();
  if (lane == 0) { red[warp] = best; ired[warp] = bi; }
  __syncthreads();
  best = red[0];
  bi = ired[0];
  for (int w = 1; w < nw; w++)
    if (red[w] > best || (red[w] == best && ired[w] < bi)) { best = red[w]; bi = ired[w]; }
  *idx = bi;
  return best;
}

/* ||A^-1||_1 estimate from the prepared factor in the workspace (Hager's method as refined by Higham:
   N. J. Higham, "FORTRAN codes for estimating the one-norm of a real or complex matrix", ACM TOMS 14
   (1988); A symmetric, so A^-T = A^-1): at most five iterations of x -> sign(A^-1 x) -> e_j, then
   the alternating test vector x_i = (-1)^i (1 + i/(m-1)).  v, u: two workspace vectors of m. */
template <typename Solve>
__device__ double inv_norm1_estimate(int m, double *v, double *u, double *red, int *ired, Solve solve)
{
  const int tid = threadIdx.x;
  for (int i = tid; i < m; i += blockDim.x) v[i] = 1.0 / m;
  __syncthreads();
  solve(v);
  double s = 0.0;
  for (int i = tid; i < m; i += blockDim.x) s += fabs(v[i]);
  double est = blk_reduce(s, red, false);
  int jprev = -1;
  for (int it = 0; it < 5; it++) {
    for (int i = tid; i < m; i += blockDim.x) u[i] = (v[i] >= 0.0) ? 1.0 : -1.0;
    __syncthreads();
    solve(u);
    int j;
    const double zmax = blk_argmax_abs(u, m, &j, red, ired);
    double ztx;
    if (jprev < 0) {
      double t = 0.0;
      for (int i = tid; i < m; i += blockDim.x) t += u[i];
      ztx = blk_reduce(t, red, false) / m;
    } else {
      ztx = u[jprev];
    }
    if (it > 0 && zmax <= ztx) break;
    for (int i = tid; i < m; i += blockDim.x) v[i] = (i == j) ? 1.0 : 0.0;
    __syncthreads();
    solve(v);
    s = 0.0;
    for (int i = tid; i < m; i += blockDim.x) s += fabs(v[i]);
    const double e2 = blk_reduce(s, red, false);
    if (e2 <= est) break;
    est = e2;
    jprev = j;
  }
  for (int i = tid; i < m; i += blockDim.x) v[i] = ((i & 1) ? -1.0 : 1.0) * (1.0 + (m > 1 ? (double)i / (m - 1) : 0.0));
  __syncthreads();
  solve(v);
  s = 0.0;
  for (int i = tid; i < m; i += blockDim.x) s += fabs(v[i]);
  const double alt = 2.0 * blk_reduce(s, red, false) / (3.0 * m);
  return fmax(est, alt);
}

/* The adjacent cells of a patch node (thread 0): first sorted point, count and offset in the patch. */
struct PatchCells {
  int cstart[8], cnt[8], off[8];
};
__device__ void patch_cells(const FactorParams &P, int node, PatchCells &C)
{
  const lgb_geom &g = P.g;
  int nxy = g.n[0] * g.n[1];
  int l = node / nxy, r = node - l * nxy, j = r / g.n[0], i = r - j * g.n[0];
  for (int s = 0; s < 8; s++) {
    int dx = s & 1, dy = (s >> 1) & 1, dz = (s >> 2) & 1;
    int ci = i - 1 + dx, cj = j - 1 + dy, cl = (g.dim == 3) ? (l - 1 + dz) : 0;
    bool ok = (g.dim == 3 || dz == 0) && ci >= 0 && ci < g.nc[0] && cj >= 0 && cj < g.nc[1] && cl >= 0 &&
              cl < g.nc[2];
    int c = ok ? ci + cj * g.nc[0] + cl * g.nc[0] * g.nc[1] : 0;
    C.cstart[s] = ok ? P.cstart[c] : 0;
    C.cnt[s] = ok ? P.cstart[c + 1] - P.cstart[c] : 0;
    C.off[s] = P.slot[node * 8 + s];
  }
}

/* The patch points (reference patch order) into X[m*dim] and their values into B[f*m + q]. */
__device__ void patch_gather(const FactorParams &P, const PatchCells &C, int m, double *X, double *B)
{
  const int dim = P.g.dim;
  for (int q = threadIdx.x; q < m; q += blockDim.x) {
    int s = 0;
    while (s < 7 && q >= C.off[s] + C.cnt[s]) s++;
    int src = C.cstart[s] + (q - C.off[s]);
    for (int d = 0; d < dim; d++) X[(size_t)q * dim + d] = P.xs[(size_t)src * dim + d];
    for (int f = 0; f < P.F; f++) B[(size_t)f * m + q] = P.fs[(size_t)src * P.F + f];
  }
}

/* The coefficients of a patch, [point][field], in both precisions, and its flags. */
__device__ void patch_store(const FactorParams &P, int node, int m, const double *B)
{
  const int F = P.F;
  const long long c0 = P.coff[node];
  for (int q = threadIdx.x; q < m; q += blockDim.x)
    for (int f = 0; f < F; f++) {
      double v = B[(size_t)f * m + q];
      P.c64[(size_t)(c0 + q) * F + f] = v;
      P.c32[(size_t)(c0 + q) * F + f] = (float)v;
    }
  /* the fields' exponents, for the fixed-point evaluation */
  __shared__ unsigned s_top;
  for (int f = 0; f < F; f++) {
    __syncthreads();
    if (threadIdx.x == 0) s_top = 0;
    __syncthreads();
    unsigned top = 0;
    for (int q = threadIdx.x; q < m; q += blockDim.x) top = max(top, (unsigned)__double2hiint(B[(size_t)f * m + q]) & 0x7fffffffu);
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_top, top);
    __syncthreads();
    if (threadIdx.x == 0) {
      const int e = (int)(s_top >> 20);
      P.cexp[(size_t)node * F + f] = e == 2047 ? LGB_CEXP_NAN : e - 1022;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    P.setup[node] = 1;
    P.solved[node] = 1;
  }
  __syncthreads();
}

__device__ __forceinline__ void count_factored(const FactorParams &P, int m)
{
  atomicAdd(&P.ctrl->factor_flops, (double)m * m * m / 3.0 + 2.0 * (double)m * m * P.F);
  atomicAdd(&P.ctrl->nfactored, 1);
}

/* One template per CTA size NT (the patch-size class's entry of the tuning table): patches of up to 64
   points, or every patch under the option factor_threads. */
template <int NT>
__global__ void __launch_bounds__(NT) k_factor(FactorParams P)
{
  __shared__ PatchCells s_cells;
  __shared__ int s_fail;
  __shared__ double s_rd;
  __shared__ double s_diag[32 * 33], s_y[4 * 32];
  __shared__ double s_red[32];
  __shared__ int s_ired[32];
  const lgb_geom &g = P.g;
  const int nwork = *P.nwork;
  const int tid = threadIdx.x;
  double *A = P.ws + (size_t)blockIdx.x * P.ws_stride;
  for (int w = blockIdx.x; w < nwork; w += gridDim.x) {
    const int node = P.work[w];
    const int m = P.pm[node];
    const int F = P.F;
    if (tid == 0) {
      patch_cells(P, node, s_cells);
      s_fail = 0;
    }
    __syncthreads();
    double *X = A + (size_t)m * m;     /* m*dim patch coordinates */
    double *B = X + (size_t)m * g.dim; /* m*F right-hand sides / solutions */
    patch_gather(P, s_cells, m, X, B);
    __syncthreads();
    const bool have_factor = P.setup[node] && P.keep;
    if (m > 0 && !have_factor) {
      /* assemble the lower triangle, column-major: A[j*m + i], i >= j */
      const double eps = g.eps_r;
      for (int j = 0; j < m; j++) {
        const double xj0 = X[(size_t)j * g.dim], xj1 = X[(size_t)j * g.dim + 1];
        const double xj2 = (g.dim == 3) ? X[(size_t)j * g.dim + 2] : 0.0;
        for (int i = j + tid; i < m; i += NT) {
          double dx = X[(size_t)i * g.dim] - xj0, dy = X[(size_t)i * g.dim + 1] - xj1, d2;
          if (g.dim == 3) {
            double dz = X[(size_t)i * g.dim + 2] - xj2;
            d2 = fma(dx, dx, fma(dy, dy, dz * dz));
          } else d2 = fma(dx, dx, dy * dy);
          A[(size_t)j * m + i] = lgb_phi<double>(g.kernel, sqrt(d2), eps);
        }
      }
      __syncthreads();
      /* 1-norm of the symmetric matrix (largest column sum of |A|) for the condition estimate */
      double anorm = 0.0;
      if (P.kappa) {
        double cm = 0.0;
        for (int j = tid; j < m; j += NT) {
          double cs = 0.0;
          for (int i = j; i < m; i++) cs += fabs(A[(size_t)j * m + i]);
          for (int k = 0; k < j; k++) cs += fabs(A[(size_t)k * m + j]);
          cm = fmax(cm, cs);
        }
        anorm = blk_reduce(cm, s_red, true);
      }
      /* Cholesky in panels of CHOL_NB columns: each panel is factored left-looking from the
         entries already updated by the earlier panels, then the trailing lower triangle is updated
         by the panel (tiles of 32 x 32, one warp per tile).  Every entry receives its updates
         -L(i,k) L(j,k) one at a time in ascending k, exactly as in an unblocked left-looking
         factorisation, so the factor is the same bit for bit; the blocking only stops each column
         from re-reading all earlier columns. */
      double *Ps = B + (size_t)m * F; /* panel rows [p0, m) x CHOL_NB, stride CHOL_NB + 1 */
      for (int p0 = 0; p0 < m && !s_fail; p0 += CHOL_NB) {
        const int nb = min(CHOL_NB, m - p0), p1 = p0 + nb;
        for (int j = p0; j < p1; j++) {
          const double *Lj = A + j; /* row j: Lj[k*m] = L(j,k) */
          for (int i = j + tid; i < m; i += NT) {
            double s = A[(size_t)j * m + i];
            for (int k = p0; k < j; k++) s -= A[(size_t)k * m + i] * Lj[(size_t)k * m];
            A[(size_t)j * m + i] = s;
          }
          __syncthreads();
          /* one thread takes the pivot's square root and its reciprocal; the column is scaled by
             multiplication (an FP64 division per entry would cost the FP64 pipe ~10 operations) */
          if (tid == 0) {
            const double dd = A[(size_t)j * m + j];
            if (!(dd > 0.0)) {
              if (atomicCAS(&P.ctrl->factor_error, 0, j + 1) == 0) P.ctrl->factor_node = node;
              s_fail = 1;
            } else {
              const double sd = sqrt(dd);
              A[(size_t)j * m + j] = sd;
              s_rd = 1.0 / sd;
            }
          }
          __syncthreads();
          if (s_fail) break;
          const double rd = s_rd;
          for (int i = j + 1 + tid; i < m; i += NT) A[(size_t)j * m + i] *= rd;
          __syncthreads();
        }
        __syncthreads();
        if (s_fail || p1 >= m) break;
        /* stage the panel's rows (row-major, padded) for the trailing update */
        for (int t = tid; t < (m - p0) * nb; t += NT) {
          const int kk = t / (m - p0), r = t - kk * (m - p0);
          Ps[(size_t)r * (CHOL_NB + 1) + kk] = A[(size_t)(p0 + kk) * m + p0 + r];
        }
        __syncthreads();
        const int T = (m - p1 + 31) / 32, ntile = T * (T + 1) / 2;
        const int lane = tid & 31, warp = tid >> 5;
        for (int t = warp; t < ntile; t += NT / 32) {
          int c = 0, rem = t;
          while (rem >= T - c) { rem -= T - c; c++; }
          const int i = p1 + 32 * (c + rem) + lane, jb = p1 + 32 * c;
          if (i >= m) continue;
          double li[CHOL_NB];
#pragma unroll
          for (int kk = 0; kk < CHOL_NB; kk++) li[kk] = (kk < nb) ? Ps[(size_t)(i - p0) * (CHOL_NB + 1) + kk] : 0.0;
          const int jend = min(jb + 32, i + 1);
          for (int j = jb; j < jend; j++) {
            const double *lj = Ps + (size_t)(j - p0) * (CHOL_NB + 1);
            double a = A[(size_t)j * m + i];
#pragma unroll
            for (int kk = 0; kk < CHOL_NB; kk++)
              if (kk < nb) a -= li[kk] * lj[kk];
            A[(size_t)j * m + i] = a;
          }
        }
        __syncthreads();
      }
      __syncthreads();
      if (s_fail) { __syncthreads(); continue; }
      prepare_diag_blocks<false>(A, m);
      if (P.kappa) {
        const double inv = inv_norm1_estimate(m, Ps, Ps + m, s_red, s_ired, [&](double *v) {
          chol_solve_group<false, 1>(A, m, v, s_diag, s_y);
        });
        if (tid == 0) P.kappa[node] = anorm * inv;
      }
      if (P.keep) {
        double *Fk = P.fac + P.foff[node];
        for (int j = 0; j < m; j++) {
          long long base = (long long)j * m - ((long long)j * (j - 1)) / 2; /* packed column j */
          for (int i = j + tid; i < m; i += NT) Fk[base + (i - j)] = A[(size_t)j * m + i];
        }
      }
      if (tid == 0) count_factored(P, m);
    } else if (m > 0) {
      if (tid == 0) atomicAdd(&P.ctrl->factor_flops, 2.0 * (double)m * m * F);
    }
    __syncthreads();
    if (m > 0) {
      if (have_factor) chol_solve<true>(P.fac + P.foff[node], m, F, B, s_diag, s_y);
      else chol_solve<false>(A, m, F, B, s_diag, s_y);
    }
    patch_store(P, node, m, B);
  }
}

/* ---- blocked factorisation with fixed-point updates -------------------------------------------- */
/* GB300 issues 2 FP64 multiply-adds per clock and SM, so the updates of the factorisation (m^3 / 6
   multiply-adds) run on the tensor cores and the integer pipe.  The kernels with a positive definite
   matrix have phi(0) <= 1, so every factor entry l is in [-1, 1] and is held in fixed point, units of
   2^-56 (lgb_fx.cuh), whose rounding is below that of FP64 from 1/8 on and below what the m rounded
   FP64 subtractions of an entry accumulate:
     - the sums over earlier block columns on the tensor cores: l = sum_i d_i 2^-(9 + 10 i) with six
       balanced digits |d_i| <= 512, exact in FP16; the products of equal weight i + j <= 5 (21 of 36)
       accumulate in FP32 and are moved to 64-bit integers every 64 columns.  Sums below 2^24 are exact.
       With row norms <= 1 (Cauchy) those with d_0 stay below 2^18 sqrt(64), and sum d_1 d_1' <= 64 2^18 by
       itself; sums of pairs of lower digits are of the order sqrt(64) 2^16.4 (sums of squares on the
       diagonal 64 2^16.4), 2^24 being some 17 standard deviations away: an estimate for digits that are not
       made to line up, not a bound.  What is left out adds up over the columns: of the products
       of weight 6 and more the squares d_3^2 on the diagonal have one sign, about m 2^-61.6 together (2^-52.6
       at 512 columns, 2^-50.6 at 2,048), which FP64's roundings of the m subtractions of a pivot exceed;
     - inside a block column as {hi, lo} integer multiply-adds (fx_mad), in 64-bit sums: |sum hi hi'|
       <= 2^56, |sum hi lo' + lo hi'| <= 2^56 sqrt(32).
   An entry beyond 1 proves a non-positive pivot in its row (a_ii - l_ij^2 < 0): it is clamped for the
   updates and the row is remembered, so the factorisation stops there at the latest.

   One CTA per patch, block columns of 32, left-looking.  For each block column the sums over all
   earlier columns are formed in tiles of 64 rows (a warp: 16 rows x 16 columns, digit slabs of one
   block column staged by cp.async) and subtracted from the kernel values, which are computed there and
   never stored (Wendland C2 in fixed point, other kernels in FP64); the block column waits in the
   workspace.  One warp factors the 32 x 32 diagonal block; then every thread solves its own rows
   against it without further barriers.

   The factor is stored by block columns of 32 columns x R_b = me - 32 b rows (me: m rounded up to
   even, so that 16-byte copies of row pairs stay aligned): the diagonal block in FP64, prepared for
   the solves as above, the rows below as {hi, lo}.  Fresh factors live in the workspace, kept ones in
   the factor pool; the solves read the same format from either.  The digits live in the workspace. */
#define BLK_NT 256
#define BLK_NB 32
#define BLK_KP 16   /* column pairs per staged slab (one block column) */
#define BLK_ROWS 64
#define BLK_ND 6    /* digits */
#define BLK_FLUSH 2 /* slabs between two moves of the FP32 sums to integers */

struct FxSolveShared {
  int2 tile[128][36];   /* backward update: 128 columns x 32 rows, padded to distinct banks */
  double d[32 * 33];    /* staged diagonal block */
  int2 yq[4][32];       /* the block's solution in fixed point, relative to 2^e */
  double ysc[4];        /* 2^(e - 56) */
};
struct FxFactorShared {
  /* digit pairs (columns 2 p, 2 p + 1) of a row; row strides of 8 mod 32 words: the fragment reads of a
     warp (four pairs x eight rows) fall in distinct banks */
  union {
    struct {
      unsigned row[2][BLK_ND][BLK_KP][BLK_ROWS + 8];
      unsigned col[2][BLK_ND][BLK_KP][BLK_NB + 8];
    };
    long long diag[BLK_NB][BLK_NB];  /* between the updates: the block's entries, [column][row] */
  };
  int2 q11[BLK_NB][BLK_NB];      /* diagonal block in fixed point, [row][column] */
  double rd[BLK_NB];
};
struct BlkShared {
  union {
    FxSolveShared s;
    FxFactorShared f;
  };
  double red[32];
  PatchCells cells;
  int ired[32];
  int fail, badrow, item;
};

/* Start of block column b in the stored factor (8-byte elements) and in the digit array (words;
   [digit][pair][row], rows from the block's first one, mh: m rounded up to a multiple of 4). */
__device__ __forceinline__ long long fx_base(int me, int b) { return 32LL * b * me - 512LL * b * (b - 1); }
__device__ __forceinline__ long long fx_dbase(int mh, int b) { return 16LL * BLK_ND * ((long long)b * mh - 16LL * b * (b - 1)); }

__device__ __forceinline__ void cp_async16(void *dst, const void *src, bool ok)
{
  const unsigned n = ok ? 16u : 0u; /* 0: zero fill */
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(n) : "memory");
}

/* Kernel value for the assembly from the squared distance (Wendland C2: lgb_sqrt_pos of (eps r)^2). */
__device__ __forceinline__ double asm_phi(int kernel, double d2, double eps)
{
  if (kernel == LGB_KERNEL_WENDLAND_C2) {
    const double s = d2 * (eps * eps);
    const double r = lgb_sqrt_pos(s);
    double u = 1.0 - r;
    if (__double2hiint(u) < 0) return 0.0; /* the sign bit: no FP64 comparison */
    const double u2 = u * u;
    return (u2 * u2) * fma(-4.0, u, 5.0);
  }
  return lgb_phi<double>(kernel, sqrt(d2), eps);
}

/* Entry (i, j) of the collocation matrix in fixed point; X: the patch coordinates, FP64 (FIXED 0) or
   eps (x - node) in fixed point (1: Wendland C2, 2: Gaussian). */
template <int FIXED>
__device__ __forceinline__ long long asm_entry(const lgb_geom &g, const double *X, int i, int j)
{
  if constexpr (FIXED != 0) {
    const long long *Z = reinterpret_cast<const long long *>(X);
    const long long dx = Z[g.dim * (size_t)i] - Z[g.dim * (size_t)j], dy = Z[g.dim * (size_t)i + 1] - Z[g.dim * (size_t)j + 1];
    const long long dz = g.dim == 3 ? Z[3 * (size_t)i + 2] - Z[3 * (size_t)j + 2] : 0;
    if constexpr (FIXED == 1) {
      const long long s = fx_dist2<3>(dx, dy, dz);
      return s < FX_ONE_I ? fx_phi_c2(s) : 0;
    } else {
      const long long s = fx_dist2_wide<3>(dx, dy, dz);
      return s < FX_EXP_END ? fx_exp_neg(s) : 0;
    }
  } else {
    const int dim = g.dim;
    const double *xi = X + (size_t)i * dim, *xj = X + (size_t)j * dim;
    const double dx = xi[0] - xj[0], dy = xi[1] - xj[1], dz = (dim == 3) ? xi[2] - xj[2] : 0.0;
    const double d2 = (dim == 3) ? fma(dx, dx, fma(dy, dy, dz * dz)) : fma(dx, dx, dy * dy);
    return __double2ll_rn(asm_phi(g.kernel, d2, g.eps_r) * FX_ONE);
  }
}

/* The balanced digits of two fixed-point values as FP16 pairs. */
__device__ __forceinline__ void fx_digits(long long a, long long b, unsigned (&h)[BLK_ND])
{
  long long v[2] = {a << 3, b << 3}; /* units of 2^-59 */
  float d[2][BLK_ND];
#pragma unroll
  for (int s = 0; s < 2; s++) {
    long long t = v[s];
#pragma unroll
    for (int i = BLK_ND - 1; i > 0; i--) {
      const int e = (int)((unsigned)t << 22) >> 22; /* the low ten bits, signed */
      d[s][i] = (float)e;
      t = (t - e) >> 10;
    }
    d[s][0] = (float)(int)t;
  }
#pragma unroll
  for (int i = 0; i < BLK_ND; i++)
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h[i]) : "f"(d[1][i]), "f"(d[0][i]));
}

__device__ __forceinline__ void blk_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1)
{
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

/* The block solution v (lane's entry, zero beyond the block) of right-hand side q into fixed point
   relative to a power of two above its largest entry (one warp).  A solution that is not finite makes
   every row it updates NaN through the scale. */
__device__ __forceinline__ void fx_pack(FxSolveShared &S, int q, int lane, double v)
{
  const unsigned top = __reduce_max_sync(0xffffffffu, (unsigned)__double2hiint(v) & 0x7fffffffu) >> 20;
  const int e = max((int)top - 1022, -966); /* |v| < 2^e, and both factors below are normal */
  const double up = __hiloint2double((1023 + 56 - e) << 20, 0);
  S.yq[q][lane] = fx_split(top == 2047 ? 0 : __double2ll_rn(v * up));
  if (lane == 0) S.ysc[q] = top == 2047 ? __hiloint2double(0x7ff80000, 0) : __hiloint2double((1023 - 56 + e) << 20, 0);
}

/* Solves L L^T X = B in place for FC (1..4) columns of B (B[q*m + i]) with the stored factor Fq, in
   blocks of 32 rows: the diagonal block is substituted in FP64 (as chol_solve_group; one warp per
   right-hand side, a warp issues an FP64 operation in 64 cycles), the other rows are updated with exact integer sums over the block and one FP64 multiply-add.  Forward:
   a thread per row, coalesced along the rows.  Backward: tiles of 128 columns x 32 rows pass through
   shared memory, two threads per column.  Bound by reading the factor (8 bytes per 9 integer
   multiply-adds with three right-hand sides). */
template <int FC>
__device__ void fx_solve_group(const double *__restrict__ Fq, int m, double *B0, FxSolveShared &S)
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nblk = (m + 31) / 32, me = (m + 1) & ~1;
  for (int b = 0; b < nblk; b++) {
    const int J = 32 * b, nb = min(32, m - J), R = me - J;
    const double *Fb = Fq + fx_base(me, b);
    for (int t = tid; t < 1024; t += BLK_NT) {
      const int c = t >> 5, r = t & 31;
      if (r >= c && r < nb) S.d[r * 33 + c] = Fb[(size_t)c * R + r];
    }
    __syncthreads();
    if (warp < FC) {
      double u = (lane < nb) ? B0[(size_t)warp * m + J + lane] : 0.0;
      for (int jj = 0; jj < nb - 1; jj++) {
        const double mij = (lane > jj && lane < nb) ? S.d[lane * 33 + jj] : 0.0;
        u = fma(-mij, __shfl_sync(0xffffffffu, u, jj), u);
      }
      const double y = u * ((lane < nb) ? S.d[lane * 33 + lane] : 0.0);
      if (lane < nb) B0[(size_t)warp * m + J + lane] = y;
      fx_pack(S, warp, lane, lane < nb ? y : 0.0);
    }
    __syncthreads();
    for (int i = J + 32 + tid; i < m; i += BLK_NT) {
      const int2 *Lr = reinterpret_cast<const int2 *>(Fb) + (i - J);
      long long hh[FC], hl[FC];
#pragma unroll
      for (int q = 0; q < FC; q++) { hh[q] = 0; hl[q] = 0; }
#pragma unroll 16
      for (int c = 0; c < 32; c++) {
        const int2 l = Lr[(size_t)c * R];
#pragma unroll
        for (int q = 0; q < FC; q++) {
          const int2 y = S.yq[q][c];
          fx_mad(hh[q], l.x, y.x);
          fx_mad(hl[q], l.x, y.y);
          fx_mad(hl[q], l.y, y.x);
        }
      }
#pragma unroll
      for (int q = 0; q < FC; q++)
        B0[(size_t)q * m + i] = fma(-(double)fx_sum(hh[q], hl[q]), S.ysc[q], B0[(size_t)q * m + i]);
    }
    __syncthreads();
  }
  for (int b = nblk - 1; b >= 0; b--) {
    const int i0 = 32 * b, nb = min(32, m - i0), R = me - i0;
    const double *Fb = Fq + fx_base(me, b);
    for (int t = tid; t < 1024; t += BLK_NT) {
      const int c = t >> 5, r = t & 31;
      if (r >= c && r < nb) S.d[r * 33 + c] = Fb[(size_t)c * R + r];
    }
    __syncthreads();
    if (warp < FC) {
      double x = (lane < nb) ? B0[(size_t)warp * m + i0 + lane] * S.d[lane * 33 + lane] : 0.0;
      for (int ii = nb - 1; ii >= 1; ii--) {
        const double mi = (lane < ii) ? S.d[ii * 33 + lane] : 0.0;
        x = fma(-mi, __shfl_sync(0xffffffffu, x, ii), x);
      }
      if (lane < nb) B0[(size_t)warp * m + i0 + lane] = x;
      fx_pack(S, warp, lane, lane < nb ? x : 0.0);
    }
    __syncthreads();
    for (int t0 = 0; t0 < i0; t0 += 128) {
      for (int t = tid; t < 128 * 16; t += BLK_NT) {
        const int c = t >> 4, i = t0 + c, bc = i >> 5;
        if (i < i0)
          cp_async16(&S.tile[c][2 * (t & 15)],
                     Fq + fx_base(me, bc) + (size_t)(i & 31) * (me - 32 * bc) + (i0 - 32 * bc) + 2 * (t & 15), true);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();
      const int c = tid >> 1, h = tid & 1, i = t0 + c;
      long long hh[FC], hl[FC];
#pragma unroll
      for (int q = 0; q < FC; q++) { hh[q] = 0; hl[q] = 0; }
      if (i < i0) {
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const int r = 4 * k + 2 * h;
          const int4 l = *reinterpret_cast<const int4 *>(&S.tile[c][r]);
#pragma unroll
          for (int q = 0; q < FC; q++) {
            const int4 y = *reinterpret_cast<const int4 *>(&S.yq[q][r]);
            fx_mad(hh[q], l.x, y.x);
            fx_mad(hl[q], l.x, y.y);
            fx_mad(hl[q], l.y, y.x);
            fx_mad(hh[q], l.z, y.z);
            fx_mad(hl[q], l.z, y.w);
            fx_mad(hl[q], l.w, y.z);
          }
        }
      }
#pragma unroll
      for (int q = 0; q < FC; q++) {
        hh[q] += __shfl_xor_sync(0xffffffffu, hh[q], 1);
        hl[q] += __shfl_xor_sync(0xffffffffu, hl[q], 1);
        if (h == 0 && i < i0)
          B0[(size_t)q * m + i] = fma(-(double)fx_sum(hh[q], hl[q]), S.ysc[q], B0[(size_t)q * m + i]);
      }
      __syncthreads();
    }
    __syncthreads();
  }
}

/* All F right-hand sides of B (B[f*m + i]), four at a time. */
__device__ void fx_solve(const double *Fq, int m, int F, double *B, FxSolveShared &S)
{
  for (int f0 = 0; f0 < F; f0 += 4) {
    double *B0 = B + (size_t)f0 * m;
    switch (min(4, F - f0)) {
    case 1: fx_solve_group<1>(Fq, m, B0, S); break;
    case 2: fx_solve_group<2>(Fq, m, B0, S); break;
    case 3: fx_solve_group<3>(Fq, m, B0, S); break;
    default: fx_solve_group<4>(Fq, m, B0, S); break;
    }
  }
}

/* 1 / sqrt(d) of a double in the single range: the single-precision root y refined by a third-order
   step (Householder's method); y^2 is exact in FP64, so the residual 1 - d y^2 is rounded once.  About
   half an ulp in five operations.  (A warp issues an FP64 operation in 64 cycles, and this chain is
   the pivot's latency.) */
__device__ __forceinline__ double fx_rsqrt(double d)
{
  float f;
  asm("rsqrt.approx.f32 %0, %1;" : "=f"(f) : "f"(__double2float_rn(d)));
  const double y = (double)f, e = fma(-d, y * y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}
/* x 2^-56 for normal x (the exponent field: no FP64 operation). */
__device__ __forceinline__ double fx_down(double x) { return __hiloint2double(__double2hiint(x) - (56 << 20), __double2loint(x)); }

/* sum_k<N q[k] v[k] of the fixed-point entries, in CH (1 or 2) chains of integer sums. */
template <int N, int CH>
__device__ __forceinline__ long long fx_dot(const int2 (&q)[BLK_NB], const int2 *v)
{
  long long hh[CH], hl[CH];
#pragma unroll
  for (int c = 0; c < CH; c++) { hh[c] = 0; hl[c] = 0; }
#pragma unroll
  for (int k = 0; k < N; k++) {
    const int2 x = v[k];
    fx_mad(hh[k % CH], q[k].x, x.x);
    fx_mad(hl[k % CH], q[k].x, x.y);
    fx_mad(hl[(k + 1) % CH], q[k].y, x.x);
  }
  return CH == 2 ? fx_sum(hh[0] + hh[CH - 1], hl[0] + hl[CH - 1]) : fx_sum(hh[0], hl[0]);
}

/* One warp factors the nb x nb diagonal block J of the block column (lane i holds row J + i,
   left-looking; S.diag: its entries): q11 and rd in shared memory, the prepared block in Fb.  Returns
   the failing column + 1, or 0.  The chain of a column (dot product, pivot root, scaling) is the
   latency of the factorisation. */
template <int J0> struct BlkCol {
  static __device__ __forceinline__ int run(FxFactorShared &S, int2 (&q)[BLK_NB], double *Fb, int J, int nb, int R, int lane,
                                            int bad, int *badrow)
  {
    if (J0 >= nb) return 0;
    const long long s = S.diag[J0][lane] - fx_dot<J0, 2>(q, S.q11[J0]);
    const long long dd = __shfl_sync(0xffffffffu, s, J0);
    if (dd <= 0 || J + J0 == bad) return J0 + 1;
    const double rs = fx_rsqrt(fx_down((double)dd));
    const double x = (double)s * rs;
    long long f = __double2ll_rn(x); /* saturates */
    if (f > FX_ONE_I + (1LL << 36) || f < -FX_ONE_I - (1LL << 36)) {
      if (lane > J0 && lane < nb) atomicMin(badrow, J + lane);
      f = f > 0 ? FX_ONE_I : -FX_ONE_I;
    }
    q[J0] = fx_split(f);
    S.q11[lane][J0] = q[J0];
    if (lane == J0) S.rd[J0] = rs;
    if (lane >= J0 && lane < nb) Fb[(size_t)J0 * R + lane] = (J0 == lane) ? rs : x * fx_down(rs);
    __syncwarp();
    if constexpr (J0 + 1 < BLK_NB) return BlkCol<J0 + 1>::run(S, q, Fb, J, nb, R, lane, bad, badrow);
    else return 0;
  }
};
__device__ __noinline__ int blk_diag(FxFactorShared &S, double *Fb, int J, int nb, int R, int *badrow)
{
  int2 q[BLK_NB];
  return BlkCol<0>::run(S, q, Fb, J, nb, R, threadIdx.x & 31, *badrow, badrow);
}
/* Block column J minus the sums over the columns before it, for the rows i0 .. i0 + 63 (all warps). */
template <int FIXED>
__device__ __noinline__ void blk_update(FxFactorShared &T, const lgb_geom &g, const unsigned *H, const double *X,
                                           long long *C, int m, int J, int i0)
{
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wr = warp & 3, wc = warp >> 2;
  const int t = lane & 3, gr = lane >> 2, nslab = J / BLK_NB, mh = (m + 3) & ~3, rows = m - J;
  float acc[BLK_ND][2][4]; /* by digit weight d + e */
  long long v[2][4];
#pragma unroll
  for (int n = 0; n < 2; n++)
#pragma unroll
    for (int r = 0; r < 4; r++) {
      v[n][r] = 0;
#pragma unroll
      for (int s = 0; s < BLK_ND; s++) acc[s][n][r] = 0.f;
    }
  auto stage = [&](int sl) { /* block column sl: [digit][pair][row] */
    const int bf = sl & 1, Rk = mh - 32 * sl;
    const unsigned *src = H + fx_dbase(mh, sl);
    {
      const int c = 4 * (tid & 15), o = i0 - 32 * sl + c;
      const bool ok = o < Rk;
#pragma unroll
      for (int d = 0; d < BLK_ND; d++)
        cp_async16(&T.row[bf][d][tid >> 4][c], src + (size_t)(16 * d + (tid >> 4)) * Rk + (ok ? o : 0), ok);
    }
    {
      const int c = 4 * (tid & 7), p = (tid >> 3) & 15, o = J - 32 * sl + c;
      const bool ok = o < Rk;
#pragma unroll
      for (int d = 0; d < BLK_ND; d += 2)
        cp_async16(&T.col[bf][d + (tid >> 7)][p][c], src + (size_t)(16 * (d + (tid >> 7)) + p) * Rk + (ok ? o : 0), ok);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (nslab > 0) stage(0);
  for (int sl = 0; sl < nslab; sl++) {
    if (sl + 1 < nslab) {
      stage(sl + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const int bf = sl & 1;
#pragma unroll
    for (int h = 0; h < BLK_KP; h += 8) {
      unsigned a[BLK_ND][4];
#pragma unroll
      for (int d = 0; d < BLK_ND; d++) {
        a[d][0] = T.row[bf][d][h + t][16 * wr + gr];
        a[d][1] = T.row[bf][d][h + t][16 * wr + gr + 8];
        a[d][2] = T.row[bf][d][h + t + 4][16 * wr + gr];
        a[d][3] = T.row[bf][d][h + t + 4][16 * wr + gr + 8];
      }
#pragma unroll
      for (int n = 0; n < 2; n++)
#pragma unroll
        for (int e = 0; e < BLK_ND; e++) {
          const unsigned b0 = T.col[bf][e][h + t][16 * wc + 8 * n + gr], b1 = T.col[bf][e][h + t + 4][16 * wc + 8 * n + gr];
#pragma unroll
          for (int d = 0; d < BLK_ND; d++)
            if (d + e < BLK_ND) blk_mma(acc[d + e][n], a[d], b0, b1);
        }
    }
    if (sl % BLK_FLUSH == BLK_FLUSH - 1 || sl + 1 == nslab) {
#pragma unroll
      for (int n = 0; n < 2; n++)
#pragma unroll
        for (int r = 0; r < 4; r++) {
          long long x = (((long long)__float2int_rn(acc[4][n][r]) << 10) + __float2int_rn(acc[5][n][r]) + (1 << 11)) >> 12;
#pragma unroll
          for (int s = 0; s < 4; s++) x += (long long)__float2int_rn(acc[s][n][r]) << (38 - 10 * s);
          v[n][r] += x;
#pragma unroll
          for (int s = 0; s < BLK_ND; s++) acc[s][n][r] = 0.f;
        }
    }
    __syncthreads();
  }
#pragma unroll
  for (int n = 0; n < 2; n++)
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int i = i0 + 16 * wr + gr + 8 * (r >> 1), jl = 16 * wc + 8 * n + 2 * t + (r & 1);
      if (i >= m || i - J < jl) continue;
      C[(size_t)jl * rows + (i - J)] = asm_entry<FIXED>(g, X, i, J + jl) - v[n][r];
    }
}

/* Rows below the diagonal block: x L11^T = c, one row per thread, left to right; each entry's sum over
   the columns before it in integers, one FP64 multiplication by the reciprocal pivot. */
template <int J0> struct BlkRow {
  static __device__ __forceinline__ bool run(const FxFactorShared &T, int2 (&q)[BLK_NB], const long long *C, int2 *Qb,
                                             unsigned *Hb, int i, int rows, int R, int Rh, long long s, long long even)
  {
    long long ahead = 0;
    if (J0 + 1 < BLK_NB) ahead = C[(size_t)(J0 + 1) * rows + i];
    s -= fx_dot<J0, 1>(q, T.q11[J0]);
    long long f = __double2ll_rn((double)s * T.rd[J0]); /* saturates */
    bool bad = false;
    if (f > FX_ONE_I + (1LL << 36) || f < -FX_ONE_I - (1LL << 36)) {
      bad = true;
      f = f > 0 ? FX_ONE_I : -FX_ONE_I;
    }
    q[J0] = fx_split(f);
    Qb[(size_t)J0 * R + i] = q[J0];
    if (J0 & 1) {
      unsigned h[BLK_ND];
      fx_digits(even, f, h);
#pragma unroll
      for (int d = 0; d < BLK_ND; d++) Hb[(size_t)(BLK_KP * d + (J0 >> 1)) * Rh + i] = h[d];
    }
    asm volatile("" ::: "memory"); /* one column's loads at a time: the row's entries fill the registers */
    if constexpr (J0 + 1 < BLK_NB) bad |= BlkRow<J0 + 1>::run(T, q, C, Qb, Hb, i, rows, R, Rh, ahead, f);
    return bad;
  }
};
__device__ __noinline__ void blk_rows(BlkShared &S, const long long *C, int2 *Qb, unsigned *Hb, int J, int rows, int R, int Rh)
{
  for (int i = BLK_NB + threadIdx.x; i < rows; i += BLK_NT) {
    int2 q[BLK_NB];
    if (BlkRow<0>::run(S.f, q, C, Qb, Hb, i, rows, R, Rh, C[i], 0)) atomicMin(&S.badrow, J + i);
  }
}

__global__ void __launch_bounds__(BLK_NT, 2) k_factor_blk(FactorParams P, int *next)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BlkShared &S = *reinterpret_cast<BlkShared *>(smem_raw);
  const lgb_geom &g = P.g;
  const int nwork = *P.nwork, F = P.F, dim = g.dim;
  const int tid = threadIdx.x, warp = tid >> 5;
  double *W = P.ws + (size_t)blockIdx.x * P.ws_stride;
  for (;;) {
    if (tid == 0) S.item = atomicAdd(next, 1);
    __syncthreads();
    const int w = S.item;
    if (w >= nwork) return;
    const int node = P.work[w], m = P.pm[node], me = (m + 1) & ~1, mh = (m + 3) & ~3;
    if (tid == 0) {
      patch_cells(P, node, S.cells);
      S.fail = 0;
      S.badrow = 0x7fffffff;
    }
    __syncthreads();
    /* workspace: digits, block column, coordinates, right-hand sides, two vectors, then the factor */
    unsigned *H = reinterpret_cast<unsigned *>(W);
    long long *C = reinterpret_cast<long long *>(W + lgb_fx_dsize(m));
    double *X = reinterpret_cast<double *>(C + (size_t)BLK_NB * m), *B = X + (size_t)m * dim, *V = B + (size_t)m * F;
    double *Fq = P.keep ? P.fac + P.foff[node]
                        : W + ((lgb_fx_dsize(m) + (long long)m * (BLK_NB + dim + F + 2) + 1) & ~1LL);
    patch_gather(P, S.cells, m, X, B);
    if (P.fixed) { /* coordinates relative to the patch node, scaled (each thread its own points) */
      const int nxy = g.n[0] * g.n[1], l = node / nxy, r = node - l * nxy, nj = r / g.n[0];
      const double c[3] = {g.O[0] + g.h[0] * (r - nj * g.n[0]), g.O[1] + g.h[1] * nj, g.O[2] + g.h[2] * l};
      for (int q = tid; q < m; q += BLK_NT)
        for (int d = 0; d < dim; d++) {
          const long long z = fx_coord(g.eps_r, X[(size_t)q * dim + d] - c[d]);
          X[(size_t)q * dim + d] = __longlong_as_double(z);
        }
    }
    __syncthreads();
    double anorm = 0.0;
    if (P.kappa) { /* 1-norm of the symmetric matrix for the condition estimate */
      double cm = 0.0;
      for (int j = tid; j < m; j += BLK_NT) {
        double cs = 0.0;
        for (int i = 0; i < m; i++)
          cs += fabs((double)(P.fixed == 1 ? asm_entry<1>(g, X, i, j)
                              : P.fixed == 2 ? asm_entry<2>(g, X, i, j) : asm_entry<0>(g, X, i, j)));
        cm = fmax(cm, cs * (1.0 / FX_ONE));
      }
      anorm = blk_reduce(cm, S.red, true);
    }
    for (int J = 0; J < m; J += BLK_NB) {
      const int nb = min(BLK_NB, m - J), rows = m - J, R = me - J, b = J / BLK_NB;
      double *Fb = Fq + fx_base(me, b);
      for (int i0 = J; i0 < m; i0 += BLK_ROWS) {
        if (P.fixed == 1) blk_update<1>(S.f, g, H, X, C, m, J, i0);
        else if (P.fixed == 2) blk_update<2>(S.f, g, H, X, C, m, J, i0);
        else blk_update<0>(S.f, g, H, X, C, m, J, i0);
      }
      __syncthreads();
      for (int q = tid; q < BLK_NB * BLK_NB; q += BLK_NT) {
        const int j = q / BLK_NB, r = q % BLK_NB;
        S.f.diag[j][r] = (r >= j && r < nb) ? C[(size_t)j * rows + r] : 0;
      }
      __syncthreads();
      if (warp == 0) {
        const int failed = blk_diag(S.f, Fb, J, nb, R, &S.badrow);
        if (failed && tid == 0) {
          if (atomicCAS(&P.ctrl->factor_error, 0, J + failed) == 0) P.ctrl->factor_node = node;
          S.fail = 1;
        }
      }
      __syncthreads();
      if (S.fail) break;
      int2 *Qb = reinterpret_cast<int2 *>(Fb);
      blk_rows(S, C, Qb, H + fx_dbase(mh, b), J, rows, R, mh - J);
      if ((m & 1) && tid < BLK_NB) Qb[(size_t)tid * R + rows] = make_int2(0, 0); /* the padding row */
      __syncthreads();
    }
    if (S.fail) continue; /* uniform: its write was followed by a barrier */
    if (P.kappa) {
      const double inv = inv_norm1_estimate(m, V, V + m, S.red, S.ired, [&](double *v) { fx_solve_group<1>(Fq, m, v, S.s); });
      if (tid == 0) P.kappa[node] = anorm * inv;
    }
    if (tid == 0) count_factored(P, m);
    fx_solve(Fq, m, F, B, S.s);
    patch_store(P, node, m, B);
  }
}

/* Re-solve of the patches with a kept factor of the blocked kernel. */
__global__ void __launch_bounds__(BLK_NT) k_solve_blk(FactorParams P, int *next)
{
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FxSolveShared &S = *reinterpret_cast<FxSolveShared *>(smem_raw);
  __shared__ PatchCells s_cells;
  __shared__ int s_item;
  const int nwork = *P.nwork, tid = threadIdx.x;
  double *W = P.ws + (size_t)blockIdx.x * P.ws_stride;
  for (;;) {
    if (tid == 0) {
      s_item = atomicAdd(next, 1);
      if (s_item < nwork) patch_cells(P, P.work[s_item], s_cells);
    }
    __syncthreads();
    if (s_item >= nwork) return;
    const int node = P.work[s_item], m = P.pm[node];
    double *X = W, *B = X + (size_t)m * P.g.dim;
    patch_gather(P, s_cells, m, X, B);
    if (tid == 0) atomicAdd(&P.ctrl->factor_flops, 2.0 * (double)m * m * P.F);
    __syncthreads();
    fx_solve(P.fac + P.foff[node], m, P.F, B, S);
    patch_store(P, node, m, B);
  }
}

extern "C" int lgb_op_factor(lgb_dev *d, void *stream)
{
  if (d->nws <= 0 || !d->ws) return 0;
  FactorParams P;
  P.g = d->g;
  P.F = d->F;
  P.keep = d->keep_factors;
  P.cstart = d->cstart;
  P.xs = d->xs;
  P.fs = d->fs;
  P.pm = d->pm;
  P.slot = d->slot;
  P.work = d->work;
  P.coff = d->coff;
  P.foff = d->foff;
  P.setup = d->setup;
  P.solved = d->solved;
  P.c64 = d->c64;
  P.c32 = d->c32;
  P.cexp = d->cexp;
  P.fac = d->fac;
  P.ws = d->ws;
  P.ws_stride = d->ws_stride;
  P.ctrl = d->ctrl;
  P.kappa = d->cond_on ? d->kappa : NULL;
  P.fixed = d->fixed;
  /* one launch per patch-size class holding patches: its CTA size, grid and workspace slots */
  for (int c = 0; c < LGB_NCLS; c++) {
    if (d->cls_cap[c] <= 0 || d->cls_grid[c] <= 0) continue;
    P.work = d->work + d->cls_off[c];
    P.nwork = &d->ctrl->nwork_c[c];
    P.ws_stride = d->cls_stride[c];
    cudaStream_t s = (cudaStream_t)stream;
    switch (d->cls_threads[c]) {
    case 0: {
      static unsigned long long opted_f = 0, opted_s = 0;
      int rc = lgb_opt_in(k_factor_blk, (int)sizeof(BlkShared), &opted_f);
      if (!rc) rc = lgb_opt_in(k_solve_blk, (int)sizeof(FxSolveShared), &opted_s);
      if (rc) return rc;
      k_factor_blk<<<d->cls_grid[c], BLK_NT, sizeof(BlkShared), s>>>(P, &d->ctrl->next_c[c]);
      if (P.keep) {
        FactorParams Q = P;
        Q.work = d->work_s + d->cls_off[c];
        Q.nwork = &d->ctrl->nwork_s[c];
        Q.ws_stride = d->cls_sstride[c];
        k_solve_blk<<<d->cls_sgrid[c], BLK_NT, sizeof(FxSolveShared), s>>>(Q, &d->ctrl->next_s[c]);
        lgb_count_launch(1);
      }
      break;
    }
    case 32: k_factor<32><<<d->cls_grid[c], 32, 0, s>>>(P); break;
    case 64: k_factor<64><<<d->cls_grid[c], 64, 0, s>>>(P); break;
    case 256: k_factor<256><<<d->cls_grid[c], 256, 0, s>>>(P); break;
    default: k_factor<128><<<d->cls_grid[c], 128, 0, s>>>(P); break;
    }
    lgb_count_launch(1);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}
