/*
 * lgb_eval32_2d.cu -- FP32-evaluation instantiations of the PU evaluation kernel (lgb_eval.cuh), 2D.
 */
#include "lgb_evalrec.cuh"
#include "lgb_optin.cuh"
#include <stdlib.h>

template <int DIM, int FP, int KER, int R>
static int launch32r(const EvalParams &P, int grid, cudaStream_t s)
{
  static unsigned long long opted = 0;
  const int nbuf = 1;
  /* at least a warp: the kernel's block table takes 3^DIM threads and its votes whole warps (units of 32
     particles are cut for the record kernel, which other fields of the same particles do not take) */
  const int threads = P.chunk_cap / R < 32 ? 32 : P.chunk_cap / R;
  /* staging buffer(s) + per-thread running sums of the R*NEN*FP per-patch partial sums */
  size_t smem = ((size_t)nbuf * P.budget + (size_t)(R * (1 << DIM) * FP + 1) * threads) * sizeof(float);
  const size_t smax = ((size_t)nbuf * P.budget + (size_t)(R * (1 << DIM) * FP + 1) * (LGB_CHUNK_MAX / R)) * sizeof(float);
  if (const int rc = lgb_opt_in(k_eval<float, DIM, FP, R, KER>, (int)smax, &opted)) return rc;
  k_eval<float, DIM, FP, R, KER><<<grid, threads, smem, s>>>(P);
  return (int)cudaGetLastError();
}

/* Two particles per thread (four per thread measured slower: fewer active lanes per work unit). */
template <int DIM, int FP, int KER>
static int launch32(const EvalParams &P, int grid, cudaStream_t s)
{
  return launch32r<DIM, FP, KER, 2>(P, grid, s);
}

/* The record-streamed kernel: EVR_NB stages of P.budget floats; per particle the PU weights (8 words) and marks of its sums
   (1), per thread the shares' support sums (2). */
template <int DIM, int KER, int RM>
static int launch_rec(const EvalParams &P, int grid, cudaStream_t s)
{
  /* opted in once to the device's largest size (a per-call size could shrink it under another thread's launch) */
  static unsigned long long opted = 0;
  const size_t smem = ((size_t)EVR_NB * P.budget + (size_t)(RM == 2 ? 2 * EVR_T * 10 : P.threads * 11)) * sizeof(float);
  if (const int rc = lgb_opt_in(k_eval_rec<DIM, DIM, KER, RM>, 227 * 1024 - 8192, &opted)) return rc;
  k_eval_rec<DIM, DIM, KER, RM><<<grid, P.threads, smem, s>>>(P);
  return (int)cudaGetLastError();
}

template <int DIM, int KER>
static int launch32_fp(const EvalParams &P, int fp, int stage, int grid, cudaStream_t s)
{
  if (stage == 1) { /* records hold the dim velocity fields */
    if (P.threads > EVR_T) return launch_rec<DIM, KER, 0>(P, grid, s);
    return P.chunk_cap <= EVR_T ? launch_rec<DIM, KER, 1>(P, grid, s) : launch_rec<DIM, KER, 2>(P, grid, s);
  }
  switch (fp) {
  case 1: return launch32<DIM, 1, KER>(P, grid, s);
  case 2: return launch32<DIM, 2, KER>(P, grid, s);
  case 3: return launch32<DIM, 3, KER>(P, grid, s);
  default: return launch32<DIM, 4, KER>(P, grid, s);
  }
}

extern "C" int lgb_eval32_launch_2d(const EvalParams *P, int fp, int ker, int stage, int grid, void *stream)
{
  cudaStream_t s = (cudaStream_t)stream;
  if (ker == KER_C2) return launch32_fp<2, KER_C2>(*P, fp, stage, grid, s);
  if (ker == KER_GAUSS) return launch32_fp<2, KER_GAUSS>(*P, fp, stage, grid, s);
  return launch32_fp<2, KER_GENERIC>(*P, fp, stage, grid, s);
}

extern "C" int lgb_build_records_2d(const EvalParams *P, int force, int grid, void *stream)
{
  k_build_records2<2, 2><<<grid, 128, 0, (cudaStream_t)stream>>>(*P, force);
  return (int)cudaGetLastError();
}
