/*
 * lgb_evalfx.cu -- instantiations of the fixed-point evaluation kernel (lgb_evalfx.cuh).
 */
#include "lgb_evalfx.cuh"

template <int DIM, int FP, int KER>
static int launch(const EvalParams &P, int grid, cudaStream_t s)
{
  k_eval_fx<DIM, FP, KER><<<grid, FXE_T, FXE_BUDGET, s>>>(P);
  return (int)cudaGetLastError();
}
template <int DIM, int KER>
static int launch_fp(const EvalParams &P, int fp, int grid, cudaStream_t s)
{
  switch (fp) {
  case 1: return launch<DIM, 1, KER>(P, grid, s);
  case 2: return launch<DIM, 2, KER>(P, grid, s);
  case 3: return launch<DIM, 3, KER>(P, grid, s);
  default: return launch<DIM, 4, KER>(P, grid, s);
  }
}

extern "C" int lgb_evalfx_launch(const EvalParams *P, int fp, int grid, void *stream)
{
  cudaStream_t s = (cudaStream_t)stream;
  const bool gauss = P->g.kernel == LGB_KERNEL_GAUSSIAN;
  if (P->g.dim == 3) return gauss ? launch_fp<3, KER_GAUSS>(*P, fp, grid, s) : launch_fp<3, KER_C2>(*P, fp, grid, s);
  return gauss ? launch_fp<2, KER_GAUSS>(*P, fp, grid, s) : launch_fp<2, KER_C2>(*P, fp, grid, s);
}
