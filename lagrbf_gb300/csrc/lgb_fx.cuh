/*
 * lgb_fx.cuh -- 64-bit fixed-point arithmetic on the integer pipe in place of FP64.
 *
 * GB300 issues 2 FP64 multiply-adds per clock and SM, but 25-55 32 x 32 + 64-bit integer ones
 * (mad.wide; the operands' register banks decide), so three integer multiply-adds for a 56-bit product
 * are four to eight times an FP64 one.  Values are integers in units of 2^-56, multiplied as
 *     t = hi 2^28 + lo,  |lo| <= 2^27:   t t' 2^-56 = hi hi' + (hi lo' + lo hi') 2^-28  (+ lo lo' 2^-56)
 * where the last product, at most a quarter unit, is left out.  Every operation below is exact up to
 * about one unit, 2^-56, which is an eighth of the rounding unit 2^-53 of FP64 at one.
 * The functions compile for the host too, where the unit tests compare them with extended precision.
 */
#pragma once
#include <math.h>
#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD static inline
struct int2 { int x, y; };
static inline int2 make_int2(int x, int y) { int2 v = {x, y}; return v; }
#endif

#define FX_ONE 72057594037927936.0 /* 2^56 */
#define FX_ONE_I (1LL << 56)

/* a += x y */
FX_HD void fx_mad(long long &a, int x, int y)
{
#ifdef __CUDA_ARCH__
  asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a) : "r"(x), "r"(y));
#else
  a += (long long)x * y;
#endif
}
/* The value of the two sums of products. */
FX_HD long long fx_sum(long long hh, long long hl) { return hh + ((hl + (1LL << 27)) >> 28); }
FX_HD int2 fx_split(long long t)
{
  const int hi = (int)((t + (1LL << 27)) >> 28);
  return make_int2(hi, (int)(t - ((long long)hi << 28)));
}
FX_HD long long fx_mul(long long a, long long b)
{
  const int2 p = fx_split(a), q = fx_split(b);
  long long hh = 0, hl = 0;
  fx_mad(hh, p.x, q.x);
  fx_mad(hl, p.x, q.y);
  fx_mad(hl, p.y, q.x);
  return fx_sum(hh, hl);
}
FX_HD long long fx_sq(long long a)
{
  const int2 p = fx_split(a);
  long long hh = 0, hl = 0;
  fx_mad(hh, p.x, p.x);
  fx_mad(hl, p.x, p.y);
  return fx_sum(hh, hl + hl);
}
/* eps d rounded to the grid with the product's rounding error, |eps d| < 64. */
FX_HD long long fx_coord(double eps, double d)
{
  const double p = eps * d, e = fma(eps, d, -p);
#ifdef __CUDA_ARCH__
  return __double2ll_rn(p * FX_ONE) + __double2ll_rn(e * FX_ONE);
#else
  return llrint(p * FX_ONE) + llrint(e * FX_ONE);
#endif
}
FX_HD float fx_rsqrtf(float f)
{
#ifdef __CUDA_ARCH__
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(f));
  return y;
#else
  return 1.0f / sqrtf(f);
#endif
}
FX_HD int fx_f2i(float f)
{
#ifdef __CUDA_ARCH__
  return __float2int_rn(f);
#else
  return (int)lrintf(f);
#endif
}

/* Squared distance of two points, or FX_ONE_I where it is 1 or more (|differences| < 2^62). */
template <int DIM> FX_HD long long fx_dist2(long long dx, long long dy, long long dz)
{
  const unsigned long long big = (unsigned long long)FX_ONE_I;
  /* |d| < 1 for every component: (d + 1) in [0, 2) as unsigned */
  bool in = (unsigned long long)(dx + FX_ONE_I) < 2 * big && (unsigned long long)(dy + FX_ONE_I) < 2 * big;
  if (DIM == 3) in = in && (unsigned long long)(dz + FX_ONE_I) < 2 * big;
  if (!in) return FX_ONE_I;
  const int2 x = fx_split(dx), y = fx_split(dy);
  long long hh = 0, hl = 0;
  fx_mad(hh, x.x, x.x);
  fx_mad(hl, x.x, x.y);
  fx_mad(hh, y.x, y.x);
  fx_mad(hl, y.x, y.y);
  if (DIM == 3) {
    const int2 z = fx_split(dz);
    fx_mad(hh, z.x, z.x);
    fx_mad(hl, z.x, z.y);
  }
  return fx_sum(hh, hl + hl);
}

/* Wendland C2 (1 - r)^4 (4 r + 1) of s = r^2 < 1.  The root: R0 = round(2^28 r) from the
   single-precision reciprocal root y of s, then two Newton corrections (s - r^2) / (2 r) with the
   residuals formed exactly in integers; the second residual is a few thousand units at most. */
FX_HD long long fx_phi_c2(long long s)
{
  const int sh = (int)(s >> 28), sl = (int)(s & 0xfffffff);
  const float f = fmaf((float)sh, 268435456.0f, (float)sl);
  const float y = fx_rsqrtf(fmaxf(f, 1.0f)); /* 2^-28 / r */
  const int R0 = fx_f2i(f * y);
  long long e = s;
  fx_mad(e, R0, -R0);
  const float yc = y * 134217728.0f; /* 2^27 */
  const int D0 = fx_f2i((float)(int)((e + 32) >> 6) * yc);
  const long long r1 = ((long long)R0 << 28) + ((long long)D0 << 6);
  const int2 q = fx_split(r1);
  long long e1 = s, hl = 0, ll = 0;
  fx_mad(e1, q.x, -q.x);
  fx_mad(hl, q.x, q.y);
  fx_mad(ll, q.y, q.y);
  e1 -= (hl + hl + (ll >> 28) + (1LL << 27)) >> 28;
  const int D1 = fx_f2i((float)(int)e1 * yc);
  long long u = FX_ONE_I - (r1 + D1);
  if (u < 0) u = 0;
  const long long u2 = fx_sq(u), u4 = fx_sq(u2);
  return fx_mul(u4, 5 * FX_ONE_I - 4 * u);
}
