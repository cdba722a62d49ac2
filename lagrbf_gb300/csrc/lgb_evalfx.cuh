/*
 * lgb_evalfx.cuh -- PU evaluation with FP64 accuracy in 64-bit fixed point (lgb_fx.cuh): the plain FP64
 * path for the Wendland C2 and Gaussian kernels.
 *
 * In FP64 a (particle, data point) pair takes about 31 FP64 instructions, and GB300 issues one for a
 * warp every 16 clocks per SM: 0.5 ns per pair and SM, whatever else the kernel does.  Here the
 * squared distance, the kernel value and the sums over the coefficients run on the integer pipe:
 * about 17 multiply-adds (mad.wide) for the kernel value and three per coefficient.  The kernel value
 * is within 12 units of 2^-56 of the exact one (rms 1.5; FP64: 31 and 3.6).
 *
 * One CTA of 128 threads per work unit (up to chunk_cap <= 128 particles of one cell), a lane per
 * particle.  The CTA walks the virtual segments of the cell's block (3^dim neighbour cells, in 3D the
 * centre cell in two halves, so that a record carries at most four patches), staging per data point
 *     { x, y, [z] } and { X_k[j, f] } for every field f and involved corner patch k
 * in shared memory: coordinates in units of the support radius relative to the evaluating cell's
 * origin, coefficients relative to a power of two above the largest one of the patch and field,
 * both fixed point, the coefficients as {hi, lo}.  Every lane reads the same record
 * (broadcast).  A segment's per-patch sums are exact 64-bit sums; after FXE_RUN records they
 * are folded, still as whole numbers, into the particle's field sums with the PU weights, in units that go by the
 * patches with a share in the particle's value: a patch of large coefficients (points that nearly coincide) costs no
 * bits where its weight is zero or small (one exponent for all patches of a cell left errors of 1e-3 there; 200K
 * particles in three dimensions 28.3 ms a pass with it, 28.8 with exponents of the patches).  Units of up to 64
 * particles divide the runs of records among their warps (a cell of 20 particles would otherwise leave three of
 * four warps idle); whole numbers make the result independent of it, and so of the unit's other particles.
 * The PU weights are fixed point too, divided at the end by an exact sum over the support nodes, which the
 * shares divide among themselves.
 */
#pragma once
#include "lgb_eval.cuh"
#include "lgb_fx.cuh"

#define FXE_T 128       /* threads */
#define FXE_RUN 32      /* records between folds (32 products below 2^56 stay within 63 bits) */
#define FXE_BUDGET 24576 /* bytes of staged records */
#define FXE_SHARE 8     /* PU weights from 2^-8 of the support sum on set the units of the fields */

/* Bytes of a record: coordinates (3D: padded to 32), coefficients. */
__host__ __device__ constexpr int fxe_len(int dim, int ninv, int fp)
{
  return (dim == 3 ? 32 : 16) + (ninv * fp * 8 + 15) / 16 * 16;
}

struct FxeShared {
  int exps[8][4];            /* exponents above the corner patches' coefficients, by field */
  int cnt[27], first[27], node[8], setup[8];
  int bad;                   /* fields with a coefficient that is not finite */
  long long off[27][3];      /* neighbour cell's origin relative to the cell's */
  int seg_v[28], seg_p0[28], seg_n[28], seg_base[28], nseg;
  int vs, pp;                /* planner cursor */
  int cell, pbeg, pn, blk, wsum;
  unsigned long long den[FXE_T];
  unsigned long long w[8][FXE_T]; /* phiW of the corners */
};

/* x 2^e for |e| <= 2044, in two steps (one factor has exponents from -1022 to 1023). */
__device__ __forceinline__ double fxe_scale(double x, int e)
{
  const int a = e >> 1, b = e - a;
  return x * __hiloint2double((1023 + a) << 20, 0) * __hiloint2double((1023 + b) << 20, 0);
}

template <int DIM, int KER>
__device__ __forceinline__ long long fxe_phi(long long dx, long long dy, long long dz)
{
  if constexpr (KER == KER_C2) {
    const long long s = fx_dist2<DIM>(dx, dy, dz);
    return s < FX_ONE_I ? fx_phi_c2(s) : 0;
  } else {
    const long long s = fx_dist2_wide<DIM>(dx, dy, dz);
    return s < FX_EXP_END ? fx_exp_neg(s) : 0;
  }
}

/* S w / 2^(64 - FXE_FINE), rounded, for a sum |S| < 2^61 and a weight w < 2^63.  The Gaussian kernel's sums cancel more:
   three bits finer (relative error of a field against long double, 2D, 350 points per patch: 2.2e-16; FP64
   3.0e-16; without them 3.9e-16; Wendland C2 2.0e-13 without, FP64 6.1e-13.  Against a 64-bit computation, whose
   own error is of that size and goes along with the FP64 kernel's, it is the other way round: 3.2e-16 and 2.3e-16). */
template <int KER> constexpr int fxe_fine = KER == KER_GAUSS ? 3 : 0;
template <int KER>
__device__ __forceinline__ long long fxe_weigh(long long s, unsigned long long w)
{
  constexpr int F = fxe_fine<KER>;
  const long long hi = (long long)__umul64hi((unsigned long long)s, w) - (s < 0 ? (long long)w : 0ll);
  return (hi << F) + (long long)(((((unsigned long long)s * w) >> (63 - F)) + 1) >> 1);
}

/* The runs of FXE_RUN records of a piece (n records of NI patches at rec) whose number is the share's (run: of
   the round, so far), for the lane's particle: the per-patch sums of a run are folded into val, two words per
   field, with the PU weights w[corner * FXE_T], which carry the patches' exponents ex[corner][field] relative to the
   particle's: w 2^(ex - ef) stays below bit 63.  A run's fold is a whole number that does not depend on which
   share does it, and so neither does their sum. */
template <int DIM, int FP, int KER, int NI>
__device__ __forceinline__ void fxe_segment(const unsigned char *rec, int n, int sh, int ns, int &run, long long px, long long py,
                                            long long pz, unsigned mask, const unsigned long long *w, const int (*ex)[4],
                                            const int (&ef)[FP], int ws, long long (&val)[FP][2])
{
  constexpr int LEN = fxe_len(DIM, NI, FP), HEAD = DIM == 3 ? 32 : 16;
  for (int p0 = 0; p0 < n; p0 += FXE_RUN, run++) {
    if ((run & (ns - 1)) != sh) continue;
    const int p1 = min(n, p0 + FXE_RUN);
    long long hh[NI * FP], hl[NI * FP];
#pragma unroll
    for (int q = 0; q < NI * FP; q++) { hh[q] = 0; hl[q] = 0; }
#pragma unroll 1
    for (int p = p0; p < p1; p++) {
      const unsigned char *r = rec + (size_t)p * LEN;
      const longlong2 xy = *reinterpret_cast<const longlong2 *>(r);
      const long long z = (DIM == 3) ? *reinterpret_cast<const long long *>(r + 16) : 0;
      const long long phi = fxe_phi<DIM, KER>(px - xy.x, py - xy.y, pz - z);
      const int2 f = fx_split(phi);
      const int4 *c = reinterpret_cast<const int4 *>(r + HEAD);
#pragma unroll
      for (int q = 0; q < NI * FP; q += 2) {
        const int4 v = c[q / 2];
        fx_mad(hh[q], f.x, v.x);
        fx_mad(hl[q], f.x, v.y);
        fx_mad(hl[q], f.y, v.x);
        if (q + 1 < NI * FP) {
          fx_mad(hh[q + 1], f.x, v.z);
          fx_mad(hl[q + 1], f.x, v.w);
          fx_mad(hl[q + 1], f.y, v.z);
        }
      }
    }
    unsigned m = mask;
#pragma unroll
    for (int j = 0; j < NI; j++) {
      const int k = __ffs(m) - 1;
      const unsigned long long wk = w[k * FXE_T];
      m &= m - 1;
#pragma unroll
      for (int f = 0; f < FP; f++) {
        const int up = ws - ef[f] + ex[k][f];
        const long long v = fxe_weigh<KER>(fx_sum(hh[j * FP + f], hl[j * FP + f]), up >= 0 ? wk << min(up, 63) : wk >> min(-up, 63));
        val[f][0] += v & 0xffffffffll;
        val[f][1] += v >> 32;
      }
    }
  }
}

template <int DIM, int FP, int KER>
__global__ void __launch_bounds__(FXE_T, 4) k_eval_fx(EvalParams P)
{
  constexpr int NEN = EGeo<DIM>::NEN, NOFF = EGeo<DIM>::NOFF, NVS = VGeo<DIM>::NVS;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ FxeShared S;
  const lgb_geom &g = P.g;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chunk = blockIdx.x;
  if (chunk >= P.chunk_start[g.ncells]) return;
  if (tid < 32) {
    /* the work unit's cell: the last cell c with chunk_start[c] <= chunk (a 32-way search) */
    int lo = 0, hi = g.ncells - 1;
    while (hi > lo) {
      const int step = (hi - lo + 32) / 32;
      const int c = min(lo + lane * step, hi);
      const unsigned le = __ballot_sync(0xffffffffu, P.chunk_start[c] <= chunk);
      const int last = 31 - __clz(le);
      const int nlo = min(lo + last * step, hi);
      hi = min(nlo + step - 1, hi);
      lo = nlo;
      if (step == 1) hi = lo;
    }
    if (tid == 0) {
      const int c = lo, q = chunk - P.chunk_start[c], nch = P.chunk_start[c + 1] - P.chunk_start[c];
      const int ncell = P.pstart[c + 1] - P.pstart[c];
      const int b0 = (int)(((long long)ncell * q) / nch), b1 = (int)(((long long)ncell * (q + 1)) / nch);
      S.cell = c;
      S.pbeg = P.pstart[c] + b0;
      S.pn = b1 - b0;
      S.wsum = 0;
      S.bad = 0;
      S.vs = 0;
      S.pp = 0;
    }
  }
  __syncthreads();
  const int cell = S.cell, pn = S.pn;
  int ci, cj, cl;
  lgb_cell_ijk(g, cell, ci, cj, cl);
  const int cc[3] = {ci, cj, cl};
  double org[3];
#pragma unroll
  for (int d = 0; d < 3; d++) org[d] = g.O[d] + g.h[d] * cc[d];
  cell_block<DIM>(P, cell, S.cnt, S.first, S.node, S.setup);
  if (tid < NOFF * DIM) {
    const int o = tid / DIM, d = tid - o * DIM;
    const int a = d == 0 ? eoff_a(o) : d == 1 ? eoff_b(o) : eoff_e(DIM, o);
    S.off[o][d] = fx_coord(g.eps_r, (g.O[d] + g.h[d] * (cc[d] + a)) - org[d]);
  }
  __syncthreads();
  if (tid < NEN * FP) {
    const int k = tid / FP, f = tid - k * FP, e = S.setup[k] ? P.cexp[(size_t)S.node[k] * P.F + P.f0 + f] : LGB_CEXP_ZERO;
    S.exps[k][f] = e == LGB_CEXP_NAN ? LGB_CEXP_ZERO : e;
    if (e == LGB_CEXP_NAN) atomicOr(&S.bad, 1 << f);
  }
  if (tid == 32) {
    int nb = 0;
    for (int o = 0; o < NOFF; o++) nb += S.cnt[o];
    S.blk = nb;
  }
  /* groups of 32 particles; a group's warps share its records and support nodes */
  const int ng = (pn + 31) / 32, ns = ng == 1 ? 4 : ng == 2 ? 2 : 1, grp = warp % ng, sh = warp / ng;
  const bool active = sh < ns;
  const int idx = 32 * grp + lane; /* lanes beyond the unit repeat its last particle */
  const int pid = P.plist[S.pbeg + min(idx, pn - 1)];
  double x[3];
  long long pq[3] = {0, 0, 0};
#pragma unroll
  for (int d = 0; d < DIM; d++) {
    x[d] = P.xp[(size_t)pid * DIM + d];
    pq[d] = fx_coord(g.eps_r, x[d] - org[d]);
  }
  S.den[tid] = 0ull;
#pragma unroll
  for (int k = 0; k < NEN; k++) S.w[k][tid] = 0ull; /* corners beyond the support */
  __syncthreads();
  if (S.blk == 0) return; /* empty neighbourhood: the value is left untouched (interpolation.c:89) */

  /* PU weights: phiW over the support nodes (exact integer sum), the corners' kept */
  int wloc = 0;
  if (active) {
    int lo[3] = {0, 0, 0}, hi[3] = {0, 0, 0};
    long long pw[3] = {0, 0, 0};
#pragma unroll
    for (int d = 0; d < DIM; d++) {
      eval_node_range(x[d], g.O[d], g.rh[d], g.n[d], g.rad_w, lo[d], hi[d]);
      pw[d] = fx_coord(g.eps_w, x[d] - org[d]);
    }
    unsigned long long den = 0;
    const int n0 = hi[0] - lo[0] + 1, n1 = hi[1] - lo[1] + 1, n2 = hi[2] - lo[2] + 1;
    for (int q = sh; q < n0 * n1 * n2; q += ns) {
      const int k = q / (n0 * n1), r = q - k * n0 * n1, j = r / n0, ijk[3] = {lo[0] + r - j * n0, lo[1] + j, lo[2] + k};
      long long dd[3] = {0, 0, 0};
#pragma unroll
      for (int d = 0; d < DIM; d++) dd[d] = pw[d] - fx_coord(g.eps_w, (g.O[d] + g.h[d] * ijk[d]) - org[d]);
      const long long s = fx_dist2<DIM>(dd[0], dd[1], dd[2]);
      const long long v = s < FX_ONE_I ? fx_phi_c2(s) : 0;
      den += (unsigned long long)v;
      wloc += v > 0;
      const int a = ijk[0] - ci, b = ijk[1] - cj, e = ijk[2] - cl;
      if ((unsigned)a < 2 && (unsigned)b < 2 && (unsigned)e < 2)
        S.w[(b ? 3 - a : a) + (DIM == 3 ? 4 * e : 0)][idx] = (unsigned long long)v; /* corner of the cell */
    }
    atomicAdd(&S.den[idx], den);
    if (idx >= pn) wloc = 0;
  }
  __syncthreads();
  /* The support sum in bit 62 (the division by it comes last), and the fields' exponents: the largest ex of the patches
     with a share of 2^-8 or more in the sum, and large enough that w 2^(ex - ef) stays below bit 63 for the others. */
  const int ws = __clzll((long long)max(S.den[idx], 1ull)) - 1;
  int ef[FP];
#pragma unroll
  for (int f = 0; f < FP; f++) ef[f] = LGB_CEXP_ZERO;
#pragma unroll
  for (int k = 0; k < NEN; k++) {
    const unsigned long long wk = S.w[k][idx];
    const int over = max(wk ? __clzll((long long)wk) - ws - 1 : INT_MAX, 0); /* bits of the sum above the weight's */
#pragma unroll
    for (int f = 0; f < FP; f++)
      if (wk) ef[f] = max(ef[f], S.exps[k][f] - (over <= FXE_SHARE ? 0 : over));
  }

  long long val[FP][2];
#pragma unroll
  for (int f = 0; f < FP; f++) val[f][0] = val[f][1] = 0;
  for (;;) {
    if (tid == 0) { /* the next round of records */
      int vs = S.vs, pp = S.pp, base = 0, nseg = 0;
      while (vs < NVS) {
        const int c = S.cnt[c_masks.vo[DIM - 2][vs]] - pp;
        if (c <= 0) { vs++; pp = 0; continue; }
        const int len = fxe_len(DIM, __popc(c_masks.vs[DIM - 2][vs]), FP), fit = (FXE_BUDGET - base) / len;
        if (fit <= 0) break;
        const int take = min(c, fit);
        S.seg_v[nseg] = vs; S.seg_p0[nseg] = pp; S.seg_n[nseg] = take; S.seg_base[nseg] = base;
        nseg++;
        base += take * len;
        pp += take;
      }
      S.vs = vs;
      S.pp = pp;
      S.nseg = nseg;
    }
    __syncthreads();
    const int nseg = S.nseg;
    if (nseg == 0) break;
    for (int i = 0; i < nseg; i++) {
      const int vs = S.seg_v[i], o = c_masks.vo[DIM - 2][vs], mask = c_masks.vs[DIM - 2][vs], ni = __popc(mask);
      const int len = fxe_len(DIM, ni, FP), n = S.seg_n[i], p0 = S.seg_p0[i];
      unsigned char *dst = smem_raw + S.seg_base[i];
      for (int t = tid; t < n * DIM; t += FXE_T) {
        const int p = t / DIM, d = t - p * DIM;
        *reinterpret_cast<long long *>(dst + (size_t)p * len + 8 * d) =
            P.xq[(size_t)(S.first[o] + p0 + p) * DIM + d] + S.off[o][d];
      }
      for (int j = 0, m = mask; j < ni; j++, m &= m - 1) {
        const int k = __ffs(m) - 1;
        const long long pos = P.coff[S.node[k]] + P.slot[S.node[k] * 8 + eslot(DIM, k, o)] + p0;
        const bool on = S.setup[k];
        for (int t = tid; t < n * FP; t += FXE_T) {
          const int p = t / FP, f = t - p * FP;
          int2 v = make_int2(0, 0);
          if (on && !((S.bad >> f) & 1)) {
            const double c = P.c64[(size_t)(pos + p) * P.F + P.f0 + f];
            /* c 2^(56 - e) by the exponent field; what is too small for it is below half a unit */
            const int up = 56 - S.exps[k][f], hi = __double2hiint(c), ec = (hi >> 20) & 2047;
            if (ec > 0 && ec + up > 0) v = fx_split(__double2ll_rn(__hiloint2double(hi + (up << 20), __double2loint(c))));
          }
          *reinterpret_cast<int2 *>(dst + (size_t)p * len + (DIM == 3 ? 32 : 16) + 8 * (j * FP + f)) = v;
        }
      }
    }
    __syncthreads();
    int run = 0;
    if (active)
      for (int i = 0; i < nseg; i++) {
        const int mask = c_masks.vs[DIM - 2][S.seg_v[i]], n = S.seg_n[i];
        const unsigned char *rec = smem_raw + S.seg_base[i];
        const unsigned long long *w = &S.w[0][idx];
        switch (__popc(mask)) {
        case 1: fxe_segment<DIM, FP, KER, 1>(rec, n, sh, ns, run, pq[0], pq[1], pq[2], mask, w, S.exps, ef, ws, val); break;
        case 2: fxe_segment<DIM, FP, KER, 2>(rec, n, sh, ns, run, pq[0], pq[1], pq[2], mask, w, S.exps, ef, ws, val); break;
        default: fxe_segment<DIM, FP, KER, 4>(rec, n, sh, ns, run, pq[0], pq[1], pq[2], mask, w, S.exps, ef, ws, val); break;
        }
      }
    __syncthreads();
  }

  /* the shares' sums through the drained staging buffer */
  long long *red = reinterpret_cast<long long *>(smem_raw);
  if (active && sh > 0)
#pragma unroll
    for (int f = 0; f < FP; f++)
      for (int h = 0; h < 2; h++) red[(((sh - 1) * FP + f) * 2 + h) * (FXE_T / 2) + idx] = val[f][h];
  __syncthreads();
  if (active && sh == 0 && idx < pn) {
    double *o = P.out + (size_t)pid * P.out_stride;
    const double den = (double)(long long)S.den[idx], sc = den > 0.0 ? __hiloint2double((1023 + 8 - fxe_fine<KER> - ws) << 20, 0) / den : 0.0;
#pragma unroll
    for (int f = 0; f < FP; f++) {
      for (int k = 1; k < ns; k++)
        for (int h = 0; h < 2; h++) val[f][h] += red[(((k - 1) * FP + f) * 2 + h) * (FXE_T / 2) + idx];
      val[f][1] += val[f][0] >> 32;
      const double v = fma((double)val[f][1], 4294967296.0, (double)(val[f][0] & 0xffffffffll)) * sc;
      o[f] = (S.bad >> f) & 1 ? __hiloint2double(0x7ff80000, 0) : fxe_scale(v, ef[f]);
    }
  }
  /* algorithmic work of this unit (the same count as the FP64 kernel) */
  for (int off = 16; off > 0; off >>= 1) wloc += __shfl_down_sync(0xffffffffu, wloc, off);
  if (lane == 0) atomicAdd(&S.wsum, wloc);
  __syncthreads();
  if (tid < 32) {
    const long long msum = emask_products<DIM>(S.cnt, S.setup);
    if (tid > 0) return;
    const int kphi = KER == KER_GAUSS ? 4 : 8;
    const long long fl = pn * ((long long)S.blk * (10 + kphi) + 2 * FP * msum + NEN * (2 * FP + 1)) + 18LL * S.wsum;
    const long long by = (long long)pn * (8 * DIM + 4 + 8 * FP) + S.blk * 8LL * DIM + msum * FP * 8;
    atomicAdd(&P.ctrl->eval_flops, (double)fl);
    atomicAdd(&P.ctrl->eval_bytes, (double)by);
  }
}
