"""The fixed-point arithmetic of lagrbf_gb300/csrc/lgb_fx.cuh (units of 2^-56), compiled for the host,
against long double: Wendland C2 of a squared distance, the distance from scaled coordinates, and
exp(-s).  Bounds: every product or rounding is within one unit, the distance adds three and the kernel's
slope in r^2 is at most 10, so a kernel value of exact s is within 16 units and one of rounded
coordinates within 48; exp(-s) is four products (4 units).  FP64 in the operation order of the FP64
kernels reaches 26, 31 and 9 units on the same inputs."""
import os
import subprocess

import lagrbf_gb300

CSRC = os.path.join(os.path.dirname(lagrbf_gb300.__file__), "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include "lgb_fx.cuh"
typedef long double Q;
static Q c2(Q r) { Q u = r < 1 ? 1 - r : 0; return u * u * u * u * (5 - 4 * u); }
int main()
{
  const Q one = FX_ONE;
  double a = 0, b = 0, c = 0, far = 0;
  srand48(7);
  for (long i = 0; i < 400000; i++) {
    const double r = i % 4 == 0 ? drand48() : i % 4 == 1 ? exp(-drand48() * 25)
                   : i % 4 == 2 ? 1 - exp(-drand48() * 30) : drand48() * 1e-7;
    long long s = i < 1000 ? i : (long long)(r * r * FX_ONE);
    if (s >= FX_ONE_I) s = FX_ONE_I - 1;
    a = fmax(a, (double)fabsl((Q)fx_phi_c2(s) - c2(sqrtl((Q)s / one)) * one));
    long long t = (long long)((i & 1 ? 40 : 1) * drand48() * FX_ONE);
    if (t >= FX_EXP_END) t = FX_EXP_END - 1;
    c = fmax(c, (double)fabsl((Q)fx_exp_neg(t) - expl(-(Q)t / one) * one));
  }
  for (long i = 0; i < 400000; i++) {
    const double eps = i & 1 ? 31 / 1.5 : 9.0, ref = drand48();
    Q d2 = 0;
    long long d[3];
    for (int k = 0; k < 3; k++) {
      const double x = ref + (2 * drand48() - 1) / 31, y = ref + (2 * drand48() - 1) / 31;
      d2 += ((Q)x - (Q)y) * ((Q)x - (Q)y);
      d[k] = fx_coord(eps, x - ref) - fx_coord(eps, y - ref);
    }
    const Q r = (Q)eps * sqrtl(d2);
    const long long s = fx_dist2<3>(d[0], d[1], d[2]), w = fx_dist2_wide<3>(d[0], d[1], d[2]);
    b = fmax(b, (double)fabsl((Q)(s < FX_ONE_I ? fx_phi_c2(s) : 0) - c2(r) * one));
    far = fmax(far, (double)fabsl((Q)w - r * r * one) / (1 + (double)r));
  }
  printf("%g %g %g %g\n", a, b, c, far);
}
"""


def test_fixed_point_kernels_against_long_double(tmp_path):
    src = tmp_path / "fx.cpp"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-O2", "-x", "c++", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o",
                    str(tmp_path / "fx"), "-lm"], check=True)
    a, b, c, far = map(float, subprocess.run([str(tmp_path / "fx")], check=True, stdout=subprocess.PIPE,
                                             text=True).stdout.split())
    assert a <= 16 and b <= 48 and c <= 4 and far <= 16
