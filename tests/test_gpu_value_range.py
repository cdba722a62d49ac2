"""Data values near the ends of the range.  Every step of the set-up, solve and evaluation is linear in the
values and scales them by powers of two exactly, so values times 2^k give the fields times 2^k, bit for bit."""
import numpy as np
import pytest

import lagrbf_gb300 as L
from lagrbf_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def fields(dim, nlat, npu, kernel, k, nf=2, prec="fp64", n=500):
    xd = W.jittered_lattice(nlat, dim, np.random.default_rng(nlat))
    fd = np.ldexp(np.random.default_rng(1).uniform(-1.0, 1.0, (len(xd), nf)), k)
    xp = np.random.default_rng(2).random((n, dim))
    # supports of 1.5 lattice spacings (Gaussian: eps = 2 / spacing): coefficients of the values' size
    shape = nlat / 1.5 if kernel == 2 else 2.0 * nlat
    c = L.LagRBFCtx(dim=dim, npartitions=[npu] * dim, overlap=W.pu_overlap(npu), nfields=nf, kernel=kernel,
                    shape_factor=shape * W.pu_overlap(npu) / npu, eval_precision=prec)
    c.fill_data(xd, fd)
    c.fill_points(xp)
    c.interpolate_c()
    f = np.zeros((n, nf))
    c.output(fvals=f)
    c.close()
    return f


@pytest.mark.parametrize("k", [-960, 1019])
@pytest.mark.parametrize("kernel", [2, 6])
@pytest.mark.parametrize("dim,nlat,npu", [(2, 16, 6), (2, 24, 5), (3, 12, 4)])
def test_powers_of_two_scale_the_fields(dim, nlat, npu, kernel, k):
    f = fields(dim, nlat, npu, kernel, 0)
    assert np.abs(f).max() > 0.1
    assert np.array_equal(fields(dim, nlat, npu, kernel, k), np.ldexp(f, k))


@pytest.mark.parametrize("n", [1, 500])
@pytest.mark.parametrize("kernel", [2, 6])
@pytest.mark.parametrize("dim,nlat,npu", [(2, 16, 6), (2, 24, 5), (3, 12, 4)])
def test_powers_of_two_scale_the_fp32_fields(dim, nlat, npu, kernel, n):
    """Coefficients up to 2^127 (1.9 times the values at most), sums below FP32's largest number."""
    f = fields(dim, nlat, npu, kernel, 0, dim, "fp32", n)
    assert np.abs(f).max() > 0.1 or n == 1
    assert np.array_equal(fields(dim, nlat, npu, kernel, 126, dim, "fp32", n), np.ldexp(f, 126))


@pytest.mark.parametrize("n", [1, 300])
def test_fp32_sums_beyond_fp32(n):
    """Coefficients of one size, whose sums do not fit FP32: not finite, as FP32 sums are; and an eighth bit lower they do
    fit (FP32 sums of 25 terms of one sign: 25 half units of 2^-24 and the kernel value's few)."""
    a = (np.arange(5) + 0.5) / 5
    xd = np.stack(np.meshgrid(a, a, indexing="ij"), -1).reshape(-1, 2)
    rad = 1.5
    r = np.sqrt(((xd[:, None] - xd[None]) ** 2).sum(2)) / rad
    v = ((1.0 - r) ** 4 * (4.0 * r + 1.0)).sum(1)  # Wendland C2, coefficients of 1
    xp = np.random.default_rng(1).uniform(0.2, 0.8, (n, 2))
    out = []
    for k, prec in ((127, "fp32"), (119, "fp32"), (119, "fp64")):
        c = L.LagRBFCtx(dim=2, npartitions=[2, 2], overlap=2.0 * rad, nfields=2, kernel=2, shape_factor=1.0, eval_precision=prec)
        c.fill_data(xd, np.repeat(np.ldexp(v, k)[:, None], 2, axis=1))
        c.fill_points(xp)
        c.interpolate_c()
        f = np.zeros((n, 2))
        c.output(fvals=f)
        out.append(f)
        c.close()
    assert not np.isfinite(out[0]).any()
    assert np.abs(out[1] / out[2] - 1.0).max() <= 4e-6


@pytest.mark.parametrize("n", [1, 300])
@pytest.mark.parametrize("a,b", [(-100, -100), (-100, 60), (-110, 0), (0, 100)])
def test_fp32_fields_of_different_sizes(a, b, n):
    """Two fields of the same values times 2^a and 2^b, even powers: each as alone."""
    xd = W.jittered_lattice(20, 2, np.random.default_rng(3))
    v = np.random.default_rng(1).uniform(-1.0, 1.0, (len(xd), 2))
    xp = np.random.default_rng(2).random((n, 2))
    out = []
    for e in ((0, 0), (a, b)):
        c = L.LagRBFCtx(dim=2, npartitions=[5, 5], overlap=W.pu_overlap(5), nfields=2, kernel=2, shape_factor=1.0,
                        eval_precision="fp32")
        c.fill_data(xd, np.ldexp(v, e))
        c.fill_points(xp)
        c.interpolate_c()
        f = np.zeros((n, 2))
        c.output(fvals=f)
        out.append(f)
        c.close()
    # the products of small kernel values and coefficients leave the normal range from 2^-126 on: 1e-6 of the field
    assert np.abs(np.ldexp(out[1], (-a, -b)) - out[0]).max() <= 1e-6 * np.abs(out[0]).max()
