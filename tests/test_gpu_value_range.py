"""Data values near the ends of the FP64 range.  Every step of the set-up, solve and FP64 evaluation is linear in the
values and scales them by powers of two exactly, so values times 2^k give the fields times 2^k, bit for bit."""
import numpy as np
import pytest

import lagrbf_gb300 as L
from lagrbf_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def fields(dim, nlat, npu, kernel, k):
    xd = W.jittered_lattice(nlat, dim, np.random.default_rng(nlat))
    fd = np.ldexp(np.random.default_rng(1).uniform(-1.0, 1.0, (len(xd), 2)), k)
    xp = np.random.default_rng(2).random((500, dim))
    # supports of 1.5 lattice spacings (Gaussian: eps = 2 / spacing): coefficients of the values' size
    shape = nlat / 1.5 if kernel == 2 else 2.0 * nlat
    c = L.LagRBFCtx(dim=dim, npartitions=[npu] * dim, overlap=W.pu_overlap(npu), nfields=2, kernel=kernel,
                    shape_factor=shape * W.pu_overlap(npu) / npu)
    c.fill_data(xd, fd)
    c.fill_points(xp)
    c.interpolate_c()
    f = np.zeros((500, 2))
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
