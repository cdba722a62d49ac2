"""Patches of very different coefficients around one cell.  Two data points that nearly coincide give the patches that hold
them coefficients some 2^40 times the values; a particle of a neighbouring cell beyond the PU support of those
patches has the value that it has without the second point, since no other patch holds it."""
import numpy as np
import pytest

import lagrbf_gb300 as L
from lagrbf_gb300 import workloads as W

pytestmark = pytest.mark.gpu

NPU = 4                        # cells of h = 1/3
RADIUS = {2: 0.95, 3: 1.17}    # PU radius in spacings: the cells' corners that a particle may be beyond


def fields(dim, nlat, n, kernel, prec, near):
    h = 1.0 / (NPU - 1)
    rad = RADIUS[dim] * h
    xd = W.jittered_lattice(nlat, dim, np.random.default_rng(nlat))
    fd = np.cos(3.0 * xd @ np.arange(1.0, dim + 1.0))[:, None] * np.arange(1.0, dim + 1.0)
    if near:  # a second point next to the one nearest to the middle of cell 0
        p = np.argmin(((xd - 0.5 * h) ** 2).sum(1))
        xd = np.concatenate([xd, xd[p:p + 1] + 1e-7 * rad])
        fd = np.concatenate([fd, fd[p:p + 1] + 1.0])
    x = h + h * np.random.default_rng(2).random((200 * n, dim))  # cell (1, .., 1) shares the node at h alone with cell 0
    xp = np.ascontiguousarray(x[((x - h) ** 2).sum(1) > (1.001 * rad) ** 2][:n])
    assert len(xp) == n
    c = L.LagRBFCtx(dim=dim, npartitions=[NPU] * dim, overlap=rad * NPU, nfields=dim, kernel=kernel, eval_precision=prec,
                    shape_factor=1.0 if kernel == 2 else nlat * rad)
    c.fill_data(xd, fd)
    c.fill_points(xp)
    c.interpolate_c()
    f = np.zeros((n, dim))
    c.output(fvals=f)
    c.close()
    return f


# whole numbers in units of 2^-60 of the largest coefficients in reach (within 2^6 of the values), of some 200 runs
# of records
@pytest.mark.parametrize("kernel", [2, 6])
@pytest.mark.parametrize("n", [1, 50, 300])
@pytest.mark.parametrize("dim,nlat", [(2, 20), (3, 9)])
def test_fp64_beyond_the_support_of_large_coefficients(dim, nlat, n, kernel):
    f, g = (fields(dim, nlat, n, kernel, "fp64", near) for near in (False, True))
    assert np.abs(f).max() > 0.1
    assert np.abs(f - g).max() <= 1e-13 * np.abs(f).max()


# whole numbers in units of 2^-40 of the largest coefficients in reach or finer, of 64 segments
@pytest.mark.parametrize("kernel", [2, 5, 6])
@pytest.mark.parametrize("n", [1, 50, 300])
@pytest.mark.parametrize("dim,nlat", [(2, 20), (3, 9)])
def test_fp32_beyond_the_support_of_large_coefficients(dim, nlat, n, kernel):
    f, g = (fields(dim, nlat, n, kernel, "fp32", near) for near in (False, True))
    assert np.abs(f).max() > 0.1
    assert np.abs(f - g).max() <= 1e-9 * np.abs(f).max()
