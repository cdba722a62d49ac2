"""The blocked patch factorisation (patches above 64 points) and its re-solve against the CPU oracle,
at patch sizes around its block and tile edges.  A PU mesh of one cell puts every data point in each
of its 2^dim patches, so the patch size is the number of points.

Tolerance: max(1e-10, 16 u kappa) max-normalised, as for the other set-up tests: the GPU's and the
oracle's factorisations round differently, and a relative change u = 2^-53 of the matrix moves the
interpolant by up to about kappa u.
"""
import numpy as np
import pytest

from oracle_lib import Oracle
import lagrbf_gb300 as L
from lagrbf_gb300 import workloads as W

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def relerr(a, b):
    den = np.abs(b).max(axis=0)
    den[den == 0] = 1.0
    return float((np.abs(a - b).max(axis=0) / den).max())


def points(m, dim, seed):
    """m jittered lattice points of [0, 1]^dim (a random subset of the smallest sufficient lattice)."""
    rng = np.random.default_rng(seed)
    n = int(np.ceil(m ** (1.0 / dim)))
    x = W.jittered_lattice(n, dim, rng)
    return np.ascontiguousarray(x[rng.permutation(len(x))[:m]])


@pytest.mark.parametrize("solve", [1, 2])
@pytest.mark.parametrize("m,dim,nf,kernel", [(64, 2, 2, 2), (65, 2, 1, 2), (66, 3, 3, 2), (95, 2, 4, 2), (96, 3, 5, 2),
                                             (97, 2, 2, 6), (127, 3, 1, 5), (128, 2, 9, 2), (129, 3, 3, 2),
                                             (160, 2, 2, 6), (161, 3, 4, 2), (257, 3, 2, 1), (300, 2, 3, 2)])
def test_factor_and_resolve_match_oracle(m, dim, nf, kernel, solve):
    xd = points(m, dim, seed=m)
    rng = np.random.default_rng(m + 1)
    xp = rng.random((200, dim))
    # Gaussian and inverse multiquadric: eps = lattice spacing^-1 keeps kappa moderate
    eps_w = 2.0 / W.pu_overlap(2)
    shape = np.ceil(m ** (1.0 / dim)) / eps_w if kernel in (5, 6) else 1.0
    opts = dict(dim=dim, npartitions=[2] * dim, overlap=W.pu_overlap(2), shape_factor=float(shape), kernel=kernel,
                nfields=nf, solve_method=solve)
    c, o = L.LagRBFCtx(**opts), Oracle(**opts)
    c.set_condition_estimates(True)
    c.fill_points(xp, pidx=np.arange(1, 201))
    assert o.fill(False, xp, pidx=np.arange(1, 201)) == 0
    for it in range(2):  # the second pass re-solves (1) or factors again (2)
        fd = rng.normal(size=(m, nf))
        c.reset_coefficients()
        c.fill_data(xd, fd)
        c.interpolate_c()
        assert o.reset() == 0 and o.fill(True, xd, fd) == 0 and o.interpolate() == 0
        f = np.zeros((200, nf))
        c.output(fvals=f)
        kap = c.condition()[1]["max"]
        assert c.stats()["max_patch"] == m
        assert relerr(f, o.output(200)[1]) <= max(1e-10, 16 * U * kap)


def test_missing_values_stay_in_their_field():
    """A NaN among the values of one field makes that field NaN and leaves the others alone."""
    m = 150
    xd = points(m, 3, seed=2)
    fd = np.random.default_rng(3).normal(size=(m, 3))
    xp = np.random.default_rng(4).random((50, 3))
    res = []
    for bad in (False, True):
        if bad:
            fd[70, 1] = np.nan
        c = L.LagRBFCtx(dim=3, npartitions=[2] * 3, overlap=W.pu_overlap(2), kernel=2, nfields=3)
        c.fill_data(xd, fd)
        c.fill_points(xp)
        c.interpolate_c()
        f = np.zeros((50, 3))
        c.output(fvals=f)
        res.append(f)
    assert np.isnan(res[1][:, 1]).all()
    assert np.array_equal(res[0][:, [0, 2]], res[1][:, [0, 2]])


@pytest.mark.parametrize("kernel,shape", [(0, 1.0), (4, 1.0), (3, 0.5)])
@pytest.mark.parametrize("m", [70, 200])
def test_not_positive_definite_is_reported(kernel, shape, m):
    """Kernels without a positive definite matrix: the same outcome as the oracle (code 81), and the
    context works afterwards."""
    xd = points(m, 2, seed=m)
    fd = np.ones((m, 1))
    xp = np.random.default_rng(1).random((20, 2))
    opts = dict(dim=2, npartitions=[2, 2], overlap=W.pu_overlap(2), shape_factor=shape, kernel=kernel, nfields=1)
    c, o = L.LagRBFCtx(**opts), Oracle(**opts)
    c.fill_data(xd, fd)
    c.fill_points(xp)
    assert o.fill(True, xd, fd) == 0 and o.fill(False, xp) == 0
    want = o.interpolate()
    if want:
        with pytest.raises(RuntimeError, match="error code 81"):
            c.interpolate_c()
    else:
        c.interpolate_c()
    assert want == 81 or kernel == 3
