"""The fixed-point FP64 evaluation (Wendland C2 and Gaussian kernels) against the CPU oracle: every
field count of a launch and of split launches, both kernels, work units of few and of many particles
(shares of the records per warp, the capacities 32, 64 and 128), cells without data, boundary cells;
and the extents where the FP64 kernel takes over.  Tolerance: max(1e-10, 16 u kappa) max-normalised
(the factorisations round differently; see test_gpu_precision.py)."""
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


def run(dim, nlat, npu, npart, nf, kernel, shape=None, overlap=None, scale=1.0, box=1.0, seed=3, xp=None, drop=None):
    rng = np.random.default_rng(seed)
    xd = W.jittered_lattice(nlat, dim, rng)
    if drop is not None:
        xd = np.ascontiguousarray(xd[drop(xd)])
    fd = rng.normal(size=(len(xd), nf)) * scale
    xp = rng.random((npart, dim)) if xp is None else xp
    ov = W.pu_overlap(npu) if overlap is None else overlap
    sh = (nlat / (npu / ov) if kernel == 6 else 1.0) if shape is None else shape
    opts = dict(dim=dim, npartitions=[npu] * dim, overlap=ov, shape_factor=float(sh), kernel=kernel, nfields=nf,
                maxCoords=[box] * dim)
    c, o = L.LagRBFCtx(**opts), Oracle(**opts)
    c.set_condition_estimates(True)
    xd, xp = xd * box, xp * box
    c.fill_data(xd, fd)
    c.fill_points(xp)
    c.interpolate_c()
    assert o.fill(True, xd, fd) == 0 and o.fill(False, xp) == 0 and o.interpolate() == 0
    f = np.zeros((len(xp), nf))
    c.output(fvals=f)
    return relerr(f, o.output(len(xp))[1]), max(1e-10, 16 * U * c.condition()[1]["max"])


@pytest.mark.parametrize("kernel", [2, 6])
@pytest.mark.parametrize("dim,nlat,npu,npart,nf", [(2, 20, 3, 1, 1), (2, 20, 3, 33, 2), (2, 24, 5, 700, 3),
                                                   (2, 24, 5, 9000, 5), (3, 12, 4, 5, 3), (3, 12, 4, 300, 4),
                                                   (3, 12, 3, 2500, 1), (3, 13, 6, 4000, 6)])
def test_matches_oracle(dim, nlat, npu, npart, nf, kernel):
    err, tol = run(dim, nlat, npu, npart, nf, kernel)
    assert err <= tol


def test_many_units_use_full_capacity():
    err, tol = run(2, 40, 9, 60000, 2, 2)
    assert err <= tol


def test_particles_on_data_points_faces_and_corners():
    x = np.random.default_rng(3)
    xd = W.jittered_lattice(14, 3, np.random.default_rng(3))
    grid = np.stack(np.meshgrid(*[np.linspace(0, 1, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)
    xp = np.concatenate([xd[::7], np.nextafter(xd[::11], 2.0).clip(0, 1), grid, x.random((50, 3))])
    err, tol = run(3, 14, 4, len(xp), 3, 2, xp=np.ascontiguousarray(xp))
    assert err <= tol


def test_empty_neighbourhoods_and_uneven_cells():
    err, tol = run(3, 16, 8, 600, 3, 2, drop=lambda x: (x[:, 0] < 0.4) | (x.sum(1) > 2.4))
    assert err <= tol


@pytest.mark.parametrize("scale", [1e-200, 1e-12, 1e150])
def test_scales_of_the_values(scale):
    err, tol = run(3, 12, 4, 300, 3, 2, scale=scale)
    assert err <= tol


@pytest.mark.parametrize("box", [1e-6, 1.0, 6.4e6])
def test_scales_of_the_box(box):
    err, tol = run(3, 12, 4, 300, 3, 2, box=box)
    assert err <= tol


@pytest.mark.parametrize("kw", [dict(shape=200.0), dict(overlap=30.0, shape=20.0), dict(kernel=1), dict(overlap=0.9)])
def test_beyond_the_fixed_point_extent(kw):
    """Supports far smaller than a cell, PU weights over many nodes (the FP64 kernel), another kernel, and
    PU supports smaller than a cell's diagonal."""
    kw = dict(dict(kernel=2), **kw)
    err, tol = run(2, 24, 5, 500, 2, kw.pop("kernel"), **kw)
    assert err <= tol


def test_precision_switch_rebins_the_work_units():
    rng = np.random.default_rng(5)
    xd = W.jittered_lattice(16, 3, rng)
    fd = W.abc_flow(xd)
    xp = rng.random((3000, 3))
    c = L.LagRBFCtx(dim=3, npartitions=[5] * 3, overlap=W.pu_overlap(5), kernel=2, nfields=3)
    c.fill_data(xd, fd)
    c.fill_points(xp)
    out = []
    for fp32 in (0, 1, 0):
        c.set_precision(fp32)
        c.interpolate_c()
        f = np.zeros((3000, 3))
        c.output(fvals=f)
        out.append(f)
    assert np.array_equal(out[0], out[2])
    assert relerr(out[1], out[0]) <= 1e-6
