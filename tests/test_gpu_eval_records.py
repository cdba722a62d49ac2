"""The FP32 record kernel at the sizes where its work split changes (particles of a unit around the
powers of two that set the shares, one to many units per cell, the capacities 32, 64 and 128), with odd
and empty cells, against the FP64 path: <= 1e-6 per component, as everywhere for the FP32 evaluation,
of the largest data value (the largest interpolated value of a set of one or two particles can be
arbitrarily close to zero, and says nothing about the size of the terms that are summed)."""
import numpy as np
import pytest

import lagrbf_gb300 as L
from lagrbf_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def fields(dim, nlat, npu, xp, kernel=2, drop=None, nfields=None):
    rng = np.random.default_rng(nlat)
    xd = W.jittered_lattice(nlat, dim, rng)
    if drop is not None:
        xd = np.ascontiguousarray(xd[drop(xd)])
    fd = W.abc_flow(xd) if dim == 3 else W.cellular_flow(xd)
    if nfields and nfields > dim:
        fd = np.concatenate([fd, xd[:, :nfields - dim] + 2.0], 1)
    eps_w = npu / W.pu_overlap(npu)
    shape = 1.0 if kernel == 2 else nlat / eps_w
    out = []
    for prec in ("fp64", "fp32"):
        c = L.LagRBFCtx(dim=dim, npartitions=[npu] * dim, overlap=W.pu_overlap(npu), shape_factor=shape, kernel=kernel,
                        nfields=fd.shape[1], eval_precision=prec)
        c.fill_data(xd, fd)
        c.fill_points(xp)
        c.interpolate_c()
        assert prec == "fp64" or c.stats()["records"] == 1
        f = np.zeros((len(xp), fd.shape[1]))
        c.output(fvals=f)
        out.append(f)
    return out + [np.abs(fd).max(axis=0)]


def err(f):
    return float((np.abs(f[1] - f[0]).max(axis=0) / f[2]).max())


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 8, 9, 16, 17, 31, 32, 33, 64, 65, 127, 128, 129, 200])
def test_particles_of_one_cell(n, dim):
    xp = 0.34 + 0.3 * np.random.default_rng(n).random((n, dim))
    assert err(fields(dim, 13 if dim == 3 else 31, 4, np.ascontiguousarray(xp))) <= 1e-6


@pytest.mark.parametrize("dim,nlat,npu,npart", [(3, 20, 9, 5000), (3, 20, 9, 20000), (3, 20, 9, 60000), (2, 60, 30, 9000),
                                                (2, 60, 30, 40000)])
def test_capacities(dim, nlat, npu, npart):
    assert err(fields(dim, nlat, npu, np.random.default_rng(1).random((npart, dim)))) <= 1e-6


@pytest.mark.parametrize("kernel", [5, 6])
def test_other_kernels(kernel):
    assert err(fields(3, 15, 5, np.random.default_rng(2).random((700, 3)), kernel=kernel)) <= 1e-6


def test_empty_and_single_point_cells():
    xp = np.random.default_rng(3).random((3000, 3))
    f = fields(3, 13, 10, xp, drop=lambda x: (x[:, 0] < 0.5) | (x[:, 1] > 0.8))
    assert err(f) <= 1e-6


def test_more_fields_than_records():
    assert err(fields(3, 14, 5, np.random.default_rng(4).random((900, 3)), nfields=5)) <= 1e-6
