"""The FP32 gather kernel where the work units are cut small: sparse particles, and more fields than the record blocks
hold or no record blocks at all.  Against the FP64 path: <= 1e-6 per component, as everywhere for the FP32
evaluation, of the largest data value."""
import numpy as np
import pytest

import lagrbf_gb300 as L
from lagrbf_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def fields(dim, nlat, npu, xp, nfields, refill=None):
    xd = W.jittered_lattice(nlat, dim, np.random.default_rng(nlat))
    fd = W.abc_flow(xd) if dim == 3 else W.cellular_flow(xd)
    fd = np.concatenate([fd] + [np.cos((k + 2) * xd[:, :1]) for k in range(nfields - dim)], 1)
    out = []
    for prec in ("fp64", "fp32"):
        c = L.LagRBFCtx(dim=dim, npartitions=[npu] * dim, overlap=W.pu_overlap(npu), shape_factor=1.0, kernel=2,
                        nfields=nfields, eval_precision=prec)
        c.fill_data(xd, fd)
        c.fill_points(xp)
        if refill:
            refill(c, xd, fd)
        c.interpolate_c()
        assert prec == "fp64" or c.stats()["records"] == (0 if refill else 1)
        f = np.zeros((len(xp), nfields))
        c.output(fvals=f)
        out.append(f)
        c.close()
    return float((np.abs(out[1] - out[0]).max(axis=0) / np.abs(fd).max(axis=0)).max())


# more cells in use than four units per SM, of 1 to 90 particles on average
@pytest.mark.parametrize("npart", [3000, 20000, 60000, 120000])
@pytest.mark.parametrize("dim,nlat,npu,nfields", [(3, 22, 12, 4), (3, 22, 12, 5), (3, 22, 12, 7), (2, 80, 37, 3), (2, 80, 37, 6)])
def test_more_fields_than_records(dim, nlat, npu, nfields, npart):
    xp = np.random.default_rng(npart).random((npart, dim))
    assert fields(dim, nlat, npu, xp, nfields) <= 1e-6


@pytest.mark.parametrize("dim,nlat,npu", [(3, 22, 12), (2, 80, 37)])
def test_records_dropped_after_the_particles(dim, nlat, npu, monkeypatch):
    """Units cut for the record blocks of the first data, and second data whose blocks are not kept."""
    xp = np.random.default_rng(5).random((9000, dim))

    def refill(c, xd, fd):
        monkeypatch.setenv("LAGRBF_RECORDS_MAX_GB", "0")
        c.fill_data(np.ascontiguousarray(xd[::-1]), np.ascontiguousarray(fd[::-1]))
        monkeypatch.delenv("LAGRBF_RECORDS_MAX_GB")

    assert fields(dim, nlat, npu, xp, dim, refill) <= 1e-6


def test_interpolation_after_advection_steps():
    """Three velocity fields from the records during the step, all four by the gather kernel at its end."""
    dim, npu, nlat = 3, 12, 22
    xd = W.jittered_lattice(nlat, dim, np.random.default_rng(1))
    fd = np.concatenate([W.abc_flow(xd), np.cos(xd[:, :1])], 1)
    xp = np.random.default_rng(2).random((9000, dim))
    out = []
    for prec in ("fp64", "fp32"):
        c = L.LagRBFCtx(dim=dim, npartitions=[npu] * dim, overlap=W.pu_overlap(npu), shape_factor=1.0, kernel=2, nfields=4,
                        eval_precision=prec, advection=True, advection_scheme=2, dt=1e-3)
        c.fill_data(xd, fd)
        c.fill_points(xp)
        c.interpolate_c()
        c.advect_interpolate_c(0.0, 1e-3)
        f = np.zeros((len(xp), 4))
        c.output(fvals=f)
        out.append(f)
        c.close()
    alive = np.abs(out[0]).max(axis=1) > 0
    # the FP32 positions differ by dt times the FP32 error; the field's Lipschitz constant is some 2 pi
    assert (np.abs(out[1] - out[0])[alive].max(axis=0) / np.abs(fd).max(axis=0)).max() <= 2e-6
