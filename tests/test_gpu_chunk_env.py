"""LAGRBF_CHUNK, the capacity of the evaluation's work units: every value from 64 to 256 is taken, in steps of 64, by each
evaluation (the fixed-point FP64 kernel: up to 128), with the same results."""
import numpy as np
import pytest

import lagrbf_gb300 as L
from lagrbf_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def fields(monkeypatch, env, prec, kernel, nf):
    if env:
        monkeypatch.setenv("LAGRBF_CHUNK", str(env))
    xd = W.jittered_lattice(12, 3, np.random.default_rng(1))
    fd = np.random.default_rng(2).uniform(-1.0, 1.0, (len(xd), nf))
    xp = np.random.default_rng(3).random((6000, 3))
    c = L.LagRBFCtx(dim=3, npartitions=[4] * 3, overlap=W.pu_overlap(4), nfields=nf, kernel=kernel, shape_factor=1.0,
                    eval_precision=prec)
    c.fill_data(xd, fd)
    c.fill_points(xp)
    c.interpolate_c()
    f = np.zeros((6000, nf))
    c.output(fvals=f)
    cap = c.stats()["chunk_cap"]
    c.close()
    monkeypatch.delenv("LAGRBF_CHUNK", raising=False)
    return f, cap


# kernel 1: the FP64 kernel; four FP32 fields: the gather kernel
@pytest.mark.parametrize("prec,kernel,nf,most", [("fp32", 2, 3, 256), ("fp32", 2, 4, 256), ("fp64", 2, 3, 128), ("fp64", 1, 3, 256)])
def test_every_capacity_is_taken(monkeypatch, prec, kernel, nf, most):
    ref = fields(monkeypatch, None, prec, kernel, nf)[0]
    for env in (64, 100, 128, 192, 255, 256):
        f, cap = fields(monkeypatch, env, prec, kernel, nf)
        assert cap == min(env // 64 * 64, most)
        assert np.array_equal(f, ref)
