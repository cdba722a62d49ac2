"""A particle's interpolated value does not depend on the other particles: evaluation work units are cut, and
their records divided among threads, by the number of particles that share a cell, and the sums are whole
numbers, so any division gives the same bits.  Sharded and repeated runs rest on it."""
import numpy as np
import pytest

import lagrbf_gb300 as L
from lagrbf_gb300 import workloads as W

pytestmark = pytest.mark.gpu


def particles(dim, npu, rng):
    """0 to some 300 particles per cell (every power of two that sets a division on either side), in no order."""
    nc = npu - 1
    counts = rng.permutation(np.r_[[0, 1, 2, 3, 5, 8, 9, 16, 17, 31, 32, 33, 63, 64, 65, 127, 128, 129, 200, 257, 300],
                                   rng.integers(0, 40, 200)])[:nc ** dim]
    ijk = np.stack(np.unravel_index(np.repeat(np.arange(len(counts)), counts), (nc,) * dim), 1)
    x = (ijk + rng.random(ijk.shape)) / nc
    return np.ascontiguousarray(x[rng.permutation(len(x))])


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("dim,kernel,nlat,npu", [(3, 2, 24, 7), (3, 6, 24, 7), (2, 2, 60, 10), (2, 1, 40, 6)])
def test_values_do_not_depend_on_the_set(dim, kernel, nlat, npu, prec):
    rng = np.random.default_rng(nlat + kernel)
    xd = W.jittered_lattice(nlat, dim, rng)
    fd = W.abc_flow(xd) if dim == 3 else W.cellular_flow(xd)
    xp = particles(dim, npu, rng)
    eps_w = npu / W.pu_overlap(npu)
    c = L.LagRBFCtx({"setup_all_patches": True}, dim=dim, npartitions=[npu] * dim, overlap=W.pu_overlap(npu),
                    shape_factor=nlat / eps_w if kernel == 6 else 1.0, kernel=kernel, nfields=dim, eval_precision=prec)
    c.fill_data(xd, fd)

    def values(x):
        c.fill_points(np.ascontiguousarray(x), pidx=np.arange(1, len(x) + 1))
        c.interpolate_c()
        f = np.zeros((len(x), dim))
        c.output(fvals=f)
        return f

    ref = values(xp)
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0.1
    perm = rng.permutation(len(xp))
    assert np.array_equal(values(xp[perm]), ref[perm])
    big = np.repeat(xp, 64, axis=0)                      # units of several hundred particles
    assert np.array_equal(values(big), np.repeat(ref, 64, axis=0))
    for share in (2, 5, len(xp) // 7):
        for first in range(min(share, 2)):
            assert np.array_equal(values(xp[first::share]), ref[first::share])
    c.close()
