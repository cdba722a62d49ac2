"""FP64 evaluation with PU supports that hardly reach a cell's middle (half a diagonal: 0.707 spacings in 2D, 0.866 in 3D),
where every PU weight is small and only their ratios count.  Against the CPU oracle, tolerance as in
test_gpu_eval_fixed.py (a weight (1 - r)^4 (4 r + 1) has the relative error 4 u / (1 - r), here below 1e-12)."""
import numpy as np
import pytest

from test_gpu_eval_fixed import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [2, 6])
@pytest.mark.parametrize("over", [1.0005, 1.01, 1.3, 1.36])
@pytest.mark.parametrize("dim,nlat,npu", [(2, 24, 5), (3, 12, 4)])
def test_particles_in_the_middle_of_the_cells(dim, nlat, npu, over, kernel):
    radius = over * 0.5 * dim ** 0.5  # in spacings
    g = np.random.default_rng(4)
    xp = (g.integers(0, npu - 1, (400, dim)) + 0.5 + 1e-4 * g.uniform(-1.0, 1.0, (400, dim))) / (npu - 1)
    ov = radius * npu / (npu - 1)
    shape = 1.0 if kernel == 2 else nlat * radius / (npu - 1)
    err, tol = run(dim, nlat, npu, 400, 2, kernel, shape=shape, overlap=ov, xp=xp)
    assert err <= tol
