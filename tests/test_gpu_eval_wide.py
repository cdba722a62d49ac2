"""FP64 evaluation with PU supports of 6.4 to 8.3 node spacings, around the radius from which the sum of the PU weights
no longer fits the fixed-point kernel (7.5 in 3D).  Against the CPU oracle, tolerance as in
test_gpu_eval_fixed.py."""
import pytest

from test_gpu_eval_fixed import run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [2, 6])
@pytest.mark.parametrize("radius", [6.4, 6.98, 7.3, 7.6, 7.98, 8.3])
@pytest.mark.parametrize("dim,nlat,npu", [(3, 20, 18), (2, 50, 20)])
def test_wide_pu_supports(dim, nlat, npu, radius, kernel):
    ov = radius * npu / (npu - 1)
    shape = radius / 1.5 if kernel == 2 else nlat * radius / (npu - 1)
    err, tol = run(dim, nlat, npu, 400, 2, kernel, shape=shape, overlap=ov)
    assert err <= tol
