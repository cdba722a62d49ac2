"""The FP32 evaluation adds the points of a cell one after the other, in the cell's order, into each patch's sum.
Four points on a square around the particle have one kernel value phi and, farther apart than the kernel's support, a
collocation matrix that is the identity: the coefficients are the data values, and the order of the additions
decides which of them cancel before the small ones are added and which absorb them."""
import numpy as np
import pytest

import lagrbf_gb300 as L

pytestmark = pytest.mark.gpu

BIG = 2.0 ** 28  # phi * BIG absorbs phi in FP32 (24 bits)
NPU = 5          # cells of 1/4; PU radius 1/2, kernel support 1/16: every coordinate and scale is exact


def value(dim, values, n, prec):
    """Interpolated first field at n particles in the middle of the square."""
    a = 9.0 / 256.0  # half a side: corners at 0.0497 from the middle, 0.0703 apart
    mid = np.full(dim, 0.375)
    xd = np.tile(mid, (5, 1))
    xd[:4, 0] += a * np.array([-1.0, 1.0, -1.0, 1.0])
    xd[:4, 1] += a * np.array([-1.0, -1.0, 1.0, 1.0])
    xd[4] += 0.1171875  # a fifth point of the cell out of reach: an odd count
    xd = xd[:len(values)]
    fd = np.repeat(np.asarray(values, dtype=np.float64)[:, None], dim, axis=1)
    c = L.LagRBFCtx(dim=dim, npartitions=[NPU] * dim, overlap=0.5 * NPU, shape_factor=8.0, kernel=2, nfields=dim,
                    eval_precision=prec)
    c.fill_data(np.ascontiguousarray(xd), np.ascontiguousarray(fd))
    c.fill_points(np.tile(mid, (n, 1)))
    c.interpolate_c()
    assert prec == "fp64" or c.stats()["records"] == 1
    f = np.zeros((n, dim))
    c.output(fvals=f)
    c.close()
    return f


def in_order(values):
    """What is left of the additions in FP32, in units of phi."""
    acc = np.float32(0)
    for v in values[:4]:
        acc = np.float32(acc + np.float32(v))
    return float(acc)


@pytest.mark.parametrize("chunk", [None, 64, 128, 256])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("values", [(BIG, -BIG, 1, 1), (BIG, -BIG, 1, 1, 3), (1, BIG, -BIG, 1), (BIG, 1, -BIG, 1, 5),
                                    (1, 1, BIG, -BIG), (BIG, 1, 1, -BIG)])
def test_points_are_added_in_order(values, dim, chunk, monkeypatch):
    if chunk:
        monkeypatch.setenv("LAGRBF_CHUNK", str(chunk))
    one = value(dim, (0, 0, 1, 0, 0), 1, "fp64")[0, 0]
    assert one > 1e-5
    want = in_order(values) * one
    for n in (1, 40, 300):
        f = value(dim, values, n, "fp32")
        # the kernel value within 1e-5 (1 - r = 0.2 at four digits fewer than FP32's seven); units of the fold below 2^-28
        assert np.abs(f - want).max() <= 1e-5 * one + 2.0 ** -26
