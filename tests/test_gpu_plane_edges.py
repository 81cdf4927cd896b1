"""FP64 products on the digit planes (oz.cu) at the edges of their passes of
64 right-hand sides, panels of few and of 17 to 32 rows and passes of several
accumulation rounds, against this library's FP64-pipe products of the same
leaves (htool's mvprod_global_to_global, types/hmatrix.hpp:1074-1182).

Tolerance: the planes keep 54 bits of each operand relative to its row, column
or panel and drop the digit pairs 2^-48 below the leading one; over the some
hundred columns of a row, of random sign, that is below 2^-48 sqrt(1000) < 2e-13."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [700, 6000, 20000])
@pytest.mark.parametrize("mu", [8, 63, 64, 65, 129])
def test_passes_and_panels(n, mu):
    pts = G.ellipsoid(n, (1.0, 0.6, 1.4), seed=n)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts)
    hm.set_digit_planes(True)
    assert hm.get_digit_planes()[1] > 0
    x = G.rhs(n, mu, seed=mu).reshape(mu, n)
    x[mu // 2] *= 1e-40  # every right-hand side keeps its own scale
    y = hm.mvprod_global_to_global(x.reshape(-1), mu).reshape(mu, n)
    assert hm.device_status() == 0
    hm.set_fp64_split(1000, 1000)
    for c in sorted({0, 1, mu // 2, mu - 1}):
        r = hm.mvprod_global_to_global(x[c].copy(), 1)
        assert np.linalg.norm(y[c] - r) < 2e-13 * np.linalg.norm(r), c


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_largest_digit_sums(sign):
    """entries and inputs whose middle digits are all -64: the plane products
    of 256 rows sum to 2^20 each, the most an accumulator can hold"""
    n, mu = 512, 64
    v = -float(32 * 128**7 + 64 * sum(128**k for k in range(2, 7))) * 2.0**-54
    pts = G.sphere(n, seed=2)
    t = H.Cluster().build(n, pts)
    lr = np.array([[0, 0, 256, 256, 1]], np.int32)
    uv = np.concatenate([np.ones(256), np.full(256, sign * v)])
    dn = np.array([[256 + 32 * k, 256 * (k % 2), 32, 256] for k in range(8)], np.int32)
    dd = np.full(8 * 32 * 256, sign * v)
    hm = H.HMatrix(t, t, 1e-6, 10.0).set_leaves(lr, uv, dn, dd)
    x = np.full(n * mu, v)
    want = sign * 256 * v * v
    hm.set_digit_planes(True)
    y = hm.mvprod_global_to_global(x, mu)
    assert np.abs(y - want).max() <= 1e-13 * abs(want)
    assert hm.device_status() == 0
