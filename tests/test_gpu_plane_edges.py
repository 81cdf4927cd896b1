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
