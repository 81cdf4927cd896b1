"""Device partialACA (partialACA.hpp:39-171) over its three size classes: a
warp, a CTA of 128 and a CTA of 256 threads per block, at the classes' edges.

Leaves and ranks equal the oracle's (its arithmetic of rows, columns and pivots
is the device's bit for bit; only the stopping estimator's sums differ in their
order), and so the factors agree to the last bits."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu


# admissible pairs of clusters of n and m points: M + N = 26 .. 192 (a warp),
# 193 .. 2048 (128 threads), beyond (256 threads), remainders of 32 included
@pytest.mark.parametrize("n,m", [(13, 13), (96, 96), (97, 96), (130, 70), (1024, 1024), (1025, 1024), (3000, 2500)])
@pytest.mark.parametrize("kernel", [H.LAPLACE, H.INV_R_EPS])
def test_one_block_of_every_class(port, n, m, kernel):
    xt, xs = G.sphere(n, seed=n), G.sphere(m, seed=m + 1) + np.array([4.0, 0.5, 0.0])
    t, s = H.Cluster(), H.Cluster()
    t.set_minclustersize(10)
    t.build(n, xt), s.build(m, xs)
    ot, os_ = port.cluster(xt), port.cluster(xs)
    for eps in (1e-3, 1e-8):
        hm = H.HMatrix(t, s, eps, 10.0).build(kernel, xt, xs)
        OH = port.hmatrix(ot, os_, xt, xs, kernel, eps, 10.0)
        lr, dn, uv, dd = hm.get_factors()
        lr_o, dn_o, uv_o, dd_o = OH.factors()
        assert np.array_equal(lr, lr_o) and np.array_equal(dn, dn_o)
        assert np.array_equal(dd, dd_o)
        if uv.size:
            assert np.max(np.abs(uv - uv_o)) <= 1e-12 * np.max(np.abs(uv_o))
