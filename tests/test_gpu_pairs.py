"""FP64 products on paired panels (pair.cu), the kernels FP64 products run
on unless the caller chose a split or a phase mode: against the oracle's
product of its own H-matrix (htool's mvprod_global_to_global,
types/hmatrix.hpp:1074-1182, restated in oracle/htool_oracle.c) and against
this library's FP64-pipe kernels, at the panels' edges.

Tolerances: the oracle comparison keeps the 1e-12 of the FP64 parity tests.
Against the FP64 pipe on the same leaves: both factors and the input are
split to 2^-48, and a sum of K terms adds at most K roundings of 2^-48 of its
partial sums; with K below 2^10 terms a slice and the terms' signs at random
that stays below 2^-48 sqrt(K) 3 < 4e-13."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu

ORACLE_TOL = 1e-12
PIPE_TOL = 4e-13


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# 12 .. 33 points: one dense leaf of an odd, an even, a full and a just cut
# panel; 513: both phases with remainders; 3000: tiles of several panels
@pytest.mark.parametrize("n", [12, 31, 32, 33, 513, 3000])
@pytest.mark.parametrize("mu", [1, 2, 3, 5, 8, 9, 15])
def test_products_at_the_panels_edges(port, n, mu):
    pts = G.ellipsoid(n, (1.0, 0.7, 1.3), seed=n)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts)
    x = G.rhs(n, mu, seed=mu)
    y = hm.mvprod_global_to_global(x, mu)
    ot = port.cluster(pts)
    assert rel(y, port.hmatrix(ot, ot, pts, pts, H.LAPLACE, 1e-6, 10.0).mvprod(x, mu)) < ORACLE_TOL
    assert np.array_equal(y, hm.mvprod_global_to_global(x, mu))
    hm.set_fp64_split(1000, 1000)
    assert rel(y, hm.mvprod_global_to_global(x, mu)) < PIPE_TOL


@pytest.mark.parametrize("mu", [1, 4])
def test_rectangular_products_and_transposes(port, mu):
    """targets and sources of different sizes; sources of more than one tile"""
    xt, xs = G.sphere(700, seed=1) + 3.0, G.cylinder(2900, seed=2)
    t, s = H.Cluster().build(700, xt), H.Cluster().build(2900, xs)
    hm = H.HMatrix(t, s, 1e-6, 10.0).build(H.INV_R_EPS, xt, xs)
    OH = port.hmatrix(port.cluster(xt), port.cluster(xs), xt, xs, H.INV_R_EPS, 1e-6, 10.0)
    x = G.rhs(2900, mu, seed=3)
    y = hm.mvprod_global_to_global(x, mu)
    assert rel(y, OH.mvprod(x, mu)) < ORACLE_TOL
    v = G.rhs(700, mu, seed=4)
    yt = hm.mvprod_transp_global_to_global(v, mu)
    a = np.sum(yt.reshape(mu, -1) * x.reshape(mu, -1), 1)
    b = np.sum(v.reshape(mu, -1) * y.reshape(mu, -1), 1)
    assert np.max(np.abs(a - b)) < 1e-11 * np.max(np.abs(b))


@pytest.mark.parametrize("mu", [1, 3, 8])
def test_values_that_are_not_finite_reach_the_output(mu):
    """an infinity or a NaN in one right-hand side makes its whole output not
    finite and leaves the others as they are"""
    n = 2000
    pts = G.sphere(n, seed=7)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts)
    x = G.rhs(n, mu, seed=8).reshape(mu, n)
    y = hm.mvprod_global_to_global(x.reshape(-1), mu).reshape(mu, n)
    for bad in (np.nan, np.inf, -np.inf):
        xb = x.copy()
        xb[mu - 1, 5] = bad
        yb = hm.mvprod_global_to_global(xb.reshape(-1), mu).reshape(mu, n)
        assert not np.any(np.isfinite(yb[mu - 1]))
        assert np.array_equal(yb[:mu - 1], y[:mu - 1])


def test_choices_of_the_caller_leave_the_panels_and_autotune_returns():
    n = 4000
    pts = G.sphere(n, seed=9)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts)
    x = G.rhs(n, 2, seed=10)
    y = hm.mvprod_global_to_global(x, 2)
    nbytes = hm.get_presplit()[1]
    for choose in (lambda: hm.set_fp64_split(0, 350), lambda: hm.set_phase1_mode("tiles"), lambda: hm.set_phase2_mode("warp"), lambda: hm.set_presplit(False)):
        choose()
        assert rel(hm.mvprod_global_to_global(x, 2), y) < PIPE_TOL
    hm.set_presplit(True)
    assert hm.autotune(2, 2) > 0
    assert hm.get_presplit()[1] == nbytes
    assert np.array_equal(hm.mvprod_global_to_global(x, 2), y)
    hm.set_precision("mixed")  # the reduced-precision products release the panels
    assert hm.get_presplit()[1] < nbytes
    hm.set_precision("fp64")
    assert hm.get_presplit()[1] == nbytes
    assert np.array_equal(hm.mvprod_global_to_global(x, 2), y)


# 1500: four warps to a panel; 12000: a warp each
@pytest.mark.parametrize("n", [1500, 12000])
def test_a_wait_that_runs_out_is_reported(n):
    """a panel whose first copy never comes: the status reports it, a
    host-pointer product fails, and the next product is the one before"""
    pts = G.sphere(n, seed=11)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts)
    x = G.rhs(n, 1, seed=12)
    y = hm.mvprod_global_to_global(x)
    try:
        H._check(H.lib.htgpu_debug_set_waits(0, 2000000, 0))
        with pytest.raises(RuntimeError, match="device wait of the product ran out"):
            hm.mvprod_global_to_global(x)
        assert hm.device_status() in (2, 3)
    finally:
        H._check(H.lib.htgpu_debug_set_waits(0, 4000000000, -1))
    hm.reset_status()
    assert np.array_equal(hm.mvprod_global_to_global(x), y)
    assert hm.device_status() == 0


# inputs of 3 072 entries are gathered by one CTA with their exponent, of
# 16 384 have the exponent from one CTA
@pytest.mark.parametrize("n,mu", [(3072, 1), (3073, 1), (1536, 2), (1537, 2), (1024, 3), (384, 8), (385, 8), (341, 9), (16384, 1), (16385, 1)])
def test_small_inputs(n, mu):
    pts = G.sphere(n, seed=n)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts)
    x = G.rhs(n, mu, seed=mu) * 1e30
    x[:n] *= 2.0**-40  # the largest entries lie behind the first right-hand side
    if mu == 1:
        x[n - 1] = 3e33
    y = np.asarray(hm.mvprod_global_to_global(x, mu)).reshape(mu, n)
    hm.set_fp64_split(1000, 1000)
    r = np.asarray(hm.mvprod_global_to_global(x, mu)).reshape(mu, n)
    assert rel(y, r) < PIPE_TOL
    assert hm.device_status() == 0
