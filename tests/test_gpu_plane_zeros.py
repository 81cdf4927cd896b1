"""Zeros among the right-hand sides of products on the digit planes (oz.cu): a
zero has no digits, whatever the exponent bound of the panel it is cut for.
htool's product of a zero input is exactly zero (mvprod_global_to_global,
types/hmatrix.hpp:1074-1182 sums products with it), and a power of two on an
input is that power on its output, bit for bit, as every right-hand side is cut
relative to its own exponents."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def product(hm, x):
    y = np.asarray(hm.mvprod_global_to_global(x.reshape(-1), x.shape[0])).reshape(x.shape[0], -1)
    assert hm.device_status() == 0
    return y


# FP64 storage: both phases on the planes; mixed: phase 1 and the dense blocks,
# which are added onto the low-rank part
@pytest.mark.parametrize("storage,eps", [("fp64", 1e-6), ("mixed", 1e-6), ("mixed", 1e-4)])
@pytest.mark.parametrize("mu", [8, 64])
def test_zero_columns(storage, eps, mu):
    n = 3000
    pts = G.sphere(n, seed=1)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, eps, 10.0).build(H.LAPLACE, pts)
    hm.set_precision(storage, 1.0)
    hm.set_digit_planes(True)
    x = G.rhs(n, mu, seed=2).reshape(mu, n)
    y = product(hm, x)
    xz = x.copy()
    xz[3] = 0.0
    xz[mu - 1] = -0.0
    yz = product(hm, xz)
    assert not np.any(yz[3]) and not np.any(yz[mu - 1])
    keep = [c for c in range(mu) if c not in (3, mu - 1)]
    assert np.array_equal(yz[keep], y[keep])
    assert not np.any(product(hm, np.zeros((mu, n))))


@pytest.mark.parametrize("mu", [8, 64])
def test_zero_forest_member(mu):
    sizes = [1500, 2100]
    sets = [G.ellipsoid(m, (1.0, 0.7, 1.2), seed=m) for m in sizes]
    t = H.Cluster.forest([H.Cluster().build(len(p), p) for p in sets])
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, t.points)
    hm.set_digit_planes(True)
    x = G.rhs(sum(sizes), mu, seed=3).reshape(mu, -1)
    assert np.all(product(hm, x) != 0.0)
    x[:, sizes[0]:] = 0.0
    y = product(hm, x)
    assert not np.any(y[:, sizes[0]:])
    assert np.all(y[:, :sizes[0]] != 0.0)


# 2^-1000: the panel's exponent bounds lie below 54, the width of the digits
@pytest.mark.parametrize("power", [-1000, -40, 900])
def test_scaled_sparse_inputs(power):
    """one dense leaf, whose coefficients are input rows, most of them zero (the
    planes are built where there are low-rank leaves: one of zero factors)"""
    n, mu = 600, 8
    t = H.Cluster().build(n, G.sphere(n, seed=4))
    rng = np.random.default_rng(5)
    D = rng.uniform(0.5, 1.5, (n, n))
    lr = np.array([[0, 0, n, n, 1]], np.int32)
    hm = H.HMatrix(t, t, 1e-6, 10.0).set_leaves(lr, np.zeros(2 * n), np.array([[0, 0, n, n]], np.int32), D.ravel(order="F"))
    hm.set_digit_planes(True)
    assert hm.get_digit_planes()[1] > 0
    x = rng.uniform(1.0, 2.0, (mu, n)) * (rng.random((mu, n)) < 0.1)
    y = product(hm, x)
    ys = product(hm, np.ldexp(x, power))
    assert np.array_equal(np.ldexp(ys, -power), y)


def test_large_entries():
    """entries far beyond single precision and right-hand sides of zeros and of a few rows"""
    n, mu = 500, 9
    t = H.Cluster().build(n, G.sphere(n, seed=6))
    rng = np.random.default_rng(7)
    D = rng.uniform(-1.0, 1.0, (n, n)) * 1e200
    lr = np.array([[0, 0, n, n, 1]], np.int32)
    hm = H.HMatrix(t, t, 1e-6, 10.0).set_leaves(lr, np.zeros(2 * n), np.array([[0, 0, n, n]], np.int32), D.ravel(order="F"))
    hm.set_digit_planes(True)
    perm = t.get_perm()
    x = np.zeros((mu, n))
    x[1, perm[7]] = 2.0
    x[8, perm[:3]] = (0.5, 0.25, -1.0)
    y = product(hm, x)[:, perm]
    assert not np.any(y[[0, 2, 3, 4, 5, 6, 7]])
    # the planes hold 54 bits of an entry relative to its row's largest
    assert np.max(np.abs(y[1] - 2.0 * D[:, 7])) <= 2.0 ** -50 * 1e200
    assert np.max(np.abs(y[8] - D[:, :3] @ (0.5, 0.25, -1.0))) <= 2.0 ** -50 * 1e200
