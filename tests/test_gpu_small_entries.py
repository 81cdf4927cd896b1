"""FP64-grade products of entries far below 1: the factors are held as float
pairs, whose lower halves run into the subnormal floats from about 2^-101 on,
against the product in extended precision.  No counterpart in the reference
(its products run on BLAS).

Tolerance: as for entries near 1 (4e-13: splits to 2^-48, sums of random sign),
and below about 2^-101 what the subnormal floats keep: entries, products and
sums to 2^-150 each, four of these for each of K terms of random sign against a
sum of size sqrt(K) times the entries' scale."""
import numpy as np
import pytest

import htool_gb300 as H

pytestmark = pytest.mark.gpu


def tol(K, scale):
    return 4e-13 + 4 * np.sqrt(K) * 2.0**-150 / scale


def leaf(scale, m, seed):
    """one dense leaf of m x m entries of the scale, a hundredth of them 2^-20 of that"""
    rng = np.random.default_rng(seed)
    D = scale * rng.standard_normal((m, m))
    D[rng.random((m, m)) < 0.01] *= 2.0**-20
    t = H.Cluster().build(m, rng.random((m, 3)))
    hm = H.HMatrix(t, t, 1e-6, 10.0).set_leaves(np.zeros((0, 5), np.int32), np.zeros(1), np.array([[0, 0, m, m]], np.int32), D.T.reshape(-1).copy())
    return hm, np.asarray(t.get_perm()), D, rng


@pytest.mark.parametrize("policy", ["fp64", "mixed"])
@pytest.mark.parametrize("e", [0, -70, -83, -95, -103, -110])
def test_scales_of_a_dense_leaf(e, policy):
    m, scale = 150, 2.0**e
    hm, perm, D, rng = leaf(scale, m, 100 - e)
    hm.set_precision(policy, 1.0)
    for mu in (1, 2, 3, 8):
        x = rng.standard_normal((mu, m))
        y = hm.mvprod_global_to_global(x.reshape(-1).copy(), mu).reshape(mu, m)
        ref = (D.astype(np.longdouble) @ x[:, perm].T.astype(np.longdouble)).T
        for c in range(mu):
            d = (y[c, perm] - ref[c]) / scale
            assert np.linalg.norm(d.astype(float)) < tol(m, scale) * np.linalg.norm((ref[c] / scale).astype(float)), (mu, c)


@pytest.mark.parametrize("mu", [1, 2, 5])
def test_small_entries_that_a_large_input_meets(mu):
    """columns 2^-110 of the others in size, against inputs 2^27 of the others':
    what they give is 2^-83 of the sum but all of the sum where those are zero"""
    m = 150
    hm, perm, D, rng = leaf(1.0, m, 7)
    D[:, :40] *= 2.0**-110
    D[:30, 40:] = 0
    hm.set_leaves(np.zeros((0, 5), np.int32), np.zeros(1), np.array([[0, 0, m, m]], np.int32), D.T.reshape(-1).copy())
    x = rng.standard_normal((mu, m))
    x[:, perm[:40]] *= 2.0**27
    y = hm.mvprod_global_to_global(x.reshape(-1).copy(), mu).reshape(mu, m)
    ref = (D.astype(np.longdouble) @ x[:, perm].T.astype(np.longdouble)).T
    # the input is brought to 1: the small columns' products stay at 2^-110
    t = tol(40, 2.0**-110)
    for c in range(mu):
        for rows, lim in ((slice(0, 30), t), (slice(30, m), 4e-13)):
            a, b = y[c, perm][rows], ref[c, rows]
            s = np.abs(b).max()
            assert np.linalg.norm(((a - b) / s).astype(float)) < lim * np.linalg.norm((b / s).astype(float)), (c, rows)
