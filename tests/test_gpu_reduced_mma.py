"""Phase 2 of reduced-precision products on mma.sync (mixed.cu): right-hand
sides in blocks of 8, 16, 32 or 64, copied 16, 8 or 4 bytes at a time.

A column's sums take the same steps wherever its block puts it, so a product
with many right-hand sides equals products of 8 of its columns bit for bit
(all scaled by the same power of two: every column's largest entry is 1).
Against the product of one right-hand side at a time, on the CUDA cores from
the same stored factors, it differs by FP32 rounding: sums of at most a few
thousand products, 2^-24 each and growing with the square root of their
number, stay below 2e-6."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def rhs(n, mu, seed):
    x = G.rhs(n, mu, seed=seed).reshape(mu, n)
    return np.ascontiguousarray(x / np.abs(x).max(axis=1, keepdims=True)).ravel()


def matrix(n, policy):
    pts = G.ellipsoid(n, (1.0, 0.7, 1.3), seed=n)
    t = H.Cluster().build(n, pts)
    return H.HMatrix(t, t, 1e-5, 10.0).build(H.LAPLACE, pts).set_precision(policy, 1.0)


@pytest.mark.parametrize("n,policy", [(47, "mixed"), (700, "fp32"), (3001, "mixed"), (3001, "bf16"), (12000, "mixed")])
def test_blocks_agree_bitwise(n, policy):
    hm = matrix(n, policy)
    hm.set_tensor_core_mode("mma.sync")
    x = rhs(n, 77, n)
    cols = lambda y, a, b: np.asarray(y).reshape(-1, n)[a:b]
    parts = [cols(hm.mvprod_global_to_global(x[c * n:(c + 8) * n], 8), 0, 8) for c in range(0, 72, 8)]
    want = np.concatenate(parts)
    for mu in (9, 10, 12, 15, 16, 17, 32, 34, 61, 64, 72):
        assert np.array_equal(cols(hm.mvprod_global_to_global(x[:mu * n], mu), 0, mu), want[:mu]), mu
    y = cols(hm.mvprod_global_to_global(x, 77), 0, 77)
    assert np.array_equal(y[:72], want)
    one = np.concatenate([cols(hm.mvprod_global_to_global(x[c * n:(c + 1) * n], 1), 0, 1) for c in (0, 40, 76)])
    assert np.linalg.norm(y[[0, 40, 76]] - one) < 2e-6 * np.linalg.norm(one)
    assert hm.device_status() == 0


def test_sums_that_are_not_finite_reach_the_result():
    """factors whose columns' scales are beyond FP32: infinite or NaN
    coefficients, which the integer split would lose"""
    n = 3001
    pts = G.sphere(n, seed=1)
    t = H.Cluster().build(n, pts)
    lr, dn, uv, dd = H.HMatrix(t, t, 1e-5, 10.0).build(H.LAPLACE, pts).get_factors()
    big = H.HMatrix(t, t, 1e-5, 10.0).set_leaves(lr, uv * 1e30, dn, dd).set_precision("mixed", 1.0)
    big.set_tensor_core_mode("mma.sync")
    y = np.asarray(big.mvprod_global_to_global(rhs(n, 16, 1), 16))
    assert not np.isfinite(y).any()
