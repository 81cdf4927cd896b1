"""Products whose result has no double: infinite with its sign, as FP64
arithmetic gives it (the products run on inputs brought to 1, so the way back
must not run over the exponent's end).  No counterpart in the reference (its
products run on BLAS).

Exact: powers of two in and out."""
import numpy as np
import pytest

import htool_gb300 as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("policy", ["fp64", "mixed"])
@pytest.mark.parametrize("mu", [1, 2, 3, 8])
def test_results_past_the_largest_double(mu, policy):
    """rows of one entry: 2^50, 1, -2^50, 2^-50 against inputs of 2^1000, and all
    rows against inputs of 1"""
    m = 64
    rng = np.random.default_rng(11)
    t = H.Cluster().build(m, rng.random((m, 3)))
    perm = np.asarray(t.get_perm())
    d = np.tile([2.0**50, 1.0, -(2.0**50), 2.0**-50], m // 4)
    hm = H.HMatrix(t, t, 1e-6, 10.0).set_leaves(np.zeros((0, 5), np.int32), np.zeros(1), np.array([[0, 0, m, m]], np.int32), np.diag(d).reshape(-1)).set_precision(policy, 1.0)
    for big in (1.0, 2.0**1000):
        x = big * 2.0 ** rng.integers(-3, 4, (mu, m)).astype(np.float64)
        with np.errstate(over="ignore"):
            want = d * x[:, perm]
        assert np.isinf(want).any() == (big > 1)
        y = hm.mvprod_global_to_global(x.reshape(-1).copy(), mu).reshape(mu, m)[:, perm]
        assert np.array_equal(y, want)
