"""A NaN in the input of a reduced-precision product on the warp-fed streams
(red.cu) reaches the rows whose leaves read it and no others: htool's products
(types/hmatrix.hpp:1074-1182) multiply a leaf with its own columns alone."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def product(hm, x):
    y = np.asarray(hm.mvprod_global_to_global(x.reshape(-1), x.shape[0])).reshape(x.shape[0], -1)
    assert hm.device_status() == 0
    return y


@pytest.mark.parametrize("mu", [1, 2, 3, 5, 8])
def test_forest_members_stay_apart(mu):
    sizes = [9000, 11000]
    sets = [G.ellipsoid(m, (1.0, 0.7, 1.2), seed=m) for m in sizes]
    t = H.Cluster.forest([H.Cluster().build(len(p), p) for p in sets])
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, t.points).set_precision("mixed", 1.0)
    assert int(hm.get_infos()["GPU_reduced_streams"]) > 0
    x = G.rhs(sum(sizes), mu, seed=1).reshape(mu, -1)
    x[:, sizes[0] - 1] = 64.0  # the largest entry, which scales the input, is the other member's
    y = product(hm, x)
    x[:, sizes[0]:] = np.nan
    yn = product(hm, x)
    assert np.all(np.isnan(yn[:, sizes[0]:]))
    assert np.array_equal(yn[:, :sizes[0]], y[:, :sizes[0]])


# h rows to a row chunk: 32 / h of its columns side by side, so that from one
# column to 64 a chunk has every number of padded columns
@pytest.mark.parametrize("policy", ["fp32", "bf16"])
@pytest.mark.parametrize("h", [1, 3, 4, 11, 16, 32])
def test_rows_of_clean_columns(policy, h):
    """row chunks of one low-rank leaf each, of 1 to 70 columns, reading either
    the clean or the NaN half of the input; far more of them than warps, in any
    order, so every warp takes clean ones after others"""
    n, k = 400000, min(40000, 400000 // h)
    rng = np.random.default_rng(h)
    t = H.Cluster().build(n, rng.random((n, 3)))
    rank = rng.integers(1, 9, k)
    rank[rng.random(k) < 0.1] = 70
    dirty = rng.random(k) < 0.5
    lr = np.zeros((k, 5), np.int32)
    lr[:, 0] = h * np.arange(k)
    lr[:, 1] = np.where(dirty, n // 2 + 8, 8)  # columns of the NaN or of the clean half
    lr[:, 2], lr[:, 3], lr[:, 4] = h, 4, rank
    uv = rng.uniform(0.5, 1.5, int((rank * (h + 4)).sum()))
    hm = H.HMatrix(t, t, 1e-6, 10.0).set_leaves(lr, uv, np.empty((0, 4), np.int32), np.empty(0)).set_precision(policy, 1.0)
    assert int(hm.get_infos()["GPU_reduced_streams"]) > 0
    perm = t.get_perm()
    clean = np.zeros(n, bool)
    for j in range(h):
        clean[h * np.flatnonzero(~dirty) + j] = True
    rows = np.zeros(n, bool)
    rows[:h * k] = True
    for mu in (1, 2, 3, 6, 8):
        xc = rng.uniform(1.0, 2.0, (mu, n))
        x = np.empty_like(xc)
        x[:, perm] = xc
        y = product(hm, x)[:, perm]
        xc[:, n // 2:] = np.nan
        x[:, perm] = xc
        yn = product(hm, x)[:, perm]
        assert np.array_equal(yn[:, clean], y[:, clean]), mu
        assert np.all(np.isnan(yn[:, rows & ~clean])), mu
