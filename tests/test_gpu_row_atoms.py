"""The final sums of a product (zsum_kernel, pair_zsum_kernel) take the target
rows in atoms of at most 32 rows, also where one leaf covers many: products of
one low-rank leaf against numpy's (htool's mvprod_global_to_global,
types/hmatrix.hpp:1074-1182, on one block).

Tolerance: as for two FP64 products on different kernels, below 4e-13 (factors
and inputs split to 2^-48, sums of random sign); reduced storage with factors of
+-1 and small integers is exact in FP32, in any order."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu

NO_DENSE = (np.empty((0, 4), np.int32), np.empty(0))


def one_leaf(nr, nc, u, v):
    t, s = H.Cluster().build(nr, G.sphere(nr, seed=1)), H.Cluster().build(nc, G.sphere(nc, seed=2))
    lr = np.array([[0, 0, nr, nc, u.shape[1]]], np.int32)
    uv = np.concatenate([u.ravel(order="F"), v.ravel(order="F")])
    return H.HMatrix(t, s, 1e-6, 10.0).set_leaves(lr, uv, *NO_DENSE), t.get_perm(), s.get_perm()


# 1 and 5 right-hand sides on the panels; 17 on the planes too
@pytest.mark.parametrize("nr", [31, 32, 33, 64, 65, 1000, 40000])
def test_one_leaf(nr):
    nc, r = 300, 3
    rng = np.random.default_rng(nr)
    u, v = rng.standard_normal((nr, r)), rng.standard_normal((r, nc))
    hm, pt, ps = one_leaf(nr, nc, u, v)
    for mu, planes in ((1, False), (5, False), (17, False), (17, True)):
        hm.set_digit_planes(planes)
        x = rng.standard_normal((mu, nc))
        want = np.empty((mu, nr))
        want[:, pt] = (u @ (v @ x[:, ps].T)).T
        y = np.asarray(hm.mvprod_global_to_global(x.ravel(), mu)).reshape(mu, nr)
        assert np.linalg.norm(y - want) < 4e-13 * np.linalg.norm(want), (mu, planes)
    assert hm.device_status() == 0


@pytest.mark.parametrize("eps", [1e-6, 1e-4])
def test_one_leaf_reduced_storage(eps):
    nr, nc, r = 1003, 64, 5
    rng = np.random.default_rng(3)
    u, v = rng.choice([-1.0, 1.0], (nr, r)), rng.choice([-1.0, 1.0], (r, nc))
    t, s = H.Cluster().build(nr, G.sphere(nr, seed=1)), H.Cluster().build(nc, G.sphere(nc, seed=2))
    uv = np.concatenate([u.ravel(order="F"), v.ravel(order="F")])
    hm = H.HMatrix(t, s, eps, 10.0).set_leaves(np.array([[0, 0, nr, nc, r]], np.int32), uv, *NO_DENSE).set_precision("fp32")
    for mu in (1, 3, 8, 11):
        x = rng.integers(-8, 9, (mu, nc)).astype(np.float64)
        want = np.empty((mu, nr))
        want[:, t.get_perm()] = (u @ (v @ x[:, s.get_perm()].T)).T
        assert np.array_equal(np.asarray(hm.mvprod_global_to_global(x.ravel(), mu)).reshape(mu, nr), want), mu


def test_more_than_2_31_outputs():
    """rows times right-hand sides past 32-bit indices, from 16 columns"""
    torch = pytest.importorskip("torch")
    nr, nc, mu = 1100003, 16, 1999
    assert nr * mu > 2**31
    if torch.cuda.mem_get_info()[0] < 100e9:
        pytest.skip("needs 100 GB of device memory")
    rng = np.random.default_rng(4)
    u, v = rng.choice([-1.0, 1.0], (nr, 1)), rng.choice([-1.0, 1.0], (1, nc))
    hm, pt, ps = one_leaf(nr, nc, u, v)
    x = rng.integers(-8, 9, (mu, nc)).astype(np.float64)
    xd = torch.from_numpy(x).cuda()
    y = torch.full((mu, nr), float("nan"), dtype=torch.float64, device="cuda")
    hm.mvprod_ptr(xd.data_ptr(), y.data_ptr(), mu, 0, torch.cuda.current_stream().cuda_stream)
    assert hm.device_status() == 0
    ud = torch.zeros(nr, dtype=torch.float64)
    ud[torch.from_numpy(pt).long()] = torch.from_numpy(u[:, 0])
    a = torch.from_numpy(x[:, ps] @ v[0]).cuda()  # small integers: exact
    ud = ud.cuda()
    for c in range(0, mu, 64):
        assert torch.equal(y[c:c + 64], a[c:c + 64, None] * ud)
