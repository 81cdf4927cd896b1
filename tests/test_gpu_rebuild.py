"""An H-matrix built again: what an earlier build and its storage left behind
takes no part in the new one's products."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("storage", ["fp32", "mixed"])
def test_rebuild_under_reduced_precision(storage):
    """built, stored in reduced precision, built again with another kernel, then a
    choice of the reduced-precision kernels: the products of a new handle"""
    n = 4000
    pts = G.sphere(n, seed=1)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.INV_R_EPS, pts)
    hm.set_precision(storage, 1.0)
    assert int(hm.get_infos()["GPU_reduced_streams"]) > 0
    hm.build(H.LAPLACE, pts)  # back in FP64
    assert int(hm.get_infos()["GPU_reduced_streams"]) == 0
    assert int(hm.get_infos()["GPU_paired_panels"]) > 0
    hm.set_phase2_dense_split(True)
    assert int(hm.get_infos()["GPU_paired_panels"]) > 0
    fresh = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts)
    for mu in (1, 3, 8):
        x = G.rhs(n, mu, seed=mu)
        assert np.array_equal(hm.mvprod_global_to_global(x, mu), fresh.mvprod_global_to_global(x, mu))
    hm.set_phase2_dense_split(False)
    for policy in (storage, "fp64"):
        hm.set_precision(policy, 1.0)
        fresh.set_precision(policy, 1.0)
        for mu in (1, 2, 8):
            x = G.rhs(n, mu, seed=mu)
            assert np.allclose(hm.mvprod_global_to_global(x, mu), fresh.mvprod_global_to_global(x, mu), rtol=0, atol=1e-12 * np.sqrt(n))
    assert hm.device_status() == 0
