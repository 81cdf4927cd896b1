"""Products where device memory is short: the copies of the factors that make
products faster (paired panels, reduced-precision streams, pre-split pairs) are
left out or given up, and the products stay.  The rest of the memory is held by
torch meanwhile.  No counterpart in the reference (host memory).

Tolerance: two FP64-grade products of the same sums, below 4e-13."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu

TOL = 4e-13
MB = 1 << 20


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


class Held:
    """all device memory but `leave` bytes, for the time of a with block"""

    def __init__(self, leave):
        self.leave = leave

    def __enter__(self):
        torch = pytest.importorskip("torch")
        torch.cuda.empty_cache()
        self.blocks = []
        for unit in (16 << 30, 1 << 30, 64 * MB, 4 * MB):
            while torch.cuda.mem_get_info()[0] >= self.leave + unit:
                self.blocks.append(torch.empty(unit, dtype=torch.uint8, device="cuda"))
        return self

    def __exit__(self, *a):
        import torch

        self.blocks.clear()
        torch.cuda.empty_cache()


def matrix(n=40000):
    pts = G.sphere(n, seed=3)
    t = H.Cluster().build(n, pts)
    return H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts)


def panels(hm):
    return int(hm.get_infos()["GPU_paired_panels"])


def test_autotune_without_room_for_the_panels():
    """the sweep over the other kernels stays with them, also past the splits
    that hold no copies and leave more memory free than at its start"""
    hm = matrix()
    n = hm.sizes()[1]
    x = G.rhs(n, 2, seed=1)
    y = hm.mvprod_global_to_global(x, 2)
    nbytes = hm.get_presplit()[1]
    hm.set_fp64_split(0, 350)
    with Held(int(0.9 * nbytes)):
        assert hm.autotune(2, 1) > 0
        assert panels(hm) == 0
        assert rel(hm.mvprod_global_to_global(x, 2), y) < TOL
    assert hm.autotune(2, 1) > 0
    assert panels(hm) > 0
    assert np.array_equal(hm.mvprod_global_to_global(x, 2), y)
    assert hm.device_status() == 0


def test_streams_without_room():
    """one leaf whose reduced columns leave no room for the streams' copy of
    them: the panels of the small dense leaf beside it are not kept either"""
    n, r, m = 1000000, 40, 64
    rng = np.random.default_rng(2)
    t = H.Cluster().build(n, rng.random((n, 3)))
    lr, dn = np.array([[0, 0, n, n, r]], np.int32), np.array([[0, 0, m, m]], np.int32)
    hm = H.HMatrix(t, t, 1e-6, 10.0).set_leaves(lr, rng.choice([-1.0, 1.0], 2 * n * r), dn, rng.choice([-1.0, 1.0], m * m))
    x = rng.integers(-2, 3, n).astype(np.float64)
    y = hm.mvprod_global_to_global(x)
    hm.set_fp64_split(1000, 1000)  # no panels, no pre-split pairs
    reduced, copy = 4 * r * 2 * n, 4 * r * n
    with Held(reduced + 110 * MB):
        hm.set_precision("fp32", 1.0)
        assert 110 * MB * 3 // 4 < copy
        assert int(hm.get_infos()["GPU_reduced_streams"]) == 0
        assert hm.get_presplit()[1] < 1.5 * 8 * m * m
        assert rel(hm.mvprod_global_to_global(x), y) < 1e-6
    hm.set_precision("fp32", 1.0)
    assert int(hm.get_infos()["GPU_reduced_streams"]) > 0
    assert hm.get_presplit()[1] >= copy + 8 * m * m
    assert rel(hm.mvprod_global_to_global(x), y) < 1e-6
    assert hm.device_status() == 0


@pytest.mark.parametrize("eps", [1e-6, 1e-4])
def test_dense_blocks_are_held_once_beside_the_factors(eps):
    """reduced storage below epsilon 1e-5: the streams' panels are the only
    other copy of the dense blocks, until products leave the streams (digit
    planes; a choice of kernels); from 1e-5 on products with 8 or more right-hand
    sides read the pre-split chunks.  The products are the same without them"""
    n, r, m = 3000, 4, 600
    rng = np.random.default_rng(3)
    t = H.Cluster().build(n, rng.random((n, 3)))
    lr, dn = np.array([[m, 0, n - m, n, r]], np.int32), np.array([[0, 0, m, m]], np.int32)
    hm = H.HMatrix(t, t, eps, 10.0).set_leaves(lr, rng.standard_normal((2 * n - m) * r), dn, rng.standard_normal(m * m)).set_precision("fp32", 1.0)
    pairs, columns = 8 * m * m, 4 * r * n
    small = pairs // 2
    chunks = eps >= 1e-5
    assert abs(hm.get_presplit()[1] - (1 + chunks) * pairs - columns) < small
    X = G.rhs(n, 9, seed=4)
    hm.set_digit_planes(True)
    assert abs(hm.get_presplit()[1] - 2 * pairs - columns) < small
    y = hm.mvprod_global_to_global(X, 9)
    hm.set_presplit(False)  # the chunks split in the kernels
    assert hm.get_presplit()[1] == 0
    assert np.array_equal(hm.mvprod_global_to_global(X, 9), y)
    hm.set_presplit(True).set_digit_planes(False)
    hm.autotune(3, 1)
    assert int(hm.get_infos()["GPU_reduced_streams"]) > 0
    y = hm.mvprod_global_to_global(X[:3 * n].copy(), 3)
    hm.set_phase2_mode("warp")
    assert abs(hm.get_presplit()[1] - pairs) < small
    assert rel(hm.mvprod_global_to_global(X[:3 * n].copy(), 3), y) < TOL
    hm.set_precision("fp64")
    assert hm.device_status() == 0


def device_bytes(before):
    """what has been taken since `before` bytes were free"""
    import torch

    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0]


def streams(hm):
    return panels(hm) + int(hm.get_infos()["GPU_reduced_streams"])


@pytest.mark.parametrize("policy", ["fp64", "mixed"])
@pytest.mark.parametrize("what", ["right-hand sides", "planes"])
def test_copies_give_way(policy, what):
    """work buffers and digit planes are allocated after the panels or streams,
    which go where the rest of the memory does not hold them"""
    torch = pytest.importorskip("torch")
    mu = 400 if what == "right-hand sides" else 8
    hm, ref = matrix().set_precision(policy, 1.0), matrix().set_precision(policy, 1.0)
    n = hm.sizes()[1]
    X = G.rhs(n, mu, seed=5)
    call = lambda h: (h.set_digit_planes(True) if what == "planes" else h).mvprod_global_to_global(X, mu)
    copies = ref.get_presplit()[1]
    for h in (hm, ref):
        h.mvprod_global_to_global(X[:n].copy(), 1)
        if what == "planes":
            h.mvprod_global_to_global(X, mu)
    free = torch.cuda.mem_get_info()[0]
    y = call(ref)
    need = device_bytes(free)
    ref.set_digit_planes(False).set_phase2_mode("warp")  # the kernels without the copies hold pre-split pairs
    freed = copies - ref.get_presplit()[1]
    assert freed > 16 * MB and need > freed // 2
    del ref
    assert streams(hm) > 0
    with Held(need - freed // 2):
        z = call(hm)
        assert streams(hm) == 0
        assert rel(z, y) < TOL
        assert rel(call(hm), y) < TOL
    assert hm.device_status() == 0


def test_transposed_twin():
    """the twin of transposed products: the least memory it takes beside a handle
    off the panels is enough beside one on them, with what its panels hold"""
    n = 40000
    x = G.rhs(n, 1, seed=6)

    def works(hm, leave):
        with Held(leave):
            try:
                hm.mvprod_transp_global_to_global(x)
                return True
            except RuntimeError as e:
                assert "out of memory" in str(e)
                return False

    hm, ref = matrix(n), matrix(n)
    copies = ref.get_presplit()[1]
    y = ref.mvprod_transp_global_to_global(x)
    ref.set_phase2_mode("warp")
    freed = copies - ref.get_presplit()[1]
    assert freed > 16 * MB
    del ref
    lo, hi = 0, 5 * copies
    while hi - lo > freed // 8:
        mid = (lo + hi) // 2
        off = matrix(n).set_phase2_mode("warp")
        lo, hi = (lo, mid) if works(off, mid) else (mid, hi)
        del off
    assert works(hm, hi - freed // 2)
    assert streams(hm) == 0
    assert rel(hm.mvprod_transp_global_to_global(x), y) < TOL
    assert hm.device_status() == 0
