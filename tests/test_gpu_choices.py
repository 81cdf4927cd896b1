"""Choices of the product's kernels: a call that sets what is set already makes
none and leaves a handle on the panels and streams it runs on; one that changes
something brings the kernels it names, whose products agree with them, and whose
waits are bounded.  No counterpart in the reference (its products run on BLAS).

Tolerance: two FP64-grade products of the same sums, below 4e-13 (both factors
and the input split to 2^-48, sums of random sign); the reduced-precision ones
take the same FP32 sums in the same order."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu

TOL = 4e-13


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def matrix(n, policy="fp64"):
    pts = G.ellipsoid(n, (1.0, 0.7, 1.3), seed=n)
    t = H.Cluster().build(n, pts)
    return H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts).set_precision(policy, 1.0)


def streams(hm):
    return tuple(int(hm.get_infos()[k]) for k in ("GPU_paired_panels", "GPU_reduced_streams"))


@pytest.mark.parametrize("policy", ["fp64", "mixed"])
def test_setting_what_is_set(policy):
    n = 3000
    hm = matrix(n, policy)
    before = streams(hm)
    assert before[policy == "mixed"] > 0
    x = G.rhs(n, 3, seed=1)
    y = hm.mvprod_global_to_global(x, 3)
    for call in (lambda: hm.set_presplit(True), lambda: hm.set_phase1_mode("stream"), lambda: hm.set_phase2_mode("producer"), lambda: hm.set_phase2_dense_split(False)):
        call()
        assert streams(hm) == before
        assert np.array_equal(hm.mvprod_global_to_global(x, 3), y)
    with pytest.raises(ValueError):
        hm.set_phase1_mode(3)
    with pytest.raises(ValueError):
        hm.set_phase2_mode(2)
    hm.set_precision("fp64")
    assert streams(hm)[0] > 0 and streams(hm)[1] == 0


@pytest.mark.parametrize("n", [31, 513, 3000])
@pytest.mark.parametrize("policy", ["fp64", "fp32", "mixed", "bf16"])
def test_either_phase2_mode_against_the_streams(n, policy):
    hm = matrix(n, policy)
    mus = (1, 2, 3, 5, 8, 9, 14)
    xs = {mu: G.rhs(n, mu, seed=mu) for mu in mus}
    ys = {mu: hm.mvprod_global_to_global(xs[mu], mu) for mu in mus}
    for mode in ("warp", "producer"):
        hm.set_phase2_mode(mode)
        assert streams(hm) == (0, 0)
        for mu in mus:
            assert rel(ys[mu], hm.mvprod_global_to_global(xs[mu], mu)) < TOL, (mu, mode)
    assert hm.device_status() == 0


@pytest.mark.parametrize("layout", ["real", "native"])
def test_complex_either_phase2_mode(layout):
    n = 3000
    pts = G.cube_surface(n, seed=5)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-5, 3.0, dtype=np.complex128, complex_layout=layout).build(H.HELMHOLTZ, pts, kernel_param=20.0).set_precision("mixed", 1.0)
    ys = {mu: hm.mvprod_global_to_global(G.rhs(n, mu, seed=mu, dtype=np.complex128), mu) for mu in (1, 2, 3)}
    for mode in ("warp", "producer"):
        hm.set_phase2_mode(mode)
        for mu, y in ys.items():
            assert rel(y, hm.mvprod_global_to_global(G.rhs(n, mu, seed=mu, dtype=np.complex128), mu)) < TOL, (mu, mode)


def test_waits_of_the_producer_kernel():
    """the producer-fed phase 2, chosen in earnest, with a chunk left out"""
    n = 6000
    hm = matrix(n)
    hm.set_phase2_mode("warp")
    hm.set_phase2_mode("producer")
    assert streams(hm) == (0, 0)
    x = G.rhs(n, 1, seed=32)
    ref = hm.mvprod_global_to_global(x)
    try:
        H._check(H.lib.htgpu_debug_set_waits(0, 2000000, 0))
        with pytest.raises(RuntimeError, match="device wait of the product ran out"):
            hm.mvprod_global_to_global(x)
        assert hm.device_status() in (2, 3)
    finally:
        H._check(H.lib.htgpu_debug_set_waits(0, 4000000000, -1))
    hm.reset_status()
    assert np.array_equal(hm.mvprod_global_to_global(x), ref)
    assert hm.device_status() == 0


@pytest.mark.parametrize("policy", ["fp32", "mixed"])
def test_autotune_of_many_right_hand_sides(policy):
    """leaves of up to 300 points: most of the work in dense blocks, which the
    digit planes take at a fifth of the streams' time where they come first;
    products with fewer right-hand sides stay on the streams.  Tolerance: FP32
    sums of up to 256 terms either way, 256 x 2^-24 at most and far less at
    random: below epsilon"""
    n, mu = 12000, 64
    pts = G.sphere(n, seed=12)
    c = H.Cluster()
    c.set_minclustersize(300)
    t = c.build(n, pts)
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts).set_precision(policy, 1.0)
    x, x3 = G.rhs(n, mu, seed=13), G.rhs(n, 3, seed=14)
    y, y3 = hm.mvprod_global_to_global(x, mu), hm.mvprod_global_to_global(x3, 3)
    before = streams(hm)
    for start in (False, True):
        hm.set_digit_planes(start)
        assert hm.autotune(mu, 3) > 0
        assert hm.get_digit_planes()[0] and hm.get_phase2_dense_split()
        assert streams(hm) == before
        assert rel(hm.mvprod_global_to_global(x, mu), y) < 1e-6
        assert np.array_equal(hm.mvprod_global_to_global(x3, 3), y3)
    assert hm.device_status() == 0
