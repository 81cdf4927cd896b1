"""Reduced-precision products off the tensor cores on the warp-fed streams
(red.cu) against the chunk and tile kernels that a choice of phase-2 mode keeps.

Both take the same FP32 sums in the same order (every FMA rounds once), so
they differ only in how those sums and the dense FP64 blocks are added up in
double-float arithmetic: by less than the 4e-13 of two FP64 products."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu

TOL = 4e-13


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("n", [31, 513, 3000])
@pytest.mark.parametrize("policy", ["fp32", "mixed", "bf16"])
def test_streams_match_the_chunk_kernels(n, policy):
    pts = G.ellipsoid(n, (1.0, 0.7, 1.3), seed=n)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-6, 10.0).build(H.LAPLACE, pts).set_precision(policy, 1.0)
    mus = (1, 2, 3, 5, 8, 9, 14)
    xs = {mu: G.rhs(n, mu, seed=mu) for mu in mus}
    ys = {mu: hm.mvprod_global_to_global(xs[mu], mu) for mu in mus}
    assert all(np.array_equal(ys[mu], hm.mvprod_global_to_global(xs[mu], mu)) for mu in mus)
    hm.set_phase2_mode("producer")
    for mu in mus:
        assert rel(ys[mu], hm.mvprod_global_to_global(xs[mu], mu)) < TOL, mu
    assert hm.autotune(3, 2) > 0  # back on the streams
    assert np.array_equal(ys[3], hm.mvprod_global_to_global(xs[3], 3))
    assert hm.device_status() == 0


@pytest.mark.parametrize("layout", ["real", "native"])
def test_complex_streams_match_the_chunk_kernels(layout):
    n = 3000
    pts = G.cube_surface(n, seed=5)
    t = H.Cluster().build(n, pts)
    hm = H.HMatrix(t, t, 1e-5, 3.0, dtype=np.complex128, complex_layout=layout).build(H.HELMHOLTZ, pts, kernel_param=20.0).set_precision("mixed", 1.0)
    ys = {mu: hm.mvprod_global_to_global(G.rhs(n, mu, seed=mu, dtype=np.complex128), mu) for mu in (1, 2, 3)}
    hm.set_phase2_mode("producer")
    for mu, y in ys.items():
        assert rel(y, hm.mvprod_global_to_global(G.rhs(n, mu, seed=mu, dtype=np.complex128), mu)) < TOL, mu


def test_rows_without_dense_leaves_and_rectangles():
    """targets far from the sources: no dense leaf, every row from reduced columns alone"""
    xt, xs = G.sphere(900, seed=1) + 4.0, G.sphere(2100, seed=2)
    t, s = H.Cluster().build(900, xt), H.Cluster().build(2100, xs)
    hm = H.HMatrix(t, s, 1e-6, 10.0).build(H.LAPLACE, xt, xs).set_precision("mixed", 1.0)
    assert hm.get_ndmat() == 0
    x = G.rhs(2100, 4, seed=3)
    y = hm.mvprod_global_to_global(x, 4)
    hm.set_phase2_mode("warp")
    assert rel(y, hm.mvprod_global_to_global(x, 4)) < TOL


@pytest.mark.parametrize("mu", [2, 8])
def test_rows_of_more_than_a_window_of_chunks(mu):
    """row chunks of more than 32 chunks: a second window of descriptors"""
    n = 3000
    rng = np.random.default_rng(7)
    pts = G.sphere(n, seed=4)
    t = H.Cluster().build(n, pts)
    lr = np.array([[0, j, 40, 50, 40] for j in range(0, n, 50)] + [[40, 0, n - 40, n, 3]], np.int32)  # offsets, sizes, rank
    uv = rng.standard_normal(int((lr[:, 4].astype(np.int64) * (lr[:, 2] + lr[:, 3])).sum()))
    assert 60 * 40 > 33 * 64  # columns of the first 40 rows, at most 64 a chunk
    hm = H.HMatrix(t, t, 1e-6, 10.0).set_leaves(lr, uv, np.empty((0, 4), np.int32), np.empty(0)).set_precision("mixed", 1.0)
    x = G.rhs(n, mu, seed=3)
    y = hm.mvprod_global_to_global(x, mu)
    hm.set_phase2_mode("warp")
    assert rel(y, hm.mvprod_global_to_global(x, mu)) < TOL
    assert hm.device_status() == 0


@pytest.mark.parametrize("policy", ["fp32", "mixed", "bf16"])
def test_narrow_tiles_exact(policy):
    """low-rank leaves of 1 to 66 columns: tiles whose columns share a warp.
    Factors of +-1 and inputs of small integers make every sum exact in FP32, in
    any order and storage"""
    n = 4096
    rng = np.random.default_rng(3)
    t = H.Cluster().build(n, G.sphere(n, seed=8))
    sizes = [(j, r) for j in (1, 3, 4, 5, 12, 16, 17, 24, 31, 32, 33, 48, 63, 64, 65, 66) for r in (1, 4, 9, 33)]
    lr = np.array([[8 * k, (67 * k) % 4000, 8, j, r] for k, (j, r) in enumerate(sizes)], np.int32)
    sign = lambda *s: rng.choice([-1.0, 1.0], s)
    uvs = [(sign(8, r), sign(r, j)) for j, r in sizes]
    uv = np.concatenate([np.concatenate([u.ravel(order="F"), v.ravel(order="F")]) for u, v in uvs])
    hm = H.HMatrix(t, t, 1e-6, 10.0).set_leaves(lr, uv, np.empty((0, 4), np.int32), np.empty(0)).set_precision(policy, 1.0)
    perm = t.get_perm()
    for mu in (1, 2):
        x = rng.integers(-8, 9, (mu, n)).astype(np.float64)
        want = np.zeros((mu, n))
        for (oi, oj, m, j, r), (u, v) in zip(lr, uvs):
            want[:, perm[oi:oi + m]] += (u @ (v @ x[:, perm[oj:oj + j]].T)).T
        y = np.asarray(hm.mvprod_global_to_global(x.ravel(), mu)).reshape(mu, n)
        assert np.array_equal(y, want), mu
