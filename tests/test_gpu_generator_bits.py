"""Generator entries on the device, whose square roots and reciprocals are
taken in integer arithmetic, bit for bit against numpy's IEEE operations:
random points, lattices (exact roots, powers of two) and scales at which the
squares are subnormal, zero or infinite (there the FP64 operations run)."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 3e-5, 7e8, 1e-150, 1e-158, 1e-170, 1e120, 1e160])
@pytest.mark.parametrize("shape", ["sphere", "lattice"])
@pytest.mark.parametrize("kernel", [0, 1])
def test_dense_entries_match_ieee(kernel, shape, scale):
    n = 1331
    if shape == "sphere":
        pts = G.sphere(n, seed=3)
    else:
        pts = np.stack(np.meshgrid(*[np.arange(11.0)] * 3), -1).reshape(-1, 3) * 0.25
    t = H.Cluster().build(n, pts)  # the tree of the points at their own scale
    pts = pts * scale
    hm = H.HMatrix(t, t, 1e-6, 1e-9).build(kernel, pts)
    lr, dn, uv, dd = hm.get_factors()
    assert lr.shape[0] == 0
    x = pts[t.get_perm()]
    off = 0
    with np.errstate(all="ignore"):
        for oi, oj, m, k in dn:
            d = x[oi:oi + m, None, :] - x[None, oj:oj + k, :]
            r = np.sqrt(d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2])
            want = 1.0 / (1e-5 + r) if kernel == 0 else np.where(r == 0.0, 0.0, 1.0 / (4.0 * np.pi * r))
            got = dd[off:off + m * k].reshape(k, m).T
            off += m * k
            assert np.array_equal(np.ascontiguousarray(got).view(np.int64), np.ascontiguousarray(want).view(np.int64))
