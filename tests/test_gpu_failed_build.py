"""A build whose host generator fails: the training samples of the rank
predictor hold the blocks that partialACA decided and none besides."""
import numpy as np
import pytest

import htool_gb300 as H
from htool_gb300 import geometry as G

pytestmark = pytest.mark.gpu


def test_samples_after_a_generator_that_fails():
    n = 1500
    pts = G.sphere(n, seed=1)
    t = H.Cluster().build(n, pts)

    class Fails(H.VirtualGenerator):
        def copy_submatrix(self, rows, cols, out):
            raise RuntimeError("no entries")

    hm = H.HMatrix(t, t, 1e-6, 10.0)
    with pytest.raises(RuntimeError, match="no entries"):
        hm.build_generator(Fails(n, n), pts, pts)
    X, y = hm.aca_samples()
    assert X.shape == (0, 10) and y.shape == (0,)
    hm.build_generator(lambda r, c: 1.0 / (1e-5 + np.linalg.norm(pts[r][:, None] - pts[c][None], axis=2)), pts, pts)
    X, y = hm.aca_samples()
    assert len(y) > 0 and np.all(y > 0)
