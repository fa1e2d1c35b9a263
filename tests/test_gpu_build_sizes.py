"""The GPU BLAS build around the sizes where its work is cut (a leaf, a warp, one block's range, a chunk
of a larger one), by SAH and by median splits, on general, tied and huge coordinates (costs that are
infinite or NaN): the records equal the host build's word for word."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["general", "tied", "huge"])
@pytest.mark.parametrize("median", [False, True])
@pytest.mark.parametrize("n", [1, 8, 9, 31, 33, 257, 1025, 2047, 2048, 2049, 5000])
def test_device_build_equals_the_host(engine, n, median, kind):
    mesh = S.clusters(n, stream=S.Stream(n + 3))
    pos = mesh.positions
    if kind == "tied":
        pos = (np.round(pos / 4.0) * 4.0).astype(np.float32)
    elif kind == "huge":
        pos = (pos * np.float32(1e30)).astype(np.float32)
        pos[::5, 0] = 3e38
        pos[1::7, 1] = 0.0
    host = A.Blas(pos, mesh.indices, median=median)
    dev = A.Blas.build_device(engine, pos, mesh.indices, median)
    assert dev.info() == host.info()
    assert np.array_equal(dev.bvh_indices(), host.bvh_indices())
    assert np.array_equal(dev.nodes(), host.nodes())
