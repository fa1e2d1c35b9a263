"""The device build's kept workspaces: bounded, given back by rt_ctx_trim and when a server is made or given a
scene, and made again by the next build."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

pytestmark = pytest.mark.gpu

KEEP = 64 << 20


def test_build_workspaces_are_given_back():
    import torch
    engine = A.Engine(0)
    mesh = S.clusters(60_000, stream=S.Stream(2))
    words = A.pack_scene(A.LAYOUT_REFLECTION, [A.Blas(mesh.positions, mesh.indices)], S.identity_instances(1))
    want = A.Blas(mesh.positions, mesh.indices).nodes()
    build = lambda: A.Blas.build_device(engine, mesh.positions, mesh.indices).nodes()  # noqa: E731
    assert engine.trim() == 0
    assert np.array_equal(build(), want)
    before = torch.cuda.mem_get_info()[0]
    freed = engine.trim()
    assert 0 < freed <= 2 * KEEP
    assert torch.cuda.mem_get_info()[0] - before >= freed // 2  # the driver frees whole pages
    assert engine.trim() == 0
    assert np.array_equal(build(), want)
    server = A.Server(engine, 1 << 30, launch_rays=1 << 12, slots=1, kernel="fast")
    assert engine.trim() == 0
    assert np.array_equal(build(), want)
    server.add_scene(A.LAYOUT_REFLECTION, words)
    assert engine.trim() == 0
    server.close()
    engine.close()
