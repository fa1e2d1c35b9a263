"""The GPU refit's climb (four lanes a node, the last inner child done takes its parent) at small trees:
one node, and trees of a few levels and many, refit twice, give the words of the host
refit and packing bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("n", [9, 17, 33, 70, 513, 20_011])
def test_refit_equals_the_host(engine, layout, n):
    import torch
    mesh = S.clusters(n, stream=S.Stream(31 + n))
    blas = A.Blas(mesh.positions, mesh.indices)
    inst = S.identity_instances(1)
    scene = engine.upload(layout, A.pack_scene(layout, [blas], inst))
    idx = torch.from_numpy(mesh.indices.view(np.int32)).cuda() if layout == A.LAYOUT_REFLECTION else None
    rng = np.random.default_rng(n)
    try:
        for _ in range(2):
            new = (mesh.positions * rng.uniform(0.5, 1.5) + rng.normal(0, 0.3, mesh.positions.shape)).astype(np.float32)
            new[::7, 1] = -0.0
            blas.refit(new)
            want = A.pack_scene(layout, [blas], inst)
            scene.refit(0, torch.from_numpy(new).cuda(), idx)
            torch.cuda.synchronize()
            base = int(want[16 + 18]) if layout == A.LAYOUT_GI else int(want[8 + 18]) & ~3
            got = scene.words()
            assert np.array_equal(got[base:], want[base:])
    finally:
        scene.release()
