"""The refit of a mesh small enough for one leaf (1 to 8 triangles, no node): its positions or triangles
are rewritten as the host's refit and packing write them, beside a larger mesh."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("n", [1, 8])
def test_a_lone_leaf_is_refit(engine, layout, n):
    import torch
    meshes = [S.clusters(k, stream=S.Stream(6 + k)) for k in (n, 60)]
    blas = [A.Blas(m.positions, m.indices) for m in meshes]
    inst = S.identity_instances(2)
    scene = engine.upload(layout, A.pack_scene(layout, blas, inst))
    first = (16 + 32 * 2) if layout == A.LAYOUT_GI else (8 + 24 * 2)
    try:
        for k in range(2):
            for m in (0, 1):
                new = (meshes[m].positions * np.float32(1.1 + 0.2 * k)).astype(np.float32)
                blas[m].refit(new)
                idx = torch.from_numpy(meshes[m].indices.view(np.int32)).cuda() if layout == A.LAYOUT_REFLECTION else None
                scene.refit(m, torch.from_numpy(new).cuda(), idx)
            want, got = A.pack_scene(layout, blas, inst), scene.words()
            base = int(want[(16 if layout == A.LAYOUT_GI else 8) + 18]) & ~3  # the meshes' words
            assert base >= first and np.array_equal(got[base:], want[base:])
    finally:
        scene.release()
