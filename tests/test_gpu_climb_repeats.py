"""The climbs that decide node boxes (a refit's, a top level's) read children that other thread blocks
have just written: repeated over a tree of many levels, with other geometry each time, every word equals
the host's each time."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from .test_gpu_move_sizes import _instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
def test_climbs_repeat(engine, layout):
    import torch
    gi = layout == A.LAYOUT_GI
    meshes = [S.clusters(n, stream=S.Stream(n), half=2.0) for n in (60_000, 3)]
    blas = [A.Blas(m.positions, m.indices) for m in meshes]
    n = 3000
    inst = _instances(n, 1)
    scene = engine.upload(layout, A.pack_scene(layout, blas, inst, tlas_mode=1))
    base = int(scene.words(16 if gi else 8, 32)[18]) & ~(0 if gi else 3)  # mesh 0's words
    idx = None if gi else torch.from_numpy(meshes[0].indices.view(np.int32)).cuda()
    try:
        for k in range(20):
            new = (meshes[0].positions * np.float32(0.9 + 0.02 * k)).astype(np.float32)
            blas[0].refit(new)
            want = A.pack_scene(layout, blas, inst, tlas_mode=0)
            scene.refit(0, torch.from_numpy(new).cuda(), idx)
            assert np.array_equal(scene.words(base), want[base:]), f"refit {k}"
        boxes = A.object_boxes(layout, blas)
        host = scene.words()
        for k in range(20):
            placed = _instances(n, 50 + k)
            host = A.move_instances_host(layout, host, placed, boxes)
            scene.move_instances(placed, boxes)
            assert np.array_equal(scene.words(), host), f"move {k}"
    finally:
        scene.release()
