"""Record rewrites, moves and refits of one scene from three threads at once: each call works on the scene
between two others, and a rewrite and a move at the end leave the host's words."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from .test_gpu_move_sizes import _instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
def test_threads_change_one_scene(engine, layout):
    import torch
    n = 300
    meshes = [S.clusters(k, stream=S.Stream(k), half=2.0) for k in (40, 700)]
    blas = [A.Blas(m.positions, m.indices) for m in meshes]
    blas[0].refit(meshes[0].positions)
    boxes = A.object_boxes(layout, blas)
    placed = [_instances(n, 1), _instances(n, 2)]
    words = [A.pack_scene(layout, blas, p, tlas_mode=1) for p in placed]
    header, stride = (16, 32) if layout == A.LAYOUT_GI else (8, 24)
    records = words[0][header:header + stride * n].reshape(n, stride)
    leading = int((records[:, 18] & ~np.uint32(3)).min())  # the records and the top level, no mesh word
    scene = engine.upload(layout, words[0])
    positions = torch.from_numpy(meshes[0].positions).cuda()
    idx = torch.from_numpy(meshes[0].indices.view(np.int32)).cuda() if layout == A.LAYOUT_REFLECTION else None
    torch.cuda.synchronize()
    errors = []

    def loop(call):
        try:
            for k in range(40):
                call(k)
        except Exception as e:  # the main thread reports it
            errors.append(e)

    calls = (lambda k: scene.update_records(words[k & 1][:leading]), lambda k: scene.move_instances(placed[k & 1], boxes, 0),
             lambda k: scene.refit(0, positions, idx, 0))
    threads = [threading.Thread(target=loop, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    try:
        assert not errors, errors
        scene.update_records(words[0][:leading])
        scene.move_instances(placed[1], boxes)
        assert np.array_equal(scene.words(), A.move_instances_host(layout, words[0], placed[1], boxes))
    finally:
        scene.release()
