"""Moves over a top level whose nodes lie past the packer's reserve (words that the upload admits): the
device refits them as the host does, bit for bit, and a rebuild afterwards uses the reserve."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from .test_gpu_move_sizes import _instances

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("far", [1, 5])
def test_far_nodes_are_refit(engine, layout, far):
    meshes = [S.clusters(k, stream=S.Stream(k), half=2.0) for k in (3, 40)]
    blas = [A.Blas(m.positions, m.indices) for m in meshes]
    boxes = A.object_boxes(layout, blas)
    host = A.pack_scene(layout, blas, _instances(2, 1), tlas_mode=0)
    base = (len(host) + 3) & ~3
    host = np.concatenate([host, np.zeros(base - len(host) + 32 * (far + 1), np.uint32)])
    node = host[base:].reshape(-1, 32)
    node[:, 24:28] = 0xFFFFFFFF
    node[0, 25] = far  # the root's only child, past the one node that two instances reserve
    node[far, 24:26] = 0x80000000, 0x80000001
    host[1:4] = base, 0, 0
    scene = engine.upload(layout, host)
    try:
        for k in range(3):
            if k == 2:
                host = host.copy()
                host[3] = 64
                scene.update_records(host[:8])
            new = _instances(2, 10 + k)
            host = A.move_instances_host(layout, host, new, boxes)
            scene.move_instances(new, boxes)
            got = scene.words()
            assert np.array_equal(got, host), f"move {k}: {int((got != host).sum())} words differ"
            assert host[3] == (1, 2, 0)[k]
    finally:
        scene.release()
