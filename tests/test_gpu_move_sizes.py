"""The device move's one-launch top-level refit and its scene bounds, at instance counts around a node,
a warp and a block, over moves in a row, after a record rewrite that changes the top level, and at
the rebuild: the words equal the host move's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

pytestmark = pytest.mark.gpu


def _instances(n, seed):
    s = S.Stream(seed)
    model = np.concatenate([S.quaternion_matrices(s, n) * s.range(0.5, 2.0, n)[:, None, None],
                            s.range(-40.0, 40.0, n, 3)[:, :, None]], axis=2).astype(np.float32)
    model[::9, 1, 3] = 0.0
    return S.Instances(model, S.affine_inverse_rows(model), (np.arange(n) % 2).astype(np.uint32))


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("n", [2, 5, 33, 130, 700])
def test_move_equals_the_host_move(engine, layout, n):
    import torch
    meshes = [S.clusters(k, stream=S.Stream(k), half=2.0) for k in (3, 40)]
    blas = [A.Blas(m.positions, m.indices) for m in meshes]
    boxes = A.object_boxes(layout, blas)
    host = A.pack_scene(layout, blas, _instances(n, 1), tlas_mode=1)
    scene = engine.upload(layout, host)
    try:
        for step in range(5):
            if step == 2:  # other instances under another tree, records and all
                host = A.pack_scene(layout, blas, _instances(n, 99), tlas_mode=1)
                scene.update_records(host)
            if step == 3:  # the refit count at its limit: the next move rebuilds
                host = host.copy()
                host[3] = 64
                scene.update_records(host[:8])
            new = _instances(n, 10 + step)
            host = A.move_instances_host(layout, host, new, boxes)
            scene.move_instances(new, boxes)
            torch.cuda.synchronize()
            dev = scene.words()
            assert np.array_equal(dev, host), f"move {step}: {int((dev != host).sum())} words differ"
    finally:
        scene.release()
