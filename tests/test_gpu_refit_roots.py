"""A refit covers every node of the BLAS that an instance may enter, not only those below the root of the
instance it was called for: nodes that this root does not reach (its record cut a subtree off, which
another instance enters at its own root), and nodes above it (another instance enters higher up, from
the start or after a rewrite of its record). Their words equal the host refit's, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("case", ["cut", "below", "raised"])
def test_every_root_is_refit(engine, layout, case):
    import torch
    gi = layout == A.LAYOUT_GI
    mesh = S.clusters(5000, stream=S.Stream(12))
    blas = A.Blas(mesh.positions, mesh.indices)
    inst = S.identity_instances(2)
    inst.mesh[:] = 0
    header, stride, root_at = (16, 32, 22) if gi else (8, 24, 20)
    w = A.pack_scene(layout, [blas], inst, tlas_mode=0)
    base, root = int(w[header + 18]) & (~0 if gi else ~3), int(w[header + root_at])
    node = w[base:base + 16 * (root + 1)].reshape(-1, 16)
    slot = next(s for s in range(4) if 0 < node[root, 6 + s] < root)  # an inner child of the root
    sub = int(node[root, 6 + slot])
    if case == "cut":  # instance 0 misses the subtree, instance 1 is the subtree
        node[root, 6 + slot] = 0xFFFFFFFF
        w[header + stride + root_at] = sub
    else:  # instance 0 is the subtree, instance 1 the whole
        w[header + root_at] = sub
    if case == "raised":
        w[header + stride + root_at] = sub
    scene = engine.upload(layout, w)
    idx = None if gi else torch.from_numpy(mesh.indices.view(np.int32)).cuda()
    try:
        for k in range(2):
            new = (mesh.positions * np.float32(1.2 + 0.3 * k)).astype(np.float32)
            blas.refit(new)
            want = A.pack_scene(layout, [blas], inst, tlas_mode=0)
            scene.refit(0, torch.from_numpy(new).cuda(), idx)
            got = scene.words()
            if case == "raised" and k == 0:
                assert np.array_equal(got[base:base + 16 * (sub + 1)], want[base:base + 16 * (sub + 1)])
                w[header + stride + root_at] = root
                scene.update_records(w[:header + 2 * stride])
                continue
            nodes = 16 * (root + (case != "cut"))  # the cut root's own boxes enclose less
            assert np.array_equal(got[base:base + nodes], want[base:base + nodes])
            after = base + 16 * (root + 1)
            assert np.array_equal(got[after:], want[after:])
    finally:
        scene.release()
