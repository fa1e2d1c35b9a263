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


def test_another_meshes_parts_are_left(engine):
    """Two GI instances over the same nodes, the second with leaves and positions of its own: a refit of the
    first, which enters a subtree, reads and writes its own parts alone."""
    import torch
    mesh = S.clusters(3000, stream=S.Stream(13))
    blas = A.Blas(mesh.positions, mesh.indices)
    inst = S.identity_instances(2)
    inst.mesh[:] = 0
    w = A.pack_scene(A.LAYOUT_GI, [blas], inst, tlas_mode=0)
    base, leaves, root = int(w[16 + 18]), int(w[16 + 19]), int(w[16 + 22])
    node = w[base:leaves].reshape(-1, 16)
    sub = next(int(c) for c in node[root, 6:10] if 0 < c < root)
    own = len(w)  # a second copy of all behind the nodes
    w = np.concatenate([w, w[leaves:]])
    w[16 + 22] = sub
    w[48 + 19:48 + 22] += own - leaves
    scene = engine.upload(A.LAYOUT_GI, w)
    try:
        for k in range(2):  # the second time from the kept topology
            new = (mesh.positions * np.float32(1.5 + k)).astype(np.float32)
            blas.refit(new)
            want = A.pack_scene(A.LAYOUT_GI, [blas], inst, tlas_mode=0)
            scene.refit(0, torch.from_numpy(new).cuda())
            got, low = scene.words(), base + 16 * (sub + 1)
            assert np.array_equal(got[base:low], want[base:low])
            assert np.array_equal(got[low:leaves], w[low:leaves]) and np.array_equal(got[own:], w[own:])
            assert np.array_equal(got[leaves:own], want[leaves:own])
        scene.refit(1, torch.from_numpy(new).cuda())
        got = scene.words()
        assert np.array_equal(got[base:own], want[base:own]) and np.array_equal(got[own:], want[leaves:own])
    finally:
        scene.release()
