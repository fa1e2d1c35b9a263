"""GI leaves whose index words lie on both sides of word 2^32 of the buffer (17 GB, nearly all zeros; the
upload admits it): the hits equal those of the same scene packed tightly."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from . import helpers as H

pytestmark = pytest.mark.gpu


def test_indices_across_the_32_bit_word(engine):
    import torch
    mesh = S.clusters(100, stream=S.Stream(17), half=6.0)
    s = S.Stream(5)
    model = np.concatenate([S.quaternion_matrices(s, 2), np.array([[-8.0, 0, 0], [8.0, 1, 2]])[:, :, None]], axis=2).astype(np.float32)
    inst = S.Instances(model, S.affine_inverse_rows(model), np.zeros(2, np.uint32))
    words = A.pack_scene(A.LAYOUT_GI, [A.Blas(mesh.positions, mesh.indices)], inst, tlas_mode=0, primitives=[True])
    words[16 + 28] = 0  # instance 0 reports position indices, instance 1 primitives
    indices, n = int(words[16 + 21]), mesh.indices.size
    far = (1 << 32) - 150  # the list crosses the line inside a leaf
    big = np.zeros(far + n, np.uint32)
    big[:len(words)] = words
    big[16 + 21] = big[48 + 21] = far
    big[far:] = words[indices:indices + n]
    rays = torch.from_numpy(H.random_rays(20_000, -16.0, 16.0, seed=4, tmax=60.0)).cuda()
    want, got = [], []
    for out, w in ((want, words), (got, big)):
        scene = engine.upload(A.LAYOUT_GI, w)
        for kernel in ("plain", "fast"):
            out += [engine.trace(scene, rays, mode, kernel) for mode in (A.CLOSEST, A.ANY_SKY)]
        hits = A.gi_closest(engine, scene, rays[:, 0:3], rays[:, 4:7], 0.0, 60.0)
        out += [hits[k].contiguous().view(torch.int32) for k in hits]
        torch.cuda.synchronize()
        scene.release()
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    hit = want[0][:, 1]
    assert bool((hit == 0).any()) and bool((hit == 1).any())
