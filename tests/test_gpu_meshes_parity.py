"""PLAIN and FAST against the oracle's restatement of the WGSL loops over scenes of several meshes, whose GI
node words start at every offset from a 16-byte boundary, with and without primitive tables, as a list
and under a top level, at launch sizes of few and of many rays: every word of every hit."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from . import helpers as H
from .test_gpu_parity import check_same, gpu_trace, oracle_words, product_words

pytestmark = pytest.mark.gpu

COUNTS = (1, 6, 9, 61, 402, 1003, 11, 12, 14)  # triangles a mesh: lone leaves, two leaves, trees


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("top", [False, True], ids=["list", "top"])
def test_meshes_at_every_offset(engine, layout, top):
    meshes = [S.clusters(n, stream=S.Stream(700 + n), half=4.0) for n in COUNTS]
    s = S.Stream(41)
    n = 40 if top else len(COUNTS)
    model = np.concatenate([S.quaternion_matrices(s, n) * s.range(0.5, 2.0, n)[:, None, None],
                            s.range(-12.0, 12.0, n, 3)[:, :, None]], axis=2).astype(np.float32)
    inst = S.Instances(model, S.affine_inverse_rows(model), (np.arange(n) % len(COUNTS)).astype(np.uint32), np.arange(n) % 5 != 3)
    prims = [k % 2 == 0 for k in range(len(meshes))] if layout == A.LAYOUT_GI else None
    w = product_words(layout, meshes, inst, 1 if top else 0, prims)
    assert np.array_equal(w, oracle_words(layout, meshes, inst, 1 if top else 0, prims))
    if layout == A.LAYOUT_GI:
        assert {int(x) & 3 for x in w[16:16 + 32 * n].reshape(n, 32)[:, 18]} == {0, 1, 2, 3}
    scene = engine.upload(layout, w)
    try:
        for count in (700, 40_000):
            rays = H.random_rays(count, -16.0, 16.0, seed=count, tmax=60.0)
            rays[::13, 4 + np.arange(len(rays[::13])) % 3] = 0.0
            rays[1::7, 3] = 2.0
            for mode in (A.CLOSEST, A.ANY_SKY, A.ANY_CASTERS):
                want, _ = O.gi_trace(w, rays, mode) if layout == A.LAYOUT_GI else O.rs_trace(w, rays, mode != 0)
                hit = want[:, 1] != (A.MISS if layout == A.LAYOUT_GI else 0)
                assert hit.any() and not hit.all()
                for kernel in ("plain", "fast"):
                    check_same(gpu_trace(engine, scene, rays, mode, kernel), hit.astype(np.uint32) if mode else want,
                               f"{kernel}, {count} rays, mode {mode}")
    finally:
        scene.release()
