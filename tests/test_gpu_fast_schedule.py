"""The FAST kernels' schedule (the warp's vote over kinds of step, lanes left idle in small launches,
results stored at a refill or at the end) and their loads (GI meshes that start at any word) change
no bit: every hit equals the PLAIN kernel's, at launch sizes around a warp, a block and a full grid
and for rays with zero, infinite and NaN components."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from . import helpers as H

pytestmark = pytest.mark.gpu

# triangle counts of the meshes of one scene: their records follow one another, so a GI mesh's node
# words start at every offset from a 16-byte boundary; leaves of 1 to 8 triangles, and a lone leaf
COUNTS = (1, 7, 8, 9, 61, 402, 1003)


@pytest.fixture(scope="module", params=[(A.LAYOUT_GI, False), (A.LAYOUT_GI, True), (A.LAYOUT_REFLECTION, True)],
                ids=["gi-list", "gi-top", "reflection-top"])
def scene(request, engine):
    layout, top = request.param
    meshes = [S.clusters(n, stream=S.Stream(900 + n), half=4.0) for n in COUNTS]
    blas = [A.Blas(m.positions, m.indices) for m in meshes]
    s = S.Stream(77)
    n = 40 if top else len(COUNTS)
    rot = S.quaternion_matrices(s, n)
    model = np.concatenate([rot * s.range(0.5, 2.0, n)[:, None, None], s.range(-12.0, 12.0, n, 3)[:, :, None]],
                           axis=2).astype(np.float32)
    inst = S.Instances(model, S.affine_inverse_rows(model), (np.arange(n) % len(COUNTS)).astype(np.uint32),
                       np.arange(n) % 5 != 3)
    words = A.pack_scene(layout, blas, inst, tlas_mode=1 if top else 0, primitives=[k % 2 == 0 for k in range(len(blas))])
    if layout == A.LAYOUT_GI:
        starts = {int(w) & 3 for w in words[16:16 + 32 * n].reshape(n, 32)[:, 18]}
        assert len(starts) > 1, "the scene should hold misaligned nodes"
    sc = engine.upload(layout, words)
    yield sc
    sc.release()


def _rays(n):
    r = H.random_rays(n, -16.0, 16.0, seed=n)
    special = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 1e-38, 1e38], np.float32)
    k = np.arange(0, n, 11)
    r[k, 4 + k % 3] = special[(k // 11) % len(special)]
    r[k[::3], (k[::3]) % 3] = special[(k[::3] // 33) % len(special)]
    r[1::7, 3] = 2.0
    r[2::7, 7] = 9.0
    return r


@pytest.mark.parametrize("mode", [A.CLOSEST, A.ANY_SKY, A.ANY_CASTERS])
@pytest.mark.parametrize("n", [1, 31, 33, 129, 4145, 40_003, 140_001])
def test_every_hit_is_the_plain_kernels(engine, scene, n, mode):
    import torch
    rays = torch.from_numpy(_rays(n)).cuda()
    want = engine.trace(scene, rays, mode, "plain")
    for refill in (1, 8, 32):
        engine.set_tuning(fast_refill=refill)
        got = engine.trace(scene, rays, mode, "fast")
        torch.cuda.synchronize()
        bad = (got != want).reshape(n, -1).any(1).nonzero().flatten()
        assert len(bad) == 0, f"refill {refill}: {len(bad)} rays differ, first {bad[:3].tolist()}"
    engine.set_tuning(fast_refill=8)
