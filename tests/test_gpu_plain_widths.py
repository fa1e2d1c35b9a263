"""PLAIN launches on both sides of each number of rays at which they spread differently over warps or take
another kernel (few rays a warp, GI closest hits that fit fewer blocks an SM, GI any hits in full
warps): every word is the oracle's, over a list of instances and under a top level."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from renderlab_b200 import api as A

from . import helpers as H
from .test_gpu_wide8_schedule import _words

pytestmark = pytest.mark.gpu

SMS = 148
# rays at which 5, 7 and 8 blocks of 4 warps an SM are full with 1 (and a quarter more), 8, 16 and 32 rays a warp
EDGES = sorted({int(SMS * 4 * blocks * width) for blocks in (5, 7, 8) for width in (1, 1.25, 8, 16, 32)})


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("top", [False, True], ids=["list", "top"])
def test_every_width_gives_the_oracles_hits(engine, layout, top):
    import torch
    words = _words(layout, top)
    base = H.random_rays(2999, -14.0, 14.0, seed=12, tmax=60.0)
    base[::17, 4] = 0.0
    scene = engine.upload(layout, words)
    try:
        for mode in (A.CLOSEST, A.ANY_SKY):
            want = O.gi_trace(words, base, mode)[0] if layout == A.LAYOUT_GI else O.rs_trace(words, base, mode != 0)[0]
            hit = want[:, 1] != (A.MISS if layout == A.LAYOUT_GI else 0)
            want = torch.from_numpy((hit.astype(np.uint32) if mode else want).view(np.int32)).cuda()
            for n in [e + d for e in EDGES for d in (0, 1)]:
                pick = torch.arange(n, device="cuda") % len(base)
                got = engine.trace(scene, torch.from_numpy(base).cuda()[pick].contiguous(), mode, "plain")
                assert torch.equal(got, want[pick]), f"{n} rays, mode {mode}"
    finally:
        scene.release()
