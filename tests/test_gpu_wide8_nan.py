"""WIDE8 rays whose range holds a NaN miss, and visit no BLAS: through an 8-wide top level, a packed one
and a flat list, alone and among other rays."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A

from . import helpers as H
from .test_gpu_wide8_schedule import _words

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("top", ["wide", "packed", "list"])
def test_nan_ranges_miss_at_once(engine, layout, top):
    import torch
    words = _words(layout, top != "list", n=50)
    scene = engine.upload(layout, words)
    scene.prepare("wide8")
    if top == "packed":
        scene.update_records(words)  # the 8-wide top level counts as stale: the packed one is walked
    rays = H.random_rays(600, -14.0, 14.0, tmax=1e3)
    rays[0::4] = np.nan
    rays[1::4, 3] = np.nan
    rays[2::4, 7] = np.nan
    try:
        d_rays = torch.from_numpy(rays).cuda()
        dead = d_rays[0::4].contiguous()
        for mode in (A.CLOSEST, A.ANY_CASTERS):
            got = engine.trace(scene, d_rays, mode, "wide8")
            assert torch.equal(got, engine.trace(scene, d_rays, mode, "wide8p"))
            hit = got != 0 if mode != A.CLOSEST else got[:, 1] != (-1 if layout == A.LAYOUT_GI else 0)
            assert not bool(hit[0::4].any() | hit[1::4].any() | hit[2::4].any()) and bool(hit[3::4].any())
            counts = engine.trace_counted(scene, dead, mode)
            assert counts["rays"] == len(dead)
            assert counts["nodes"] == counts["triangles"] == 0, counts
            assert top != "wide" or counts["top_nodes"] == 0, counts
    finally:
        scene.release()
