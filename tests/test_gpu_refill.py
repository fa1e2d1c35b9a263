"""Launches of more rays than the GPU holds lanes, so that lanes take new rays while results of ended ones
wait to be stored: every refill width, the packet walk and a batch of both modes give the same records,
which are the FP64 oracle's where it is asked. And host batches of several chunks each, smaller than
the staging slots, give the records of the device launches."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from . import helpers as H
from .test_gpu_wide8 import check_any, check_closest
from .test_gpu_wide8_schedule import _words

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("top", [False, True], ids=["list", "top"])
def test_refills_agree(engine, layout, top):
    import torch
    words = _words(layout, top)
    n = 200_003
    rays = H.random_rays(n, -14.0, 14.0, seed=8, tmax=40.0)
    d_rays = torch.from_numpy(rays).cuda()
    split = n // 2 + 13
    scene = engine.upload(layout, words)
    scene.prepare("wide8")
    try:
        whole = {}
        for mode in (A.CLOSEST, A.ANY_CASTERS):
            whole[mode] = engine.trace(scene, d_rays, mode, "wide8p")
            some = np.arange(0, n, 97)
            got = whole[mode].cpu().numpy().view(np.uint32)[some]
            ref64, ident64 = O.fp64_trace(words, rays[some], layout, any_hit=mode != A.CLOSEST)
            if mode == A.CLOSEST:
                check_closest(layout, got, ref64, ident64, "closest")
            else:
                check_any(got.reshape(-1), rays[some], ref64, "any hit")
        for refill in (1, 8, 32):
            engine.set_tuning(wide8_refill=refill)
            for mode in whole:
                assert torch.equal(engine.trace(scene, d_rays, mode, "wide8"), whole[mode]), f"refill {refill}, mode {mode}"
            mixed = engine.trace_batches(scene, [(d_rays[:split], A.CLOSEST), (d_rays[split:], A.ANY_CASTERS)], "wide8")
            assert torch.equal(mixed[0], whole[A.CLOSEST][:split]) and torch.equal(mixed[1], whole[A.ANY_CASTERS][split:])
    finally:
        engine.set_tuning(wide8_refill=8)
        scene.release()


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
def test_host_batches_of_several_chunks(engine, layout):
    import torch
    mesh = S.clusters(30_000, stream=S.Stream(4))
    scene = engine.upload(layout, A.pack_scene(layout, [A.Blas(mesh.positions, mesh.indices)], S.identity_instances(1)))
    scene.prepare("wide8")
    engine.reserve(1 << 20)
    batches = [(H.random_rays(n, -110.0, 110.0, seed=n, tmax=300.0), mode, kernel)
               for n, mode, kernel in ((700_001, A.CLOSEST, "wide8"), (600_003, A.ANY_SKY, "wide8"), (3, A.CLOSEST, "plain"),
                                       (300_000, A.ANY_CASTERS, "fast"))]
    try:
        got = engine.trace_host_batches(scene, batches)
        for (rays, mode, kernel), out in zip(batches, got):
            want = engine.trace(scene, torch.from_numpy(rays).cuda(), mode, kernel).cpu().numpy().view(np.uint32)
            assert np.array_equal(out.reshape(want.shape), want), (len(rays), mode, kernel)
            assert out.any()
    finally:
        scene.release()
