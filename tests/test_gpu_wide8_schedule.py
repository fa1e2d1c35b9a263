"""The WIDE8 walks' schedules change no result: the per-ray walk at every refill width and the packet
walk write the same records at launch sizes around a warp and a block, with the FP64 oracle's hits,
over a flat list of instances and over a top level; and a plan made over a flat list stays right
when the records then gain a top level."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from . import helpers as H
from .test_gpu_wide8 import check_any, check_closest

pytestmark = pytest.mark.gpu


def _words(layout, top, n=23):
    meshes = [S.clusters(k, stream=S.Stream(400 + k), half=4.0) for k in (5, 60, 700)]
    s = S.Stream(55)
    rot = S.quaternion_matrices(s, n)
    model = np.concatenate([rot * s.range(0.5, 2.0, n)[:, None, None], s.range(-10.0, 10.0, n, 3)[:, :, None]],
                           axis=2).astype(np.float32)
    inst = S.Instances(model, S.affine_inverse_rows(model), (np.arange(n) % 3).astype(np.uint32))
    return A.pack_scene(layout, [A.Blas(m.positions, m.indices) for m in meshes], inst, tlas_mode=1 if top else 0)


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("top", [False, True], ids=["list", "top"])
@pytest.mark.parametrize("n", [1, 31, 33, 129, 2049])
def test_schedules_agree(engine, layout, top, n):
    import torch
    words = _words(layout, top)
    rays = H.random_rays(n, -14.0, 14.0, seed=3 + n, tmax=1e3)
    d_rays = torch.from_numpy(rays).cuda()
    scene = engine.upload(layout, words)
    scene.prepare("wide8")
    try:
        for mode in (A.CLOSEST, A.ANY_CASTERS):
            first = None
            for kernel, refill in (("wide8", 1), ("wide8", 8), ("wide8", 32), ("wide8p", 32)):
                engine.set_tuning(wide8_refill=refill)
                got = engine.trace(scene, d_rays, mode, kernel).cpu().numpy().view(np.uint32)
                first = got if first is None else first
                assert np.array_equal(got, first), f"{kernel} refill {refill}"
            ref64, ident64 = O.fp64_trace(words, rays, layout, any_hit=mode != A.CLOSEST)
            if mode == A.CLOSEST:
                check_closest(layout, first, ref64, ident64, f"n {n}")
            else:
                check_any(first.reshape(-1), rays, ref64, f"n {n}")
    finally:
        engine.set_tuning(wide8_refill=8)
        scene.release()


def test_a_flat_plan_outlives_a_new_top_level(engine):
    import torch
    layout = A.LAYOUT_REFLECTION
    words = _words(layout, True, n=50)
    flat = words.copy()
    flat[1] = 0  # no top level: a list of 50 instances
    rays = torch.from_numpy(H.random_rays(3000, -14.0, 14.0, tmax=1e3)).cuda()
    scene = engine.upload(layout, flat)
    scene.prepare("wide8")
    plan = engine.plan(scene, [(rays, A.CLOSEST)], "wide8")
    try:
        plan.launch()
        before = plan.hits[0].clone()
        scene.update_records(words)
        plan.hits[0].zero_()
        plan.launch()
        torch.cuda.synchronize()
        assert torch.equal(plan.hits[0], before)
        scene.prepare("wide8")
        assert torch.equal(engine.trace(scene, rays, A.CLOSEST, "wide8"), before)
    finally:
        plan.close()
        scene.release()


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
def test_the_default_stack_gives_the_local_stack_results(layout):
    """Where no placement was set, any-hit launches over a flat scene take the shared stack; the flags
    are the local stack's through single launches, batches and plans (direct and captured)."""
    import torch
    mesh = S.clusters(20_000, stream=S.Stream(8))
    words = A.pack_scene(layout, [A.Blas(mesh.positions, mesh.indices)], S.identity_instances(1))
    rays = torch.from_numpy(H.random_rays(30_011, -120.0, 120.0, seed=6, tmax=300.0)).cuda()
    batches = [(rays[:7], A.ANY_CASTERS), (rays[7:], A.ANY_SKY)]
    got = {}
    for stack in ("", "local"):
        engine = A.Engine(0)
        if stack:
            engine.set_tuning(wide8_stack=A.STACKS[stack])
        scene = engine.upload(layout, words)
        scene.prepare("wide8")
        assert scene.wide8_depth() <= 16 and engine.tuning()["wide8_stack"] == A.STACKS["local"]
        out = [engine.trace(scene, rays, A.ANY_CASTERS, "wide8")] + engine.trace_batches(scene, batches, "wide8")
        for graph in (False, True):
            plan = engine.plan(scene, batches, "wide8", graph=graph)
            plan.launch()
            torch.cuda.synchronize()
            out += [h.clone() for h in plan.hits]
            plan.close()
        assert engine.stats()["stack_overflows"] == 0
        got[stack] = out
        scene.release()
        engine.close()
    assert all(torch.equal(a, b) for a, b in zip(got[""], got["local"]))
    assert any(bool(h.any()) for h in got[""])
