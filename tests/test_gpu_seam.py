"""The seam's functions over separate origin / direction / range arrays (one launch, rt_trace_split) give
the bits of the same rays traced from a ray buffer by the PLAIN kernel, at ray counts around each
number of rays a warp, for strided views and for ranges given once or per ray; arguments that the
one launch does not take go through a buffer."""
from __future__ import annotations

import numpy as np
import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from . import helpers as H

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[A.LAYOUT_GI, A.LAYOUT_REFLECTION], ids=["gi", "reflection"])
def scene(request, engine):
    mesh, inst = S.cubes_instanced(12)
    inst.casts = np.arange(len(inst)) % 4 != 1
    sc = engine.upload(request.param, A.pack_scene(request.param, [A.Blas(mesh.positions, mesh.indices)], inst, tlas_mode=1))
    yield sc
    sc.release()


@pytest.mark.parametrize("n", [1, 33, 4736, 4737, 9473, 37_889, 75_777, 151_553])
def test_seam_equals_the_ray_buffer(engine, scene, n):
    import torch
    rays = torch.from_numpy(H.random_rays(n, -14.0, 14.0, seed=n, tmax=40.0)).cuda()
    rays[::5, 3] = 0.5
    rays[::7, 4] = 0.0
    closest = engine.trace(scene, rays, A.CLOSEST, "plain")
    blocked = {m: engine.trace(scene, rays, m, "plain") != 0 for m in (A.ANY_SKY, A.ANY_CASTERS)}
    o, d, tmin, tmax = rays[:, 0:3], rays[:, 4:7], rays[:, 3].contiguous(), rays[:, 7].contiguous()
    for oo, dd in ((o, d), (o.contiguous(), d.contiguous())):  # strided views, and arrays of their own
        if scene.layout == A.LAYOUT_GI:
            got = A.gi_closest(engine, scene, oo, dd, tmin, tmax)
            want = A.decode_gi(closest)
            for k in want:  # NaN-free: compare the bits
                assert torch.equal(got[k].contiguous().view(torch.int32), want[k].contiguous().view(torch.int32)), k
        else:
            t, rec = A.rs_trace(engine, scene, oo, dd, tmin, tmax)
            assert torch.equal(t.contiguous().view(torch.int32), closest[:, 0]) and torch.equal(rec, closest[:, 1:5])
            assert torch.equal(A.rs_blocked(engine, scene, oo, dd, tmin, tmax), blocked[A.ANY_CASTERS])
    rays[:, 3], rays[:, 7] = 0.0, 40.0
    want = engine.trace(scene, rays, A.ANY_CASTERS, "plain") == 0
    for tm in (40.0, 40, torch.full((n,), 40.0, device="cuda"), torch.tensor(40.0, device="cuda"), np.float32(40.0)):
        assert torch.equal(A.gi_visible_within(engine, scene, o, d, tm), want)
    rays[:, 7] = 1e20
    assert torch.equal(A.gi_visible(engine, scene, o, d), engine.trace(scene, rays, A.ANY_SKY, "plain") == 0)
    assert torch.equal(A.gi_visible(engine, scene, o, d, kernel="fast"), A.gi_visible(engine, scene, o, d))
    # double arrays go through a ray buffer, as before
    assert torch.equal(A.gi_visible(engine, scene, o.double(), d.double()), A.gi_visible(engine, scene, o, d))


def test_seam_without_rays(engine, scene):
    import torch
    none = torch.empty((0, 3), device="cuda")
    assert A.gi_visible(engine, scene, none, none).shape == (0,)
