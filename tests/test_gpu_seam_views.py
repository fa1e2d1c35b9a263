"""The seam's functions read the values of the tensors that they are given, not their memory: a negated
view (torch keeps a flag instead of negating the memory) gives the hits of its negated copy."""
from __future__ import annotations

import pytest

from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from . import helpers as H

pytestmark = pytest.mark.gpu


def test_negated_views_are_read_as_their_values(engine):
    import torch
    mesh, inst = S.cubes_instanced(12)
    scene = engine.upload(A.LAYOUT_REFLECTION, A.pack_scene(A.LAYOUT_REFLECTION, [A.Blas(mesh.positions, mesh.indices)], inst))
    rays = torch.from_numpy(H.random_rays(500, -14.0, 14.0, seed=3, tmax=40.0)).cuda()
    o, d, tmax = rays[:, 0:3].contiguous(), rays[:, 4:7].contiguous(), rays[:, 7].contiguous()
    try:
        want = A.rs_trace(engine, scene, o, d, 0.0, tmax)
        neg = [torch._neg_view(-x) for x in (o, d, tmax)]
        assert all(x.is_neg() for x in neg) and torch.equal(neg[0], o)
        for args in ((neg[0], d, tmax), (o, neg[1], tmax), (o, d, neg[2])):
            got = A.rs_trace(engine, scene, args[0], args[1], 0.0, args[2])
            assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
        assert bool((want[1][:, 0] != 0).any()) and not bool(torch.equal(A.rs_trace(engine, scene, -o, d, 0.0, tmax)[0], want[0]))
    finally:
        scene.release()
