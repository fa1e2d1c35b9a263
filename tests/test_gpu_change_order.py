"""A move or a refit returns with its work queued on the caller's stream; what is called next on the
scene sees its result all the same: host-buffer traces, word reads, record rewrites, a prepare, traces
and further changes on other streams. The stream is kept busy in front of the change, so that it
is still queued when the next call is made."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from renderlab_b200 import api as A
from renderlab_b200 import scenes as S

from . import helpers as H

pytestmark = pytest.mark.gpu

LAYOUTS = pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
STREAMS = pytest.mark.parametrize("side", [False, True], ids=["default", "side"])
BUSY = 1_000_000  # cycles


def _instances(n, seed):
    s = S.Stream(seed)
    model = np.concatenate([S.quaternion_matrices(s, n) * s.range(0.5, 2.0, n)[:, None, None],
                            s.range(-40.0, 40.0, n, 3)[:, :, None]], axis=2).astype(np.float32)
    return S.Instances(model, S.affine_inverse_rows(model), (np.arange(n) % 2).astype(np.uint32))


class Moved:
    """A scene with a top level and its words as the host moves them."""

    def __init__(self, engine, layout, n=2500):
        meshes = [S.clusters(k, stream=S.Stream(k), half=2.0) for k in (3, 40)]
        blas = [A.Blas(m.positions, m.indices) for m in meshes]
        self.engine, self.layout, self.n = engine, layout, n
        self.boxes = A.object_boxes(layout, blas)
        self.host = A.pack_scene(layout, blas, _instances(n, 1), tlas_mode=1)
        self.scene = engine.upload(layout, self.host)
        self.rays = H.random_rays(64, -40.0, 40.0, seed=5, tmax=200.0)

    def want(self, seed):
        return A.move_instances_host(self.layout, self.host, _instances(self.n, seed), self.boxes)

    def move(self, seed, stream, busy=True):
        import torch
        new = _instances(self.n, seed)
        self.host = A.move_instances_host(self.layout, self.host, new, self.boxes)
        with torch.cuda.stream(stream):
            if busy:
                torch.cuda._sleep(BUSY)
            self.scene.move_instances(new, self.boxes)

    def hits(self):
        return (O.gi_trace(self.host, self.rays, 0) if self.layout == A.LAYOUT_GI else O.rs_trace(self.host, self.rays, False))[0]


def _stream(side):
    import torch
    return torch.cuda.Stream() if side else torch.cuda.default_stream()


@pytest.fixture
def moved(engine, layout):
    m = Moved(engine, layout)
    yield m
    m.scene.release()


@LAYOUTS
@STREAMS
def test_a_host_trace_sees_the_move(moved, side):
    stream = _stream(side)
    for k in range(70):  # past a rebuild of the top level
        moved.move(100 + k, stream, busy=k % 2 == 0)
        got = moved.engine.trace_host(moved.scene, moved.rays, A.CLOSEST, "fast")
        want = moved.hits()
        assert np.array_equal(got.reshape(want.shape), want), f"move {k}"


@LAYOUTS
@STREAMS
def test_reads_and_rewrites_see_the_move(moved, side):
    import torch
    stream = _stream(side)
    for k in range(6):
        moved.move(10 + k, stream)
        assert np.array_equal(moved.scene.words(), moved.host)
    for k in range(3):  # a rewrite of the records comes after the moves queued before it
        other = moved.want(50 + k)
        moved.move(20 + k, stream)
        moved.scene.update_records(other)
        torch.cuda.synchronize()
        moved.host = other
        assert np.array_equal(moved.scene.words(), other)
    moved.scene.prepare("wide8")
    moved.move(30, stream)
    moved.scene.prepare("wide8")  # its top level is made from the moved records
    rays = torch.from_numpy(moved.rays).cuda()
    got = moved.engine.trace(moved.scene, rays, A.CLOSEST, "wide8")
    fresh = moved.engine.upload(moved.layout, moved.host)
    fresh.prepare("wide8")
    assert torch.equal(got, moved.engine.trace(fresh, rays, A.CLOSEST, "wide8"))
    fresh.release()


@LAYOUTS
def test_other_streams_see_the_move(moved):
    import torch
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    rays = torch.from_numpy(moved.rays).cuda()
    batch = [(rays, A.CLOSEST)]
    plan = moved.engine.plan(moved.scene, batch, "fast")
    torch.cuda.synchronize()
    for k in range(8):
        moved.move(40 + k, (a, b)[k % 2])  # moves in turn on two streams: as if on one
        with torch.cuda.stream((b, a)[k % 2]):
            got = [moved.engine.trace(moved.scene, rays, A.CLOSEST, kernel) for kernel in ("plain", "fast")]
            got += moved.engine.trace_batches(moved.scene, batch, "fast")
            plan.launch()
        torch.cuda.synchronize()
        want = moved.hits()
        for h in got + plan.hits:
            assert np.array_equal(h.cpu().numpy().view(np.uint32).reshape(want.shape), want), f"move {k}"
    for k in range(8):
        moved.move(60 + k, (a, b)[k % 2], busy=k == 0)
    assert np.array_equal(moved.scene.words(), moved.host)
    plan.close()


@LAYOUTS
def test_a_captured_trace_sees_the_move_and_a_move_is_not_captured(moved):
    import torch
    rays = torch.from_numpy(moved.rays).cuda()
    hits = moved.engine.trace(moved.scene, rays, A.CLOSEST, "fast")
    stream, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
    before = moved.host
    moved.move(7, torch.cuda.Stream())
    with torch.cuda.graph(graph, stream=stream):
        moved.engine.trace(moved.scene, rays, A.CLOSEST, "fast", hits=hits)
        with pytest.raises(A.RtError):
            moved.scene.move_instances(_instances(moved.n, 8), moved.boxes)
    graph.replay()
    torch.cuda.synchronize()
    want = moved.hits()
    assert np.array_equal(hits.cpu().numpy().view(np.uint32).reshape(want.shape), want)
    assert np.array_equal(moved.scene.words(), moved.host) and not np.array_equal(before, moved.host)
    del graph


@LAYOUTS
@STREAMS
def test_a_host_trace_sees_the_refit(engine, layout, side):
    import torch
    stream = _stream(side)
    mesh = S.clusters(20_000, stream=S.Stream(3))
    blas = A.Blas(mesh.positions, mesh.indices)
    inst = S.identity_instances(1)
    words = A.pack_scene(layout, [blas], inst)
    scene = engine.upload(layout, words)
    base = int(words[16 + 18]) if layout == A.LAYOUT_GI else int(words[8 + 18]) & ~3
    idx = torch.from_numpy(mesh.indices.view(np.int32)).cuda() if layout == A.LAYOUT_REFLECTION else None
    rays = H.random_rays(64, -90.0, 90.0, seed=9, tmax=400.0)
    torch.cuda.synchronize()
    try:
        for k in range(12):
            new = (mesh.positions * np.float32(0.97 ** (k + 1))).astype(np.float32)
            blas.refit(new)
            words = words.copy()
            words[base:] = A.pack_scene(layout, [blas], inst)[base:]
            with torch.cuda.stream(stream):
                d_new = torch.from_numpy(new).cuda()
                torch.cuda._sleep(BUSY)
                scene.refit(0, d_new, idx)
            got = engine.trace_host(scene, rays, A.CLOSEST, "fast")
            want = (O.gi_trace(words, rays, 0) if layout == A.LAYOUT_GI else O.rs_trace(words, rays, False))[0]
            assert np.array_equal(got.reshape(want.shape), want), f"refit {k}"
    finally:
        torch.cuda.synchronize()
        scene.release()
