"""The instance records that the packers and moves are given: whatever indexable values a caller holds (integer
arrays of any width, floats, lists, tensors, mappings, rows of more than eight words), each record holds
int(value) in 32 bits, as ctypes stores it."""
from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest

from renderlab_b200 import api as A

N = 5


def _one_by_one(layout, inst):
    arr = (A.RtInstance * N)()
    get = lambda name: getattr(inst, name, None)  # noqa: E731
    for i in range(N):
        r = arr[i]
        r.model[:] = np.asarray(inst.model, np.float32).reshape(N, 12)[i].tolist()
        r.rows[:] = np.asarray(inst.rows, np.float32).reshape(N, 12)[i].tolist()
        r.mesh = int(inst.mesh[i])
        r.slot = int(get("slot")[i]) if get("slot") is not None else i
        r.casts_shadow = int(bool(get("casts")[i])) if get("casts") is not None else 1
        r.near_base = int(get("near_base")[i]) if get("near_base") is not None else 0
        if get("extra") is not None:
            for k in range(8):
                r.extra[k] = int(get("extra")[i][k])
        elif get("casts") is not None and layout == A.LAYOUT_GI:
            r.extra[3] = 0 if get("casts")[i] else 1
    return bytes(arr)


def _tensor(x):
    import torch
    return torch.tensor(x)


FIELDS = {
    "none": {},
    "uint32": dict(slot=np.arange(N, dtype=np.uint32) + 7, casts=np.arange(N) % 2 == 0),
    "int64": dict(slot=np.array([-1, 2 ** 40 + 3, 0, 1, -2 ** 31]), near_base=np.arange(N, dtype=np.int16) - 2),
    "uint64": dict(slot=np.array([2 ** 63 + 5, 2 ** 64 - 1, 0, 1, 2], np.uint64)),
    "floats": dict(slot=np.array([0.9, 1.0, -1.5, 3e9, 4.2]), casts=[0.0, 0.5, 1, "", "x"]),
    "longer": dict(slot=list(range(20)), casts=[True] * 9, extra=np.arange(20 * 11).reshape(20, 11)),
    "wide lists": dict(slot=[2 ** 70 + 1, -1, True, 3.7, np.uint8(9)], near_base=["1", 2, 3, 4, 5]),
    "mapping": dict(slot={i: 10 * i for i in range(N)}, casts={i: i % 2 for i in range(N)}),
    "tensors": dict(slot=_tensor([5, 4, 3, 2, 1]), casts=_tensor([True, False, True, True, False]), near_base=_tensor([1.0] * N)),
    "ragged extra": dict(extra=[[i + k for k in range(8 + i)] for i in range(N)], casts=np.zeros(N, bool)),
    "extra tensor": dict(extra=_tensor([[i * 8 + k for k in range(8)] for i in range(N)])),
}


@pytest.mark.parametrize("layout", [A.LAYOUT_GI, A.LAYOUT_REFLECTION])
@pytest.mark.parametrize("name", FIELDS)
def test_records_hold_every_value(layout, name):
    eye = np.tile(np.eye(3, 4, dtype=np.float32), (N, 1, 1))
    inst = SimpleNamespace(model=eye * 2, rows=eye / 2, mesh=[0, 1, 0, 1, 2], **FIELDS[name])
    arr, n = A._instance_array(layout, inst)
    assert n == N and bytes(arr) == _one_by_one(layout, inst)


@pytest.mark.parametrize("bad", [dict(slot=[1, 2]), dict(slot=np.arange(2)), dict(casts=np.ones(3, bool)), dict(extra=np.zeros((2, 8), int)),
                                 dict(extra=[[1] * 7] * N)])
def test_too_few_values_are_refused(bad):
    eye = np.tile(np.eye(3, 4, dtype=np.float32), (N, 1, 1))
    with pytest.raises(IndexError):
        A._instance_array(A.LAYOUT_GI, SimpleNamespace(model=eye, rows=eye, mesh=np.zeros(N, int), **bad))
