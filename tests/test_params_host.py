"""Shapes of the per-atom parameters before they reach the engine: what the device copies may read, and
what the host path broadcasts or refuses; the device that the copies are queued on.  No GPU: the library is
a stand-in that records its calls."""
import contextlib
import ctypes
import types

import numpy as np
import pytest
import torch

from dmff_b200 import engine
from dmff_b200.engine import AdmpEngine, DispEngine

N = 4


class _Lib:
    def __init__(self):
        self.calls = []

    def dmffb_admp_set_params(self, h, Q, pol, thole):
        vals = lambda p, m: None if p is None else np.ctypeslib.as_array((ctypes.c_double * m).from_address(p.value)).copy()  # noqa: E731
        self.calls.append((vals(Q, 9 * N).reshape(N, 9), vals(pol, N), vals(thole, N)))
        return 0

    def dmffb_disp_set_params(self, h, c, a, b, q):
        vals = lambda p, m: None if p is None else np.ctypeslib.as_array((ctypes.c_double * m).from_address(p.value)).copy()  # noqa: E731
        self.calls.append((vals(c, 3 * N), vals(a, N), vals(b, N), vals(q, N)))
        return 0


def _engine(cls, lib):
    eng = cls.__new__(cls)
    eng.lib, eng.h, eng.n, eng.device = lib, None, N, -1  # device -1: no CUDA device is entered
    return eng


def _z(*shape):
    return torch.zeros(shape, dtype=torch.float64)


@pytest.mark.parametrize("Q,pol,thole,ok", [
    (_z(N, 9), None, None, True),
    (_z(N, 4), _z(N), _z(N, 1), True),
    (_z(N, 0), None, None, True),
    (_z(N - 1, 9), None, None, False),
    (_z(N + 1, 9), None, None, False),
    (_z(1, 9), None, None, False),
    (_z(N, 10), None, None, False),
    (_z(9 * N), None, None, False),
    (_z(N, 9), _z(N - 1), _z(N), False),
    (_z(N, 9), _z(N), _z(1), False),
    (_z(N, 9), _z(N + 1), _z(N + 1), False),
    (_z(N, 9), _z(N), None, False),
])
def test_what_the_device_copies_may_read(Q, pol, thole, ok):
    assert _engine(AdmpEngine, None)._per_atom(Q, pol, thole) is ok


def test_host_path_broadcasts_and_refuses():
    lib = _Lib()
    eng = _engine(AdmpEngine, lib)
    eng.set_params(np.arange(4.0)[None], 1.0 + np.arange(N), np.full(N + 1, 0.3))  # one row; a longer array
    Q, pol, thole = lib.calls.pop()
    assert np.array_equal(Q, np.tile(np.r_[0.0, 1, 2, 3, 0, 0, 0, 0, 0], (N, 1)))
    assert np.array_equal(pol, 1.0 + np.arange(N)) and np.array_equal(thole, np.full(N, 0.3))
    eng.set_params(_z(N, 9), _z(N, 1), None)  # the engine answers a missing thole
    assert lib.calls.pop()[2] is None
    for args in ((_z(N - 1, 9),), (_z(N, 10),), (_z(N, 9), _z(N - 1), _z(N)), (_z(N, 9), _z(N), _z(1))):
        with pytest.raises(ValueError):
            eng.set_params(*args)
    assert not lib.calls


@pytest.mark.parametrize("c,rest,ok", [
    (_z(N, 3), (None, None, None), True),
    (_z(N, 3), (_z(N), _z(N, 1), _z(N)), True),
    (_z(3, N), (None, None, None), False),
    (_z(3 * N), (None, None, None), False),
    (_z(N - 1, 3), (None, None, None), False),
    (_z(N, 1), (None, None, None), False),
    (_z(N, 3), (_z(N), _z(N - 1), _z(N)), False),
    (_z(N, 3), (_z(N), _z(N), _z(1)), False),
])
def test_what_the_dispersion_device_copies_may_read(c, rest, ok):
    assert _engine(DispEngine, None)._per_atom(c, *rest) is ok


def test_dispersion_host_path():
    lib = _Lib()
    eng = _engine(DispEngine, lib)
    eng.set_params(np.arange(3.0 * N), *(np.full(N + 1, float(k)) for k in range(3)))  # flat, longer arrays
    c, a, b, q = lib.calls.pop()
    assert np.array_equal(c, np.arange(3.0 * N)) and [x[0] for x in (a, b, q)] == [0.0, 1.0, 2.0]
    for args in ((_z(N, 1),), (_z(N - 1, 3),), (_z(N, 3), _z(N), _z(N - 1), _z(N))):
        with pytest.raises(ValueError):
            eng.set_params(*args)
    assert not lib.calls


@pytest.mark.parametrize("cls,name,args", [
    (AdmpEngine, "dmffb_admp_set_params_device", (_z(N, 4), _z(N), _z(N))),
    (DispEngine, "dmffb_disp_set_params_device", (_z(N, 3), None, None, None)),
])
def test_device_path_enters_the_engines_device(monkeypatch, cls, name, args):
    """Buffers are allocated and kernels launched there: both go by the current device."""
    current, seen = [], []

    @contextlib.contextmanager
    def device(d):
        current.append(d)
        yield
        current.pop()

    monkeypatch.setattr(engine, "_on_device", lambda *a: True)
    monkeypatch.setattr(torch.cuda, "device", device)
    monkeypatch.setattr(torch.cuda, "current_stream", lambda d: types.SimpleNamespace(cuda_stream=0))
    lib = types.SimpleNamespace(**{name: lambda *a: seen.append(list(current)) or 0})
    _engine(cls, lib).set_params(*args)
    assert seen == [[-1]]
