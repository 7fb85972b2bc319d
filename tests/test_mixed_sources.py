"""Sources whose rays do not all start without a collider or owner (no GPU: the
library is a stand-in that notes what it is given): every ray is launched once,
with the arrays that are needed."""
from types import SimpleNamespace

import numpy as np
import pytest
from test_device_of_calls import _Torch

from ehss_b200 import _lib, engine


@pytest.mark.parametrize('call', ['trace', 'query'])
@pytest.mark.parametrize('n,differ', [(1, 0), (3000, 0), (3000, 1000), (3000, 1), (40000, 0), (40000, 13000), (40000, 2), (70000, 0),
                                      (70000, 23000), (70000, 2)])
def test_rays_are_launched_once(monkeypatch, call, n, differ):
    fake, launched = _Torch(), []
    lib = SimpleNamespace(
        ehss_trace_host_workspace_bytes=lambda n, out: 0,
        ehss_trace_host=lambda scene, n, cap, prec, o, d, last, bounces, *rest: launched.append((n, last, bounces)) or 0,
        ehss_pa_anyhit=lambda scene, n, o, d, owners, *rest: launched.append((n, owners, None)) or 0)
    monkeypatch.setattr(engine, 'torch', lambda: fake)
    monkeypatch.setattr(engine, 'stream_handle', lambda device: 0)
    monkeypatch.setattr(_lib, 'load', lambda: lib)
    scene = SimpleNamespace(device='cuda:0', ptr=256, n_atoms=5, exterior=False)
    last = np.full(n, -1)
    if differ:
        last[1:-1:(n - 2) // differ] = 3                 # the ends do not
    d = np.tile([0., 0., 1.], (n, 1))
    if call == 'trace':
        engine.GPUEHSSTransport(scene).trace(engine.EHSSSource(d, d, d, np.ones(n), last, np.zeros(n, dtype=int), 't'))
    else:
        index = engine.SphereIndex.__new__(engine.SphereIndex)
        index.scene = scene
        index.query(SimpleNamespace(origins=d, directions=d, owners=last))
    (rays, given, bounces), = launched
    assert rays == n and (given is not None) == (differ > 0) and bounces is None


@pytest.mark.parametrize('value', [-1, 0])
def test_uniform_arrays(value):
    for n in (1, 7, 100):
        a = np.full(n, value)
        assert engine._unless(a, value) is None
        for other in (5, -1 - value, -7):
            a[n // 2] = other
            assert engine._unless(a, value) is a
    assert engine._unless(np.empty(0, dtype=np.int64), value) is not None
    a = np.full(100000, value)
    assert engine._unless(a, value) is None and engine._seems_all(a, value)
    a[::3] = 7
    assert engine._unless(a, value) is a and not engine._seems_all(a, value)
