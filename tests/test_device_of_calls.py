"""Explicit-ray calls launch on their scene's device (no GPU: the library and
torch's CUDA calls are stand-ins), also from a thread whose current device is
another: the handle of a default stream does not name one."""
import contextlib
import threading
from types import SimpleNamespace

import numpy as np
import pytest
import torch as real

from ehss_b200 import _lib, engine


class _Torch:
    """torch with page-locked and device memory replaced by host memory, and a current device per thread."""

    def __init__(self):
        self.local = threading.local()
        stream = SimpleNamespace(cuda_stream=0, synchronize=lambda: None)
        self.cuda = SimpleNamespace(device=self._device, current_stream=lambda device=None: stream)

    def current(self):
        return getattr(self.local, 'device', 'cuda:0')

    @contextlib.contextmanager
    def _device(self, device):
        before, self.local.device = self.current(), device
        try:
            yield
        finally:
            self.local.device = before

    def empty(self, *a, **kw):
        return real.zeros(*a, dtype=kw['dtype'])

    zeros = empty

    def from_numpy(self, a):
        t = real.from_numpy(a)
        return SimpleNamespace(is_pinned=lambda: True, data_ptr=t.data_ptr, copy_=lambda other, **kw: t.copy_(other),
                               to=lambda device, **kw: t)

    def __getattr__(self, name):
        return getattr(real, name)


@pytest.mark.parametrize('call', ['trace', 'query'])
def test_launch_on_the_scene_device(monkeypatch, call):
    fake, seen = _Torch(), []

    def launch(*args):
        seen.append(fake.current())
        return 0
    lib = SimpleNamespace(ehss_trace_host_workspace_bytes=lambda n, out: 0, ehss_trace_host=launch, ehss_pa_anyhit=launch)
    monkeypatch.setattr(engine, 'torch', lambda: fake)
    monkeypatch.setattr(engine, 'stream_handle', lambda device: 0)
    monkeypatch.setattr(_lib, 'load', lambda: lib)
    scene = SimpleNamespace(device='cuda:1', ptr=256, n_atoms=5, exterior=False)
    d = np.tile([0., 0., 1.], (4, 1))
    if call == 'trace':
        source = engine.EHSSSource(np.zeros((4, 3)), d, d, np.ones(4), np.array([-1, 2, 2, -1]), np.zeros(4, dtype=int), 't')
        engine.GPUEHSSTransport(scene).trace(source)
    else:
        index = engine.SphereIndex.__new__(engine.SphereIndex)
        index.scene = scene
        index.query(SimpleNamespace(origins=np.zeros((4, 3)), directions=d, owners=np.array([-1, 2, 2, -1])))
    assert seen and set(seen) == {'cuda:1'} and fake.current() == 'cuda:0'
