"""Warm-up of the served form (no GPU: builds are recorded): some build of it
takes each of the builder's paths, whatever sizes the caller names."""
import pytest

from ehss_b200.serve import DeviceExecutor


@pytest.mark.parametrize('sizes', [None, (300,), (64, 1536, 4096, 12000)])
def test_every_builder_path_is_warmed_up(sizes):
    ex = DeviceExecutor.__new__(DeviceExecutor)
    built, traced = [], []
    ex.build = lambda structures: built.append((len(structures), max(len(r) for _, r in structures))) or [structures]
    ex.trace = traced.append
    ex.warmup(*(() if sizes is None else (sizes,)))
    assert len(traced) == len(sizes or (64, 4096, 12000))
    for lone, low, high in ((True, 1, 1024), (True, 1025, 2048), (True, 2049, 8192), (False, 1, 2048), (False, 2049, 8192),
                            (True, 8193, 1 << 27)):
        assert any((count <= 8) == lone and low <= n <= high for count, n in built), (lone, low, high)
