"""The one-CTA tree builder at the edges of its instances (1024, 2048, 8192
atoms; half and quarter sorts; one or two CTAs an SM; node boxes in shared or
global memory): its scenes equal the device-wide builder's byte for byte."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shapes(sizes):
    from ehss_b200 import workloads as W
    rng = np.random.default_rng(4)
    out = [W.globule(n, n)[:2] for n in sizes]
    out.append((np.zeros((40, 3)), np.full(40, 1.5)))                                           # equal keys only
    out.append((rng.normal(size=(700, 3)) * [30., 1., .1], np.full(700, 1.7)))                  # a thin sheet
    return out


def _bytes(batch, i):
    off = batch.scene_ptrs[i] - batch.scene_buf.data_ptr()
    return batch.scene_buf[off:off + int(batch._sizes[i])].cpu().numpy()


@pytest.mark.parametrize('leaf_size', [1, 14])
@pytest.mark.parametrize('exterior', [False, True])
@pytest.mark.parametrize('sizes,copies', [
    ((1, 2, 15, 511, 512, 513, 1023, 1024), 1), ((1025, 2047, 2048), 1), ((2049, 4096, 4097, 8192), 1), ((6500,), 1),
    ((20, 300, 1500), 40), ((17, 900), 60), ((2500, 40), 40)])
def test_scenes_equal_the_device_wide_builder(sizes, copies, exterior, leaf_size):
    from ehss_b200 import workloads as W
    from ehss_b200.batch import BatchScenes
    shapes = _shapes(sizes) * copies
    small = BatchScenes(shapes, leaf_size=leaf_size, exterior=exterior)
    wide = BatchScenes(shapes + [W.globule(8300, 1)[:2]], leaf_size=leaf_size, exterior=exterior)
    for batch in (small, wide):
        batch.scene_buf.zero_()                          # alignment padding is never written
        batch.build()
    for i in range(len(shapes)):
        assert np.array_equal(_bytes(small, i), _bytes(wide, i)), (i, len(shapes[i][1]))
