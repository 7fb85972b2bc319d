"""Batches on either side of the numbers of structures and atoms up to which one
CTA makes each tree: a structure's scene is the same byte for byte in both."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bytes(batch, i):
    off = batch.scene_ptrs[i] - batch.scene_buf.data_ptr()
    return batch.scene_buf[off:off + int(batch._sizes[i])].cpu().numpy()


@pytest.mark.parametrize('exterior', [False, True])
@pytest.mark.parametrize('largest', [3, 1024, 2048, 2049, 6144, 6145, 8192])
def test_eight_and_nine_structures(largest, exterior):
    from ehss_b200 import workloads as W
    from ehss_b200.batch import BatchScenes
    sizes = [largest, 1, 2, 14, 15, 300, 777, 40, 5]
    shapes = [W.globule(min(n, largest), n)[:2] for n in sizes]
    eight, nine = BatchScenes(shapes[:8], exterior=exterior), BatchScenes(shapes, exterior=exterior)
    alone = BatchScenes(shapes[8:], exterior=exterior)
    for batch in (eight, nine, alone):
        batch.scene_buf.zero_()                          # alignment padding is never written
        batch.build()
    for i in range(8):
        assert np.array_equal(_bytes(eight, i), _bytes(nine, i)), i
    assert np.array_equal(_bytes(alone, 0), _bytes(nine, 8))
