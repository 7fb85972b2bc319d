"""Batches whose staged and uploaded coordinates differ: a build uses the
centres of the coordinates that the device holds, whichever were staged last."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _frames():
    from ehss_b200 import workloads as W
    first = [W.globule(n, n)[:2] for n in (40, 300)]
    second = [(c * 1.1 + 7., r) for c, r in first]
    return first, second


def _bytes(batch):
    return batch.scene_buf.cpu().numpy()[batch.scene_ptrs[0] - batch.scene_buf.data_ptr():]


def _built(structures, exterior, change=lambda batch: None):
    from ehss_b200.batch import BatchScenes
    batch = BatchScenes(structures, exterior=exterior)
    batch.scene_buf.zero_()                              # alignment padding is never written
    batch.upload()
    change(batch)
    batch.build(upload=False)
    return batch


@pytest.mark.parametrize('exterior', [False, True])
def test_staging_the_next_frame_leaves_the_uploaded_one(exterior):
    first, second = _frames()
    want = _built(first, exterior)
    got = _built(first, exterior, lambda batch: batch.stage(second))
    for i in range(len(first)):
        assert got.info(i).center[:] == want.info(i).center[:] and got.info(i).radius == want.info(i).radius
    assert np.array_equal(_bytes(got)[:int(sum(got._sizes))], _bytes(want)[:int(sum(want._sizes))])


def test_coordinates_written_on_the_device():
    import torch
    first, second = _frames()
    want = _built(second, False)
    flat = torch.from_numpy(np.concatenate([c.ravel() for c, _ in second]))
    got = _built(first, False, lambda batch: batch.d_xyz.copy_(flat))
    for i in range(len(first)):
        assert got.info(i).center[:] == want.info(i).center[:] and got.info(i).radius == want.info(i).radius


def test_build_before_an_upload_is_not_centred():
    """Nothing uploaded yet: the coordinates are whatever the caller put there."""
    import torch
    from ehss_b200.batch import BatchScenes
    first, second = _frames()
    batch = BatchScenes(first)
    batch.d_xyz.copy_(torch.from_numpy(np.concatenate([c.ravel() for c, _ in second])))
    batch.d_r.copy_(torch.from_numpy(np.concatenate([r for _, r in second])))
    batch.build(upload=False)
    assert batch.info(1).center[:] == _built(second, False).info(1).center[:]
