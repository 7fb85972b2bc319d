"""Host threads that build batches and count grids of different sizes at the
same time, each on a stream of its own: no call fails and every result is the
single thread's."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_concurrent_builds_and_grids():
    import torch
    import ehss_b200 as eb
    from ehss_b200 import workloads as W
    from ehss_b200.adaptive_pa import grid_counts
    from ehss_b200.batch import BatchScenes
    shapes = {n: W.globule(n, n)[:2] for n in (200, 1500, 3000, 7000)}
    sizes = {200: (2, 4096), 1500: (16, 512), 3000: (16, 64), 7000: (4, 1024)}     # directions and grid of each thread
    scenes = {n: eb.Scene(*s) for n, s in shapes.items()}

    def work(n):
        batch = BatchScenes([shapes[n]], exterior=True)
        batch.scene_buf.zero_()                          # alignment padding is never written
        batch.build()
        return batch.scene_buf.cpu().numpy()[batch.scene_ptrs[0] - batch.scene_buf.data_ptr():][:int(batch._sizes[0])], \
            grid_counts(scenes[n], *sizes[n], 3)[0]
    want = {n: work(n) for n in shapes}
    failures = []
    start = threading.Barrier(len(shapes))

    def loop(n):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                start.wait(60)
                for _ in range(60):
                    got = work(n)
                    if not all(np.array_equal(a, b) for a, b in zip(got, want[n])):
                        raise AssertionError(f'{n} atoms: another result than one thread gives')
        except Exception as e:
            failures.append(f'{n} atoms: {type(e).__name__}: {e}')
    torch.cuda.synchronize()
    threads = [threading.Thread(target=loop, args=(n,)) for n in shapes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[:3]
