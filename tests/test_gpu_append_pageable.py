"""Appends from pageable host memory: a thread's first ones take no longer than
those that follow (no pinned buffers are made for them), a chunk alone is copied
plainly also where there are such buffers, and the blobs of chunks before and after
they come in are those of the same voxels on the device."""
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CHUNK = 256 ** 3


def test_first_appends(gpu, tmp_path):
    """Three threads, one after another: pinning three 8 MiB buffers takes 10 ms and
    more, a driver's own allocation now and then as long."""
    import torch
    import volumes
    dev = [volumes.region(60 + i, (0, 0, 0), (256, 256, 256), 0.9, device="cuda").contiguous() for i in range(3)]
    host = [d.cpu().numpy() for d in dev]
    torch.cuda.synchronize()
    extra, errors = [], []

    def run(path):
        try:
            with gpu.open(path, 256 * 32, 256, 256, 6.0) as a:
                for i in range(3):   # the thread's other buffers, and the blobs wanted
                    assert a.append_chunks(0, [(0, 0, i)], [dev[i].data_ptr()], 6.0, on_device=True) == 0
                t = []
                for k in range(12):
                    t0 = time.perf_counter()
                    assert a.append_chunks(0, [(0, 0, 3 + k)], [host[k % 3]], 6.0) == 0
                    t.append(time.perf_counter() - t0)
                extra.append(t[0] - float(np.median(t[1:6])))
                # 15 to 29: calls of several chunks, the buffers made in the second; 30, 31: alone again
                for c0, n in ((15, 10), (25, 5)):
                    assert a.append_chunks(0, [(0, 0, c) for c in range(c0, c0 + n)], [host[(c - 15) % 3] for c in
                                                                                       range(c0, c0 + n)], 6.0) == 0
                assert a.append_chunks(0, [(0, 0, 30)], [host[0]], 6.0) == 0
                pinned = torch.from_numpy(host[0]).pin_memory().numpy()
                assert a.append_chunks(0, [(0, 0, 31)], [pinned], 6.0) == 0
                for c in range(3, 32):
                    i = 0 if c >= 30 else (c - 3) % 3
                    co, want = a.chunk_offset(0, 0, 0, c), a.chunk_offset(0, 0, 0, i)
                    for b in range(0, 4096, 61):
                        at = b >> 8, (b >> 4) & 15, b & 15
                        assert a.block_blob(co, *at) == a.block_blob(want, *at), (c, b)
        except BaseException as e:   # handed to the test
            errors.append(e)

    for k in range(3):
        th = threading.Thread(target=run, args=(str(tmp_path / f"a{k}.mca"),))
        th.start()
        th.join()
        if errors:
            raise errors[0]
    assert min(extra) < 6e-3, extra
