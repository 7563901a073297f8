"""Appends publish in two steps -- a blob is placed in the file, then its hash is
written and its slot set. While two threads append, a third brings the device mirror
up to date again and again and reads what is published, as it is: every published
chunk has its hash on the host and in the mirror, and its voxels; at the end the
whole archive verifies on both."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CHUNK = 256 ** 3


def test_readers_beside_appends(gpu, oracle, tmp_path):
    import torch
    import volumes
    dev = [volumes.region(70 + i, (0, 0, 0), (256, 256, 256), 0.85, device="cuda").contiguous() for i in range(3)]
    torch.cuda.synchronize()
    want, errors, done = {}, [], threading.Event()
    path = str(tmp_path / "p.mca")
    with gpu.open(path, 256 * 40, 512, 256, 6.0) as a:
        for i in range(3):   # row 0 of LOD 1: the blobs wanted
            assert a.append_chunks(1, [(0, 0, i)], [dev[i].data_ptr()], 6.0, on_device=True) == 0
            co = a.chunk_offset(1, 0, 0, i)
            want[i] = np.array(a.decode_chunk(co))

        def writer(row, group):
            try:
                for x0 in range(0, 36, group):
                    at = [(0, row, x) for x in range(x0, x0 + group)]
                    assert a.append_chunks(0, at, [dev[(x + row) % 3].data_ptr() for x in range(x0, x0 + group)], 6.0,
                                           on_device=True) == 0
            except BaseException as e:   # shown below
                errors.append(repr(e))

        def reader():
            try:
                out = np.empty(CHUNK, np.uint8)
                d_out = torch.empty(CHUNK, dtype=torch.uint8, device="cuda")
                k = rounds = 0
                while not done.is_set() or rounds == 0:
                    rounds += 1
                    rc, base, n = a.sync_device()
                    assert rc == 0
                    row, x = (k // 36) % 2, k % 36
                    k += 7
                    co = a.chunk_offset(0, 0, row, x)
                    if not co:
                        continue
                    # published: hashed on the host; the mirror as of now holds the same blob
                    data = np.memmap(path, np.uint8, "r")
                    assert data[co + 4:co + 12].any(), co
                    assert a.decode_chunks_dev([co], d_out.data_ptr()) == 0
                    torch.cuda.synchronize()
                    assert np.array_equal(d_out.cpu().numpy(), want[(x + row) % 3].reshape(-1)), (row, x)
                    gpu.L.mc_archive_decode_chunk(a.a, co, out.ctypes.data, 0)
                    assert np.array_equal(out, want[(x + row) % 3].reshape(-1)), (row, x)
            except BaseException as e:   # shown below
                errors.append(repr(e))

        ws = [threading.Thread(target=writer, args=(0, 4)), threading.Thread(target=writer, args=(1, 1))]
        r = threading.Thread(target=reader)
        for t in ws + [r]:
            t.start()
        for t in ws:
            t.join()
        done.set()
        r.join()
        assert not errors, errors[:3]
        rc, base, n = a.sync_device()
        data = np.fromfile(path, np.uint8)[:n]
        assert rc == 0 and gpu.L.mc_verify_archive(data.ctypes.data, n, 0) == 0
        assert gpu.L.mc_b200_verify_archive_dev(data.ctypes.data, base, n, 0) == 0   # the mirror's bytes hashed
        for row in range(2):
            for x in range(36):
                co = a.chunk_offset(0, 0, row, x)
                blob = data[co:co + _blob_len(data, co)]
                assert oracle.blob_hash(blob.tobytes()) == int(blob[4:12].view(np.uint64)[0]), (row, x)
                assert co + blob.size <= n


def _blob_len(data, co):
    fml = int(data[co + 12]) | int(data[co + 13]) << 8
    np_ = int(np.unpackbits(data[co + 14 + fml:co + 14 + fml + 512]).sum())
    at = co + 14 + fml + 512
    return 14 + fml + 512 + 2 * np_ + int(data[at:at + 2 * np_].copy().view(np.uint16).astype(np.int64).sum())
