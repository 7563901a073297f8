"""The encoder's symbol pool: the device memory that a group of chunks takes, and
groups with more levels and corrections than the pool is first made for (noise
with a tight bound), whose blobs are the oracle's all the same and leave the
thread's encoder as good as before. Each in a thread of its own: a thread keeps
its encoder's buffers."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CHUNK = 256 ** 3


def _in_thread(f):
    out = []

    def run():
        try:
            out.append(f())
        except BaseException as e:   # handed to the test
            out.append(e)
    t = threading.Thread(target=run)
    t.start()
    t.join()
    if isinstance(out[0], BaseException):
        raise out[0]
    return out[0]


def test_memory_of_eight_chunks(gpu, tmp_path):
    """1160 MiB: payload slots 544, symbols 768 less what the first chunk took of both."""
    import torch
    v = torch.full((8, 256, 256, 256), 90, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()

    def run():
        with gpu.open(str(tmp_path / "m.mca"), 2048, 256, 256, 6.0) as a:
            assert a.append_chunks(0, [(0, 0, 0)], [v[0].data_ptr()], 6.0, on_device=True) == 0
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            assert a.append_chunks(0, [(0, 0, c) for c in range(8)], [v[c].data_ptr() for c in range(8)], 6.0,
                                   on_device=True) == 0
            torch.cuda.synchronize()
            return before - torch.cuda.mem_get_info()[0]
    assert _in_thread(run) <= 1160 << 20


@pytest.mark.parametrize("n,q,tau", [(1, 2.5, 1), (2, 2.5, 1), (1, 0.25, 0)])
def test_dense_symbols(gpu, oracle, tmp_path, n, q, tau):
    import torch
    rng = np.random.default_rng(n)
    base = rng.integers(1, 256, (16, 16, 16, 16, 16, 16)).astype(np.uint8)   # 4096 blocks of noise
    # 32 distinct ones, so that the oracle codes few
    base = base.reshape(4096, 16, 16, 16)[rng.integers(0, 32, 4096)]
    want = {}
    vox = np.ascontiguousarray(base.reshape(16, 16, 16, 16, 16, 16).transpose(0, 3, 1, 4, 2, 5)).reshape(256, 256, 256)
    smooth = np.full((256, 256, 256), 70, np.uint8)
    d = torch.from_numpy(np.stack([vox, smooth])).cuda()
    torch.cuda.synchronize()

    def run():
        with gpu.open(str(tmp_path / "d.mca"), 1024, 256, 256, q) as a:
            kw = {"ctx_q": q, "ctx_tau": tau} if tau else {}
            # sparse, dense, sparse again, dense again
            for c, src in ((0, [1] * n), (n, [0] * n)):
                assert a.append_chunks(0, [(0, 0, (c + k) % 4) for k in range(n)], [d[s].data_ptr() for s in src], q,
                                       on_device=True, **kw) == 0
            for b in range(0, 4096, 7):
                key = base[b].tobytes()
                if key not in want:
                    want[key] = oracle.enc_block(base[b], q, tau)
                z, y, x = b >> 8, (b >> 4) & 15, b & 15
                for k in range(n):
                    co = a.chunk_offset(0, 0, 0, (n + k) % 4)
                    assert a.block_blob(co, z, y, x) == want[key], (b, k)
            one = oracle.enc_block(smooth[:16, :16, :16], q, tau)
            assert a.block_blob(a.chunk_offset(0, 0, 0, 0), 3, 4, 5) == one
            # the single-block call shares the pool
            assert gpu.enc_block(base[0], q, tau) == want[base[0].tobytes()]
        return sum(len(w) for w in want.values())
    assert _in_thread(run) > 0
    if tau:   # the case is what it says: more than 6144 symbols a block
        b = base[0]
        plain = oracle.enc_block(b, q, 0)
        off = np.abs(oracle.dec_block(plain, q).reshape(b.shape).astype(int) - b.astype(int)) > tau
        assert np.count_nonzero(oracle.dec_levels(plain, q)[0]) + np.count_nonzero(off) > 6144
