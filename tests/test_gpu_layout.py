"""The batch layout made on the device (arena ranges and processing order), at
item counts around its CTAs' 1024 items and with every length class in use:
absent blocks, the shortest payloads and ones past 4092 bytes; and the
reconstruction's dealing of blocks to CTAs, one or two at a time, around the
count where it changes. Whole numbers: equality with the oracle's block
decoder."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def chunk(gpu, oracle, tmp_path_factory):
    """A chunk whose blocks repeat 61 distinct ones, and those blocks' voxels."""
    q, rng = 0.25, np.random.default_rng(23)
    distinct = [np.zeros((16, 16, 16), np.uint8), np.full((16, 16, 16), 90, np.uint8)]
    for i in range(59):
        distinct.append(np.clip(rng.normal(128, 0.02 * 1.17 ** i, (16, 16, 16)), 1, 255).astype(np.uint8))
    lens = [len(oracle.enc_block(b, q)) for b in distinct]
    assert min(lens[1:]) < 32 and max(lens) > 4092
    want = [oracle.dec_block(oracle.enc_block(b, q), q).reshape(16, 16, 16) if b.any() else b for b in distinct]
    pick = rng.integers(0, len(distinct), 4096)
    vox = np.stack([distinct[p] for p in pick]).reshape(16, 16, 16, 16, 16, 16).transpose(0, 3, 1, 4, 2, 5)
    a = gpu.open(str(tmp_path_factory.mktemp("lay") / "l.mca"), 256, 256, 256, q)
    assert a.append_ctx(0, 0, 0, 0, np.ascontiguousarray(vox).reshape(256, 256, 256), q, 0) == 0
    yield a, pick, np.stack(want)
    a.close()


@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1024, 1025, 2048, 4096, 6001])
def test_item_counts(chunk, n):
    import torch
    a, pick, want = chunk
    at = np.random.default_rng(n).integers(0, 4096, n)
    boxes = [(16 * int(b >> 8), 16 * int(b >> 4 & 15), 16 * int(b & 15)) for b in at]
    out = torch.full((n, 4096), 0xA7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert a.read_regions_dev(0, boxes, 16, 16, 16, out.data_ptr(), 4096) == 0
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().reshape(n, 16, 16, 16), want[pick[at]])


def test_nothing_coded(chunk):
    import torch
    a, pick, want = chunk
    air = [int(i) for i in np.flatnonzero(pick == 0)]
    out = torch.full((len(air), 4096), 0xA7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert a.read_regions_dev(0, [(16 * (b >> 8), 16 * (b >> 4 & 15), 16 * (b & 15)) for b in air], 16, 16, 16,
                              out.data_ptr(), 4096) == 0
    torch.cuda.synchronize()
    assert not out.any()


@pytest.mark.parametrize("over", [-1, 0, 1, 2, 2 * 9 * 148 + 1])
def test_blocks_per_cta(chunk, over):
    """Around 64 blocks for each of the reconstruction's CTAs (9 per SM)."""
    import torch
    a, pick, want = chunk
    n = 64 * 9 * torch.cuda.get_device_properties(0).multi_processor_count + over
    short = np.flatnonzero(pick < 20)     # payloads of a few dozen bytes: one batch holds them all
    at = short[np.random.default_rng(5).integers(0, len(short), n)]
    boxes = [(16 * int(b >> 8), 16 * int(b >> 4 & 15), 16 * int(b & 15)) for b in at]
    out = torch.full((n + 1, 4096), 0xA7, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert a.read_regions_dev(0, boxes, 16, 16, 16, out.data_ptr(), 4096) == 0
    torch.cuda.synchronize()
    ref = torch.from_numpy(want.reshape(-1, 4096)).cuda()[torch.from_numpy(pick[at]).cuda()]
    assert torch.equal(out[:n], ref) and bool((out[n] == 0xA7).all())
