"""The one-pass deblocking kernel against the oracle where its tiles can go
wrong: tiles cut by the volume's edges on either side of a face, a single row,
plane or vector, the longest row, a face in the last plane, and the sizes and
qualities just past its rule (a face in a plane's last row, a gate above the
half-precision bound, rows off a 16-byte boundary). Whole numbers: equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [(16, 16, 16), (17, 18, 32), (33, 20, 48), (12, 13, 16), (5, 36, 64), (20, 4, 32), (1, 32, 48), (50, 17, 32),
         (34, 34, 1024), (19, 21, 1040), (40, 28, 80)]


@pytest.mark.parametrize("nz,ny,nx", SIZES)
def test_tiles(gpu, oracle, nz, ny, nx):
    import torch
    rng = np.random.default_rng(nz * 10007 + ny * 101 + nx)
    lv = rng.integers(0, 256, (2, (nz + 15) // 16, (ny + 15) // 16, (nx + 15) // 16))
    near = np.repeat(np.repeat(np.repeat(lv, 16, 1), 16, 2), 16, 3)[:, :nz, :ny, :nx]
    vols = np.stack([np.clip(near[0] // 8 + 100 + rng.integers(-4, 5, near[0].shape), 0, 255),
                     np.clip(near[1] + rng.integers(-30, 31, near[1].shape), 0, 255)]).astype(np.uint8)
    vols[rng.random(vols.shape) < 0.03] = 0
    for q in (0.5, 6.0, 62.0, 62.4, 300.0):
        for shift in (0, 8):
            buf = torch.full((vols.size + 64,), 0xA7, dtype=torch.uint8, device="cuda")
            buf[shift:shift + vols.size] = torch.from_numpy(vols.ravel()).cuda()
            torch.cuda.synchronize()
            assert gpu.deblock_dev(buf.data_ptr() + shift, 2, vols[0].size, nz, ny, nx, q) == 0
            got = buf.cpu().numpy()
            for c in range(2):
                want = oracle.deblock(vols[c].copy(), q)
                at = shift + c * vols[0].size
                assert np.array_equal(got[at:at + vols[0].size].reshape(nz, ny, nx), want), (q, shift, c)
            assert (got[:shift] == 0xA7).all() and (got[shift + vols.size:] == 0xA7).all()
