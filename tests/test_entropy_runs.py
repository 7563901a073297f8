"""The entropy steps at the places where a run of zeros, a band, the density
window or an Exp-Golomb escape ends: blocks with chosen coefficients, coded by
the oracle and decoded by the stage-1 device code built for the host (see
test_entropy_host_emulation.py), and on the GPU coded and decoded through every
entropy kernel. Whole numbers: equality with the oracle."""
import numpy as np
import pytest

from test_entropy_host_emulation import _check, emu  # noqa: F401  (emu: the host build, a fixture)


def _basis():
    k, n = np.arange(16)[:, None], np.arange(16)[None, :]
    c = np.cos(np.pi * (2 * n + 1) * k / 32) * np.sqrt(2.0 / 16)
    c[0] = 0.25
    return c


def _block(scan, places):
    """Voxels whose transform is large at the given (scan position, amplitude)s."""
    co = np.zeros(4096)
    for p, a in places:
        co[scan[p]] = a
    c = _basis()
    v = np.einsum("zyx,zk,yl,xm->klm", co.reshape(16, 16, 16), c, c, c, optimize=True)
    return np.clip(np.rint(v + 128), 1, 255).astype(np.uint8)


def _scan(oracle):
    s = np.zeros(4096, np.uint16)
    oracle.L.or_scan_table(s.ctypes.data)
    return s


ENDS = [56, 364, 1128, 2240, 3280, 3876, 4076]   # the first position past each band


def _blocks(oracle):
    scan = _scan(oracle)
    rng = np.random.default_rng(17)
    out = [_block(scan, [(0, 30.0)]), _block(scan, [(4095, 60.0)]), np.full((16, 16, 16), 77, np.uint8)]
    for gap in range(0, 24):       # two, three and four ones this far apart: windows of every density class
        for n in (2, 3, 4):
            out.append(_block(scan, [(5 + i * (gap + 1), 40.0 + 9 * i) for i in range(n)] + [(900, 60.0)]))
    for e in ENDS:                 # coefficients around a band's end, alone and behind a run
        for d in range(-6, 6):
            out.append(_block(scan, [(max(0, e + d), 70.0), (min(4095, e + 9), 90.0)]))
    for a in (20.0, 60.0, 150.0, 400.0, 900.0):   # magnitudes up the ladder and into escapes
        out.append(_block(scan, [(0, a), (1, -a / 2), (2, a / 3), (9, -a / 4), (30, a / 5)]))
    for _ in range(20):            # dense and sparse noise
        out.append(np.clip(rng.normal(128, rng.choice([2, 10, 60]), (16, 16, 16)), 0, 255).astype(np.uint8))
    return out


@pytest.mark.parametrize("q", [0.25, 1.0, 6.0])
def test_runs_on_the_host(emu, oracle, q):  # noqa: F811
    for i, b in enumerate(_blocks(oracle)):
        _check(emu, oracle, oracle.enc_block(b, q), q, f"block {i} q {q}")


@pytest.mark.gpu
@pytest.mark.parametrize("q,tau", [(0.25, 0), (1.0, 4), (6.0, 0), (6.0, 1)])
def test_runs_on_the_gpu(gpu, oracle, tmp_path, q, tau):
    """One chunk holding the blocks: the coder gives the oracle's payloads, and
    every share of the two entropy kernels its voxels."""
    blocks = _blocks(oracle)
    vox = np.zeros((256, 256, 256), np.uint8)
    for i, b in enumerate(blocks):
        z, y, x = (i * 7) % 4096 >> 8, (i * 7) >> 4 & 15, (i * 7) & 15
        vox[16 * z:16 * z + 16, 16 * y:16 * y + 16, 16 * x:16 * x + 16] = b
    with gpu.open(str(tmp_path / "r.mca"), 256, 256, 256, q) as a:
        assert a.append_ctx(0, 0, 0, 0, vox, q, tau) == 0
        co = a.chunk_offset(0, 0, 0, 0)
        for i, b in enumerate(blocks):
            z, y, x = (i * 7) % 4096 >> 8, (i * 7) >> 4 & 15, (i * 7) & 15
            want = oracle.enc_block(b, q, tau)
            assert a.block_blob(co, z, y, x) == want, i
            if i % 8 == 0:
                assert np.array_equal(a.decode_block(co, z, y, x).reshape(-1), oracle.dec_block(want, q).reshape(-1)), i
        ref = None
        try:
            for share in (0, 1, 3, -1):
                assert gpu.L.mc_b200_set_entropy_solo(share) == 0
                got = a.decode_chunk(co).copy()
                ref = got if ref is None else ref
                assert np.array_equal(got, ref), share
        finally:
            gpu.L.mc_b200_set_entropy_solo(-1)
        for i, b in enumerate(blocks):
            z, y, x = (i * 7) % 4096 >> 8, (i * 7) >> 4 & 15, (i * 7) & 15
            want = oracle.dec_block(oracle.enc_block(b, q, tau), q).reshape(16, 16, 16)
            got = ref.reshape(256, 256, 256)[16 * z:16 * z + 16, 16 * y:16 * y + 16, 16 * x:16 * x + 16]
            assert np.array_equal(got, want), i
