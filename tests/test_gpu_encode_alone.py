"""The single-block coder (mc_enc_block): its payloads against the oracle's where
its runs, bands, density classes, rungs, escapes, corrections and carries end, and
its time next to the same block's decode -- one thread codes what one thread
decodes, so the two are of a size."""
import time

import numpy as np
import pytest

from test_entropy_runs import _blocks

pytestmark = pytest.mark.gpu


def _noise(rng):
    return rng.integers(1, 256, (16, 16, 16)).astype(np.uint8)


@pytest.mark.parametrize("q,tau", [(0.25, 0), (1.0, 0), (1.0, 4), (6.0, 0), (6.0, 1), (40.0, 0), (40.0, 2)])
def test_payloads(gpu, oracle, q, tau):
    rng = np.random.default_rng(5)
    # at q = 0.25 enough written words for a carry past the held bytes (one in 65536)
    blocks = _blocks(oracle) + [_noise(rng) for _ in range(8 if q > 0.25 else 160)]
    blocks += [np.zeros((16, 16, 16), np.uint8), (rng.random((16, 16, 16)) < 0.5).astype(np.uint8) * 255]
    for i, b in enumerate(blocks):
        assert gpu.enc_block(b, q, tau) == oracle.enc_block(b, q, tau), i


def _median(f):
    f()
    t = []
    for _ in range(9):
        t0 = time.perf_counter()
        f()
        t.append(time.perf_counter() - t0)
    return sorted(t)[4]


@pytest.mark.parametrize("q,tau", [(0.5, 0), (1.0, 4), (24.0, 4)])
def test_time_beside_the_decode(gpu, q, tau):
    """At most twice the decode's time (dense blocks; a coder that pays every
    lane's step for its one lane takes 3.2 times at q = 0.5)."""
    b = _noise(np.random.default_rng(6))
    pay = gpu.enc_block(b, q, tau)
    assert _median(lambda: gpu.enc_block(b, q, tau)) < 2.0 * _median(lambda: gpu.dec_block(pay, q))
