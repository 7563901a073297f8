"""Which kernels a deblocking call launches, counted as the nodes of a captured
graph: none for an axis without faces, one for all three axes where tiles of the
whole volume pay, one per axis where they would read and write rows that no face
touches or leave most of a warp idle; and the voxels either way."""
import numpy as np
import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CASES = [((16, 16, 16), 0), ((1, 16, 16), 0), ((512, 1, 16), 1), ((1, 512, 16), 1), ((8, 8, 512), 1), ((16, 256, 64), 2),
         ((256, 16, 1008), 2), ((256, 40, 16), 2), ((40, 40, 32), 3), ((24, 24, 96), 3), ((24, 24, 640), 3),
         ((32, 32, 1024), 3), ((40, 40, 64), 1), ((100, 100, 48), 1), ((256, 256, 256), 1), ((40, 40, 896), 1), ((100, 100, 912), 3),
         ((40, 33, 256), 3), ((40, 40, 72), 3)]


def _launches(gpu, oracle, size, q):
    import torch
    from cuda.bindings import runtime as rt
    nz, ny, nx = size
    rng = np.random.default_rng(nz * 7919 + ny * 31 + nx)
    vol = np.clip(100 + rng.integers(-6, 7, size), 1, 255).astype(np.uint8)
    d = torch.from_numpy(vol).cuda()
    s = torch.cuda.Stream()
    gpu.deblock_dev(d.data_ptr(), 1, vol.size, nz, ny, nx, q, s.cuda_stream)   # not the first call under capture
    s.synchronize()
    assert np.array_equal(d.cpu().numpy(), oracle.deblock(vol.copy(), q))
    h = s.cuda_stream
    assert rt.cudaStreamBeginCapture(h, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == 0
    rc = gpu.deblock_dev(d.data_ptr(), 1, vol.size, nz, ny, nx, q, h)
    err, graph = rt.cudaStreamEndCapture(h)
    assert rc == 0 and err == 0
    try:
        err, _, n = rt.cudaGraphGetNodes(graph, 0)
        assert err == 0
        return n
    finally:
        rt.cudaGraphDestroy(graph)


@pytest.mark.parametrize("size,launches", CASES)
def test_launches(gpu, oracle, size, launches):
    assert _launches(gpu, oracle, size, 6.0) == launches


@pytest.mark.parametrize("q", [0.5, 6.0, 62.0, 62.4, 100.0])
def test_what_the_benchmark_reports(gpu, oracle, monkeypatch, q):
    monkeypatch.syspath_prepend(ROOT)
    import bench
    assert len(bench.deblock_kernels(q)) == _launches(gpu, oracle, (256, 256, 256), q)
