"""Which kernels a deblocking call launches, counted as the nodes of a captured
graph: none for an axis without faces, one for all three axes where tiles of the
whole volume pay, one per axis where they would read and write rows that no face
touches or leave most of a warp idle; and the voxels either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CASES = [((16, 16, 16), 0), ((1, 16, 16), 0), ((512, 1, 16), 1), ((1, 512, 16), 1), ((8, 8, 512), 1), ((16, 256, 64), 2),
         ((256, 16, 1008), 2), ((256, 40, 16), 2), ((40, 40, 32), 3), ((24, 24, 96), 3), ((24, 24, 640), 3),
         ((32, 32, 1024), 3), ((40, 40, 64), 1), ((100, 100, 48), 1), ((256, 256, 256), 1), ((40, 40, 896), 1), ((100, 100, 912), 3),
         ((40, 33, 256), 3), ((40, 40, 72), 3)]


@pytest.mark.parametrize("size,launches", CASES)
def test_launches(gpu, oracle, size, launches):
    import torch
    from cuda.bindings import runtime as rt
    nz, ny, nx = size
    rng = np.random.default_rng(nz * 7919 + ny * 31 + nx)
    vol = np.clip(100 + rng.integers(-6, 7, size), 1, 255).astype(np.uint8)
    d = torch.from_numpy(vol).cuda()
    s = torch.cuda.Stream()
    gpu.deblock_dev(d.data_ptr(), 1, vol.size, nz, ny, nx, 6.0, s.cuda_stream)   # not the first call under capture
    s.synchronize()
    assert np.array_equal(d.cpu().numpy(), oracle.deblock(vol.copy(), 6.0))
    h = s.cuda_stream
    assert rt.cudaStreamBeginCapture(h, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)[0] == 0
    rc = gpu.deblock_dev(d.data_ptr(), 1, vol.size, nz, ny, nx, 6.0, h)
    err, graph = rt.cudaStreamEndCapture(h)
    assert rc == 0 and err == 0
    try:
        err, _, n = rt.cudaGraphGetNodes(graph, 0)
        assert err == 0 and n == launches
    finally:
        rt.cudaGraphDestroy(graph)
