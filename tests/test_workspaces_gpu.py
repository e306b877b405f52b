"""Device memory that the library keeps: how it grows and how much a small
context takes, by the device's free memory."""
import numpy as np
import pytest

from pbf_gb300 import render as Rd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_renderer_workspace_grows_by_half():
    """A scene that emits particles: after the first tiled frame there is room
    for half as many again without another allocation."""
    W, H = 640, 360
    dp = torch.from_numpy(np.random.default_rng(1).random((1100000, 4)).astype(np.float32) - 0.5).cuda()
    r = Rd.FilteredParticleFluid(W, H)
    r.setConfig(filterSize=16, particleRadius=0.04)
    r.set_camera(Rd.reference_camera(W, H))
    r.render(dp.data_ptr(), 1000)
    before = free_bytes()
    r.render(dp.data_ptr(), 700000)
    first = free_bytes()
    assert 16 * 700000 <= before - first <= 24 * 700000 + (4 << 20)
    for n in (700001, 800000, 950000, 1049999, 700000):
        r.render(dp.data_ptr(), n)
        assert free_bytes() == first
    r.close()
