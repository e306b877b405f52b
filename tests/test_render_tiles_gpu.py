"""The splat at the edges of its split over warps and of its two-phase path (a
first share, the tiles' depth test, volume sprites summed by tile), bit for bit
against the restatement: the particle counts where they change, crowded tiles,
sprites too large for a tile's window, and maps whose sides are no multiple of
a tile."""
import numpy as np
import pytest

from oracle import oracle as O
from pbf_gb300 import render as Rd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,W,H,R,spread", [(32767, 321, 177, 0.02, 0.5), (32768, 321, 177, 0.02, 0.5),
                                            (40001, 640, 360, 0.02, 0.03), (33000, 203, 95, 0.2, 0.6),
                                            (50000, 1023, 577, 0.01, 2.5), (524287, 1280, 820, 0.01, 0.5),
                                            (524288, 1280, 820, 0.01, 0.5), (524288, 1023, 1031, 0.01, 2.5),
                                            (600001, 1031, 1023, 0.02, 0.03), (3000, 1031, 1023, 0.02, 0.3),
                                            (10001, 320, 200, 0.05, 0.3), (393215, 1600, 880, 0.01, 2.5),
                                            (393216, 1600, 880, 0.01, 2.5), (655359, 320, 200, 0.01, 0.5),
                                            (655360, 320, 200, 0.01, 0.5)])
def test_two_phase_splat(n, W, H, R, spread):
    rng = np.random.default_rng(n + W)
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = 0.2 + spread * (rng.random((n, 3)) - 0.5)
    p[: n // 50, :3] = [1.6, 1.6, 0.0] + 0.3 * rng.random((n // 50, 3))  # close to the camera at (2, 2, 0)
    p = p[rng.permutation(n)]
    scene = rng.random((H, W)).astype(np.float32) * 0.03
    cam = Rd.reference_camera(W, H)
    want = O.render(p, W, H, cam["view"], cam["projection"], R, 16, scene.copy())
    r = Rd.FilteredParticleFluid(W, H)
    r.setConfig(filterSize=16, particleRadius=R)
    r.set_camera(cam)
    dp = torch.from_numpy(p).cuda()
    for _ in range(2):  # the workspace and the maps of the first frame are reused
        ds = torch.from_numpy(scene).cuda()
        r.render(dp.data_ptr(), n, ds.data_ptr())
        torch.cuda.synchronize()
        for got, ref in zip((r.depth(), r.volume(), ds.cpu().numpy()), want):
            assert np.array_equal(got.view(np.uint32), np.asarray(ref, np.float32).view(np.uint32))
    r.close()
