"""The splat where the sprites' size decides how it is drawn (at once or tiled,
particles per warp, keys read ahead): particle counts and radii on both sides
of each line, bit for bit against the restatement."""
import numpy as np
import pytest

from oracle import oracle as O
from pbf_gb300 import render as Rd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def radius_of(side, H):
    """The radius whose sprites are `side` pixels across at the distance of the
    origin from the reference's camera (8 ** 0.5), fov 50."""
    return side * 2.0 * 8.0 ** 0.5 * float(np.tan(np.pi / 180.0 * 25.0)) / H


@pytest.mark.parametrize("n,W,H,side", [
    (393215, 1280, 819, 16.0), (393216, 1280, 819, 16.0),                       # the least number for tiles
    (393216, 1280, 819, 24.9), (393216, 1280, 819, 25.1),                       # the largest sprites for them
    (524288, 1280, 820, 4.30), (524288, 1280, 820, 4.32),                       # fill 9.5e3
    (149999, 320, 200, 5.6), (150000, 320, 200, 5.6), (150000, 320, 200, 5.8),  # 16 a warp
    (299999, 640, 360, 3.9), (300000, 640, 360, 3.9), (300000, 640, 360, 4.1),  # 32 a warp
    (450000, 960, 540, 0.7),
    (60000, 500, 300, 4.9), (60000, 500, 300, 5.1),                             # keys read ahead
    (400000, 1280, 819, 6.4), (400000, 1280, 819, 6.6), (400000, 1280, 819, 10.6), (800000, 1280, 819, 6.6)])
def test_radius_lines(n, W, H, side):
    rng = np.random.default_rng(n + W)
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = 1.2 * (rng.random((n, 3)) - 0.5)
    cam = Rd.reference_camera(W, H)
    R = radius_of(side, H)
    want = O.render(p, W, H, cam["view"], cam["projection"], R, 16, None)
    r = Rd.FilteredParticleFluid(W, H)
    r.setConfig(filterSize=16, particleRadius=R)
    r.set_camera(cam)
    dp = torch.from_numpy(p).cuda()
    r.render(dp.data_ptr(), n)
    for got, ref in zip((r.depth(), r.volume()), want):
        assert np.array_equal(got.view(np.uint32), np.asarray(ref, np.float32).view(np.uint32))
    r.close()


def test_one_renderer_across_the_lines():
    """Frames of one renderer above and below the tiled line, with more and
    fewer particles than its workspace has held."""
    W, H, R = 1280, 819, 0.02
    cam = Rd.reference_camera(W, H)
    rng = np.random.default_rng(3)
    p = np.zeros((700000, 4), np.float32)
    p[:, :3] = 1.2 * (rng.random((len(p), 3)) - 0.5)
    dp = torch.from_numpy(p).cuda()
    r = Rd.FilteredParticleFluid(W, H)
    r.setConfig(filterSize=16, particleRadius=R)
    r.set_camera(cam)
    for n in (400000, 20000, 450001, 393215, 700000, 400000, 0, 699999):
        want = O.render(p[:n], W, H, cam["view"], cam["projection"], R, 16, None)
        r.render(dp.data_ptr(), n)
        for got, ref in zip((r.depth(), r.volume()), want):
            assert np.array_equal(got.view(np.uint32), np.asarray(ref, np.float32).view(np.uint32))
    r.close()
