"""The splat on maps whose volume tiles take more than one round of the scan that
places them (1,024 tiles a round), bit for bit against the restatement: just
under and over a round, over two, and a map with one tile row."""
import numpy as np
import pytest

from oracle import oracle as O
from pbf_gb300 import render as Rd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,W,H,R,spread", [(400003, 1584, 1488, 0.006, 2.0), (400003, 1632, 1488, 0.006, 2.0),
                                            (393217, 3001, 1601, 0.003, 2.5), (655361, 16384, 48, 0.02, 2.5)])
def test_many_volume_tiles(n, W, H, R, spread):
    rng = np.random.default_rng(W)
    p = np.zeros((n, 4), np.float32)
    p[:, :3] = 0.2 + spread * (rng.random((n, 3)) - 0.5)
    cam = Rd.reference_camera(W, H)
    want = O.render(p, W, H, cam["view"], cam["projection"], R, 16, None)
    r = Rd.FilteredParticleFluid(W, H)
    r.setConfig(filterSize=16, particleRadius=R)
    r.set_camera(cam)
    dp = torch.from_numpy(p).cuda()
    for _ in range(2):
        r.render(dp.data_ptr(), n)
        for got, ref in zip((r.depth(), r.volume()), want):
            assert np.array_equal(got.view(np.uint32), np.asarray(ref, np.float32).view(np.uint32))
    r.close()
