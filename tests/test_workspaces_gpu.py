"""Device memory that the library keeps: how it grows and how much a small
context takes, by the device's free memory."""
import numpy as np
import pytest

from oracle import oracle as O
from pbf_gb300 import NeighborSearch, scenes
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


def test_small_search_contexts_stay_small():
    """A context of 100 points on 6^3 cells needs some 20 KB: 256 of them on one
    stream, each with a search done, stay within 64 KB each."""
    n, dims = 100, (6, 6, 6)
    dp = torch.from_numpy(np.random.default_rng(1).random((n, 4)).astype(np.float32)).cuda()
    stream = torch.cuda.Stream()

    def contexts(count):
        made = [NeighborSearch((0.0, 0.0, 0.0), (6.0,) * 3, dims, n, stream=stream.cuda_stream) for _ in range(count)]
        for ns in made:
            ns.run(dp.data_ptr(), n)
            ns.sync()
        return made

    torch.cuda.synchronize()
    kept = contexts(64)
    before = free_bytes()
    kept += contexts(256)
    assert before - free_bytes() <= 256 * (64 << 10)
    for ns in kept:
        ns.close()


@pytest.mark.parametrize("dims", [(5, 4, 3), (40, 40, 40), (260, 256, 256)])
@pytest.mark.parametrize("most", [3072, 32 * 3072, 40 * 3072])
def test_one_context_for_many_and_few_points(dims, most):
    """The passes of few tiles and those of many share a context's scratch: one
    to four passes, contexts made for either, used up and down."""
    rng = np.random.default_rng(most)
    cfg = scenes.base_config(kernel_radius=1.0 / max(dims), grid_dim=dims, max_particles=most)
    cells = int(np.prod(dims))
    ns = NeighborSearch((0.0, 0.0, 0.0), [float(np.float32(d)) for d in dims], dims, most)
    for n in (most, 1, most // 2 + 1, 33 * 3072 + 5, 3073, 32 * 3072, 100, most):
        if n > most:
            continue
        pts = np.zeros((n, 4), np.float32)
        pts[:, :3] = rng.random((n, 3)) ** 2
        ref = O.neighbor_search(cfg, pts)
        pos = torch.from_numpy(pts).cuda()
        out = {k: torch.full((m,), -1, dtype=torch.int32, device="cuda")
               for k, m in (("keys", n), ("cell_count", cells), ("cell_offset", cells + 1), ("order", n), ("rank", n))}
        ns.run(pos.data_ptr(), n, *(out[k].data_ptr() for k in ("keys", "cell_count", "cell_offset", "order", "rank")))
        ns.sync()
        for k, v in out.items():
            assert np.array_equal(v.cpu().numpy().view(np.uint32), ref[k]), k
    ns.close()
