"""Neighbour lists of the stand-alone search at the edges of their kernels:
partial warps, runs of more than 32 candidates, lists longer than the rows a
warp stages in shared memory, and a capacity that is one entry short."""
import numpy as np
import pytest

from oracle import oracle as O
from pbf_gb300 import _lib as L
from pbf_gb300 import NeighborSearch, scenes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def search(cfg, pts, capacity):
    n = len(pts)
    dims, _ = O.grid_dims(cfg)
    inv = [float(np.float32(float(dims[a]) / (cfg.domain_max[a] - cfg.domain_min[a]))) for a in range(3)]
    ns = NeighborSearch(list(cfg.domain_min), inv, list(dims), n)
    pos = torch.from_numpy(pts).cuda()
    off = torch.full((n + 1,), -1, dtype=torch.int32, device="cuda")
    lst = torch.full((capacity + 8,), -1, dtype=torch.int32, device="cuda")
    ns.run(pos.data_ptr(), n)
    rc, total = ns.lists(pos.data_ptr(), n, cfg.kernel_radius, off.data_ptr(), lst.data_ptr(), capacity)
    ns.close()
    return rc, total, off.cpu().numpy().view(np.uint32), lst.cpu().numpy().view(np.uint32)


@pytest.mark.parametrize("n,spread", [(1, 1.0), (31, 0.1), (33, 0.1), (257, 0.08), (700, 0.03), (5003, 0.2)])
def test_lists_at_the_edges(n, spread):
    rng = np.random.default_rng(n)
    pts = np.zeros((n, 4), np.float32)
    pts[:, :3] = 0.45 + spread * rng.random((n, 3))
    cfg = scenes.base_config(max_particles=n)
    ref = O.neighbor_search(cfg, pts, lists=True, capacity=n * min(n, 1024))
    want = len(ref["nbr_list"])
    rc, total, off, lst = search(cfg, pts, want)
    assert rc == 0 and total == want
    assert np.array_equal(off, ref["nbr_offset"])
    assert np.array_equal(lst[:want], ref["nbr_list"])
    assert (lst[want:] == 0xffffffff).all()
    rc, total, off, lst = search(cfg, pts, want - 1)  # one short: refused, nothing written
    assert rc == L.PBF_ECAPACITY and total == want
    assert np.array_equal(off, ref["nbr_offset"])
    assert (lst == 0xffffffff).all()


@pytest.mark.parametrize("n", [1, 3072, 3073, 32 * 3072, 32 * 3072 + 1])
@pytest.mark.parametrize("dims", [(5, 4, 3), (40, 40, 40), (100, 70, 120)])
def test_search_at_the_tile_edges(n, dims):
    """One to four radix passes at the edges of a tile and of the range that
    sorts from the tiles' counts directly; a second search on the same context
    finds its scratch cleared."""
    rng = np.random.default_rng(n)
    cfg = scenes.base_config(kernel_radius=1.0 / max(dims), grid_dim=dims, max_particles=n)
    ns = None
    for _ in range(2):
        pts = np.zeros((n, 4), np.float32)
        pts[:, :3] = rng.random((n, 3)) ** 2
        ref = O.neighbor_search(cfg, pts)
        cells = int(np.prod(dims))
        if ns is None:
            ns = NeighborSearch((0.0, 0.0, 0.0), [float(np.float32(d)) for d in dims], dims, n)
        pos = torch.from_numpy(pts).cuda()
        out = {k: torch.full((m,), -1, dtype=torch.int32, device="cuda")
               for k, m in (("keys", n), ("cell_count", cells), ("cell_offset", cells + 1), ("order", n), ("rank", n))}
        ns.run(pos.data_ptr(), n, *(out[k].data_ptr() for k in ("keys", "cell_count", "cell_offset", "order", "rank")))
        ns.sync()
        for k, v in out.items():
            assert np.array_equal(v.cpu().numpy().view(np.uint32), ref[k]), k
    ns.close()
