"""Neighbour lists whose total does not fit 32 bits: every point of one crowd is
a neighbour of all, so n points have n^2 entries."""
import pytest

from pbf_gb300 import _lib as L
from pbf_gb300 import NeighborSearch

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,capacity", [(300, 90000), (300, 89999), (65535, 1000), (65536, 0), (65536, 1000),
                                        (65537, 200000), (70001, 1000)])
def test_totals_above_32_bits_are_refused(n, capacity):
    pos = torch.full((n, 4), 0.5, device="cuda")
    off = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
    lst = torch.full((capacity + 8,), -1, dtype=torch.int32, device="cuda")
    ns = NeighborSearch((0.0, 0.0, 0.0), (10.0,) * 3, (10,) * 3, n)
    ns.run(pos.data_ptr(), n)
    rc, total = ns.lists(pos.data_ptr(), n, 0.1, off.data_ptr(), lst.data_ptr(), capacity)
    assert total == min(n * n, 0xFFFFFFFF)
    if n * n <= capacity:
        assert rc == L.PBF_OK
        want = torch.arange(n, dtype=torch.int32, device="cuda").repeat(n)
        assert torch.equal(lst[: n * n], want)
        assert bool((lst[n * n:] == -1).all())
    else:
        assert rc == L.PBF_ECAPACITY
        assert bool((lst == -1).all())
    ns.sync()
    ns.close()
