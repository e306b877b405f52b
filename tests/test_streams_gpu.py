"""Kernels that are set up beside the end of the stream's previous one: handles,
searches and renderers side by side on streams of their own, and between a
caller's kernels on the caller's stream; and the passes with several lanes a
slot where the walls jitter."""
import numpy as np
import pytest

from pbf_gb300 import _lib as L
from pbf_gb300 import PBF, NeighborSearch, scenes
from pbf_gb300 import render as Rd

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FIELDS = (L.FIELD_POSITION, L.FIELD_VELOCITY, L.FIELD_ACCELERATION, L.FIELD_PREDICTED)


class DeviceArray:
    def __init__(self, ptr, shape):
        self.__cuda_array_interface__ = dict(data=(int(ptr), False), shape=tuple(shape), typestr="<f4", version=3)


def simulator(fp, substeps, graph, iterations, stream=None):
    sc = scenes.reference_scene("boundary_small")
    cfg = scenes.copy_config(sc.config)
    cfg.fp_mode, cfg.substeps = fp, substeps
    cfg.options.iterations = iterations
    cfg.stream = stream.cuda_stream if stream is not None else None
    sim = PBF(cfg)
    sim.set_particles(sc.particles)
    f = sc.field
    sim.set_boundary_field(f["res"], f["origin"], f["extent"], f["sdf"], f["vol"])
    sim.enable_graph(graph)
    return sim


def fields(sim):
    sim.synchronize()
    return [np.asarray(sim.copy_field(f)).view(np.uint32) for f in FIELDS]


def test_side_by_side():
    """Three simulators, a search and a renderer in turn, none waited for, give
    what each gives alone."""
    args = [(L.FP_FAST, 2, True, 4), (L.FP_EXACT, 1, True, 3), (L.FP_FAST, 1, False, 5)]
    alone = []
    for a in args:
        with simulator(*a) as sim:
            sim.step(12)
            alone.append(fields(sim))
    n, dim = 20011, 40
    g = torch.Generator(device="cuda").manual_seed(2)
    pos = torch.rand((n, 4), generator=g, device="cuda")
    out = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3)]
    ns = NeighborSearch((0.0,) * 3, (float(dim),) * 3, (dim,) * 3, n)
    search = lambda: ns.run(pos.data_ptr(), n, d_keys=out[0].data_ptr(), d_order=out[1].data_ptr(),
                            d_rank=out[2].data_ptr())
    W, H = 320, 200
    r = Rd.FilteredParticleFluid(W, H)
    r.set_camera(Rd.reference_camera(W, H))
    torch.cuda.synchronize()
    search()
    ns.sync()
    want = [o.clone() for o in out]
    r.render(pos.data_ptr(), n)
    depth, volume = r.depth().copy(), r.volume().copy()
    for o in out:
        o.zero_()
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    sims = [simulator(*a) for a in args]
    for k in range(12):
        for sim in sims:
            sim.step(1)
        search()
        if k % 4 == 0:
            r.render(pos.data_ptr(), n, stream=stream.cuda_stream)
    for sim, w in zip(sims, alone):
        for a, b in zip(fields(sim), w):
            assert np.array_equal(a, b)
        sim.close()
    ns.sync()
    for a, b in zip(out, want):
        assert torch.equal(a, b)
    assert np.array_equal(r.depth(), depth) and np.array_equal(r.volume(), volume)
    ns.close()
    r.close()


def test_search_between_the_callers_kernels():
    """The caller's kernels on the same stream make the points just before each
    search, read its results just after and change the points again."""
    n, dim, rounds = 5003, 24, 30
    stream = torch.cuda.Stream()
    ns = NeighborSearch((0.0,) * 3, (float(dim),) * 3, (dim,) * 3, n, stream=stream.cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(5)
    base = torch.rand((n, 4), generator=g, device="cuda")
    pos, keys = torch.empty_like(base), torch.zeros(n, dtype=torch.int32, device="cuda")
    order, rank = torch.zeros_like(keys), torch.zeros_like(keys)
    got = torch.zeros((rounds, 3, n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        for k in range(rounds):
            torch.remainder(base + k / 37.0, 1.0, out=pos)
            ns.run(pos.data_ptr(), n, d_keys=keys.data_ptr(), d_order=order.data_ptr(), d_rank=rank.data_ptr())
            got[k, 0], got[k, 1], got[k, 2] = keys, order, rank
    stream.synchronize()
    for k in range(rounds):
        torch.remainder(base + k / 37.0, 1.0, out=pos)
        torch.cuda.synchronize()
        ns.run(pos.data_ptr(), n, d_keys=keys.data_ptr(), d_order=order.data_ptr(), d_rank=rank.data_ptr())
        ns.sync()
        assert torch.equal(got[k], torch.stack([keys, order, rank])), k
    ns.close()


@pytest.mark.parametrize("graph", [False, True])
def test_step_between_the_callers_kernels(graph):
    """The caller's kernel reads the positions right after each frame, with the
    next frame queued behind it."""
    stream = torch.cuda.Stream()
    frames = 10
    with simulator(L.FP_FAST, 1, graph, 4, stream) as sim:
        pos = torch.as_tensor(DeviceArray(sim.position, (sim.particleCount, 4)), device="cuda")
        got = torch.zeros((frames,) + tuple(pos.shape), device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            for k in range(frames):
                sim.step(1)
                got[k].copy_(pos)
        stream.synchronize()
    with simulator(L.FP_FAST, 1, False, 4) as sim:
        pos = torch.as_tensor(DeviceArray(sim.position, (sim.particleCount, 4)), device="cuda")
        for k in range(frames):
            sim.step(1)
            sim.synchronize()
            assert torch.equal(got[k].view(torch.int32), pos.view(torch.int32)), k


@pytest.mark.parametrize("fp,n", [(L.FP_EXACT, 2000), (L.FP_EXACT, 20000), (L.FP_FAST, 2000), (L.FP_FAST, 6000)])
def test_lanes_at_jittering_walls(fp, n):
    """Particles pressed against all six walls: several lanes a slot against one
    (persistent grids), the hash jitter on."""
    rng = np.random.default_rng(n)
    cfg = scenes.base_config(fp_mode=fp, max_particles=n, max_neighbors=1024)
    assert cfg.wall_jitter > 0
    pts = np.zeros((n, 4), np.float32)
    pts[:, :3] = 0.02 + 0.96 * rng.random((n, 3))
    axis, side = rng.integers(0, 3, n), rng.integers(0, 2, n)
    pts[np.arange(n), axis] = np.where(side == 0, 0.001 * rng.random(n), 1.0 - 0.001 * rng.random(n))
    vel = np.zeros((n, 4), np.float32)
    vel[np.arange(n), axis] = np.where(side == 0, -2.0, 2.0)
    out = []
    for ctas in (0, 4):
        with PBF(cfg) as sim:
            sim.set_particles(pts)
            sim.set_velocities(vel)
            sim.set_launch(ctas_per_sm=ctas)
            sim.step(3)
            out.append(fields(sim))
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    x = out[0][0].view(np.float32)[:, :3]
    assert ((x < 2e-4) | (x > 1 - 2e-4)).any(axis=1).mean() > 0.3
