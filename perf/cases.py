"""The work that users of this package have it do, as cases that can be timed.

A case is a dict of plain values; `prepare` makes what a program holds before
the call (a simulator with a scene in motion, a search context, a renderer),
`run` is one pass through the package's public calls, `work` the bytes and
operations that the pass cannot do without and `exact` what the pass returns
when its formulas are evaluated in 64 bits with plain torch.

Simulation states come from the scene's own lattice, jittered by the seed and
carried on for some substeps by the bit-exact mode, so the timed step starts
from fluid in motion and the same seed always gives the same bits.  The wall
jitter (a hash of the position's float bits, 1e-4 by default) is off: with it
the last bit of a position would decide where a particle at a wall goes.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "webgpu-fluid-simulation_gb300"))
import pbf_gb300 as pbf  # noqa: E402
from pbf_gb300 import _lib as L, scenes  # noqa: E402
from pbf_gb300.render import reference_camera  # noqa: E402


def listed():
    return [
        # a small interactive scene at the reference's constants: one substep per call, latency and launches count
        dict(name="step_2k_call", kind="step", scene="reference", nx=13, ny=13, nz=13, iterations=5, settle=60,
             fp="fast", graph=False, learned=-1),
        # the dam break of the benchmark: 16,384 particles, volume map, one graph-replayed frame of 2 substeps
        dict(name="step_dam_16k", kind="step", scene="dam", nx=32, ny=16, nz=32, iterations=4, settle=60, fp="fast",
             graph=True, learned=-1),
        # the reference's Cube Drop preset with its GUI options (5 iterations, no volume map): one substep per call
        dict(name="step_cube_drop_69k", kind="step", scene="reference", nx=41, ny=41, nz=41, iterations=5, settle=60,
             fp="fast", graph=False, learned=-1),
        # the reference's Boundary preset (torus volume map) in the mode that is bit-identical with the reference method
        dict(name="step_exact_torus_69k", kind="step", scene="torus", nx=41, ny=41, nz=41, iterations=5, settle=80,
             fp="exact", graph=True, learned=-1),
        # the benchmark's large scene after its impact, plain solve, the launch shape its autotuner picks
        dict(name="step_sphere_1m", kind="step", scene="sphere", nx=128, ny=64, nz=128, iterations=4, settle=190,
             fp="fast", graph=True, learned=-1),
        # the same with the learned start and one plain iteration
        dict(name="step_sphere_1m_learned", kind="step", scene="sphere", nx=128, ny=64, nz=128, iterations=4,
             settle=190, fp="fast", graph=True, learned=1),
        # uneven independent dam breaks, 3 or 4 iterations each, stepped together
        dict(name="batch_16", kind="batch", count=16, n_min=4096, n_max=262144, settle=60),
        # the neighbour search on its own: a small scene's points on the reference's 40^3 grid, odd count
        dict(name="search_5k", kind="search", n=5003, dim=40, dist="uniform"),
        # ... and the benchmark's largest
        dict(name="search_16m", kind="search", n=1 << 24, dim=128, dist="uniform"),
        # neighbour lists in the reference's layout for a cloud of uneven density
        dict(name="lists_200k", kind="lists", n=200003, dim=40, dist="clumps"),
        # a full-HD frame of the screen-space depth and thickness maps
        dict(name="render_1080p_1m", kind="render", n=1 << 20, width=1920, height=1080, filter_size=32),
        # one training epoch of the learned start's network on traced rows held by the host
        dict(name="train_200k", kind="train", rows=200000, batch=8192, epochs=1),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "batch", "search", "search", "lists", "render", "train"])
    if kind == "step":
        scene = rng.choice(["reference", "torus", "dam", "sphere", "sphere"])
        m = _log(rng, 12, 41) if scene in ("reference", "torus") else _log(rng, 16, 96)
        dims = [max(8, int(m * rng.uniform(0.7, 1.1))) for _ in range(3)]
        if scene in ("reference", "torus"):
            dims = [min(d, 41) for d in dims]
        if scene == "dam":
            dims = [min(max(dims[0], 16), 60), min(dims[1], 24), min(max(dims[2], 16), 60)]
        if scene == "sphere":
            dims[1] = min(dims[1], 64)
        learned = 1 if scene == "sphere" and rng.random() < 0.4 else -1
        fp = "exact" if learned < 0 and rng.random() < 0.2 else "fast"
        settle = 2 * (rng.randint(94, 98) if scene == "sphere" else rng.randint(10, 20) if scene == "dam" else rng.randint(20, 40))
        return dict(kind="step", scene=scene, nx=dims[0], ny=dims[1], nz=dims[2], iterations=rng.choice([3, 4, 5]),
                    settle=settle, fp=fp, graph=rng.random() < 0.6, learned=learned)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(3, 16), n_min=_log(rng, 2048, 16384),
                    n_max=_log(rng, 32768, 262144), settle=2 * rng.randint(20, 30))
    if kind == "search":
        return dict(kind="search", n=_log(rng, 4000, 1 << 24), dim=rng.choice([24, 40, 64, 128]),
                    dist=rng.choice(["uniform", "clumps"]))
    if kind == "lists":
        return dict(kind="lists", n=_log(rng, 5000, 400000), dim=rng.choice([32, 40]), dist=rng.choice(["uniform", "clumps"]))
    if kind == "render":
        w = _log(rng, 320, 1920)
        return dict(kind="render", n=_log(rng, 4000, 1 << 20), width=w, height=int(w * rng.uniform(0.5, 0.56)),
                    filter_size=rng.choice([7, 16, 32]))
    return dict(kind="train", rows=_log(rng, 20000, 300000), batch=rng.choice([2048, 8192, 8000]), epochs=1)


# ---- inputs ---------------------------------------------------------------------------
class _DeviceArray:
    """A device buffer of the library, for torch.as_tensor (no copy).  The
    tensor keeps this object, and with it the buffer's owner, alive."""

    def __init__(self, ptr, shape, owner):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(int(ptr), False), shape=tuple(shape), typestr="<f4", version=3)


def _wrap(ptr, shape, owner):
    return torch.as_tensor(_DeviceArray(ptr, shape, owner), device="cuda")


@functools.lru_cache(maxsize=None)
def _field(shapes, res, origin, extent, h, quadrature):
    return scenes.generate_field(list(shapes), res, origin, extent, h, quadrature=quadrature)


def _map_of(args, res=None, quadrature=8):
    fix = lambda v: tuple(float(x) for x in v)  # noqa: E731
    shapes = tuple((int(k), fix(c), fix(s)) for k, c, s in args["shapes"])
    return _field(shapes, tuple(res or args["res"]), fix(args["origin"]), fix(args["extent"]), float(args["h"]), quadrature)


@functools.lru_cache(maxsize=None)
def _torus():
    return scenes.load_cdm_npz("torus")


def _scene(case, seed):
    """(config, particles, volume map or None) of a stepped scene."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    if case["scene"] in ("reference", "torus"):
        cfg = scenes.base_config()
        r = cfg.particle_radius
        d = 2 * r
        top = 0.9 if case["scene"] == "reference" else 0.95
        lo = np.array([0.5 - nx * d / 2, top - ny * d, 0.5 - nz * d / 2])
        if case["scene"] == "torus":  # close above the ring (its top is near y = 0.4)
            lo[1] = 0.36
        else:
            lo[1] = 0.02
        field = _torus() if case["scene"] == "torus" else None
    elif case["scene"] == "dam":
        cfg, _, args = scenes.dam_break_16k_spec()
        r = cfg.particle_radius
        d = 2 * r
        box = (2 * nx * d, 1.25 * max(ny, 16) * d, nz * d)
        cfg.domain_max[:] = box
        lo = np.array([r, r, r])
        half = tuple(b / 2 for b in box)
        field = _map_of(dict(shapes=[(L.SHAPE_BOX_CONTAINER, half, half)], res=(64, 64, 64), origin=(0, 0, 0), extent=box, h=4 * r))
    else:
        cfg, _, args = scenes.sphere_drop_spec(nx=8, ny=8, nz=8)
        r = cfg.particle_radius
        d = 2 * r
        lo = np.array([(3.3 - nx * d) / 2 + r, 0.85 + r, (3.3 - nz * d) / 2 + r])
        field = _map_of(args)
    i = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3)
    pts = np.zeros((nx * ny * nz, 4), np.float32)
    pts[:, :3] = lo + d * i + 0.1 * r * rng.uniform(-1, 1, (len(i), 3))
    cfg.max_particles = len(pts)
    cfg.max_neighbors = 128
    cfg.wall_jitter = 0.0
    cfg.options.iterations = case["iterations"]
    return cfg, pts, field


def _set_field(sim, f):
    if f is not None:
        sim.set_boundary_field(f["res"], f["origin"], f["extent"], f["sdf"], f["vol"])


def _snapshot(sim):
    return sim.positions(), sim.velocities(), sim.copy_field(L.FIELD_ACCELERATION)


def _settled(cfg, pts, field, substeps):
    """The scene after some substeps of the bit-exact mode: x, v and a by id."""
    c = scenes.copy_config(cfg)
    c.fp_mode = L.FP_EXACT
    with pbf.PBF(c) as sim:
        sim.set_particles(pts)
        _set_field(sim, field)
        sim.enable_graph(True)
        sim.step(substeps // int(c.substeps))
        return _snapshot(sim)


def _model():
    """The learned start's network, set by hand so that every run has the same
    (training sums in no fixed order): two units of each layer pass on the
    density error between 0 and 0.04, the others are seeded and go nowhere.
    The slope is what rows traced from the plain solve of this scene give."""
    m = pbf.mlp_init(7)
    p = np.array(m.params)
    w1, b1, w2, b2, w3 = p[:512].reshape(8, 64), p[512:576], p[576:4672].reshape(64, 64), p[4672:4736], p[4736:4800]
    w1[:, :2], w2[:, :2], w2[:2], w3[:] = 0.0, 0.0, 0.0, 0.0
    w1[0, :2], b1[1] = 1.0, -16.0                    # silu(400 f0) and silu(400 f0 - 16) ...
    w2[0, 0], w2[1, 0], w2[0, 1], w2[1, 1] = 1.0, -1.0, 1.0, -1.0
    b2[1], w3[0] = 0.0, -1.0                         # ... their difference, at most 16
    m.params[:] = p.tolist()
    m.feat_mean[:] = [0.0, 0.0, 33.0, 0.25, 0.0, 0.0, 0.0, 0.0]
    m.feat_inv_std[:] = [400.0, 1e4, 0.1, 4.0, 10.0, 1.0, 1.0, 1.0]
    m.lam_scale = 2.5e-3 / 400.0
    return m


def _cloud(n, dist, dim, seed):
    """n float4 points of the unit cube on the GPU: uniform, or 64 clumps."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dist == "uniform":
        xyz = torch.rand((n, 3), generator=g, device="cuda")
    else:
        centres = torch.rand((64, 3), generator=g, device="cuda")
        which = torch.randint(0, 64, (n,), generator=g, device="cuda")
        sigma = 2.0 / dim * max(1.0, n / 64 / 4000) ** (1 / 3)
        xyz = centres[which] + sigma * torch.randn((n, 3), generator=g, device="cuda")
    pts = torch.zeros((n, 4), device="cuda")
    pts[:, :3] = xyz.clamp_(0.0, 1.0 - 2.0 ** -24)
    return pts


def _block(n, seed):
    """n points of a jittered 0.5^3 block under the reference's camera."""
    m = math.ceil(n ** (1 / 3))
    g = torch.Generator(device="cuda").manual_seed(seed)
    i = torch.arange(n, device="cuda")
    pts = torch.zeros((n, 4), device="cuda")
    for a, q in enumerate((i % m, i // m % m, i // (m * m))):
        pts[:, a] = 0.25 + 0.5 / m * (q + 0.2 * (torch.rand(n, generator=g, device="cuda") - 0.5))
    return pts


def _rows(case, seed):
    """Training rows with the ranges of the traced features."""
    n = case["rows"]
    rng = np.random.default_rng(seed)
    f = np.empty((n, 8), np.float32)
    f[:, 0] = 0.03 * rng.standard_normal(n)
    f[:, 1] = -1e-5 * rng.random(n)
    f[:, 2] = rng.integers(12, 50, n)
    f[:, 3] = rng.gamma(4.0, 0.05, n)
    f[:, 4] = 0.01 * rng.standard_normal(n)
    f[:, 5] = np.where(rng.random(n) < 0.9, 2.0, rng.random(n))
    f[:, 6] = np.where(f[:, 5] < 1.0, 3.0 * rng.random(n), 0.0)
    f[:, 7] = rng.integers(0, 2, n)
    t = (-3e-5 * np.maximum(f[:, 0] + 0.3 * f[:, 4] + 0.002 * f[:, 6], 0.0) * (0.8 + 0.01 * f[:, 2])).astype(np.float32)
    return f, t


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        cfg, pts, field = _scene(case, seed)
        state = _settled(cfg, pts, field, case["settle"])
        if case["fp"] == "exact":
            cfg.fp_mode = L.FP_EXACT
        sim = pbf.PBF(cfg)
        if case["scene"] == "sphere" and case["fp"] == "fast":
            sim.set_launch(block=128, ctas_per_sm=0, cell_ratio=0.5, build=L.BUILD_THREAD)
        sim.set_state(*state)
        _set_field(sim, field)
        if case["learned"] >= 0:
            sim.set_learned(_model(), iterations=case["learned"], fallback_bound=0.2)
        sim.enable_graph(case["graph"])
        sim.synchronize()
        return dict(case=case, sim=sim, position=_wrap(sim.position, (sim.particleCount, 4), sim))
    if kind == "batch":
        cfg, scs, fields = scenes.batch_scenes_spec(case["count"], case["n_min"], case["n_max"], seed=3, field_res=(32, 32, 32))
        cfg.wall_jitter = 0.0
        cfg.max_neighbors = 128
        scs = [dict(s, field=_map_of(f, quadrature=4), positions=scenes.jitter(s["positions"], 0.05 * cfg.particle_radius, 64 * seed + q))
               for q, (s, f) in enumerate(zip(scs, fields))]
        c = scenes.copy_config(cfg)
        c.fp_mode = L.FP_EXACT
        with pbf.PBFBatch(c, scs) as sim:
            sim.step(case["settle"] // int(c.substeps))
            state = _snapshot(sim)
        at = 0
        for s in scs:
            n = len(s["positions"])
            s["positions"] = state[0][at:at + n]
            at += n
        sim = pbf.PBFBatch(cfg, scs)
        sim.set_velocities(state[1])
        sim.set_accelerations(state[2])
        sim.enable_graph(True)
        sim.synchronize()
        return dict(case=case, sim=sim, scenes=scs, position=_wrap(sim.position, (sim.particleCount, 4), sim))
    if kind in ("search", "lists"):
        n, dim = case["n"], case["dim"]
        pts = _cloud(n, case["dist"], dim, seed)
        ns = pbf.NeighborSearch((0.0, 0.0, 0.0), (dim,) * 3, (dim,) * 3, n)
        new = lambda k: torch.zeros(k, dtype=torch.int32, device="cuda")  # noqa: E731
        out = dict(keys=new(n), cell_count=new(dim ** 3), cell_offset=new(dim ** 3 + 1), order=new(n), rank=new(n))
        torch.cuda.synchronize()
        s = dict(case=case, ns=ns, pts=pts, out=out)
        if kind == "lists":
            s["offset"] = new(n + 1)
            s["list"] = new(96 * n)  # room for the densest cloud
            torch.cuda.synchronize()
        return s
    if kind == "render":
        fluid = pbf.FilteredParticleFluid(case["width"], case["height"])
        fluid.setConfig(filterSize=case["filter_size"])
        fluid.set_camera(reference_camera(case["width"], case["height"]))
        pts = _block(case["n"], seed)
        torch.cuda.synchronize()
        w, h = case["width"], case["height"]
        return dict(case=case, fluid=fluid, pts=pts, depth=_wrap(fluid.device_map(L.RENDER_DEPTH), (h, w), fluid),
                    volume=_wrap(fluid.device_map(L.RENDER_VOLUME), (h // 2, w // 2), fluid))
    f, t = _rows(case, seed)
    return dict(case=case, feat=f, target=t, seed=seed)


# ---- one pass ---------------------------------------------------------------------------
def _search(s):
    o = s["out"]
    s["ns"].run(s["pts"].data_ptr(), len(s["pts"]), o["keys"].data_ptr(), o["cell_count"].data_ptr(),
                o["cell_offset"].data_ptr(), o["order"].data_ptr(), o["rank"].data_ptr())


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("step", "batch"):
        sim = s["sim"]
        if case.get("graph", True):
            sim.step(1)
        else:
            sim.run()
        v = _wrap(L.load().pbf_velocity_device(sim._h), s["position"].shape, sim)
        return dict(x=s["position"][:, :3], density=s["position"][:, 3], v=v[:, :3])
    if kind == "search":
        _search(s)
        return s["out"]
    if kind == "lists":
        _search(s)
        s["ns"].lists(s["pts"].data_ptr(), len(s["pts"]), 1.0 / case["dim"], s["offset"].data_ptr(), s["list"].data_ptr(),
                      len(s["list"]))
        return dict(offset=s["offset"], list=s["list"])
    if kind == "render":
        s["fluid"].render(s["pts"].data_ptr(), len(s["pts"]))
        return dict(depth=s["depth"], volume=s["volume"])
    m = pbf.mlp_init(s["seed"])
    pbf.mlp_fit_normalization(m, s["feat"], s["target"])
    loss = pbf.mlp_train(m, s["feat"], s["target"], epochs=case["epochs"], batch=case["batch"], lr=3e-3, seed=s["seed"])
    return dict(params=pbf.mlp_params(m), loss=loss)


# ---- what a pass cannot do without ---------------------------------------------------------
def _particles(case):
    if case["kind"] == "batch":  # the mean of the log-uniform counts
        a, b = case["n_min"], case["n_max"]
        return int(case["count"] * (b - a) / math.log(b / a))
    return case["nx"] * case["ny"] * case["nz"]


def work(case):
    kind = case["kind"]
    if kind in ("step", "batch"):
        n = _particles(case)
        learned = case.get("learned", -1)
        iters = case.get("iterations", 4) if learned < 0 else learned + 0.5
        sub = 2 if kind == "batch" or (case["graph"] and case["scene"] in ("dam", "sphere")) else 1
        pairs = 34.0 * n * sub  # neighbours, itself included
        # distance test, the two sums of an iteration, density, vorticity and cohesion, viscosity and curvature
        flops = pairs * (8 + iters * (27 + 18) + 12 + 60 + 40) + (9e3 * n * sub if learned >= 0 else 0)
        # x, v and a in and out, and the by-id positions (with density) and velocities
        return dict(bytes=n * (6 * 16 + 2 * 16), flops=flops)
    if kind == "search":
        return dict(bytes=case["n"] * (16 + 4 + 4 + 4) + 8 * case["dim"] ** 3, flops=9.0 * case["n"])
    if kind == "lists":  # about 4.2 points a cell volume where the cloud is uniform, more in clumps
        pairs = case["n"] * max(8.0, 4.2 * case["n"] / case["dim"] ** 3)
        return dict(bytes=case["n"] * (16 + 4) + 4 * pairs, flops=8 * pairs)
    if kind == "render":
        px = case["width"] * case["height"]
        side = 0.02 / 2.3 * case["height"] / 0.93  # pixels across a sprite of the fluid block
        frags = case["n"] * (0.785 * side ** 2 + side ** 2)
        return dict(bytes=16 * case["n"] + px * 4 + px, flops=8.0 * frags + 64.0 * px)
    rows = case["rows"] // case["batch"] * case["batch"] * case["epochs"]
    return dict(bytes=36.0 * case["rows"] + 8 * 4801, flops=6.0 * 4672 * rows)


# ---- 64 bits ------------------------------------------------------------------------------
def _f(v):
    return float(np.float32(v))


def _pairs(x, h, lo, hi):
    """(i, j) of every pair within h, itself included, and how many each has."""
    n = len(x)
    dim = [max(1, int((hi[a] - lo[a]) / h)) for a in range(3)]
    cell = torch.stack([((x[:, a] - lo[a]) * (dim[a] / (hi[a] - lo[a]))).floor().long().clamp(0, dim[a] - 1) for a in range(3)], 1)
    key = (cell[:, 0] * dim[1] + cell[:, 1]) * dim[2] + cell[:, 2]
    order = torch.argsort(key)
    start = torch.zeros(dim[0] * dim[1] * dim[2] + 1, dtype=torch.long, device=x.device)
    start[1:] = torch.bincount(key, minlength=len(start) - 1).cumsum(0)
    got = []
    zlo, zhi = (cell[:, 2] - 1).clamp(min=0), (cell[:, 2] + 1).clamp(max=dim[2] - 1)
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            cx, cy = cell[:, 0] + dx, cell[:, 1] + dy
            ok = (cx >= 0) & (cx < dim[0]) & (cy >= 0) & (cy < dim[1])
            row = (cx.clamp(0, dim[0] - 1) * dim[1] + cy.clamp(0, dim[1] - 1)) * dim[2]
            b, e = start[row + zlo], start[row + zhi + 1]
            cnt = torch.where(ok, e - b, 0)
            first = cnt.cumsum(0) - cnt
            i = torch.repeat_interleave(torch.arange(n, device=x.device), cnt)
            j = order[torch.arange(len(i), device=x.device) - first[i] + b[i]]
            keep = ((x[i] - x[j]) ** 2).sum(1) <= h * h
            got.append((i[keep], j[keep]))
    return torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])


class _Map64:
    """Cubic 32-node interpolation of a volume map (.cdm node layout)."""

    def __init__(self, f, quirk):
        self.res = [int(v) for v in f["res"]]
        self.origin = [_f(v) for v in f["origin"]]
        self.extent = [_f(v) for v in f["extent"]]
        self.sdf, self.vol = (torch.as_tensor(np.asarray(f[k], np.float32), device="cuda").double() for k in ("sdf", "vol"))
        self.quirk = quirk

    def sample(self, x, r, h):
        """(x_b, V_b) of each point."""
        nx, ny, nz = self.res
        u = [(x[:, a] - self.origin[a]) * (self.res[a] / self.extent[a]) for a in range(3)]
        c = [u[a].floor().long().clamp(0, self.res[a] - 1) for a in range(3)]
        s = [2.0 * (u[a] - u[a].floor()) - 1.0 for a in range(3)]
        i, j, k = c
        nc = (nx + 1) * (ny + 1) * (nz + 1)
        ney0 = nc + 2 * nx * (ny + 1) * (nz + 1)
        nez0 = ney0 + (nx + 1) * 2 * ny * (nz + 1)
        idx, fn, grad = [], [], []
        r2 = s[0] ** 2 + s[1] ** 2 + s[2] ** 2
        for m in range(8):
            b = [m & 1, m >> 1 & 1, m >> 2 & 1]
            idx.append(((k + b[2]) * (ny + 1) + j + b[1]) * (nx + 1) + i + b[0])
            g = [2 * v - 1 for v in b]
            t = [1 + g[a] * s[a] for a in range(3)]
            p, q = t[0] * t[1] * t[2], 9 * r2 - 19
            fn.append(p * q / 64)
            grad.append([(g[a] * t[(a + 1) % 3] * t[(a + 2) % 3] * q + 18 * p * s[a]) / 64 for a in range(3)])
        for ax in range(3):
            av, aw = (ax + 1) % 3, (ax + 2) % 3
            for m in range(8):
                e, bw, bv = m & 1, m >> 1 & 1, m >> 2 & 1
                if ax == 0:    # v = y, w = z
                    idx.append(nc + ((k + bw) * (ny + 1) + j + bv) * (2 * nx) + 2 * i + e)
                elif ax == 1:  # v = z, w = x
                    idx.append(ney0 + ((i + bw) * (nz + 1) + k + bv) * (2 * ny) + 2 * j + e)
                else:          # v = x, w = y
                    idx.append(nez0 + ((j + bw) * (nx + 1) + i + bv) * (2 * nz) + 2 * k + e)
                sg, gv, gw = 2 * e - 1, 2 * bv - 1, 2 * bw - 1
                q, lin = 1 - s[ax] ** 2, 1 + 3 * sg * s[ax]
                tv, tw = 1 + gv * s[av], 1 + gw * s[aw]
                fn.append(9 / 64 * q * lin * tv * tw)
                d = [None] * 3
                d[ax] = 9 / 64 * tv * tw * (-2 * s[ax] * lin + 3 * sg * q)
                d[av], d[aw] = 9 / 64 * q * lin * gv * tw, 9 / 64 * q * lin * tv * gw
                grad.append(d)
        dist = sum(f * self.sdf[n] for f, n in zip(fn, idx))
        g = torch.stack([sum(d[a] * self.sdf[n] for d, n in zip(grad, idx)) * (2 * self.res[a] / self.extent[a]) for a in range(3)], 1)
        if self.quirk:
            for a, b in ((11, 10), (15, 14), (25, 24), (27, 26), (29, 28), (31, 30)):
                idx[a] = idx[b]
        vol = sum(f * self.vol[n] for f, n in zip(fn, idx))
        gl = g.norm(dim=1, keepdim=True)
        on = (dist > 0) & (dist < h) & (gl[:, 0] > 1e-9) & (vol > 0)
        xb = x - torch.clamp(dist + 0.5 * r, min=2 * r)[:, None] * g / gl.clamp(min=1e-30)
        return torch.where(on[:, None], xb, torch.zeros_like(xb)), torch.where(on, vol, torch.zeros_like(vol))


class _Fluid64:
    """Substeps of the method (time integration, search, solver iterations,
    density, vorticity, XSPH and surface tension) in 64 bits."""

    def __init__(self, cfg, lo, hi, iterations, field, state, model=None, learned=0):
        self.c, self.iterations, self.model, self.learned = cfg, iterations, model, learned
        self.h, self.r, self.rho0, self.dt = _f(cfg.kernel_radius), _f(cfg.particle_radius), _f(cfg.rest_density), _f(cfg.time_step)
        self.V = 0.9 * (2 * self.r) ** 3
        self.m = self.V * self.rho0
        self.lo, self.hi = [_f(v) for v in lo], [_f(v) for v in hi]
        self.tlo, self.thi = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (self.lo, self.hi))
        self.map = _Map64(field, cfg.volume_quirk) if field is not None else None
        self.x, self.v, self.a = (torch.as_tensor(q[:, :3], device="cuda").double() for q in state)
        self.rho = torch.zeros_like(self.x[:, 0])

    def clamp(self, x):
        return torch.maximum(torch.minimum(x, self.thi), self.tlo)

    def sum(self, w):
        out = torch.zeros((len(self.x),) + w.shape[1:], dtype=torch.float64, device="cuda")
        return out.index_add_(0, self.i, w)

    def geometry(self, d):
        r = d.norm(dim=1)
        return r, torch.where(r > 0, 1 / r.clamp(min=1e-300), torch.zeros_like(r))

    def poly6(self, r):
        return 315 / (64 * math.pi * self.h ** 9) * torch.clamp(self.h ** 2 - r ** 2, min=0) ** 3

    def spiky(self, d, r, ir):
        return (-45 / (math.pi * self.h ** 6) * torch.clamp(self.h - r, min=0) ** 2 * ir)[:, None] * d

    def boundary(self, x):
        if self.map is None:
            return torch.zeros_like(x), torch.zeros_like(x[:, 0])
        out = [self.map.sample(q, self.r, self.h) for q in x.split(1 << 18)]
        return torch.cat([q[0] for q in out]), torch.cat([q[1] for q in out])

    def multipliers(self, x, xb, vb):
        d = x[self.i] - x[self.j]
        r, ir = self.geometry(d)
        g = self.spiky(d, r, ir)
        grad, sum2, dens = self.V * self.sum(g), self.V ** 2 * self.sum((g * g).sum(1)), self.V * self.sum(self.poly6(r))
        rb, irb = self.geometry(x - xb)
        grad = grad + vb[:, None] * self.spiky(x - xb, rb, irb)
        dens = dens + vb * self.poly6(rb)
        return -torch.clamp(dens - 1, min=0) / ((grad * grad).sum(1) + sum2 + _f(self.c.lambda_eps))

    def project(self, x, lam, xb, vb):
        d = x[self.i] - x[self.j]
        r, ir = self.geometry(d)
        pu = self.V * self.sum((lam[self.i] + lam[self.j])[:, None] * self.spiky(d, r, ir))
        rb, irb = self.geometry(x - xb)
        pu = pu + (vb * lam)[:, None] * self.spiky(x - xb, rb, irb)
        return self.clamp(x + 0.5 * pu)

    def network(self, x, xb, vb):  # (of the features, only the density error has weight: _model)
        r = self.geometry(x[self.i] - x[self.j])[0]
        rb = self.geometry(x - xb)[0]
        f = torch.zeros((len(x), 8), dtype=torch.float64, device="cuda")
        f[:, 0] = self.V * self.sum(self.poly6(r)) + vb * self.poly6(rb) - 1
        t = lambda v: torch.tensor(np.array(v, np.float32), device="cuda").double()  # noqa: E731
        p, z = t(self.model.params), (f - t(self.model.feat_mean)) * t(self.model.feat_inv_std)
        z = torch.nn.functional.silu(z @ p[:512].view(8, 64) + p[512:576])
        z = torch.nn.functional.silu(z @ p[576:4672].view(64, 64) + p[4672:4736])
        return (z @ p[4736:4800] + p[4800]) * _f(self.model.lam_scale)

    def substep(self):
        o = self.c.options
        g = torch.tensor([0.0, -_f(o.gravity), 0.0], dtype=torch.float64, device="cuda")
        x0 = self.x
        x = self.clamp(x0 + self.dt * (self.v + self.dt * (g + self.a)))
        self.i, self.j = _pairs(x, self.h, self.lo, self.hi)
        rounds = self.iterations
        if self.model is not None:
            xb, vb = self.boundary(x)
            x = self.project(x, self.network(x, xb, vb), xb, vb)
            rounds = self.learned
        for _ in range(rounds):
            xb, vb = self.boundary(x)
            x = self.project(x, self.multipliers(x, xb, vb), xb, vb)
        i, j = self.i, self.j
        d = x[i] - x[j]
        r, ir = self.geometry(d)
        w, gw = self.poly6(r), self.spiky(d, r, ir)
        rho = self.m * self.sum(w)
        v = (x - x0) / self.dt
        vd = v[j] - v[i]
        om = self.sum((self.m / rho[j])[:, None] * torch.linalg.cross(vd, gw))
        nm = self.h * self.sum((self.m / rho[j])[:, None] * gw)
        ol = om.norm(dim=1)
        vu = self.sum((w / rho[j])[:, None] * vd)
        eta = self.sum((ol[j] / rho[j])[:, None] * gw)
        t = torch.clamp(self.h - r, min=0) ** 3 * r ** 3
        spline = torch.where(r > 0.5 * self.h, t, 2 * t - self.h ** 6 / 64) * (r <= self.h)
        coh = self.m * (32 / (math.pi * self.h ** 9) * spline * ir)[:, None] * d
        ten = -self.sum((2 * self.rho0 / (rho[i] + rho[j]))[:, None] * (coh + nm[i] - nm[j]))
        el = eta.norm(dim=1, keepdim=True)
        en = torch.where(el > 0, eta / el.clamp(min=1e-300), torch.zeros_like(eta))
        self.a = (_f(o.xsph) / self.dt * self.m * vu + _f(o.vorticity) * torch.linalg.cross(en, om)
                  + _f(o.surface_tension) * ten)
        self.x, self.v, self.rho = x, v, rho


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        cfg, pts, field = _scene(case, seed)
        state = _settled(cfg, pts, field, case["settle"])
        model = _model() if case["learned"] >= 0 else None
        parts = [_Fluid64(cfg, cfg.domain_min, cfg.domain_max, case["iterations"], field, state, model, case["learned"])]
        substeps = int(cfg.substeps) if case["graph"] else 1
    elif kind == "batch":
        s = prepare(case, seed)
        state = _snapshot(s["sim"])
        parts, at, cfg = [], 0, s["sim"].config
        for sc in s["scenes"]:
            mine = [q[at:at + len(sc["positions"])] for q in state]
            parts.append(_Fluid64(cfg, sc["domain_min"], sc["domain_max"], sc["iterations"], sc["field"], mine))
            at += len(sc["positions"])
        substeps = int(cfg.substeps)
    else:
        # whole numbers (search, lists); coverage of pixels decided in 32 bits (render); sums in no fixed order (train)
        return None
    for p in parts:
        for _ in range(substeps):
            p.substep()
    return dict(x=torch.cat([p.x for p in parts]), density=torch.cat([p.rho for p in parts]), v=torch.cat([p.v for p in parts]))
