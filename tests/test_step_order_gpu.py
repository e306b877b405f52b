"""The substep's sort with the state moved along, and the buffers that a
substep hands to the next one: cells around the size where the block sort
takes over, and single substeps mixed with graph replays."""
import numpy as np
import pytest

from oracle import oracle as O
from pbf_gb300 import _lib as L
from pbf_gb300 import PBF, scenes

pytestmark = pytest.mark.gpu

FIELDS = (L.FIELD_POSITION, L.FIELD_VELOCITY, L.FIELD_ACCELERATION, L.FIELD_PREDICTED, L.FIELD_NEIGHBOR_COUNT)


@pytest.mark.parametrize("n,build", [(1023, L.BUILD_THREAD), (1025, L.BUILD_THREAD), (1500, L.BUILD_THREAD),
                                     (1500, L.BUILD_CELLBLOCK_MASK)])
def test_crowded_cell_bitexact(n, build):
    """n particles in one cell (its particles sorted by the block radix path
    above 1,024) beside a loose cloud: one exact substep, then the order."""
    rng = np.random.default_rng(n)
    cfg = scenes.base_config(fp_mode=L.FP_EXACT, max_particles=n + 300, max_neighbors=2048)
    cfg.options.iterations = 3
    pts = np.zeros((n + 300, 4), np.float32)
    pts[:n, :3] = 0.5 + 0.004 + 0.016 * rng.random((n, 3))
    pts[n:, :3] = 0.3 + 0.4 * rng.random((300, 3))
    pts = pts[rng.permutation(n + 300)]
    orc = O.Oracle(cfg, 32)
    orc.set_particles(pts)
    orc.substep(1)
    with PBF(cfg) as sim:
        sim.set_particles(pts)
        sim.set_launch(build=build)
        sim.run()
        for f in FIELDS:
            ref = orc.field(f)
            got = sim.copy_field(f)
            assert np.array_equal(got, ref.astype(got.dtype)), f
        order = sim.search_state("order")
        keys = sim.search_state("keys")
        assert np.array_equal(order, np.lexsort([np.arange(n + 300), keys]).astype(np.uint32))
        count = sim.search_state("cell_count", cells=sim.scene_info(0)["cells"])
        assert np.array_equal(count, np.bincount(keys, minlength=len(count)))


@pytest.mark.parametrize("fp", [L.FP_EXACT, L.FP_FAST])
@pytest.mark.parametrize("substeps", [1, 2])
def test_single_substeps_between_graph_frames(fp, substeps):
    """run() between graph-replayed frames leaves the other state buffers
    current: the same result as stepping eagerly throughout."""
    sc = scenes.reference_scene("cube_small")
    cfg = scenes.copy_config(sc.config)
    cfg.fp_mode, cfg.substeps = fp, substeps
    out = []
    for graph in (False, True):
        with PBF(cfg) as sim:
            sim.set_particles(sc.particles)
            sim.enable_graph(graph)
            sim.step(2)
            sim.run()
            sim.step(3)
            sim.run()
            sim.run()
            sim.step(2)
            sim.synchronize()
            out.append([sim.copy_field(f) for f in FIELDS])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
