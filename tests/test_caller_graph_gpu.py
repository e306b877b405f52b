"""Substeps that a caller records into a CUDA graph of its own, on its own
stream: dropped, replayed, and mixed with eager steps and with the handle's
captured frames, always the same bits as plain stepping."""
import numpy as np
import pytest

from pbf_gb300 import _lib as L
from pbf_gb300 import PBF, PBFBatch, mlp_init, scenes

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FIELDS = (L.FIELD_POSITION, L.FIELD_VELOCITY, L.FIELD_ACCELERATION, L.FIELD_PREDICTED, L.FIELD_NEIGHBOR_COUNT)


def simulator(fp, substeps, stream, iterations=4):
    sc = scenes.reference_scene("cube_small")
    cfg = scenes.copy_config(sc.config)
    cfg.fp_mode, cfg.substeps = fp, substeps
    cfg.options.iterations = iterations
    cfg.stream = stream.cuda_stream if stream is not None else None
    sim = PBF(cfg)
    sim.set_particles(sc.particles)
    return sim


def recorded(stream, call):
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=stream, capture_error_mode="thread_local"):
        call()
    return g


def replay(stream, graph):
    with torch.cuda.stream(stream):
        graph.replay()


def state(sim):
    sim.synchronize()
    cells = sim.scene_info(0)["cells"]
    return [np.asarray(sim.copy_field(f)) for f in FIELDS] + [sim.search_state("order"),
                                                             sim.search_state("cell_count", cells=cells)]


def same(a, b):
    assert len(a) == len(b)
    for x, y in zip(a, b):
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32))


def plain(fp, substeps, frames, iterations=4):
    with simulator(fp, substeps, None, iterations) as sim:
        sim.step(frames)
        return state(sim)


@pytest.mark.parametrize("fp", [L.FP_EXACT, L.FP_FAST])
@pytest.mark.parametrize("own_graph", [False, True])
def test_frame_recorded_before_the_first_step(fp, own_graph):
    """A frame recorded on a new handle, an eager frame before its first
    replay, then replays and eager frames in turn."""
    stream = torch.cuda.Stream()
    with simulator(fp, 2, stream) as sim:
        g = recorded(stream, lambda: sim.step(1))
        sim.enable_graph(own_graph)
        sim.step(1)
        same(state(sim), plain(fp, 2, 1))
        replay(stream, g)
        same(state(sim), plain(fp, 2, 2))
        sim.step(2)
        replay(stream, g)
        replay(stream, g)
        sim.step(1)
        same(state(sim), plain(fp, 2, 7))


@pytest.mark.parametrize("fp", [L.FP_EXACT, L.FP_FAST])
@pytest.mark.parametrize("own_graph", [False, True])
def test_recorded_frame_that_is_dropped(fp, own_graph):
    stream = torch.cuda.Stream()
    with simulator(fp, 2, stream) as sim:
        sim.enable_graph(own_graph)
        sim.step(1)
        before = state(sim)
        g = recorded(stream, lambda: sim.step(1))
        same(state(sim), before)
        del g
        sim.step(3)
        same(state(sim), plain(fp, 2, 4))


def test_own_frames_and_a_recorded_one_take_turns():
    """The handle has a captured frame before the caller records one; single
    substeps in pairs between replays leave either count buffer current."""
    stream = torch.cuda.Stream()
    with simulator(L.FP_EXACT, 2, stream) as sim:
        sim.enable_graph(True)
        sim.step(2)
        g = recorded(stream, lambda: sim.step(2))
        sim.run()
        sim.run()
        replay(stream, g)
        sim.step(1)
        sim.run()
        sim.run()
        replay(stream, g)
        sim.step(1)
        same(state(sim), plain(L.FP_EXACT, 2, 10))


@pytest.mark.parametrize("first,then", [(3, 4), (4, 3), (3, 5)])
def test_predicted_positions_after_a_replay(first, then):
    """An odd number of iterations ends in the other buffer of the predicted
    positions: the field is the last substep's whoever ran it."""
    stream = torch.cuda.Stream()
    with simulator(L.FP_EXACT, 2, stream, first) as sim:
        g = recorded(stream, lambda: sim.step(1))
        sim.setConfig({"iteration": then})
        sim.step(1)
        replay(stream, g)
        got = state(sim)
    with simulator(L.FP_EXACT, 2, None, then) as sim:
        sim.step(1)
        sim.setConfig({"iteration": first})
        sim.step(1)
        same(got, state(sim))


def test_recorded_on_the_handles_own_stream():
    """The caller records the stream that the handle made and handed out."""
    with simulator(L.FP_EXACT, 2, None) as sim:
        sim.step(1)
        stream = torch.cuda.ExternalStream(sim.stream)
        g = recorded(stream, lambda: sim.step(1))
        sim.run()
        sim.run()
        replay(stream, g)
        sim.step(1)
        same(state(sim), plain(L.FP_EXACT, 2, 4))


@pytest.mark.parametrize("kind", ["learned", "batch", "field", "cellblock"])
def test_recorded_frames_of_other_routes(kind):
    """The learned start (side stream and fallback in the recorded graph), 16
    small scenes in one batch, a volume map and the cell-block passes."""

    def make(stream):
        if kind == "batch":
            cfg, sc, fa = scenes.batch_scenes_spec(count=16, n_min=300, n_max=900, seed=3, field_res=(8, 8, 8))
            cfg, sc = scenes.build_batch((cfg, sc, fa), quadrature=4)
            cfg.stream = stream.cuda_stream if stream is not None else None
            return PBFBatch(cfg, sc)
        if kind == "cellblock":
            sim = simulator(L.FP_FAST, 2, stream)
            sim.set_launch(build=L.BUILD_CELLBLOCK_MASK)
            return sim
        sc = scenes.reference_scene("boundary_small")
        cfg = scenes.copy_config(sc.config)
        cfg.fp_mode, cfg.substeps = L.FP_FAST, 2
        cfg.stream = stream.cuda_stream if stream is not None else None
        sim = PBF(cfg)
        sim.set_particles(sc.particles)
        f = sc.field
        sim.set_boundary_field(f["res"], f["origin"], f["extent"], f["sdf"], f["vol"])
        if kind == "learned":
            sim.set_learned(mlp_init(3), iterations=1, fallback_bound=0.02)
        return sim

    def bits(sim):
        sim.synchronize()
        return [np.asarray(sim.copy_field(f)).view(np.uint32) for f in FIELDS]

    stream = torch.cuda.Stream()
    with make(stream) as sim:
        g = recorded(stream, lambda: sim.step(1))
        sim.step(1)
        replay(stream, g)
        replay(stream, g)
        sim.enable_graph(True)
        sim.step(2)
        replay(stream, g)
        got = bits(sim)
    with make(None) as sim:
        sim.step(6)
        same(got, bits(sim))


def test_first_captured_frame_is_refused_under_the_callers_capture():
    """A handle with no captured frame yet cannot capture one inside the
    caller's capture; the capture and the handle stay usable."""
    stream = torch.cuda.Stream()
    x = torch.zeros(1, device="cuda")
    with simulator(L.FP_EXACT, 2, stream) as sim:
        sim.enable_graph(True)

        def body():
            with pytest.raises(L.PBFError):
                sim.step(1)
            x.add_(1.0)

        g = recorded(stream, body)
        sim.step(2)
        replay(stream, g)
        same(state(sim), plain(L.FP_EXACT, 2, 2))
        assert float(x) == 1.0
