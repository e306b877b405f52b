"""The neighbour passes with several lanes a slot (small scenes) against the same passes with one lane a slot, bit for bit, at the sizes where
the number of lanes changes and where a warp or block is partly filled."""
import numpy as np
import pytest

from pbf_gb300 import _lib as L
from pbf_gb300 import PBF, scenes

pytestmark = pytest.mark.gpu

FIELDS = (L.FIELD_POSITION, L.FIELD_VELOCITY, L.FIELD_ACCELERATION, L.FIELD_PREDICTED, L.FIELD_OMEGA, L.FIELD_NORMAL,
          L.FIELD_LAMBDA, L.FIELD_DELTA_P)


@pytest.mark.parametrize("field", [False, True])
@pytest.mark.parametrize("fp,n", [(L.FP_EXACT, n) for n in (1, 2, 7, 9, 33, 1025, 1 << 14, (1 << 14) + 1, 1 << 15,
                                                            (1 << 15) + 1)] +
                         [(L.FP_FAST, n) for n in (1, 9, 1025, 1 << 12, (1 << 12) + 1, 1 << 13, (1 << 13) + 1)])
def test_lanes_equal_one_lane(fp, n, field):
    """Persistent grids (ctas_per_sm) take one lane a slot at every size."""
    rng = np.random.default_rng(n)
    sc = scenes.reference_scene("boundary_small")
    cfg = scenes.copy_config(sc.config)
    cfg.fp_mode, cfg.max_particles, cfg.max_neighbors = fp, n, 1024
    side = 0.04 * max(n, 8) ** (1.0 / 3.0) * 0.5
    pts = np.zeros((n, 4), np.float32)
    pts[:, :3] = 0.5 + min(side, 0.9) * (rng.random((n, 3)) - 0.5)
    pts[: n // 20, :3] = 0.5 + 0.05 * (rng.random((n // 20, 3)) - 0.5)  # long lists
    f, out = sc.field, []
    for ctas in (0, 4):
        with PBF(cfg) as sim:
            sim.set_particles(pts)
            sim.set_launch(ctas_per_sm=ctas)
            if field:
                sim.set_boundary_field(f["res"], f["origin"], f["extent"], f["sdf"], f["vol"])
            sim.set_capture(True)
            sim.step(2)
            sim.synchronize()
            out.append([sim.copy_field(q) for q in FIELDS])
    for a, b in zip(*out):
        assert np.array_equal(np.asarray(a).view(np.uint32), np.asarray(b).view(np.uint32))
