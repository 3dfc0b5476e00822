"""The smoothing's estimated tries decide as the exact ones do: one smoothing
call, replayed on the oracle's coloring, ends on the oracle's bits on meshes
that press the estimate's error bound: flat elements, a metric stretched up
to the bound's limit and past it, coordinates far from the origin, areas next
to the orientation threshold."""
import numpy as np
import pytest

from trinity_b200.meshgen import GridMesh, field_multi, grid_mesh

# name: (side, jitter, scale x, scale y, offset, field factor of y)
CASES = {
    "plain": (31, 0.3, 1.0, 1.0, 0.0, 1.0),
    "flat": (23, 0.3, 1.0, 1e-3, 0.0, 1.0),
    "stretched": (23, 0.3, 1.0, 1e-2, 0.0, 1e3),
    "far": (23, 0.3, 1.0, 1.0, 3e5, 1.0),
    "very_far": (17, 0.3, 1.0, 1.0, 4e7, 1.0),
    "tiny": (23, 0.35, 8e-4, 2e-3, 0.0, 1.0),
    "large": (23, 0.3, 3e4, 1e3, 0.0, 1.0),
    "one": (2, 0.3, 1.0, 1.0, 0.0, 1.0),
}


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(2, 7), (4, 5), (8, 4)])
@pytest.mark.parametrize("name", sorted(CASES))
def test_smoothing_ends_on_the_oracles_bits(oracle_built, name, shape):
    from tests.helpers import gpu_mesh, gpu_state
    from tests.oracle_lib import Oracle
    from trinity_b200.api import Metrics, Partit, Smooth
    side, jit, sx, sy, off, f = CASES[name]
    m = grid_mesh(side, jit, 5)
    u = field_multi(m.points) + np.sin(f * m.points[:, 1])
    m = GridMesh(m.points * np.array([sx, sy]) + off, m.tris, m.edges, m.corners)
    o = Oracle(m, u, capa_scale=4)
    o.metric(0.8, 2)
    o.smooth(2)
    g = gpu_mesh(m, u, dict(bucket=64, depth=2, rounds=1), capa_scale=4)
    cfg = g.get_tune()
    cfg["smooth_lanes"], cfg["smooth_regs"] = shape
    g.set_tune(cfg)
    g.set_replay(o.log())
    Metrics(g, 0.8, 2).run()
    Smooth(g, Partit(g, 8), 2).run()
    d = gpu_state(g).diff(o.state())
    g.close()
    assert not d
