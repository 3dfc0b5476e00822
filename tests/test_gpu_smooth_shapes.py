"""Every launch shape the smoothing can take (2, 4 or 8 lanes a vertex, two,
three or four blocks a multiprocessor) can be asked for, beside the default that
picks one by the class's length: on the oracle's coloring each ends on the
oracle's bits, and in the mixed form all end on the same mesh."""
import numpy as np
import pytest

from tests.test_gpu_smooth_tries import CASES
from trinity_b200.meshgen import GridMesh, field_multi, grid_mesh

SHAPES = [(lanes, regs) for lanes in (2, 4, 8) for regs in (0, 1, 2)]


def mesh_of(name):
    side, jit, sx, sy, off, f = CASES[name]
    m = grid_mesh(side, jit, 5)
    u = field_multi(m.points) + np.sin(f * m.points[:, 1])
    return GridMesh(m.points * np.array([sx, sy]) + off, m.tris, m.edges, m.corners), u


def smoothed(name, shape, precision, log=None):
    from tests.helpers import gpu_mesh, gpu_state
    from trinity_b200.api import Metrics, Partit, Smooth
    m, u = mesh_of(name)
    g = gpu_mesh(m, u, dict(bucket=64, depth=2, rounds=1), capa_scale=4)
    cfg = g.get_tune()
    assert (cfg["smooth_lanes"], cfg["smooth_regs"]) == (2, 7)   # by the class's length
    g.set_tune(dict(cfg, smooth_lanes=shape[0], smooth_regs=shape[1]))
    if log is None:
        g.set_precision(precision)
    else:
        g.set_replay(log)
    Metrics(g, 0.8, 2).run()
    Smooth(g, Partit(g, 8), 2).run()
    st = gpu_state(g)
    g.close()
    return st


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_every_shape_ends_on_the_oracles_bits(oracle_built, name):
    from tests.oracle_lib import Oracle
    m, u = mesh_of(name)
    o = Oracle(m, u, capa_scale=4)
    o.metric(0.8, 2)
    o.smooth(2)
    for shape in SHAPES + [(2, 7), (1, 7)]:
        assert not smoothed(name, shape, "fp64", o.log()).diff(o.state()), shape


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_every_shape_ends_on_the_same_mesh_mixed(name):
    want = smoothed(name, (2, 7), "mixed")
    for shape in SHAPES:
        assert not smoothed(name, shape, "mixed").diff(want), shape
