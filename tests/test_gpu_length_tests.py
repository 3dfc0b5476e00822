"""Length and orientation tests decide as the computed lengths do: refinement
and coarsening, replayed on the oracle's decisions, end on the oracle's bits
on meshes that press the tests' margins: a graded and a stretched metric (the
threshold lies between the two endpoint lengths of many edges), a uniform one
(the endpoint lengths agree), flat elements next to the orientation threshold,
coordinates far from the origin; and in the mixed form the oracle's mesh is
what the free mode's invariants ask for."""
import numpy as np
import pytest

from trinity_b200.meshgen import GridMesh, field_multi, field_shock, grid_mesh

# name: (side, jitter, scale x, scale y, offset, field, target)
CASES = {
    "graded": (31, 0.3, 1.0, 1.0, 0.0, "multi", 0.7),
    "shock": (40, 0.0, 1.0, 1.0, 0.0, "shock", 0.5),
    "uniform": (23, 0.3, 1.0, 1.0, 0.0, "square", 0.4),
    "flat": (23, 0.3, 1.0, 2e-3, 0.0, "multi", 0.6),
    "far": (23, 0.3, 1.0, 1.0, 3e5, "multi", 0.6),
    "tiny": (23, 0.35, 8e-4, 2e-3, 0.0, "multi", 0.5),
    "large": (23, 0.3, 3e4, 1e3, 0.0, "multi", 0.6),
    "two": (2, 0.2, 1.0, 1.0, 0.0, "multi", 0.6),
}


def _mesh(name):
    side, jit, sx, sy, off, field, target = CASES[name]
    m = grid_mesh(side, jit, 9)
    u = {"multi": field_multi, "shock": field_shock, "square": lambda p: (p ** 2).sum(1)}[field](m.points)
    return GridMesh(m.points * np.array([sx, sy]) + off, m.tris, m.edges, m.corners), u, target


@pytest.mark.gpu
@pytest.mark.parametrize("name", sorted(CASES))
def test_refine_and_coarsen_end_on_the_oracles_bits(oracle_built, name):
    from tests.helpers import gpu_mesh, gpu_state
    from tests.oracle_lib import Oracle
    from trinity_b200.api import Coarse, Metrics, Partit, Refine
    m, u, target = _mesh(name)
    o = Oracle(m, u, capa_scale=12, bucket=128)
    o.metric(target, 2)
    o.refine(1)
    o.coarsen()
    g = gpu_mesh(m, u, dict(bucket=128, depth=1, rounds=1), capa_scale=12)
    g.set_options(exact_sum=True)   # an empty log (nothing collapses) leaves the replay mode off
    g.set_replay(o.log())
    Metrics(g, target, 2).run()
    Refine(g, 1).run()
    Coarse(g, Partit(g, 8)).run()
    d = gpu_state(g).diff(o.state())
    g.close()
    assert not d


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", ["graded", "shock", "uniform", "two"])
def test_both_searches_find_the_same_targets(name, precision):
    from tests.helpers import check_invariants, gpu_mesh, gpu_state
    from trinity_b200.api import Coarse, Metrics, Partit, Refine
    m, u, target = _mesh(name)
    states = []
    for lanes in (1, 8, 16):
        g = gpu_mesh(m, u, dict(bucket=128, depth=1, rounds=1), capa_scale=12)
        g.set_precision(precision)
        g.set_tune(dict(g.get_tune(), group_lanes=lanes, group_max=1 << 20))
        Metrics(g, target, 2).run()
        Refine(g, 1).run()
        Coarse(g, Partit(g, 8)).run()
        states.append(gpu_state(g))
        g.close()
    assert not states[1].diff(states[0]) and not states[2].diff(states[0])
    check_invariants(states[0])
