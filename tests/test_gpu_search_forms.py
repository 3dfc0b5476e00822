"""The collapse search by one lane a vertex, by lanes that share one, and inside
the launch that runs the levels of short lists: the launch shapes choose as
they say, and the targets, so the coarsened meshes, are the same, on meshes
whose first levels list more than the 4,096 vertices of that launch and on one
with fewer, with vertices of long rows among them."""
import numpy as np
import pytest

from tests.test_gpu_noalloc_forms import cut_in_three
from trinity_b200.meshgen import GridMesh, field_multi, grid_mesh


def cut_mesh(side):
    m = grid_mesh(side, 0.1, 3)
    pts, tris = cut_in_three(side)
    return GridMesh(pts, tris, m.edges, m.corners)


MESHES = {"grid130": lambda: grid_mesh(130, 0.25, 7), "cut60": lambda: cut_mesh(60), "grid20": lambda: grid_mesh(20, 0.25, 7)}
# launch shapes, and what runs with them: (lists for the filter kernels, lists for the level loop)
SHAPES = {"one": dict(group_lanes=1), "lanes4": dict(group_lanes=4, group_max=1 << 20),
          "lanes8": dict(group_lanes=8, group_max=1 << 20), "lanes16": dict(group_lanes=16, group_max=1 << 20),
          "short": dict(group_lanes=8, group_max=300), "none": dict(group_lanes=16, group_max=0), "default": dict()}


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", sorted(MESHES))
def test_all_forms_find_the_same_targets(name, precision):
    from tests.helpers import check_invariants, gpu_state
    from tests.oracle_lib import tags_of
    from trinity_b200 import _lib
    from trinity_b200.api import Coarse, Mesh, Metrics, Partit
    m = MESHES[name]()
    states = {}
    for shape, cfg in SHAPES.items():
        g = Mesh((m.nb_nodes, m.nb_elems), 128, 1, 0, 1, capa_scale=1)
        g.set_precision(precision)
        g.load_arrays(m.points, m.tris, tags_of(m), field_multi(m.points))
        g.set_tune(dict(g.get_tune(), **cfg))
        Metrics(g, 0.3, 2).run()
        _lib.profile_enable(True)
        Coarse(g, Partit(g, 8)).run()
        ran = {e["kernel"]: e["launches"] for e in _lib.profile_read() if e["launches"]}
        _lib.profile_enable(False)
        states[shape] = gpu_state(g)
        g.close()
        if shape in ("one", "none"):
            assert ran["coarsen_filter"] > 3 and "coarsen_tail" not in ran
        else:
            assert ran["coarsen_tail"] == 1
            assert ("coarsen_filter" in ran) == (m.nb_nodes > min(4096, cfg.get("group_max", 4096)))
    want = states["one"]
    assert np.mean(want.alive == 0) > 0.2
    check_invariants(want)
    for shape, st in states.items():
        assert not st.diff(want), shape
