"""A small mesh is colored by one cluster launch, a larger one by a cooperative
grid, a captured round by a launch a round: the same rounds of the same rule,
so a round of stage calls and a captured round end in the same state, bit for
bit, on both sides of the size where the form changes, with the fewest
vertices, with vertices of long rows, and with few colors."""
import numpy as np
import pytest

from tests.helpers import gpu_state
from tests.test_gpu_patch import wheel
from trinity_b200.meshgen import field_multi, field_shock, grid_mesh

MESHES = {"grid%d" % s: (lambda s=s: grid_mesh(s, 0.2, 9)) for s in (1, 2, 60, 128, 190, 201, 203, 230)}
MESHES.update({"wheel%d" % k: (lambda k=k: wheel(k)) for k in (6, 9, 30)})


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(MESHES))
def test_round_equals_captured_round(name):
    from tests.oracle_lib import tags_of
    from trinity_b200.api import Coarse, Mesh, Metrics, Partit, Refine, Smooth, Swap
    m = MESHES[name]()
    u = field_multi(m.points) if name.startswith("grid") else field_shock(m.points, 7.0, 0.2)
    got = []
    for graph in (False, True):
        g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 1, capa_scale=8 if m.nb_nodes > 9000 else 400)
        g.load_arrays(m.points, m.tris, tags_of(m), u)
        Metrics(g, 0.9, 2).run()
        h = Partit(g, 8)
        for _ in range(2):
            if graph:
                g.round_graph(1)
            else:
                for k in (Refine(g, 1), Coarse(g, h), Swap(g), Smooth(g, h, 1)):
                    k.run()
        got.append(gpu_state(g))
        g.close()
    assert not got[1].diff(got[0])


@pytest.mark.gpu
@pytest.mark.parametrize("side", [9, 100])
def test_few_colors(side):
    """With Partit(n <= 6): five colors, vertices that find none are left."""
    from tests.oracle_lib import tags_of
    from trinity_b200.api import Mesh, Metrics, Partit, Smooth
    m = grid_mesh(side, 0.25, 4)
    out = []
    for _ in range(2):
        g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 1, capa_scale=4)
        g.load_arrays(m.points, m.tris, tags_of(m), field_multi(m.points))
        Metrics(g, 0.9, 2).run()
        Smooth(g, Partit(g, 1), 1).run()
        out.append(g.export())
        g.close()
    assert all(np.array_equal(a, b) for a, b in zip(*out))
    assert not np.array_equal(out[0][0], m.points)
