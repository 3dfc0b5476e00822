"""Forms of one rule on the same input, bit for bit: the gradient smoothing by
one lane a vertex and by eight (the class's length chooses, so the same
vertices are moved beside a large grid that is smoothed too and beside the same
grid held fixed), for stencils that fit the lanes and that do not, and the swap
matchings inside the level loop's cluster and as a captured round's launches,
in both precisions."""
import numpy as np
import pytest

from tests.test_gpu_patch import wheel
from trinity_b200.meshgen import field_multi, field_shock, grid_mesh


def union(meshes):
    """Disjoint meshes side by side; boundary tags of each."""
    from tests.oracle_lib import tags_of
    pts, tris, tags, n = [], [], [], 0
    for k, m in enumerate(meshes):
        pts.append(m.points + [1.5 * k, 0.0])
        tris.append(m.tris + n)
        tags.append(tags_of(m))
        n += m.nb_nodes
    return np.concatenate(pts), np.concatenate(tris).astype(np.int32), np.concatenate(tags)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("objective,follows", [("sum", False), ("sum", True), ("log", False), ("log", True)])
def test_gradient_moves_by_one_lane_and_by_eight(objective, follows, precision):
    from trinity_b200.api import GradientSmooth, Mesh, Metrics, Partit
    small = [wheel(k, 4) for k in (3, 6, 8, 9, 16, 17, 30)] + [grid_mesh(40, 0.3, 5)]
    for m in small[:-1]:
        m.points[0] += 0.02
    pts, tris, tags = union(small + [grid_mesh(760, 0.3, 3)])   # its classes: some 10^5 vertices
    n = sum(m.nb_nodes for m in small)
    u = field_shock(pts, 5.0, 0.1)
    held = tags.copy()
    held[n:] = 4
    got = []
    for t in (tags, held):
        g = Mesh((len(pts), len(tris)), 64, 1, 0, 1, capa_scale=1)
        g.set_precision(precision)
        g.load_arrays(pts, tris, t, u)
        Metrics(g, 0.7, 2).run()
        GradientSmooth(g, Partit(g, 8), 3, objective=objective, tensor_follows=follows).run()
        p, ten, _, _, _ = g.export()
        q = g.qualities()
        got.append((p[:n], ten[:n], q[:sum(m.nb_elems for m in small)], p[n:]))
        g.close()
    (p1, t1, q1, rest1), (p8, t8, q8, rest8) = got
    assert np.any(p1 != pts[:n], axis=1).mean() > 0.2 and np.array_equal(rest8, pts[n:]) and not np.array_equal(rest1, rest8)
    for a, b in ((p1, p8), (t1, t8), (q1, q8)):
        assert np.array_equal(a.view(np.uint64), b.view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("match", ["greedy", "gain", "row_order"])
@pytest.mark.parametrize("name", ["grid24", "grid150", "wheel30"])
def test_matchings_in_the_level_loop_and_captured(name, match, precision):
    from tests.helpers import gpu_state
    from tests.oracle_lib import tags_of
    from trinity_b200.api import Coarse, Mesh, Metrics, Partit, Refine, Smooth, Swap
    m = wheel(30) if name == "wheel30" else grid_mesh(int(name[4:]), 0.25, 9)
    u = field_shock(m.points, 7.0, 0.2) if name == "wheel30" else field_multi(m.points)
    got = []
    for graph in (False, True):
        g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 1, capa_scale=8 if m.nb_nodes > 9000 else 100)
        g.set_precision(precision)
        g.set_swap_match(match)
        g.load_arrays(m.points, m.tris, tags_of(m), u)
        Metrics(g, 0.8, 2).run()
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
