"""The patch sums where a patch has more ids than the thread's column keeps,
and one fewer, and as many: fans that meet in a vertex. Against the C oracle
bit for bit; an odd number of elements, so that the last line of records is
not full."""
import numpy as np
import pytest

from trinity_b200.meshgen import GridMesh, field_shock


def fans(extra):
    """Vertex 0 in 4 elements with 7 neighbours; extra[i] more elements, with
    vertices of their own, at neighbour i + 1: 4 + sum(extra) ids."""
    ang = 2 * np.pi * np.arange(7) / 7
    pts = [[0.5, 0.5]] + [[0.5 + 0.2 * np.cos(a), 0.5 + 0.2 * np.sin(a)] for a in ang]
    tris = [[0, 1, 2], [0, 3, 4], [0, 5, 6], [0, 6, 7]]
    for i, n in enumerate(extra):
        for k in range(n):
            a, b = 2 * np.pi * (k + 0.1) / n, 2 * np.pi * (k + 0.8) / n
            x, y = pts[i + 1]
            r = 0.05 + 0.003 * k
            pts += [[x + r * np.cos(a), y + r * np.sin(a)], [x + r * np.cos(b), y + r * np.sin(b)]]
            tris.append([i + 1, len(pts) - 2, len(pts) - 1])
    return GridMesh(np.array(pts), np.array(tris, np.int32), np.zeros((0, 2), np.int32), np.zeros(0, np.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("extra", [[6, 6, 6, 6, 6, 6, 6], [7, 6, 6, 7, 7, 5, 6], [7, 7, 6, 6, 7, 6, 6], [7, 7, 7, 7, 7, 6, 7]],
                         ids=["46", "48", "49", "52"])
def test_patch_at_the_columns_end(oracle_built, extra):
    from tests.oracle_lib import Oracle, tags_of
    from trinity_b200.api import Mesh, Metrics
    m = fans(extra)
    u = field_shock(m.points, 7.0, 0.2)
    o = Oracle(m, u, bucket=64)
    o.metric(0.8, 2)
    g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 1, capa_scale=1)
    g.load_arrays(m.points, m.tris, tags_of(m), u)
    g.set_options(exact_sum=True)
    Metrics(g, 0.8, 2).run()
    got = g.export()[1]
    g.close()
    assert np.array_equal(got.view(np.uint64), o.state().tensor.view(np.uint64))
