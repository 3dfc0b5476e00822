"""An export with the tensors where the mesh fills its capacity: points and
tensors of every vertex wait in the staging buffer."""
import numpy as np
import pytest

from trinity_b200.meshgen import field_shock, grid_mesh


def renumbered(g):
    pts, ten, tri, alive, _ = g.export()
    newid = np.cumsum(alive.astype(np.int64)) - 1
    return pts[alive == 1], newid[tri[tri[:, 0] >= 0]].astype(np.int32), ten[alive == 1]


def same(got, want):
    return all(np.array_equal(np.ascontiguousarray(a).view(np.uint8), np.ascontiguousarray(b).view(np.uint8))
               for a, b in zip(got, want))


def make(side, scale):
    from tests.oracle_lib import tags_of
    from trinity_b200.api import Mesh
    m = grid_mesh(side, 0.2, 5)
    g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 2, capa_scale=scale)
    g.load_arrays(m.points, m.tris, tags_of(m), field_shock(m.points, 7.0, 0.2))
    return m, g


@pytest.mark.gpu
@pytest.mark.parametrize("side", [2, 3, 15, 16, 47])
def test_export_without_room_to_spare(side):
    m, g = make(side, 1)
    from trinity_b200.api import Metrics
    p0, t0, m0 = g.export_compact()
    assert np.array_equal(p0, m.points) and np.array_equal(t0, m.tris) and not m0.any()
    Metrics(g, 0.8, 2).run()
    want = renumbered(g)
    assert same(g.export_compact(), want)
    p, t, ten = g.export_compact(with_tensor=False)
    assert ten is None and same((p, t), want[:2])
    g.close()
