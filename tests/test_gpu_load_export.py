"""Loading in one pass and exporting with one read back: a reload after an
adaptation has to start as a fresh load does, and an export has to be the
renumbering of the raw state where the staging buffer holds the vertices and
the triangles and where it does not (no room to spare, with the tensor), at
sides whose counts end inside a 16-byte store of flags."""
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


@pytest.mark.gpu
@pytest.mark.parametrize("side", [15, 47])
def test_reload_and_export_after_adapting(side):
    from trinity_b200.api import Coarse, Metrics, Partit, Refine, Smooth, Swap
    m, g = make(side, 8)
    h = Partit(g, 8)

    def adapt():
        Metrics(g, 0.8, 2).run()
        for k in (Refine(g, 1), Coarse(g, h), Swap(g), Smooth(g, h, 1)):
            k.run()
        return renumbered(g)

    first = adapt()
    nv, ne = first[0].shape[0], first[1].shape[0]
    assert same(g.export_compact(), first)
    for extra in (0, 5, 40000):       # exactly enough, less than the slots in use, more
        out = (np.empty((nv + extra, 2)), np.empty((ne + extra, 3), np.int32), np.empty((nv + extra, 3)))
        got = g.export_compact(out=out)
        assert same(got, first) and got[0].base is out[0]
    for cut in range(3):
        out = [np.empty((nv, 2)), np.empty((ne, 3), np.int32), np.empty((nv, 3))]
        out[cut] = out[cut][:-1]
        with pytest.raises(ValueError):
            g.export_compact(out=tuple(out))
    g.reload()
    p, t, ten = g.export_compact()
    assert np.array_equal(p, m.points) and np.array_equal(t, m.tris) and not ten.any()
    assert same(adapt(), first)
    g.close()
