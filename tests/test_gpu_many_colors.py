"""Partit with more colors than the eight classes that are smoothed: the class
offsets stay inside their words, whatever the number. On meshes whose vertices
never need a ninth color the smoothing ends where eight colors end, the counts
are what they were, and the mesh can be refined on; by one cluster (a small
mesh) and by the grid (a larger one)."""
import numpy as np
import pytest

from trinity_b200.meshgen import field_multi, grid_mesh


@pytest.mark.gpu
@pytest.mark.parametrize("side", [30, 230])
@pytest.mark.parametrize("kind", ["laplacian", "gradient"])
def test_smoothing_with_many_colors(side, kind):
    from tests.oracle_lib import tags_of
    from trinity_b200.api import GradientSmooth, Mesh, Metrics, Partit, Refine, Smooth
    m = grid_mesh(side, 0.2, 9)
    g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 1, capa_scale=4)
    g.load_arrays(m.points, m.tris, tags_of(m), field_multi(m.points))
    want = None
    for n in (9, 10, 11, 18, 19, 25, 31, 64):
        g.reload()
        Metrics(g, 0.9, 2).run()
        (Smooth(g, Partit(g, n), 1) if kind == "laplacian" else GradientSmooth(g, Partit(g, n), 2)).run()
        assert g.counts() == (m.nb_nodes, m.nb_elems, m.nb_nodes, m.nb_elems)
        smoothed = g.export()
        Refine(g, 1).run()
        got = [*smoothed, *g.export()]
        if want is None:
            want = got
            assert np.any(smoothed[0] != m.points)
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), n
    g.close()
