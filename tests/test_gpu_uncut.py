"""Refinement where the two ends of an edge measure it differently: a metric
clamped to one size, so that the endpoint tensors agree but for their last
bits, on a grid whose edges are as long as the splitting threshold. Elements
that stay uncut leave the slots they had reserved erased, also after another
mesh of the same handle has used those slots."""
import numpy as np
import pytest

from trinity_b200.meshgen import field_multi, grid_mesh

SIDE = 16


@pytest.mark.gpu
def test_uncut_elements_leave_no_triangles():
    from tests.helpers import gpu_state, signed_areas
    from tests.oracle_lib import tags_of
    from trinity_b200.api import Mesh, Metrics, Refine
    m = grid_mesh(SIDE)
    g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 1, capa_scale=8)
    g.load_arrays(m.points, m.tris, tags_of(m), field_multi(m.points))
    uncut = 0
    for k in range(-12, 13):
        g.reload()
        Metrics(g, 3.0, 2).run()   # fills the slots behind the input's
        Refine(g, 1).run()
        used = g.counts()[1]
        g.reload()
        h = 1.0 / SIDE / np.sqrt(2.0)
        Metrics(g, 1e5, 2, h_min=h * (1 + k * 1.2e-16), h_max=0.4).run()
        Refine(g, 1).run()
        st = gpu_state(g)
        assert used > m.nb_elems and st.elems.shape[0] > m.nb_elems
        erased = st.elems[:, 0] < 0
        assert np.all(st.elems[erased] == -1)
        live = st.elems[~erased]
        assert live.min() >= 0 and live.max() < st.points.shape[0]
        # an uncut element keeps its own area, a cut one hands it on
        assert abs(signed_areas(st.points, live).sum() - 1.0) < 1e-12
        uncut += int(erased.sum())
    g.close()
    assert uncut > 0
