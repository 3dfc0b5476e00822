"""Edges just past the splitting threshold whose two endpoint lengths agree but
for a unit in the last place, in single precision, where the ratio of the two
may round to 1 and the computed length is then not a number: a metric clamped to
one size on a grid whose edges are longer, or shorter, than the threshold by a
few parts in 1e5. Above it every edge is split, below it the diagonals alone;
at side, offset and direction of the edges that vary."""
import numpy as np
import pytest

from trinity_b200.meshgen import GridMesh, grid_mesh


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("off", [1.1e-5, 1.25e-5, 1.4e-5, 1.6e-5, 3e-5, -1.1e-5, -1.25e-5, -1.4e-5, -1.6e-5, -3e-5])
def test_edges_next_to_the_threshold(off, precision):
    from tests.helpers import check_invariants, gpu_mesh, gpu_state
    from trinity_b200.api import Metrics, Refine
    for side, angle in ((16, 0.0), (40, 0.3), (57, 1.1)):
        m = grid_mesh(side)
        c, s = np.cos(angle), np.sin(angle)
        x, y = m.points.T
        u = 3 * x * x + 2 * y * y + x * y + 0.05 * np.sin(9 * x + 4 * y)
        pts = m.points @ np.array([[c, s], [-s, c]])
        g = gpu_mesh(GridMesh(pts, m.tris, m.edges, m.corners), u, dict(bucket=64, depth=1, rounds=1), capa_scale=5)
        g.set_precision(precision)
        Metrics(g, 1e5, 2, h_min=1.0 / side / np.sqrt(2.0) / (1.0 + off), h_max=0.4).run()
        Refine(g, 1).run()
        st = gpu_state(g)
        g.close()
        if precision == "fp64":   # the mixed form's mid-points are another matter
            check_invariants(st)
        assert st.active_elems().shape[0] == m.nb_elems * (4 if off > 0 else 2), (side, angle)
