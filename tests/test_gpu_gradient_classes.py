"""Gradient smoothing of a mesh with color classes on both sides of the length
from which one lane moves a vertex instead of eight: no element turns or falls
below its old stencil minimum, the objective grows, and two runs agree bit for
bit."""
import numpy as np
import pytest

from trinity_b200.meshgen import field_multi, grid_mesh


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("side", [620, 760])
def test_long_classes_improve(side, precision):
    from tests.helpers import gpu_state, signed_areas
    from tests.oracle_lib import tags_of
    from trinity_b200.api import GradientSmooth, Mesh, Metrics, Partit
    m = grid_mesh(side, 0.3, 3)
    runs = []
    for _ in range(2):
        g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 1, capa_scale=1)
        g.set_precision(precision)
        g.load_arrays(m.points, m.tris, tags_of(m), field_multi(m.points))
        Metrics(g, 0.7, 2).run()
        before = g.qualities()
        GradientSmooth(g, Partit(g, 8), 2, objective="sum", tensor_follows=False).run()
        runs.append((gpu_state(g), before, g.qualities()))
        g.close()
    (st, before, after), (again, _, _) = runs
    assert not st.diff(again)
    assert np.mean(np.any(st.points != m.points, axis=1)) > 0.2
    # a vertex moves only where all its elements end counter-clockwise (the
    # input has a few that are not)
    assert np.all((signed_areas(st.points, st.elems) > 0) | (signed_areas(m.points, m.tris) <= 0))
    assert after.sum() > before.sum()
    assert after.min() >= before.min() * (1 - (1e-12 if precision == "fp64" else 1e-5))
