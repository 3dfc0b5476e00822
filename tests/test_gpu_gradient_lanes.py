"""Gradient smoothing where a stencil fits the lanes that share it and where
it does not: centres of 6, 8, 9, 16, 17 and 30 elements. No element turns or
falls below its old stencil minimum, the objective grows, and the moved vertex
is the one of the elements' exact objective (qualities recomputed from the
mesh equal the ones the moves stored)."""
import numpy as np
import pytest

from tests.test_gpu_patch import wheel
from trinity_b200.meshgen import field_shock


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("objective,follows", [("sum", False), ("log", True)])
@pytest.mark.parametrize("k", [6, 8, 9, 16, 17, 30])
def test_gradient_moves_improve_every_stencil_size(k, objective, follows, precision):
    from tests.helpers import gpu_state, signed_areas
    from tests.oracle_lib import tags_of
    from trinity_b200.api import GradientSmooth, Mesh, Metrics, Partit
    m = wheel(k, 4)
    m.points[0] += 0.02            # off the centre: there is something to gain
    u = field_shock(m.points, 5.0, 0.1)
    g = Mesh((m.nb_nodes, m.nb_elems), 64, 1, 0, 1, capa_scale=4)
    g.set_precision(precision)
    g.load_arrays(m.points, m.tris, tags_of(m), u)
    Metrics(g, 0.8, 2).run()
    before = g.qualities()
    GradientSmooth(g, Partit(g, 8), 3, objective=objective, tensor_follows=follows).run()
    st, after = gpu_state(g), g.qualities()
    g.close()
    assert np.any(st.points != m.points)
    assert np.all(signed_areas(st.points, st.elems) > 1e-9)
    f = np.log if objective == "log" else (lambda q: q)
    if not follows:                # the tensors are the old ones: the sums compare
        assert f(after).sum() > f(before).sum()
        assert after.min() >= before.min() * (1 - (1e-12 if precision == "fp64" else 1e-5))
