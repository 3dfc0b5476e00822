"""The patch sums of the metric recovery and of its adjoint, where the patch
fits the registers and where it does not: rows of 8 entries and more, rings of
7 vertices and more, buckets whose rows are not 16-byte aligned. The recovery
against the C oracle bit for bit, the adjoint against the FP64 autograd
restatement."""
import numpy as np
import pytest

from trinity_b200.meshgen import GridMesh, field_shock, grid_mesh


def wheel(k: int, rings: int = 3) -> GridMesh:
    """A centre of degree k inside `rings` rings of k vertices each."""
    ang = 2 * np.pi * (np.arange(k) + 0.1) / k
    pts = [[0.5, 0.5]]
    for r in range(1, rings + 1):
        pts += [[0.5 + 0.45 * r / rings * np.cos(a + 0.2 * r), 0.5 + 0.45 * r / rings * np.sin(a + 0.2 * r)] for a in ang]
    at = lambda r, i: 1 + (r - 1) * k + i % k   # noqa: E731
    tris = [[0, at(1, i), at(1, i + 1)] for i in range(k)]
    for r in range(1, rings):
        for i in range(k):
            tris += [[at(r, i), at(r + 1, i), at(r + 1, i + 1)], [at(r, i), at(r + 1, i + 1), at(r, i + 1)]]
    edges = [[at(rings, i), at(rings, i + 1)] for i in range(k)]
    return GridMesh(np.array(pts), np.array(tris, np.int32), np.array(edges, np.int32), np.zeros(0, np.int32))


MESHES = {"grid2": lambda: grid_mesh(2, 0.2, 1), "grid13": lambda: grid_mesh(13, 0.25, 2),
          "wheel3": lambda: wheel(3), "wheel7": lambda: wheel(7), "wheel8": lambda: wheel(8),
          "wheel9": lambda: wheel(9), "wheel30": lambda: wheel(30)}


@pytest.mark.gpu
@pytest.mark.parametrize("bucket", [64, 66])
@pytest.mark.parametrize("name", sorted(MESHES))
def test_recovery_matches_the_oracle(oracle_built, name, bucket):
    from tests.oracle_lib import Oracle, tags_of
    from trinity_b200.api import Mesh, Metrics
    m = MESHES[name]()
    u = field_shock(m.points, 7.0, 0.2)
    o = Oracle(m, u, bucket=bucket)
    o.metric(0.8, 2)
    want = o.state().tensor
    g = Mesh((m.nb_nodes, m.nb_elems), bucket, 1, 0, 1, capa_scale=4)
    g.load_arrays(m.points, m.tris, tags_of(m), u)
    g.set_options(exact_sum=True)
    Metrics(g, 0.8, 2).run()
    got = g.export()[1]
    g.close()
    assert np.array_equal(got.view(np.uint64), want.view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("bucket", [64, 66])
@pytest.mark.parametrize("name", ["grid13", "wheel8", "wheel9", "wheel30"])
def test_adjoint_matches_autograd(name, bucket):
    """To 1e-7 of the largest entry: the bound the adjoint has on grids."""
    import torch
    from tests import adjoint_ref
    from tests.oracle_lib import tags_of
    from trinity_b200.api import Mesh
    m = MESHES[name]()
    u = field_shock(m.points, 7.0, 0.2)
    J, gxy, gu = adjoint_ref.gradients(adjoint_ref.Topology(m.points, m.tris), m.points, u, target_factor=0.8, p=2)
    g = Mesh((m.nb_nodes, m.nb_elems), bucket, 1, 0, 1, capa_scale=4)
    g.load_arrays(m.points, m.tris, tags_of(m), u)
    j, a, b = g.quality_adjoint(torch.from_numpy(m.points).cuda(), torch.from_numpy(u).cuda(), target_factor=0.8)
    a, b = a.cpu().numpy(), b.cpu().numpy()
    g.close()
    assert abs(j - J) <= 1e-10 * abs(J)
    assert np.abs(a - gxy).max() <= 1e-7 * np.abs(gxy).max()
    assert np.abs(b - gu).max() <= 1e-7 * np.abs(gu).max()
