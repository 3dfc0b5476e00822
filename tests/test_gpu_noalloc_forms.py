"""The allocation-free recovery where one cluster serves the vertices whose
rows do not fit the registers and where they are too many and the whole chip
does (2,048 of them): the same tensors, bit for bit, as trn_metric_run, with a
smaller mesh after a larger one, and the same refusals."""
import ctypes

import numpy as np
import pytest

from trinity_b200.meshgen import field_multi, grid_mesh

TRN_ERR_CAPACITY, TRN_ERR_INVALID = 1, 3


def cut_in_three(side, jitter=0.1):
    """A grid whose triangles are each cut at their centre: interior vertices
    of 12 elements and of 3."""
    m = grid_mesh(side, jitter, 3)
    n = m.nb_nodes + np.arange(m.nb_elems)
    tris = np.concatenate([np.stack([m.tris[:, i], m.tris[:, (i + 1) % 3], n], 1) for i in range(3)])
    return np.concatenate([m.points, m.points[m.tris].mean(1)]), tris.astype(np.int32)


def noalloc(pts, tris, u):
    import torch
    from trinity_b200._lib import lib
    f = lib().trn_metric_noalloc
    i, d, vp = ctypes.c_int, ctypes.c_double, ctypes.c_void_p
    f.argtypes, f.restype = [i, i, vp, vp, vp, d, i, d, d, vp, vp], i
    t = [torch.from_numpy(a).cuda() for a in (pts, tris, u)]
    out = torch.full((len(pts), 3), float("nan"), dtype=torch.float64, device="cuda")
    rc = f(len(pts), len(tris), t[0].data_ptr(), t[1].data_ptr(), t[2].data_ptr(), 0.8, 2, 1e-9, 0.4, out.data_ptr(),
           torch.cuda.current_stream().cuda_stream)
    return rc, out.cpu().numpy()


def by_mesh(pts, tris, u):
    from trinity_b200.api import Mesh, Metrics
    g = Mesh((len(pts), len(tris)), 64, 1, 0, 1, capa_scale=1)
    g.load_arrays(pts, tris, np.zeros(len(pts), np.uint8), u)
    Metrics(g, 0.8, 2).run()
    ten = g.export()[1]
    g.close()
    return ten


@pytest.mark.gpu
def test_both_forms_give_the_mesh_recovery():
    for side in (70, 25, 26, 4, 72):   # 1,926 and 2,081 vertices on the two sides of the line
        pts, tris = cut_in_three(side)
        u = field_multi(pts)
        rc, got = noalloc(pts, tris, u)
        assert rc == 0
        assert np.array_equal(got.view(np.uint64), by_mesh(pts, tris, u).view(np.uint64)), side


@pytest.mark.gpu
def test_refusals_where_many_rows_are_long():
    pts, tris = cut_in_three(60)
    u = field_multi(pts)
    bad = tris.copy()
    bad[777, 1] = len(pts)
    assert noalloc(pts, bad, u)[0] == TRN_ERR_INVALID
    full = tris.copy()
    full[:40, 0] = 5    # 40 elements and more around one vertex
    assert noalloc(pts, full, u)[0] == TRN_ERR_CAPACITY
    rc, got = noalloc(pts, tris, u)
    assert rc == 0 and np.isfinite(got).all()
