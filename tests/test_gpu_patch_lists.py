"""The metric recovery where more than 32,768 vertices have rows too long for
the registers and each is summed by one lane instead of a warp: FP64 against
the C oracle bit for bit; the mixed form against the same mesh alone, few enough
for warps, when the larger one is four copies of it."""
import numpy as np
import pytest

from tests.test_gpu_noalloc_forms import cut_in_three
from trinity_b200.meshgen import GridMesh, field_multi

NONE = np.zeros((0, 2), np.int32), np.zeros(0, np.int32)


def recover(pts, tris, u, precision, exact=False, target=1.0):
    from trinity_b200.api import Mesh, Metrics
    g = Mesh((len(pts), len(tris)), 64, 1, 0, 1, capa_scale=1)
    g.set_precision(precision)
    g.load_arrays(pts, tris, np.zeros(len(pts), np.uint8), u)
    g.set_options(exact_sum=exact)
    Metrics(g, target, 2).run()
    ten = g.export()[1]
    g.close()
    return ten


@pytest.mark.gpu
@pytest.mark.parametrize("side", [103, 104, 110])   # 32,034, 32,657 and 36,521 vertices, all listed
def test_long_lists_match_the_oracle(oracle_built, side):
    from tests.oracle_lib import Oracle
    pts, tris = cut_in_three(side)
    u = field_multi(pts)
    o = Oracle(GridMesh(pts, tris, *NONE), u, capa_scale=1, bucket=64, tags=np.zeros(len(pts), np.uint8))
    o.metric(0.8, 2)
    got = recover(pts, tris, u, "fp64", True, 0.8)
    assert np.array_equal(got.view(np.uint64), o.state().tensor.view(np.uint64))


@pytest.mark.gpu
@pytest.mark.parametrize("precision,bound", [("fp64", 1e-12), ("mixed", 1e-6)])
def test_copies_recover_what_one_does(precision, bound):
    """Up to the global scale, whose sum over the copies is rounded
    differently: some ulps of the form's arithmetic."""
    pts, tris = cut_in_three(60)
    u = field_multi(pts)
    n = len(pts)
    # exact shifts, so that the copies' differences of coordinates are the same
    scale = 2.0 ** 30
    pts = np.round(pts * scale) / scale
    one = recover(pts, tris, u, precision)
    all4 = recover(np.concatenate([pts + [2.0 * k, 0.0] for k in range(4)]),
                   np.concatenate([tris + k * n for k in range(4)]).astype(np.int32), np.tile(u, 4), precision)
    size = np.abs(one).max(1, keepdims=True)
    for k in range(4):
        assert np.all(np.abs(all4[k * n:(k + 1) * n] - one) <= bound * size)
