"""The adaptation work that the package's speed is measured on: sizes, inputs
and entry points as a solver's program uses them.

A case is a dict; ``kind`` says which entry points one pass goes through:

* ``noalloc``  metric recovery of one small mesh in the caller's own device
  buffers (trn_metric_noalloc): a solver on a fixed memory budget, every
  time step.
* ``metric``   a new nodal field for a loaded mesh, metric recovery, and the
  mesh with its metric back in host memory.
* ``adjoint``  the quality functional with its gradients (forward and
  backward), device tensors in and out: one step of a mesh optimisation.
* ``smooth``   metric recovery, then smart-Laplacian smoothing.
* ``gradient`` metric recovery, then gradient smoothing.
* ``coarsen``  metric recovery with a small target, then edge collapses: a
  mesh that is too fine for its field.
* ``swap``     metric recovery, then edge flips alone: a better
  triangulation of points that have to stay.
* ``adapt``    the whole call: a mesh from host arrays, metric recovery,
  ``rounds`` of refine / coarsen / swap / smooth, the adapted mesh back.
* ``batch``    many meshes of uneven size adapted at once.

Meshes are the unit-square grids of ``trinity_b200.meshgen`` (``side`` quads a
side, interior vertices moved by ``jitter`` of the spacing), fields its shock
and its sum of a shock, a bump and waves. Host arrays are pinned, as a program
that adapts in a loop keeps them.
"""
from __future__ import annotations

import ctypes
import os

# many meshes adapt at once on one stream each; read when CUDA starts
os.environ.setdefault("CUDA_DEVICE_MAX_CONNECTIONS", "32")

import numpy as np
import torch

from trinity_b200 import api, meshgen
from trinity_b200._lib import lib

H_MIN, H_MAX = api.EPSILON, api.H_MAX


def listed():
    return [
        # the smallest call, all latency: a coarse mesh recovered every step
        dict(name="noalloc_20", kind="noalloc", side=20, target=0.9, norm=2),
        # a new field on the 2M-triangle mesh
        dict(name="metric_fp64_1000", kind="metric", side=1000, jitter=0.2, target=0.7, norm=2, precision="fp64"),
        # an ordinary mesh of odd size, metric arithmetic in single precision
        dict(name="metric_mixed_317", kind="metric", side=317, jitter=0.2, target=0.7, norm=2, precision="mixed"),
        # an optimisation step on a large mesh, and a small one in single precision
        dict(name="adjoint_fp64_700", kind="adjoint", side=700, jitter=0.3, target=0.7, norm=2, precision="fp64", recover=True),
        dict(name="adjoint_mixed_151", kind="adjoint", side=151, jitter=0.3, target=0.7, norm=2, precision="mixed", recover=True),
        # the steps of a round called by themselves
        dict(name="smooth_fp64_600", kind="smooth", side=600, jitter=0.2, target=0.7, norm=2, precision="fp64", depth=2),
        dict(name="gradient_fp64_251", kind="gradient", side=251, jitter=0.3, target=0.7, norm=2, precision="fp64", steps=5),
        dict(name="coarsen_mixed_501", kind="coarsen", side=501, jitter=0.2, target=0.3, norm=2, precision="mixed"),
        # the whole call: the small workload (unjittered, one level a round),
        # a million odd triangles in the mixed form, the 2M-triangle workload
        dict(name="adapt_fp64_100", kind="adapt", side=100, jitter=0.0, field="shock", target=0.9, norm=2, precision="fp64",
             rounds=3, depth=1, bucket=64, scale=8),
        dict(name="adapt_mixed_707", kind="adapt", side=707, jitter=0.2, field="multi", target=0.7, norm=2, precision="mixed",
             rounds=3, depth=2, bucket=128, scale=4),
        dict(name="adapt_fp64_1000", kind="adapt", side=1000, jitter=0.2, field="multi", target=0.7, norm=2, precision="fp64",
             rounds=3, depth=2, bucket=128, scale=4),
        # sixteen meshes of 32 to 256 quads a side, as the batched workload has them
        dict(name="batch_16", kind="batch", count=16, lo=32, hi=256, jitter=0.05, target=0.8, norm=2, rounds=3, depth=1, threads=8),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["noalloc", "metric", "metric", "adjoint", "adjoint", "smooth", "gradient", "coarsen", "swap",
                       "adapt", "adapt", "adapt", "batch"])
    precision = rng.choice(["fp64", "fp64", "mixed"])
    jitter = round(rng.uniform(0.05, 0.3), 3)
    if kind == "noalloc":
        return dict(kind=kind, side=_log(rng, 12, 126), target=round(rng.uniform(0.5, 1.0), 3), norm=rng.choice([1, 2, 4]))
    if kind == "batch":
        lo = _log(rng, 32, 64)
        return dict(kind=kind, count=rng.randint(4, 16), lo=lo, hi=_log(rng, 2 * lo, 240), jitter=jitter, target=round(rng.uniform(0.6, 0.9), 3),
                    norm=2, rounds=rng.randint(1, 3), depth=1, threads=rng.choice([4, 8]))
    side = _log(rng, 40, 900 if kind != "gradient" else 300)
    case = dict(kind=kind, side=side, jitter=jitter, target=round(rng.uniform(0.5, 0.9), 3), norm=rng.choice([1, 2, 4]), precision=precision)
    if kind == "adjoint":
        case.update(recover=rng.random() < 0.75)
    elif kind == "smooth":
        case.update(depth=rng.randint(1, 3))
    elif kind == "gradient":
        case.update(steps=rng.randint(2, 8))
    elif kind == "coarsen":
        case.update(target=round(rng.uniform(0.2, 0.5), 3))
    elif kind == "adapt":
        depth = rng.randint(1, 2)
        case.update(side=_log(rng, 40, 800), field="multi" if depth == 2 else rng.choice(["shock", "multi"]), norm=2,
                    rounds=rng.randint(1, 3), depth=depth, bucket=128, scale=8)
    return case


# ------------------------------------------------------------------ inputs
def _tags(m):
    """Boundary vertices 4, corners 12."""
    t = np.zeros(m.nb_nodes, np.uint8)
    t[m.edges.ravel()] = 4
    t[m.corners] = 12
    return t


def _pinned(a):
    t = torch.empty(a.shape, dtype=torch.from_numpy(a[:0]).dtype, pin_memory=True)
    t.numpy()[...] = a
    return t.numpy()


def _mesh_of(case, seed):
    m = meshgen.grid_mesh(case["side"], case.get("jitter", 0.0), seed)
    r = np.random.default_rng(seed)
    if case.get("field", "multi" if case.get("jitter") else "shock") == "shock":
        u = meshgen.field_shock(m.points, r.uniform(40.0, 60.0), r.uniform(0.2, 0.3))
    else:
        u = meshgen.field_multi(m.points)
    return m, u


def _out(nv, nt):
    """Where the adapted mesh goes: points, triangles, metric."""
    return tuple(torch.zeros(s, dtype=d, pin_memory=True).numpy()
                 for s, d in (((nv, 2), torch.float64), ((nt, 3), torch.int32), ((nv, 3), torch.float64)))


# the coarsest meshes under the steepest shocks grow more than the batched
# workload's own eight-fold, for some of the shocks that a seed draws
_BATCH_SCALE = 16


def _batch_inputs(case, seed):
    """The sides are the case's; the shocks come from the seed. The vertices
    are moved a little: on an exact grid two triangles can be exactly as good
    either way round, and once in some thousand meshes flip without end."""
    r = np.random.default_rng(seed)
    for side, _, _ in meshgen.batch_specs(case["count"], 5, case["lo"], case["hi"]):
        m = meshgen.grid_mesh(side, case["jitter"], seed)
        yield m, meshgen.field_shock(m.points, r.uniform(10.0, 100.0), r.uniform(0.0, 0.3))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        p = meshgen.BATCH_PARAMS
        meshes = []
        for m, u in _batch_inputs(case, seed):
            g = api.Mesh((m.nb_nodes, m.nb_elems), p["bucket"], case["depth"], 0, case["rounds"], capa_scale=_BATCH_SCALE)
            g.load_arrays(m.points, m.tris, _tags(m), u)
            g.set_swap_match(p["swap_match"])
            meshes.append(g)
        # one buffer for all meshes, each at its own offset
        room = np.cumsum([(0, 0)] + [(8 * n, 8 * t) for n, t in (g.counts()[:2] for g in meshes)], axis=0)
        out = _out(*room[-1])
        outs = [(out[0][a:c], out[1][b:d], out[2][a:c]) for (a, b), (c, d) in zip(room[:-1], room[1:])]
        return dict(case=case, meshes=meshes, out=out, outs=outs)
    m, u = _mesh_of(case, seed)
    if kind == "noalloc":
        dev = torch.device("cuda")
        f = lib().trn_metric_noalloc
        i, d, vp = ctypes.c_int, ctypes.c_double, ctypes.c_void_p
        f.argtypes, f.restype = [i, i, vp, vp, vp, d, i, d, d, vp, vp], i
        return dict(case=case, call=f, nv=m.nb_nodes, nt=m.nb_elems, pts=torch.from_numpy(m.points).to(dev),
                    tris=torch.from_numpy(m.tris).to(dev), u=torch.from_numpy(u).to(dev),
                    ten=torch.empty((m.nb_nodes, 3), dtype=torch.float64, device=dev))
    depth, rounds = case.get("depth", 1), case.get("rounds", 1)
    g = api.Mesh((m.nb_nodes, m.nb_elems), case.get("bucket", 128), depth, 0, rounds, capa_scale=case.get("scale", 4))
    if kind != "adjoint":
        g.set_precision(case["precision"])
    arrays = (m.points, m.tris, _tags(m), u)
    s = dict(case=case, mesh=g, metric=api.Metrics(g, case["target"], case["norm"]))
    heur = api.Partit(g, 8)
    if kind == "adapt":
        s["arrays"] = tuple(_pinned(a) for a in arrays)
        s["steps"] = [api.Refine(g, depth), api.Coarse(g, heur), api.Swap(g), api.Smooth(g, heur, depth)]
        s["out"] = _out(2 * m.nb_nodes + 20000, 2 * m.nb_elems + 40000)
        return s
    g.load_arrays(*arrays)
    if kind == "metric":
        s["u"] = _pinned(u)
    elif kind == "adjoint":
        s["metric"].run()   # the metric of a fixed-metric call
        s["xy"] = torch.from_numpy(m.points).cuda()
        s["u"] = torch.from_numpy(u).cuda() if case["recover"] else None
        return s
    elif kind == "smooth":
        s["steps"] = [api.Smooth(g, heur, depth)]
    elif kind == "gradient":
        s["steps"] = [api.GradientSmooth(g, heur, case["steps"])]
    elif kind == "coarsen":
        s["steps"] = [api.Coarse(g, heur)]
    elif kind == "swap":
        s["steps"] = [api.Swap(g)]
    s["out"] = _out(m.nb_nodes, m.nb_elems)
    return s


def _fetch(g, out):
    """The adapted mesh in its leading rows of the program's buffers."""
    points, tris, _ = g.export_compact(out=out)
    return dict(vertices=points.shape[0], triangles=tris.shape[0], points=out[0], tris=out[1], tensor=out[2])


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "noalloc":
        rc = s["call"](s["nv"], s["nt"], s["pts"].data_ptr(), s["tris"].data_ptr(), s["u"].data_ptr(), case["target"],
                       case["norm"], H_MIN, H_MAX, s["ten"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError(f"trn_metric_noalloc: {rc}")
        return dict(tensor=s["ten"])
    if kind == "batch":
        for g in s["meshes"]:
            g.reload()
        api.batch_adapt(s["meshes"], case["target"], case["norm"], case["rounds"], case["depth"], threads=case["threads"])
        sizes = [[a.shape[0] for a in g.export_compact(out=o)[:2]] for g, o in zip(s["meshes"], s["outs"])]
        return dict(sizes=np.array(sizes), points=s["out"][0], tris=s["out"][1], tensor=s["out"][2])
    g = s["mesh"]
    if kind == "adjoint":
        J, gxy, gu = g.quality_adjoint(s["xy"], s["u"], target_factor=case["target"], Lp_norm=case["norm"],
                                       precision=case["precision"])
        return dict(J=J, gxy=gxy, gu=gu)
    if kind == "metric":
        g.set_solution(s["u"])
        s["metric"].run()
        return _fetch(g, s["out"])
    if kind == "adapt":
        g.load_arrays(*s["arrays"])
    else:
        g.reload()
    s["metric"].run()
    for _ in range(case.get("rounds", 1)):
        for k in s["steps"]:
            k.run()
    return _fetch(g, s["out"])


def work(case):
    """Inputs once, outputs once; operations: per element its gradient and
    Hessian terms (100) and quality (150), per vertex the patch sums, tensor
    functions and moves, per recovery, pass or round."""
    kind = case["kind"]
    if kind == "batch":
        sides = [s for s, _, _ in meshgen.batch_specs(case["count"], 5, case["lo"], case["hi"])]
    else:
        sides = [case["side"]]
    V = sum((s + 1) ** 2 for s in sides)
    T = sum(2 * s * s for s in sides)
    recover = V * 600.0 + T * 100.0
    if kind in ("noalloc", "metric"):
        return dict(bytes=V * (16 + 8 + 24) + T * 12 + (T * 12 + V * 16 if kind == "metric" else 0), flops=recover)
    if kind == "adjoint":
        back = 2.0 if case["recover"] else 0.0
        return dict(bytes=V * (16 + 16 + 24 + (16 if back else 0)) + T * 12, flops=back * recover + T * 400.0)
    io = V * (16 + 8 + 1) + T * 12 + V * (16 + 24) + T * 12
    if kind in ("coarsen", "swap"):
        return dict(bytes=io, flops=recover + V * 1500.0)
    if kind in ("smooth", "gradient"):
        passes = case["depth"] if kind == "smooth" else case["steps"]
        return dict(bytes=io, flops=recover + passes * V * 3000.0)
    return dict(bytes=io, flops=recover + case["rounds"] * (V * 3000.0 + case["depth"] * V * 3000.0))


# ------------------------------------------------------------------ in 64 bits
def _eig(a, b, c):
    """Eigenvalues (descending in the pair's own order) and unit vectors of
    [[a, b], [b, c]]; a tensor with b*b < 1e-9 counts as diagonal, as the
    recovery's definition has it."""
    diag = (b * b < 1e-9).detach()
    bs = torch.where(diag, torch.ones_like(b), b)
    root = torch.sqrt(0.25 * (a - c) ** 2 + bs * bs)
    mid = 0.5 * (a + c)
    x = torch.where((a >= c).detach(), 0.5 * (a - c) + root, bs)
    y = torch.where((a >= c).detach(), bs, 0.5 * (c - a) + root)
    n = torch.sqrt(x * x + y * y)
    one, zero = torch.ones_like(a), torch.zeros_like(a)
    l0, l1 = torch.where(diag, a, mid + root), torch.where(diag, c, mid - root)
    return l0, l1, torch.where(diag, one, x / n), torch.where(diag, zero, y / n)


def _tensor(l0, l1, x, y):
    """l0 (x,y)(x,y)^T + l1 (-y,x)(-y,x)^T as (m11, m12, m22)."""
    return l0 * x * x + l1 * y * y, (l0 - l1) * x * y, l0 * y * y + l1 * x * x


class _Patches:
    """The means over the elements around a vertex and around its neighbours."""

    def __init__(self, pts, tri):
        V, T = pts.shape[0], tri.shape[0]
        e = torch.cat([tri[:, [0, 1]], tri[:, [1, 2]], tri[:, [2, 0]]])
        e = torch.cat([e, e.flip(1)])
        edge = torch.unique(e[:, 0] * V + e[:, 1])
        src, dst = edge // V, edge % V
        # vertices beside each corner of each element, itself among them
        deg = torch.bincount(src, minlength=V)
        off = torch.cumsum(deg, 0) - deg
        corner = tri.reshape(-1)
        el = torch.arange(T, device=tri.device).repeat_interleave(3)
        n = deg[corner]
        at = torch.arange(int(n.sum()), device=tri.device) - (torch.cumsum(n, 0) - n).repeat_interleave(n)
        v = torch.cat([corner, dst[off[corner].repeat_interleave(n) + at]])
        el = torch.cat([el, el.repeat_interleave(n)])
        key = torch.unique(v * T + el)
        self.v, self.e, self.V, self.tri = key // T, key % T, V, tri
        p = pts[tri]
        self.area = 0.5 * ((p[:, 1, 0] - p[:, 0, 0]) * (p[:, 2, 1] - p[:, 0, 1]) - (p[:, 2, 0] - p[:, 0, 0]) * (p[:, 1, 1] - p[:, 0, 1]))
        q = torch.stack([p[:, [1, 2, 0], 1] - p[:, [2, 0, 1], 1], p[:, [2, 0, 1], 0] - p[:, [1, 2, 0], 0]], 2)
        self.basis = q * (2 / self.area)[:, None, None]   # four times the P1 gradients
        self.total = self._sum(self.area[:, None])

    def _sum(self, f):
        return torch.zeros((self.V, f.shape[1]), dtype=f.dtype, device=f.device).index_add(0, self.v, f[self.e])

    def mean(self, f):
        return self._sum(f * self.area[:, None]) / self.total


def _recover(P, u, target, norm):
    g = P.mean((u[P.tri][:, :, None] * P.basis).sum(1))
    h = P.mean((g[P.tri][:, :, :, None] * P.basis[:, :, None, :]).sum(1).reshape(-1, 4))
    l0, l1, x, y = _eig(h[:, 0], 0.5 * (h[:, 1] + h[:, 2]), h[:, 3])
    l0, l1 = torch.clamp(l0.abs(), min=1e-9), torch.clamp(l1.abs(), min=1e-9)
    s = (l0 * l1) ** (-1.0 / (2 * norm + 2))
    a, b, c = _tensor(l0 * s, l1 * s, x, y)
    density = torch.sqrt(a * c - b * b)[P.tri].sum(1) / 3
    scale = float(int(np.floor(P.V * target))) / (density * P.area).sum()
    l0, l1, x, y = _eig(a, b, c)
    lo, hi = 1 / H_MAX ** 2, 1 / H_MIN ** 2
    return _tensor(torch.clamp(l0 * scale, lo, hi), torch.clamp(l1 * scale, lo, hi), x, y)


def _quality(xy, tri, ten):
    l0, l1, x, y = _eig(*ten)
    lt = torch.stack(_tensor(torch.log(l0), torch.log(l1), x, y), 1)
    mean = lt[tri].sum(1) / 3
    l0, l1, x, y = _eig(mean[:, 0], mean[:, 1], mean[:, 2])
    a, b, c = _tensor(torch.exp(l0), torch.exp(l1), x, y)
    p = xy[tri]
    d = p[:, [1, 2, 0]] - p
    ln = torch.sqrt(a[:, None] * d[:, :, 0] ** 2 + 2 * b[:, None] * d[:, :, 0] * d[:, :, 1] + c[:, None] * d[:, :, 1] ** 2)
    perim = ln.sum(1)
    area = 0.5 * (d[:, 0, 0] * -d[:, 2, 1] + d[:, 2, 0] * d[:, 0, 1]).abs()
    m = torch.minimum(perim / 3, 3 / perim)
    return area * 12 * np.sqrt(3.0) * (m * (2 - m)) ** 3 * torch.sqrt(a * c - b * b) / perim ** 2


def exact(case, seed):
    if case["kind"] not in ("noalloc", "metric", "adjoint"):
        return None   # the meshes that rounds end with are the heuristics' choices
    m, u = _mesh_of(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    pts, tri = torch.from_numpy(m.points).to(dev), torch.from_numpy(m.tris).to(dev).long()
    u = torch.from_numpy(u).to(dev)
    P = _Patches(pts, tri)
    if case["kind"] != "adjoint":
        ten = torch.stack(_recover(P, u, case["target"], case["norm"]), 1)
        return dict(tensor=ten) if case["kind"] == "noalloc" else dict(vertices=None, triangles=None, points=pts, tris=None, tensor=ten)
    xy = pts.clone().requires_grad_(True)
    u = u.requires_grad_(case["recover"])
    J = _quality(xy, tri, _recover(P, u, case["target"], case["norm"])).sum()
    J.backward()
    return dict(J=float(J.detach()), gxy=xy.grad, gu=u.grad)
