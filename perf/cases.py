"""The framework's work as measured cases: elastic boundary-element operator
applies, their farfields (direct, panels of right-hand sides, fast multipole),
interior evaluation, nearfield assembly and a constrained solve, each through
the entry point a program calls.

A case is a dict of plain values; `kind` says which entry point it goes through:

  apply     RegularizedSparseIntegralOp.dot: one full operator apply, as a
            Krylov solver or a time stepper makes it
  far       TriToTriDirectFarfieldOp.dot: the direct farfield alone (all
            seven kernels; one surface on itself, or a fault's slip seen on
            a surface)
  panel     TriToTriDirectFarfieldOp.dot_panel_device: the farfield of many
            right-hand sides at once (batched and served solves)
  fmm       FMMFarfieldOp: the treecode / FMM farfield of large meshes
  interior  InteriorOp.dot: a boundary field evaluated at points off the
            surface
  nearfield RegularizedNearfieldIntegralOp: the singular and near-singular
            pair integrals of an operator build (a remeshed or moved surface)
  solve     iterative_solve: a constrained FP64 GMRES solve

Device arrays in, device arrays out, except where the call takes host arrays
by its nature (nearfield, solve).  Meshes: seeded topographic surfaces over
[-10, 10]^2 (grid spacing and relief of the 59,858-triangle benchmark
surface, cut to any triangle count), planar faults, and surfaces with a
dipping fault below.
"""
import math

import numpy as np
import torch

from tectosaur_b200.fmm.tsfmm import FMMFarfieldOp
from tectosaur_b200.interior import InteriorOp
from tectosaur_b200.mesh.mesh_gen import concat_no_dedupe, make_rect
from tectosaur_b200.nearfield.nearfield_op import RegularizedNearfieldIntegralOp
from tectosaur_b200.ops.sparse_farfield_op import TriToTriDirectFarfieldOp
from tectosaur_b200.ops.sparse_integral_op import RegularizedSparseIntegralOp
from tectosaur_b200.simple_solver import (free_edge_vertices, iterative_solve,
                                          shared_vertex_matrix)

PARAMS = [1.0, 0.25]          # shear modulus, Poisson's ratio
KERNELS = {"U": "elasticU3", "T": "elasticT3", "A": "elasticA3", "H": "elasticH3",
           "RT": "elasticRT3", "RA": "elasticRA3", "RH": "elasticRH3"}
# quadrature orders (coincident, edge, vertex, near) and near threshold of
# every configuration of the repository
NQ_CO, NQ_EA, NQ_VA, NQ_NEAR, NEAR = 6, 6, 6, 5, 2.5
# points of the far rule by order, and FMA-counted operations per ordered
# point pair of the hoisted forms (bench.py's and the reference's own counts)
RULE_PTS = {1: 3, 2: 4, 3: 7}
PAIR_FLOPS = {"U": 28, "T": 63, "A": 63, "H": 102, "RT": 45, "RA": 45, "RH": 36}


def listed():
    return [
        # one FP64 apply on the smallest configuration (722 triangles): a
        # GMRES step of the plain solve, where launches and latency count
        dict(name="apply-rh-f64-722", kind="apply", kernel="RH", dtype="f64", n=722, nq_far=2),
        # the headline configuration: FP32 apply of 59,858 triangles, direct
        # farfield on all pairs + nearfield blocks
        dict(name="apply-rh-f32-59858", kind="apply", kernel="RH", dtype="f32", n=59858, nq_far=1),
        # FP64 residual of a mixed-precision solve on a mid-size mesh
        dict(name="far-rh-f64-12290", kind="far", kernel="RH", dtype="f64", n=12290, n_src=0,
             nq_far=2),
        # displacement/traction of fault slip on a surface: two different
        # triangle sets, odd sizes
        dict(name="far-rt-f32-9461x2311", kind="far", kernel="RT", dtype="f32", n=9461, n_src=2311,
             nq_far=1),
        # an unregularised kernel on one surface (the reference's default
        # kernels), FP32
        dict(name="far-h-f32-5003", kind="far", kernel="H", dtype="f32", n=5003, n_src=0,
             nq_far=1),
        # 16 right-hand sides of a served mesh, one tensor-core panel
        dict(name="panel-rh-f32-16x32258", kind="panel", kernel="RH", dtype="f32", n=32258, rhs=16,
             nq_far=2),
        # a ragged panel (11 right-hand sides) of the other regularised kernel
        dict(name="panel-rt-f32-11x7441", kind="panel", kernel="RT", dtype="f32", n=7441, rhs=11,
             nq_far=1),
        # FP32 FMM apply of a large surface + fault mesh
        dict(name="fmm-rh-f32-p8-119656", kind="fmm", kernel="RH", dtype="f32", n=119656, nq_far=1,
             order=8, mode="fmm", leaf=128),
        # FP64 FMM apply: the residual of a solve on a large mesh
        dict(name="fmm-rh-f64-p10-72200", kind="fmm", kernel="RH", dtype="f64", n=72200, nq_far=2,
             order=10, mode="fmm", leaf=128),
        # displacements at points in the volume from slip on the surface
        dict(name="interior-t-f32-2500x1682", kind="interior", kernel="T", dtype="f32", n=1682,
             points=2500, nq_far=2),
        # pair integrals of an operator build
        dict(name="nearfield-rh-f64-3042", kind="nearfield", kernel="RH", dtype="f64", n=3042,
             nq_far=2),
        # the whole plain solve: continuity + free edges, FP64 to 1e-8
        dict(name="solve-rh-f64-722", kind="solve", kernel="RH", dtype="f64", n=722, nq_far=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply", "far", "far", "panel", "fmm", "interior", "nearfield"])
    dt = rng.choice(["f32", "f64"])
    if kind == "apply":
        return dict(kind=kind, kernel="RH", dtype=dt,
                    n=_log_int(rng, 300, 45000 if dt == "f32" else 12000),
                    nq_far=rng.choice([1, 2]))
    if kind == "far":
        K = rng.choice(["U", "T", "A", "H", "RT", "RA", "RH", "RH"])
        hi = 16000 if dt == "f32" else 5000
        return dict(kind=kind, kernel=K, dtype=dt, n=_log_int(rng, 200, hi),
                    n_src=rng.choice([0, 0, _log_int(rng, 200, hi)]),
                    nq_far=rng.choice([1, 1, 2, 3]))
    if kind == "panel":
        K = rng.choice(["RH", "RH", "RT"])
        return dict(kind=kind, kernel=K, dtype="f32", n=_log_int(rng, 700, 30000),
                    rhs=rng.randint(2, 24), nq_far=1 if K == "RT" else rng.choice([1, 2, 3]))
    if kind == "fmm":
        return dict(kind=kind, kernel=rng.choice(["U", "RT", "RA", "RH", "RH", "RH"]), dtype=dt,
                    n=_log_int(rng, 8000, 110000 if dt == "f32" else 60000),
                    nq_far=rng.choice([1, 2]), order=rng.choice([6, 8, 10]),
                    mode=rng.choice(["fmm", "fmm", "treecode"]), leaf=rng.choice([64, 128]))
    if kind == "interior":
        return dict(kind=kind, kernel=rng.choice(["U", "T", "A", "H"]), dtype=dt,
                    n=_log_int(rng, 300, 8000), points=_log_int(rng, 500, 10000),
                    nq_far=rng.choice([1, 2, 3]))
    return dict(kind=kind, kernel="RH", dtype=dt, n=_log_int(rng, 400, 8000),
                nq_far=rng.choice([1, 2]))


# ---- inputs ---------------------------------------------------------------------

def _surface(n, rng, half=10.0):
    """A topographic surface of n triangles over [-half, half]^2 (single
    precision coordinates, so both precisions see the same mesh)."""
    cells = max(1, int(math.ceil(n / 2)))
    nx = int(math.ceil(math.sqrt(cells)))
    ny = int(math.ceil(cells / nx))
    pts, tris = make_rect(nx + 1, ny + 1, [[-half, -half, 0], [half, -half, 0],
                                           [half, half, 0], [-half, half, 0]])
    pts = np.array(pts, dtype=np.float64)
    h = 2.0 * half / max(nx, ny)
    # the benchmark surface's hill and roughness (0.17 of the grid spacing)
    pts[:, 2] = (0.05 * half * np.exp(-(pts[:, 0] ** 2 + pts[:, 1] ** 2) / (0.08 * half * half))
                 + 0.17 * h * rng.standard_normal(pts.shape[0]))
    return pts.astype(np.float32).astype(np.float64), np.asarray(tris)[:n].copy()


def _fault(n, half=5.0):
    """A plane dipping 30 degrees below the surface, n triangles."""
    cells = max(1, int(math.ceil(n / 2)))
    nx = int(math.ceil(math.sqrt(cells)))
    ny = int(math.ceil(cells / nx))
    y1, z1 = 2 * half * math.cos(math.pi / 6), -1.0 - 2 * half * math.sin(math.pi / 6)
    pts, tris = make_rect(nx + 1, ny + 1, [[-half, -half, -1.0], [half, -half, -1.0],
                                           [half, -half + y1, z1], [-half, -half + y1, z1]])
    pts = np.array(pts, dtype=np.float64)
    return pts.astype(np.float32).astype(np.float64), np.asarray(tris)[:n].copy()


def _inputs(case, seed):
    """(pts, tris, obs, src, x): mesh, triangle subsets and the input vectors
    (a host FP64 array holding single precision values)."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    kind = case["kind"]
    if kind == "fmm":
        n_f = n // 4
        pts, tris = concat_no_dedupe(_surface(n - n_f, rng), _fault(n_f))
        obs = src = np.arange(n)
    elif kind == "far" and case["n_src"]:
        pts, tris = concat_no_dedupe(_surface(n, rng), _fault(case["n_src"]))
        obs, src = np.arange(n), np.arange(n, n + case["n_src"])
    elif kind == "solve":
        # the solve's planar fault: the grid stays regular, the load is seeded
        g = int(round(math.sqrt(n / 2.0))) + 1
        pts, tris = make_rect(g, g, [[-1, -1, 0], [-1, 1, 0], [1, 1, 0], [1, -1, 0]])
        pts, tris = np.asarray(pts, np.float64), np.asarray(tris)
        obs = src = np.arange(tris.shape[0])
    elif kind == "nearfield":
        # one surface (the block structure follows from it); the seed draws
        # the elastic parameters the blocks hold
        pts, tris = _surface(n, np.random.default_rng(n), half=1.0)
        obs = src = np.arange(n)
    elif kind == "apply" and n < 2000:
        pts, tris = _surface(n, rng, half=1.0)
        obs = src = np.arange(n)
    else:
        pts, tris = _surface(n, rng)
        obs = src = np.arange(n)
    R = case.get("rhs", 1)
    x = rng.standard_normal((R, 9 * src.shape[0])).astype(np.float32).astype(np.float64)
    return pts, tris, obs, src, (x if kind == "panel" else x[0]), rng


def _interior_points(case, rng):
    """Points over the fault area, more than four triangle sizes off it."""
    n = case["points"]
    p = rng.uniform(-9.0, 9.0, (n, 3))
    p[:, 2] = 4.5 * 20.0 / math.sqrt(case["n"] / 2.0) + 1.0 + rng.uniform(0.0, 3.0, n)
    ns = rng.standard_normal((n, 3))
    ns /= np.linalg.norm(ns, axis=1)[:, None]
    f = lambda a: a.astype(np.float32).astype(np.float64)  # noqa: E731
    return f(p), f(ns)


def _ft(case):
    return np.float32 if case["dtype"] == "f32" else np.float64


def _dev(a, case):
    return torch.from_numpy(np.ascontiguousarray(a)).to("cuda").to(
        torch.float32 if case["dtype"] == "f32" else torch.float64)


def prepare(case, seed):
    pts, tris, obs, src, x, rng = _inputs(case, seed)
    K, ft, kind = KERNELS[case["kernel"]], _ft(case), case["kind"]
    if kind in ("apply", "solve"):
        op = RegularizedSparseIntegralOp(
            NQ_CO, NQ_EA, NQ_VA, case["nq_far"], NQ_NEAR, NEAR, K, K, PARAMS, pts, tris, ft,
            TriToTriDirectFarfieldOp, keep_uncorrected=False)
        if kind == "solve":
            cm = shared_vertex_matrix(tris, free_edge_vertices(tris))
            return dict(kind=kind, op=op, cm=cm, rhs=x)
        return dict(kind=kind, op=op, x=_dev(x, case))
    if kind == "far":
        op = TriToTriDirectFarfieldOp(case["nq_far"], K, PARAMS, pts, tris, ft, obs, src)
        return dict(kind=kind, op=op, x=_dev(x, case))
    if kind == "panel":
        op = TriToTriDirectFarfieldOp(case["nq_far"], K, PARAMS, pts, tris, ft, obs, src)
        X = _dev(x, case)
        return dict(kind=kind, op=op, x=X, y=torch.empty_like(X))
    if kind == "fmm":
        op = FMMFarfieldOp(3.0, case["leaf"], case["order"], mode=case["mode"])(
            case["nq_far"], K, PARAMS, pts, tris, ft, obs, src)
        return dict(kind=kind, op=op, x=_dev(x, case))
    if kind == "interior":
        p, ns = _interior_points(case, rng)
        op = InteriorOp(p, ns, (pts, tris), K, 4.0, 6, case["nq_far"], NQ_NEAR, PARAMS, ft)
        return dict(kind=kind, op=op, x=_dev(x, case))
    params = [float(rng.uniform(0.5, 2.0)), float(rng.uniform(0.1, 0.4))]
    return dict(kind=kind, args=(pts, tris, obs, src, NQ_CO, NQ_EA, NQ_VA, case["nq_far"], NQ_NEAR,
                                 NEAR, K, K, params, ft))


def run(state):
    kind = state["kind"]
    if kind == "panel":
        return state["op"].dot_panel_device(state["x"], state["y"])
    if kind == "nearfield":
        op = RegularizedNearfieldIntegralOp(*state["args"], keep_uncorrected=False)
        return dict(blocks=op.bsr.data, indices=op.bsr.indices, indptr=op.bsr.indptr)
    if kind == "solve":
        return iterative_solve(state["op"], state["cm"], state["rhs"])
    return state["op"].dot(state["x"])


# ---- what a pass cannot do without ------------------------------------------------

# near pairs per triangle at threshold 2.5 on these surfaces (5,477,848 blocks
# of 59,858 triangles on the benchmark surface), by class, and the points of
# their rules: coincident / edge / vertex rules of order 6, near rule 361
NEAR_PER_TRI = 91.5
NEAR_CLASS_POINTS = (1 * 2592 + 3 * 6480 + 9 * 2592) + (NEAR_PER_TRI - 13) * 361


def work(case):
    kind, n = case["kind"], case["n"]
    r = 4 if case["dtype"] == "f32" else 8
    q = RULE_PTS[case["nq_far"]]
    f = PAIR_FLOPS[case["kernel"]]
    far = lambda no, ns: float(no) * ns * q * q * f  # noqa: E731
    mesh = lambda m: m * (12 + 1.5 * r)  # noqa: E731  triangles + vertices
    if kind == "apply":
        near = n * NEAR_PER_TRI
        return dict(bytes=near * (81 * r + 4) + 18.0 * r * n + mesh(n),
                    flops=far(n, n) + near * 162)
    if kind == "far":
        m = case["n_src"] or n
        return dict(bytes=9.0 * r * (n + m) + mesh(n + m), flops=far(n, m))
    if kind == "panel":
        # the geometry of a pair once, then its 3x3 products per vector
        return dict(bytes=18.0 * r * n * case["rhs"] + mesh(n),
                    flops=float(n) * n * (q * q * 29 + 63 * case["rhs"]))
    if kind == "fmm":
        # linear in n: near leaves pair by pair (27 leaves of leaf/2
        # triangles), expansions of (p+1)(p+2)(p+3)/6 terms over 189 boxes
        # of the interaction list a leaf
        p = case["order"]
        terms = (p + 1) * (p + 2) * (p + 3) * (p + 4) * (p + 5) * (p + 6) / 720.0
        leaf = case["leaf"] / 2.0
        return dict(bytes=18.0 * r * n + mesh(n),
                    flops=far(n, 27 * leaf) + (n / leaf) * 189 * terms * 42)
    if kind == "interior":
        m = case["points"]
        return dict(bytes=r * (9.0 * n + 6.0 * m) + 8.0 * 3 * m + mesh(n), flops=float(n) * m * q * f)
    if kind == "nearfield":
        return dict(bytes=n * NEAR_PER_TRI * (81 * r + 4) + mesh(n),
                    flops=n * NEAR_CLASS_POINTS * 200.0)
    # solve: about 25 applies of the operator
    return dict(bytes=25 * n * NEAR_PER_TRI * (81 * r + 4), flops=25 * (far(n, n) + n * NEAR_PER_TRI * 162))


def tolerance(case):
    kind = case["kind"]
    if kind == "solve":
        # iterates that both meet the 1e-8 residual (1.5e-8 from the 1e-12 one)
        return dict(rel=1e-7)
    if case["dtype"] == "f64":
        return dict(rel=1e-11)
    # FP32: about four times the distance seen from the 64-bit values
    if kind == "fmm":
        return dict(rel=3e-5)   # rounding of the expansions: 3e-6 to 7e-6
    if kind == "panel":
        return dict(rel=3e-5)   # split TF32 products: 3e-6 to 7e-6
    if kind == "nearfield":
        return dict(rel=1.5e-5)  # batched and per-class sums: 3.4e-6 apart
    if kind == "far" and case["kernel"] in ("T", "A"):
        return dict(rel=2e-5)   # r^-2 at touching triangles
    if kind == "far" and case["kernel"] == "H":
        return dict(rel=8e-5)   # r^-3 at touching triangles: 7e-6 to 2e-5
    return dict(rel=1e-5)


# ---- 64-bit values -----------------------------------------------------------------

def _rule(order):
    """The triangle rules of degree 2, 3 and 5 (3, 4 and 7 points) on the unit
    triangle, weights summing to 1/2."""
    if order == 1:
        a = [(2 / 3, 1 / 6), (1 / 6, 2 / 3), (1 / 6, 1 / 6)]
        return np.array(a), np.full(3, 1 / 6)
    if order == 2:
        a = [(1 / 3, 1 / 3), (0.6, 0.2), (0.2, 0.6), (0.2, 0.2)]
        return np.array(a), np.array([-27, 25, 25, 25]) / 96.0
    s = math.sqrt(15.0)
    out, w = [(1 / 3, 1 / 3)], [9 / 80.0]
    for sg in (-1, 1):
        c = (6 + sg * s) / 21
        out += [(1 - 2 * c, c), (c, 1 - 2 * c), (c, c)]
        w += [(155 + sg * s) / 2400.0] * 3
    return np.array(out), np.array(w)


def _t(a):
    return torch.as_tensor(np.asarray(a, dtype=np.float64), device="cuda")


class _Tris:
    """Geometry of triangles in 64 bits: rule points, normal, Jacobian,
    surface curls of the basis."""

    def __init__(self, pts, tris, order):
        v = _t(np.asarray(pts)[np.asarray(tris)])
        q, w = _rule(order)
        self.b = _t(np.stack([1 - q[:, 0] - q[:, 1], q[:, 0], q[:, 1]], axis=1))  # (q, 3)
        self.w = _t(w)
        e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        un = torch.linalg.cross(v[:, 2] - v[:, 0], v[:, 2] - v[:, 1])
        self.J = torch.linalg.norm(un, dim=1)
        self.nrm = un / self.J[:, None]
        self.sc = torch.stack([e1 - e2, e2, -e1], dim=1) / self.J[:, None, None]  # (n, basis, 3)
        self.x = torch.einsum("qb,nbd->nqd", self.b, v)
        self.n, self.q = v.shape[0], q.shape[0]


def _inv(x, y):
    """1 / |y - x| for all pairs, 0 where the points coincide."""
    r2 = (x[:, 0:1] - y[None, :, 0]).square_()
    for d in (1, 2):
        D = x[:, d:d + 1] - y[None, :, d]
        r2.addcmul_(D, D)
    inv = r2.rsqrt_()
    return inv.masked_fill_(torch.isinf(inv), 0.0)


def _blocks(n_x, n_y, rows=8192, cols=16384):
    for i in range(0, n_x, rows):
        for j in range(0, n_y, cols):
            yield slice(i, i + rows), slice(j, j + cols)


def _point_field(K, x, nx, y, ny, a, step=1 << 25):
    """sum_y K(x, y) a(y) of the U/T/A/H point kernels, pairs with r = 0 left
    out."""
    mu, nu = PARAMS
    out = torch.empty_like(x)
    rows = max(1, step // max(1, y.shape[0]))
    dot = lambda u, v: (u * v).sum(-1)  # noqa: E731
    for i in range(0, x.shape[0], rows):
        D = y[None] - x[i:i + rows, None]
        inv = _inv(x[i:i + rows], y)
        s = a[None]
        N, M = ny[None], nx[i:i + rows, None]
        if K == "U":
            c = 1 / (16 * math.pi * mu * (1 - nu))
            v = (c * inv)[..., None] * ((3 - 4 * nu) * s + (dot(D, s) * inv ** 2)[..., None] * D)
        elif K in ("T", "A"):
            c0, c1 = (1 - 2 * nu) / (8 * math.pi * (1 - nu)), 3 / (8 * math.pi * (1 - nu))
            nn, sg = (N, -1.0) if K == "T" else (M, 1.0)
            rn, ds = dot(nn, D), dot(D, s)
            nb = nn.expand(D.shape)
            # c0 r^-3 (-(n.D) s + s' ((n.s) D - (D.s) n)) and c1 r^-5 (n.D)(D.s) D
            t = -rn[..., None] * s + sg * (ds[..., None] * nb - dot(nn, s)[..., None] * D)
            v = (-sg * c0 * inv ** 3)[..., None] * t + (sg * c1 * inv ** 5 * rn * ds)[..., None] * D
        else:
            Q = mu / (4 * math.pi * (1 - nu)) * inv ** 3
            rn, rm = inv * dot(N, D), inv * dot(M, D)
            mn, sn, sm = dot(M, N), dot(s, N), dot(s, M)
            sd = inv * dot(s, D)
            A, B, C = Q * 3 * rn, Q * (1 - 2 * nu), Q * 3 * nu
            MT = Q * (-1 + 4 * nu) * sn + A * (1 - 2 * nu) * sd
            NT = B * sm + C * sd * rm
            DT = inv * (B * 3 * sn * rm + C * sd * mn + A * (nu * sm - 5 * sd * rm))
            ST = A * nu * rm + B * mn
            v = (N * NT[..., None] + M * MT[..., None] + D * DT[..., None] + s * ST[..., None])
        out[i:i + rows] = v.sum(1)
    return out


def _moments(x, y, charge, quad):
    """sum_y [ c / r + (D D^T m) / r^3 ] per point x, D = y - x: charge c and
    quad m (n_y, 3, J) -> (n_x, 3, J)."""
    ny, J = y.shape[0], charge.shape[2]
    ym = torch.einsum("yk,ykj->yj", y, quad)                      # y . m
    cols = torch.cat([torch.einsum("yd,yj->ydj", y, ym).reshape(ny, -1), ym,
                      torch.einsum("yd,ykj->ydkj", y, quad).reshape(ny, -1),
                      quad.reshape(ny, -1)], dim=1)
    ch = charge.reshape(ny, -1)
    F = torch.zeros((x.shape[0], 3 * J), dtype=x.dtype, device=x.device)
    G = torch.zeros((x.shape[0], cols.shape[1]), dtype=x.dtype, device=x.device)
    for i, j in _blocks(x.shape[0], ny):
        inv = _inv(x[i], y[j])
        F[i] += inv @ ch[j]
        G[i] += inv.pow_(3) @ cols[j]
    F, a = F.reshape(-1, 3, J), G[:, :3 * J].reshape(-1, 3, J)
    b = G[:, 3 * J:4 * J]
    c = G[:, 4 * J:13 * J].reshape(-1, 3, 3, J)                   # d, k, j
    m = G[:, 13 * J:].reshape(-1, 3, J)
    xm = torch.einsum("xk,xkj->xj", x, m)
    return (F + a - torch.einsum("xd,xj->xdj", x, b) - torch.einsum("xk,xdkj->xdj", x, c)
            + torch.einsum("xd,xj->xdj", x, xm))


def _dipoles(x, y, v):
    """sum_y (v . D) / r^3, v (n_y, m, 3): (n_x, m)."""
    ny, m = v.shape[0], v.shape[1]
    cols = torch.cat([torch.einsum("ymk,yk->ym", v, y), v.reshape(ny, -1)], dim=1)
    G = torch.zeros((x.shape[0], 4 * m), dtype=x.dtype, device=x.device)
    for i, j in _blocks(x.shape[0], ny):
        G[i] += _inv(x[i], y[j]).pow_(3) @ cols[j]
    return G[:, :m] - torch.einsum("xmk,xk->xm", G[:, m:].reshape(-1, m, 3), x)


def _far(K, o, s, x):
    """The direct farfield in 64 bits of the inputs x (R, 9 per source
    triangle): (R, 9 per observation triangle)."""
    mu, nu = PARAMS
    R = x.shape[0]
    xi = _t(x).reshape(R, s.n, 3, 3)                                # (r, n, basis, component)
    sw = s.J[:, None] * s.w[None]                                   # (n, q)
    xo, yo = o.x.reshape(-1, 3), s.x.reshape(-1, 3)

    def contract(F):                                                # (points, 3, R) -> (r, n, b, d)
        return torch.einsum("nq,qb,nqdr->rnbd", o.J[:, None] * o.w[None], o.b,
                            F.reshape(o.n, o.q, 3, R))

    inp = torch.einsum("qb,rnbd,nq->nqdr", s.b, xi, sw)             # (n, q, 3, r)
    ssc = torch.einsum("nbj,rnbd->ndjr", s.sc, xi)                  # (n, d, j, r)
    if K == "RH":
        c0 = mu / (8 * math.pi * (1 - nu))
        eye = torch.eye(3, dtype=torch.float64, device="cuda")[None, :, :, None]
        P = (2 * (1 - nu) * torch.einsum("nddr->nr", ssc)[:, None, None] * eye
             + 4 * nu * ssc.transpose(1, 2) - 2 * ssc)
        ch = (c0 * sw)[..., None, None, None] * P[:, None]
        qd = (c0 * sw)[..., None, None, None] * (-2 * ssc)[:, None]
        F = _moments(xo, yo, ch.reshape(-1, 3, 3 * R), qd.reshape(-1, 3, 3 * R))
        W = torch.einsum("q,nqdjr->ndjr", o.w, F.reshape(o.n, o.q, 3, 3, R))
        return torch.einsum("n,nbj,ndjr->rnbd", o.J, o.sc, W).reshape(R, -1)
    eps = torch.zeros((3, 3, 3), dtype=torch.float64, device="cuda")
    for i, j, k in ((0, 1, 2), (1, 2, 0), (2, 0, 1)):
        eps[i, j, k], eps[i, k, j] = 1.0, -1.0
    c8 = -1 / (8 * math.pi * (1 - nu))
    if K == "RT":
        curl = torch.einsum("mpj,njmr->npr", eps, ssc)
        ch = (sw[..., None, None] * curl[:, None]).reshape(-1, 3, R)
        F = _moments(xo, yo, (1 - 2 * nu) * c8 * ch, c8 * ch)
        v = torch.einsum("nqdr,nk->nqdrk", inp, s.nrm).reshape(-1, 3 * R, 3)
        return contract(F - _dipoles(xo, yo, v).reshape(-1, 3, R) / (4 * math.pi)).reshape(R, -1)
    if K == "RA":
        ch = inp.reshape(-1, 3, R)
        F = _moments(xo, yo, (1 - 2 * nu) * c8 * ch, c8 * ch)
        U = torch.einsum("q,nqkr->nkr", o.w, F.reshape(o.n, o.q, 3, R))
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        v = torch.einsum("nqdr,kl->nqdrkl", inp, eye).reshape(-1, 9 * R, 3)
        G = _dipoles(xo, yo, v).reshape(o.n, o.q, 3, R, 3)
        G = torch.einsum("nqdrk,nk->nqdr", G, o.nrm) / (4 * math.pi)
        curl = torch.einsum("n,nbm,mdk,nkr->rnbd", o.J, o.sc, eps, U)
        return (contract(G) - curl).reshape(R, -1)
    rep = lambda t: t.nrm[:, None].expand(t.n, t.q, 3).reshape(-1, 3)  # noqa: E731
    F = _point_field(K, xo, rep(o), yo, rep(s), inp[..., 0].reshape(-1, 3))  # one input
    return contract(F[..., None]).reshape(1, -1)


def exact(case, seed):
    """The same values in 64 bits by direct summation.  None for the kinds
    whose values hold the singular pair integrals (apply, nearfield, solve),
    and where the direct sum would take too long."""
    kind, K = case["kind"], case["kernel"]
    if kind in ("apply", "nearfield", "solve"):
        return None
    pts, tris, obs, src, x, rng = _inputs(case, seed)
    s = _Tris(pts, tris[src], case["nq_far"])
    if kind == "interior":
        p, ns = _interior_points(case, rng)
        xi = torch.einsum("qb,nbd->nqd", s.b, _t(x).reshape(s.n, 3, 3))
        a = (xi * (s.J[:, None] * s.w)[..., None]).reshape(-1, 3)
        ny = s.nrm[:, None].expand(s.n, s.q, 3).reshape(-1, 3)
        return _point_field(K, _t(p), _t(ns), s.x.reshape(-1, 3), ny, a).reshape(-1)
    o = s if obs is src else _Tris(pts, tris[obs], case["nq_far"])
    return _far(K, o, s, x) if kind == "panel" else _far(K, o, s, x[None])[0]
