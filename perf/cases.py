"""The work that programs have this library do, as timed cases.

A case is a dict of plain values.  ``listed()`` names twelve of them, ``draw``
gives more of the same ranges, ``prepare`` makes what a program holds before
the call (geometry from a seed, resident batches, scenes, servers), ``run`` is
one pass through the public entry points, ``work`` counts what a pass cannot
do without, and ``exact`` is the same answer in 64 bits from plain torch.

Volumes, gradients and Hessians leave the library in float64 containers that
hold FP32-accurate values (form factors and contractions run in FP32, or in
split 16-bit operands with FP32 sums).  The programs here keep them as the
float32 values they are.

Kinds of case:

  pair     intersection volume of two geometries from host memory, the
           reference's own call: collision tests, one pair at a time
  matrix   a simulation or similarity step: new DoFs for resident objects,
           their form factors, the volume matrix at a chosen precision
  solid    one large scanned or simulated mesh: form factors on a fine k-grid
           and its volume
  surfels  a training step on point clouds: volumes of all pairs, gradients
           with respect to every position and normal
  dofs     a training step on rigid or affine bodies: volumes and gradients
           with respect to every DoF (affine), or every vertex (mesh DoFs)
  align    one Newton evaluation of the alignment caller: value, gradient,
           Gauss-Newton Hessian for a new pose
  serve    a burst of scene queries to a resident server, translated or
           partly rotated
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from pointint_gb300 import align, core, geometry as G, pointint_cpp
from pointint_gb300._lib import DOF_AFFINE, DOF_TRIANGLE_MESH, GEOM_DISK, GEOM_TRIANGLE, SIM_ALL
from pointint_gb300.kgrid import standard_kgrid
from pointint_gb300.serving import Server

DIRECTIONS = {3: 6, 9: 38, 29: 302, 59: 1202, 131: 5810}  # bundled Lebedev rules: order -> directions
MEASURES = ("ochiai", "jaccard", "dice")


def listed():
    return [
        # the smallest call: two small point clouds on a coarse grid, where the host path and the launches are the time
        {"name": "pair_clouds", "kind": "pair", "a": "disks", "a_n": 777, "b": "gaussians", "b_n": 1001, "order": 9, "radial": 16},
        # the reference's own example: a box against a 1,280-triangle sphere, N_k = 9,664
        {"name": "pair_box_sphere", "kind": "pair", "a": "box", "a_n": 12, "b": "sphere", "b_n": 3, "order": 29, "radial": 32},
        # an ordinary scene of every element type, odd counts, radii that are no multiple of anything, plain FP32
        {"name": "matrix_mixed_37", "kind": "matrix", "spheres": 13, "level": 3, "boxes": 11, "clouds": 7, "splats": 6, "surfels": 1333,
         "order": 29, "radial": 45, "precision": "fp32"},
        # the 256-object volume matrix, N_k = 76,928, split-precision contraction
        {"name": "matrix_256", "kind": "matrix", "spheres": 128, "level": 4, "boxes": 128, "clouds": 0, "splats": 0, "surfels": 0,
         "order": 59, "radial": 64, "precision": "fp16x3"},
        # the largest mesh: a star-shaped solid of 200,000 triangles, N_k = 743,680
        {"name": "solid_200k", "kind": "solid", "frequency": 100, "order": 131, "radial": 128},
        # a training step on clouds of 50,000 disks
        {"name": "surfels_8x50k", "kind": "surfels", "objects": 8, "surfels": 50000, "gaussian": False, "order": 59, "radial": 64},
        # a small training step on Gaussians
        {"name": "surfels_gauss_small", "kind": "surfels", "objects": 3, "surfels": 1500, "gaussian": True, "order": 29, "radial": 32},
        # a training step on affine bodies
        {"name": "dofs_affine_24", "kind": "dofs", "spheres": 12, "boxes": 12, "level": 4, "vertices": False, "order": 59, "radial": 64},
        # a training step on the vertices of a few meshes
        {"name": "dofs_vertices_4", "kind": "dofs", "spheres": 4, "boxes": 0, "level": 3, "vertices": True, "order": 29, "radial": 32},
        # the alignment caller's Newton evaluation, 5,120 moving triangles
        {"name": "align_step", "kind": "align", "level": 4, "order": 59, "radial": 64, "measure": "dice"},
        # one query of a 256-object scene over resident form factors: latency of the contraction path
        {"name": "serve_translated", "kind": "serve", "library": 24, "tris_lo": 1000, "tris_hi": 5000, "scenes": 1, "objects": 256,
         "p_rot": 0.0, "order": 59, "radial": 64},
        # a burst of scenes, a fifth of whose objects are rotated (their form factors are evaluated again)
        {"name": "serve_rotated", "kind": "serve", "library": 16, "tris_lo": 1000, "tris_hi": 50000, "scenes": 4, "objects": 47,
         "p_rot": 0.2, "order": 59, "radial": 64},
    ]


def draw(rng):
    def log(lo, hi):
        return int(min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))

    kind = rng.choice(("pair", "matrix", "solid", "surfels", "dofs", "align", "serve"))
    if kind == "pair":
        order = rng.choice((9, 29))
        side = {}
        for s in "ab":
            shape = rng.choice(("disks", "gaussians", "sphere", "box"))
            side[s] = shape
            side[s + "_n"] = 12 if shape == "box" else rng.randint(1, 4) if shape == "sphere" else log(100, 4000)
        return {"kind": kind, **side, "order": order, "radial": rng.randint(16, 48)}
    if kind == "matrix":
        total = log(3, 256)
        mixed = total <= 64 and rng.random() < 0.5
        parts = [0, 0, 0, 0]
        for _ in range(total):
            parts[rng.randrange(4 if mixed else 2)] += 1
        return {"kind": kind, "spheres": parts[0], "level": rng.randint(2, 4), "boxes": parts[1], "clouds": parts[2], "splats": parts[3],
                "surfels": log(300, 5000) if mixed else 0, "order": rng.choice((29, 59)), "radial": rng.choice((32, 45, 64)),
                "precision": rng.choice(("fp32", "fp16x3", "bf16x3", "tf32x3"))}
    if kind == "solid":
        return {"kind": kind, "frequency": log(15, 100), "order": rng.choice((29, 59, 131)), "radial": rng.randint(32, 128)}
    if kind == "surfels":
        return {"kind": kind, "objects": rng.randint(2, 8), "surfels": log(500, 50000), "gaussian": rng.random() < 0.5,
                "order": rng.choice((29, 59)), "radial": rng.choice((32, 45, 64))}
    if kind == "dofs":
        vertices = rng.random() < 0.5
        return {"kind": kind, "spheres": rng.randint(1, 12), "boxes": 0 if vertices else rng.randint(0, 12), "level": rng.randint(2, 4),
                "vertices": vertices, "order": rng.choice((29, 59)), "radial": rng.choice((32, 45, 64))}
    if kind == "align":
        return {"kind": kind, "level": rng.randint(2, 4), "order": rng.choice((29, 59)), "radial": rng.choice((32, 45, 64)),
                "measure": rng.choice(MEASURES)}
    rotated = rng.random() < 0.5
    return {"kind": kind, "library": rng.randint(8, 24), "tris_lo": 1000, "tris_hi": log(2000, 20000), "scenes": rng.randint(1, 6),
            "objects": log(2, 64 if rotated else 256), "p_rot": 0.2 if rotated else 0.0, "order": 59, "radial": 64}


# ---------------------------------------------------------------------------
# Inputs.  Base meshes and k-grids are what a program loads once; shapes,
# poses and samples come from the seed.

@functools.lru_cache(maxsize=None)
def _grid(order, radial):
    return standard_kgrid(order, radial)


@functools.lru_cache(maxsize=None)
def _icosphere(level):
    return G.icosphere(level)


@functools.lru_cache(maxsize=None)
def _geodesic(frequency):
    """A geodesic sphere with the real spherical harmonics of degree <= 8 at its vertices."""
    V, F = G.geodesic_sphere(frequency)
    Y = G._real_sph_harm_basis(8, np.arccos(np.clip(V[:, 2], -1.0, 1.0)), np.arctan2(V[:, 1], V[:, 0]))
    return V, F, Y


def _stretch(rng, lo=0.5, hi=1.5):
    return G.random_rotation(rng) @ np.diag(rng.uniform(lo, hi, size=3)) @ G.random_rotation(rng).T


def _cloud(rng, n, gaussian, center):
    """n surfels sampled area-uniformly from a stretched sphere, radius sqrt(area / (pi n))."""
    V, F = _icosphere(3)
    P, N, share = G.sample_surface(V @ _stretch(rng).T + center, F, n, rng)
    rho = np.full(n, math.sqrt(share / math.pi))
    return G.make_gaussian_splat(P, N, rho, np.full(n, share)) if gaussian else G.make_point_cloud(P, N, rho, True)


def _one(rng, shape, n):
    """A geometry of the pair cases, near the origin."""
    at = rng.uniform(-0.6, 0.6, size=3)
    if shape == "box":
        V, F = G.create_unit_cube_mesh()
        return G.make_triangle_mesh(V * rng.uniform(0.7, 1.3, size=3) + at, F)
    if shape == "sphere":
        V, F = _icosphere(n)
        return G.make_triangle_mesh(V @ _stretch(rng, 0.8, 1.2).T + at, F)
    return _cloud(rng, n, shape == "gaussians", at)


def _objects(rng, c):
    """The matrix cases' objects: spheres and boxes under random affine maps, then clouds and splats, centres in [0, 8]^3."""
    objs = []
    Vs, Fs = _icosphere(c["level"])
    sphere = G.make_triangle_mesh(Vs, Fs)
    box = G.make_triangle_mesh(*G.create_unit_cube_mesh())
    for _ in range(c["spheres"]):
        objs.append(G.SceneObject(sphere, DOF_AFFINE, G.affine_dofs(_stretch(rng), rng.uniform(0.0, 8.0, size=3))))
    for _ in range(c["boxes"]):
        objs.append(G.SceneObject(box, DOF_AFFINE, G.affine_dofs(G.random_rotation(rng) * rng.uniform(0.5, 2.0), rng.uniform(0.0, 8.0, size=3))))
    for i in range(c.get("clouds", 0) + c.get("splats", 0)):
        geom = _cloud(rng, c["surfels"], i >= c["clouds"], np.zeros(3))
        objs.append(G.SceneObject(geom, DOF_AFFINE, G.affine_dofs(G.random_rotation(rng), rng.uniform(0.0, 8.0, size=3))))
    return objs


def _scene_objects(rng, c):
    """The training steps' objects, close enough together to overlap."""
    if c["kind"] == "surfels":
        return [G.SceneObject(_cloud(rng, c["surfels"], c["gaussian"], rng.uniform(0.0, 2.0, size=3))) for _ in range(c["objects"])]
    objs = []
    Vs, Fs = _icosphere(c["level"])
    sphere = G.make_triangle_mesh(Vs, Fs)
    for _ in range(c["spheres"]):
        A, t = _stretch(rng), rng.uniform(0.0, 3.0, size=3)
        if c["vertices"]:
            objs.append(G.SceneObject(sphere, DOF_TRIANGLE_MESH, Vs @ A.T + t))
        else:
            objs.append(G.SceneObject(sphere, DOF_AFFINE, G.affine_dofs(A, t)))
    box = G.make_triangle_mesh(*G.create_unit_cube_mesh())
    for _ in range(c["boxes"]):
        objs.append(G.SceneObject(box, DOF_AFFINE, G.affine_dofs(G.random_rotation(rng) * rng.uniform(0.5, 2.0), rng.uniform(0.0, 3.0, size=3))))
    return objs


def _solid(rng, frequency):
    V, F, Y = _geodesic(frequency)
    r = np.maximum(1.0 + Y @ rng.normal(0.0, 0.05, size=Y.shape[1]), 0.5)
    return G.make_triangle_mesh(V * r[:, None], F)


def _aligned(rng, c):
    """Fixed geometry, moving geometry and a pose near the fit."""
    V, F = _icosphere(c["level"])
    fixed = G.make_triangle_mesh(V @ _stretch(rng, 0.7, 1.3).T, F)
    moving = G.make_triangle_mesh(V @ _stretch(rng, 0.7, 1.3).T, F)
    return fixed, moving, G.affine_dofs(np.eye(3) + 0.1 * rng.standard_normal((3, 3)), 0.15 * rng.standard_normal(3))


def _library(rng, c):
    """Geodesic spheres of log-uniform triangle counts, half of them stretched; and the scenes asked for."""
    lib = []
    for i in range(c["library"]):
        t = math.exp(rng.uniform(math.log(c["tris_lo"]), math.log(c["tris_hi"])))
        V, F, _ = _geodesic(int(min(50, max(7, round(math.sqrt(t / 20.0))))))
        lib.append(G.SceneObject(G.make_triangle_mesh(V @ (_stretch(rng).T if i % 2 else np.eye(3)), F)))
    scenes = []
    for _ in range(c["scenes"]):
        n = c["objects"]
        which = rng.integers(0, c["library"], size=n).astype(np.int32)
        turn = np.stack([G.random_rotation(rng) if rng.random() < c["p_rot"] else np.eye(3) for _ in range(n)]) if c["p_rot"] else None
        scenes.append((which, turn, rng.normal(0.0, 0.5, size=(n, 3))))
    return lib, scenes


def prepare(case, seed):
    c, rng = case, np.random.default_rng(seed)
    kg = _grid(c["order"], c["radial"])
    s = {"case": c, "kg": kg}
    if c["kind"] == "pair":
        s["a"], s["b"] = _one(rng, c["a"], c["a_n"]), _one(rng, c["b"], c["b_n"])
        return s
    kg.handle()
    if c["kind"] == "matrix":
        objs = _objects(rng, c)
        s["batch"] = core.ObjectBatch(objs)
        s["theta"] = torch.tensor(np.concatenate([o.dofs for o in objs]), device="cuda")
    elif c["kind"] == "solid":
        s["batch"] = core.ObjectBatch([G.SceneObject(_solid(rng, c["frequency"]))])
    elif c["kind"] == "surfels":
        s["scene"] = core.Scene(kg, _scene_objects(rng, c))
        s["centers"], s["normals"] = (t.requires_grad_() for t in s["scene"].surfel_params())
    elif c["kind"] == "dofs":
        s["scene"] = core.Scene(kg, _scene_objects(rng, c))
        s["theta"] = s["scene"].dofs().requires_grad_()
    elif c["kind"] == "align":
        fixed, moving, s["pose"] = _aligned(rng, c)
        s["aligner"] = align.Aligner(fixed, moving, kg)
        s["V1"] = s["aligner"].fixed_volume()
    else:
        lib, s["scenes"] = _library(rng, c)
        s["server"] = Server(kg, lib, hbm_budget_bytes=4 << 30)
    return s


def run(state):
    s, c = state, state["case"]
    kg = s["kg"]
    if c["kind"] == "pair":
        return pointint_cpp.compute_intersection_volume_cuda(s["a"], s["b"], kg)
    if c["kind"] == "matrix":
        s["batch"].set_all_dofs(s["theta"])
        amax = torch.empty(len(s["batch"]), dtype=torch.float32, device="cuda")
        J = core.form_factors(kg, s["batch"], True, row_amax=amax)
        return {"J": J, "V": core.contract(kg, J, c["precision"], row_amax=amax).float()}
    if c["kind"] == "solid":
        J = core.form_factors(kg, s["batch"], True)
        return {"J": J, "V": core.contract(kg, J, "fp32").float()}
    if c["kind"] == "surfels":
        V = s["scene"].volume_matrix_of_surfels(s["centers"], s["normals"])
        gc, gn = torch.autograd.grad(V.sum(), (s["centers"], s["normals"]))
        return {"V": V.detach().float(), "centers": gc.float(), "normals": gn.float()}
    if c["kind"] == "dofs":
        V = s["scene"].volume_matrix_of_dofs(s["theta"])
        (g,) = torch.autograd.grad(V.sum(), (s["theta"],))
        return {"V": V.detach().float(), "theta": g.float()}
    if c["kind"] == "align":
        r = s["aligner"].similarity(s["pose"], c["measure"], s["V1"], SIM_ALL)
        return {"value": r.value, "similarity": r.similarity, "gradient": r.gradient.astype(np.float32), "hessian": r.hessian.astype(np.float32)}
    srv = s["server"]
    tickets = [srv.submit(which, turn, shift) for which, turn, shift in s["scenes"]]
    out = [srv.wait(t).astype(np.float32) for t in tickets]
    for t in tickets:
        srv.release(t)
    return out


def _counts(c):
    """(triangles, surfels) of each object whose form factors one pass evaluates, and the rows of the volume matrix."""
    tri = {"box": lambda n: 12, "sphere": lambda n: 20 * 4 ** n}
    if c["kind"] == "pair":
        return [(tri[c[s]](c[s + "_n"]), 0) if c[s] in tri else (0, c[s + "_n"]) for s in "ab"], 2
    if c["kind"] in ("matrix", "dofs"):
        e = [(20 * 4 ** c["level"], 0)] * c["spheres"] + [(12, 0)] * c["boxes"]
        e += [(0, c.get("surfels", 0))] * (c.get("clouds", 0) + c.get("splats", 0))
        return e, len(e)
    if c["kind"] == "solid":
        return [(20 * c["frequency"] ** 2, 0)], 1
    if c["kind"] == "surfels":
        return [(0, c["surfels"])] * c["objects"], c["objects"]
    if c["kind"] == "align":
        return [(20 * 4 ** c["level"], 0)], 14
    mean = (c["tris_hi"] - c["tris_lo"]) / math.log(c["tris_hi"] / c["tris_lo"])  # of a log-uniform count
    return [(mean, 0)] * round(c["scenes"] * c["objects"] * c["p_rot"]), c["objects"]


def work(case):
    """Elements read and results written once; every element projected on every direction that a centrally symmetric grid leaves
    (three dot products, once more for each direction of a gradient), every form factor combined with every other."""
    c = case
    elems, n = _counts(c)
    directions = DIRECTIONS[c["order"]]
    Q = directions * c["radial"]
    n_elem = sum(t + s for t, s in elems)
    source = sum(112 * t + 64 * s for t, s in elems)
    project = 18 * n_elem * directions / 2
    pairs = c.get("scenes", 1) * n * (n + 1) / 2
    gradient = c["kind"] in ("surfels", "dofs", "align")
    rows = 8 * Q * (c["library"] if c["kind"] == "serve" else len(elems) if c["kind"] in ("matrix", "solid") else 0)
    out = 8 * c.get("scenes", 1) * n * n + (48 * n_elem if gradient else 0)
    return {"bytes": source + rows + out, "flops": project * (2 if gradient else 1) + 4 * Q * pairs}


# ---------------------------------------------------------------------------
# The same answers in 64 bits, from the definitions: plain torch, chunked.
#
#   triangle  A(k) = -2 (k.S)/|k| e^{ik.m} e[da, db, dc], S the area vector,
#             m the centroid, e[..] the second divided difference of e^{iz}
#             at the vertices' phases relative to the centroid
#   disk      A(k) = area (k'.n)/|k| 2 J1(x)/x e^{ik.c}, x = rho |k'_perp|,
#             k' = A^T k for a cloud moved by the linear part A
#   Gaussian  A(k) = w (k'.n)/|k| e^{-sigma^2 |k'_perp|^2 / 2} e^{ik.c}
#   volumes   V_ij = Re sum_q w_q conj(A_i) A_j / (8 pi^3)
#
# A(-k) = -conj A(k), so one direction of each antipodal pair is summed.

SCALE = 1.0 / (8.0 * math.pi ** 3)
MOST_VALUES = 3e10        # element x node values of one exact() without gradients (about 15 s)
MOST_DERIVATIVES = 3e9    # with gradients
CHUNK = 1 << 24


class _DiskFactor(torch.autograd.Function):
    """2 J1(x)/x as a function of y = x^2, with its derivative -J2(x)/x^2."""

    @staticmethod
    def forward(ctx, y):
        ctx.save_for_backward(y)
        x = y.clamp(min=0.25).sqrt()
        big = 2.0 * torch.special.bessel_j1(x) / x
        return torch.where(y < 0.25, _DiskFactor.series(y, 1), big)

    @staticmethod
    def backward(ctx, g):
        (y,) = ctx.saved_tensors
        x = y.clamp(min=0.25).sqrt()
        j2 = 2.0 * torch.special.bessel_j1(x) / x - torch.special.bessel_j0(x)
        return g * torch.where(y < 0.25, -0.25 * _DiskFactor.series(y, 2) * 0.5, -j2 / (x * x))

    @staticmethod
    def series(y, nu):
        """nu! sum_m (-y/4)^m / (m! (m + nu)!)"""
        t = torch.ones_like(y)
        s = t
        for m in range(1, 10):
            t = t * (-0.25 * y) / (m * (m + nu))
            s = s + t
        return s


def _triangle_terms(a, e1, e2, d, k, spread):
    """Terms [L, N, M] as (re, im) of triangles (a, e1, e2) at directions d and radii k; `spread` bounds k |edge|."""
    m = (a + (e1 + e2) / 3.0) @ d.T
    S = 0.5 * torch.linalg.cross(e1, e2) @ d.T
    s1, s2 = e1 @ d.T, e2 @ d.T
    da = -(s1 + s2) / 3.0
    db, dc = da + s1, da + s2
    k = k[:, None, None]
    g = -2.0 * S
    # Taylor series of e[da, db, dc] about the centroid, through the complete homogeneous symmetric polynomials
    mu = 0.5 * (da * da + db * db + dc * dc)
    nu = da * db * dc
    top = 5  # the last term, odd: those after it are below 1e-17 of the first
    while top < 13 and min(spread, 0.7) ** (top + 1) / math.factorial(top + 3) > 1e-18:
        top += 2
    h = [torch.ones_like(mu), torch.zeros_like(mu), mu]
    for n in range(3, top + 1):
        h.append(mu * h[n - 2] + nu * h[n - 3])
    k2 = k * k
    re, im = k2 * torch.zeros_like(mu), k2 * torch.zeros_like(mu)
    for n in range(top - 1, -1, -2):
        re = torch.addcmul((-1) ** (n // 2 + 1) / math.factorial(n + 2) * h[n], re, k2)
    for n in range(top, 2, -2):
        im = torch.addcmul((-1) ** ((n + 1) // 2) / math.factorial(n + 2) * h[n], im, k2)
    im = im * (k2 * k)
    if spread > 0.7:
        lo, hi = torch.minimum(torch.minimum(da, db), dc), torch.maximum(torch.maximum(da, db), dc)
        mid = da + db + dc - lo - hi
        D = k * (hi - lo)
        wide = D > 0.7
        D = torch.where(wide, D, torch.ones_like(D))
        x, y = 0.5 * k * (mid + hi), 0.5 * k * (lo + mid)
        sx, sy = torch.sinc(0.5 / math.pi * k * (hi - mid)), torch.sinc(0.5 / math.pi * k * (mid - lo))
        re = torch.where(wide, -(torch.sin(x) * sx - torch.sin(y) * sy) / D, re)
        im = torch.where(wide, (torch.cos(x) * sx - torch.cos(y) * sy) / D, im)
    c, s = torch.cos(k * m), torch.sin(k * m)
    return g * (c * re - s * im), g * (c * im + s * re)


def _surfel_terms(c, n, size, weight, A, d, k, disk):
    v = d @ A  # rows: A^T d
    vn = n @ v.T
    perp = (v * v).sum(-1) - vn * vn
    k = k[:, None, None]
    y = k * k * (size * size)[:, None] * perp.clamp(min=0.0)
    f = weight[:, None] * vn * (_DiskFactor.apply(y) if disk else torch.exp(-0.5 * y))
    p = k * (c @ d.T)
    return f * torch.cos(p), f * torch.sin(p)


class _Exact64:
    """The k-grid in 64 bits, one direction of each antipodal pair, and the objects' form factors on it."""

    def __init__(self, kg, order, radial):
        self.M, self.L = DIRECTIONS[order], radial
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        dirs = torch.tensor(kg.dirs[: self.M], device=dev)
        self.k = torch.tensor(kg.kmag.reshape(radial, self.M)[:, 0].copy(), device=dev)
        self.w = torch.tensor(kg.w.reshape(radial, self.M), device=dev)
        mate = (dirs @ dirs.T).argmin(1)
        index = torch.arange(self.M, device=dev)
        assert bool(((dirs + dirs[mate]).abs().amax(1) < 1e-9).all()) and bool((mate[mate] == index).all())
        self.half = index[index < mate]
        self.mate = mate[self.half]
        self.d = dirs[self.half]
        self.weight = self.w[:, self.half] + self.w[:, self.mate]  # Re(conj A_i A_j) is the same at k and -k
        self.dev = dev

    def t(self, x):
        return torch.tensor(np.ascontiguousarray(x), dtype=torch.float64, device=self.dev)

    def source(self, obj):
        """What an object's terms are made from: (kind, differentiable parameters, constants)."""
        e = obj.geom.elems
        if obj.geom.type == GEOM_TRIANGLE:
            if obj.dof_type == DOF_TRIANGLE_MESH:
                return "mesh", [self.t(obj.dofs)], [torch.tensor(e["vid"].astype(np.int64), device=self.dev)]
            return "tri", [self.t(obj.dofs)], [self.t(e["a"]), self.t(e["e1"]), self.t(e["e2"])]
        kind = "disk" if obj.geom.type == GEOM_DISK else "gauss"
        size, weight = ("rho", "area") if kind == "disk" else ("sigma", "w")
        return kind, [self.t(obj.dofs), self.t(e["c"]), self.t(e["n"])], [self.t(e[size]), self.t(e[weight])]

    def count(self, objs):
        return sum(o.geom.num_elements() for o in objs) * len(self.half) * self.L

    def terms(self, kind, params, const, lo, hi, d, k, k_max):
        t, A = params[0][:3], params[0][3:12].reshape(3, 3)
        if kind in ("tri", "mesh"):
            if kind == "mesh":
                P = params[0].reshape(-1, 3)
                v = [P[const[0][lo:hi, i]] for i in range(3)]
                a, e1, e2 = v[0], v[1] - v[0], v[2] - v[0]
            else:
                a, e1, e2 = const[0][lo:hi] @ A.T + t, const[1][lo:hi] @ A.T, const[2][lo:hi] @ A.T
            with torch.no_grad():
                edge = max(float(x.detach().norm(dim=1).max()) for x in (e1, e2, e2 - e1))
            return _triangle_terms(a, e1, e2, d, k, k_max * edge)
        c = params[1][lo:hi] @ A.T + t
        return _surfel_terms(c, params[2][lo:hi], const[0][lo:hi], const[1][lo:hi], A, d, k, kind == "disk")

    def chunks(self, n):
        """(element range, direction range, radius range) blocks of at most CHUNK values; radii in groups of similar k."""
        rs = max(1, self.L // 8)
        ns = max(1, min(n, CHUNK // (rs * 32)))
        ms = max(1, min(len(self.half), CHUNK // (rs * ns)))
        for r in range(0, self.L, rs):
            for m in range(0, len(self.half), ms):
                for e in range(0, n, ns):
                    yield e, min(n, e + ns), slice(m, m + ms), slice(r, r + rs)

    def amplitudes(self, obj):
        """A [L, half of the directions], complex128."""
        kind, params, const = self.source(obj)
        out = torch.zeros((self.L, len(self.half)), dtype=torch.complex128, device=self.dev)
        with torch.no_grad():
            for lo, hi, m, r in self.chunks(obj.geom.num_elements()):
                re, im = self.terms(kind, params, const, lo, hi, self.d[m], self.k[r], float(self.k[r].max()))
                out[r, m] += torch.complex(re.sum(1), im.sum(1))
        return out

    def rows(self, A):
        """sqrt(w)-scaled rows over all nodes, q = r M + j, from the amplitudes of half the directions."""
        full = torch.zeros((len(A), self.L, self.M), dtype=torch.complex128, device=self.dev)
        full[:, :, self.half] = A
        full[:, :, self.mate] = -A.conj()
        return (full * self.w.sqrt()).reshape(len(A), -1)

    def volumes(self, A):
        X = (A * self.weight.sqrt()).reshape(len(A), -1)
        return (X.real @ X.real.T + X.imag @ X.imag.T) * SCALE

    def pullback(self, obj, B):
        """Gradient of Re sum_q weight conj(A) B / (8 pi^3) with respect to the object's parameters."""
        kind, params, const = self.source(obj)
        params = [p.requires_grad_() for p in params]
        total = [torch.zeros_like(p) for p in params]
        X = B * self.weight * SCALE
        for lo, hi, m, r in self.chunks(obj.geom.num_elements()):
            re, im = self.terms(kind, params, const, lo, hi, self.d[m], self.k[r], float(self.k[r].max()))
            loss = (re.sum(1) * X.real[r, m] + im.sum(1) * X.imag[r, m]).sum()
            for t, g in zip(total, torch.autograd.grad(loss, params, allow_unused=True)):
                if g is not None:
                    t += g
        return total

    def tangents(self, obj):
        """dA/dtheta over the 12 affine DoFs [12, L, half of the directions], complex128."""
        kind, params, const = self.source(obj)
        out = torch.zeros((12, self.L, len(self.half)), dtype=torch.complex128, device=self.dev)
        for i in range(12):
            unit = torch.zeros_like(params[0])
            unit[i] = 1.0
            for lo, hi, m, r in self.chunks(obj.geom.num_elements()):
                def f(theta):
                    re, im = self.terms(kind, [theta] + params[1:], const, lo, hi, self.d[m], self.k[r], float(self.k[r].max()))
                    return re.sum(1), im.sum(1)
                re, im = torch.func.jvp(f, (params[0],), (unit,))[1]
                out[i, r, m] += torch.complex(re, im)
        return out


def _moved(obj, turn, shift):
    """A library object under x' = R x + t on top of its DoFs."""
    A, t = obj.dofs[3:].reshape(3, 3), obj.dofs[:3]
    R = np.eye(3) if turn is None else turn
    return G.SceneObject(obj.geom, DOF_AFFINE, G.affine_dofs(R @ A, R @ t + shift))


def exact(case, seed):
    c, rng = case, np.random.default_rng(seed)
    X = _Exact64(_grid(c["order"], c["radial"]), c["order"], c["radial"])
    if c["kind"] == "pair":
        objs = [G.SceneObject(_one(rng, c[s], c[s + "_n"])) for s in "ab"]
        return float(X.volumes(torch.stack([X.amplitudes(o) for o in objs]))[0, 1])
    if c["kind"] in ("matrix", "solid"):
        objs = _objects(rng, c) if c["kind"] == "matrix" else [G.SceneObject(_solid(rng, c["frequency"]))]
        if X.count(objs) > MOST_VALUES:
            return None
        A = torch.stack([X.amplitudes(o) for o in objs])
        return {"J": X.rows(A), "V": X.volumes(A)}
    if c["kind"] in ("surfels", "dofs"):
        objs = _scene_objects(rng, c)
        if X.count(objs) > MOST_DERIVATIVES:
            return None
        A = torch.stack([X.amplitudes(o) for o in objs])
        B = 2.0 * A.sum(0)  # of the sum of all V_ij
        grads = [X.pullback(o, B) for o in objs]
        out = {"V": X.volumes(A)}
        if c["kind"] == "dofs":
            return {**out, "theta": torch.cat([g[0] for g in grads])}
        return {**out, "centers": torch.cat([g[1] for g in grads]), "normals": torch.cat([g[2] for g in grads])}
    if c["kind"] == "align":
        fixed, moving, pose = _aligned(rng, c)
        o1, o2 = G.SceneObject(fixed), G.SceneObject(moving, DOF_AFFINE, pose)
        A1, A2 = X.amplitudes(o1), X.amplitudes(o2)
        gram = X.volumes(torch.cat([A1[None], A2[None], X.tangents(o2)])).cpu().numpy()
        return _similarity64(gram, c["measure"])
    lib, scenes = _library(rng, c)
    used = [(i, which[i], turn is not None and not np.array_equal(turn[i], np.eye(3))) for which, turn, _ in scenes for i in range(len(which))]
    base = sorted({w for _, w, turned in used})
    if X.count([lib[w] for w in base]) + X.count([lib[w] for _, w, turned in used if turned]) > MOST_VALUES:
        return None
    still = {w: X.amplitudes(lib[w]) for w in base}
    out = []
    for which, turn, shift in scenes:
        A = []
        for i, w in enumerate(which):
            if turn is not None and not np.array_equal(turn[i], np.eye(3)):
                A.append(X.amplitudes(_moved(lib[w], turn[i], shift[i])))
            else:  # a translation is a phase
                p = X.k[:, None] * (X.d @ X.t(shift[i]))[None, :]
                A.append(still[w] * torch.polar(torch.ones_like(p), p))
        out.append(X.volumes(torch.stack(A)))
    return out


def _similarity64(gram, measure):
    """-log of the similarity of a fixed (row 0) and a moving (row 1) solid, its gradient and Gauss-Newton Hessian over the moving
    solid's DoFs (rows 2..), in which the intersection's own second derivatives are dropped."""
    V1, Vi, V2 = gram[0, 0], gram[0, 1], gram[1, 1]
    gi, g2, H2 = gram[2:, 0], 2.0 * gram[2:, 1], 2.0 * gram[2:, 2:]
    # s(Vi, V2): first and second partial derivatives
    if measure == "ochiai":
        s = Vi / math.sqrt(V1 * V2)
        si, s2, sii, si2, s22 = s / Vi, -0.5 * s / V2, 0.0, -0.5 * s / (Vi * V2), 0.75 * s / V2 ** 2
    elif measure == "jaccard":
        D = V1 + V2 - Vi
        s = Vi / D
        si, s2 = (D + Vi) / D ** 2, -Vi / D ** 2
        sii, si2, s22 = 2.0 * (D + Vi) / D ** 3, -(D + 2.0 * Vi) / D ** 3, 2.0 * Vi / D ** 3
    else:
        D = V1 + V2
        s = 2.0 * Vi / D
        si, s2, sii, si2, s22 = 2.0 / D, -2.0 * Vi / D ** 2, 0.0, -2.0 / D ** 2, 4.0 * Vi / D ** 3
    gs = si * gi + s2 * g2
    Hs = s2 * H2 + sii * np.outer(gi, gi) + si2 * (np.outer(gi, g2) + np.outer(g2, gi)) + s22 * np.outer(g2, g2)
    return {"value": -math.log(s), "similarity": s, "gradient": -gs / s, "hessian": np.outer(gs, gs) / s ** 2 - Hs / s}
