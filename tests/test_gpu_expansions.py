"""Edges of the expansion, splitting and ordering paths against the FP64 oracle.

Tolerances are the FP32 contract of the other parity tests, fixed beforehand:
form factors ||dJ|| <= 2e-6 ||J|| and max |dJ| <= 1e-5 max |J|; gradients 1e-5
of the largest entry; Hessian blocks 1e-5; FP32 contraction 1e-5 conditioned.

Element counts straddle the leaf (4), the summation chunk (16), the cluster
(64), the staged tiles (128), the smallest object that is reordered (2,048) and
the largest segment one block orders (8,192).
"""
import numpy as np
import pytest
import torch

import pointint_gb300 as pg
from pointint_gb300 import core, geometry as G
from pointint_gb300.kgrid import KGrid, standard_kgrid
from test_gpu_gradients import assert_grad_close
from test_gpu_hessian import block_errors
from test_gpu_parity import check_J, cond_rel_err, gpu_J, shapes, to_oracle
from test_gpu_precision import fp64_contract

pytestmark = pytest.mark.gpu


def radial_order(kg, perm):
    """The tensor grid with its radii taken in the order perm."""
    M = kg.num_nodes // len(perm)
    sel = (np.asarray(perm)[:, None] * M + np.arange(M)[None, :]).reshape(-1)
    return KGrid(kg.dirs[sel], kg.kmag[sel], kg.w[sel])


@pytest.mark.parametrize("order", ["descending", "shuffled"])
def test_tensor_grid_with_radii_in_any_order(cuda, orc, order):
    """Radii that do not ascend take no expansions, and a block's first radius
    is not its smallest."""
    L = 61  # a partly empty block as well
    perm = np.arange(L)[::-1] if order == "descending" else np.random.default_rng(5).permutation(L)
    kg = radial_order(standard_kgrid(9, L), perm)
    rng = np.random.default_rng(1)
    objs = [shapes(k, rng) for k in ("cube", "ico3", "mesh_dof", "disks_affine", "gauss")]
    check_J(gpu_J(kg, objs), orc.form_factor_matrix(to_oracle(orc, objs), kg.dirs, kg.kmag))


KINDS3 = ["tri", "disk", "gauss"]
COUNTS = [1, 3, 4, 5, 15, 17, 63, 64, 65, 127, 129, 2047, 2048, 2049, 8192, 8193]


def patch(kind, n, seed, shift=(0.0, 0.0, 0.0), affine=False):
    """n elements scattered over a unit sphere in random order, each of the size
    that n of them cover it with: an open surface, or one whose elements overlap."""
    rng = np.random.default_rng(1000 * n + seed)
    P = rng.normal(size=(n, 3))
    N = P / np.linalg.norm(P, axis=1, keepdims=True)
    size = 2.0 / np.sqrt(n)
    if kind == "tri":
        V = (N[:, None, :] + size * 0.5 * rng.normal(size=(n, 3, 3))).reshape(-1, 3)
        geom = G.make_triangle_mesh(V, np.arange(3 * n).reshape(n, 3))
    elif kind == "disk":
        geom = G.make_point_cloud(N, N, size * rng.uniform(0.5, 1.0, n))
    else:
        geom = G.make_gaussian_splat(N, N, 0.5 * size * rng.uniform(0.5, 1.0, n), np.full(n, 4 * np.pi / n))
    A = np.eye(3) + (0.2 * rng.normal(size=(3, 3)) if affine else 0.0)
    return G.SceneObject(geom, pg.DOF_AFFINE, G.affine_dofs(A, shift))


def check_J_weighted(kg, orc, objs):
    """check_J on the sqrt|w|-weighted form factors, in which every radius counts
    (an open surface's plain ones grow like 1/k towards k = 0)."""
    Jo = orc.form_factor_matrix(to_oracle(orc, objs), kg.dirs, kg.kmag) * np.sqrt(np.abs(kg.w))[:, None]
    check_J(gpu_J(kg, objs, True), Jo)


@pytest.fixture(scope="module")
def kg64():
    return standard_kgrid(9, 64)  # 38 directions, 19 of them evaluated: a part of one warp


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("kind", KINDS3)
def test_form_factors_at_edge_element_counts(cuda, orc, kg64, kind, n):
    check_J_weighted(kg64, orc, [patch(kind, n, 1, (0.3, -0.2, 0.5), affine=True)])


@pytest.mark.parametrize("L", [7, 8, 9, 31, 32, 47, 48, 49, 288, 289])
def test_radius_counts_around_the_expansions_limits(cuda, orc, L):
    """Expansions from 8 to 288 radii; 32 radii a thread block of eight, 48 the
    Jacobian's groups."""
    kg = standard_kgrid(3, L)
    check_J_weighted(kg, orc, [patch(k, 130, 2, (0.1, 0.2, 0.3), affine=True) for k in KINDS3])


@pytest.mark.parametrize("n", [1, 63, 64, 65, 129, 2049])
@pytest.mark.parametrize("kind", KINDS3)
def test_gradients_at_edge_element_counts(cuda, orc, kg64, kind, n):
    """AffineDoF gradients of a pair (the adjoint's expansions, its clusters'
    last one partly empty) and, for triangles, Gauss-Newton blocks (the
    Jacobian's expansions, which surfels do not take)."""
    o1, o2 = patch(kind, n, 3, (0.1, 0.0, -0.2), affine=True), patch("tri", 80, 4, (0.4, 0.1, 0.0))
    got = core.pair_volume_hessian_host(kg64, o1, o2)
    a, b = to_oracle(orc, [o1, o2])
    ref = orc.pair_volume(a, b, (kg64.dirs, kg64.kmag, kg64.w), orc.VOLUME_ONLY | orc.GRADIENT | orc.HESSIAN)
    assert_grad_close(got["grad_geom1"], ref["grad_geom1"], what=f"{kind} {n} grad1")
    assert_grad_close(got["grad_geom2"], ref["grad_geom2"], what=f"{kind} {n} grad2")
    if kind != "tri":
        return
    H11, H22 = ref["hessian_geom1"], ref["hessian_geom2"]
    for key, Hi, Hj in (("hessian_geom1", H11, H11), ("hessian_geom2", H22, H22), ("hessian_cross", H11, H22)):
        fro, _ = block_errors(got[key], ref[key], Hi, Hj)
        assert fro <= 1e-5, (key, fro)


def test_vertex_gradients_of_a_reordered_mesh(cuda, orc, kg64):
    """2,420 triangles (reordered) with vertex DoFs: gradients stay with their vertices."""
    V, F = G.geodesic_sphere(11)
    assert len(F) > 2048
    objs = [G.SceneObject(G.make_triangle_mesh(V, F), pg.DOF_TRIANGLE_MESH, V.reshape(-1)), patch("disk", 100, 5, (0.5, 0, 0))]
    _, grad = core.volume_matrix_grad_host(kg64, objs)
    _, ref, _ = orc.volume_matrix(to_oracle(orc, objs), (kg64.dirs, kg64.kmag, kg64.w), orc.VOLUME_ONLY | orc.GRADIENT)
    assert_grad_close(grad[0][1], ref[0][1], what="vertices")


@pytest.mark.parametrize("kind", ["disk", "gauss"])
def test_surfel_gradients_of_a_reordered_cloud(cuda, orc, kg64, kind):
    """2,049 surfels: the gradients come back in the caller's order."""
    objs = [patch(kind, 2049, 6), patch(kind, 65, 7)]
    scene = core.Scene(kg64, objs)
    c, n = (t.requires_grad_(True) for t in scene.surfel_params())
    scene.volume_matrix_of_surfels(c, n).sum().backward()
    gp, gn = orc.surfel_param_grad(to_oracle(orc, objs), (kg64.dirs, kg64.kmag, kg64.w), np.ones((2, 2)))
    assert_grad_close(c.grad.cpu().numpy(), gp, what="dL/dc")
    assert_grad_close(n.grad.cpu().numpy(), gn, what="dL/dn")


@pytest.mark.parametrize("n", [1, 2, 4, 5, 8, 9, 33, 63, 64, 65])
@pytest.mark.parametrize("Q", [3, 1001])
def test_few_row_contraction(cuda, n, Q):
    """n <= 64 rows take the FP32 contraction of their own; weights of both signs,
    a node count that is no multiple of anything."""
    rng = np.random.default_rng(100 * n + Q)
    dirs = rng.normal(size=(Q, 3))
    dirs /= np.linalg.norm(dirs, axis=1, keepdims=True)
    w = rng.uniform(0.5, 1.5, Q)
    w[::5] *= -1.0
    kg = KGrid(dirs, rng.uniform(0.1, 5.0, Q), w)
    J = (rng.normal(size=(n, Q)) + 1j * rng.normal(size=(n, Q))).astype(np.complex64)
    V = core.contract(kg, torch.from_numpy(J).cuda(), "fp32").cpu().numpy()
    R = fp64_contract(J, w)
    # conditioned by the sums of magnitudes: with weights of both signs the diagonal may cancel too
    scale = fp64_contract(np.abs(J.real) + 1j * np.abs(J.imag), np.abs(w))
    assert np.array_equal(V, V.T)
    assert (np.abs(V - R) / scale).max() <= 1e-6


@pytest.mark.parametrize("dirs_kept", ["every second", "one of each pair"])
def test_serving_on_a_grid_with_unpaired_directions(cuda, orc, dirs_kept):
    """Rows hold the evaluated directions only, weighted with their antipode where
    the grid has it."""
    from pointint_gb300.serving import Server
    full = standard_kgrid(9, 16)
    M = full.num_nodes // 16
    keep = np.arange(0, M, 2) if dirs_kept == "every second" else full.direction_pairs()[:, 0]
    sel = (np.arange(16)[:, None] * M + np.asarray(keep)[None, :]).reshape(-1)
    kg = KGrid(full.dirs[sel], full.kmag[sel], full.w[sel])
    rng = np.random.default_rng(3)
    lib = [patch("tri", 300, 8), patch("disk", 200, 9), patch("gauss", 100, 10), shapes("ico3", rng)]
    rots = np.array([np.eye(3), G.random_rotation(rng), G.random_rotation(rng), np.eye(3), G.random_rotation(rng)])
    trans = rng.normal(0.0, 0.4, size=(5, 3))
    ids = [0, 1, 2, 3, 3]
    moved = []
    for i, R, t in zip(ids, rots, trans):
        d = lib[i].dofs
        moved.append(G.SceneObject(lib[i].geom, pg.DOF_AFFINE, G.affine_dofs(R @ d[3:].reshape(3, 3), R @ d[:3] + t)))
    ref, _, _ = orc.volume_matrix(to_oracle(orc, moved), (kg.dirs, kg.kmag, kg.w))
    with Server(kg, lib, precision="fp16x3", autotune=False) as srv:
        V = srv.query(ids, rots, trans)
    assert cond_rel_err(V, ref).max() <= 1e-4


def test_serving_precision_of_disjoint_objects(cuda):
    """Serving rows keep the grid's direction order: small volumes of disjoint
    objects, conditioned at 1e-3 sqrt(V_ii V_jj), within 3e-5 of an FP64
    contraction in the mean over scenes (2e-5 is the plain path's own level with
    the FP16 split; rows in compact groups of directions measured 5.3e-5)."""
    from pointint_gb300.serving import Server
    kg = standard_kgrid(59, 64)
    V3, F3 = G.icosphere(3)
    worst = []
    for seed in range(4):
        rng = np.random.default_rng(seed)
        objs = []
        for i in range(40):
            A = G.random_rotation(rng) @ np.diag(rng.uniform(0.5, 1.5, 3))
            V, F = (V3, F3) if i % 2 else G.box_mesh(rng.uniform(0.5, 2.0, 3))
            objs.append(G.SceneObject(G.make_triangle_mesh(V, F), pg.DOF_AFFINE, G.affine_dofs(A, rng.uniform(0, 3, 3))))
        tr = rng.normal(0.0, 0.5, (40, 3))
        with Server(kg, objs, precision="fp16x3", autotune=False) as srv:
            V = srv.query(np.arange(40), None, tr)
        moved = [G.SceneObject(o.geom, o.dof_type, np.concatenate([o.dofs[:3] + t, o.dofs[3:]])) for o, t in zip(objs, tr)]
        X = torch.view_as_real(core.form_factors(kg, core.ObjectBatch(moved), True)).reshape(40, -1).double()
        worst.append(cond_rel_err(V, ((X @ X.T) / (8 * np.pi ** 3)).cpu().numpy()).max())
    print(f"\nserved disjoint objects: {worst}")
    assert np.mean(worst) <= 3e-5


@pytest.mark.parametrize("kind", ["ico4", "cube", "cloud", "splat"])
def test_each_small_radius_on_its_own(cuda, orc, kg64, kind):
    """The form factors at every radius below k = 1, each against its own norm
    (closed surfaces: A(k) ~ k, the elements' zeroth moments cancelling): the
    2e-6 norm contract radius by radius, plus what the rounding of the
    elements' own area vectors leaves (two FP32 roundings each, independent)."""
    if kind == "ico4":
        obj = G.SceneObject(G.make_triangle_mesh(*G.icosphere(4)), pg.DOF_AFFINE, G.affine_dofs(np.eye(3), [0.3, -0.2, 0.5]))
    elif kind == "cube":
        obj = shapes("cube", np.random.default_rng(0))
    elif kind == "cloud":
        obj = G.SceneObject(G.make_point_cloud(*G.create_sphere_pointcloud(3000)))
    else:
        obj = G.SceneObject(G.make_gaussian_splat(*G.create_sphere_gaussians(3000)))
    L = 64
    Jo = orc.form_factor_matrix(to_oracle(orc, [obj]), kg64.dirs, kg64.kmag)[:, 0].reshape(L, -1)
    Jg = gpu_J(kg64, [obj])[0].reshape(L, -1)
    k = kg64.kmag.reshape(L, -1)[:, 0]
    n = obj.geom.num_elements()
    inputs = 2.0 ** -23 * 4 * np.pi / np.sqrt(n) * np.sqrt(Jo.shape[1])  # sqrt(sum area^2) over the directions
    err, tol = np.linalg.norm(Jg - Jo, axis=1), 2e-6 * np.linalg.norm(Jo, axis=1) + inputs
    print(f"\n{kind}: worst radius {(err / tol)[k < 1].max():.2f} of the tolerance")
    assert (err <= tol)[k < 1].all()


def test_jacobian_translation_rows_at_each_small_radius(cuda, orc, kg64):
    """dA/dt = i k A radius by radius below k = 1, to the tolerance of the form
    factors above times k."""
    obj = G.SceneObject(G.make_triangle_mesh(*G.icosphere(4)), pg.DOF_AFFINE,
                        G.affine_dofs(np.diag([1.4, 0.9, 0.6]), [0.3, -0.2, 0.5]))
    L = 64
    got = core.dof_jacobian(kg64, core.ObjectBatch([obj])).cpu().numpy()[:3] / np.sqrt(kg64.w)
    Jo = orc.form_factor_matrix(to_oracle(orc, [obj]), kg64.dirs, kg64.kmag)[:, 0]
    ref = 1j * (kg64.dirs * kg64.kmag[:, None]).T * Jo
    k = kg64.kmag.reshape(L, -1)[:, 0]
    norm = lambda x: np.linalg.norm(x.reshape(3, L, -1), axis=(0, 2))
    inputs = 2.0 ** -23 * 4 * np.pi * 1.4 * 0.9 / np.sqrt(5120) * np.sqrt(Jo.size / L) * k
    assert (norm(got - ref) <= 2e-6 * norm(ref) + inputs)[k < 1].all()


def test_one_shot_calls_from_several_threads(cuda, kg64):
    """Host entry points take their device memory from a shared pool: concurrent
    calls give the serial calls' results, bit for bit."""
    import threading
    scenes = [[patch("tri", 200 + 50 * i, i), patch("disk", 300, 20 + i)] for i in range(4)]
    serial = [core.volume_matrix_host(kg64, s) for s in scenes]
    got = [[None] * 3 for _ in scenes]

    def work(i):
        for r in range(3):
            got[i][r] = core.volume_matrix_host(kg64, scenes[i])

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(g is not None and np.array_equal(g, serial[i]) for i in range(4) for g in got[i])
