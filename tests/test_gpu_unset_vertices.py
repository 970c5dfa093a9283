"""TriangleMeshDoF triangles with unset vertex ids contribute nothing: their
element gradients are exactly zero, also in a patch far from the object's
origin (where such a triangle is stored) beside triangles that are set."""
import numpy as np
import pytest

import pointint_gb300 as pg
from pointint_gb300 import core, geometry as G
from pointint_gb300.kgrid import standard_kgrid
from test_gpu_gradients import assert_grad_close
from test_gpu_parity import to_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("unset", [[0], [5], [1, 2, 3, 30], [64], list(range(32, 36))],
                         ids=["first", "mixed leaf", "several", "last", "whole leaf"])
@pytest.mark.parametrize("size", [1e-1, 1e-3, 1e-5])
def test_unset_triangles_have_zero_gradients(cuda, orc, unset, size):
    rng = np.random.default_rng(len(unset))
    n = 65                                       # two full patches and one triangle
    ctr = np.where(np.arange(n) % 64 < 32, 1.0, -1.0)[:, None] * np.array([1.0, 0.3, -0.2])
    V = (ctr[:, None, :] + size * rng.normal(size=(n, 3, 3))).reshape(-1, 3)
    geom = G.make_triangle_mesh(V, np.arange(3 * n).reshape(n, 3))
    geom.elems["vid"][unset] = -1
    P, N, R = G.create_sphere_pointcloud(100)
    objs = [G.SceneObject(geom, pg.DOF_TRIANGLE_MESH, V.reshape(-1)), G.SceneObject(G.make_point_cloud(P, N, R))]
    kg = standard_kgrid(9, 64)
    batch = core.ObjectBatch(objs)
    W = np.ones((2, 2))
    tri, _ = core.element_gradients(kg, batch, core.form_factors(kg, batch), W)
    tri = tri.cpu().numpy()
    assert np.isfinite(tri).all()
    assert (tri[unset] == 0).all()
    _, grad = core.volume_matrix_grad_host(kg, objs)
    _, ref, _ = orc.volume_matrix(to_oracle(orc, objs), (kg.dirs, kg.kmag, kg.w), orc.VOLUME_ONLY | orc.GRADIENT)
    assert_grad_close(grad[0][1], ref[0][1], what="vertices")
