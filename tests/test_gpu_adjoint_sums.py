"""The adjoint adds every direction's contribution compensated.

Directions come in groups of eight equal ones (the kernels stage eight at a
time), the first with weight 1, the others with 2^-26: each of those is less than half a unit
in the last place of the first, so a plain FP32 sum over the eight loses them
all, 7 2^-26 = 1.0e-7 of the gradient.  Weights are powers of four, so every
contribution scales exactly, and gradients under the large and the small
weights alone give what the sum should be.  What rounds otherwise (the last
place of each element's total) has no sign in common, so the slope of the
difference over the gradients stays below 2e-8.
"""
import numpy as np
import pytest

import pointint_gb300 as pg
from pointint_gb300 import core, geometry as G
from pointint_gb300.kgrid import KGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_radii", [2, 16])
@pytest.mark.parametrize("kind", ["tri", "disk", "gauss"])
def test_small_contributions_are_kept(cuda, kind, n_radii):
    rng = np.random.default_rng(0)
    d = rng.normal(size=(64, 3))
    d[:, 2] = np.abs(d[:, 2]) + 0.1                 # no antipodes
    dirs = np.repeat(d / np.linalg.norm(d, axis=1, keepdims=True), 8, axis=0)
    M = len(dirs)
    k = np.linspace(0.7, 3.0, n_radii)
    first = np.tile(np.arange(M) % 8 == 0, n_radii)

    if kind == "tri":
        geom = G.make_triangle_mesh(*G.icosphere(2))
    elif kind == "disk":
        geom = G.make_point_cloud(*G.create_sphere_pointcloud(256))
    else:
        geom = G.make_gaussian_splat(*G.create_sphere_gaussians(256))
    batch = core.ObjectBatch([G.SceneObject(geom, pg.DOF_AFFINE, G.affine_dofs(np.diag([1.4, 0.9, 0.6]), [0.1, 0.2, 0.3]))])

    def grads(w):
        kg = KGrid(np.tile(dirs, (n_radii, 1)), np.repeat(k, M), w)
        tri, surf = core.element_gradients(kg, batch, core.form_factors(kg, batch), np.ones((1, 1)))
        return (tri if kind == "tri" else surf).cpu().numpy().astype(np.float64)

    eps = 2.0 ** -26
    large, small = grads(np.where(first, 1.0, 0.0)), grads(np.where(first, 0.0, 1.0))
    got, want = grads(np.where(first, 1.0, eps)), large + eps * small
    slope = ((got - want) * large).sum(0) / (large * large).sum(0)   # per kind of entry
    print(f"\n{kind} {n_radii}: slopes {slope.min():.1e} .. {slope.max():.1e}")
    assert np.abs(slope).max() <= 2e-8, slope
