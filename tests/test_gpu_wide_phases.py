"""The gap phases k (v - u), k (w - v) of wide triangles keep the radius as a
double-float: with the projections exact in FP32, the form factor's error does
not grow with the phase.

One triangle with projections 0, g, -g on the z direction (its centroid at 0):
e[..] = (cos kg - 1) / (kg)^2.  What rounds: three phasors (1.5e-7 each at most,
the pair's difference at the scale of 1), three reciprocals and a few products,
so 2e-6 of the envelope 2 / (kg)^2 bounds the error; a radius rounded to FP32
would leave kg 2^-24, 6e-4 at kg = 1e4.
"""
import numpy as np
import pytest

import pointint_gb300 as pg
from pointint_gb300 import core, geometry as G
from pointint_gb300.kgrid import KGrid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_radii", [2, 4, 7, 8, 32, 65])
@pytest.mark.parametrize("g", [1.0, 0.125])
def test_gap_phases(cuda, n_radii, g):
    k = np.sort(np.random.default_rng(n_radii).uniform(20.0 / g, 1.0e4 / g, n_radii))
    kg = KGrid(np.tile([0.0, 0.0, 1.0], (n_radii, 1)), k, np.ones(n_radii))
    V = np.array([[0, 0, 0], [1, 0, g], [0, 1, -g]], dtype=np.float64)
    obj = G.SceneObject(G.make_triangle_mesh(V, np.array([[0, 1, 2]])), pg.DOF_AFFINE,
                        G.affine_dofs(np.eye(3), np.zeros(3)))
    A = core.form_factors(kg, core.ObjectBatch([obj]), False).cpu().numpy()[0]
    ref = -2 * 0.5 * (np.cos(k * g) - 1) / (k * g) ** 2     # -2 (khat . S) e[..], S_z = 1/2
    err = np.abs(A - ref) / (2 / (k * g) ** 2)
    print(f"\nlargest error over the envelope {err.max():.1e}")
    assert err.max() <= 2e-6, err
