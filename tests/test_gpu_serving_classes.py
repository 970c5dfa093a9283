"""Serving evaluations by size of object: up to 256 elements, up to 1,024, up to 4,096, more.

A row is the same whatever evaluations share its batch (bit for bit, with and
without graphs), and small objects do not pay for the large ones' split.
Volumes are held to the 1e-4 of the other serving tests, against the plain path.
"""
import time

import numpy as np
import pytest

import pointint_gb300 as pg
from pointint_gb300 import core, geometry as G
from pointint_gb300.kgrid import standard_kgrid
from pointint_gb300.serving import Server
from test_gpu_expansions import patch
from test_gpu_parity import cond_rel_err

pytestmark = pytest.mark.gpu

SIZES = [1, 12, 255, 256, 257, 1023, 1024, 1025, 4095, 4096, 4097, 6000]


def moved(o, R, t):
    return G.SceneObject(o.geom, o.dof_type, G.affine_dofs(R @ o.dofs[3:].reshape(3, 3), R @ o.dofs[:3] + t))


@pytest.mark.parametrize("use_graphs", [True, False])
@pytest.mark.parametrize("kind", ["tri", "disk"])
def test_rows_do_not_depend_on_the_batch(cuda, kind, use_graphs):
    kg = standard_kgrid(9, 32)
    lib = [patch(kind, n, 5) for n in SIZES]
    rng = np.random.default_rng(0)
    scenes = []
    for i in range(len(lib)):                     # each size with another, one of them rotated
        ids = [i, (3 * i + 1) % len(lib)]
        scenes.append((ids, np.stack([G.random_rotation(rng), np.eye(3)]), rng.normal(0, 0.3, (2, 3))))
    with Server(kg, lib, autotune=False, use_graphs=use_graphs, max_batch_queries=1, inflight_batches=1) as srv:
        alone = [srv.query(*s) for s in scenes]
    with Server(kg, lib, autotune=False, use_graphs=use_graphs) as srv:
        for order in (range(len(scenes)), reversed(range(len(scenes)))):
            tickets = {i: srv.submit(*scenes[i]) for i in order}
            for i, t in tickets.items():
                assert np.array_equal(srv.wait(t), alone[i]), SIZES[i]
    for (ids, R, T), V in zip(scenes, alone):
        ref = core.volume_matrix(kg, [moved(lib[o], r, t) for o, r, t in zip(ids, R, T)]).cpu().numpy()
        assert cond_rel_err(V, ref).max() <= 1e-4


def test_small_objects_are_not_split(cuda):
    """200 rotated boxes have 1/43 of the elements of 20 rotated meshes of 5,120
    triangles; split over as many CTAs they took longer than those."""
    kg = standard_kgrid(59, 64)
    rng = np.random.default_rng(1)
    box = G.SceneObject(G.make_triangle_mesh(*G.box_mesh([1.0, 1.3, 0.7])))
    ico = G.SceneObject(G.make_triangle_mesh(*G.icosphere(4)))

    def best(srv, obj, n):
        R, T, times = np.stack([G.random_rotation(rng) for _ in range(n)]), rng.normal(0, 0.5, (n, 3)), []
        for _ in range(8):
            t0 = time.perf_counter()
            srv.query([obj] * n, R, T)
            times.append(time.perf_counter() - t0)
        return min(times)

    with Server(kg, [box, ico], autotune=False) as srv:
        boxes, meshes = best(srv, 0, 200), best(srv, 1, 20)
    print(f"\n200 boxes {boxes * 1e6:.0f} us, 20 meshes {meshes * 1e6:.0f} us")
    assert boxes < meshes
