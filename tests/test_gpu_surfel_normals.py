"""Surfels whose normals are not of unit length, as an optimiser's steps on raw
normals leave them.  For a disk |k'|^2 - (k'.n)^2 counts as 0 where a normal
longer than 1 makes it negative, at every radius and in every path (the
expansions at small k, the direct sum, the gradients).

Tolerances: the FP32 contract of the parity tests (form factors 2e-6 of the
norm and 1e-5 of the largest entry, volumes 1e-5 conditioned).
"""
import numpy as np
import pytest
import torch

import pointint_gb300 as pg
from pointint_gb300 import core, geometry as G
from pointint_gb300.kgrid import standard_kgrid
from test_gpu_expansions import check_J_weighted, patch
from test_gpu_parity import cond_rel_err, to_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def kg64():
    return standard_kgrid(9, 64)


def scaled_normals(obj, length):
    """obj with normals of the given length (Gaussians and disks share the record's layout)."""
    rows = obj.geom.elems.view(np.float64).reshape(-1, 8)
    rows[:, 3:6] *= length
    return obj


@pytest.mark.parametrize("n", [1, 64, 2049])
@pytest.mark.parametrize("length", [0.5, 0.99, 1.01, 1.05, 1.5])
def test_disks(cuda, orc, kg64, n, length):
    obj = scaled_normals(patch("disk", n, 11, (0.2, -0.1, 0.4), affine=True), length)
    check_J_weighted(kg64, orc, [obj])
    # radius by radius where the expansions apply, to the largest value there
    Jo = orc.form_factor_matrix(to_oracle(orc, [obj]), kg64.dirs, kg64.kmag)[:, 0].reshape(64, -1)
    Jg = core.form_factors(kg64, core.ObjectBatch([obj]), False).cpu().numpy().reshape(64, -1)
    err, top = np.abs(Jg - Jo).max(1), np.abs(Jo).max(1)
    k = kg64.kmag.reshape(64, -1)[:, 0]
    assert (err <= 1e-5 * top)[k < 2].all(), (err / top)[k < 2].max()


@pytest.mark.parametrize("length", [0.5, 0.9])
def test_gaussians(cuda, orc, kg64, length):
    check_J_weighted(kg64, orc, [scaled_normals(patch("gauss", 130, 12, affine=True), length)])


def test_volumes_of_long_normals(cuda, orc, kg64):
    objs = [scaled_normals(patch("disk", n, n, (0.1 * i, 0.0, 0.2)), 1.05) for i, n in enumerate((1, 64, 2049))]
    ref, _, _ = orc.volume_matrix(to_oracle(orc, objs), (kg64.dirs, kg64.kmag, kg64.w))
    assert cond_rel_err(core.volume_matrix_host(kg64, objs), ref).max() <= 1e-5


def test_one_object_has_one_definition(cuda, kg64):
    """A disk seen along its normal, |n| > 1: the factor 2 J1(x)/x is 1 whatever
    the radius, so A(k) d.n / |d.n| is the area times |n| at every k."""
    N = np.array([[0.0, 0.0, 1.05]])
    geom = G.make_point_cloud(np.zeros((1, 3)), N, np.array([0.3]))
    geom.elems.view(np.float64).reshape(-1, 8)[:, 3:6] = N  # (whatever the packing does to normals)
    from pointint_gb300.kgrid import KGrid
    k = kg64.kmag.reshape(64, -1)[:, 0]
    kg = KGrid(np.tile([0.0, 0.0, 1.0], (64, 1)), k, np.ones(64))
    A = core.form_factors(kg, core.ObjectBatch([G.SceneObject(geom, pg.DOF_AFFINE, G.affine_dofs(np.eye(3), np.zeros(3)))]),
                          False).cpu().numpy()[0]
    area = np.pi * 0.3 ** 2
    assert np.abs(A - 1.05 * area)[k > 1e-6].max() <= 1e-5 * area
