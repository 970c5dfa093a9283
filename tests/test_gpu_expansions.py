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
