"""The footprint counts the resident solve's plan: the default (persistent) form
holds the same scene arrays as the two-reduction launches, which have no plan."""
import numpy as np
import pytest

from mfem_gb300 import abi
from mfem_gb300._lib import load
from mfem_gb300.build import build
from mfem_gb300.desc import SceneSpec
from mfem_gb300.meshgen import cube_grid, enu_to_lame, face_mask


def footprint(dims, prec, kern, solver=abi.SOLVER_EIGEN_CG_DIAG):
    from mfem_gb300 import gpu
    build()
    load()
    V, T = cube_grid(*dims, 0.05)
    lam, mu = enu_to_lame(2e5, 0.4)
    return gpu.footprint(SceneSpec(V_rest=V, tets=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam),
                                   is_fixed=face_mask(V, 0, "min"), dt=1 / 60, precision=prec, pcg_kernel=kern,
                                   linear_solver=solver))


@pytest.mark.parametrize("prec", [abi.PRECISION_MIXED, abi.PRECISION_FP64])
@pytest.mark.parametrize("dims", [(1, 1, 1), (13, 9, 9), (20, 17, 23)])
def test_plan_is_counted(prec, dims):
    rows = dims[0] * (dims[1] + 1) * (dims[2] + 1)
    slices = -(-rows // 32)
    plan = footprint(dims, prec, abi.PCG_KERNEL_PERSISTENT) - footprint(dims, prec, abi.PCG_KERNEL_SPLIT)
    records = 768 * (slices if prec == abi.PRECISION_FP64 else -(-slices // 8))
    exchanged = 32 * rows * (3 if prec == abi.PRECISION_FP64 else 1)
    # (a row of a grid has at least its own block and three neighbours')
    assert plan >= records + exchanged + 2 * 4 * rows
    assert plan <= 2 * (records + exchanged) + 100 * 32 * slices + 8192


def test_forms_without_a_plan():
    d = (13, 9, 9)
    for prec in (abi.PRECISION_MIXED, abi.PRECISION_FP64):
        m = abi.SOLVER_MINRES_ID
        assert footprint(d, prec, abi.PCG_KERNEL_PERSISTENT, m) == footprint(d, prec, abi.PCG_KERNEL_SPLIT, m)
    auto = footprint(d, abi.PRECISION_FP64, abi.PCG_KERNEL_AUTO)
    assert auto > footprint(d, abi.PRECISION_FP64, abi.PCG_KERNEL_FUSED)
