"""The stopping test |r|^2 < max(tol^2 |b|^2, DBL_MIN) of the mixed PCG forms at
tolerances whose square, or the tolerance itself, lies outside FP32's range:
the threshold is formed in FP64, so that a tolerance no FP32 residual can meet
counts as zero, a negative one as its magnitude and a huge one is met at once."""
import numpy as np
import pytest

from mfem_gb300 import abi, gpu
from mfem_gb300.desc import SceneSpec
from mfem_gb300.meshgen import cube_grid, enu_to_lame, face_mask

pytestmark = pytest.mark.gpu

KERNELS = [abi.PCG_KERNEL_AUTO, abi.PCG_KERNEL_FUSED, abi.PCG_KERNEL_SPLIT, abi.PCG_KERNEL_PERSISTENT]


def run(dims, kern, tol):
    V, T = cube_grid(*dims, 0.05)
    lam, mu = enu_to_lame(2e5, 0.4)
    sc = gpu.Scene(SceneSpec(V_rest=V, tets=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam),
                             is_fixed=face_mask(V, 0, "min"), dt=1 / 60, body_force=(0.0, -9.8, 0.0),
                             max_newton_iterations=2, iterative_solver_tolerance=tol, max_iterative_solver_iters=60,
                             precision=abi.PRECISION_MIXED, pcg_kernel=kern))
    st = sc.step(raise_on_error=False)
    x = sc.positions()
    sc.close()
    return st.cg_iterations, x


@pytest.mark.parametrize("kern", KERNELS)
@pytest.mark.parametrize("dims", [(7, 5, 5), (13, 9, 9)])  # 252 and 1,300 free rows: one tile and six
@pytest.mark.parametrize("tol,same_as", [(9e-38, 0.0), (1e-38, 0.0), (1e-40, 0.0), (1e-44, 0.0), (1e-200, 0.0),
                                         (-0.05, 0.05)])
def test_tolerances_out_of_fp32s_range(gpu_lib, dims, kern, tol, same_as):
    (n, x), (n0, x0) = run(dims, kern, tol), run(dims, kern, same_as)
    assert n == n0 > 0
    assert np.array_equal(x, x0)


@pytest.mark.parametrize("kern", KERNELS)
@pytest.mark.parametrize("tol", [2.0, 1e20, 1e39])
def test_a_tolerance_above_one_is_met_before_the_first_iteration(gpu_lib, kern, tol):
    assert run((7, 5, 5), kern, tol)[0] == 0
