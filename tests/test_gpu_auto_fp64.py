"""FP64 scenes of at most four PCG tiles that leave the PCG form to the library:
a scene takes the same steps, bitwise, alone and in a batch, one step or several
a call, as the resident solve of the two-reduction iteration."""
import numpy as np
import pytest

from mfem_gb300 import abi, gpu
from mfem_gb300.desc import SceneSpec
from mfem_gb300.meshgen import cube_grid, enu_to_lame, face_mask

pytestmark = pytest.mark.gpu


def scenes(n):
    out = []
    for i in range(n):
        V, T = cube_grid(6 + i, 3, 2, 0.1)  # 72 free rows and more: one tile each
        lam, mu = enu_to_lame(3e5, 0.4)
        out.append(gpu.Scene(SceneSpec(
            V_rest=V, tets=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam), is_fixed=face_mask(V, 0, "min"),
            dt=1 / 60, body_force=(0.0, -9.8, 0.0), max_newton_iterations=6, iterative_solver_tolerance=1e-10,
            precision=abi.PRECISION_FP64, pcg_kernel=abi.PCG_KERNEL_AUTO)))
    return out


@pytest.mark.parametrize("n", [2, 4])
@pytest.mark.parametrize("one_call", [False, True])
def test_alone_and_in_a_small_batch(gpu_lib, n, one_call):
    a, b = scenes(n), scenes(n)
    batch = gpu.Batch(b)
    if one_call:
        batch.step_n(3)
    else:
        for _ in range(3):
            batch.step()
    assert gpu.kernel_stats(batch.handle)["k_cg_solve"][1] > 0
    for x, y in zip(a, b):
        for _ in range(3):
            x.step()
        p, q = x.get_state(), y.get_state()
        for k in ("x", "v", "s", "R"):
            assert np.array_equal(p[k], q[k]), k
    batch.close()
