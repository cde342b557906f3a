"""The single-reduction resident solve in ticks (mfem_gpu_batch_step_n), whose
sums and scalars are the first warp's: bitwise the steps of each scene alone in
single launches, with blocks of one and of two tiles, scenes of one block, of up
to 32 tiles and of more (another path of the sums), both preconditioners, and an
iteration limit inside a tick."""
import numpy as np
import pytest

from mfem_gb300 import abi, gpu
from mfem_gb300.desc import SceneSpec
from mfem_gb300.meshgen import cube_grid, enu_to_lame, face_mask

pytestmark = pytest.mark.gpu


def scene(dims, **kw):
    V, T = cube_grid(*dims, 0.05)
    lam, mu = enu_to_lame(2e5, 0.4)
    return gpu.Scene(SceneSpec(V_rest=V, tets=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam),
                               is_fixed=face_mask(V, 0, "min"), dt=1 / 60, body_force=(0.0, -9.8, 0.0),
                               max_newton_iterations=3, iterative_solver_tolerance=1e-6,
                               precision=abi.PRECISION_MIXED, pcg_kernel=abi.PCG_KERNEL_FUSED,
                               **{"max_iterative_solver_iters": 400, **kw}))


# tiles: 1 + 6 + 33 (a block each); 5 x 34 + 6 (pairs of tiles); 1 (no exchange)
@pytest.mark.parametrize("dims", [[(7, 5, 5), (13, 9, 9), (16, 21, 23)], [(20, 17, 23)] * 5 + [(13, 9, 9)], [(7, 5, 5)]])
@pytest.mark.parametrize("kw", [{}, dict(linear_solver=abi.SOLVER_GPU_PCG_BLOCK), dict(max_iterative_solver_iters=131)])
def test_ticks_equal_single_launches(gpu_lib, dims, kw):
    a, b = [scene(d, **kw) for d in dims], {d: scene(d, **kw) for d in set(dims)}
    batch = gpu.Batch(a)
    stats, _ = batch.step_n(2)
    solves, iters = (gpu.kernel_stats(batch.handle)[k][1] for k in ("k_cg_solve", "k_cgf_iter"))
    assert solves > 0 and iters == 3 * solves
    cg = {}
    for d, x in b.items():
        cg[d] = sum(x.step(raise_on_error=False).cg_iterations for _ in range(2))
        assert gpu.kernel_stats(x.solo_batch_handle())["k_cg_solve"][1] == 0
    for d, x, st in zip(dims, a, stats):
        assert st.cg_iterations == cg[d]
        p, q = x.get_state(), b[d].get_state()
        for k in ("x", "v", "s", "R"):
            assert np.array_equal(p[k], q[k]), (d, k)
    batch.close()
