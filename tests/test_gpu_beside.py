"""Batches stepped side by side (mfem_gpu_batches_step_n): those whose resident
solves would only take turns on the SMs run the launches while they are beside
each other and the resident solve alone; small ones stay resident; with the same
bits."""
import numpy as np
import pytest

from mfem_gb300 import abi, gpu
from mfem_gb300.desc import SceneSpec
from mfem_gb300.meshgen import cube_grid, enu_to_lame, face_mask

pytestmark = pytest.mark.gpu


def scenes(dims, n, kern):
    V, T = cube_grid(*dims, 0.05)
    lam, mu = enu_to_lame(2e5, 0.4)
    return [gpu.Scene(SceneSpec(V_rest=V, tets=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam),
                                is_fixed=face_mask(V, 0, "min"), dt=1 / 60, body_force=(0.0, -9.8, 0.0),
                                max_newton_iterations=4, iterative_solver_tolerance=1e-5,
                                max_iterative_solver_iters=300, precision=abi.PRECISION_MIXED, pcg_kernel=kern))
            for _ in range(n)]


def solves_and_iters(batch):
    ks = gpu.kernel_stats(batch.handle)
    return ks["k_cg_solve"][1], ks["k_cgf_iter"][1]


# 10 scenes of 33 tiles a lane: more than two tiles an SM; 3 of five tiles: 15 SMs
@pytest.mark.parametrize("dims,n,turns", [((20, 20, 20), 10, True), ((13, 9, 9), 3, False)])
def test_two_lanes(gpu_lib, dims, n, turns):
    a, b = scenes(dims, 2 * n, abi.PCG_KERNEL_FUSED), scenes(dims, n, abi.PCG_KERNEL_FUSED)
    lanes, alone = gpu.Lanes(a, lanes=2), gpu.Batch(b)
    lanes.step_n(3)
    alone.step_n(3)
    solves, iters = solves_and_iters(alone)
    assert solves > 0 and iters == 3 * solves
    for batch in lanes.batches:
        solves, iters = solves_and_iters(batch)
        if turns:  # (but for the last ticks of the lane that ends later)
            assert iters - 3 * solves > 16 * 4 * solves
        else:
            assert solves > 0 and iters == 3 * solves
    for x in a:
        assert np.array_equal(x.positions(), b[0].positions())
    lanes.close()
    alone.close()


def test_single_scenes_in_lanes_take_turns(gpu_lib):
    """Two scenes of 113 tiles, left to the library (the two-reduction solve):
    three quarters of the SMs each, in turns."""
    a = scenes((30, 30, 30), 3, abi.PCG_KERNEL_AUTO)
    lanes = gpu.Lanes(a[:2], lanes=2)
    lanes.step_n(1)
    a[2].step()
    for batch in lanes.batches:
        ks = gpu.kernel_stats(batch.handle)
        assert ks["k_cg_solve"][1] > 0 and ks["k_cg_spmv"][1] == 0
    for x in a[:2]:
        assert np.array_equal(x.positions(), a[2].positions())
    lanes.close()
