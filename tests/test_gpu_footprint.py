"""mfem_gpu_scene_footprint covers what a scene allocates on the device when it is
created and stepped, the resident solve's plan included."""
import pytest

import coop_calls

pytestmark = pytest.mark.gpu


# (4 to 1,300 free rows; 8,568; 86k, whose solve streams the matrix)
@pytest.mark.parametrize("prec,kern", [("D", "PERSISTENT"), ("D", "AUTO"), ("M", "PERSISTENT"), ("M", "AUTO")])
@pytest.mark.parametrize("dims", [(1, 1, 1), (10, 2, 2), (13, 9, 9), (20, 17, 23), (57, 32, 45)])
def test_scene_and_plan_fit(gpu_lib, tmp_path, prec, kern, dims):
    if dims[0] > 50 and (prec, kern) != ("M", "AUTO"):
        pytest.skip("no plan at this size")
    coop_calls.run(tmp_path, "", f"""
    from mfem_gb300 import abi, gpu
    from mfem_gb300.desc import SceneSpec
    from mfem_gb300.meshgen import cube_grid, enu_to_lame, face_mask
    gpu.set_tuning(0)
    V, T = cube_grid(*{dims}, 0.05)
    lam, mu = enu_to_lame(2e5, 0.4)
    s = SceneSpec(V_rest=V, tets=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam), is_fixed=face_mask(V, 0, "min"),
                  dt=1 / 60, body_force=(0.0, -9.8, 0.0), max_newton_iterations=1, max_iterative_solver_iters=20,
                  precision=abi.PRECISION_{"FP64" if prec == "D" else "MIXED"}, pcg_kernel=abi.PCG_KERNEL_{kern})
    at = lib.malloc_bytes()
    sc = gpu.Scene(s)
    made = lib.malloc_bytes() - at
    sc.step(raise_on_error=False)
    used = lib.malloc_bytes() - at
    assert any("k_cgr" in n for n in launched()) and used > made
    assert used <= gpu.footprint(s), (made, used, gpu.footprint(s))
    """)
