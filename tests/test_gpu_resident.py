"""The resident PCG (one cooperative launch a solve, the matrix in shared
memory): a scene that left the PCG form to the library takes the same steps,
bitwise, as with the launches of that form, and the default (persistent) form
the same as the two-reduction launches.  Sizes at the edges of its blocks (a
slice is 32 rows, a reduction tile 256, 32 tiles change the sum's path, 152
blocks an SM's share) and options that change its loop: block Jacobi, the
residual replacement every 25 iterations, the iteration limit."""
import numpy as np
import pytest

from mfem_gb300 import abi, configs, gpu
from mfem_gb300.desc import SceneSpec
from mfem_gb300.meshgen import cube_grid, enu_to_lame, face_mask

pytestmark = pytest.mark.gpu

M, D = abi.PRECISION_MIXED, abi.PRECISION_FP64
AUTO, FUSED, SPLIT, PERS = (abi.PCG_KERNEL_AUTO, abi.PCG_KERNEL_FUSED, abi.PCG_KERNEL_SPLIT,
                            abi.PCG_KERNEL_PERSISTENT)


def spec(dims, prec, kern, **kw):
    V, T = cube_grid(*dims, 0.05)
    lam, mu = enu_to_lame(2e5, 0.4)
    rng = np.random.default_rng(11)
    fixed = face_mask(V, 0, "min")
    V = V + rng.uniform(-0.005, 0.005, V.shape) * (fixed == 0)[:, None]
    s = SceneSpec(V_rest=V, tets=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam), is_fixed=fixed, dt=1 / 60,
                  max_newton_iterations=4, iterative_solver_tolerance=1e-6, newton_residual_tolerance=1e-5,
                  max_iterative_solver_iters=2000, precision=prec, pcg_kernel=kern)
    for k, v in kw.items():
        setattr(s, k, v)
    return s


def run(s, steps=2):
    sc = gpu.Scene(s)
    stats = [sc.step(raise_on_error=False) for _ in range(steps)]
    st = sc.get_state()
    ks = gpu.kernel_stats(sc.solo_batch_handle())
    n = sc.n_free
    sc.close()
    return [(q.status, q.newton_iterations, q.cg_iterations) for q in stats], st, ks["k_cg_solve"][1], n


def same(a, b):
    assert a[0] == b[0]
    for k in ("x", "v", "s", "R"):
        assert np.array_equal(a[1][k], b[1][k]), k


# (free rows: 4, 32, 36, 252, 264, 1300, 8448 = 33 tiles)
DIMS = [(1, 1, 1), (2, 3, 3), (4, 2, 2), (7, 5, 5), (11, 3, 5), (13, 9, 9), (16, 21, 23)]


@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("prec", [M, D])
def test_persistent_equals_the_two_reduction_launches(gpu_lib, dims, prec):
    a, b = run(spec(dims, prec, PERS)), run(spec(dims, prec, SPLIT))
    assert a[2] > 0 and b[2] == 0
    same(a, b)


@pytest.mark.parametrize("dims,kern", [((4, 2, 2), FUSED), ((7, 5, 5), FUSED), ((11, 3, 5), FUSED), ((13, 9, 9), SPLIT),
                                       ((60, 27, 25), SPLIT)])  # the last: 171 tiles, two blocks an SM
def test_auto_equals_the_launches_of_its_form(gpu_lib, dims, kern):
    a, b = run(spec(dims, M, AUTO)), run(spec(dims, M, kern))
    assert a[2] > 0 and b[2] == 0
    same(a, b)


@pytest.mark.parametrize("dims,prec,ref", [((7, 5, 5), M, FUSED), ((13, 9, 9), M, SPLIT), ((7, 5, 5), D, SPLIT)])
@pytest.mark.parametrize("kw", [dict(linear_solver=abi.SOLVER_GPU_PCG_BLOCK), dict(max_iterative_solver_iters=1),
                                dict(max_iterative_solver_iters=25), dict(max_iterative_solver_iters=26),
                                dict(iterative_solver_tolerance=0.5)])
def test_options(gpu_lib, dims, prec, ref, kw):
    same(run(spec(dims, prec, AUTO, **kw)), run(spec(dims, prec, ref, **kw)))


def test_lanes_of_resident_batches_side_by_side(gpu_lib):
    """Batches of different sizes whose resident solves together outnumber
    the SMs, stepped from several threads at once."""
    specs = [spec(d, M, FUSED) for d in [(16, 21, 23)] * 5 + [(7, 5, 5), (13, 9, 9), (20, 20, 20), (24, 20, 21)]]
    a, b = [gpu.Scene(s) for s in specs], [gpu.Scene(s) for s in specs]
    lanes, one = gpu.Lanes(a, lanes=3), gpu.Batch(b)
    s1, _ = lanes.step_n(3)
    s2, _ = one.step_n(3)
    for x, y, p, q in zip(a, b, s1, s2):
        assert p.cg_iterations == q.cg_iterations
        assert np.array_equal(x.positions(), y.positions())
    lanes.close()
    one.close()


# (free rows: 4,864 and 4,896, the last with one slice a block and the first
# with two; 9,728 and 9,760, two and four; 17,550: 69 tiles, the sum's third group)
@pytest.mark.parametrize("dims", [(19, 15, 15), (17, 17, 15), (19, 15, 31), (61, 15, 9), (26, 26, 24)])
def test_fp64_blocks_of_one_two_and_four_slices(gpu_lib, dims):
    kw = dict(max_iterative_solver_iters=40)
    a, b = run(spec(dims, D, PERS, **kw), 1), run(spec(dims, D, SPLIT, **kw), 1)
    assert a[2] > 0 and b[2] == 0
    same(a, b)


# (free rows: 86,526 = 338 tiles, three a block; 223,138 = 872 tiles, six)
@pytest.mark.parametrize("dims,kw", [((57, 32, 45), {}), ((57, 32, 45), dict(linear_solver=abi.SOLVER_GPU_PCG_BLOCK)),
                                     ((57, 32, 45), dict(max_iterative_solver_iters=7)), ((59, 60, 61), {})])
def test_blocks_of_several_tiles_that_stream_the_matrix(gpu_lib, dims, kw):
    a, b = run(spec(dims, M, AUTO, **kw), 1), run(spec(dims, M, FUSED, **kw), 1)
    same(a, b)


def test_batch_of_scenes_whose_blocks_hold_several_tiles(gpu_lib):
    """18 scenes together of more than two tiles an SM (one to 35 tiles each):
    the steps are those of each scene alone in single launches."""
    specs = [spec(d, M, FUSED) for d in [(20, 20, 20)] * 10 + [(7, 5, 5), (13, 9, 9), (4, 2, 2), (16, 21, 23)] * 2]
    one = [gpu.Scene(s) for s in specs]
    ref = [run(s, 2) for s in (specs[0], *specs[10:14])]
    batch = gpu.Batch(one)
    batch.step_n(2)
    for sc, i in zip(one, [0] * 10 + [1, 2, 3, 4] * 2):
        st = sc.get_state()
        for k in ("x", "v", "s", "R"):
            assert np.array_equal(st[k], ref[i][1][k]), (i, k)
    batch.close()
