"""Cooperative launches that the runtime refuses (a stream or process limited to
a part of the SMs): the forms that need no co-residency run instead.  And waits
between their blocks that run out.  Each test runs in a child process whose
cooperative launches go through a stand-in."""
import pytest

import coop_calls

pytestmark = pytest.mark.gpu

SCENE = """
from mfem_gb300 import abi, gpu
from mfem_gb300.desc import SceneSpec
from mfem_gb300.meshgen import cube_grid, enu_to_lame, face_mask
def scene(dims, prec, kern, **kw):
    V, T = cube_grid(*dims, 0.05)
    lam, mu = enu_to_lame(2e5, 0.4)
    return gpu.Scene(SceneSpec(V_rest=V, tets=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam),
                               is_fixed=face_mask(V, 0, "min"), dt=1 / 60, body_force=(0.0, -9.8, 0.0),
                               max_newton_iterations=3, iterative_solver_tolerance=1e-6, precision=prec,
                               max_iterative_solver_iters=400, pcg_kernel=kern, **kw))
M, D = abi.PRECISION_MIXED, abi.PRECISION_FP64
"""


def test_allocation_free_solve(gpu_lib, tmp_path):
    # (980 rows: 31 blocks; both solves to 1e-10, their sums in another order)
    coop_calls.run(tmp_path, SCENE, """
    import torch
    from mfem_gb300._lib import load
    sc = scene((20, 6, 6), D, abi.PCG_KERNEL_SPLIT, linear_solver=abi.SOLVER_GPU_PCG_BLOCK)
    sc.step()
    rp, col, val, rhs = sc.get_system()
    dev = [torch.from_numpy(np.ascontiguousarray(a).ravel()).cuda() for a in (rp, col, val, rhs)]
    x = torch.zeros(3 * sc.n_free, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    def solve():
        it, err = C.c_int32(-1), C.c_double(-1)
        x.zero_()
        torch.cuda.synchronize()
        rc = load().mfem_gpu_bsr_pcg_noalloc(sc.n_free, sc.nnzb, *[C.c_void_p(a.data_ptr()) for a in dev],
                                             C.c_void_p(x.data_ptr()), 3000, C.c_double(1e-10), None, C.byref(it),
                                             C.byref(err))
        return rc, it.value, x.cpu().numpy()
    rc, it, ref = solve()
    assert rc == 0 and it > 0 and any("k_na_resident" in n for n in launched())
    for on, runs in ((1, False), (1, False), (0, True)):
        lib.coop_refuse(on)
        rc, n, y = solve()
        assert rc == 0 and abs(n - it) <= max(2, it // 50), (rc, n, it)
        assert any("k_na_resident" in k for k in launched()) == runs
        assert np.abs(y - ref).max() <= 1e-7 * np.abs(ref).max()
    # rows that nobody sends: the wait runs out, the next solve is as ever
    lib.coop_drop(1)
    assert solve()[0] == abi.ERR_TIMEOUT
    lib.coop_drop(0)
    rc, n, y = solve()
    assert rc == 0 and n == it and np.array_equal(y, ref)
    """)


@pytest.mark.parametrize("form", ["split", "fused", "ticks"])
def test_scenes_that_leave_the_form_to_the_library(gpu_lib, tmp_path, form):
    """Six tiles: the two-reduction solve; one tile: the single-reduction loop;
    a batch of those in ticks.  The launches take the same steps, bitwise."""
    coop_calls.run(tmp_path, SCENE, f"""
    form = {form!r}
    def steps():
        if form == "ticks":
            s = [scene(d, M, abi.PCG_KERNEL_FUSED) for d in [(13, 9, 9), (7, 5, 5)]]
            b = gpu.Batch(s)
            b.step_n(2)
            h = b.handle
        else:
            s = [scene((13, 9, 9) if form == "split" else (7, 5, 5), M, abi.PCG_KERNEL_AUTO)]
            for _ in range(2):
                s[0].step(raise_on_error=False)
            h = s[0].solo_batch_handle()
        return [x.positions() for x in s], gpu.kernel_stats(h)["k_cg_solve"][1], launched()
    ref, n, names = steps()
    kernel = dict(split="k_cgr_split", fused="k_cgr_fused", ticks="k_cgr_fused")[form]
    assert n > 0 and any(kernel in k for k in names), names
    lib.coop_refuse(1)
    got, n, names = steps()
    assert n == 0 and not names
    assert all(np.array_equal(a, b) for a, b in zip(ref, got))
    """)


@pytest.mark.parametrize("nx,ny,kernel", [(12, 8, "t2_pcg_res2"), (64, 20, "t2_pcg_res")])  # 99 and 1,302 free rows
def test_sheets(gpu_lib, tmp_path, nx, ny, kernel):
    # (Newton's converged states of forms that add in another order: 1e-9 of
    # the sheet apart; the bound is the one on parity, 1e-6)
    coop_calls.run(tmp_path, "", f"""
    from mfem_gb300 import abi
    from mfem_gb300.desc import Tri2dSpec
    from mfem_gb300.meshgen import enu_to_lame, square_grid
    from mfem_gb300.tri2d import Tri2dScene
    def steps():
        V, T = square_grid({nx}, {ny}, 1.0 / {nx})
        lam, mu = enu_to_lame(1e5, 0.45)
        sc = Tri2dScene(Tri2dSpec(V_rest=V, tris=T, mu=np.full(len(T), float(mu)), lam=np.full(len(T), float(lam)),
                                  density_const=1000.0, bc_type=abi.BC_HANGENDS, bc_ratio=0.01, bc_axis=0, dt=0.0333,
                                  body_force=(0.0, -9.8, 0.0), max_newton_iterations=10,
                                  max_linesearch_iterations=20, max_iterative_solver_iters=10000,
                                  iterative_solver_tolerance=1e-10))
        st = [sc.step().status for _ in range(steps_)]
        x = sc.get_state()["x"]
        sc.close()
        return np.array(x), st, launched()
    steps_ = 2
    ref, st, names = steps()
    assert any({kernel!r} in k for k in names), names
    # rows that nobody sends: the wait runs out, the next sheet is as ever
    lib.coop_drop(1)
    steps_ = 1
    assert steps()[1] == [abi.ERR_TIMEOUT]
    lib.coop_drop(0)
    steps_ = 2
    again, st, names = steps()
    assert abi.ERR_TIMEOUT not in st and np.array_equal(again, ref)
    lib.coop_refuse(1)
    got, st, names = steps()
    assert not names
    assert np.abs(got - ref).max() <= 1e-6, np.abs(got - ref).max()
    """)


# k_cgr_split (6, 33 and 263 tiles), k_cgr_split64, k_cgr_wide; in ticks k_cgr_fused of 8 and of 16 warps
@pytest.mark.parametrize("dims,prec,kern,n", [
    ((13, 9, 9), "M", "PERSISTENT", 1), ((16, 21, 23), "M", "PERSISTENT", 1), ((40, 40, 40), "M", "PERSISTENT", 1),
    ((13, 9, 9), "D", "PERSISTENT", 1), ((57, 32, 45), "M", "AUTO", 1), ((13, 9, 9), "M", "FUSED", 3),
    ((20, 17, 23), "M", "FUSED", 5)])
def test_a_wait_that_runs_out(gpu_lib, tmp_path, dims, prec, kern, n):
    """The last block is left out of the grid, so that the others wait for sums
    nobody sends until their limit of two seconds, then leave: the step reports
    the timeout, and the next solves, on this scene and others, are as ever."""
    coop_calls.run(tmp_path, SCENE, f"""
    import time
    from mfem_gb300._lib import MfemError
    gpu.set_tuning(0)
    def make():
        s = [scene({dims}, {prec}, abi.PCG_KERNEL_{kern}) for _ in range({n})]
        return s, gpu.Batch(s)
    def step(b):
        return b.step_n(1) if {n} > 1 else b.step()
    s, b = make()
    snap = [x.snapshot() for x in s]
    step(b)
    assert any("k_cgr" in k for k in launched())
    ref = [x.positions() for x in s]
    lib.coop_drop(1)
    t, u = make()
    t0 = time.perf_counter()
    try:
        step(u)
        assert False, "no timeout"
    except MfemError as e:
        assert e.status == abi.ERR_TIMEOUT, e.status
    waited = time.perf_counter() - t0
    assert 1.9 < waited < 20, waited
    lib.coop_drop(0)
    direct = {kern!r} == "PERSISTENT"  # (graphs keep the grid they were captured with)
    for x, q in zip(t if direct else s, snap):
        x.restore(q)
    step(u if direct else b)
    assert all(np.array_equal(x.positions(), r) for x, r in zip(t if direct else s, ref))
    v, c = make()
    step(c)
    assert all(np.array_equal(x.positions(), r) for x, r in zip(v, ref))
    """)


def test_which_resident_kernel_runs(gpu_lib, tmp_path):
    """The kernels behind the comparisons with the launches in
    test_gpu_resident.py: that the resident ones ran, at each of their sizes."""
    coop_calls.run(tmp_path, SCENE, """
    gpu.set_tuning(0)
    A, P, F = abi.PCG_KERNEL_AUTO, abi.PCG_KERNEL_PERSISTENT, abi.PCG_KERNEL_FUSED
    block = dict(linear_solver=abi.SOLVER_GPU_PCG_BLOCK)
    # (mangled template arguments: Lb = scaled or not, Li = threads)
    for dims, prec, kern, kw, name in [
            ((7, 5, 5), M, A, {}, "k_cgr_fusedILb1ELi256E"), ((7, 5, 5), M, A, block, "k_cgr_fusedILb0ELi256E"),
            ((11, 3, 5), M, A, {}, "k_cgr_fusedILb1ELi512E"), ((13, 9, 9), M, A, {}, "k_cgr_splitILi256E"),
            ((13, 9, 9), M, A, block, "k_cgr_splitILi256E"), ((60, 27, 25), M, A, {}, "k_cgr_splitILi512E"),
            ((57, 32, 45), M, A, {}, "k_cgr_wideILb1E"), ((57, 32, 45), M, A, block, "k_cgr_wideILb0E"),
            ((59, 60, 61), M, A, {}, "k_cgr_wideILb1E"), ((2, 3, 3), M, P, {}, "k_cgr_splitILi256E"),
            ((7, 5, 5), D, A, {}, "k_cgr_split64"), ((19, 15, 15), D, P, {}, "k_cgr_split64"),
            ((26, 26, 24), D, P, {}, "k_cgr_split64")]:
        s = scene(dims, prec, kern, **kw)
        launched()
        s.step(raise_on_error=False)
        names = launched()
        assert names and all(name in k for k in names), (dims, kern, kw, names)
        assert gpu.kernel_stats(s.solo_batch_handle())["k_cg_solve"][1] > 0
        s.close()
    # the batch of 18 scenes on more than two tiles an SM, and lanes of small ones
    s = [scene(d, M, F) for d in [(20, 20, 20)] * 10 + [(7, 5, 5), (13, 9, 9), (4, 2, 2), (16, 21, 23)] * 2]
    b = gpu.Batch(s)
    b.step_n(1)
    assert all("k_cgr_wide" in k for k in launched()) and gpu.kernel_stats(b.handle)["k_cg_solve"][1] > 0
    b.close()
    lanes = gpu.Lanes(s[10:], lanes=3)
    lanes.step_n(1)
    assert {"k_cgr_fused" in k for k in launched()} == {True}
    assert all(gpu.kernel_stats(x.handle)["k_cg_solve"][1] > 0 for x in lanes.batches)
    lanes.close()
    """)
