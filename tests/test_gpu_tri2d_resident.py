"""The 2-D path's resident PCG at the sizes where its blocks change: fewer
rows than a block's 32, exactly as many and one more, 4 to 32 blocks, the
last size of the two-reduction form (1,024 rows) and the first of the
single-reduction form, two blocks an SM, and a sheet too large to be resident
(the grid form); each against the FP64 oracle within 1e-8 of the bounding-box
diagonal after two steps, with equal Newton counts."""
import numpy as np
import pytest

from mfem_gb300.desc import Tri2dSpec
from mfem_gb300.meshgen import enu_to_lame, face_mask, square_grid

pytestmark = pytest.mark.gpu


# free rows: 6, 32, 33, 63, 110, 500, 600, 1,024, 1,025, 2,800, 10,100
@pytest.mark.parametrize("nx,ny", [(2, 2), (4, 7), (3, 10), (7, 8), (10, 10), (20, 24), (24, 24), (32, 31), (41, 24),
                                   (40, 69), (100, 100)])
def test_sizes_match_the_oracle(gpu_lib, nx, ny):
    import oracle
    from mfem_gb300.tri2d import Tri2dScene
    V, T = square_grid(nx, ny, 1.0 / max(nx, ny))
    lam, mu = enu_to_lame(1e5, 0.4)
    fixed = face_mask(V, 0, "min")
    sp = Tri2dSpec(V_rest=V, tris=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam), is_fixed=fixed, dt=0.01,
                   max_newton_iterations=3, iterative_solver_tolerance=1e-10, max_iterative_solver_iters=5000)
    o, g = oracle.OracleTri2d(sp), Tri2dScene(sp)
    for _ in range(2 if g.n_free < 5000 else 1):
        so, sg = o.step(), g.step()
        assert (sg.status, sg.newton_iterations) == (so.status, so.newton_iterations)
    xo, xg = o.get_state()["x"], g.get_state()["x"]
    assert np.abs(xg - xo).max() < 1e-8 * np.linalg.norm(np.ptp(xo, axis=0))
    assert np.abs(xo - V).max() > 1e-5
    g.close()


def test_resident_and_grid_forms_agree_on_a_large_sheet(gpu_lib):
    """Past the resident form's capacity the grid form runs; one Newton
    iteration of a 90,000-vertex sheet meets the tolerance."""
    from mfem_gb300.tri2d import Tri2dScene
    V, T = square_grid(300, 299, 1.0 / 300)
    lam, mu = enu_to_lame(1e4, 0.4)
    sp = Tri2dSpec(V_rest=V, tris=T, mu=np.full(len(T), mu), lam=np.full(len(T), lam),
                   is_fixed=face_mask(V, 0, "min"), dt=0.003, max_newton_iterations=1,
                   iterative_solver_tolerance=1e-8, max_iterative_solver_iters=5000)
    g = Tri2dScene(sp)
    st = g.step()
    assert st.cg_error < 1e-8 and 0 < st.cg_iterations < 5000
    g.close()
