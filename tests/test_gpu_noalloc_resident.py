"""The allocation-free PCG's resident form and what it hands back to the
launches: block rows at the edges of its blocks (32 rows a slice, an SM's
share, the capacity), rows too long for a block's slots, a halo too large for
its table, and patterns or diagonals that are refused.  The solution must meet
the tolerance it reports (true residual in FP64 on the host: the recursive
residual's drift over a few hundred iterations of a well-conditioned system
stays far below the factor 10 allowed)."""
import ctypes as C

import numpy as np
import pytest
import torch

from mfem_gb300 import abi
from mfem_gb300._lib import load

pytestmark = pytest.mark.gpu
TOL = 1e-10


def solve(rp, col, val, b, max_iters=2000, tol=TOL):
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (rp, col, val.ravel(), b)]
    x = torch.full((len(b),), float("nan"), dtype=torch.float64, device="cuda")
    it, err = C.c_int32(-1), C.c_double(-1.0)
    torch.cuda.synchronize()
    rc = load().mfem_gpu_bsr_pcg_noalloc(len(rp) - 1, len(col), *(d.data_ptr() for d in dev), x.data_ptr(), max_iters,
                                         tol, None, C.byref(it), C.byref(err))
    return rc, it.value, err.value, x.cpu().numpy()


def system(n, edges, seed=0):
    """Mass plus springs along edges (pairs of rows): SPD, 3x3 blocks."""
    rng = np.random.default_rng(seed)
    e = np.unique(np.sort(np.asarray(edges, dtype=np.int64).reshape(-1, 2), axis=1), axis=0)
    e = e[e[:, 0] != e[:, 1]]
    d = rng.standard_normal((len(e), 3))
    B = d[:, :, None] * d[:, None, :] + 0.2 * np.eye(3)
    diag = np.tile(np.eye(3), (n, 1, 1))
    np.add.at(diag, e[:, 0], B)
    np.add.at(diag, e[:, 1], B)
    row = np.concatenate([e[:, 0], e[:, 1], np.arange(n)])
    col = np.concatenate([e[:, 1], e[:, 0], np.arange(n)])
    val = np.concatenate([-B, -B, diag])
    order = np.lexsort((col, row))
    rp = np.zeros(n + 1, np.int32)
    np.cumsum(np.bincount(row, minlength=n), out=rp[1:])
    return rp, col[order].astype(np.int32), val[order], rng.standard_normal(3 * n)


def residual(rp, col, val, b, x):
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    y = np.zeros((len(rp) - 1, 3))
    np.add.at(y, rows, np.einsum("kij,kj->ki", val, x.reshape(-1, 3)[col]))
    return np.linalg.norm(b - y.ravel()) / np.linalg.norm(b)


def chain(n, reach=6):
    i = np.arange(n)
    return np.concatenate([np.stack([i[:-k], i[k:]], 1) for k in range(1, min(reach, n - 1) + 1)]) if n > 1 else []


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 97, 4864, 4865, 9120, 32768])
def test_sizes(gpu_lib, n):
    s = system(n, chain(n), n)
    rc, it, err, x = solve(*s)
    assert rc == abi.OK and 0 <= it < 2000 and err <= TOL  # (one row: exact at once, not counted)
    assert residual(*s, x) <= 10 * TOL
    assert np.array_equal(x, solve(*s)[3])  # the same bits again


@pytest.mark.parametrize("kind", ["long_row", "wide", "long_rows_partly_resident"])
def test_shapes(gpu_lib, kind):
    rng = np.random.default_rng(3)
    if kind == "long_row":        # 600 entries in one row: more slots than a block keeps
        n, e = 2000, np.concatenate([chain(2000), np.stack([np.zeros(600, int), rng.integers(1, 2000, 600)], 1)])
    elif kind == "wide":          # neighbours anywhere: the halo outgrows the table
        n, e = 30000, rng.integers(0, 30000, (200000, 2))
    else:                         # 61 entries a row: a block's slots outgrow its shared memory
        n, e = 12000, chain(12000, 30)
    s = system(n, e, 5)
    rc, it, err, x = solve(*s)
    assert rc == abi.OK and err <= TOL
    assert residual(*s, x) <= 10 * TOL


def test_limits_and_refusals(gpu_lib):
    rp, col, val, b = system(500, chain(500), 9)
    rc, it, err, x = solve(rp, col, val, b, max_iters=4)
    assert (rc, it) == (abi.ERR_CG_MAXITER, 4) and err > TOL
    assert solve(rp, col, val, 0 * b)[:3] == (abi.OK, 0, 0.0)
    assert solve(rp, col, val, b, tol=2.0)[:3] == (abi.OK, 0, 1.0)
    nan = b.copy()
    nan[7] = np.nan
    assert solve(rp, col, val, nan)[0] == abi.ERR_NONFINITE
    bad = col.copy()
    bad[rp[40]] = 500
    assert solve(rp, bad, val, b)[0] == abi.ERR_INVALID
    short = rp.copy()
    short[100] = short[99] - 1
    assert solve(short, col, val, b)[0] == abi.ERR_INVALID
    # and the next good system solves
    rc, _, err, x = solve(rp, col, val, b)
    assert rc == abi.OK and residual(rp, col, val, b, x) <= 10 * TOL


@pytest.mark.parametrize("n", [14592, 14593])  # three and four slices a block: each its own build of the kernel
def test_sizes_at_the_change_of_kernel(gpu_lib, n):
    test_sizes(gpu_lib, n)
