"""BiCGSTAB's kernels (csrc/nlgb_krylov.cu) where their layout changes: one CTA
to one per SM (256 rows each, 38,912 rows), CTAs of 256 and of 1024 threads
(622,592 rows), tiles that do and do not fill a CTA's quarters, rows that do not divide, one or several threads per
row, and chunks of sixteen iterations cut anywhere -- against the definition
(the true residual of the returned x) and the step count of the oracle's
BiCGSTAB on the small systems."""
import numpy as np
import pytest

from graphitethree_gb300 import solver, systems

pytestmark = pytest.mark.gpu

EPS = 1e-10


@pytest.mark.parametrize("nx,ny,layout", [
    (1, 1, None), (16, 16, None), (257, 1, None), (40, 33, (1, 64)), (40, 33, (4, 256)), (40, 33, (32, 320)),
    (73, 59, (2, 1024)), (256, 152, None), (1201, 33, (1, 192)), (311, 257, (1, 64)), (640, 611, None),
    (801, 777, None)])
def test_kernels(gpu_ok, oracle_mod, nx, ny, layout):
    cd = systems.convection_diffusion(nx, ny, seed=nx + ny)
    b = cd.rhs[0]
    M = solver.Matrix(cd.rp, cd.ci, cd.va)
    if layout:
        M.set_layout(*layout)
    x, info = M.solve_krylov(b, eps=EPS)
    assert info.status == "converged"
    # the recursion's residual drifts from the true one by rounding: a few
    # |A||x| eps64 an iteration, below EPS |b| for these diagonally dominant rows
    assert info.true_rel_residual <= 2 * EPS
    r = b - oracle_mod.spmv(cd.rp, cd.ci, cd.va, x)
    assert np.linalg.norm(r) <= 2 * EPS * np.linalg.norm(b)
    if cd.n <= 1400:
        its = oracle_mod.bicgstab(cd.rp, cd.ci, cd.va, b, eps=EPS, jacobi=True)[2]
        assert abs(info.iterations - its) <= max(3, its // 10)


@pytest.mark.parametrize("max_iter", [0, 1, 15, 16, 17, 31, 33])
def test_cut_anywhere(gpu_ok, max_iter):
    cd = systems.convection_diffusion(300, 200, seed=7)
    M = solver.Matrix(cd.rp, cd.ci, cd.va)
    x, info = M.solve_krylov(cd.rhs[0], eps=1e-14, max_iter=max_iter)
    assert info.iterations == max_iter
    assert np.array_equal(x, np.zeros(cd.n)) == (max_iter == 0)


@pytest.mark.parametrize("b", ["zero", "nan", "inf"])
def test_no_solution(gpu_ok, b):
    cd = systems.convection_diffusion(40, 33, seed=7)
    M = solver.Matrix(cd.rp, cd.ci, cd.va)
    v = np.full(cd.n, {"zero": 0.0, "nan": np.nan, "inf": np.inf}[b])
    x, info = M.solve_krylov(v)
    # |r|^2 = |b|^2 = inf passes |r|^2 <= eps^2 |b|^2 before the first iteration
    assert info.status == ("breakdown" if b == "nan" else "converged")
    assert info.iterations <= 1 and (b != "zero" or not x.any())
