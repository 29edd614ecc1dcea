"""GMRES step kernels (csrc/nlgb_krylov.cu) where their layout changes: one
CTA to one per SM (256 rows each, 38,912 rows), rows that do and do not
divide, groups of eight Krylov vectors, the longest restart, and one or
several threads per row -- against the definition (the true residual of the
returned x) and the step count of the oracle's GMRES on the small systems."""
import numpy as np
import pytest

from graphitethree_gb300 import solver, systems

pytestmark = pytest.mark.gpu

EPS = 1e-10


@pytest.mark.parametrize("nx,ny,restart,tpr", [
    (1, 1, 5, 0), (16, 16, 1, 0), (257, 1, 7, 0), (16, 17, 8, 0), (40, 33, 9, 4), (40, 33, 64, 0), (40, 33, 100, 32),
    (256, 152, 17, 0), (1201, 33, 16, 2), (311, 257, 30, 0)])
def test_step_kernels(gpu_ok, oracle_mod, nx, ny, restart, tpr):
    cd = systems.convection_diffusion(nx, ny, seed=nx + restart)
    b = cd.rhs[0]
    M = solver.Matrix(cd.rp, cd.ci, cd.va)
    if tpr:
        M.set_layout(tpr, 0)
    x, info = M.solve_krylov(b, method="gmres", eps=EPS, restart=restart)
    assert info.status == "converged"
    # the solver stops on its own true residual; here it is recomputed with
    # other rounding: |Ax| is at most a few |b| (diagonally dominant rows)
    r = b - oracle_mod.spmv(cd.rp, cd.ci, cd.va, x)
    assert np.linalg.norm(r) <= (EPS + 1e-14) * np.linalg.norm(b)
    if cd.n <= 1400:
        ref = oracle_mod.gmres(cd.rp, cd.ci, cd.va, b, eps=EPS, restart=min(restart, 64))
        assert abs(info.iterations - ref[2]) <= 1
