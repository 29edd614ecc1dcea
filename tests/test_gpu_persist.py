"""The persistent single-system kernel (csrc/nlgb_persist.cuh) against the
phase kernels launched one by one (NLGB_EAGER_SOLVE): the same iterates bit
for bit, at the sizes where its layout changes -- one tile, one cluster,
cluster to grid (64 / 65 tiles), one to nine tiles per CTA, every number of
threads per row, tiles of one to several passes -- and for columns in no
order (large halos, and halos that do not fit and take the graph)."""
import os

import numpy as np
import pytest

from graphitethree_gb300 import _lib, meshes, solver, systems

pytestmark = pytest.mark.gpu


def _both(M, b, precision, **kw):
    os.environ["NLGB_EAGER_SOLVE"] = "1"
    try:
        want = M.solve(b, precision=precision, **kw)
    finally:
        del os.environ["NLGB_EAGER_SOLVE"]
    got = M.solve(b, precision=precision, **kw)
    for (x, i), (y, j) in [(got, want)]:
        assert np.array_equal(x, y)
        assert (i.status, i.iterations, i.refinement_steps) == (j.status, j.iterations, j.refinement_steps)
        assert (i.rel_residual, i.true_rel_residual) == (j.rel_residual, j.true_rel_residual)


def _system(kind, nx, ny):
    V, F = meshes.height_field(nx, ny, 3)
    if kind == "lscm":
        M, rhs, _ = solver.build_lscm(V, F)
        return M, rhs
    return solver.build_fairing(V, F, 1e-2)[0], 1e-2 * V[:, 0]


@pytest.mark.parametrize("precision", ["double", "mixed", "df"])
@pytest.mark.parametrize("kind,nx,ny,layout", [
    ("fairing", 3, 3, None), ("lscm", 4, 3, None), ("fairing", 16, 8, None), ("fairing", 43, 3, None),
    ("fairing", 33, 31, None), ("lscm", 41, 29, None),
    ("fairing", 128, 64, None), ("fairing", 8193, 1, None), ("fairing", 2731, 3, None),
    ("lscm", 73, 59, (1, 192)), ("lscm", 73, 59, (4, 64)), ("lscm", 73, 59, (8, 512)),
    ("lscm", 73, 59, (16, 320)), ("lscm", 73, 59, (32, 128)), ("fairing", 150, 131, (2, 64)),
    ("fairing", 363, 291, None), ("fairing", 394, 394, None), ("fairing", 640, 611, None)])
def test_matches_phase_kernels(gpu_ok, kind, nx, ny, layout, precision):
    M, b = _system(kind, nx, ny)
    if layout:
        M.set_layout(*layout)
    _both(M, b, precision, max_iter=300)


@pytest.mark.parametrize("n", [900, 20000, 120000])
def test_columns_in_no_order(gpu_ok, n):
    """A symmetric diagonally dominant matrix with random columns: every
    column is in some CTA's halo (at 120,000 rows they do not fit)."""
    rng = np.random.default_rng(n)
    i = np.repeat(np.arange(n), 6)
    j = rng.integers(0, n, i.shape[0])
    w = rng.uniform(0.1, 1.0, i.shape[0])
    d = np.full(n, 1e-3)
    np.add.at(d, i, w)
    np.add.at(d, j, w)
    k = np.arange(n)
    rp, ci, va = systems.csr_from_coo(n, np.concatenate([i, j, k]), np.concatenate([j, i, k]),
                                      np.concatenate([-w, -w, d]))
    M = solver.Matrix(rp, ci, va)
    b = rng.standard_normal(n)
    for precision in ("double", "mixed"):
        _both(M, b, precision, max_iter=150)


def test_long_solve_crosses_launches(gpu_ok):
    """More iterations than one launch runs, and a true-residual continuation."""
    M, b = _system("lscm", 90, 80)
    _both(M, b, "double", eps=1e-12)
    M, b = _system("lscm", 60, 50)
    _both(M, b, "double", eps=1e-13)


@pytest.mark.parametrize("b", ["zero", "nan"])
def test_no_iteration(gpu_ok, b):
    M, rhs = _system("fairing", 40, 30)
    v = np.zeros_like(rhs) if b == "zero" else np.full_like(rhs, np.nan)
    x, i = M.solve(v)
    assert i.iterations == 0 and i.status == ("converged" if b == "zero" else "breakdown")


def _band(n, per_row, seed):
    """Diagonally dominant, random columns within a band, about per_row nonzeros a row."""
    rng = np.random.default_rng(seed)
    m = n * (per_row - 1) // 2
    i = rng.integers(0, n, m)
    j = i + rng.integers(1, max(2, min(2500, n // 3)), m)
    i, j = i[j < n], j[j < n]
    w = rng.uniform(0.1, 1.0, i.shape[0])
    d = np.full(n, 1e-3)
    np.add.at(d, i, w)
    np.add.at(d, j, w)
    k = np.arange(n)
    rp, ci, va = systems.csr_from_coo(n, np.concatenate([i, j, k]), np.concatenate([j, i, k]),
                                      np.concatenate([-w, -w, d]))
    return solver.Matrix(rp, ci, va), rng.standard_normal(n)


@pytest.mark.parametrize("n,per_row", [(300, 60), (2048, 30), (2049, 30), (2177, 110), (8192, 200), (8193, 24),
                                       (20000, 300)])
def test_long_rows(gpu_ok, n, per_row):
    """A cluster up to 16 tiles, a grid from 17 on; many nonzeros outside the registers."""
    M, b = _band(n, per_row, n)
    assert M.threads_per_row > 2
    for precision in ("double", "mixed", "df"):
        _both(M, b, precision, max_iter=60)
    xs, infos, _ = solver.batch_solve([M, M], [b, 2.0 * b], max_iter=60)
    for x, i, s in zip(xs, infos, (1.0, 2.0)):
        y, j = M.solve(s * b, max_iter=60)
        assert np.array_equal(x, y) and i.iterations == j.iterations


@pytest.mark.parametrize("precision", ["double", "df"])
@pytest.mark.parametrize("case", ["tiles_above_512_rows", "larger_than_l2"])
def test_one_kernel_per_iteration_where_the_persistent_one_does_not_fit(gpu_ok, case, precision):
    if case == "larger_than_l2":
        M, b = _band(60_000, 230, 1)
    else:
        M, b = _system("lscm", 70, 61)
        M.set_layout(2, 576)
    _both(M, b, precision, max_iter=40)
    before = _lib.load().nlgb_kernel_launches()
    info = M.solve(b, precision=precision, max_iter=40)[1]
    assert info.iterations == 40
    assert _lib.load().nlgb_kernel_launches() - before < 2 * info.iterations      # three phases: 3 and more
    _both(M, b, precision, eps=1e-13, max_iter=1500)                              # continuations too


@pytest.mark.parametrize("side", [12, 110])      # a cluster, a grid
def test_a_mixed_solve_that_ends_at_once_queues_few_kernels(gpu_ok, side):
    """Ten reliable updates are expected at 1e-10, three kernels each; a solve
    that is over before does not queue them all (the fewest of some calls: the
    host sees the end when it comes)."""
    M, b = _system("fairing", side, side)
    x, info = M.solve(b, precision="mixed", eps=1e-12)
    assert info.status == "converged"
    launches = []
    for _ in range(8):
        before = _lib.load().nlgb_kernel_launches()
        y, again = M.solve(b, x0=x, precision="mixed")
        launches.append(_lib.load().nlgb_kernel_launches() - before)
        assert again.status == "converged" and again.iterations == 0 and np.array_equal(x, y)
    assert min(launches) < 20


@pytest.mark.parametrize("kind,nx,ny", [("fairing", 47, 46), ("fairing", 90, 91), ("lscm", 46, 44), ("lscm", 46, 46)])
def test_cluster_and_grid_by_threads_per_row(gpu_ok, kind, nx, ny):
    """17 and 64 tiles of one thread per row: a cluster; 32 and 34 of two: both sides."""
    M, b = _system(kind, nx, ny)
    for precision in ("double", "mixed", "df"):
        _both(M, b, precision, max_iter=60)
