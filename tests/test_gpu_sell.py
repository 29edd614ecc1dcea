"""Sliced layout of large matrices with two threads per row (csrc/nlgb_sell.cu):
the products and the phase-kernel iterates are those of the CRS kernels bit for
bit -- short last tiles and passes, tiles that are not a multiple of a pass,
rows without entries -- and matrices it does not suit keep the CRS kernels."""
import ctypes
import os
import threading

import numpy as np
import pytest
import torch

from graphitethree_gb300 import _lib, meshes, solver, systems
from graphitethree_gb300.nlvector import Vector

pytestmark = pytest.mark.gpu


def _check(M, rng):
    x = rng.standard_normal(M.n)
    x[:3] = [np.inf, -np.inf, np.nan]          # reach only their own rows
    y = [M.spmv(x) for _ in range(7)]          # the layout is built by the fifth
    assert all(np.array_equal(y[0], v, equal_nan=True) for v in y)


@pytest.mark.parametrize("tile", [1024, 1088, 576, 4096])
def test_lscm_products_and_iterates(gpu_ok, tile):
    V, F = meshes.height_field(331, 307, 5)
    M, b, _ = solver.build_lscm(V, F)
    M.set_layout(2, tile)                       # (above 512 rows: phase kernels)
    _check(M, np.random.default_rng(1))
    os.environ["NLGB_EAGER_SOLVE"] = "1"
    try:
        want = M.solve(b, max_iter=60)
    finally:
        del os.environ["NLGB_EAGER_SOLVE"]
    x, i = M.solve(b, max_iter=60)
    assert np.array_equal(x, want[0]) and i.iterations == want[1].iterations
    assert i.true_rel_residual == want[1].true_rel_residual
    M.set_layout(2, 832)                        # another layout: rebuilt
    _check(M, np.random.default_rng(2))


@pytest.mark.parametrize("kind", ["empty_rows", "one_dense_row", "uneven"])
def test_rows_of_any_length(gpu_ok, kind):
    n = 170_000
    rng = np.random.default_rng(7)
    lens = rng.integers(10, 19, n)
    if kind == "empty_rows":
        lens[rng.random(n) < 0.05] = 0
    elif kind == "one_dense_row":
        lens[n // 2] = 700                      # more than 255 per lane
    else:
        lens[::64] = 300
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(lens)
    i = np.repeat(np.arange(n), lens)
    ci = (i + rng.integers(-300, 300, rp[-1])) % n
    va = rng.standard_normal(rp[-1])
    M = solver.Matrix(rp, ci, va)
    M.set_layout(2, 1024)
    x = rng.standard_normal(n)
    y = [M.spmv(x) for _ in range(7)]
    assert all(np.array_equal(y[0], v) for v in y)


def test_products_and_solves_of_one_matrix_in_two_threads(gpu_ok):
    """Whichever thread asks first builds the layout, and both find it whole."""
    V, F = meshes.height_field(331, 307, 6)
    first, b, _ = solver.build_lscm(V, F)
    first.set_layout(2, 1024)
    x = np.random.default_rng(3).standard_normal(first.n)
    y = first.spmv(x)
    want = first.solve(b, max_iter=40)[0]
    for _ in range(6):
        M, _, _ = solver.build_lscm(V, F)
        M.set_layout(2, 1024)
        start, bad = threading.Barrier(2), []

        def products():
            start.wait()
            for _ in range(12):
                if not np.array_equal(M.spmv(x), y):
                    bad.append("product")

        def solves():
            start.wait()
            for _ in range(3):
                if not np.array_equal(M.solve(b, max_iter=40)[0], want):
                    bad.append("solve")
        threads = [threading.Thread(target=f) for f in (products, solves)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert not bad
        M.close()


@pytest.mark.parametrize("side,built", [(600, True), (1500, False)])     # 10 and 63 million nonzeros
def test_solves_of_the_largest_matrices_keep_the_crs_kernels(gpu_ok, side, built):
    """The layout costs two kernels; with other threads per row it is not built."""
    V, F = meshes.height_field(side, side, 1)
    M, b, _ = solver.build_lscm(V, F)
    launches = []
    for tpr in (4, 2):
        M.set_layout(tpr, M.tile_rows)
        before = _lib.load().nlgb_kernel_launches()
        M.solve(b, max_iter=4)
        launches.append(_lib.load().nlgb_kernel_launches() - before)
    assert launches[1] - launches[0] == (2 if built else 0)


def test_timed_products_are_the_products_asked_for(gpu_ok):
    """As many kernels as products, and what a layout costs is not in the time."""
    L = _lib.load()
    V, F = meshes.height_field(808, 808, 1)
    M, _, _ = solver.build_lscm(V, F)
    x, y, ms = Vector(np.ones(M.n)), Vector(M.n), ctypes.c_double()
    times = []
    for reps in (3, 3, 3):
        assert L.nlgb_spmv_timed(M.handle, x.tensor.data_ptr(), y.tensor.data_ptr(), reps, ctypes.byref(ms)) == 0
        times.append(ms.value)
    assert max(times[1:]) < 1.5 * times[0]
    before = L.nlgb_kernel_launches()
    assert L.nlgb_spmv_timed(M.handle, x.tensor.data_ptr(), y.tensor.data_ptr(), 10, ctypes.byref(ms)) == 0
    assert L.nlgb_kernel_launches() - before == 10


def _launches_of_products(M, x, y, count):
    L = _lib.load()
    before = L.nlgb_kernel_launches()
    for _ in range(count):
        assert L.nlgb_spmv(M.handle, x.tensor.data_ptr(), y.tensor.data_ptr()) == 0
    return L.nlgb_kernel_launches() - before


# 2.8 M nonzeros: too few to gain; 9.4 M: laid out (two kernels) once that has paid; 63 M: too many
@pytest.mark.parametrize("side,extra", [(320, 0), (580, 2), (1500, 0)])
def test_products_are_laid_out_where_that_pays(gpu_ok, side, extra):
    V, F = meshes.height_field(side, side, 1)
    M, _, _ = solver.build_lscm(V, F)
    x, y = Vector(np.random.default_rng(4).standard_normal(M.n)), Vector(M.n)
    assert _launches_of_products(M, x, y, 256) == 256
    first = y.tensor.clone()
    assert _launches_of_products(M, x, y, 2) == 2 + extra
    assert torch.equal(y.tensor, first)


@pytest.mark.parametrize("tile", [1024, 576])
def test_products_use_the_layout_of_a_solve(gpu_ok, tile):
    V, F = meshes.height_field(331, 307, 5)
    M, b, _ = solver.build_lscm(V, F)
    M.set_layout(2, tile)
    x = np.random.default_rng(1).standard_normal(M.n)
    x[:3] = [np.inf, -np.inf, np.nan]          # reach only their own rows
    y = M.spmv(x)
    M.solve(b, max_iter=3)
    for _ in range(2):
        assert np.array_equal(M.spmv(x), y, equal_nan=True)


@pytest.mark.parametrize("kind", ["short_and_empty", "one_row_of_500", "one_dense_row"])
def test_rows_of_any_length_in_the_layout_of_a_solve(gpu_ok, kind):
    """A solve lays the matrix out (two kernels) unless a lane would get more
    than 255 nonzeros; the products that follow keep their bits."""
    n = 170_000 + 77                            # a short last tile and pass
    rng = np.random.default_rng(11)
    lens = rng.integers(12, 19, n)
    if kind == "short_and_empty":
        lens[rng.random(n) < 0.02] = 0
        lens[rng.random(n) < 0.02] = 1
    else:
        lens[n // 2] = 500 if kind == "one_row_of_500" else 700
    rp = np.zeros(n + 1, np.int64)
    rp[1:] = np.cumsum(lens)
    i = np.repeat(np.arange(n), lens)
    ci = (i + rng.integers(-300, 300, rp[-1])) % n
    va = rng.standard_normal(rp[-1])
    x = rng.standard_normal(n)
    M = solver.Matrix(rp, ci, va)
    M.set_layout(2, 1024)
    y = M.spmv(x)
    launches = []
    for _ in range(2):
        before = _lib.load().nlgb_kernel_launches()
        M.solve(x, max_iter=1)
        launches.append(_lib.load().nlgb_kernel_launches() - before)
    assert np.array_equal(M.spmv(x), y)
    assert launches[0] - launches[1] == (1 if kind == "one_dense_row" else 2)
