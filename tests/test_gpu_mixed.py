"""Mixed precision beyond the persistent kernel's range: the graph, whose solution
update is due at most once in a pass of four iterations, against the phase
kernels launched one by one, bit for bit; row lengths on both sides of the three
nonzeros that a thread of the FP32 product has in flight; and products that are
subnormal or not finite, which leave the integer path of the conversion."""
import os

import numpy as np
import pytest

from graphitethree_gb300 import meshes, solver, systems

pytestmark = pytest.mark.gpu


def _eager(M, b, **kw):
    os.environ["NLGB_EAGER_SOLVE"] = "1"
    try:
        return M.solve(b, precision="mixed", **kw)
    finally:
        del os.environ["NLGB_EAGER_SOLVE"]


def _same(got, want):
    (x, i), (y, j) = got, want
    assert np.array_equal(x, y, equal_nan=True)
    assert (i.status, i.iterations, i.refinement_steps) == (j.status, j.iterations, j.refinement_steps)


@pytest.mark.parametrize("max_iter", [1, 4, 7, 40, 5000])
@pytest.mark.parametrize("nx,ny", [(700, 600), (1024, 700)])
def test_updates_inside_and_at_the_end_of_a_pass(gpu_ok, nx, ny, max_iter):
    V, F = meshes.height_field(nx, ny, 3)
    M = solver.build_fairing(V, F, 1e-2)[0]
    got = M.solve(1e-2 * V[:, 0], precision="mixed", max_iter=max_iter)
    _same(got, _eager(M, 1e-2 * V[:, 0], max_iter=max_iter))
    if max_iter == 5000:
        assert got[1].status == "converged" and got[1].true_rel_residual < 1e-8


def _band(n, half, scale):
    i = np.repeat(np.arange(n), half)
    j = np.minimum(i + np.tile(np.arange(1, half + 1), n), n - 1)
    i, j = i[i != j], j[i != j]
    w = np.full(i.shape[0], 0.25)
    d = np.full(n, 0.5)
    np.add.at(d, i, w)
    np.add.at(d, j, w)
    k = np.arange(n)
    rp, ci, va = systems.csr_from_coo(n, np.concatenate([i, j, k]), np.concatenate([j, i, k]),
                                      np.concatenate([-w, -w, d]) * scale)
    return solver.Matrix(rp, ci, va)


@pytest.mark.parametrize("threads", [1, 2, 4])
@pytest.mark.parametrize("half", [0, 1, 2, 3, 4, 6])
def test_row_lengths(gpu_ok, half, threads):
    n = 1500
    M = _band(n, half, 1.0) if half else solver.Matrix(np.arange(n + 1), np.arange(n), np.full(n, 0.5))
    M.set_layout(threads, 256)
    x = np.sin(np.arange(n))
    b = M.spmv(x) if half else 0.5 * x
    got, info = M.solve(b, precision="mixed", eps=1e-12)
    # |e| <= cond * relres * |b| / |A|min: the spectrum of a band system lies in [0.5, 0.5 + 4 * 0.25 * half]
    assert info.status == "converged"
    assert np.linalg.norm(got - x) <= 1e-11 * np.linalg.norm(b) / 0.5
    _same((got, info), _eager(M, b, eps=1e-12))


@pytest.mark.parametrize("scale", [1e-19, 1e-21, 1e-24, 1e18, 1e30])
def test_products_out_of_the_normal_range(gpu_ok, scale):
    M = _band(1500, 2, 1.0)
    b = np.sin(np.arange(1500)) * scale
    _same(M.solve(b, precision="mixed", max_iter=40), _eager(M, b, max_iter=40))


def test_chunk_with_many_updates(gpu_ok):
    """A chunk in which many passes end early: an update every few iterations."""
    sq = systems.fairing_system(1300, 1000, seed=3, n_rhs=1)
    x, info = solver.Matrix(sq.rp, sq.ci, sq.va).solve(sq.rhs[0], precision="mixed", inner_eps=0.5)
    srv = solver.Server(precision="mixed", inner_eps=0.5, epoch_ms=20.0)   # the second chunk: about 300 iterations
    xs, infos, _ = srv.wait(srv.submit_square(sq))
    srv.close()
    assert infos[0].status == info.status == "converged"
    assert infos[0].refinement_steps > 20
    _same((xs[0], infos[0]), (x, info))


def _wide_band(n, offset):
    """Rows of 5 and more nonzeros with the farthest at `offset`, 2^21 nonzeros and more."""
    k = np.arange(n)
    i, j, w = [k], [k], [np.full(n, 6.5)]
    for d, v in ((1, -1.0), (700, -1.0), (offset, -1.0)):
        a = np.arange(n - d)
        i += [a, a + d]
        j += [a + d, a]
        w += [np.full(n - d, v)] * 2
    return solver.Matrix(*systems.csr_from_coo(n, np.concatenate(i), np.concatenate(j), np.concatenate(w)))


@pytest.mark.parametrize("threads", [1, 2, 8])
@pytest.mark.parametrize("offset", [32767, 32768])   # 16-bit columns; one too far for them
def test_columns_relative_to_the_row(gpu_ok, offset, threads):
    n = 700000
    b = np.sin(np.arange(n))
    M = _wide_band(n, offset)
    M.set_layout(threads, 0)
    want = _eager(M, b)                    # before any graph: 32-bit columns
    got = M.solve(b, precision="mixed")
    assert got[1].status == "converged" and got[1].true_rel_residual <= 1e-10
    _same(got, want)
    _same(_eager(M, b), want)
