"""Batches on the persistent single-system kernel (csrc/nlgb_batch.cu): its
layouts (one to four tiles per CTA; one CTA, one cluster, cluster to grid at 64 / 65
tiles, more than four tiles per CTA), more systems than run at a time, matrices
used twice, mixed systems that continue in FP64, a layout changed between two
batches, two threads with the same matrices, and both sides of the rule that
chooses it -- the iterates of the single-system solver bit for bit."""
import threading
import time

import numpy as np
import pytest

from graphitethree_gb300 import _lib, meshes, solver

pytestmark = pytest.mark.gpu


def _system(kind, nx, ny, seed=3):
    V, F = meshes.height_field(nx, ny, seed)
    if kind == "lscm":
        M, rhs, _ = solver.build_lscm(V, F)
        return M, rhs
    return solver.build_fairing(V, F, 1e-2)[0], 1e-2 * V[:, 0]


def _check(systems, **kw):
    want = [M.solve(b, **kw) for M, b in systems]
    xs, infos, secs = solver.batch_solve([M for M, _ in systems], [b for _, b in systems], **kw)
    assert secs > 0
    for x, i, (y, j) in zip(xs, infos, want):
        assert np.array_equal(x, y)
        assert (i.status, i.iterations, i.refinement_steps) == (j.status, j.iterations, j.refinement_steps)


@pytest.mark.parametrize("precision", ["double", "mixed", "df"])
@pytest.mark.parametrize("sizes", [
    [("fairing", 3, 3)], [("lscm", 4, 3), ("fairing", 32, 16)], [("fairing", 37, 17), ("fairing", 128, 64)],
    [("fairing", 131, 64), ("lscm", 41, 29)], [("fairing", 363, 291)], [("fairing", 640, 600), ("fairing", 20, 20)]])
def test_layouts(gpu_ok, sizes, precision):
    _check([_system(*s) for s in sizes], precision=precision, max_iter=300)


@pytest.mark.parametrize("n,side", [(40, 12), (400, 8)])   # here; in the batched kernel
def test_more_systems_than_run_at_a_time(gpu_ok, n, side):
    _check([_system("fairing", side + k % 7, side, k) for k in range(n)], precision="mixed")


def test_a_matrix_twice_and_a_new_layout(gpu_ok):
    M, b = _system("lscm", 60, 50)
    F, c = _system("fairing", 150, 131)
    _check([(M, b), (F, c), (M, 2.0 * b), (F, -c)])
    M.set_layout(4, 256)
    _check([(M, b), (F, c), (M, 2.0 * b)])


def test_mixed_continues_in_fp64(gpu_ok):
    _check([_system("lscm", 70, 60), _system("lscm", 30, 20)], precision="mixed", eps=1e-12)


@pytest.mark.parametrize("max_iter", [0, 1, 1023, 1024, 1025])
def test_iteration_limits(gpu_ok, max_iter):
    _check([_system("lscm", 90, 80), _system("fairing", 40, 30)], max_iter=max_iter, eps=1e-13)


def test_two_threads_share_matrices(gpu_ok):
    systems = [_system("lscm", 50, 40), _system("fairing", 120, 100), _system("lscm", 33, 31)]
    mats, bs = [M for M, _ in systems], [b for _, b in systems]
    got = [None, None]

    def run(k):
        got[k] = [solver.batch_solve(mats[::1 - 2 * k], bs[::1 - 2 * k])[0][::1 - 2 * k] for _ in range(5)]
    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    want = [M.solve(b)[0] for M, b in systems]
    for k in range(2):
        for xs in got[k]:
            for x, y in zip(xs, want):
                assert np.array_equal(x, y)


def test_threads_with_other_layouts_of_a_matrix(gpu_ok):
    """A matrix alone (a tile per CTA) and among many (four): each batch keeps
    the tables that it runs on while the other thread's replaces the matrix's."""
    M, b = _system("lscm", 60, 50)
    many = [(M, b)] + [_system("fairing", 90, 80 + k, k) for k in range(12)]
    want = [m.solve(c)[0] for m, c in many]
    bad = []

    def run(systems, expect):
        for _ in range(6):
            xs = solver.batch_solve([m for m, _ in systems], [c for _, c in systems])[0]
            bad.extend(k for k, (x, y) in enumerate(zip(xs, expect)) if not np.array_equal(x, y))
    threads = [threading.Thread(target=run, args=a) for a in ((many[:1], want[:1]), (many, want))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("count", [1, 2, 3, 5, 9])
def test_tiles_per_cta_follow_the_batch(gpu_ok, count):
    _check([_system("lscm", 60, 50 + k, k) for k in range(count)] + [_system("fairing", 150, 131)])


@pytest.mark.parametrize("route", ["batch", "server"])
def test_the_host_sleeps_while_a_long_chunk_runs(gpu_ok, route):
    V, F = meshes.height_field(250, 240, 3)
    M, b, _ = solver.build_lscm(V, F)
    M.solve(b, max_iter=2)
    srv = solver.Server(precision="double", epoch_ms=20.0)
    wall, cpu = time.perf_counter(), time.process_time()
    if route == "batch":
        solver.batch_solve([M], [b])
    else:
        srv.wait(srv.submit_mesh("lscm", V, F))
    wall, cpu = time.perf_counter() - wall, time.process_time() - cpu
    srv.close()
    assert cpu < 0.5 * wall


# quick systems run in one launch of the batched kernel (a few launches in all), longer ones here
@pytest.mark.parametrize("count,side,precision,here", [
    (5, 4, "double", False), (5, 20, "double", True), (20, 10, "mixed", False), (20, 30, "mixed", True),
    (60, 12, "df", False), (60, 30, "df", True)])
def test_batches_of_quick_systems(gpu_ok, count, side, precision, here):
    systems = [_system("fairing", side, side, k) for k in range(count)]
    _check(systems, precision=precision)
    before = _lib.load().nlgb_kernel_launches()
    solver.batch_solve([M for M, _ in systems], [b for _, b in systems], precision=precision)
    launches = _lib.load().nlgb_kernel_launches() - before
    assert (launches >= 3 * count) == here


@pytest.mark.parametrize("precision", ["mixed", "df"])
def test_a_batch_and_a_solve_convert_one_matrix(gpu_ok, precision):
    """Whichever comes first converts the values, on a stream of its own; the
    other waits for them."""
    V, F = meshes.height_field(331, 307, 6)
    first, b, _ = solver.build_lscm(V, F)
    want = first.solve(b, precision=precision, max_iter=8)[0]
    for _ in range(10):
        M, _, _ = solver.build_lscm(V, F)
        start, got = threading.Barrier(2), {}

        def batch():
            start.wait()
            got["batch"] = solver.batch_solve([M], [b], precision=precision, max_iter=8)[0][0]

        def solve():
            start.wait()
            got["solve"] = M.solve(b, precision=precision, max_iter=8)[0]
        threads = [threading.Thread(target=f) for f in (batch, solve)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        assert np.array_equal(got["batch"], want) and np.array_equal(got["solve"], want)
        M.close()
