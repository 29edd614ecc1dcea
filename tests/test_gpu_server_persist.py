"""Chunks of the server on the persistent kernel (csrc/nlgb_persist.cuh): where
their layout changes (four tiles per CTA; one CTA, one cluster, cluster to grid
at 64 / 65 tiles, more than four tiles per CTA), every precision, a mixed system
that continues in FP64, a budget without room for the tables, and a load that
changes between systems that fit and systems that do not -- the same iterates
bit for bit as the single-system solver."""
import threading
import time

import numpy as np
import pytest

from graphitethree_gb300 import meshes, solver, systems

pytestmark = pytest.mark.gpu


def _check(srv, reqs, precision):
    want = [solver.Matrix(s.rp, s.ci, s.va).solve(s.rhs[0], precision=precision) for s in reqs]
    tickets = [srv.submit_square(s) for s in reqs]
    for t, (y, j) in zip(tickets, want):
        xs, infos, _ = srv.wait(t)
        assert infos[0].status == j.status == "converged"
        assert np.array_equal(xs[0], y)
        assert (infos[0].iterations, infos[0].refinement_steps) == (j.iterations, j.refinement_steps)


@pytest.mark.parametrize("precision", ["double", "mixed", "df"])
@pytest.mark.parametrize("sizes", [[(3, 3)], [(32, 16)], [(37, 17)], [(128, 64)], [(131, 64)], [(363, 291)],
                                   [(640, 600)], [(20, 20), (150, 131), (90, 80), (33, 31), (200, 180), (5, 4)]])
def test_sizes(gpu_ok, sizes, precision):
    srv = solver.Server(precision=precision, epoch_ms=0.5)
    _check(srv, [systems.fairing_system(nx, ny, seed=nx, n_rhs=1) for nx, ny in sizes], precision)
    srv.close()


def test_mixed_continues_in_fp64(gpu_ok):
    V, F = meshes.height_field(70, 60, 3)
    M, rhs, _ = solver.build_lscm(V, F)
    x, info = M.solve(rhs, precision="mixed", eps=1e-12)
    srv = solver.Server(precision="mixed", eps=1e-12)
    xs, infos, _ = srv.wait(srv.submit_mesh("lscm", V, F))
    srv.close()
    assert infos[0].status == info.status
    assert np.array_equal(xs[0], x) and infos[0].iterations == info.iterations


def test_no_room_for_tables(gpu_ok):
    sq = systems.fairing_system(200, 180, seed=2, n_rhs=1)
    srv = solver.Server(precision="double")
    srv.wait(srv.submit_square(sq))
    peak = srv.stats()["peak_bytes"]
    srv.close()
    srv = solver.Server(precision="double", budget_bytes=peak - 1024)
    _check(srv, [sq], "double")
    assert srv.stats()["peak_bytes"] <= peak - 1024
    srv.close()


def test_load_changes(gpu_ok):
    small = [systems.fairing_system(60 + 10 * i, 50 + 7 * i, seed=i, n_rhs=1) for i in range(6)]
    large = systems.fairing_system(1300, 1000, seed=3, n_rhs=1)
    srv = solver.Server(precision="mixed", epoch_ms=1.0)
    _check(srv, small + [large] + small, "mixed")
    _check(srv, [large] + small, "mixed")
    srv.close()


def test_more_work_than_the_persistent_kernel_gains_on(gpu_ok):
    """Enough mid-size systems that their chunks run as graphs, then the last
    of them on the persistent kernel again."""
    srv = solver.Server(precision="double", epoch_ms=1.0)
    _check(srv, [systems.fairing_system(360 + 4 * i, 300, seed=i, n_rhs=1) for i in range(12)] +
           [systems.fairing_system(60, 50 + i, seed=i, n_rhs=1) for i in range(8)], "double")
    srv.close()


@pytest.mark.parametrize("side", [33, 110])      # a cluster, a grid
def test_a_mixed_chunk_keeps_to_its_budget(gpu_ok, side, tmp_path, monkeypatch):
    """A new system's first chunk is a probe of 16 iterations, also where reliable
    updates end the kernel's launches sooner."""
    sq = systems.fairing_system(side, side, seed=3, n_rhs=1)
    want, info = solver.Matrix(sq.rp, sq.ci, sq.va).solve(sq.rhs[0], precision="mixed", inner_eps=0.5)
    monkeypatch.setenv("NLGB_SERVER_TRACE", str(tmp_path / "trace"))
    srv = solver.Server(precision="mixed", inner_eps=0.5)
    xs, infos, _ = srv.wait(srv.submit_square(sq))
    srv.close()
    assert np.array_equal(xs[0], want) and infos[0].iterations == info.iterations
    chunks = [line.split(",") for line in (tmp_path / "trace").read_text().splitlines() if line.startswith("C,")]
    assert 0 < int(chunks[0][6]) - int(chunks[0][5]) <= 16


def test_a_wide_system_leaves_room_for_small_ones(gpu_ok):
    """Beside a system of 613 tiles, whose chunks last 50 ms, a small request is
    admitted and solved without waiting for their ends."""
    V, F = meshes.height_field(280, 280, 1)
    small = [systems.fairing_system(40, 40, seed=i, n_rhs=1) for i in range(4)]
    srv = solver.Server(precision="double", epoch_ms=50.0)
    srv.wait(srv.submit_square(small[3]))
    wide = srv.submit_mesh("lscm", V, F)
    time.sleep(0.03)
    lat = [srv.wait(srv.submit_square(s))[2] for s in small[:3]]
    _, infos, wide_lat = srv.wait(wide)
    srv.close()
    assert infos[0].status == "converged" and wide_lat > sum(lat)     # it ran all the while
    assert sorted(lat)[1] < 0.025


@pytest.mark.parametrize("streams", [6, 12])     # SMs left over, but too few; none left over
def test_a_wide_system_among_a_stream_of_small_ones(gpu_ok, streams):
    V, F = meshes.height_field(200, 200, 1)      # 625 tiles, 0.1 s alone
    small = [meshes.height_field(60, 60, i) for i in range(8)]
    M, b, _ = solver.build_lscm(V, F)
    want = M.solve(b)[0]
    srv = solver.Server(precision="double")
    stop = threading.Event()

    def feed(i):
        while not stop.is_set():
            srv.wait(srv.submit_mesh("lscm", *small[i % 8]))
            i += 1
    threads = [threading.Thread(target=feed, args=(i,)) for i in range(streams)]
    for t in threads:
        t.start()
    time.sleep(0.1)
    got = []
    waiter = threading.Thread(target=lambda t: got.append(srv.wait(t)), args=(srv.submit_mesh("lscm", V, F),))
    waiter.start()
    waiter.join(4.0)
    in_time = not waiter.is_alive()              # beside the stream, not after it
    stop.set()
    for t in threads + [waiter]:
        t.join()
    srv.close()
    assert in_time and np.array_equal(got[0][0][0], want)


def test_chunks_on_the_persistent_kernel_are_counted_apart(gpu_ok):
    small, large = systems.fairing_system(90, 80, seed=1, n_rhs=1), systems.fairing_system(1300, 1000, seed=3, n_rhs=1)
    for sq, here in ((small, True), (large, False)):
        srv = solver.Server(precision="double")
        srv.wait(srv.submit_square(sq))
        st = srv.stats()
        srv.close()
        part = (st["persist_chunks"], st["persist_algo_bytes"])
        assert part == ((st["epochs"], st["epoch_algo_bytes"]) if here else (0, 0.0))
        assert abs(st["persist_s"] - (st["kernel_s"] if here else 0.0)) < 1e-9
