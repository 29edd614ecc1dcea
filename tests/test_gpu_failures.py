"""Failure paths that a running kernel can reach, exercised without faulting
the GPU:

* a team barrier of the persistent kernel whose wait runs out: with a test
  limit of 50 ms and a first team planned for one CTA more than it is given
  (test hooks NLGB_BARRIER_TIMEOUT_MS / NLGB_TEST_TEAM_SHORTFALL, read when
  a batch runner starts), the barrier gives up, the kernel flags the error
  and returns, the call reports a device error, and the GPU stays usable;
* the solve server's abort, raised while a graph solve (serial mode) or a
  persistent epoch (batched mode) is running: the host-mapped abort flag
  (polled by the graph's guard kernel once per while-loop pass) or the next
  epoch boundary stops the work, the request ends as aborted with the
  iterations it ran."""
import json
import os
import subprocess
import sys
import time
from pathlib import Path

import numpy as np
import pytest

from graphitethree_gb300 import solver, systems

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parents[1]

BARRIER_SCRIPT = r"""
import json, sys, time
sys.path.insert(0, sys.argv[1])
from graphitethree_gb300 import solver, systems
M, rhs, _ = solver.assemble(systems.lscm_system(40, 40, seed=4))
out = {}
t0 = time.perf_counter()
try:
    solver.batch_solve([M], [rhs[0]])
    out["batch"] = "ok"
except solver.SolverError as e:
    out["batch"] = str(e)
out["batch_s"] = time.perf_counter() - t0
x, info = M.solve(rhs[0])          # graph executor: the context is still usable
out["after"] = info.status
out["after_true"] = info.true_rel_residual
print(json.dumps(out))
"""


def test_team_barrier_timeout_is_reported_and_the_gpu_stays_usable(gpu_ok):
    env = dict(os.environ, NLGB_BARRIER_TIMEOUT_MS="50", NLGB_TEST_TEAM_SHORTFALL="1")
    p = subprocess.run([sys.executable, "-c", BARRIER_SCRIPT, str(ROOT)], env=env, capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    out = json.loads(p.stdout.strip().splitlines()[-1])
    assert "barrier timed out" in out["batch"], out
    assert out["batch_s"] < 10.0
    assert out["after"] == "converged" and out["after_true"] <= 1e-10


def _lscm_square(side, seed):
    M, rhs, _ = solver.assemble(systems.lscm_system(side, side, seed=seed))
    rp, ci, va = M.download()
    return systems.SquareSystem(M.n, rp, ci, va, rhs[:1].copy())


def test_abort_stops_a_running_serial_graph_solve(gpu_ok):
    big = _lscm_square(600, 7)                      # ~720k unknowns: ~60k iterations, seconds
    srv = solver.Server(precision="double", mode="serial")
    t = srv.submit_square(big)
    time.sleep(0.5)                                  # the graph solve is running
    t_abort = time.perf_counter()
    srv.abort()
    ok, x, infos, lat = srv.wait_result(t)
    waited = time.perf_counter() - t_abort
    srv.close()
    assert not ok and infos[0].status == "aborted"
    assert 0 < infos[0].iterations < 5 * big.n
    assert waited < 2.0


def test_abort_stops_batched_epochs(gpu_ok):
    big = _lscm_square(600, 8)
    small = systems.fairing_system(60, 50, seed=9)
    srv = solver.Server(precision="double", mode="batched")
    t_big = srv.submit_square(big)
    t_small = srv.submit_square(small)
    _, info_small, _ = srv.wait(t_small)             # the small request completes normally
    assert all(i.status == "converged" for i in info_small)
    time.sleep(0.5)
    t_abort = time.perf_counter()
    srv.abort()
    ok, x, infos, lat = srv.wait_result(t_big)
    waited = time.perf_counter() - t_abort
    st = srv.stats()
    srv.close()
    assert not ok and infos[0].status == "aborted"
    assert 0 < infos[0].iterations < 5 * big.n      # the iterations run before the abort
    assert waited < 2.0
    assert st["completed"] == 1 and st["failed"] == 1


PERSIST_SCRIPT = r"""
import json, os, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from graphitethree_gb300 import meshes, solver
V, F = meshes.height_field(72, 57, 4)            # 65 tiles: a grid, whose CTAs wait for alpha and beta
M, b, _ = solver.build_lscm(V, F)
out = {}
for p in ("double", "mixed", "df"):
    out[p] = M.solve(b, precision=p)[1].status
    try:
        solver.batch_solve([M], [b], precision=p)
        out["batch " + p] = "ok"
    except solver.SolverError as e:
        out["batch " + p] = str(e)
    srv = solver.Server(precision=p)
    out["server " + p] = srv.wait_result(srv.submit_mesh("lscm", V, F))[2][0].status
    srv.close()
os.environ.pop("NLGB_TEST_PERSIST_SHORTFALL")
x, i = M.solve(b)                                # the same handle, the same context
out["after"] = [i.status, bool(np.array_equal(solver.batch_solve([M], [b])[0][0], x))]
srv = solver.Server(precision="double")
xs, infos, _ = srv.wait(srv.submit_mesh("lscm", V, F))
out["after server"] = [infos[0].status, bool(np.array_equal(xs[0], x))]
srv.close()
print(json.dumps(out))
"""


def test_wait_of_the_persistent_kernel_runs_out(gpu_ok):
    """Every wait for alpha is given up after 50 ms.  The CTA that writes the
    state on the device is the one that is missing, so that the error word alone
    tells of it: each route reports a device error, and goes on afterwards."""
    env = dict(os.environ, NLGB_BARRIER_TIMEOUT_MS="50", NLGB_TEST_PERSIST_SHORTFALL="1")
    p = subprocess.run([sys.executable, "-c", PERSIST_SCRIPT, str(ROOT)], env=env, capture_output=True,
                       text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    out = json.loads(p.stdout.strip().splitlines()[-1])
    for name in ("double", "mixed", "df"):
        assert out[name] == out["server " + name] == "device_err", out
        assert "timed out" in out["batch " + name], out
    assert out["after"] == out["after server"] == ["converged", True]


@pytest.mark.parametrize("side,n_rhs", [(33, 12000), (110, 4000)])      # a cluster, a grid
def test_abort_between_reliable_updates_of_a_few_iterations(gpu_ok, side, n_rhs):
    """Right-hand sides that take three iterations per reliable update and converge in ten."""
    sq = systems.fairing_system(side, side, lam=30.0, seed=3, n_rhs=1)
    sq.rhs = np.ascontiguousarray(np.repeat(sq.rhs, n_rhs, axis=0))
    srv = solver.Server(precision="mixed", mode="serial")
    t = srv.submit_square(sq)
    time.sleep(0.6)
    t_abort = time.perf_counter()
    srv.abort()
    ok, x, infos, lat = srv.wait_result(t)
    waited = time.perf_counter() - t_abort
    srv.close()
    assert not ok and "aborted" in [i.status for i in infos]
    assert "converged" in [i.status for i in infos] and waited < 0.5


REFUSE_SCRIPT = r"""
import json, os, sys
sys.path.insert(0, sys.argv[1])
import numpy as np
from graphitethree_gb300 import meshes, solver
meshes_ = [meshes.height_field(72, 57, 4), meshes.height_field(30, 20, 5)]      # a grid, a cluster
def run():
    out = []
    for p in ("double", "mixed", "df"):
        systems = [solver.build_lscm(V, F)[:2] for V, F in meshes_]
        out += [M.solve(b, precision=p) for M, b in systems]
        xs, infos, _ = solver.batch_solve([M for M, _ in systems], [b for _, b in systems], precision=p)
        out += list(zip(xs, infos))
        srv = solver.Server(precision=p, epoch_ms=1.0)
        for t in [srv.submit_mesh("lscm", V, F) for V, F in meshes_]:
            xs, infos, _ = srv.wait(t)
            out.append((xs[0], infos[0]))
        srv.close()
    return out
refused = run()
del os.environ["NLGB_TEST_PERSIST_REFUSE"]
want = run()
print(json.dumps([[i.status, i.iterations == j.iterations, bool(np.array_equal(x, y))]
                  for (x, i), (y, j) in zip(refused, want)]))
"""


@pytest.mark.parametrize("first", [1, 2, 7, 30])
def test_a_refused_launch_of_the_persistent_kernel_falls_back_to_the_graphs(gpu_ok, first):
    """From the first launch on, or in the middle of a solve, a batch or a chunk."""
    p = subprocess.run([sys.executable, "-c", REFUSE_SCRIPT, str(ROOT)],
                       env=dict(os.environ, NLGB_TEST_PERSIST_REFUSE=str(first)), capture_output=True, text=True,
                       timeout=300)
    assert p.returncode == 0, p.stderr
    out = json.loads(p.stdout.strip().splitlines()[-1])
    assert len(out) == 18 and all(o[1:] == [True, True] for o in out), out
