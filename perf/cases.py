"""The work a user of the library has it do, as cases to time and compare.

Kinds of case (all through the package's public entry points):

* ``spmv``    y = A x on a resident matrix with device vectors;
* ``solve``   one Jacobi-PCG solve on a resident matrix (fairing or LSCM
              systems; FP64, mixed and double-float precision; host vectors for
              the small calls, device vectors for the large ones);
* ``build``   mesh -> CRS system on the GPU, read back to the host;
* ``opennl``  the OpenNL context sequence on a least-squares row stream
              (assembly, solve, read-back);
* ``atlas``   many uneven charts in one batched solve;
* ``krylov``  BiCGSTAB / GMRES(30) on a non-symmetric system;
* ``serve``   a burst of mesh requests to the solve server.

Meshes are the repository's seeded height fields (an nx x ny vertex grid, one
random diagonal per quad, eight Gaussian bumps).
"""
import math

import numpy as np
import torch

from graphitethree_gb300 import _lib, meshes, solver, systems
from graphitethree_gb300.nlvector import Vector

LAMBDA = 1e-2     # fairing: L + LAMBDA I
NOISE = 1e-3      # positional noise of the fairing right-hand sides


def listed():
    return [
        # The product with a large LSCM normal matrix, vectors kept on the
        # device: what a scripting user calls in a loop.
        {"name": "spmv_lscm_808", "kind": "spmv", "system": "lscm", "nx": 808, "ny": 808},
        # The smallest solve a mesh command makes (1k vertices): launches and
        # latency, host vectors as a C caller has them.
        {"name": "solve_fairing_33x31", "kind": "solve", "system": "fairing", "nx": 33, "ny": 31,
         "precision": "double"},
        # The plain LSCM parameterisation of a 256 x 256 patch in FP64.
        {"name": "solve_lscm_256", "kind": "solve", "system": "lscm", "nx": 256, "ny": 256,
         "precision": "double"},
        # Fairing of an ordinary patch with odd sides, mixed precision.
        {"name": "solve_fairing_363x291_mixed", "kind": "solve", "system": "fairing", "nx": 363, "ny": 291,
         "precision": "mixed"},
        # Fairing of a 2048 x 2048 patch, FP64 and mixed: one coordinate.
        {"name": "solve_fairing_2048", "kind": "solve", "system": "fairing", "nx": 2048, "ny": 2048,
         "precision": "double"},
        {"name": "solve_fairing_2048_mixed", "kind": "solve", "system": "fairing", "nx": 2048, "ny": 2048,
         "precision": "mixed"},
        # The LSCM system of a 640 x 481 mesh, built and read back as CRS.
        {"name": "build_lscm_640x481", "kind": "build", "system": "lscm", "nx": 640, "ny": 481},
        # The voxel interpolation of the optimal-transport plugin, as an
        # OpenNL caller runs it: rows in, least squares, variables out.
        {"name": "opennl_voxel_48x40x37", "kind": "opennl", "nx": 48, "ny": 40, "nz": 37},
        # Charts of an atlas (log-uniform sides, aspect 1 to 4), one launch.
        {"name": "atlas_40", "kind": "atlas", "charts": 40, "side_min": 16, "side_max": 128,
         "precision": "double"},
        # Non-symmetric systems (upwind convection-diffusion).
        {"name": "bicgstab_1024", "kind": "krylov", "method": "bicgstab", "nx": 1024, "ny": 1024},
        {"name": "gmres_601x523", "kind": "krylov", "method": "gmres", "nx": 601, "ny": 523},
        # Requests of the serving stream that arrive together (LSCM and
        # fairing, 1k to 20k vertices), AUTO precision.
        {"name": "serve_burst_24", "kind": "serve", "requests": 24, "vmin": 1000, "vmax": 20000},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: sizes log-uniform over the ranges of the listed ones."""
    kind = rng.choice(["spmv", "solve", "solve", "solve", "solve", "build", "opennl", "atlas", "krylov", "krylov",
                       "serve"])
    if kind == "spmv":
        system = rng.choice(["lscm", "fairing"])
        return {"kind": kind, "system": system, "nx": _log_int(rng, 40, 800), "ny": _log_int(rng, 40, 800)}
    if kind == "solve":
        system = rng.choice(["fairing", "fairing", "lscm"])
        if system == "lscm":
            nx = _log_int(rng, 20, 230)
            return {"kind": kind, "system": system, "nx": nx, "ny": max(16, int(nx * rng.uniform(0.5, 1.0))),
                    "precision": "double"}
        nx = _log_int(rng, 30, 2000)
        return {"kind": kind, "system": system, "nx": nx, "ny": max(24, int(nx * rng.uniform(0.5, 1.0))),
                "precision": rng.choice(["double", "mixed", "df"])}
    if kind == "build":
        return {"kind": kind, "system": rng.choice(["lscm", "fairing"]), "nx": _log_int(rng, 30, 600),
                "ny": _log_int(rng, 30, 480)}
    if kind == "opennl":
        return {"kind": kind, "nx": _log_int(rng, 7, 46), "ny": _log_int(rng, 7, 40), "nz": _log_int(rng, 5, 36)}
    if kind == "atlas":
        return {"kind": kind, "charts": _log_int(rng, 4, 38), "side_min": 16, "side_max": rng.randint(48, 120),
                "precision": "double"}
    if kind == "krylov":
        method = rng.choice(["bicgstab", "gmres"])
        top = 1000 if method == "bicgstab" else 580
        nx = _log_int(rng, 60, top)
        return {"kind": kind, "method": method, "nx": nx, "ny": max(40, int(nx * rng.uniform(0.5, 0.9)))}
    return {"kind": kind, "requests": rng.randint(6, 22), "vmin": 1000, "vmax": _log_int(rng, 4000, 18000)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _rng(seed, tag):
    return np.random.default_rng([int(seed), tag])


def _mesh(nx, ny, seed):
    return meshes.height_field(nx, ny, int(seed))


def _fairing_rhs(V, seed, k=1):
    P = V[:, :k].T
    return np.ascontiguousarray(LAMBDA * (P + _rng(seed, 7919).normal(0.0, NOISE, P.shape)))


def _charts(case, seed):
    # the mix of sizes is one atlas's; the surfaces differ with the seed
    nx, ny = meshes.chart_sizes(case["charts"], 17, case["side_min"], case["side_max"])
    return [(int(nx[i]), int(ny[i]), int(seed) * 1009 + i) for i in range(case["charts"])]


def _requests(case, seed):
    rng = np.random.default_rng(23)     # sizes and kinds: one burst; surfaces from the seed
    out = []
    for i in range(case["requests"]):
        nv = math.exp(rng.uniform(math.log(case["vmin"]), math.log(case["vmax"])))
        kind = "lscm" if int(rng.integers(0, 2)) == 0 else "fairing"
        side = max(4, int(round(math.sqrt(nv))))
        V, F = _mesh(side, side, int(seed) * 1013 + i)
        out.append((kind, V, F, _fairing_rhs(V, int(seed) * 1013 + i, 3) if kind == "fairing" else None))
    return out


def _large(case):
    return case["nx"] * case["ny"] > 20_000


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind in ("spmv", "solve"):
        V, F = _mesh(case["nx"], case["ny"], seed)
        if case["system"] == "lscm":
            M, rhs, _ = solver.build_lscm(V, F)
        else:
            M, _ = solver.build_fairing(V, F, LAMBDA)
            rhs = _fairing_rhs(V, seed)[0]
        s["M"] = M
        if kind == "spmv":
            s["x"] = Vector(_rng(seed, 3).standard_normal(M.n))
            s["y"] = Vector(M.n)
        elif _large(case):
            s["b"] = Vector(rhs)
        else:
            s["b"] = np.array(rhs)
    elif kind == "build":
        s["V"], s["F"] = _mesh(case["nx"], case["ny"], seed)
        n, nnz = _sizes(case)
        # read-back buffers for the largest CRS of these sides (the corners'
        # degrees depend on the diagonals); what is not filled stays zero
        s["rp"] = torch.zeros(n + 1, dtype=torch.int32).pin_memory().numpy()
        s["ci"] = torch.zeros(nnz, dtype=torch.int32).pin_memory().numpy()
        s["va"] = torch.zeros(nnz, dtype=torch.float64).pin_memory().numpy()
    elif kind == "opennl":
        s["rows"] = systems.voxel_rows(case["nx"], case["ny"], case["nz"], int(seed))
    elif kind == "atlas":
        s["mats"], s["b"] = [], []
        for nx, ny, sd in _charts(case, seed):
            M, rhs, _ = solver.build_lscm(*_mesh(nx, ny, sd))
            s["mats"].append(M)
            s["b"].append(rhs)
    elif kind == "krylov":
        sq = systems.convection_diffusion(case["nx"], case["ny"], int(seed))
        s["M"] = solver.Matrix(sq.rp, sq.ci, sq.va)
        s["b"] = sq.rhs[0]
    else:
        s["requests"] = _requests(case, seed)
        s["server"] = solver.Server(budget_bytes=20e9, precision="auto")
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "spmv":
        _lib.load().nlgb_spmv(s["M"].handle, s["x"].tensor.data_ptr(), s["y"].tensor.data_ptr())
        return s["y"].tensor
    if kind == "solve":
        if isinstance(s["b"], Vector):
            x = Vector(len(s["b"]))
            s["M"].solve_device(s["b"].tensor.data_ptr(), x.tensor.data_ptr(), precision=case["precision"])
            return x.tensor
        return s["M"].solve(s["b"], precision=case["precision"])[0]
    if kind == "build":
        rhs = None
        if case["system"] == "lscm":
            M, rhs, _ = solver.build_lscm(s["V"], s["F"])
        else:
            M, _ = solver.build_fairing(s["V"], s["F"], LAMBDA)
        _lib.load().nlgb_matrix_download(M.handle, s["rp"].ctypes.data_as(_lib.i32p),
                                         s["ci"].ctypes.data_as(_lib.i32p), s["va"].ctypes.data_as(_lib.f64p))
        out = {"rp": s["rp"], "ci": s["ci"], "va": s["va"]}
        if rhs is not None:
            out["rhs"] = rhs
        M.close()
        return out
    if kind == "opennl":
        return solver.solve_opennl(s["rows"])[0]
    if kind == "atlas":
        return solver.batch_solve(s["mats"], s["b"], precision=case["precision"])[0]
    if kind == "krylov":
        return s["M"].solve_krylov(s["b"], method=case["method"])[0]
    srv = s["server"]
    tickets = [srv.submit_mesh(k, V, F, b=b, lam=LAMBDA) for k, V, F, b in s["requests"]]
    return [srv.wait(t)[0] for t in tickets]


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------
def _edges(nx, ny):
    return (nx - 1) * ny + nx * (ny - 1) + (nx - 1) * (ny - 1)


def _nnz(system, nx, ny):
    pairs = nx * ny + 2 * _edges(nx, ny)
    return 4 * pairs if system == "lscm" else pairs


def _sizes(case):
    """Rows and an upper bound of the nonzeros of a built system."""
    nv = case["nx"] * case["ny"]
    return (2 * nv - 4 if case["system"] == "lscm" else nv), _nnz(case["system"], case["nx"], case["ny"])


def _iterations(system, nx, ny):
    """About how many PCG iterations 1e-10 takes."""
    return 0.66 * max(nx, ny) ** 1.77 if system == "lscm" else min(320.0, 8.0 * max(nx, ny))


def _solve_work(system, nx, ny, precision):
    n = 2 * nx * ny - 4 if system == "lscm" else nx * ny
    nnz, it = _nnz(system, nx, ny), _iterations(system, nx, ny)
    # per iteration the matrix (values and columns), the row pointers, and
    # x, r, p (read and written) and 1 / diagonal once each
    vb = 4 if precision == "mixed" else 8
    return it * ((vb + 4) * nnz + 4 * n + 7 * vb * n), it * (2 * nnz + 12 * n)


def work(case):
    kind = case["kind"]
    if kind == "spmv":
        n, nnz = _sizes(case)
        return {"bytes": 12 * nnz + 20 * n, "flops": 2 * nnz}
    if kind == "solve":
        b, f = _solve_work(case["system"], case["nx"], case["ny"], case["precision"])
        return {"bytes": b, "flops": f}
    if kind == "build":
        n, nnz = _sizes(case)
        nv, nt = case["nx"] * case["ny"], 2 * (case["nx"] - 1) * (case["ny"] - 1)
        return {"bytes": 24 * nv + 12 * nt + 12 * nnz + 4 * n, "flops": 80 * nt}
    if kind == "opennl":
        n = case["nx"] * case["ny"] * case["nz"]
        free, nnz, it = 0.7 * n, 0.7 * n * 18, 90
        return {"bytes": 7 * n * 12 + 12 * nnz + it * (12 * nnz + 60 * free), "flops": it * (2 * nnz + 12 * free)}
    if kind == "krylov":
        n = case["nx"] * case["ny"]
        it = (230 if case["method"] == "bicgstab" else 420) * max(case["nx"], case["ny"]) / 1024
        if case["method"] == "bicgstab":
            return {"bytes": it * (2 * 12 * 5 * n + 13 * 8 * n), "flops": it * (20 * n + 24 * n)}
        return {"bytes": it * (12 * 5 * n + 17 * 3 * 8 * n), "flops": it * (10 * n + 17 * 8 * n)}
    if kind == "atlas":
        w = [_solve_work("lscm", nx, ny, case["precision"]) for nx, ny, _ in _charts(case, 1)]
    else:
        rng = np.random.default_rng(23)
        w = []
        for _ in range(case["requests"]):
            nv = math.exp(rng.uniform(math.log(case["vmin"]), math.log(case["vmax"])))
            lscm = int(rng.integers(0, 2)) == 0
            side = max(4, int(round(math.sqrt(nv))))
            b, f = _solve_work("lscm" if lscm else "fairing", side, side, "double" if lscm else "mixed")
            w.append((b, f) if lscm else (3 * b, 3 * f))
    return {"bytes": sum(b for b, _ in w), "flops": sum(f for _, f in w)}


# ---------------------------------------------------------------------------
# The same results from plain torch in 64 bits
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _csr(n, i, j, a):
    m = torch.sparse_coo_tensor(torch.stack([i, j]), a, (n, n)).coalesce()
    i, j = m.indices()
    rp = torch.zeros(n + 1, dtype=torch.int64, device=i.device)
    rp[1:] = torch.cumsum(torch.bincount(i, minlength=n), 0)
    return torch.sparse_csr_tensor(rp, j, m.values(), (n, n))


def _cot_matrix(V, F):
    V, F = torch.from_numpy(V).to(_dev()), torch.from_numpy(F).to(_dev()).long()
    n = V.shape[0]
    I, J, A = [], [], []
    for k in range(3):
        o, i, j = F[:, k], F[:, (k + 1) % 3], F[:, (k + 2) % 3]
        u, v = V[i] - V[o], V[j] - V[o]
        w = 0.5 * (u * v).sum(1) / torch.linalg.cross(u, v).norm(dim=1)
        I += [i, j, i, j]
        J += [j, i, i, j]
        A += [-w, -w, w, w]
    d = torch.arange(n, device=V.device)
    return _csr(n, torch.cat(I + [d]), torch.cat(J + [d]),
                torch.cat(A + [torch.full((n,), LAMBDA, dtype=torch.float64, device=V.device)]))


def _lscm_matrix(V, F):
    """The normal matrix over the free variables and its right-hand side
    (vertex 0 pinned at (0, 0), the last one at (1, 1))."""
    V, F = torch.from_numpy(V).to(_dev()), torch.from_numpy(F).to(_dev()).long()
    nv = V.shape[0]
    e1, e2 = V[F[:, 1]] - V[F[:, 0]], V[F[:, 2]] - V[F[:, 0]]
    x1 = e1.norm(dim=1)
    X = e1 / x1[:, None]
    N = torch.linalg.cross(e1, e2)
    Y = torch.linalg.cross(N / N.norm(dim=1)[:, None], X)
    x2, y2 = (e2 * X).sum(1), (e2 * Y).sum(1)
    s = 1.0 / torch.sqrt(x1 * y2)
    a = [(x2 - x1) * s, -x2 * s, x1 * s]
    b = [y2 * s, -y2 * s, torch.zeros_like(s)]
    var = torch.stack([2 * F[:, 0], 2 * F[:, 0] + 1, 2 * F[:, 1], 2 * F[:, 1] + 1, 2 * F[:, 2], 2 * F[:, 2] + 1], 1)
    re = torch.stack([a[0], -b[0], a[1], -b[1], a[2], -b[2]], 1)
    im = torch.stack([b[0], a[0], b[1], a[1], b[2], a[2]], 1)
    K = re[:, :, None] * re[:, None, :] + im[:, :, None] * im[:, None, :]
    i = var[:, :, None].expand(-1, 6, 6).reshape(-1)
    j = var[:, None, :].expand(-1, 6, 6).reshape(-1)
    K = K.reshape(-1)
    n = 2 * nv - 4
    free_i, free_j = (i >= 2) & (i < 2 * nv - 2), (j >= 2) & (j < 2 * nv - 2)
    at = free_i & (j >= 2 * nv - 2)          # the last vertex is at (1, 1)
    rhs = torch.zeros(n, dtype=torch.float64, device=V.device)
    rhs.index_add_(0, i[at] - 2, -K[at])
    both = free_i & free_j
    return _csr(n, i[both] - 2, j[both] - 2, K[both]), rhs


def _diagonal(M):
    rp, j = M.crow_indices(), M.col_indices()
    i = torch.repeat_interleave(torch.arange(M.shape[0], device=j.device), rp[1:] - rp[:-1])
    d = torch.zeros(M.shape[0], dtype=torch.float64, device=j.device)
    d.index_add_(0, i[i == j], M.values()[i == j])
    return d


def _cg(mul, b, diag, tol, most):
    x, r = torch.zeros_like(b), b.clone()
    z = r / diag
    p, rho, stop = z.clone(), r @ z, float(b @ b) * tol * tol
    for k in range(most):
        q = mul(p)
        alpha = rho / (p @ q)
        x += alpha * p
        r -= alpha * q
        z = r / diag
        new = r @ z
        p = z + (new / rho) * p
        rho = new
        if k % 32 == 31 and float(r @ r) <= stop:
            break
    return x


def _spd(mul, b, diag, tol=1e-12, most=40000):
    """The solution of an SPD system: CG, then one correction of its residual."""
    x = _cg(mul, b, diag, tol, most)
    return x + _cg(mul, b - mul(x), diag, 1e-3, most)


def _bicgstab(mul, b, diag, tol, most=4000):
    x, r = torch.zeros_like(b), b.clone()
    rh, p, rho, stop = r.clone(), r.clone(), r @ r, float(b @ b) * tol * tol
    for k in range(most):
        y = p / diag
        v = mul(y)
        alpha = rho / (rh @ v)
        t0 = r - alpha * v
        z = t0 / diag
        t = mul(z)
        omega = (t @ t0) / (t @ t)
        x += alpha * y + omega * z
        r = t0 - omega * t
        if k % 16 == 15 and float(r @ r) <= stop:
            break
        new = rh @ r
        p = r + (new / rho) * (alpha / omega) * (p - omega * v)
        rho = new
    return x


def _solution(system, V, F, rhs=None):
    if system == "lscm":
        M, rhs = _lscm_matrix(V, F)
    else:
        M, rhs = _cot_matrix(V, F), torch.from_numpy(rhs).to(_dev())
    return _spd(lambda v: M @ v, rhs, _diagonal(M)).cpu()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("spmv", "solve"):
        V, F = _mesh(case["nx"], case["ny"], seed)
        if kind == "spmv":
            M = _lscm_matrix(V, F)[0] if case["system"] == "lscm" else _cot_matrix(V, F)
            return (M @ torch.from_numpy(_rng(seed, 3).standard_normal(M.shape[0])).to(_dev())).cpu()
        return _solution(case["system"], V, F, _fairing_rhs(V, seed)[0])
    if kind == "build":
        V, F = _mesh(case["nx"], case["ny"], seed)
        M, rhs = _lscm_matrix(V, F) if case["system"] == "lscm" else (_cot_matrix(V, F), None)
        fill = (0, _sizes(case)[1] - M.values().numel())
        out = {"rp": M.crow_indices().int().cpu(), "ci": torch.nn.functional.pad(M.col_indices().int(), fill).cpu(),
               "va": torch.nn.functional.pad(M.values(), fill).cpu()}
        if rhs is not None:
            out["rhs"] = rhs.cpu()
        return out
    if kind == "opennl":
        return _voxel_solution(case, seed)
    if kind == "atlas":
        return [_solution("lscm", *_mesh(nx, ny, sd)) for nx, ny, sd in _charts(case, seed)]
    if kind == "krylov":
        sq = systems.convection_diffusion(case["nx"], case["ny"], int(seed))
        M = torch.sparse_csr_tensor(torch.from_numpy(sq.rp).long(), torch.from_numpy(sq.ci).long(),
                                    torch.from_numpy(sq.va), (sq.n, sq.n)).to(_dev())
        d, b = _diagonal(M), torch.from_numpy(sq.rhs[0]).to(_dev())
        mul = lambda v: M @ v   # noqa: E731
        x = _bicgstab(mul, b, d, 1e-12)
        return (x + _bicgstab(mul, b - mul(x), d, 1e-3)).cpu()
    out = []
    for k, V, F, b in _requests(case, seed):
        out.append(torch.stack([_solution(k, V, F, r) for r in (b if b is not None else [None])]))
    return out


def _voxel_solution(case, seed):
    rs = systems.voxel_rows(case["nx"], case["ny"], case["nz"], int(seed))
    dev, n = _dev(), rs.n_vars
    A = torch.sparse_csr_tensor(torch.from_numpy(rs.row_ptr).long(), torch.from_numpy(rs.var).long(),
                                torch.from_numpy(rs.val), (n, n)).to(dev)   # n rows over all variables
    free = torch.from_numpy(rs.locked == 0).to(dev)
    known = torch.from_numpy(rs.values[0]).to(dev) * (~free)
    At = _csr(n, A.col_indices(), torch.repeat_interleave(torch.arange(n, device=dev), 7), A.values())
    mul = lambda v: (At @ (A @ (v * free))) * free + v * (~free)   # noqa: E731
    diag = torch.zeros(n, dtype=torch.float64, device=dev)
    diag.index_add_(0, A.col_indices(), A.values() ** 2)
    diag = torch.where(free, diag, torch.ones_like(diag))
    x = _spd(mul, -(At @ (A @ known)) * free, diag)
    return (torch.where(free, x, known))[None, :].cpu()
