"""nlgb_add_rows' bulk path against nlBegin(NL_ROW)/nlCoefficient/nlEnd(NL_ROW)
one call at a time: runs of plain rows broken by rows that name a variable
twice, long and empty rows (the limit of 32 coefficients), locked variables,
weights, several systems, and calls with fewer coefficients than variables."""
import numpy as np
import pytest

from graphitethree_gb300 import opennl as nl
from graphitethree_gb300 import solver, systems

pytestmark = pytest.mark.gpu


def _rows(n, seed, lengths, n_systems=1, twice=0.2, locked=0.1, weighted=True):
    rng = np.random.default_rng(seed)
    ptr, var, val = [0], [], []
    for r in range(n):                       # a row per variable keeps A^T A regular
        v = rng.choice(n, min(n, int(rng.choice(lengths))), replace=False)
        if len(v) and rng.random() < twice:
            v = np.concatenate([v, v[:1]])
        v = np.concatenate([[r], v[v != r]]) if len(v) else v
        var += list(v)
        val += list(rng.uniform(-1, 1, len(v)) + 3.0 * (v == r))
        ptr.append(len(var))
    for r in range(n):
        var.append(r)
        val.append(1.0)
        ptr.append(len(var))
    m = len(ptr) - 1
    return systems.RowStream(
        n_vars=n, least_squares=True, row_ptr=np.array(ptr, np.int64), var=np.array(var, np.int32),
        val=np.array(val), rhs=rng.standard_normal((m, n_systems)),
        weight=rng.uniform(0.5, 2.0, m) if weighted else None,
        locked=(rng.random(n) < locked).astype(np.uint8), values=rng.standard_normal((n_systems, n)))


@pytest.mark.parametrize("lengths,n_systems,weighted", [
    ([1, 2, 5], 1, False), ([0, 3], 1, True), ([6, 31, 32, 33, 40], 2, True), ([7], 3, False)])
@pytest.mark.parametrize("twice", [0.0, 0.3, 1.0])
def test_same_system(gpu_ok, lengths, n_systems, weighted, twice):
    rs = _rows(60, 5, lengths, n_systems, twice, weighted=weighted)
    a, ia = solver.solve_opennl(rs, eps=1e-12)
    b, ib = solver.solve_opennl(rs, eps=1e-12, per_call=True)
    assert ia["status"] == ib["status"] == "converged" and ia["nnz"] == ib["nnz"]
    assert ia["iterations"] == ib["iterations"] and np.array_equal(a, b)


def test_few_rows_per_call(gpu_ok):
    """One row at a time (fewer coefficients than variables)."""
    rs = _rows(40, 9, [4], twice=0.5, locked=0.0, weighted=False)
    want, _ = solver.solve_opennl(rs, eps=1e-12)
    ctx = nl.nlNewContext()
    nl.nlSolverParameteri(nl.NL_NB_VARIABLES, rs.n_vars)
    nl.nlSolverParameteri(nl.NL_LEAST_SQUARES, nl.NL_TRUE)
    nl.nlSolverParameterd(nl.NL_THRESHOLD, 1e-12)
    nl.nlBegin(nl.NL_SYSTEM)
    nl.nlgbSetVariables(rs.values, rs.locked)
    nl.nlBegin(nl.NL_MATRIX)
    for r in range(rs.n_rows):
        k = slice(rs.row_ptr[r], rs.row_ptr[r + 1])
        n = rs.row_ptr[r + 1] - rs.row_ptr[r]
        assert nl.nlgbAddRows(np.array([0, n]), rs.var[k], rs.val[k], rs.rhs[r]) == 0
    assert nl.nlgbAddRows(np.array([0, 1]), np.array([-1]), np.array([1.0])) != 0
    assert nl.nlgbAddRows(np.array([0, 1]), np.array([40]), np.array([1.0])) != 0
    nl.nlEnd(nl.NL_MATRIX)
    nl.nlEnd(nl.NL_SYSTEM)
    assert nl.nlSolve()
    got = nl.nlgbGetVariables(1, rs.n_vars)
    nl.nlDeleteContext(ctx)
    assert np.array_equal(got, want)
