"""Normal-equation merge (csrc/nlgb_assembly.cu) at the limits of its three
paths -- one thread per row up to 24 rows and 32 columns per variable, one
warp up to 256 candidates, one CTA above -- bit for bit against the oracle."""
import numpy as np
import pytest

from graphitethree_gb300 import solver, systems

pytestmark = pytest.mark.gpu


def _stream(degree, width, n_vars, seed, n_systems=1):
    """`degree` rows of `width` coefficients per variable on average, variable
    0 in exactly `degree` of them, some variables locked or in no row."""
    rng = np.random.default_rng(seed)
    n_rows = max(degree, n_vars * degree // width)
    var = np.stack([rng.choice(np.arange(1, n_vars), width, replace=False) for _ in range(n_rows)])
    var[:degree, 0] = 0
    locked = (rng.random(n_vars) < 0.1).astype(np.uint8)
    locked[0] = 0
    return systems.RowStream(
        n_vars=n_vars, row_ptr=np.arange(0, n_rows * width + 1, width, dtype=np.int64),
        var=var.reshape(-1).astype(np.int32), val=rng.standard_normal(n_rows * width),
        rhs=rng.standard_normal((n_rows, n_systems)), locked=locked,
        values=np.where(locked, rng.standard_normal((n_systems, n_vars)), 0.0), least_squares=True,
        weight=rng.uniform(0.5, 2.0, n_rows))


@pytest.mark.parametrize("degree,width,n_vars,n_systems", [
    (1, 1, 2, 1), (3, 2, 40, 1), (12, 6, 700, 3), (24, 2, 200, 1), (25, 2, 200, 1), (16, 3, 33, 1), (16, 3, 34, 2),
    (7, 12, 300, 1), (40, 6, 128, 1), (43, 6, 500, 1), (60, 20, 257, 1)])
def test_merge_paths_bit_exact(gpu_ok, oracle_mod, degree, width, n_vars, n_systems):
    rs = _stream(degree, width, n_vars, 1000 * degree + width, n_systems)
    rp, ci, va, rhs = oracle_mod.assemble_rowstream(rs)
    M, grhs, _ = solver.assemble(rs)
    g_rp, g_ci, g_va = M.download()
    assert np.array_equal(g_rp, rp) and np.array_equal(g_ci, ci)
    assert np.array_equal(g_va, va)
    assert np.array_equal(grhs, rhs)
