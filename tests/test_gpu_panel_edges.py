"""Factorization tasks at the edges of their shapes: small panels whose width is not a multiple
of the 8-column pieces, with off-diagonal parts around what a warp (24 rows), a block (192
rows) and the fused external update (128 rows) take; diagonal blocks narrower than 64 and row
tiles that end inside a warp's 16 rows; both schedules, Cholesky and LDL^T.  Factor and
solution agree with the CPU oracle to 1e-12, the other GPU tests' bound (condition below 1e3)."""
import numpy as np
import pytest

from sympack_b200 import DistSparseMatrix, generators as G
from test_gpu_solve_edges import bordered, oracle_for, solver

pytestmark = pytest.mark.gpu
TOL = 1e-12
WIDTHS = [1, 7, 8, 9, 17, 24, 31, 32, 33, 40, 65, 100]


@pytest.mark.parametrize("schedule", ["persistent", "steps"])
@pytest.mark.parametrize("dec", ["LL", "LDL"])
@pytest.mark.parametrize("border", [2, 15, 25, 127, 128, 129, 210, 400])
def test_panel_tasks_match_the_oracle(border, dec, schedule):
    A = DistSparseMatrix.from_lower_csc(*bordered(WIDTHS, border, border + 1))
    M = solver(A, decomposition=dec, factor_schedule=schedule)
    w = np.diff(M.GetSupernodalPartition())
    assert set(w.tolist()) >= {7, 9, 17, 31, 33, 65}
    f = oracle_for(M, A, dec == "LDL")
    Lo = f.factor()
    assert np.max(np.abs(M.GetFactor() - Lo)) <= TOL * np.max(np.abs(Lo))
    b = np.random.default_rng(2).standard_normal((A.size, 3))
    M.Solve(b)
    x, xo = M.GetSolution(nrhs=3), f.solve(b)
    assert np.max(np.abs(x - xo)) <= TOL * np.max(np.abs(xo))
    M.close()


@pytest.mark.parametrize("schedule", ["persistent", "steps"])
@pytest.mark.parametrize("dec", ["LL", "LDL"])
@pytest.mark.parametrize("width,border", [(65, 60), (65, 123), (80, 60), (96, 32), (110, 1)])
def test_small_panels_wider_than_64_columns(width, border, dec, schedule):
    """plan_small_max_w above 64: panels up to the widest that fit in shared memory (110 columns,
    96 KB), D of LDL^T kept beside the column tables of the fused update."""
    A = DistSparseMatrix.from_lower_csc(*bordered([width, width], border, width + border))
    M = solver(A, decomposition=dec, factor_schedule=schedule, plan_small_max_w=4096)
    assert width in np.diff(M.GetSupernodalPartition())
    f = oracle_for(M, A, dec == "LDL")
    Lo = f.factor()
    assert np.max(np.abs(M.GetFactor() - Lo)) <= TOL * np.max(np.abs(Lo))
    b = np.random.default_rng(3).standard_normal((A.size, 2))
    M.Solve(b)
    x, xo = M.GetSolution(nrhs=2), f.solve(b)
    assert np.max(np.abs(x - xo)) <= TOL * np.max(np.abs(xo))
    M.close()


@pytest.mark.parametrize("dec", ["LL", "LDL"])
def test_update_tiles_see_the_panels_finished_before_them(dec):
    """Bulk copies of the update tiles read panels that other blocks of the same launch have just
    stored; the step sequence, a launch per step, has no such hand-over.  Both agree every time."""
    A = DistSparseMatrix.from_lower_csc(*(G.stencil27(16, 16, 16, 1e-2) if dec == "LL" else G.quasi_definite_3d(16, 16, 16)))
    M, S = (solver(A, decomposition=dec, factor_schedule=k) for k in ("persistent", "steps"))
    Ls = S.GetFactor()
    for _ in range(20):
        M.DistributeMatrix(A)
        M.Factorize()
        assert np.max(np.abs(M.GetFactor() - Ls)) <= TOL * np.max(np.abs(Ls))
    M.close()
    S.close()


@pytest.mark.parametrize("schedule", ["persistent", "steps"])
@pytest.mark.parametrize("dec", ["LL", "LDL"])
@pytest.mark.parametrize("widths,border", [([1] * 70, 1), ([1] * 40, 31), ([3, 4] * 20, 4), ([5, 7] * 15, 9), ([12] * 9, 30), ([30] * 5, 20)])
def test_launches_of_tiny_panels(widths, border, dec, schedule):
    """Panels of up to 32, 256 and 1,024 entries, the sizes up to which a launch of them takes 32,
    64 and 128 threads a panel; pieces that end before their eighth column."""
    A = DistSparseMatrix.from_lower_csc(*bordered(widths, border, len(widths)))
    M = solver(A, decomposition=dec, factor_schedule=schedule)
    f = oracle_for(M, A, dec == "LDL")
    Lo = f.factor()
    assert np.max(np.abs(M.GetFactor() - Lo)) <= TOL * np.max(np.abs(Lo))
    M.close()


@pytest.mark.parametrize("column", [0, 5, 12, 40])
def test_a_bad_pivot_is_reported_where_it_is(column):
    """The first non-positive pivot's column, in a piece's interior and beyond the first piece."""
    from sympack_b200.solver import NotSPDError
    n, cp, ri, v = bordered([60, 20], 30, 4)
    v = v.copy()
    v[cp[column] - 1] = -1.0  # the diagonal entry (first of its column)
    with pytest.raises(NotSPDError, match=f"column {column + 1}$"):
        solver(DistSparseMatrix.from_lower_csc(n, cp, ri, v))


@pytest.mark.parametrize("schedule", ["persistent", "steps"])
def test_diagonal_entries_are_the_rounded_square_roots(schedule):
    """Pivots that no update touches: diagonal matrices (one-column panels) and the first column
    of dense 64-column and wider blocks.  L_kk is sqrt's result, bit for bit."""
    d = np.random.default_rng(5).uniform(1e-3, 1e3, 2000)
    n = len(d)
    M = solver(DistSparseMatrix.from_lower_csc(n, np.arange(1, n + 2), np.arange(1, n + 1, dtype=np.int32), d),
               factor_schedule=schedule)
    assert np.array_equal(M.GetFactor()[M.GetOrdering()[1] - 1], np.sqrt(d))
    M.close()
    for seed in range(20):
        n, cp, ri, v = bordered([40, 70], 30, seed)
        M = solver(DistSparseMatrix.from_lower_csc(n, cp, ri, v), factor_schedule=schedule)
        L, pos = M.GetFactor(), 0
        xs, (xl, li), perm = M.GetSupernodalPartition(), M.GetStructure(), M.GetOrdering()[0]
        for s in range(len(xs) - 1):
            c = perm[xs[s] - 1]
            if c in (1, 41):  # the first column of each block
                assert L[pos] == np.sqrt(v[cp[c - 1] - 1])
            pos += (xs[s + 1] - xs[s]) * (xl[s + 1] - xl[s])
        M.close()
