"""The automatic schedule of the FP32 form: the persistent launch for short factorizations with
the engine that has a task body, the level-ordered sequence otherwise, and whatever is asked
for explicitly.  Host-only handles: the choice needs no GPU."""
import pytest

from sympack_b200 import DistSparseMatrix, generators as G, symPACKMatrix2D, symPACKOptions


def launches(A, **opt):
    M = symPACKMatrix2D()
    M.Init(symPACKOptions(device=-1, **opt))
    M.SymbolicFactorization(A)
    inf = M.info()
    M.close()
    return inf.factor_launches, inf.factor_tasks


@pytest.mark.parametrize("precision,engine,schedule,persistent", [
    ("FP32_IR", "tcgen05-tma", "auto", True),
    ("FP32_IR", "tcgen05-tma", "steps", False),
    ("FP32_IR", "tcgen05-tma", "persistent", True),
    ("FP32_IR", "tcgen05", "auto", False),
    ("FP32_IR", "mma.sync", "persistent", False),
    ("FP64", "tcgen05-tma", "auto", True),
    ("FP64", "tcgen05-tma", "steps", False),
])
def test_schedule_of_a_short_factorization(precision, engine, schedule, persistent):
    A = DistSparseMatrix.from_lower_csc(*G.stencil27(14, 14, 14, 1e-2))
    n, tasks = launches(A, precision=precision, fp32_engine=engine, factor_schedule=schedule)
    assert (n == 1) == persistent and (tasks > 0) == persistent


def test_a_long_fp32_factorization_keeps_the_step_sequence():
    A = DistSparseMatrix.from_lower_csc(*G.stencil27(54, 54, 54, 1e-2))  # 7e11 flops
    assert launches(A, precision="FP32_IR")[0] > 1
    assert launches(A, precision="FP32_IR", factor_schedule="persistent")[0] == 1
