"""The automatic schedule of the FP32 form: the persistent launch for short factorizations with
the engine that has a task body, the level-ordered sequence otherwise, and whatever is asked
for explicitly.  Host-only handles: the choice needs no GPU."""
import pytest

from sympack_b200 import DistSparseMatrix, generators as G, symPACKMatrix2D, symPACKOptions


def launches(A, offsets=None, **opt):
    M = symPACKMatrix2D()
    M.Init(symPACKOptions(device=-1, **opt))
    if offsets is None:
        M.SymbolicFactorization(A)
    else:
        M.SymbolicFactorizationBatch(A, offsets)
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


@pytest.mark.parametrize("count,persistent", [(10, True), (300, False)])
def test_a_wide_batch_keeps_the_step_sequence(count, persistent):
    """Many small systems: a few launches take a level of all of them, where the persistent
    launch would take them a block per SM.  What is asked for explicitly stays."""
    n, cp, ri, v, offsets = G.block_diagonal([G.laplacian_2d(30, 30, 1e-3)] * count)
    A = DistSparseMatrix.from_lower_csc(n, cp, ri, v)
    assert (launches(A, offsets, precision="FP32_IR")[0] == 1) == persistent
    assert launches(A, offsets, precision="FP32_IR", factor_schedule="persistent")[0] == 1
    assert launches(A, offsets, precision="FP32_IR", factor_schedule="steps")[0] > 1
    assert launches(A, offsets)[0] == 1  # FP64
