"""The staged form of compute_quotient_values against the oracle: rows of
shared memory up to the largest and, beyond it, the general form; fewer
points than a block; columns read in part, in any order, from both rows;
registers that are read again after the assertion of their value, or never
written by an instruction of their own.  Every comparison is exact.
"""
import numpy as np
import pytest

from pico_b200 import TwoAdicDomain, TwoAdicFriPcs
from pico_b200 import fields as F
from pico_b200.quotient import OPS, ConstraintBuilder, compute_quotient_values

pytestmark = pytest.mark.gpu
FIELDS = [0, 1]


def _check(gpu, orc, f, logn, log_qd, prog, main, alpha_seed):
    alpha = F.random_matrix(f, 0, 4, alpha_seed)[0]
    _, pd = TwoAdicFriPcs(gpu, f, max(1, log_qd)).commit([(TwoAdicDomain(logn), main)])
    got = compute_quotient_values(gpu, prog, logn, log_qd, (pd, 0), alpha=alpha)
    want = orc.quotient_values(f, logn, log_qd, prog, orc.on_quotient_domain(f, main, log_qd), alpha=alpha)
    pd.release()
    assert (got == want).all()


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("logn,log_qd", [(1, 0), (1, 1), (4, 1), (6, 2), (8, 0)])
@pytest.mark.parametrize("cols", [1, 7, 8, 9, 100, 212, 215, 300])
def test_columns_read_from_both_rows(gpu, orc, f, logn, log_qd, cols):
    # the words read are about 2 * cols: the staged form holds 440
    width = cols + 3
    rng = np.random.default_rng(cols)
    bld = ConstraintBuilder()
    for c in rng.permutation(cols):
        bld.when_transition().assert_eq(bld.main(int(c), True), bld.main(int(c)) * bld.main(int(c + 3)))
    bld.when_first_row().assert_zero(bld.main(0))
    bld.when_last_row().assert_eq(bld.main(width - 1, True), bld.const(7))
    _check(gpu, orc, f, logn, log_qd, bld.program(f), F.random_matrix(f, logn, width, 900 + cols), 901)


@pytest.mark.parametrize("f", FIELDS)
def test_registers_read_and_written_again(gpu, orc, f):
    o = {k: v for k, v in OPS.items()}
    prog = np.array([
        [o["MAIN"], 0, 2, 0], [o["MAIN"], 1, 0, 1], [o["TRANSITION"], 2, 0, 0],
        [o["MUL"], 3, 0, 1], [o["ASSERT"], 0, 3, 0],   # read again below
        [o["ADD"], 4, 3, 2], [o["ASSERT"], 0, 4, 0],   # not read again: written below
        [o["MAIN"], 4, 1, 0], [o["ADD"], 0, 0, 4],     # a register that held a column is written
        [o["MAIN"], 0, 1, 1], [o["SUB"], 0, 0, 0], [o["ASSERT"], 0, 0, 0],
        [o["SUB"], 5, 3, 1], [o["ASSERT"], 0, 5, 0], [o["ASSERT"], 0, 5, 0],
        [o["MUL"], 6, 5, 5], [o["ASSERT"], 0, 2, 0],   # of another value than the instruction before it made
        [o["ASSERT"], 0, 6, 0],
        [o["EMB"], 0, 1, 0], [o["MUL"], 1, 1, 1], [o["EMULB"], 0, 0, 1], [o["EASSERT"], 0, 0, 0],
        [o["ADD"], 7, 1, 1], [o["ASSERT"], 0, 7, 0], [o["EMB"], 1, 7, 0], [o["EASSERT"], 0, 1, 0],
        [o["MUL"], 7, 7, 2], [o["ASSERT"], 0, 7, 0],
    ], dtype=np.uint32)
    _check(gpu, orc, f, 6, 1, prog, F.random_matrix(f, 6, 3, 910), 911)
