"""The assertion sum of compute_quotient_values at the ends of its range:
no assertion, one, many base and extension ones in turn, and values and
challenges of 0 and p - 1, against the oracle.  Every comparison is exact.
"""
import numpy as np
import pytest

from pico_b200 import TwoAdicDomain, TwoAdicFriPcs
from pico_b200 import fields as F
from pico_b200.quotient import ConstraintBuilder, compute_quotient_values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f", [0, 1])
@pytest.mark.parametrize("alpha_word", [0, 1, None])  # Monty words 0, 1 and p - 1
@pytest.mark.parametrize("asserts", [0, 1, 2, 70])
def test_assertion_sum_ends(gpu, orc, f, alpha_word, asserts):
    logn, w = 5, 3
    p = F.P[f]
    main = F.random_matrix(f, logn, w, 700 + asserts)
    main[:, 1] = p - 1
    main[:, 2] = 0
    bld = ConstraintBuilder()
    top, ch = bld.const(F.from_monty(f, np.array([p - 1], dtype=np.uint32))[0]), bld.challenge(0)
    for k in range(asserts):
        bld.assert_zero([top, bld.main(k % w), ch, ch * bld.main(1)][k % 4])
    prog = bld.program(f)
    alpha = np.full(4, p - 1 if alpha_word is None else alpha_word, dtype=np.uint32)
    chal = np.full((1, 4), p - 1, dtype=np.uint32)
    _, pd = TwoAdicFriPcs(gpu, f, 1).commit([(TwoAdicDomain(logn), main)])
    got = compute_quotient_values(gpu, prog, logn, 1, (pd, 0), perm_challenges=chal, alpha=alpha)
    want = orc.quotient_values(f, logn, 1, prog, orc.on_quotient_domain(f, main, 1), perm_challenges=chal, alpha=alpha)
    assert (got == want).all()
    pd.release()
