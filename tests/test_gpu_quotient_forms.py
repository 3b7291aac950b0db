"""Both forms of the quotient kernel on either side of the rule that chooses
between them, against the oracle: wide and extension-heavy programs over more
points than a wave (the general form, although their rows would fit in shared
memory), op-heavy ones (staged), and every instruction in the general form
(more words read than a row of shared memory holds).  Every comparison is exact.
"""
import numpy as np
import pytest

from pico_b200 import TwoAdicDomain, TwoAdicFriPcs
from pico_b200 import fields as F
from pico_b200.quotient import ConstraintBuilder, compute_quotient_values

pytestmark = pytest.mark.gpu
FIELDS = [0, 1]


def _check(gpu, orc, f, logn, log_qd, prog, main, perm=None, prep=None, **kw):
    b = max(1, log_qd)
    mats = [m for m in (main, perm, prep) if m is not None]
    _, pd = TwoAdicFriPcs(gpu, f, b).commit([(TwoAdicDomain(logn), m) for m in mats])
    refs, cpu = {}, {}
    if perm is not None:  # base words, four per extension column
        refs["permutation"] = (pd, 1)
        q = orc.on_quotient_domain(f, perm, log_qd)
        cpu["perm_q"] = q.reshape(q.shape[0], -1, 4)
    if prep is not None:
        refs["preprocessed"] = (pd, len(mats) - 1)
        cpu["prep_q"] = orc.on_quotient_domain(f, prep, log_qd)
    alpha = F.random_matrix(f, 0, 4, 931)[0]
    got = compute_quotient_values(gpu, prog, logn, log_qd, (pd, 0), alpha=alpha, **refs, **kw)
    want = orc.quotient_values(f, logn, log_qd, prog, orc.on_quotient_domain(f, main, log_qd), alpha=alpha, **cpu, **kw)
    pd.release()
    assert (got == want).all()


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("cols,reps,ext", [(60, 0, 0), (100, 0, 0), (100, 100, 0), (130, 0, 0), (20, 0, 10)])
def test_more_points_than_a_wave(gpu, orc, f, cols, reps, ext):
    logn = 15
    rng = np.random.default_rng(cols + reps)
    bld = ConstraintBuilder()
    for c in range(cols):
        bld.when_transition().assert_eq(bld.main(c, True), bld.main(c) * bld.main((c + 1) % cols))
    for _ in range(reps):
        x, y, z = (int(v) for v in rng.integers(0, cols, 3))
        bld.assert_zero(bld.main(x) * bld.main(y) - bld.main(z))
    for j in range(ext):
        z, zn = bld.permutation(j), bld.permutation(j, True)
        bld.when_transition().assert_zero((zn - z) * (bld.challenge(0) + bld.main(0)) - bld.main(1))
    perm = F.random_matrix(f, logn, 4 * ext, 933) if ext else None
    chal = F.random_matrix(f, 1, 4, 934)
    _check(gpu, orc, f, logn, 1, bld.program(f), F.random_matrix(f, logn, cols, 932), perm, perm_challenges=chal)


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("logn,log_qd", [(1, 0), (5, 1), (8, 2)])
def test_every_instruction_in_the_general_form(gpu, orc, f, logn, log_qd):
    cols = 450  # words read: a row of shared memory holds fewer
    bld = ConstraintBuilder()
    z, zn, pre = bld.permutation(0), bld.permutation(1, True), bld.preprocessed(1, True)
    bld.when_first_row().assert_eq(bld.main(0), bld.public(0))
    bld.when_last_row().assert_eq(bld.main(1, True), bld.public(1) + bld.const(5))
    bld.when_transition().assert_zero((zn - z) * (bld.challenge(0) + bld.main(2)) - pre)
    bld.assert_zero(z * bld.preprocessed(0) + bld.regional_cumulative_sum())
    bld.assert_eq(bld.main(3), bld.global_cumulative_sum(7))
    x = bld.main(0)
    for c in range(1, cols):
        x = x + bld.main(c)
    bld.assert_zero(x * x)
    bld.assert_zero(zn)
    rng = np.random.default_rng(5)
    word = lambda *s: F.to_monty(f, rng.integers(0, F.P[f], size=s, dtype=np.uint64).astype(np.uint32).ravel()).reshape(s)
    _check(gpu, orc, f, logn, log_qd, bld.program(f), F.random_matrix(f, logn, cols, 940), F.random_matrix(f, logn, 8, 941),
           F.random_matrix(f, logn, 2, 942), public_values=word(2), perm_challenges=word(2, 4), regional_sum=word(4),
           global_sum=word(14))
