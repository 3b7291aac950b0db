"""compute_quotient_values called from several threads on one context, with
programs whose rows of shared memory differ from a few words to the most the
staged form holds, and beyond it the general form: every call succeeds and
every result is the one the call gives alone.
"""
import threading

import numpy as np
import pytest

from pico_b200 import TwoAdicDomain, TwoAdicFriPcs
from pico_b200 import fields as F
from pico_b200.quotient import ConstraintBuilder, compute_quotient_values

pytestmark = pytest.mark.gpu
CALLS = 60


def _program(f, cols):
    bld = ConstraintBuilder()
    for c in range(cols):
        bld.when_transition().assert_eq(bld.main(c, True), bld.main(c) * bld.main((c + 1) % cols))
    return bld.program(f)


@pytest.mark.parametrize("f", [0, 1])
def test_programs_of_different_widths_at_once(gpu, orc, f):
    logn, widths = 6, [2, 200, 12, 100, 230, 3]  # words a row: about twice the width
    alpha = F.random_matrix(f, 0, 4, 920)[0]
    mains = [F.random_matrix(f, logn, w, 921 + w) for w in widths]
    progs = [_program(f, w) for w in widths]
    pcs = TwoAdicFriPcs(gpu, f, 1)
    _, pd = pcs.commit([(TwoAdicDomain(logn), m) for m in mains])
    want = [orc.quotient_values(f, logn, 1, p, orc.on_quotient_domain(f, m, 1), alpha=alpha)
            for p, m in zip(progs, mains)]
    errors = []
    start = threading.Barrier(len(widths))

    def work(i):
        try:
            start.wait()
            for _ in range(CALLS):
                got = compute_quotient_values(gpu, progs[i], logn, 1, (pd, i), alpha=alpha)
                if not (got == want[i]).all():
                    raise AssertionError(f"width {widths[i]}: another result than alone")
        except Exception as e:  # noqa: BLE001  (reported below, with its width)
            errors.append((widths[i], repr(e)))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(widths))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    pd.release()
    assert not errors, errors
