"""Commits whose heights' LDEs share launches (device inputs, batched form):
every one-pass height in one launch next to three-pass ones, below and above
the size from which the tallest group's LDE runs by itself, against the oracle.
Field elements: every comparison is exact.
"""
import numpy as np
import pytest

from pico_b200 import TwoAdicDomain, TwoAdicFriPcs
from pico_b200 import fields as F

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("f,b", [(0, 1), (1, 2)])
@pytest.mark.parametrize("tallest", [None, (18, 66)])
def test_every_height_in_one_commit(gpu, orc, f, b, tallest):
    import torch

    shapes = [(h, 1 + (7 * h) % 23) for h in range(14)] + ([tallest] if tallest else [])
    traces = [F.random_matrix(f, h, w, 70 + h) for h, w in shapes]
    want_root, want_ldes, _ = orc.pcs_commit(f, traces, [F.lde_shift(f)] * len(traces), b, want_ldes=True)
    dev = [torch.from_numpy(t.view(np.int32)).cuda() for t in traces]
    root, pd = TwoAdicFriPcs(gpu, f, b).commit([(TwoAdicDomain(h), t) for (h, _), t in zip(shapes, dev)])
    for i, want in enumerate(want_ldes):
        assert (pd.lde(i) == want).all(), shapes[i]
    pd.release()
    assert (root == want_root).all()
