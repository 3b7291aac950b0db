"""The 16-lanes-per-state Poseidon2 kernels (few rows, narrow tree levels)
against the oracle: every split of a narrow tree into launches with digests
injected at every level, warps whose two rows differ in width, row counts and
widths around the lines between the row-hashing kernels, and the resumable
form.  All values are field elements: every comparison is exact.
"""
import numpy as np
import pytest

from pico_b200 import MerkleTreeMmcs, TwoAdicFriPcs, new_challenger
from pico_b200 import fields as F

pytestmark = pytest.mark.gpu
FIELDS = [0, 1]


def _dev(a):
    import torch

    return torch.from_numpy(a.view(np.int32)).cuda()


def _check(gpu, orc, f, mats, **how):
    want_root, want_layers = orc.mmcs_commit(f, mats, want_layers=True)
    given = mats if how.pop("host", False) else [_dev(m) for m in mats]
    root, pd = MerkleTreeMmcs(gpu, f).commit(given, **how)
    top = max(m.shape[0] for m in mats).bit_length() - 1
    got = np.concatenate([pd.digest_layer(level) for level in range(top + 1)])
    pd.release()
    assert (got == want_layers).all()
    assert (root == want_root).all()


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("top", [0, 1, 2, 5, 6, 7, 8, 9, 13, 14, 15])
def test_narrow_trees_with_rows_at_every_level(gpu, orc, f, top):
    # heights 2^top .. 2^0: every level of the tree takes an injected digest, and
    # the short groups put rows of different widths into one warp
    _check(gpu, orc, f, [F.random_matrix(f, h, 1 + (5 * h) % 19, 60 + h) for h in range(top, -1, -1)])


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("log_rows", [4, 12, 13, 14])
@pytest.mark.parametrize("widths", [[8], [9], [3, 13]])
@pytest.mark.parametrize("form", ["batched", "plain", "host"])
def test_row_hashing_lines(gpu, orc, f, log_rows, widths, form):
    mats = [F.random_matrix(f, log_rows, w, 80 + i) for i, w in enumerate(widths)]
    _check(gpu, orc, f, mats, plain=form == "plain", host=form == "host")


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("log_trace", [1, 6, 12, 13])
def test_fri_rounds_from_each_leaf_count(gpu, orc, f, log_trace):
    cw = orc.coset_lde(f, orc.random_matrix(f, log_trace, 4, 90), 1, F.lde_shift(f))
    want = orc.fri_commit_phase(f, cw, 1, 0)
    got = TwoAdicFriPcs(gpu, f, 1).fri_commit_phase(_dev(cw), challenger=new_challenger())
    assert (got.roots == want[0]).all() and (got.betas == want[1]).all() and (got.final_poly == want[2]).all()


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("observed", [0, 1, 7])
def test_challenger_with_pending_values(gpu, orc, f, observed):
    # the device challenger starts with values still in its buffer
    cw = orc.coset_lde(f, orc.random_matrix(f, 5, 4, 91), 1, F.lde_shift(f))
    values = F.to_monty(f, F.uniform(f, 7, 92))[:observed]
    oc, gc = orc.new_challenger(), new_challenger()
    for v in values:
        orc.challenger_observe(f, oc, int(v))
    import ctypes as C

    gpu.lib.pico_gpu_challenger_observe(f, C.byref(gc), values.ctypes.data_as(C.POINTER(C.c_uint32)), observed)
    want = orc.fri_commit_phase(f, cw, 1, 0, challenger=oc)
    got = TwoAdicFriPcs(gpu, f, 1).fri_commit_phase(_dev(cw), challenger=gc)
    assert (got.betas == want[1]).all() and (got.roots == want[0]).all()
    assert orc.challenger_sample(f, oc) == _sample(gpu, f, gc)


def _sample(gpu, f, ch):
    import ctypes as C

    out = C.c_uint32()
    assert gpu.lib.pico_gpu_challenger_sample(f, C.byref(ch), C.byref(out), 1) == 0
    return out.value
