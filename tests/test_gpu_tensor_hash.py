"""The tensor-core Poseidon2 kernels (launches of at least 2^16 states) against
the oracle, where their tiling and sponge handling can go wrong: state counts
around the dispatch line and a tile of 128, row widths around the rate of 8
(partial chunks keep the other rate words), rows of several matrices, digests
injected at a tall level, and the resumable form of plain and host commits.
All values are field elements: every comparison is exact.
"""
import numpy as np
import pytest

from pico_b200 import MerkleTreeMmcs, Poseidon2, TwoAdicFriPcs, new_challenger
from pico_b200 import fields as F

pytestmark = pytest.mark.gpu
FIELDS = [0, 1]
LINE = 1 << 16  # states from which launches use the tensor cores


def _dev(a):
    import torch

    return torch.from_numpy(a.view(np.int32)).cuda()


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("n", [LINE - 1, LINE, LINE + 1, LINE + 129, 2 * 296 * 4 * 128 + 77])
def test_permute_state_counts(gpu, orc, f, n):
    st = F.to_monty(f, F.uniform(f, 16 * n, 21)).reshape(n, 16)
    st[0] = 0
    st[1] = F.P[f] - 1  # the largest canonical words
    d = _dev(st.copy())
    Poseidon2(gpu, f).permute(d)
    assert (d.cpu().numpy().view(np.uint32) == orc.permute(f, st)).all()


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("widths", [[1], [7], [8], [9], [16], [3, 6, 8], [17, 0, 2]])
@pytest.mark.parametrize("form", ["batched", "plain", "host"])
def test_row_widths(gpu, orc, f, widths, form):
    mats = [F.random_matrix(f, 16, w, 30 + i) if w else np.zeros((LINE, 0), np.uint32) for i, w in enumerate(widths)]
    want_root, want_layers = orc.mmcs_commit(f, mats, want_layers=True)
    given = mats if form == "host" else [_dev(m) if m.size else m for m in mats]
    if form != "host" and any(not m.size for m in mats):
        import torch

        given = [torch.empty((LINE, 0), dtype=torch.int32, device="cuda") if not m.size else g
                 for m, g in zip(mats, given)]
    root, pd = MerkleTreeMmcs(gpu, f).commit(given, plain=form == "plain")
    assert (root == want_root).all()
    assert (pd.digest_layer(0).ravel() == np.asarray(want_layers).ravel()[: 8 * LINE]).all()
    pd.release()


@pytest.mark.parametrize("f", FIELDS)
def test_injection_at_a_tall_level(gpu, orc, f):
    # 2^18 leaves; rows of 2^17 and 2^16 meet levels compressed on the tensor cores, 2^15 the quad form
    mats = [F.random_matrix(f, h, w, 40 + h) for h, w in ((18, 5), (17, 11), (16, 8), (15, 3))]
    want_root = orc.mmcs_commit(f, mats)
    root, pd = MerkleTreeMmcs(gpu, f).commit([_dev(m) for m in mats])
    pd.release()
    assert (root == want_root).all()


@pytest.mark.parametrize("f", FIELDS)
def test_fri_fold_and_hash(gpu, orc, f):
    # first rounds hash 2^17 and 2^16 leaves on the tensor cores, the next 2^15 one thread per leaf
    cw = orc.coset_lde(f, orc.random_matrix(f, 17, 4, 50), 1, F.lde_shift(f))
    want = orc.fri_commit_phase(f, cw, 1, 0)
    got = TwoAdicFriPcs(gpu, f, 1).fri_commit_phase(_dev(cw), challenger=new_challenger())
    assert (got.roots == want[0]).all() and (got.betas == want[1]).all() and (got.final_poly == want[2]).all()
