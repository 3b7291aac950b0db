"""Waits of the tensor-core Poseidon2 kernels that run out (an arrival that
nothing makes, pico_gpu_test_expire_tensor_waits): the kernels give up after a
bounded number of tries, the call reports it instead of returning void results,
and the context goes on working, the failure not charged to a later call.
"""
import numpy as np
import pytest

from pico_b200 import MerkleTreeMmcs, PicoError, Poseidon2, TwoAdicFriPcs, abi, new_challenger
from pico_b200 import fields as F

pytestmark = pytest.mark.gpu
FIELDS = [0, 1]
TRIES = 1 << 10  # the products themselves have long arrived by then
ROWS = 1 << 16


@pytest.fixture
def expired(gpu):
    def switch(on):
        abi.check(gpu.lib.pico_gpu_test_expire_tensor_waits(gpu.handle, TRIES if on else -1))

    yield switch
    switch(False)


def _dev(a):
    import torch

    return torch.from_numpy(a.view(np.int32)).cuda()


def _reported(call):
    with pytest.raises(PicoError) as e:
        call()
    assert e.value.status == abi.PICO_ERR_CUDA
    assert "ran out" in str(e.value)


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("form", ["batched", "host"])
def test_row_hashing(gpu, orc, expired, f, form):
    mats = [F.random_matrix(f, 16, w, 400 + w) for w in (9, 5)]
    want = orc.mmcs_commit(f, mats)
    given = mats if form == "host" else [_dev(m) for m in mats]
    m = MerkleTreeMmcs(gpu, f)
    reserved = gpu.memory()[0]
    expired(True)
    _reported(lambda: m.commit(given))
    expired(False)
    assert gpu.memory()[0] == reserved
    root, pd = m.commit(given)
    pd.release()
    assert (root == want).all()


@pytest.mark.parametrize("f", FIELDS)
def test_fri_commit_phase(gpu, orc, expired, f):
    cw = orc.coset_lde(f, orc.random_matrix(f, 17, 4, 50), 1, F.lde_shift(f))
    want = orc.fri_commit_phase(f, cw, 1, 0)
    pcs = TwoAdicFriPcs(gpu, f, 1)
    expired(True)
    _reported(lambda: pcs.fri_commit_phase(_dev(cw), challenger=new_challenger()))
    expired(False)
    got = pcs.fri_commit_phase(_dev(cw), challenger=new_challenger())
    assert (got.roots == want[0]).all() and (got.final_poly == want[2]).all()


@pytest.mark.parametrize("f", FIELDS)
@pytest.mark.parametrize("device", [True, False])
def test_permutation(gpu, orc, expired, f, device):
    st = F.to_monty(f, F.uniform(f, 16 * ROWS, 21)).reshape(ROWS, 16)
    want = orc.permute(f, st)
    p = Poseidon2(gpu, f)
    expired(True)
    _reported(lambda: p.permute(_dev(st) if device else st.copy()))
    expired(False)
    # the record is gone: an unrelated call is not charged with it
    m = F.random_matrix(f, 4, 3, 1)
    root, pd = MerkleTreeMmcs(gpu, f).commit([m])
    pd.release()
    assert (root == orc.mmcs_commit(f, [m])).all()
    d = _dev(st) if device else st.copy()
    p.permute(d)
    assert ((d.cpu().numpy().view(np.uint32) if device else d) == want).all()
