"""Key-cache builds on both sides of the sizes where a build's kernels run beside or after one another: the
signatures and verification results of the keys at the build's ends (needs a B200)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _limit(mode, blocks_per_sm):
    """The most keys whose secret-row transforms take at most that many blocks (8 polynomials each) per SM."""
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return blocks_per_sm * sms * 8 // {2: 13, 3: 18, 5: 24}[mode]


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("blocks_per_sm", [4, 48])
@pytest.mark.parametrize("over", [0, 1])
def test_builds_at_the_limits(cuda_ok, oracle, mode, blocks_per_sm, over):
    import torch

    from cudilithium_b200.engine import Engine, pack_messages
    nk = _limit(mode, blocks_per_sm) + over
    pk, sk = oracle.keypair_batch(mode, nk, rand_index=600)
    idx = np.unique(np.concatenate([[0, 1, nk // 2, nk - 2, nk - 1], np.arange(3, nk, 97)])).astype(np.uint32)
    m = np.random.default_rng(nk).integers(0, 256, (len(idx), 32), dtype=np.uint8)
    want = oracle.sign_batch(mode, m, sk[idx])
    eng = Engine(mode, max_keys=nk, max_items=len(idx))
    d_sk, d_pk = torch.from_numpy(sk.reshape(-1)).cuda(), torch.from_numpy(pk.reshape(-1)).cuda()
    d_msgs, offs, lens = pack_messages(m)
    sig = torch.zeros(want.size, dtype=torch.uint8, device="cuda")
    ret = torch.full((len(idx),), 7, dtype=torch.int32, device="cuda")
    for _ in range(3):  # builds and batches in a row on one stream: each waits for the one before
        eng.set_secret_keys(d_sk)
        eng.sign(sig, d_msgs, offs, lens, idx)
        eng.set_public_keys(d_pk)
        eng.verify(ret, sig, d_msgs, offs, lens, idx)
    torch.cuda.synchronize()
    eng.last_status()
    assert np.array_equal(sig.cpu().numpy().reshape(len(idx), -1), want) and not bool(ret.any())
    eng.close()
