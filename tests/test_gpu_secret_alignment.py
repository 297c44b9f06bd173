"""Secret-key cache rows built from packed keys at every byte alignment, and key generation into device
arrays at word and odd addresses, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_keys_at_every_alignment(cuda_ok, oracle, mode, shift):
    import torch

    import cudilithium_b200 as cd
    from cudilithium_b200 import _lib
    from cudilithium_b200.engine import Engine, pack_messages
    n = 5
    d = cd.Dilithium(mode)
    seeds = np.random.default_rng(shift).integers(0, 256, (n, 32), dtype=np.uint8)
    opk, osk = oracle.keypair_seeds(mode, seeds)
    pool, pitch = cd.alloc_pool(d.keypair_row_bytes(), n)
    pk = torch.zeros(n * d.params.pk_bytes + shift, dtype=torch.uint8, device="cuda")
    sk = torch.zeros(n * d.params.sk_bytes + shift, dtype=torch.uint8, device="cuda")
    d_seeds = torch.from_numpy(seeds.reshape(-1)).cuda()
    _lib.check(cd.lib.cudil_keypair_dev(mode, pk.data_ptr() + shift, sk.data_ptr() + shift, d_seeds.data_ptr(), pool.data_ptr(),
                                        pitch, n, None, 0), "keypair")
    torch.cuda.synchronize()
    assert np.array_equal(pk.cpu().numpy()[shift:].reshape(n, -1), opk)
    assert np.array_equal(sk.cpu().numpy()[shift:].reshape(n, -1), osk)
    m = np.random.default_rng(7).integers(0, 256, (n, 40), dtype=np.uint8)
    d_msgs, offs, lens = pack_messages(m)
    eng = Engine(mode, max_keys=n, max_items=n)
    eng.set_secret_keys(sk[shift:])
    sig = torch.zeros(n * d.params.sig_bytes, dtype=torch.uint8, device="cuda")
    eng.sign(sig, d_msgs, offs, lens, np.arange(n, dtype=np.uint32))
    torch.cuda.synchronize()
    eng.close()
    assert np.array_equal(sig.cpu().numpy().reshape(n, -1), oracle.sign_batch(mode, m, osk))
