"""Word-wise unpacking and 64-bit product sums against the oracle, at every byte alignment of the inputs.

The verifier reads z fields (18 or 20 bits) and t1 fields (10 bits) as aligned words around an array that
may start at any byte; the last key of a misaligned packed array takes byte loads, so that no word past the
array is read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_verify_at_every_alignment(cuda_ok, oracle, mode, shift):
    import torch

    from cudilithium_b200.engine import Engine, pack_messages
    n, nk = 9, 3
    pk, sk = oracle.keypair_batch(mode, nk, rand_index=900 + shift)
    m = np.random.default_rng(shift).integers(0, 256, (n, 45), dtype=np.uint8)
    idx = (np.arange(n) % nk).astype(np.uint32)
    sig = oracle.sign_batch(mode, m, sk[idx])
    sig[4, 40] ^= 1
    want = np.zeros(n, np.int32)
    want[4] = -1
    # packed keys and signatures `shift` bytes into exactly large enough buffers
    d_pk = torch.from_numpy(np.concatenate([np.zeros(shift, np.uint8), pk.reshape(-1)])).cuda()[shift:]
    d_sig = torch.from_numpy(np.concatenate([np.zeros(shift, np.uint8), sig.reshape(-1)])).cuda()[shift:]
    d_msgs, offs, lens = pack_messages(m)
    eng = Engine(mode, max_keys=nk, max_items=n)
    eng.set_public_keys(d_pk)
    d_ret = torch.full((n,), 7, dtype=torch.int32, device="cuda")
    eng.verify(d_ret, d_sig, d_msgs, offs, lens, idx)
    torch.cuda.synchronize()
    eng.close()
    assert np.array_equal(d_ret.cpu().numpy(), want)
