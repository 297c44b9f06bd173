"""The engine's verification kernels against the oracle: batch sizes at the edges of their grids (one warp
or four per block, one hash state per thread or per pair), and each kind of rejection."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("n", [1, 33, 1184, 1185, 9473])
def test_verify_matches_oracle(cuda_ok, oracle, mode, n):
    import torch

    from cudilithium_b200 import _lib
    from cudilithium_b200.engine import Engine, pack_messages
    p = _lib.params(mode)
    nk, base = 5, 60
    rng = np.random.default_rng(n)
    pk, sk = oracle.keypair_batch(mode, nk, rand_index=n)
    kb = (np.arange(base) % nk).astype(np.uint32)
    mb = rng.integers(0, 256, (base, 75), dtype=np.uint8)
    sb = oracle.sign_batch(mode, mb, sk[kb])
    pick = rng.integers(0, base, n)
    idx, m, sig = kb[pick], mb[pick], sb[pick].copy()
    # a damaged c~, z, hint position, hint count, padding byte, or message; every seventh row is intact
    zlen = p.l * p.polyz_packed
    for i in range(n):
        kind = i % 7
        if kind == 0:
            sig[i, rng.integers(0, 32)] ^= 1 << rng.integers(0, 8)
        elif kind == 1:
            sig[i, 32 + rng.integers(0, zlen)] ^= 1 << rng.integers(0, 8)
        elif kind == 2:
            sig[i, 32 + zlen + rng.integers(0, 20)] ^= 1 << rng.integers(0, 8)
        elif kind == 3:
            sig[i, 32 + zlen + p.omega + rng.integers(0, p.k)] ^= 1 << rng.integers(0, 8)
        elif kind == 4:
            sig[i, 32 + zlen + p.omega - 1] ^= 1
        elif kind == 5:
            m = m.copy() if i == 5 else m
            m[i, 3] ^= 4
    want = oracle.verify_batch(mode, sig, m, pk[idx])
    d_msgs, offs, lens = pack_messages(m)
    eng = Engine(mode, max_keys=nk, max_items=n)
    eng.set_public_keys(torch.from_numpy(pk.reshape(-1)).cuda())
    d_ret = torch.full((n,), 9, dtype=torch.int32, device="cuda")
    eng.verify(d_ret, torch.from_numpy(sig.reshape(-1)).cuda(), d_msgs, offs, lens, idx)
    torch.cuda.synchronize()
    eng.close()
    assert np.array_equal(d_ret.cpu().numpy(), want)
    if n > 7:
        assert (want == 0).any() and (want == -1).any()


def test_verify_keeps_the_last_signing_nonces(cuda_ok, oracle):
    """last_nonces reports the last signing batch also after a verification on the same engine."""
    import torch

    from cudilithium_b200.engine import Engine, pack_messages
    n = 50
    pk, sk = oracle.keypair_batch(2, 3, rand_index=8)
    m = np.random.default_rng(1).integers(0, 256, (n, 20), dtype=np.uint8)
    idx = (np.arange(n) % 3).astype(np.uint32)
    want, att = oracle.sign_batch(2, m, sk[idx], return_attempts=True)
    d_msgs, offs, lens = pack_messages(m)
    eng = Engine(2, max_keys=3, max_items=n)
    eng.set_secret_keys(torch.from_numpy(sk.reshape(-1)).cuda())
    eng.set_public_keys(torch.from_numpy(pk.reshape(-1)).cuda())
    sig = torch.zeros(n * eng.params.sig_bytes, dtype=torch.uint8, device="cuda")
    ret = torch.full((n,), 5, dtype=torch.int32, device="cuda")
    eng.sign(sig, d_msgs, offs, lens, idx)
    eng.verify(ret, sig, d_msgs, offs, lens, idx)
    torch.cuda.synchronize()
    assert np.array_equal(sig.cpu().numpy().reshape(n, -1), want) and not ret.cpu().numpy().any()
    assert np.array_equal(eng.last_nonces(n).astype(np.int64) + 1, np.asarray(att, np.int64))
    eng.sign(sig, d_msgs, offs, lens, idx)  # and the next signing batch is unaffected
    torch.cuda.synchronize()
    assert np.array_equal(sig.cpu().numpy().reshape(n, -1), want)
    eng.close()
