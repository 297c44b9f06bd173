"""Staged signer (rounds over the whole GPU) against the oracle: batch sizes at the edges of its grids,
speculation from none to the deepest, one and several rounds, nonce limits, and pinned host output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _inputs(oracle, mode, n, nk, seed):
    import torch

    from cudilithium_b200.engine import pack_messages
    pk, sk = oracle.keypair_batch(mode, nk, rand_index=seed)
    rng = np.random.default_rng(seed)
    m = rng.integers(0, 256, (n, 33), dtype=np.uint8)
    idx = rng.integers(0, nk, n).astype(np.uint32)
    want = oracle.sign_batch(mode, m, sk[idx])
    return torch.from_numpy(sk.reshape(-1)).cuda(), pack_messages(m), idx, want


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("n,spec", [(1, 1), (1, 16), (31, 2), (257, 1), (257, 512), (1185, 16), (2400, 4)])
def test_staged_matches_oracle(cuda_ok, oracle, mode, n, spec):
    import torch

    from cudilithium_b200.engine import Engine
    sk, (d_msgs, offs, lens), idx, want = _inputs(oracle, mode, n, min(n, 7), 40 + n)
    eng = Engine(mode, max_keys=7, max_items=n)
    eng.set_spec_slots(spec)
    eng.set_secret_keys(sk)
    d_sig = torch.zeros(n * eng.params.sig_bytes, dtype=torch.uint8, device="cuda")
    h_sig = torch.zeros(n * eng.params.sig_bytes, dtype=torch.uint8, pin_memory=True)
    for out in (d_sig, h_sig):
        eng.sign(out, d_msgs, offs, lens, idx)
        torch.cuda.synchronize()
        eng.last_status()
        assert np.array_equal(out.cpu().numpy().reshape(n, -1), want)
    eng.close()


def test_staged_nonce_limit_marks_the_rest(cuda_ok, oracle):
    """Three nonces an item: the items that accept one of them are signed, the others are marked."""
    import ctypes

    import torch

    from cudilithium_b200._lib import CUDIL_ERR_TIMEOUT, lib
    from cudilithium_b200.engine import Engine
    mode, n = 2, 900
    sk, (d_msgs, offs, lens), idx, want = _inputs(oracle, mode, n, 7, 77)
    for spec in (1, 64):
        eng = Engine(mode, max_keys=7, max_items=n)
        eng.set_spec_slots(spec)
        eng.set_limits(nonce_limit=3)
        eng.set_secret_keys(sk)
        d_sig = torch.zeros(n * eng.params.sig_bytes, dtype=torch.uint8, device="cuda")
        eng.sign(d_sig, d_msgs, offs, lens, idx)
        torch.cuda.synchronize()
        att, err = ctypes.c_ulonglong(), ctypes.c_uint32()
        assert lib.cudil_engine_last_status(eng.h, ctypes.byref(att), ctypes.byref(err)) == CUDIL_ERR_TIMEOUT
        assert err.value == 2 and att.value <= 3 * n
        nonces, rows = eng.last_nonces(n), d_sig.cpu().numpy().reshape(n, -1)
        out = nonces == 0xFFFFFFFE
        assert 0 < out.sum() < n and np.all(nonces[~out] < 3)
        assert np.array_equal(rows[~out], want[~out]) and not rows[out].any()
        eng.close()


@pytest.mark.parametrize("mode,n,longest", [(2, 2000, 40000), (5, 1200, 60000)])
def test_staged_mixed_lengths_in_two_parts(cuda_ok, oracle, mode, n, longest):
    """Lengths that make the batch sign in two parts (the longest messages hashed meanwhile)."""
    import torch

    from cudilithium_b200.engine import Engine, pack_messages
    rng = np.random.default_rng(mode)
    pk, sk = oracle.keypair_batch(mode, 5, rand_index=3)
    lens = np.exp(rng.uniform(np.log(1), np.log(longest), n)).astype(np.uint32)
    lens[[3, 700]] = longest, 0
    m = rng.integers(0, 256, (n, longest), dtype=np.uint8)
    idx = rng.integers(0, 5, n).astype(np.uint32)
    want = oracle.sign_batch(mode, m, sk[idx], mlens=lens)
    d_msgs, offs, plens = pack_messages([m[i, :lens[i]].tobytes() for i in range(n)])
    assert np.array_equal(plens, lens)
    eng = Engine(mode, max_keys=5, max_items=n)
    eng.set_secret_keys(torch.from_numpy(sk.reshape(-1)).cuda())
    sig = torch.zeros(n * eng.params.sig_bytes, dtype=torch.uint8, device="cuda")
    eng.sign(sig, d_msgs, offs, lens, idx)
    torch.cuda.synchronize()
    eng.last_status()
    assert np.array_equal(sig.cpu().numpy().reshape(n, -1), want)
    eng.close()


@pytest.mark.parametrize("n", [9471, 9472, 9473])
def test_hash_pairs_and_threads_agree(cuda_ok, oracle, n):
    """Around the item count where one hash state per thread pair becomes one per thread (148 SMs: 9472)."""
    import cudilithium_b200 as cd
    d = cd.Dilithium(2)
    pk, sk = d.keypair(n, rand_index=5)
    opk, osk = oracle.keypair_batch(2, n, rand_index=5)
    assert np.array_equal(pk, opk) and np.array_equal(sk, osk)
    m = np.random.default_rng(n).integers(0, 256, (n, 200), dtype=np.uint8)
    sig = d.sign(m, sk, exec_threshold=n)
    assert np.array_equal(sig, oracle.sign_batch(2, m, sk))
    bad = sig.copy()
    bad[::7, 5] ^= 1
    assert np.array_equal(d.verify(bad, m, pk), np.where(np.arange(n) % 7 == 0, -1, 0))
