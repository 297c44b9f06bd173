"""The phased persistent kernel after the staged rounds: it finishes the items that the enqueued rounds
left (needs a B200).

The host enqueues as many rounds as usual keys' acceptance rate calls for, so batches of such keys hardly
ever leave an item.  Here nonce limits and keys with a low acceptance rate do."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FILL = 0xA5
EXHAUSTED = 0xFFFFFFFE


def _sign(eng, batch, n):
    """Signs into rows filled with FILL: (rows, status, error bits)."""
    import torch

    from cudilithium_b200._lib import lib
    d_msgs, offs, lens, idx = batch
    sig = torch.full((n * eng.params.sig_bytes,), FILL, dtype=torch.uint8, device="cuda")
    eng.sign(sig, d_msgs, offs, lens, idx)
    torch.cuda.synchronize()
    a, e = ctypes.c_ulonglong(), ctypes.c_uint32()
    rc = lib.cudil_engine_last_status(eng.h, ctypes.byref(a), ctypes.byref(e))
    return sig.cpu().numpy().reshape(n, -1), rc, e.value


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("n", [1, 32, 293])
def test_items_out_of_nonces_end_the_kernel(cuda_ok, oracle, mode, threads, n):
    """One round, deeper than the nonce limit, is all that is enqueued: every item it leaves reaches the
    persistent kernel without a nonce to try, and the first claim of a block takes its pending count to
    zero.  The block has to leave as a whole, with those items marked, and the next batch is signed."""
    import torch

    from cudilithium_b200._lib import CUDIL_ERR_TIMEOUT, CUDIL_OK
    from cudilithium_b200.engine import Engine, pack_messages
    pk, sk = oracle.keypair_batch(mode, 5, rand_index=81)
    m = np.random.default_rng(810 + mode).integers(0, 256, (n, 48), dtype=np.uint8)
    idx = (np.arange(n) % 5).astype(np.uint32)
    want, att = oracle.sign_batch(mode, m, sk[idx], return_attempts=True)
    batch = (*pack_messages(m), idx)
    eng = Engine(mode, max_keys=5, max_items=n, threads=threads, spec_slots=64)
    eng.set_secret_keys(torch.from_numpy(sk.reshape(-1)).cuda())
    for limit in (1, 2):
        ok = att <= limit
        eng.set_limits(nonce_limit=limit)
        rows, rc, err = _sign(eng, batch, n)
        nonces = eng.last_nonces(n)
        assert (rc, err) == ((CUDIL_OK, 0) if ok.all() else (CUDIL_ERR_TIMEOUT, 2))
        assert np.array_equal(nonces[ok] + 1, att[ok]) and np.all(nonces[~ok] == EXHAUSTED)
        assert np.array_equal(rows[ok], want[ok]) and np.all(rows[~ok] == FILL)
    eng.set_limits()
    rows, rc, err = _sign(eng, batch, n)
    assert (rc, err) == (CUDIL_OK, 0) and np.array_equal(rows, want)
    eng.close()


def _hard_keys(oracle, mode, nk, seed):
    """Valid encodings of secret keys whose t0 coefficients are all large: most attempts carry more hints
    than omega allows, so an item takes around 60 to 100 of them."""
    p = oracle.params(mode)
    low, eta_bytes = {2: (3000, 96), 3: (4000, 128), 5: (3300, 96)}[mode]
    _, sk = oracle.keypair_batch(mode, nk, rand_index=seed)
    rng = np.random.default_rng(seed)
    t0 = rng.integers(low, 4096, (nk, p.k * 256)) * rng.choice([-1, 1], (nk, p.k * 256))
    bits = ((4096 - t0)[:, :, None] >> np.arange(13)) & 1
    sk = sk.copy()
    sk[:, 96 + (p.k + p.l) * eta_bytes:] = np.packbits(bits.astype(np.uint8).reshape(nk, -1), axis=1, bitorder="little")
    return sk


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("threads", [128, 256])
@pytest.mark.parametrize("n,spec", [(1, 1), (45, 128), (300, 1), (600, 16)])
def test_items_left_by_the_rounds_are_signed(cuda_ok, oracle, mode, threads, n, spec):
    """The enqueued rounds end with items still pending; the persistent kernel goes on from their next nonce."""
    import torch

    from cudilithium_b200._lib import CUDIL_OK
    from cudilithium_b200.engine import Engine, pack_messages
    sk = _hard_keys(oracle, mode, 7, 9)
    m = np.random.default_rng(n + mode).integers(0, 256, (n, 40), dtype=np.uint8)
    idx = (np.arange(n) % 7).astype(np.uint32)
    want, att = oracle.sign_batch(mode, m, sk[idx], return_attempts=True)
    eng = Engine(mode, max_keys=7, max_items=n, threads=threads, spec_slots=spec)
    eng.set_secret_keys(torch.from_numpy(sk.reshape(-1)).cuda())
    rows, rc, err = _sign(eng, (*pack_messages(m), idx), n)
    assert (rc, err) == (CUDIL_OK, 0)
    assert np.array_equal(rows, want)
    assert np.array_equal(eng.last_nonces(n) + 1, att)
    # (only the persistent kernel counts cycles, and only where it found something pending)
    assert n == 1 or eng.last_phases()["total"] > 0
    eng.close()


@pytest.mark.parametrize("mode,n,longest", [(2, 1500, 30000), (5, 700, 30000)])
def test_items_left_by_both_parts_are_signed(cuda_ok, oracle, mode, n, longest):
    """The same for mixed lengths, signed in two parts where the length model says so."""
    import torch

    from cudilithium_b200._lib import CUDIL_OK
    from cudilithium_b200.engine import Engine, pack_messages
    rng = np.random.default_rng(mode)
    sk = _hard_keys(oracle, mode, 5, 10)
    lens = np.exp(rng.uniform(0, np.log(longest), n)).astype(np.uint32)
    lens[[3, 400]] = longest, 0
    m = rng.integers(0, 256, (n, longest), dtype=np.uint8)
    idx = rng.integers(0, 5, n).astype(np.uint32)
    want, att = oracle.sign_batch(mode, m, sk[idx], mlens=lens, return_attempts=True)
    eng = Engine(mode, max_keys=5, max_items=n)
    eng.set_secret_keys(torch.from_numpy(sk.reshape(-1)).cuda())
    rows, rc, err = _sign(eng, (*pack_messages([m[i, :lens[i]].tobytes() for i in range(n)]), idx), n)
    assert (rc, err) == (CUDIL_OK, 0)
    assert np.array_equal(rows, want) and np.array_equal(eng.last_nonces(n) + 1, att)
    assert eng.last_phases()["total"] > 0
    eng.close()


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("threads", [128, 256])
def test_phased_kernel_signs_whole_batches(cuda_ok, oracle, mode, threads):
    """With a lock bound below the default the phased kernel signs the batch alone, from its first nonce:
    ordinary keys with uneven lengths, and keys that take many attempts."""
    import torch

    from cudilithium_b200._lib import CUDIL_OK
    from cudilithium_b200.engine import Engine, pack_messages
    n = 150
    rng = np.random.default_rng(mode + threads)
    sk = np.concatenate([oracle.keypair_batch(mode, 4, rand_index=90)[1], _hard_keys(oracle, mode, 2, 11)])
    lens = rng.integers(0, 300, n).astype(np.uint32)
    lens[:6] = [0, 1, 135, 136, 137, 8]
    m = rng.integers(0, 256, (n, 300), dtype=np.uint8)
    idx = (np.arange(n) % 6).astype(np.uint32)
    want, att = oracle.sign_batch(mode, m, sk[idx], mlens=lens, return_attempts=True)
    batch = (*pack_messages([m[i, :lens[i]].tobytes() for i in range(n)]), idx)
    eng = Engine(mode, max_keys=6, max_items=n, threads=threads)
    eng.set_secret_keys(torch.from_numpy(sk.reshape(-1)).cuda())
    eng.set_limits(lock_spins=(1 << 22) - 1)
    for spec in (1, 16, 2 * threads):
        eng.set_spec_slots(spec)
        rows, rc, err = _sign(eng, batch, n)
        assert (rc, err) == (CUDIL_OK, 0)
        assert np.array_equal(rows, want) and np.array_equal(eng.last_nonces(n) + 1, att)
        assert eng.last_phases()["total"] > 0
    eng.close()


def test_bounds_checked_build_finds_nothing(cuda_ok):
    """The tests above in the bounds-checked build: the same results and a clean error word."""
    import os
    import subprocess
    import sys
    from pathlib import Path
    root = Path(__file__).resolve().parents[1]
    lib = root / "cudilithium_b200" / "libcudilithium_b200_bc.so"
    if not lib.exists():
        subprocess.run([sys.executable, str(root / "cudilithium_b200" / "build.py"), "--bounds-check"], check=True)
    run = ("import ctypes, sys, pytest\n"
           f"rc = pytest.main(['-x', '-q', '-p', 'no:cacheprovider', '-k', 'not bounds_checked', {str(Path(__file__))!r}])\n"
           "from cudilithium_b200._lib import LIB_PATH, lib\n"
           "err = ctypes.c_uint32(0xFFFFFFFF)\n"
           "assert lib.cudil_bounds_check_status(ctypes.byref(err), 1) == 0\n"
           "print('tests', int(rc), LIB_PATH.name, 'error word', err.value)\n")
    r = subprocess.run([sys.executable, "-c", run], cwd=root, env=dict(os.environ, CUDIL_LIB=str(lib)), capture_output=True,
                       text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-3000:]
    assert r.stdout.strip().splitlines()[-1] == f"tests 0 {lib.name} error word 0", r.stdout[-2000:]
