"""The phased persistent kernel after the staged rounds: it finishes the items that the enqueued rounds
left (needs a B200).

The host enqueues as many rounds as usual keys' acceptance rate calls for, so batches of such keys hardly
ever leave an item.  Here nonce limits do."""
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
