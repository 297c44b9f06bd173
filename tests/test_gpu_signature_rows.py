"""Signature rows at every byte alignment, in device and in pinned host memory, from every signer kernel: the
rows' neighbours and the bytes around them stay as they are (needs a B200)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("kernel", ["staged", "phased", 1, 5])
def test_rows_at_every_byte(cuda_ok, oracle, mode, kernel):
    import torch

    from cudilithium_b200.engine import Engine, pack_messages
    n = 9
    pk, sk = oracle.keypair_batch(mode, 3, rand_index=21)
    m = np.random.default_rng(mode).integers(0, 256, (n, 20), dtype=np.uint8)
    idx = (np.arange(n) % 3).astype(np.uint32)
    want = oracle.sign_batch(mode, m, sk[idx]).reshape(-1)
    d_msgs, offs, lens = pack_messages(m)
    eng = Engine(mode, max_keys=3, max_items=n)
    eng.set_secret_keys(torch.from_numpy(sk.reshape(-1)).cuda())
    if kernel == "phased":
        eng.set_limits(lock_spins=(1 << 22) - 1)
    elif kernel != "staged":
        eng.set_sign_kernel(kernel)
    for place in ({"device": "cuda"}, {"pin_memory": True}):
        for shift in range(4):
            buf = torch.full((want.size + 16,), 0xA5, dtype=torch.uint8, **place)
            eng.sign(buf[8 + shift:], d_msgs, offs, lens, idx)
            torch.cuda.synchronize()
            eng.last_status()
            got = buf.cpu().numpy()
            assert np.array_equal(got[8 + shift:8 + shift + want.size], want)
            assert np.all(got[:8 + shift] == 0xA5) and np.all(got[8 + shift + want.size:] == 0xA5)
    eng.close()
