"""Device memory of an engine, which an admission budget is compared with, and verification batches larger
than the scratch holds packed w1' for (needs a B200)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one cached key pair and no items: the two cache rows, and at most 480 bytes of queue block
KEY_BYTES = {2: 50144, 3: 85984, 5: 147424}
# mu and rho' (128), four words of winner state (16), the metadata of an item (20)
ITEM_BYTES = 164
TURN = 1 << 18  # signatures of one turn of the verifier (kVerifyTurn)


@pytest.mark.parametrize("mode", [2, 3, 5])
def test_engine_bytes_per_key_and_item(cuda_ok, mode):
    from cudilithium_b200.engine import Engine
    eng = Engine(mode, max_keys=1, max_items=0, budget_bytes=KEY_BYTES[mode])
    assert eng.device_bytes <= KEY_BYTES[mode]
    eng.close()
    sizes = []
    for items in (1, 1_000_000, 4_000_000):
        eng = Engine(mode, max_keys=0, max_items=items)
        sizes.append(eng.device_bytes)
        eng.close()
    assert sizes[1] - sizes[0] <= 999_999 * ITEM_BYTES
    assert sizes[2] - sizes[1] <= 3_000_000 * ITEM_BYTES
    eng = Engine(mode, max_keys=0, max_items=4_000_000, budget_bytes=sizes[0] + 3_999_999 * ITEM_BYTES)
    eng.close()


@pytest.mark.parametrize("mode", [2, 5])
@pytest.mark.parametrize("n", [TURN, TURN + 1, 2 * TURN + 37])
def test_verify_in_turns(cuda_ok, oracle, mode, n):
    """61 signatures over and over; one of each damaged copy's 61 rejected, at both sides of a turn's end too."""
    import torch

    from cudilithium_b200.engine import Engine
    nk, ns = 3, 61
    pk, sk = oracle.keypair_batch(mode, nk, rand_index=17)
    m = np.random.default_rng(mode).integers(0, 256, (ns, 24), dtype=np.uint8)
    key = (np.arange(ns) % nk).astype(np.uint32)
    sig = torch.from_numpy(oracle.sign_batch(mode, m, sk[key])).cuda()
    at = np.arange(n) % ns
    d_sig = sig[torch.from_numpy(at).cuda()].contiguous()
    bad = np.unique(np.concatenate([np.arange(5, n, 1009), [0, TURN - 1, min(TURN, n - 1), n - 1]]))
    d_sig[torch.from_numpy(bad).cuda(), 40] ^= 4
    want = np.zeros(n, np.int32)
    want[bad] = -1
    eng = Engine(mode, max_keys=nk, max_items=n)
    eng.set_public_keys(torch.from_numpy(pk.reshape(-1)).cuda())
    ret = torch.full((n,), 9, dtype=torch.int32, device="cuda")
    eng.verify(ret, d_sig.reshape(-1), torch.from_numpy(m.reshape(-1)).cuda(), at * 24, np.full(n, 24), key[at])
    torch.cuda.synchronize()
    assert np.array_equal(ret.cpu().numpy(), want)
    eng.close()
