"""Where device key generation (cudil_keypair_dev) may write its keys: device memory at any byte, pinned host
memory, and no pageable host memory (needs a B200)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _keypair_dev(mode, n, seeds, pk_ptr, sk_ptr):
    import torch

    import cudilithium_b200 as cd
    pool, pitch = cd.alloc_pool(cd.Dilithium(mode).keypair_row_bytes(), n)
    d_seeds = torch.from_numpy(seeds.reshape(-1)).cuda()
    rc = cd.lib.cudil_keypair_dev(mode, pk_ptr, sk_ptr, d_seeds.data_ptr(), pool.data_ptr(), pitch, n, None, 0)
    torch.cuda.synchronize()
    return rc


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("n", [1, 37])
def test_device_and_pinned_outputs(cuda_ok, oracle, mode, n):
    import torch
    p = oracle.params(mode)
    seeds = np.random.default_rng(mode * 100 + n).integers(0, 256, (n, 32), dtype=np.uint8)
    want = oracle.keypair_seeds(mode, seeds)

    def buf(size, shift, pinned):
        b = torch.zeros(size + 8, dtype=torch.uint8, **({"pin_memory": True} if pinned else {"device": "cuda"}))
        return b[shift:shift + size]

    for pk_at, sk_at in ((0, False), (0, False)), ((0, True), (0, True)), ((0, False), (0, True)), ((0, True), (0, False)), \
            ((1, False), (0, False)), ((0, False), (2, False)), ((3, True), (1, True)):
        pk, sk = buf(n * p.pk_bytes, *pk_at), buf(n * p.sk_bytes, *sk_at)
        assert _keypair_dev(mode, n, seeds, pk.data_ptr(), sk.data_ptr()) == 0
        assert np.array_equal(pk.cpu().numpy().reshape(n, -1), want[0])
        assert np.array_equal(sk.cpu().numpy().reshape(n, -1), want[1])


@pytest.mark.parametrize("pageable", ["pk", "sk", "both"])
def test_pageable_outputs_are_refused(cuda_ok, oracle, pageable):
    """A kernel's write to memory that the device cannot access would end the context: the call returns an
    error before it queues anything, and the next one is right."""
    import torch
    mode, n = 2, 5
    p = oracle.params(mode)
    seeds = np.random.default_rng(3).integers(0, 256, (n, 32), dtype=np.uint8)
    host = {k: np.full(n * b, 0xA5, np.uint8) for k, b in (("pk", p.pk_bytes), ("sk", p.sk_bytes))}
    dev = {k: torch.zeros(v.size, dtype=torch.uint8, device="cuda") for k, v in host.items()}
    at = {k: host[k].ctypes.data if pageable in (k, "both") else dev[k].data_ptr() for k in host}
    assert _keypair_dev(mode, n, seeds, at["pk"], at["sk"]) != 0
    assert all(np.all(v == 0xA5) for v in host.values())
    assert not any(bool(v.any()) for v in dev.values())
    assert _keypair_dev(mode, n, seeds, dev["pk"].data_ptr(), dev["sk"].data_ptr()) == 0
    want = oracle.keypair_seeds(mode, seeds)
    assert np.array_equal(dev["pk"].cpu().numpy().reshape(n, -1), want[0])
    assert np.array_equal(dev["sk"].cpu().numpy().reshape(n, -1), want[1])
