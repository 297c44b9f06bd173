"""Signing and verification batches on a stream that is being captured are refused: their metadata would be
read from the engine's staging buffer when the graph runs, after other calls have rewritten it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [2, 5])
@pytest.mark.parametrize("lens", ["equal", "mixed"])
def test_batches_on_a_capturing_stream_are_refused(cuda_ok, oracle, mode, lens):
    import torch

    from cudilithium_b200 import CudilError
    from cudilithium_b200.engine import Engine, pack_messages
    n = 40
    rng = np.random.default_rng(mode)
    pk, sk = oracle.keypair_batch(mode, 3, rand_index=4)
    mlens = np.full(n, 32) if lens == "equal" else rng.integers(0, 3000, n)
    m = rng.integers(0, 256, (n, 3000), dtype=np.uint8)
    idx = (np.arange(n) % 3).astype(np.uint32)
    want = oracle.sign_batch(mode, m, sk[idx], mlens=mlens.astype(np.uint32))
    d_msgs, offs, ml = pack_messages([m[i, :mlens[i]].tobytes() for i in range(n)])
    eng = Engine(mode, max_keys=3, max_items=n)
    eng.set_secret_keys(torch.from_numpy(sk.reshape(-1)).cuda())
    eng.set_public_keys(torch.from_numpy(pk.reshape(-1)).cuda())
    sig = torch.zeros(n * eng.params.sig_bytes, dtype=torch.uint8, device="cuda")
    ret = torch.full((n,), 7, dtype=torch.int32, device="cuda")
    x = torch.zeros(8, device="cuda")
    for _ in range(2):  # an engine without and with an earlier batch
        torch.cuda.synchronize()
        st, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st, capture_error_mode="relaxed"):
            x += 1
            with pytest.raises(CudilError):
                eng.sign(sig, d_msgs, offs, ml, idx, stream=st)
            with pytest.raises(CudilError):
                eng.verify(ret, sig, d_msgs, offs, ml, idx, stream=st)
        sig.zero_()
        before = float(x[0])
        graph.replay()
        torch.cuda.synchronize()
        assert float(x[0]) == before + 1 and not bool(sig.any())
        eng.sign(sig, d_msgs, offs, ml, idx)
        ret.fill_(7)
        eng.verify(ret, sig, d_msgs, offs, ml, idx)
        torch.cuda.synchronize()
        eng.last_status()
        assert np.array_equal(sig.cpu().numpy().reshape(n, -1), want) and not bool(ret.any())
    eng.close()
