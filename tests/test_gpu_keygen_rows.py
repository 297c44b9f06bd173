"""Key generation at the edges of its row blocks (128 / L rows (key, i) per block) against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [2, 3, 5])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 9, 25, 65])
def test_keypair_row_block_edges(cuda_ok, oracle, mode, n):
    import cudilithium_b200 as cd
    seeds = np.random.default_rng(n).integers(0, 256, (n, 32), dtype=np.uint8)
    pk, sk = cd.Dilithium(mode).keypair(n, seeds=seeds)
    opk, osk = oracle.keypair_seeds(mode, seeds)
    assert np.array_equal(pk, opk) and np.array_equal(sk, osk)
