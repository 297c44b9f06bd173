"""The engine's longest-first order (csrc/length_order.cuh, host code) against numpy's stable sort: equal
lengths stay in item order."""
import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "cudilithium_b200" / "csrc"


@pytest.fixture(scope="module")
def order(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "o.cpp").write_text(f'#include "{CSRC / "length_order.cuh"}"\n'
                             'extern "C" void order(unsigned *o, unsigned *t, const unsigned *l, size_t n)\n'
                             '{ cudil::order_longest_first(o, t, l, n); }\n')
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-o", str(d / "o.so"), str(d / "o.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "o.so")).order

    def call(lens):
        out, tmp = np.full(len(lens) + 1, 0xFFFFFFFF, np.uint32), np.zeros(len(lens), np.uint32)
        fn(ctypes.c_void_p(out.ctypes.data), ctypes.c_void_p(tmp.ctypes.data), ctypes.c_void_p(lens.ctypes.data),
           ctypes.c_size_t(len(lens)))
        assert out[-1] == 0xFFFFFFFF
        return out[:-1]
    return call


@pytest.mark.parametrize("n", [1, 2, 63, 64, 65, 2048, 5001])
@pytest.mark.parametrize("longest", [0, 1, 2047, 2048, 65536, (1 << 22) - 1, 1 << 22, 0xFFFFFFFF])
def test_order_is_the_stable_descending_one(order, n, longest):
    rng = np.random.default_rng([n, longest])
    uniform = rng.integers(0, longest + 1, n).astype(np.uint32)
    logs = np.exp(rng.uniform(0, np.log(longest + 1.0), n)).clip(0, longest).astype(np.uint32)
    few = rng.choice(np.array([0, longest // 3, longest], np.uint32), n)
    for lens in (uniform, logs, few, np.sort(uniform), np.sort(uniform)[::-1].copy()):
        want = np.argsort(-lens.astype(np.int64), kind="stable")
        assert np.array_equal(order(lens), want)
