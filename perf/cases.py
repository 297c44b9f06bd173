"""Performance cases of the batched Dilithium framework.

A case is one call (or one short sequence of calls) that a program makes through the public entry
points: the fused engine (`Engine`, `EnginePipeline`), the drop-in API of the reference's shape
(`Dilithium.crypto_sign_*`), batched key generation and the NTT product.  `listed()` names the
cases, `draw(rng)` gives another one of the same ranges, `prepare(case, seed)` makes the inputs and
handles a program has in hand before the call, `run(state)` makes one pass and returns its outputs,
`work(case)` is the input and output traffic and the arithmetic the call cannot do without, and
`exact(case, seed)` the NTT product computed plainly in 64-bit integers.

Signatures, verification results and keys are bytes and whole numbers with one right value.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import cudilithium_b200 as cd
from cudilithium_b200 import _lib
from cudilithium_b200.engine import Engine, EnginePipeline

Q = 8380417


def listed():
    return [
        # one signature with a resident key: the latency of the smallest call (a signing service's
        # idle path)
        dict(name="sign_one_d2", op="sign", mode=2, n=1, keys=1, mlen_min=32, mlen_max=32, fresh=False, seeded=False),
        # the repository's headline batch: 10 000 short messages, one key per message, so the key
        # caches are built for the batch and the batch is signed
        dict(name="sign_batch_d2", op="sign", mode=2, n=10000, keys=10000, mlen_min=32, mlen_max=32, fresh=True, seeded=False),
        # a stream of such batches over two engines, as a bulk signer runs them
        dict(name="sign_stream_d2", op="stream", mode=2, n=10000, keys=10000, mlen_min=32, mlen_max=32, batches=4),
        # documents of 32 B to 64 KiB under a resident set of keys (the repository's log-uniform workload)
        dict(name="sign_varlen_d3", op="sign", mode=3, n=16384, keys=1024, mlen_min=32, mlen_max=65536, fresh=False, seeded=False),
        # a mid-size ragged request batch of the largest parameter set, randomized from a seed
        dict(name="sign_seeded_d5", op="sign", mode=5, n=1531, keys=97, mlen_min=1, mlen_max=4099, fresh=False, seeded=True),
        # the largest batch: bulk signing under resident keys
        dict(name="sign_large_d2", op="sign", mode=2, n=65536, keys=1024, mlen_min=32, mlen_max=32, fresh=False, seeded=False),
        # verification at scale with resident public keys, a tenth of the signatures damaged
        dict(name="verify_cached_d5", op="verify", mode=5, n=65536, keys=256, mlen_min=32, mlen_max=32, fresh=False, bad=0.1),
        # verification of a batch from as many signers: public-key caches built for the batch
        dict(name="verify_fresh_d2", op="verify", mode=2, n=10000, keys=10000, mlen_min=32, mlen_max=32, fresh=True, bad=0.02),
        # a small ragged verification request
        dict(name="verify_small_d3", op="verify", mode=3, n=33, keys=5, mlen_min=7, mlen_max=1021, fresh=False, bad=0.1),
        # batched key generation (device buffers), the reference's bench batch
        dict(name="keypair_d2", op="keypair", mode=2, n=10000),
        # the drop-in API on host buffers: sign, then verify, a batch of 1024
        dict(name="dropin_d3", op="dropin", mode=3, n=1024, mlen=59, threshold=4096),
        # the NTT product over a large array of polynomials (the repository's microbenchmark)
        dict(name="ntt_mul", op="ntt", npolys=1 << 20),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.499)))))))


# largest batch drawn per parameter set
_SIGN_CAP = {2: 49152, 3: 32768, 5: 24576}
_VERIFY_CAP = {2: 65536, 3: 65536, 5: 65536}
_KEYS_CAP = {2: 16384, 3: 12288, 5: 8192}


def draw(rng):
    op = rng.choice(["sign", "sign", "sign", "stream", "verify", "verify", "keypair", "dropin", "ntt"])
    if op == "ntt":
        return dict(op="ntt", npolys=_log_int(rng, 1, 1 << 20))
    mode = rng.choice([2, 3, 5])
    if op == "keypair":
        return dict(op="keypair", mode=mode, n=_log_int(rng, 1, _KEYS_CAP[mode]))
    if op == "dropin":
        n = _log_int(rng, 1, 4096)
        return dict(op="dropin", mode=mode, n=n, mlen=_log_int(rng, 1, 4096), threshold=max(64, rng.choice([1, 2, 4]) * n))
    if op == "stream":
        n = _log_int(rng, 64, 8192 if mode == 2 else 4096)
        lo = _log_int(rng, 1, 256)
        return dict(op="stream", mode=mode, n=n, keys=n, mlen_min=lo, mlen_max=lo + _log_int(rng, 1, 1024),
                    batches=rng.choice([2, 3, 4]))
    fresh = rng.random() < 0.3
    n = _log_int(rng, 1, _KEYS_CAP[mode] if fresh else (_SIGN_CAP if op == "sign" else _VERIFY_CAP)[mode])
    lo = _log_int(rng, 1, 4096)
    # the messages of a batch stay below 128 MiB
    hi = max(lo, min(_log_int(rng, 1, 65536), (128 << 20) // n))
    keys = n if fresh else min(n, _log_int(rng, 1, 1024))
    c = dict(op=op, mode=mode, n=n, keys=keys, mlen_min=min(lo, hi), mlen_max=hi, fresh=fresh)
    if op == "sign":
        c["seeded"] = rng.random() < 0.3
    else:
        c["bad"] = rng.choice([0.02, 0.1])
    return c


# ---------------------------------------------------------------------------- inputs


class State:
    """What a program holds between calls: handles, inputs and output buffers of a case."""


def _dev_bytes(gen, n):
    return torch.randint(0, 256, (max(int(n), 1),), dtype=torch.uint8, device="cuda", generator=gen)


def _keys(mode, n, gen):
    """n key pairs from random seeds, packed, on the device."""
    d = cd.Dilithium(mode)
    pool, pitch = cd.alloc_pool(d.keypair_row_bytes(), n)
    seeds = _dev_bytes(gen, n * 32)
    pk = torch.empty(n * d.params.pk_bytes, dtype=torch.uint8, device="cuda")
    sk = torch.empty(n * d.params.sk_bytes, dtype=torch.uint8, device="cuda")
    _lib.check(cd.lib.cudil_keypair_dev(mode, pk.data_ptr(), sk.data_ptr(), seeds.data_ptr(), pool.data_ptr(), pitch, n,
                                        None, 0), "keypair")
    torch.cuda.synchronize()
    return pk, sk


def _lengths(case, rng):
    """Message lengths, log-uniform between mlen_min and mlen_max."""
    lo, hi = case["mlen_min"], case["mlen_max"]
    if lo == hi:
        return np.full(case["n"], lo, np.uint32)
    v = np.exp(rng.uniform(math.log(lo), math.log(hi + 0.499), case["n"]))
    return np.clip(np.rint(v), lo, hi).astype(np.uint32)


def _messages(case, rng, gen):
    """Random messages in one device buffer at 8-byte aligned offsets: (buffer, offsets, lengths)."""
    lens = _lengths(case, rng)
    padded = (lens.astype(np.uint64) + np.uint64(7)) // np.uint64(8) * np.uint64(8)
    ends = np.cumsum(padded, dtype=np.uint64)
    return _dev_bytes(gen, int(ends[-1]) + 8), ends - padded, lens


def _key_index(case, rng):
    n, keys = case["n"], case["keys"]
    if keys == n:
        return np.arange(n, dtype=np.uint32)
    return rng.integers(0, keys, n).astype(np.uint32)


def prepare(case, seed):
    op = case["op"]
    rng = np.random.default_rng([int(seed), 7])
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed) * 1000003 + 17)
    s = State()
    s.case = case
    if op == "ntt":
        n = case["npolys"]
        s.a = torch.randint(-Q + 1, Q, (n, 256), dtype=torch.int32, device="cuda", generator=gen)
        s.b = torch.randint(-Q + 1, Q, (n, 256), dtype=torch.int32, device="cuda", generator=gen)
        s.out = torch.empty_like(s.a)
        return s
    mode, n = case["mode"], case["n"]
    d = cd.Dilithium(mode)
    pm = d.params
    s.d = d
    if op == "keypair":
        s.pool, s.pitch = cd.alloc_pool(d.keypair_row_bytes(), n)
        s.seeds = _dev_bytes(gen, n * 32)
        s.pk = torch.empty(n * pm.pk_bytes, dtype=torch.uint8, device="cuda")
        s.sk = torch.empty(n * pm.sk_bytes, dtype=torch.uint8, device="cuda")
        return s
    if op == "dropin":
        mlen, t = case["mlen"], case["threshold"]
        pk, sk = _keys(mode, n, gen)
        s.pk, s.sk, s.m = cd.pinned(pk.numel()), cd.pinned(sk.numel()), cd.pinned(n * mlen)
        s.pk.copy_(pk)
        s.sk.copy_(sk)
        s.m.copy_(_dev_bytes(gen, n * mlen))
        s.sig = cd.pinned(n * pm.sig_bytes)
        s.ret = torch.empty(n, dtype=torch.int32, pin_memory=True)
        s.spool, s.sp = cd.alloc_pool(d.sign_row_bytes(mlen), n)
        s.tpool, s.tp = cd.alloc_pool(d.sign_temp_row_bytes(), t)
        s.vpool, s.vp = cd.alloc_pool(d.verify_row_bytes(mlen), n)
        s.lut = cd.TaskLut(n, t)
        return s
    if op == "stream":
        s.pipe = EnginePipeline(mode, max_keys=n, max_items=n, depth=2)
        s.batches = []
        for _ in range(case["batches"]):
            _, sk = _keys(mode, n, gen)
            m, offs, lens = _messages(case, rng, gen)
            sig = torch.empty(n * pm.sig_bytes, dtype=torch.uint8, device="cuda")
            s.batches.append((sig, m, offs, lens, _key_index(case, rng), sk))
        return s
    # sign / verify through one engine
    s.pk, s.sk = _keys(mode, case["keys"], gen)
    s.m, s.offs, s.lens = _messages(case, rng, gen)
    s.kidx = _key_index(case, rng)
    s.sig = torch.empty(n * pm.sig_bytes, dtype=torch.uint8, device="cuda")
    s.engine = Engine(mode, max_keys=case["keys"], max_items=n)
    s.rho_seed = rng.integers(0, 256, 32, dtype=np.uint8).tobytes()
    if op == "sign":
        if not case["fresh"]:
            s.engine.set_secret_keys(s.sk)
        return s
    s.engine.set_secret_keys(s.sk)
    s.engine.sign(s.sig, s.m, s.offs, s.lens, s.kidx)
    torch.cuda.synchronize()
    bad = np.flatnonzero(rng.random(n) < case["bad"]).astype(np.int64)
    if len(bad):  # one bit of each damaged signature
        at = torch.from_numpy(bad * pm.sig_bytes + rng.integers(0, pm.sig_bytes, len(bad))).cuda()
        bit = torch.from_numpy((1 << rng.integers(0, 8, len(bad))).astype(np.uint8)).cuda()
        s.sig[at] ^= bit
    s.ret = torch.empty(n, dtype=torch.int32, device="cuda")
    if not case["fresh"]:
        s.engine.set_public_keys(s.pk)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------- one pass


def run(s):
    case = s.case
    op = case["op"]
    if op == "ntt":
        return cd.ntt_mul(s.a, s.b, out=s.out)
    if op == "keypair":
        _lib.check(cd.lib.cudil_keypair_dev(case["mode"], s.pk.data_ptr(), s.sk.data_ptr(), s.seeds.data_ptr(),
                                            s.pool.data_ptr(), s.pitch, case["n"], None, 0), "keypair")
        return {"pk": s.pk, "sk": s.sk}
    if op == "dropin":
        n, mlen, sb = case["n"], case["mlen"], s.d.CRYPTO_BYTES
        s.d.crypto_sign_signature(s.sig, sb, [0], s.m, mlen, mlen, s.sk, s.spool, s.sp, s.tpool, s.tp, s.lut,
                                  case["threshold"], n)
        s.d.crypto_sign_verify(s.ret, s.sig, sb, sb, s.m, mlen, mlen, s.pk, s.vpool, s.vp, n)
        return {"sig": s.sig, "ret": s.ret}
    if op == "stream":
        for sig, m, offs, lens, kidx, sk in s.batches:
            s.pipe.sign(sig, m, offs, lens, kidx, d_sk=sk)
        s.pipe.join()
        return [b[0] for b in s.batches]
    if op == "verify":
        if case["fresh"]:
            s.engine.set_public_keys(s.pk)
        s.engine.verify(s.ret, s.sig, s.m, s.offs, s.lens, s.kidx)
        return s.ret
    if case["fresh"]:
        s.engine.set_secret_keys(s.sk)
    if case["seeded"]:
        s.engine.sign(s.sig, s.m, s.offs, s.lens, s.kidx, rho_seed=s.rho_seed, rho_counter=0)
    else:
        s.engine.sign(s.sig, s.m, s.offs, s.lens, s.kidx)
    return s.sig


# ---------------------------------------------------------------------------- work


# 32-bit integer operations: one Keccak-f[1600] permutation (24 rounds of 180 three-input logic
# operations and funnel shifts), one transform of 256 coefficients (1024 butterflies of five), one
# modular product
_PERM, _NTT, _MUL = 24 * 180, 1024 * 5, 4
# attempts per signature (the reciprocal of the acceptance probability of the parameter set)
_ATTEMPTS = {2: 4.25, 3: 5.1, 5: 3.85}


def _absorb(nbytes):
    return nbytes // 136 + 1


def work(case):
    op = case["op"]
    if op == "ntt":
        n = case["npolys"]
        return {"bytes": 3 * 1024 * n, "flops": n * (2 * _NTT + 256 * _MUL)}
    pm = _lib.params(case["mode"])
    K, L, n = pm.k, pm.l, case["n"]
    expand_a = K * L * 5 * _PERM
    product = K * L * 256 * _MUL + K * _NTT
    if op == "keypair":
        ops = expand_a + (1 + (K + L) * 2 + _absorb(pm.pk_bytes)) * _PERM + L * _NTT + product
        return {"bytes": n * (32 + pm.pk_bytes + pm.sk_bytes), "flops": n * ops}
    w1 = K * pm.polyw1_packed
    # attempt: y, w = A y, challenge, and the products c s1, c s2 of a rejected attempt's first checks
    attempt = (L * 5 + _absorb(64 + w1) + 1) * _PERM + (L + 1 + 2) * _NTT + product
    final = (L + 2 * K) * (_NTT + 256 * _MUL)
    sk_ntt = (L + 2 * K) * _NTT
    ver = (_absorb(64 + w1) + 1) * _PERM + (L + 1) * _NTT + product + K * 256 * _MUL
    pk_build = expand_a + _absorb(pm.pk_bytes) * _PERM + K * _NTT
    if op == "dropin":
        mu = _absorb(32 + case["mlen"]) * _PERM
        ops = 2 * mu + _PERM + expand_a + sk_ntt + _ATTEMPTS[case["mode"]] * attempt + final + pk_build + ver
        return {"bytes": n * (2 * case["mlen"] + pm.sk_bytes + pm.pk_bytes + 2 * pm.sig_bytes + 4), "flops": n * ops}
    lo, hi = case["mlen_min"], case["mlen_max"]
    mean = lo if lo == hi else (hi - lo) / math.log(hi / lo)
    mu = (mean / 136 + 1) * _PERM
    batches = case.get("batches", 1)
    fresh = case.get("fresh", op == "stream")
    if op == "verify":
        ops = n * (mu + ver) + (case["keys"] * pk_build if fresh else 0)
        key_bytes = case["keys"] * (pm.pk_bytes if fresh else 32 + (K * L + K) * 1024)
        return {"bytes": int(n * (mean + pm.sig_bytes + 4) + key_bytes), "flops": int(ops)}
    ops = n * (mu + _PERM + _ATTEMPTS[case["mode"]] * attempt + final)
    ops += case["keys"] * (expand_a + sk_ntt) if fresh else 0
    key_bytes = case["keys"] * (pm.sk_bytes if fresh else 96 + (K * L + L + 2 * K) * 1024)
    return {"bytes": int(batches * (n * (mean + pm.sig_bytes) + key_bytes)), "flops": int(batches * ops)}


# ---------------------------------------------------------------------------- exact values


def _centred(v):
    v %= Q
    return v - Q if v > (Q - 1) // 2 else v


def _signed32(v):
    return ((v + (1 << 31)) & 0xFFFFFFFF) - (1 << 31)


def _montmul(a, b):
    """a * b * 2^-32 mod q in (-q, q), on int64 tensors (the representative the scheme's Montgomery
    reduction gives)."""
    p = a * b
    t = _signed32(_signed32(p) * 58728449)
    return (p - t * Q) >> 32


def exact(case, seed):
    """The NTT product in 64-bit integers: the scheme's butterfly network with Montgomery products
    (twiddles 2^32 * 1753^brv8(i) mod q, final factor 41978).  Keys, signatures and verification
    results are bytes and whole numbers, compared as they are."""
    if case["op"] != "ntt" or case["npolys"] > 1 << 20:
        return None
    zetas = [0] + [_centred((1 << 32) * pow(1753, int(f"{i:08b}"[::-1], 2), Q)) for i in range(1, 256)]
    s = prepare(case, seed)
    dev = s.a.device
    z = torch.tensor(zetas, dtype=torch.int64, device=dev)
    out = torch.empty_like(s.a)
    step = 1 << 15
    for p0 in range(0, case["npolys"], step):
        x = s.a[p0:p0 + step].to(torch.int64)
        n = x.shape[0]
        length, k = 128, 1
        while length >= 1:
            v = x.view(n, 128 // length, 2, length)
            w = z[k:k + 128 // length].view(1, -1, 1)
            t = _montmul(v[:, :, 1], w.expand_as(v[:, :, 1]))
            v[:, :, 1] = v[:, :, 0] - t
            v[:, :, 0] += t
            k += 128 // length
            length //= 2
        x = _montmul(x, s.b[p0:p0 + step].to(torch.int64))
        length, k = 1, 255
        while length <= 128:
            v = x.view(n, 128 // length, 2, length)
            blocks = 128 // length
            w = -z[k - blocks + 1:k + 1].flip(0).view(1, -1, 1)
            a, b = v[:, :, 0].clone(), v[:, :, 1].clone()
            v[:, :, 0] = a + b
            v[:, :, 1] = _montmul(a - b, w.expand_as(b))
            k -= blocks
            length *= 2
        out[p0:p0 + step] = _montmul(x, torch.full_like(x, 41978)).to(torch.int32)
    return out
