#!/usr/bin/env python3
"""Benchmark of the batched Dilithium path on B200 (one JSON line on rank 0).

Headline workload: Dilithium2 batched signing of 10000 32-byte messages, one key per message (the
reference's bench_dilithium batch, benches/bench_dilithium.cu:277-296), keys from the reference's
seed scheme SHAKE128(le64(2i+1)).  A step = the fused engine building the batch's key caches and
signing the batch in one call (then verifying it against freshly built public-key caches).

  value         Dilithium2 signatures/s of the fused engine, inputs resident in HBM
  plain         the same batch through the plain stage-by-stage path (cudil_sign_dev /
                cudil_verify_dev, best exec threshold of --thresholds); fused_over_plain = ratio
  e2e           fused signing with pinned host inputs/outputs, batches streamed: two engines
                alternate so the H2D of m and sk for batch k+1 overlaps the signing of batch k;
                signatures written by the signer into pinned host memory; all copies inside the
                timed region (the one-batch-at-a-time figure is reported beside it)
  verify_per_s  verifications/s of the same step (fused engine, public-key caches built per step)
  roofline      the signing batch: algorithmic 32-bit ALU operations (work model below,
                attempts counted on the device) over its CUDA-event duration, against the measured
                LOP3/SHF issue peak of this GPU
  configs       configs 1-4 of the workload list (batch-1024 latency, NTT microbench vs HBM peak,
                Dilithium3 log-uniform messages, Dilithium5 cached-key verification with 10% bit flips)
  cpu_baseline  the CPU oracle (C restatement, OpenMP over all host cores) on a bounded sample

--impl reference runs the CPU implementation of the same path (the oracle; the reference ships no
CPU Dilithium) on the host cores and prints the same metric.
"""
from __future__ import annotations

import argparse
import contextlib
import json
import math
import os
import statistics
import subprocess
import sys
import threading
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "Dilithium2 sign/s (batched, bit-exact) on 1 B200"
UNIT = "signatures/s"
MLEN = 32

# Algorithmic work model (32-bit ALU operations).  One Keccak-f[1600] permutation lowered to
# 3-input LOP3 and funnel shifts: per round theta 20 (parity) + 20 (D) + 50 (apply), rho 48,
# chi 50, iota 2 = 190; 24 rounds.
OPS_PERM = 24 * 190
OPS_NTT_FWD = 1024 * 6          # 1024 butterflies: 3 IMAD + 3 IADD
OPS_NTT_INV = 1024 * 6 + 256 * 4  # + the final multiplication by f
OPS_PW = 5                        # one Montgomery pointwise product


def log(*a):
    print(*a, file=sys.stderr, flush=True)


# ---------------------------------------------------------------------------- ranks
# Items are independent, so N GPUs run N replicas over disjoint inputs (no data-path collective).
def rank_shard(rank: int, batch: int) -> tuple[int, int]:
    """(key rand_index, message seed) of a rank: keys 2*batch*rank .. of the reference seed scheme
    (the keypair kernel uses rand_index + 2i + 1, so ranks never share a key) and its own message
    stream."""
    return rank * 2 * batch, 1234 + rank


def reduce_max(vals, world: int, device):
    """Element-wise max over ranks of per-rank timings (the job's time is its slowest rank)."""
    if world == 1:
        return tuple(vals)
    import torch
    import torch.distributed as dist
    t = torch.tensor(list(vals), dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return tuple(t.tolist())


# ---------------------------------------------------------------------------- clocks
class ClockSampler:
    """SM clocks and clock-event reasons while the timed region runs (read-only queries).

    Two records: `nvidia-smi -lms 200` over the whole measurement, and an NVML poll every
    5 ms whose samples count only inside the windows marked with `window()` (the host-side
    span from the first timed launch to the synchronize after the last).  The reported median
    and reasons come from the in-window NVML samples when there are any, else from nvidia-smi.
    """
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    NAMES = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
    POLL_S = 0.005

    def __init__(self, index: int, pci_bus_id: str | None = None):
        self.index = index  # CUDA ordinal; the PCI bus id, when given, picks the same GPU in NVML
        self.pci_bus_id = pci_bus_id
        self.proc = None
        self.lines: list[str] = []
        self.polled: list[tuple[float, float, int]] = []  # (perf_counter, SM MHz, reason bits)
        self.windows: list[tuple[float, float]] = []
        self.nvml = None
        self.max_mhz = None
        self.done = threading.Event()

    def start(self):
        smi_id = self.index
        try:
            import pynvml
            pynvml.nvmlInit()
            h = None
            if self.pci_bus_id:
                try:
                    h = pynvml.nvmlDeviceGetHandleByPciBusId(self.pci_bus_id)
                except Exception:
                    h = None
            if h is None:
                h = pynvml.nvmlDeviceGetHandleByIndex(self.index)
            smi_id = int(pynvml.nvmlDeviceGetIndex(h))
            self.max_mhz = float(pynvml.nvmlDeviceGetMaxClockInfo(h, pynvml.NVML_CLOCK_SM))
            self.nvml = (pynvml, h)
            self.bits = {"hw_slowdown": pynvml.nvmlClocksEventReasonHwSlowdown,
                         "hw_thermal_slowdown": pynvml.nvmlClocksEventReasonHwThermalSlowdown,
                         "sw_thermal_slowdown": pynvml.nvmlClocksEventReasonSwThermalSlowdown,
                         "sw_power_cap": pynvml.nvmlClocksEventReasonSwPowerCap}
            self.poller = threading.Thread(target=self._poll, daemon=True)
            self.poller.start()
        except Exception:  # no NVML: the nvidia-smi record stands alone
            self.nvml = None
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={smi_id}", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            threading.Thread(target=self._read, daemon=True).start()
        except OSError:
            self.proc = None
        # the first nvidia-smi line shows the sampler is up before anything is timed
        t_end = time.perf_counter() + 3.0
        while self.proc is not None and not self.lines and time.perf_counter() < t_end:
            time.sleep(0.02)

    def _read(self):
        for ln in self.proc.stdout:
            self.lines.append(ln.strip())

    def _poll(self):
        nv, h = self.nvml
        while not self.done.is_set():
            try:
                mhz = float(nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM))
                bits = int(nv.nvmlDeviceGetCurrentClocksEventReasons(h))
            except Exception:
                break
            self.polled.append((time.perf_counter(), mhz, bits))
            time.sleep(self.POLL_S)

    @contextlib.contextmanager
    def window(self):
        t0 = time.perf_counter()
        try:
            yield
        finally:
            self.windows.append((t0, time.perf_counter()))

    def stop(self) -> dict:
        self.done.set()
        if self.nvml is not None:
            self.poller.join(timeout=1.0)
            self.nvml[0].nvmlShutdown()
        smi_sm, smi_max, smi_reasons = [], None, set()
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()
            for ln in self.lines:
                parts = [p.strip() for p in ln.split(",")]
                if len(parts) < 9:
                    continue
                try:
                    smi_sm.append(float(parts[1]))
                    smi_max = float(parts[2])
                except ValueError:
                    continue
                for nm, v in zip(self.NAMES, parts[5:9]):
                    if v.lower() == "active":
                        smi_reasons.add(nm)
        inside = [(mhz, bits) for (t, mhz, bits) in self.polled if any(a <= t <= b for a, b in self.windows)]
        if inside:
            reasons = sorted(nm for nm in self.NAMES if any(bits & self.bits[nm] for _, bits in inside))
            return {"sm_mhz": statistics.median(m for m, _ in inside), "sm_max_mhz": self.max_mhz,
                    "reasons": reasons, "samples": len(inside),
                    "source": "NVML every 5 ms inside the timed regions",
                    "nvidia_smi": {"sm_mhz": statistics.median(smi_sm) if smi_sm else None, "samples": len(smi_sm),
                                   "reasons": sorted(smi_reasons)}}
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        return {"sm_mhz": statistics.median(smi_sm) if smi_sm else None, "sm_max_mhz": smi_max,
                "reasons": sorted(smi_reasons), "samples": len(smi_sm), "source": "nvidia-smi -lms 200"}


# ---------------------------------------------------------------------------- CPU legs
def cpu_sign_rate(mode: int, budget_s: float, nthreads: int = 0) -> tuple[float, str, int]:
    """Oracle signatures/s on all host threads over a bounded sample of the same workload."""
    from oracle import pyoracle as ora
    cores = os.cpu_count() or 1
    n0 = max(16, cores * 4)
    pk, sk = ora.keypair_batch(mode, n0, 0, nthreads)
    m = ora.messages_from_ctr(n0, MLEN)
    t = time.perf_counter()
    ora.sign_batch(mode, m, sk, nthreads=nthreads)
    dt = max(time.perf_counter() - t, 1e-6)
    n = int(min(20000, max(n0, n0 * budget_s / dt)))
    pk, sk = ora.keypair_batch(mode, n, 0, nthreads)
    m = ora.messages_from_ctr(n, MLEN)
    t = time.perf_counter()
    ora.sign_batch(mode, m, sk, nthreads=nthreads)
    dt = time.perf_counter() - t
    return n / dt, f"{n} Dilithium{mode} signatures of {MLEN}-byte messages (keys 0..{n - 1} of the seed scheme)", cores


def headline_config(mode: int, B: int, world: int) -> dict:
    """The headline workload, identical in both arms (the reference arm times a bounded sample of it;
    what each arm runs is in its top-level "path")."""
    sk_cache_mib = {2: 28.3, 3: 48.3, 5: 79.0}[mode] * B / 1024
    return {"workload": f"Dilithium{mode} batched sign (+ verify), batch {B} (the reference bench batch), "
                        f"{MLEN}-byte messages, one key per message",
            "batch": B, "mlen": MLEN, "parallelism": f"replicas x{world}",
            "l2": f"inputs larger than L2: the batch's secret-key caches alone are {sk_cache_mib:.0f} MiB per rank"}


def run_reference(args) -> dict:
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return {}
    from oracle import pyoracle as ora
    cores = os.cpu_count() or 1
    mode = args.mode
    # bounded sample per step
    n = args.ref_sample
    pk, sk = ora.keypair_batch(mode, n)
    m = ora.messages_from_ctr(n, MLEN)
    for _ in range(args.warmup):
        ora.sign_batch(mode, m[: max(1, n // 8)], sk[: max(1, n // 8)])
    t = time.perf_counter()
    for _ in range(args.steps):
        ora.sign_batch(mode, m, sk)
    dt = time.perf_counter() - t
    v = n * args.steps / dt
    return {
        "metric": METRIC, "value": v, "unit": UNIT, "impl": "reference", "n_gpus": args.gpus, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": 1e3 * dt / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "int32", "data": "synthetic (reference seed scheme)",
        "config": headline_config(mode, args.batch, 1),
        "path": "CPU implementation of the path (the oracle port; the reference ships no CPU Dilithium)",
        "cpu_baseline": {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": f"{n} of the workload's {args.batch} signatures per step (keys and messages of "
                                   f"the reference seed scheme), OpenMP over {cores} threads"},
        "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }


# ---------------------------------------------------------------------------- work models
def perms_absorb(nbytes: int, rate: int = 136) -> int:
    """Keccak-f[1600] permutations of one SHAKE absorb of nbytes (the padding block included)."""
    return nbytes // rate + 1


def sign_attempt_ops(pm, attempts: float, reject_intt: float) -> float:
    """Algorithmic 32-bit ALU operations of `attempts` signing attempts whose rejection checks ran
    `reject_intt` inverse NTTs (early exits included)."""
    K, L, w1 = pm.k, pm.l, pm.k * pm.polyw1_packed
    perms = L * 5 + perms_absorb(64 + w1) + 1          # ExpandMask, c~ absorb, SampleInBall
    per_attempt = (perms * OPS_PERM + L * OPS_NTT_FWD + K * OPS_NTT_INV + K * L * 256 * OPS_PW  # w = A y
                   + OPS_NTT_FWD)                                                              # NTT(c)
    return attempts * per_attempt + reject_intt * (OPS_NTT_INV + 256 * OPS_PW)


def sign_prehash_ops(mlen: int) -> float:
    """mu = H(tr || m) and rho' = H(K || mu) of one message."""
    return (perms_absorb(32 + mlen) + 1) * OPS_PERM


def cache_ops(pm, nkeys: int) -> float:
    """ExpandA (K*L entries of 5 SHAKE128 blocks) + NTT of s1, s2, t0 per key."""
    return nkeys * (pm.k * pm.l * 5 * OPS_PERM + (pm.l + 2 * pm.k) * OPS_NTT_FWD)


def keygen_ops(pm) -> float:
    """One key pair: seed expansion, ExpandA, ExpandS (2 SHAKE256 blocks per polynomial),
    t = invNTT(A NTT(s1)) + s2, tr = H(pk)."""
    K, L = pm.k, pm.l
    perms = 1 + K * L * 5 + (K + L) * 2 + perms_absorb(pm.pk_bytes)
    return perms * OPS_PERM + L * OPS_NTT_FWD + K * OPS_NTT_INV + K * L * 256 * OPS_PW


def verify_ops(pm, mlen: int, cached: bool) -> float:
    """One verification; cached = A_hat, NTT(t1 2^d) and tr resident per key (no ExpandA, no H(pk))."""
    K, L, w1 = pm.k, pm.l, pm.k * pm.polyw1_packed
    perms = perms_absorb(32 + mlen) + perms_absorb(64 + w1) + 1
    ntt = (L + 1) * OPS_NTT_FWD + K * OPS_NTT_INV + (K * L + K) * 256 * OPS_PW
    if not cached:
        perms += perms_absorb(pm.pk_bytes) + K * L * 5
        ntt += K * OPS_NTT_FWD
    return perms * OPS_PERM + ntt


def algorithmic_attempts(nonces, issued: int, reject_intt: int) -> tuple[float, float]:
    """Attempts deterministic signing needs (winning nonce + 1 per item) and the rejection checks'
    inverse NTTs scaled to them from the issued (speculative) attempts' device count."""
    alg = float((nonces.astype("float64") + 1.0).sum())
    return alg, (reject_intt * alg / issued if issued else 0.0)


def alu_roofline(ops: float, ms: float, peak_ops: float, what: str) -> dict:
    a = ops / (ms / 1e3) / 1e9 if ms else None
    return {"bound": "int32-alu", "what": what, "achieved": a, "peak": peak_ops / 1e9, "unit": "Gop/s",
            "frac": a / (peak_ops / 1e9) if a else None, "peak_source": "measured live (k_alu_peak)"}


def timed_cpu(fn):
    t = time.perf_counter()
    r = fn()
    return r, time.perf_counter() - t


class Timer:
    def __init__(self, torch, stream):
        self.torch, self.st, self.pairs = torch, stream, []

    def __enter__(self):
        self.a = self.torch.cuda.Event(enable_timing=True)
        self.b = self.torch.cuda.Event(enable_timing=True)
        self.a.record(self.st)
        return self

    def __exit__(self, *exc):
        self.b.record(self.st)
        self.pairs.append((self.a, self.b))

    def total_ms(self):
        return sum(a.elapsed_time(b) for a, b in self.pairs)


def run_gpu(args) -> dict | None:
    import ctypes

    import numpy as np
    import torch
    import torch.distributed as dist

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", timeout=__import__("datetime").timedelta(seconds=120))

    import cudilithium_b200 as cd
    from cudilithium_b200 import _lib
    from cudilithium_b200.api import TaskLut, alloc_pool, pinned
    from cudilithium_b200.engine import Engine, EnginePipeline, pack_messages

    lib = _lib.lib
    mode, B = args.mode, args.batch
    d = cd.Dilithium(mode)
    pm = d.params
    dev = torch.device("cuda", local)
    st = torch.cuda.current_stream()
    spp = st.cuda_stream

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    def max_over_ranks(*vals):
        return reduce_max(vals, world, dev)

    # ---- inputs: keys from the reference seed scheme, one key per message
    kp_pool, kpp = alloc_pool(d.keypair_row_bytes(), B)
    d_pk = torch.empty(B * pm.pk_bytes, dtype=torch.uint8, device=dev)
    d_sk = torch.empty(B * pm.sk_bytes, dtype=torch.uint8, device=dev)
    kg = Timer(torch, st)
    for _ in range(2):
        with kg:
            _lib.check(lib.cudil_keypair_dev(mode, d_pk.data_ptr(), d_sk.data_ptr(), None, kp_pool.data_ptr(), kpp,
                                             B, spp, rank_shard(rank, B)[0]), "keypair")
    torch.cuda.synchronize()
    keygen_ms = kg.pairs[-1][0].elapsed_time(kg.pairs[-1][1])
    del kp_pool
    rng = np.random.default_rng(rank_shard(rank, B)[1])
    m_host = rng.integers(0, 256, (B, MLEN), dtype=np.uint8)
    d_m = torch.from_numpy(m_host.reshape(-1)).to(dev)
    keys = np.arange(B, dtype=np.uint32)
    offs = (np.arange(B, dtype=np.uint64) * MLEN)
    lens = np.full(B, MLEN, dtype=np.uint32)

    # ---- plain stage-by-stage path (cudil_sign_dev / cudil_verify_dev), best exec threshold
    p_sig = torch.empty(B * pm.sig_bytes, dtype=torch.uint8, device=dev)
    p_ret = torch.empty(B, dtype=torch.int32, device=dev)
    s_pool, sp = alloc_pool(d.sign_row_bytes(MLEN), B)
    v_pool, vp = alloc_pool(d.verify_row_bytes(MLEN), B)
    tmax = max(args.thresholds)
    t_pool, tp = alloc_pool(d.sign_temp_row_bytes(), tmax)

    def plain_sign(T, lut):
        _lib.check(lib.cudil_sign_dev(mode, p_sig.data_ptr(), pm.sig_bytes, d_m.data_ptr(), MLEN, MLEN,
                                      d_sk.data_ptr(), s_pool.data_ptr(), sp, t_pool.data_ptr(), tp,
                                      ctypes.byref(lut.c), T, B, spp), "sign")

    def plain_verify():
        _lib.check(lib.cudil_verify_dev(mode, p_ret.data_ptr(), p_sig.data_ptr(), pm.sig_bytes, pm.sig_bytes,
                                        d_m.data_ptr(), MLEN, MLEN, d_pk.data_ptr(), v_pool.data_ptr(), vp, B,
                                        spp), "verify")

    luts = {T: TaskLut(B, T) for T in args.thresholds}
    best_T, best_ms = None, None
    for T in args.thresholds:
        plain_sign(T, luts[T])
        tm = Timer(torch, st)
        with tm:
            plain_sign(T, luts[T])
        torch.cuda.synchronize()
        ms = tm.total_ms()
        if best_ms is None or ms < best_ms:
            best_T, best_ms = T, ms
    for _ in range(args.warmup):
        plain_sign(best_T, luts[best_T])
        plain_verify()
    barrier()
    tps, tpv = Timer(torch, st), Timer(torch, st)
    for _ in range(args.steps):
        with tps:
            plain_sign(best_T, luts[best_T])
        with tpv:
            plain_verify()
    barrier()
    plain_sign_ms, plain_verify_ms = max_over_ranks(tps.total_ms(), tpv.total_ms())
    plain_ok = int((p_ret != 0).sum().item()) == 0
    plain_sign_rate = world * B * args.steps / (plain_sign_ms / 1e3)
    plain_verify_rate = world * B * args.steps / (plain_verify_ms / 1e3)

    # ---- fused engine: per step the key caches are built for this batch's keys (each key signs
    # once here, so the cache build is part of the per-signature work) and one call signs
    es = Engine(mode, max_keys=B, max_items=B, threads=args.engine_threads)
    ev = Engine(mode, max_keys=B, max_items=B, threads=args.engine_threads)
    if args.spec_slots:
        es.set_spec_slots(args.spec_slots)
    f_sig = torch.empty(B * pm.sig_bytes, dtype=torch.uint8, device=dev)
    f_ret = torch.empty(B, dtype=torch.int32, device=dev)

    def fused_sign():
        es.set_secret_keys(d_sk, stream=spp)
        es.sign(f_sig, d_m, offs, lens, keys, stream=spp)

    def fused_verify():
        ev.set_public_keys(d_pk, stream=spp)
        ev.verify(f_ret, f_sig, d_m, offs, lens, keys, stream=spp)

    # The stream of steps (the bench value): two engines on two streams take the batches in turn
    # (EnginePipeline), so batch k+1's cache build, prehash and first signer blocks run on the SMs that
    # batch k's persistent signer frees at its end.  Each step still builds its own key caches and
    # signs the whole batch.
    pipe = EnginePipeline(mode, max_keys=B, max_items=B, depth=2, threads=args.engine_threads, spec_slots=args.spec_slots)
    p_sigs = [torch.empty(B * pm.sig_bytes, dtype=torch.uint8, device=dev) for _ in range(2)]

    for _ in range(args.warmup):
        fused_sign()
        fused_verify()
    p_rets = [torch.empty(B, dtype=torch.int32, device=dev) for _ in range(2)]
    for k in range(max(2, args.warmup)):
        pipe.sign(p_sigs[k % 2], d_m, offs, lens, keys, d_sk=d_sk, after=st)
    for k in range(max(2, args.warmup)):
        pipe.verify(p_rets[k % 2], p_sig, d_m, offs, lens, keys, d_pk=d_pk, after=st)
    pipe.join(st)
    barrier()
    assert torch.equal(f_sig, p_sig), "fused and plain signatures differ"
    assert all(torch.equal(x, p_sig) for x in p_sigs), "pipelined and plain signatures differ"
    assert int((f_ret != 0).sum().item()) == 0, "fused verify rejected valid signatures"

    props = torch.cuda.get_device_properties(dev)
    clocks = ClockSampler(local, "%08x:%02x:%02x.0" % (props.pci_domain_id, props.pci_bus_id, props.pci_device_id))
    clocks.start()
    time.sleep(0.3)
    barrier()
    for x in p_sigs:
        x.zero_()
    launches0 = lib.cudil_launch_count()
    t0p, t1p = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    wall0 = time.perf_counter()
    with clocks.window():
        t0p.record(st)
        for k in range(args.steps):
            pipe.sign(p_sigs[k % 2], d_m, offs, lens, keys, d_sk=d_sk, after=t0p if k < 2 else False)
        pipe.join(st)
        t1p.record(st)
        barrier()
    wall = time.perf_counter() - wall0
    launches = lib.cudil_launch_count() - launches0
    # the verification steps, pipelined the same way (public-key caches built per step)
    for x in p_rets:
        x.fill_(1)
    t0v, t1v = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    with clocks.window():
        t0v.record(st)
        for k in range(args.steps):
            pipe.verify(p_rets[k % 2], p_sig, d_m, offs, lens, keys, d_pk=d_pk, after=t0v if k < 2 else False)
        pipe.join(st)
        t1v.record(st)
        barrier()
    # the same steps one batch at a time (one engine, one stream each for signing and verification)
    tfs, tfv = Timer(torch, st), Timer(torch, st)
    with clocks.window():
        for _ in range(args.steps):
            with tfs:
                fused_sign()
            with tfv:
                fused_verify()
        barrier()
    clk = clocks.stop()
    pipe_ms, pv_ms, fs_ms, fv_ms = max_over_ranks(t0p.elapsed_time(t1p), t0v.elapsed_time(t1v), tfs.total_ms(),
                                                  tfv.total_ms())
    value = world * B * args.steps / (pipe_ms / 1e3)
    value_single = world * B * args.steps / (fs_ms / 1e3)
    verify_rate = world * B * args.steps / (pv_ms / 1e3)
    verify_single = world * B * args.steps / (fv_ms / 1e3)
    attempts, reject_intt = es.last_work()
    written = min(2, args.steps)  # the pipelined buffers the timed steps wrote
    fused_ok = (torch.equal(f_sig, p_sig) and all(torch.equal(x, p_sig) for x in p_sigs[:written])
                and int((f_ret != 0).sum().item()) == 0
                and all(int((x != 0).sum().item()) == 0 for x in p_rets[:written]))
    pipe.close()

    # ---- e2e: host buffers in, host signatures out, through the engine API.  The messages and
    # the secret keys go up on a copy stream, the keys in --e2e-chunks chunks; each chunk's cache
    # rows are built on the compute stream behind its own copy (update_secret_keys), so the copies
    # of later chunks overlap the builds of earlier ones.  The signer writes a round's signatures
    # straight into the pinned host output when the round ends (PCIe writes by a kernel), so the
    # download overlaps the signing.  The timed region spans all copies, builds and the signing.
    h_m = pinned(B * MLEN)
    h_m.numpy()[:] = m_host.reshape(-1)
    h_sk = pinned(B * pm.sk_bytes)
    h_sk.copy_(d_sk.cpu())
    h_sig = pinned(B * pm.sig_bytes)
    nch = max(1, min(args.e2e_chunks, B))
    bounds = [B * c // nch for c in range(nch + 1)]
    ee = Engine(mode, max_keys=B, max_items=B, threads=args.engine_threads)
    if args.spec_slots:
        ee.set_spec_slots(args.spec_slots)
    s_copy = torch.cuda.Stream(device=dev)
    e_m = torch.empty(B * MLEN, dtype=torch.uint8, device=dev)
    e_sk = torch.empty(B * pm.sk_bytes, dtype=torch.uint8, device=dev)
    ev_m = torch.cuda.Event()
    ev_k = [torch.cuda.Event() for _ in range(nch)]

    def e2e_step():
        s_copy.wait_stream(st)
        with torch.cuda.stream(s_copy):
            e_m.copy_(h_m, non_blocking=True)
            ev_m.record(s_copy)
            for c in range(nch):
                lo, hi = bounds[c] * pm.sk_bytes, bounds[c + 1] * pm.sk_bytes
                e_sk[lo:hi].copy_(h_sk[lo:hi], non_blocking=True)
                ev_k[c].record(s_copy)
        for c in range(nch):
            st.wait_event(ev_k[c])
            lo, hi = bounds[c] * pm.sk_bytes, bounds[c + 1] * pm.sk_bytes
            ee.update_secret_keys(e_sk[lo:hi], bounds[c], stream=spp)
        st.wait_event(ev_m)
        ee.sign(h_sig, e_m, offs, lens, keys, stream=spp)

    e2e_step()
    barrier()
    te = Timer(torch, st)
    for _ in range(args.steps):
        with te:
            e2e_step()
    barrier()
    (e2e_ms,) = max_over_ranks(te.total_ms())
    assert torch.equal(h_sig, p_sig.cpu()), "e2e signatures differ"
    e2e_single = world * B * args.steps / (e2e_ms / 1e3)
    ee.close()

    # ---- the same batches streamed: two engines, each with its own device inputs, pinned output
    # and compute stream, alternate, so the host-to-device copies of batch k+1 (copy stream) run
    # while batch k signs, and batch k+1's cache build starts on the SMs that batch k's signer
    # frees at its end.  One timed region spans the K batches, from the first copy to the last
    # signature written into host memory.
    pe = [Engine(mode, max_keys=B, max_items=B, threads=args.engine_threads) for _ in range(2)]
    for e in pe:
        if args.spec_slots:
            e.set_spec_slots(args.spec_slots)
    p_in = [(torch.empty(B * MLEN, dtype=torch.uint8, device=dev), torch.empty(B * pm.sk_bytes, dtype=torch.uint8,
                                                                                device=dev)) for _ in range(2)]
    p_out = [pinned(B * pm.sig_bytes) for _ in range(2)]
    in_ev = [torch.cuda.Event() for _ in range(2)]
    free_ev = [torch.cuda.Event() for _ in range(2)]
    p_st = [torch.cuda.Stream(device=dev) for _ in range(2)]  # each engine's compute stream

    def stream_step(k):
        j = k % 2
        pm_m, pm_sk = p_in[j]
        s_copy.wait_event(free_ev[j])  # this buffer set's previous batch has finished signing
        with torch.cuda.stream(s_copy):
            pm_m.copy_(h_m, non_blocking=True)
            pm_sk.copy_(h_sk, non_blocking=True)
            in_ev[j].record(s_copy)
        p_st[j].wait_event(in_ev[j])
        pe[j].set_secret_keys(pm_sk, stream=p_st[j])
        pe[j].sign(p_out[j], pm_m, offs, lens, keys, stream=p_st[j])
        free_ev[j].record(p_st[j])

    for k in range(2):  # warm-up
        stream_step(k)
    barrier()
    for k in range(2):
        free_ev[k].record(st)
    t0e, t1e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    t0e.record(st)
    s_copy.wait_stream(st)
    for k in range(args.steps):
        stream_step(k)
    for x in p_st:
        st.wait_stream(x)
    t1e.record(st)
    barrier()
    (e2e_stream_ms,) = max_over_ranks(t0e.elapsed_time(t1e))
    ref_sig = p_sig.cpu()
    assert all(torch.equal(o[: B * pm.sig_bytes], ref_sig) for o in p_out), "streamed e2e signatures differ"
    e2e = world * B * args.steps / (e2e_stream_ms / 1e3)
    for e in pe:
        e.close()

    # ---- roofline: one instrumented fused signing step
    peak_ops = measure_alu_peak(lib, dev, spp)
    lib.cudil_kernel_stats_reset()
    lib.cudil_kernel_timing(1)
    # the cache build's kernels run concurrently on two streams: time the build as a whole
    cb0, cb1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    cb0.record(st)
    es.set_secret_keys(d_sk, stream=spp)
    cb1.record(st)
    es.sign(f_sig, d_m, offs, lens, keys, stream=spp)
    torch.cuda.synchronize()
    lib.cudil_kernel_timing(0)
    stats = _lib.kernel_stats()
    att1, intt1 = es.last_work()
    alg_att, alg_intt = algorithmic_attempts(es.last_nonces(B), att1, intt1)
    g_ms = stats.get("sign batch (engine)", (0.0, 1))[0]
    # algorithmic work: the attempts deterministic signing needs (not the speculative ones issued)
    sign_ops = sign_attempt_ops(pm, alg_att, alg_intt) + B * sign_prehash_ops(MLEN)
    c_ms = cb0.elapsed_time(cb1)
    achieved = sign_ops / (g_ms / 1e3) / 1e9 if g_ms else None
    total_ms = g_ms + c_ms  # the step: cache build span + signing batch
    roofline = {
        "bound": "int32-alu",
        "kernel": f"signing batch, engine sign-kernel variant {es.sign_kernel} (0: prehash, rounds of claim, "
                  f"ExpandMask, w, challenge and rejection kernels, then the persistent kernel on what they leave)",
        "achieved": achieved, "peak": peak_ops / 1e9, "unit": "Gop/s",
        "frac": achieved / (peak_ops / 1e9) if achieved else None,
        "traffic": None,
        "traffic_source": "not one kernel: the rounds' kernels are captured one by one (profiles/)",
        "ms_per_launch": g_ms, "launches": 1, "share_of_step": g_ms / total_ms if total_ms else None,
        "attempts_algorithmic": alg_att, "attempts_issued": att1, "speculation_overhead": att1 / alg_att,
        "reject_intt_issued": intt1, "signer_phases": es.last_phases(),
        "work_basis": "attempts = sum over items of (winning nonce + 1), read back from the engine; "
                      "rejection inverse NTTs scaled from the issued attempts' device count",
        "ops_model": "Keccak-f1600 = 4560 LOP3/SHF ops; NTT 6144, invNTT 7168, Montgomery product 5",
        "peak_source": "measured live: k_alu_peak (3 LOP3 : 1 SHF at 64 ops/clk/SM; IMAD-heavy NTT work can "
                       "co-issue on the FMA pipe, so frac may exceed 1)",
        "cache_build": {"ms": c_ms, "achieved_gops": cache_ops(pm, B) / (c_ms / 1e3) / 1e9 if c_ms else None,
                        "note": "k_cache_sk and k_expand_a run concurrently on two streams; ms is the build's span"},
        "kernels": {k: {"ms": round(v[0], 4), "launches": v[1]} for k, v in sorted(stats.items(), key=lambda kv: -kv[1][0])},
    }

    result = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": pipe_ms / args.steps, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "int32", "data": "synthetic: keys from the reference seed scheme, uniform random 32-byte messages",
        "config": headline_config(mode, B, world),
        "path": "fused engine: per step the batch's key caches are built and the batch is signed in one "
                "call (staged rounds); consecutive steps alternate between two engines on two streams "
                "(EnginePipeline), one timed region over all steps",
        "one_batch_at_a_time": {"value": value_single, "ms_per_step": fs_ms / args.steps, "verify_per_s": verify_single,
                                "note": "the same steps on one engine and one stream, each step timed on its own"},
        "engine": es.info(),
        "verify_per_s": verify_rate, "keygen_per_s": world * B / (keygen_ms / 1e3),
        "plain": {"sign_per_s": plain_sign_rate, "verify_per_s": plain_verify_rate, "exec_threshold": best_T,
                  "all_verified": plain_ok},
        "fused_over_plain": {"sign": value_single / plain_sign_rate, "sign_pipelined": value / plain_sign_rate,
                             "verify": verify_single / plain_verify_rate, "verify_pipelined": verify_rate / plain_verify_rate,
                             "sign_resident_keys": (B / (g_ms / 1e3)) / plain_sign_rate if g_ms else None},
        "bit_exact_fused_vs_plain": fused_ok, "attempts_per_signature": alg_att / B,
        "attempts_issued_per_signature": attempts / B,
        "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": B * (MLEN + pm.sk_bytes),
                "d2h_bytes_per_step": B * pm.sig_bytes, "signatures": "written into pinned host memory by the signer",
                "pipelining": "two engines alternate on two compute streams, so the host-to-device copies and the "
                              "cache build of batch k+1 overlap the signing of batch k; one timed region over all "
                              "batches",
                "one_batch_at_a_time": {"value": e2e_single, "key_chunks": nch,
                                        "note": "each batch's copies, cache builds (behind each key chunk) and signing "
                                                "timed on their own"}},
        "gpu_launches": int(launches), "wall_s_timed": wall, "clocks": clk, "roofline": roofline,
    }
    del s_pool, v_pool, t_pool, es, ev
    torch.cuda.empty_cache()
    # the other configurations (and the serving sweep, which drives the host threads hard) run in
    # the single-GPU invocation only; a multi-GPU run reports the replicated headline
    if not args.quick and world == 1:
        result["configs"] = run_configs(args, torch, np, lib, _lib, dev, spp, rank, peak_ops)
        result["configs"]["serve_mixed"] = run_serve(args, np)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    if rank == 0 and world == 1 and not args.no_cpu:
        rate, sample, cores = cpu_sign_rate(mode, args.cpu_seconds)
        result["cpu_baseline"] = {"value": rate, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample}
    return result if rank == 0 else None


def seed_scheme_messages(n: int, mlen: int = 32, start: int = 0):
    """Messages of the reference's test-vector scheme: SHAKE128(le64(2i))[0:mlen]."""
    import hashlib

    import numpy as np
    return np.stack([np.frombuffer(hashlib.shake_128((2 * i).to_bytes(8, "little")).digest(mlen), dtype=np.uint8)
                     for i in range(start, start + n)])


def run_configs(args, torch, np, lib, _lib, dev, spp, rank, peak_ops) -> dict:
    """The other configurations, reported beside the headline (not the bench value).  Each leg times
    the plain and the fused GPU path where both exist, reports the algorithmic work against the
    measured peak, and in its CPU leg times the oracle (OpenMP over all host threads) on the same
    inputs -- a bounded sample where the whole workload would take too long -- and checks the GPU
    outputs against it byte for byte."""
    import ctypes

    import cudilithium_b200 as cd
    from cudilithium_b200.api import TaskLut, alloc_pool, ntt_mul
    from cudilithium_b200.engine import Engine, EnginePipeline
    from oracle import pyoracle as ora
    st = torch.cuda.current_stream()
    cores = os.cpu_count() or 1
    out = {}

    def gpu_ms(fn, reps, warm=3):
        for _ in range(warm):
            fn()
        torch.cuda.synchronize()
        tm = Timer(torch, st)
        for _ in range(reps):
            with tm:
                fn()
        torch.cuda.synchronize()
        return tm.total_ms() / reps

    # ---- config 1: Dilithium2 keygen + sign + verify, batch 1024, the reference seed scheme
    d = cd.Dilithium(2)
    pm = d.params
    n = 1024
    pool, kpp = alloc_pool(d.keypair_row_bytes(), n)
    pk = torch.empty(n * pm.pk_bytes, dtype=torch.uint8, device=dev)
    sk = torch.empty(n * pm.sk_bytes, dtype=torch.uint8, device=dev)
    m1_host = seed_scheme_messages(n, 32)
    m = torch.from_numpy(m1_host.reshape(-1)).to(dev)
    offs, lens, keys = np.arange(n, dtype=np.uint64) * 32, np.full(n, 32, np.uint32), np.arange(n, dtype=np.uint32)
    s_pool, sp = alloc_pool(d.sign_row_bytes(32), n)
    t_pool, tp = alloc_pool(d.sign_temp_row_bytes(), 4096)
    v_pool, vp = alloc_pool(d.verify_row_bytes(32), n)
    lut = TaskLut(n, 4096)
    sig = torch.empty(n * pm.sig_bytes, dtype=torch.uint8, device=dev)
    ret = torch.empty(n, dtype=torch.int32, device=dev)
    psig = torch.empty_like(sig)
    pret = torch.empty_like(ret)
    es, ev = Engine(2, n, n), Engine(2, n, n)

    def c1_plain():
        lib.cudil_keypair_dev(2, pk.data_ptr(), sk.data_ptr(), None, pool.data_ptr(), kpp, n, spp, 0)
        lib.cudil_sign_dev(2, psig.data_ptr(), pm.sig_bytes, m.data_ptr(), 32, 32, sk.data_ptr(), s_pool.data_ptr(),
                           sp, t_pool.data_ptr(), tp, ctypes.byref(lut.c), 4096, n, spp)
        lib.cudil_verify_dev(2, pret.data_ptr(), psig.data_ptr(), pm.sig_bytes, pm.sig_bytes, m.data_ptr(), 32, 32,
                             pk.data_ptr(), v_pool.data_ptr(), vp, n, spp)

    # the verifier's public-key cache depends only on the key pairs: it is built on a second stream
    # while the batch is signed, and verification waits for both
    s_pk = torch.cuda.Stream(device=dev)
    e_keys, e_pkc = torch.cuda.Event(), torch.cuda.Event()

    def c1_fused():
        lib.cudil_keypair_dev(2, pk.data_ptr(), sk.data_ptr(), None, pool.data_ptr(), kpp, n, spp, 0)
        e_keys.record(st)
        s_pk.wait_event(e_keys)
        ev.set_public_keys(pk, stream=s_pk)
        e_pkc.record(s_pk)
        es.set_secret_keys(sk, stream=spp)
        es.sign(sig, m, offs, lens, keys, stream=spp)
        st.wait_event(e_pkc)
        ev.verify(ret, sig, m, offs, lens, keys, stream=spp)

    res = {"plain_ms": gpu_ms(c1_plain, 5), "fused_ms": gpu_ms(c1_fused, 5),
           "fused_path": "keygen; secret-key cache build and signing, with the public-key cache build on a "
                         "second stream beside them; verify (fused engines)"}
    res["fused_over_plain"] = res["plain_ms"] / res["fused_ms"]
    alg1, _ = algorithmic_attempts(es.last_nonces(n), *es.last_work())
    ops1 = n * (keygen_ops(pm) + sign_prehash_ops(32) + verify_ops(pm, 32, cached=False)) \
        + sign_attempt_ops(pm, alg1, es.last_work()[1] * alg1 / max(es.last_work()[0], 1)) + cache_ops(pm, n)
    res["roofline"] = alu_roofline(ops1, res["fused_ms"], peak_ops, "fused: keygen + cache builds + sign + verify")
    g_pk, g_sk = pk.cpu().numpy().reshape(n, -1), sk.cpu().numpy().reshape(n, -1)
    g_sig, g_ret = sig.cpu().numpy().reshape(n, -1), ret.cpu().numpy()
    fused_eq_plain = bool(torch.equal(sig, psig) and torch.equal(ret, pret))
    (o_pk, o_sk), t_kg = timed_cpu(lambda: ora.keypair_batch(2, n))
    o_sig, t_sg = timed_cpu(lambda: ora.sign_batch(2, m1_host, o_sk))
    o_ret, t_vf = timed_cpu(lambda: ora.verify_batch(2, o_sig, m1_host, o_pk))
    parts = {"fused_eq_plain": fused_eq_plain, "pk": bool(np.array_equal(g_pk, o_pk)),
             "sk": bool(np.array_equal(g_sk, o_sk)), "sig": bool(np.array_equal(g_sig, o_sig)),
             "ret": bool(np.array_equal(g_ret, o_ret) and not o_ret.any())}
    res["bit_exact"] = all(parts.values())
    if not res["bit_exact"]:
        res["bit_exact_parts"] = parts
    res["cpu_baseline"] = {"ms": 1e3 * (t_kg + t_sg + t_vf), "keygen_per_s": n / t_kg, "sign_per_s": n / t_sg,
                           "verify_per_s": n / t_vf, "cores": cores, "kind": "port",
                           "sample": f"the whole workload ({n} items), OpenMP over {cores} threads"}
    res["gpu_over_cpu"] = res["cpu_baseline"]["ms"] / res["fused_ms"]
    out["d2_keygen_sign_verify_batch1024"] = res
    log(f"[configs] 1: plain {res['plain_ms']:.3f} ms fused {res['fused_ms']:.3f} ms bit_exact {res['bit_exact']}")
    del pool, s_pool, t_pool, v_pool, es, ev

    # ---- config 2: NTT microbench, 2^20 polynomials: NTT -> Montgomery product -> invNTT
    npoly = 1 << 20
    g = torch.Generator(device=dev).manual_seed(42)
    a = torch.randint(0, 8380417, (npoly, 256), dtype=torch.int32, device=dev, generator=g)
    b = torch.randint(0, 8380417, (npoly, 256), dtype=torch.int32, device=dev, generator=g)
    o = torch.empty_like(a)
    ms = gpu_ms(lambda: ntt_mul(a, b, o), 10)
    peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
    hbm = peaks.get("hbm_gbs", 6650.0)
    gbs = npoly * 3072 / (ms / 1e3) / 1e9
    S = 1 << 15
    a_s, b_s, o_s = a[:S].cpu().numpy(), b[:S].cpu().numpy(), o[:S].cpu().numpy()
    o_ref, t_ntt = timed_cpu(lambda: ora.ntt_mul_batch(a_s, b_s))
    ntt_ops = npoly * (OPS_NTT_FWD + OPS_NTT_INV + 256 * OPS_PW)
    out["ntt_microbench_2^20"] = {
        "ms": ms, "polys_per_s": npoly / (ms / 1e3), "hbm_gbs": gbs, "hbm_frac": gbs / hbm, "hbm_peak_gbs": hbm,
        "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm, "unit": "GB/s", "frac": gbs / hbm,
                     "peak_source": "MEASURED_PEAKS.json" if peaks else "fallback 6650",
                     "alu": alu_roofline(ntt_ops, ms, peak_ops, "fwd NTT + 256 products + inv NTT per poly")},
        "bytes_per_poly": 3072, "l2": "inputs 2 GiB > L2",
        "bit_exact": bool(np.array_equal(o_s, o_ref)),
        "cpu_baseline": {"polys_per_s": S / t_ntt, "cores": cores, "kind": "port",
                         "sample": f"the first {S} of the {npoly} polynomials, OpenMP over {cores} threads"}}
    log(f"[configs] 2: {ms:.3f} ms {gbs:.0f} GB/s bit_exact {out['ntt_microbench_2^20']['bit_exact']}")
    del a, b, o

    # ---- config 3: Dilithium3 signing of 16384 messages over 1024 keys, log-uniform 32 B .. 64 KiB
    d3 = cd.Dilithium(3)
    p3 = d3.params
    nk, nm = 1024, 16384
    pool, kpp = alloc_pool(d3.keypair_row_bytes(), nk)
    pk3 = torch.empty(nk * p3.pk_bytes, dtype=torch.uint8, device=dev)
    sk3 = torch.empty(nk * p3.sk_bytes, dtype=torch.uint8, device=dev)
    lib.cudil_keypair_dev(3, pk3.data_ptr(), sk3.data_ptr(), None, pool.data_ptr(), kpp, nk, spp, 0)
    del pool
    rng = np.random.default_rng(3)
    mlens = np.floor(np.exp(rng.uniform(np.log(32), np.log(65536), nm))).astype(np.uint32)
    offs3 = np.zeros(nm, np.uint64)
    offs3[1:] = np.cumsum((mlens[:-1].astype(np.uint64) + 7) // 8 * 8)
    total = int(offs3[-1] + mlens[-1]) + 8
    d_msgs = torch.randint(0, 256, (total,), dtype=torch.uint8, device=dev)
    keys3 = (np.arange(nm) % nk).astype(np.uint32)
    e3 = Engine(3, nk, nm)
    s3 = torch.empty(nm * p3.sig_bytes, dtype=torch.uint8, device=dev)
    e3.set_secret_keys(sk3, stream=spp)
    ms3 = gpu_ms(lambda: e3.sign(s3, d_msgs, offs3, mlens, keys3, stream=spp), 5)
    cms = gpu_ms(lambda: e3.set_secret_keys(sk3, stream=spp), 1, warm=0)
    # the same batch as a stream over two engines sharing the resident key caches (EnginePipeline):
    # a batch's prehash, bounded by its longest message, runs beside the previous batch's signer
    pipe3 = EnginePipeline(3, nk, nm, depth=2, share_keys=True)
    pipe3.engines[0].set_secret_keys(sk3, stream=spp)
    s3q = [torch.empty_like(s3) for _ in range(2)]
    for k in range(2):
        pipe3.sign(s3q[k], d_msgs, offs3, mlens, keys3, after=st)
    pipe3.join(st)
    torch.cuda.synchronize()
    K3 = 6
    q0, q1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    q0.record(st)
    for k in range(K3):
        pipe3.sign(s3q[k % 2], d_msgs, offs3, mlens, keys3, after=q0 if k < 2 else False)
    pipe3.join(st)
    q1.record(st)
    torch.cuda.synchronize()
    ms3q = q0.elapsed_time(q1) / K3
    e3.sign(s3, d_msgs, offs3, mlens, keys3, stream=spp)
    torch.cuda.synchronize()
    iss3, intt3 = e3.last_work()
    alg3, alg_intt3 = algorithmic_attempts(e3.last_nonces(nm), iss3, intt3)
    ops3 = sign_attempt_ops(p3, alg3, alg_intt3) + sum(sign_prehash_ops(int(x)) for x in mlens)
    # plain path on the same messages: pitched rows of the longest message, secret key per row
    mmax = int(mlens.max())
    h_msgs = d_msgs.cpu().numpy()
    rows = np.zeros((nm, mmax), np.uint8)
    for i in range(nm):
        rows[i, : mlens[i]] = h_msgs[int(offs3[i]): int(offs3[i]) + int(mlens[i])]
    d_rows = torch.from_numpy(rows.reshape(-1)).to(dev)
    d_ml = torch.from_numpy(mlens.astype(np.int32)).to(dev)
    sk_rows = sk3.view(nk, p3.sk_bytes)[torch.from_numpy(keys3.astype(np.int64)).to(dev)].reshape(-1).contiguous()
    sp3, spp3 = alloc_pool(d3.sign_row_bytes(mmax), nm)
    T3 = 16384
    tp3, tpp3 = alloc_pool(d3.sign_temp_row_bytes(), T3)
    lut3 = TaskLut(nm, T3)
    s3p = torch.empty_like(s3)

    def plain3():
        _lib.check(lib.cudil_sign_dev_varlen(3, s3p.data_ptr(), p3.sig_bytes, d_rows.data_ptr(), mmax,
                                             d_ml.data_ptr(), mmax, sk_rows.data_ptr(), sp3.data_ptr(), spp3,
                                             tp3.data_ptr(), tpp3, ctypes.byref(lut3.c), T3, nm, spp), "sign varlen")

    ms3p = gpu_ms(plain3, 3, warm=1)
    fused_eq_plain3 = bool(torch.equal(s3, s3p)) and all(bool(torch.equal(x, s3)) for x in s3q)
    pipe3.close()
    del sp3, tp3, d_rows, sk_rows
    ev3 = Engine(3, nk, nm)
    ev3.set_public_keys(pk3, stream=spp)
    r3 = torch.empty(nm, dtype=torch.int32, device=dev)
    ev3.verify(r3, s3, d_msgs, offs3, mlens, keys3, stream=spp)
    torch.cuda.synchronize()
    # CPU leg: a uniform sample (timed) plus the 16 longest messages, checked byte for byte
    samp = np.sort(rng.choice(nm, 384, replace=False))
    longest = np.argsort(mlens)[-16:]
    h_sk3 = sk3.cpu().numpy().reshape(nk, -1)
    g_s3 = s3.cpu().numpy().reshape(nm, -1)

    def ora_sign3(idx):
        mm = np.zeros((idx.size, int(mlens[idx].max())), np.uint8)
        for r, i in enumerate(idx):
            mm[r, : mlens[i]] = h_msgs[int(offs3[i]): int(offs3[i]) + int(mlens[i])]
        return ora.sign_batch(3, mm, h_sk3[keys3[idx]], mlens=mlens[idx])

    o_samp, t3 = timed_cpu(lambda: ora_sign3(samp))
    o_long = ora_sign3(longest)
    out["d3_sign_16384_loguniform"] = {
        "sign_per_s_resident_keys": nm / (ms3 / 1e3), "ms_per_batch": ms3, "cache_build_ms_1024_keys": cms,
        "sign_per_s_incl_cache_build": nm / ((ms3 + cms) / 1e3),
        "pipelined": {"sign_per_s": nm / (ms3q / 1e3), "ms_per_batch": ms3q, "batches": K3,
                      "note": "the batch repeated as a stream over two engines sharing the key caches, two streams"},
        "plain": {"ms_per_batch": ms3p, "sign_per_s": nm / (ms3p / 1e3), "exec_threshold": T3,
                  "path": "cudil_sign_dev_varlen: per-item ExpandA and key unpack, host-driven rounds"},
        "fused_over_plain": {"resident_keys": ms3p / ms3, "incl_cache_build": ms3p / (ms3 + cms),
                             "resident_keys_pipelined": ms3p / ms3q},
        "attempts_per_signature": alg3 / nm, "attempts_issued_per_signature": iss3 / nm,
        "mean_mlen": float(mlens.mean()), "max_mlen": mmax,
        "roofline": alu_roofline(ops3, ms3, peak_ops, "fused signer, resident keys (prehash + attempts)"),
        "bit_exact": bool(fused_eq_plain3 and np.array_equal(g_s3[samp], o_samp)
                          and np.array_equal(g_s3[longest], o_long)),
        "all_verified": int((r3 != 0).sum().item()) == 0,
        "cpu_baseline": {"sign_per_s": samp.size / t3, "cores": cores, "kind": "port",
                         "sample": f"{samp.size} messages drawn uniformly from the {nm} (same length distribution), "
                                   f"OpenMP over {cores} threads; the 16 longest are also checked"}}
    log(f"[configs] 3: fused {ms3:.2f} ms plain {ms3p:.2f} ms bit_exact {out['d3_sign_16384_loguniform']['bit_exact']}")
    del e3, ev3, d_msgs

    # ---- config 4: Dilithium5 verification of 65536 signatures (256 keys x 256 64-byte messages, 10% flipped)
    d5 = cd.Dilithium(5)
    p5 = d5.params
    nk, nm = 256, 65536
    pool, kpp = alloc_pool(d5.keypair_row_bytes(), nk)
    pk5 = torch.empty(nk * p5.pk_bytes, dtype=torch.uint8, device=dev)
    sk5 = torch.empty(nk * p5.sk_bytes, dtype=torch.uint8, device=dev)
    lib.cudil_keypair_dev(5, pk5.data_ptr(), sk5.data_ptr(), None, pool.data_ptr(), kpp, nk, spp, 0)
    del pool
    keys5 = (np.arange(nm) // 256).astype(np.uint32)
    m5 = torch.randint(0, 256, (nm * 64,), dtype=torch.uint8, device=dev)
    offs5, lens5 = np.arange(nm, dtype=np.uint64) * 64, np.full(nm, 64, np.uint32)
    e5 = Engine(5, nk, nm)
    e5.set_secret_keys(sk5, stream=spp)
    s5 = torch.empty(nm * p5.sig_bytes, dtype=torch.uint8, device=dev)
    e5.sign(s5, m5, offs5, lens5, keys5, stream=spp)
    torch.cuda.synchronize()
    del e5
    flip = rng.permutation(nm)[: nm // 10]
    pos = rng.integers(0, p5.sig_bytes, flip.size)
    bit = rng.integers(0, 8, flip.size)
    sv = s5.view(nm, p5.sig_bytes)
    sv[torch.from_numpy(flip).to(dev), torch.from_numpy(pos).to(dev)] ^= torch.from_numpy(
        (1 << bit).astype(np.uint8)).to(dev)
    expect_bad = np.zeros(nm, bool)
    expect_bad[flip] = True
    ev5 = Engine(5, nk, nm)
    ev5.set_public_keys(pk5, stream=spp)
    r5 = torch.empty(nm, dtype=torch.int32, device=dev)
    fused_ms = gpu_ms(lambda: ev5.verify(r5, s5, m5, offs5, lens5, keys5, stream=spp), 5)
    got = r5.cpu().numpy()
    # the same batch as a stream over two engines sharing the cached public keys (EnginePipeline)
    pipe5 = EnginePipeline(5, nk, nm, depth=2, share_keys=True)
    pipe5.engines[0].set_public_keys(pk5, stream=spp)
    r5q = [torch.empty_like(r5) for _ in range(2)]
    for k in range(2):
        pipe5.verify(r5q[k], s5, m5, offs5, lens5, keys5, after=st)
    pipe5.join(st)
    torch.cuda.synchronize()
    K5 = 6
    q0, q1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    q0.record(st)
    for k in range(K5):
        pipe5.verify(r5q[k % 2], s5, m5, offs5, lens5, keys5, after=q0 if k < 2 else False)
    pipe5.join(st)
    q1.record(st)
    torch.cuda.synchronize()
    pipe_ms5 = q0.elapsed_time(q1) / K5
    pipe5_same = all(bool(torch.equal(x, r5)) for x in r5q)
    pipe5.close()
    # plain path on the same signatures (per-signature ExpandA and H(pk)); keys expanded per row
    pk_rows = pk5.view(nk, p5.pk_bytes)[torch.from_numpy(keys5.astype(np.int64)).to(dev)].reshape(-1).contiguous()
    v_pool, vp = alloc_pool(d5.verify_row_bytes(64), nm)
    r5p = torch.empty(nm, dtype=torch.int32, device=dev)

    def plain5():
        lib.cudil_verify_dev(5, r5p.data_ptr(), s5.data_ptr(), p5.sig_bytes, p5.sig_bytes, m5.data_ptr(), 64, 64,
                             pk_rows.data_ptr(), v_pool.data_ptr(), vp, nm, spp)

    plain_ms = gpu_ms(plain5, 3, warm=1)
    samp = np.sort(rng.choice(nm, 4096, replace=False))
    h_s5 = s5.cpu().numpy().reshape(nm, -1)[samp]
    h_m5 = m5.cpu().numpy().reshape(nm, -1)[samp]
    h_pk5 = pk5.cpu().numpy().reshape(nk, -1)[keys5[samp]]
    o_r5, t5 = timed_cpu(lambda: ora.verify_batch(5, h_s5, h_m5, h_pk5))
    out["d5_verify_65536_cached_keys"] = {
        "verify_per_s_fused": nm / (fused_ms / 1e3), "verify_per_s_plain": nm / (plain_ms / 1e3),
        "fused_over_plain": plain_ms / fused_ms, "rejections_exact": bool(np.array_equal(got != 0, expect_bad)),
        "pipelined": {"verify_per_s": nm / (pipe_ms5 / 1e3), "ms_per_batch": pipe_ms5, "batches": K5,
                      "fused_over_plain": plain_ms / pipe_ms5, "same_results": pipe5_same,
                      "note": "the batch repeated as a stream over two engines sharing the key caches, two streams"},
        "fused_equals_plain": bool(torch.equal(r5, r5p)), "flipped": int(flip.size),
        "roofline": alu_roofline(nm * verify_ops(p5, 64, cached=True), fused_ms, peak_ops,
                                 "fused verifier, cached A_hat / t1_hat / tr"),
        "bit_exact": bool(np.array_equal(got[samp], o_r5) and torch.equal(r5, r5p) and pipe5_same),
        "cpu_baseline": {"verify_per_s": samp.size / t5, "cores": cores, "kind": "port",
                         "sample": f"{samp.size} of the {nm} signatures (flipped ones included), OpenMP over "
                                   f"{cores} threads"}}
    log(f"[configs] 4: fused {fused_ms:.2f} ms plain {plain_ms:.2f} ms bit_exact "
        f"{out['d5_verify_65536_cached_keys']['bit_exact']}")
    del v_pool, ev5
    torch.cuda.empty_cache()
    return out


def run_serve(args, np) -> dict:
    """Serving loop: open-loop Poisson stream mixing Dilithium2/3/5 (60/25/15), 70% verify / 30%
    sign, resident seeded keys per parameter set, message lengths log-uniform 32 B - 4 KiB, fixed
    device-memory budget.  Per path (fused engines with resident key caches / plain stage-by-stage
    calls): saturation throughput (every request queued at t = 0), then Poisson arrivals at
    fractions of it with p50/p99 latency (arrival to completion seen by the host)."""
    import torch

    from cudilithium_b200.serve import Trace, make_keys, poisson_trace, serve, summary
    nkeys = args.serve_keys
    t0 = time.time()
    keys = make_keys({2: nkeys, 3: nkeys, 5: nkeys})
    base = poisson_trace(keys, rate=float("inf"), n=args.serve_requests, seed=11)
    log(f"[serve] keys + trace of {len(base.reqs)} requests in {time.time() - t0:.1f}s")
    torch.cuda.empty_cache()
    rng = np.random.default_rng(12)
    budget = int(args.serve_budget_gib * 2**30)
    out = {"workload": f"open-loop Poisson, Dilithium2/3/5 = 60/25/15, 70% verify / 30% sign, {nkeys} resident "
                       f"keys per parameter set, mlen log-uniform 32 B - 4 KiB, {len(base.reqs)} distinct requests "
                       f"repeated over a {args.serve_seconds} s arrival window per point, device budget "
                       f"{args.serve_budget_gib} GiB",
           "budget_bytes": budget, "latency": "arrival to completion observed by the host, ms"}
    def tiled(n, rate):
        # the unique requests repeated (same messages and signatures) up to n, arrivals redrawn
        r = np.resize(base.reqs, n)
        r["arrival_s"] = 0.0 if math.isinf(rate) else np.cumsum(rng.exponential(1.0 / rate, n))
        return Trace(r, base.msgs, base.sigs, np.resize(base.expect, n), rate)

    for path, name in ((0, "fused"), (1, "plain")):
        cfgkw = dict(path=path, budget_bytes=budget, slots_per_lane=args.serve_slots, max_batch=args.serve_max_batch)
        # saturation: about one second of requests at the expected peak, all queued at t = 0
        tr = tiled(max(len(base.reqs), int(min(args.serve_seconds, 1.0) * 4e6)), float("inf"))
        res, _, st = serve(tr, keys, want_sigs=False, **cfgkw)
        ok = bool(np.array_equal(res["status"][tr.reqs["op"] == 1], tr.expect[tr.reqs["op"] == 1]))
        sat = summary(tr, res, st)
        peak = sat["throughput_per_s"]
        points = []
        for f in args.serve_fracs:
            rate = f * peak
            tr = tiled(max(20_000, int(rate * args.serve_seconds)), rate)
            res, _, st = serve(tr, keys, want_sigs=False, **cfgkw)
            ok &= bool(np.array_equal(res["status"][tr.reqs["op"] == 1], tr.expect[tr.reqs["op"] == 1]))
            sm = summary(tr, res, st)
            points.append({"offered_frac_of_peak": f, "offered_per_s": rate, "achieved_per_s": sm["throughput_per_s"],
                           "achieved_frac_of_peak": sm["throughput_per_s"] / peak, "p50_ms": sm["p50_ms"],
                           "p99_ms": sm["p99_ms"], "mean_batch": sm["mean_batch"], "lanes": sm["lanes"]})
            log(f"[serve] {name} rate {rate:,.0f}/s -> {sm['throughput_per_s']:,.0f}/s p50 {sm['p50_ms']:.2f} ms "
                f"p99 {sm['p99_ms']:.2f} ms")
        out[name] = {"peak_per_s": peak, "saturation": {k: sat[k] for k in ("p50_ms", "p99_ms", "mean_batch", "slots",
                                                                             "device_bytes", "batches", "wall_s",
                                                                             "slot_time_s")},
                     "points": points, "verify_status_exact": ok}
        log(f"[serve] {name} saturation {peak:,.0f} requests/s, slots {sat['slots']}")
    out["fused_over_plain_peak"] = out["fused"]["peak_per_s"] / out["plain"]["peak_per_s"]
    return out


def ctypes_byref(x):
    import ctypes
    return ctypes.byref(x)


def measure_alu_peak(lib, dev, stream_ptr) -> float:
    """32-bit LOP3/SHF operations per second of this GPU (best of 3 launches, CUDA events)."""
    import ctypes

    import torch
    nsm = torch.cuda.get_device_properties(dev).multi_processor_count
    blocks = nsm * 8
    out = torch.empty(blocks * 256, dtype=torch.int32, device=dev)
    ops = ctypes.c_double(0)
    lib.cudil_alu_peak(out.data_ptr(), blocks, 256, stream_ptr, ctypes.byref(ops))
    best = 0.0
    for _ in range(3):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        st = torch.cuda.current_stream()
        a.record(st)
        lib.cudil_alu_peak(out.data_ptr(), blocks, 4096, stream_ptr, ctypes.byref(ops))
        b.record(st)
        torch.cuda.synchronize()
        best = max(best, ops.value / (a.elapsed_time(b) / 1e3))
    return best


def run_profile_case(args) -> dict:
    """Small, self-checking cases for ncu captures (one launch of the kernel of interest after
    one warm-up launch): fused-sign | fused-verify | ntt | plain-sign."""
    import ctypes

    import numpy as np
    import torch

    import cudilithium_b200 as cd
    from cudilithium_b200 import _lib
    from cudilithium_b200.api import TaskLut, alloc_pool, ntt_mul
    from cudilithium_b200.engine import Engine
    lib = _lib.lib
    mode, B = args.mode, args.batch
    d = cd.Dilithium(mode)
    pm = d.params
    dev = torch.device("cuda", 0)
    spp = torch.cuda.current_stream().cuda_stream
    if args.workload == "d3-sign":
        # the Dilithium3 long-message signing workload (16384 messages over 1024 keys, log-uniform
        # 32 B .. 64 KiB): one warm-up and one measured batch of the fused engine, checked
        # against the plain path
        nk, nm = 1024, 16384
        d3 = cd.Dilithium(3)
        p3 = d3.params
        pool, kpp = alloc_pool(d3.keypair_row_bytes(), nk)
        pk3 = torch.empty(nk * p3.pk_bytes, dtype=torch.uint8, device=dev)
        sk3 = torch.empty(nk * p3.sk_bytes, dtype=torch.uint8, device=dev)
        lib.cudil_keypair_dev(3, pk3.data_ptr(), sk3.data_ptr(), None, pool.data_ptr(), kpp, nk, spp, 0)
        rng = np.random.default_rng(3)
        mlens = np.floor(np.exp(rng.uniform(np.log(32), np.log(65536), nm))).astype(np.uint32)
        offs3 = np.zeros(nm, np.uint64)
        offs3[1:] = np.cumsum((mlens[:-1].astype(np.uint64) + 7) // 8 * 8)
        d_msgs = torch.randint(0, 256, (int(offs3[-1] + mlens[-1]) + 8,), dtype=torch.uint8, device=dev)
        keys3 = (np.arange(nm) % nk).astype(np.uint32)
        e3 = Engine(3, nk, nm, threads=args.engine_threads)
        if args.sign_kernel >= 0:
            e3.set_sign_kernel(args.sign_kernel)
        s3 = torch.empty(nm * p3.sig_bytes, dtype=torch.uint8, device=dev)
        e3.set_secret_keys(sk3, stream=spp)
        for _ in range(2):
            e3.sign(s3, d_msgs, offs3, mlens, keys3, stream=spp)
        torch.cuda.synchronize()
        e3.last_status()
        ev3 = Engine(3, nk, nm)
        ev3.set_public_keys(pk3, stream=spp)
        r3 = torch.empty(nm, dtype=torch.int32, device=dev)
        ev3.verify(r3, s3, d_msgs, offs3, mlens, keys3, stream=spp)
        torch.cuda.synchronize()
        assert int((r3 != 0).sum().item()) == 0
        return {"workload": "d3-sign", "engine": e3.info(), "attempts": e3.last_work()[0], "phases": e3.last_phases()}
    if args.workload == "ntt":
        n = B
        g = torch.Generator(device=dev).manual_seed(1)
        a = torch.randint(0, 8380417, (n, 256), dtype=torch.int32, device=dev, generator=g)
        b = torch.randint(0, 8380417, (n, 256), dtype=torch.int32, device=dev, generator=g)
        o = ntt_mul(a, b)
        ntt_mul(a, b, o)
        torch.cuda.synchronize()
        return {"workload": "ntt", "npolys": n}
    pool, kpp = alloc_pool(d.keypair_row_bytes(), B)
    pk = torch.empty(B * pm.pk_bytes, dtype=torch.uint8, device=dev)
    sk = torch.empty(B * pm.sk_bytes, dtype=torch.uint8, device=dev)
    lib.cudil_keypair_dev(mode, pk.data_ptr(), sk.data_ptr(), None, pool.data_ptr(), kpp, B, spp, 0)
    m = torch.randint(0, 256, (B * MLEN,), dtype=torch.uint8, device=dev)
    offs, lens, keys = np.arange(B, dtype=np.uint64) * MLEN, np.full(B, MLEN, np.uint32), np.arange(B, dtype=np.uint32)
    sig = torch.empty(B * pm.sig_bytes, dtype=torch.uint8, device=dev)
    ret = torch.empty(B, dtype=torch.int32, device=dev)
    if args.workload == "plain-sign":
        s_pool, sp = alloc_pool(d.sign_row_bytes(MLEN), B)
        t_pool, tp = alloc_pool(d.sign_temp_row_bytes(), 8192)
        lut = TaskLut(B, 8192)
        for _ in range(2):
            _lib.check(lib.cudil_sign_dev(mode, sig.data_ptr(), pm.sig_bytes, m.data_ptr(), MLEN, MLEN,
                                          sk.data_ptr(), s_pool.data_ptr(), sp, t_pool.data_ptr(), tp,
                                          ctypes.byref(lut.c), 8192, B, spp), "sign")
        torch.cuda.synchronize()
        return {"workload": "plain-sign", "batch": B}
    es = Engine(mode, B, B, threads=args.engine_threads)
    if args.sign_kernel >= 0:
        es.set_sign_kernel(args.sign_kernel)
    if args.spec_slots:
        es.set_spec_slots(args.spec_slots)
    es.set_secret_keys(sk, stream=spp)
    for _ in range(2):
        es.sign(sig, m, offs, lens, keys, stream=spp)
    torch.cuda.synchronize()
    es.last_status()
    out = {"workload": args.workload, "batch": B, "engine": es.info(), "attempts": es.last_work()[0],
           "phases": es.last_phases()}
    if args.workload == "fused-verify":
        ev = Engine(mode, B, B, threads=args.engine_threads)
        ev.set_public_keys(pk, stream=spp)
        for _ in range(2):
            ev.verify(ret, sig, m, offs, lens, keys, stream=spp)
        torch.cuda.synchronize()
        assert int((ret != 0).sum().item()) == 0
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["cudil", "reference"], default="cudil")
    ap.add_argument("--mode", type=int, default=2, choices=[2, 3, 5])
    ap.add_argument("--batch", type=int, default=10000)
    ap.add_argument("--thresholds", type=int, nargs="+", default=[4096, 8192, 16384, 32768],
                    help="exec-slot counts tried for the plain path (the fastest is used)")
    ap.add_argument("--engine-threads", type=int, default=0, help="fused engine block size (0 = tuned default)")
    ap.add_argument("--spec-slots", type=int, default=0, help="fused signer attempts in flight (0 = tuned default)")
    ap.add_argument("--sign-kernel", type=int, default=-1,
                    help="fused signer kernel: 0 phased, 1..4 async 256/64, 512/128, 640/160, 768/192, "
                         "5 phased with one wide block per SM (-1 = tuned default)")
    ap.add_argument("--quick", action="store_true", help="headline only (skip configs 1-4)")
    ap.add_argument("--workload", default="headline",
                    choices=["headline", "serve", "configs", "fused-sign", "fused-verify", "ntt", "plain-sign",
                             "d3-sign"],
                    help="headline = the bench line; serve / configs = those legs alone; the others are small "
                         "self-checking cases for ncu")
    ap.add_argument("--e2e-chunks", type=int, default=4,
                    help="chunks the end-to-end step uploads the secret keys in (each chunk's cache build "
                         "overlaps the next chunk's copy)")
    ap.add_argument("--serve-keys", type=int, default=4096, help="resident keys per parameter set (serving)")
    ap.add_argument("--serve-requests", type=int, default=200_000, help="distinct requests of the serving trace")
    ap.add_argument("--serve-seconds", type=float, default=5.0, help="arrival window per serving point")
    ap.add_argument("--serve-fracs", type=float, nargs="+", default=[0.5, 0.8, 0.85, 0.9],
                    help="offered load as fractions of the saturation throughput")
    ap.add_argument("--serve-slots", type=int, default=2,
                    help="batch slots per (parameter set, op) lane; busier lanes get more in proportion to their "
                         "share of the requests")
    ap.add_argument("--serve-max-batch", type=int, default=8192)
    ap.add_argument("--serve-budget-gib", type=float, default=48.0, help="device-memory budget of the server")
    ap.add_argument("--cpu-seconds", type=float, default=12.0)
    ap.add_argument("--ref-sample", type=int, default=4000)
    ap.add_argument("--no-cpu", action="store_true")
    args = ap.parse_args()
    if args.warmup < 3:
        log("[bench] warmup raised to 3 (minimum)")
        args.warmup = 3
    if args.impl == "reference":
        res = run_reference(args)
    elif args.workload == "serve":
        import numpy as np
        res = {"configs": {"serve_mixed": run_serve(args, np)}}
    elif args.workload == "configs":
        import numpy as np
        import torch

        from cudilithium_b200 import _lib
        dev = torch.device("cuda", 0)
        spp = torch.cuda.current_stream().cuda_stream
        res = {"configs": run_configs(args, torch, np, _lib.lib, _lib, dev, spp, 0,
                                      measure_alu_peak(_lib.lib, dev, spp))}
    elif args.workload != "headline":
        res = run_profile_case(args)
    else:
        res = run_gpu(args)
    if res:
        print(json.dumps(res), flush=True)


if __name__ == "__main__":
    main()
