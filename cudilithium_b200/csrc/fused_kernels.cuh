// Fused / persistent form of the batched path (no reference counterpart; the reference drives
// every rejection round from the host, src/api.cu:218-441).
//
//  * Per-key resident cache (built once per key, reused by every message of that key):
//      secret rows  [rho | K | tr | pad..256 | A_hat (K*L polys) | s1_hat | s2_hat | t0_hat]
//      public rows  [rho | tr | pad..256 | A_hat (K*L polys) | t1_hat = NTT(t1 * 2^d)]
//  * k_fused_prehash  one thread (few messages: a pair) per message, longest first: mu, rho' = H(K||mu)
//  * k_fused_sign     ONE persistent kernel for all signing attempts of a batch.  Block b owns the
//                     items b, b + grid, ...; every item has a next-nonce counter, so its nonces are
//                     issued in increasing order, and attempts whose item already has an accepted
//                     smaller nonce are skipped.  Each block claims up to A attempts of its pending
//                     items at a time (speculating more deeply as they run out) and runs them in two
//                     phases per iteration: a Keccak phase (ExpandMask, thread per (attempt, j)
//                     stream; the challenge, thread per attempt) and an NTT phase (w = A*y, 16-thread
//                     group per attempt; rejection checks + hints, warp per attempt).  An accepted
//                     attempt lowers the item's best nonce with atomicMin and, under a per-item lock
//                     with a bounded spin, publishes its signature only if it still holds the
//                     minimum -- the same smallest-accepted-nonce result as deterministic signing
//                     (src/api.cu:388-411).  k_fused_sign_async (fused_sign_async.cuh) runs the same
//                     queue without block-wide phases.
//
// The staged signer (fused_sign_staged.cuh) and the verifier (fused_verify.cuh) work on the same caches.
#pragma once

#include "keypair_kernels.cuh"
#include "verify_kernels.cuh"

namespace cudil {

template <int MODE>
struct Cache {
    using PM = P<MODE>;
    static constexpr int K = PM::K, L = PM::L;
    static constexpr size_t POLY = N * sizeof(int32_t);
    // secret-key rows
    static constexpr size_t SK_RHO = 0, SK_KEY = 32, SK_TR = 64;
    static constexpr size_t SK_MAT = 256;
    static constexpr size_t SK_S1 = SK_MAT + (size_t)K * L * POLY;
    static constexpr size_t SK_S2 = SK_S1 + (size_t)L * POLY;
    static constexpr size_t SK_T0 = SK_S2 + (size_t)K * POLY;
    static constexpr size_t SK_ROW = SK_T0 + (size_t)K * POLY;
    // public-key rows
    static constexpr size_t PK_RHO = 0, PK_TR = 32;
    static constexpr size_t PK_MAT = 256;
    static constexpr size_t PK_T1 = PK_MAT + (size_t)K * L * POLY;
    static constexpr size_t PK_ROW = PK_T1 + (size_t)K * POLY;
    // per-message prologue output: mu | rho'
    static constexpr size_t ITEM_BYTES = 128;
    // per-attempt slot of the persistent signer
    static constexpr size_t SL_Y = 0;
    static constexpr size_t SL_W0 = align256((size_t)L * PM::POLYZ_PACKED);
    static constexpr size_t SL_W1P = SL_W0 + (size_t)K * POLY;
    static constexpr size_t SL_CM = SL_W1P + align256(PM::W1PACKED_BYTES);
    static constexpr size_t SL_SIG = SL_CM + 256;
    // w1 as bytes, thread-major (byte 16 t + m = coefficient t + 16 m), for the hint computation
    static constexpr size_t SL_W1B = SL_SIG + align256(PM::SIG_BYTES);
    static constexpr size_t SLOT = SL_W1B + (size_t)K * 256;
};

// Queue / status block shared by the engine kernels (one per engine, device memory).
struct FusedQueue {
    unsigned int done_items;
    // bit 0: a bounded publication-lock wait gave up; bit 1: an item reached its nonce limit (with no
    // accepted nonce its signature row is not written); bit 2: an asynchronous signer block gave up
    // after its idle-poll limit
    unsigned int error;
    unsigned long long attempts;
    unsigned int n;            // items in the current batch
    unsigned int pad;
    unsigned long long intt;   // inverse NTTs run by the rejection checks (for work accounting)
    unsigned int iters;        // signer block-iterations (summed over blocks)
    unsigned int pad2;
    unsigned long long cyc[4]; // signer cycles per phase summed over blocks: claim, keccak, ntt, total
    // asynchronous signer, summed over warps: cycles in reject / w / challenge / ExpandMask / claim /
    // idle polls, then the number of each
    unsigned long long jobs[12];
    // seeded randomized signing (set per batch by the host): rho' of item i is
    // SHAKE256(rho_seed || le64(rho_counter + i), 64); rho_seeded = 0 keeps the other rho' sources
    unsigned long long rho_counter;
    unsigned rho_seeded;
    unsigned pad3;
    uint32_t rho_seed[8];
};

// ------------------------------------------------------------------ cache builders

// Secret rows from packed secret keys (dense, SK_BYTES each): rho, K, tr copied; s1, s2, t0
// unpacked and transformed.  One group per polynomial (+ group p == L+2K copies the seeds).
template <int MODE>
__global__ void __launch_bounds__(kBlock) k_cache_sk(const uint8_t *sk, uint8_t *rows, size_t pitch, int n) {
    using PM = P<MODE>;
    using C = Cache<MODE>;
    constexpr int K = PM::K, L = PM::L, NP = L + 2 * K + 1;
    __shared__ int32_t sm[kGroupsPerBlock * NTT_SMEM_WORDS];
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const int it = gid / NP, p = gid % NP;
    if (it >= n) return;
    Group g = make_group(sm, threadIdx.x >> 4);
    const uint8_t *s = sk + (size_t)it * PM::SK_BYTES;
    uint8_t *row = rows + (size_t)it * pitch;
    if (p == NP - 1) {
        // rho | K | tr are the first 96 bytes of sk
        for (int b = g.t; b < 96; b += 16) row[b] = s[b];
        return;
    }
    int32_t x[16];
    unpack_secret<MODE>(x, s, p, g.t);
    const size_t dst = p < L ? C::SK_S1 + (size_t)p * C::POLY
                             : (p < L + K ? C::SK_S2 + (size_t)(p - L) * C::POLY : C::SK_T0 + (size_t)(p - L - K) * C::POLY);
    ntt16s(x, g.sm, g.gmask, g.t);
    store16_chunks(reinterpret_cast<int32_t *>(row + dst), x, g.t);
}

// Public rows: tr = H(pk) and rho (thread or thread pair per key) ...
template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kBlock) k_cache_pk_tr(const uint8_t *pk, uint8_t *rows, size_t pitch, int n) {
    using PM = P<MODE>;
    using C = Cache<MODE>;
    using Sp = Shake256<PAIR>;
    const int it = (blockIdx.x * blockDim.x + threadIdx.x) / Sp::LANES;
    const bool on = it < n;
    if (!PAIR && !on) return;
    const uint8_t *p = pk + (size_t)(on ? it : 0) * PM::PK_BYTES;
    uint8_t *row = rows + (size_t)(on ? it : 0) * pitch;
    // pk rows of a dense array may start at any byte
    struct Src {
        const uint8_t *p;
        bool words;  // 4-byte aligned
        __device__ uint2 lane(long long g) const {
            if (words && g * 8 + 8 <= PM::PK_BYTES) {
                const uint32_t *q = reinterpret_cast<const uint32_t *>(p + g * 8);
                return make_uint2(q[0], q[1]);
            }
            return load_lane_bytes(p + g * 8, (int)(PM::PK_BYTES - g * 8));
        }
        __device__ uint32_t word(long long g, int h) const {
            const long long off = g * 8 + 4 * h;
            if (words && off + 4 <= PM::PK_BYTES) return *reinterpret_cast<const uint32_t *>(p + off);
            return off < PM::PK_BYTES ? load_lane_bytes(p + off, (int)(PM::PK_BYTES - off)).x : 0u;
        }
    } src{p, (reinterpret_cast<uintptr_t>(p) & 3u) == 0u};
    Sp sp;
    sp.hash(src, PM::PK_BYTES, on);
    if (!on) return;
    sp.template store<4>(row + C::PK_TR);
    if (!PAIR || sp.half() == 0)
        for (int b = 0; b < 32; ++b) row[C::PK_RHO + b] = p[b];
}

// ... and t1_hat = NTT(t1 * 2^d) (group per polynomial).
template <int MODE>
__global__ void __launch_bounds__(kBlock) k_cache_pk_t1(const uint8_t *pk, uint8_t *rows, size_t pitch, int n) {
    using PM = P<MODE>;
    using C = Cache<MODE>;
    constexpr int K = PM::K;
    __shared__ int32_t sm[kGroupsPerBlock * NTT_SMEM_WORDS];
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const int it = gid / K, i = gid % K;
    if (it >= n) return;
    Group g = make_group(sm, threadIdx.x >> 4);
    const uint8_t *t1p = pk + (size_t)it * PM::PK_BYTES + SEEDBYTES + (size_t)i * POLYT1_PACKED;
    int32_t x[16];
    if ((reinterpret_cast<uintptr_t>(t1p) & 3u) == 0u) {
        uint32_t v[16];
        unpack_strided<10>(v, t1p, g.t);
#pragma unroll
        for (int m = 0; m < 16; ++m) x[m] = (int32_t)(v[m] << D);
    } else {  // the last key's words would reach past the buffer
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int bit = (g.t + 16 * m) * 10, byte = bit >> 3, sh = bit & 7;
            const uint32_t v = ((uint32_t)t1p[byte] | ((uint32_t)t1p[byte + 1] << 8)) >> sh;  // sh + 10 <= 16
            x[m] = (int32_t)((v & 0x3FFu) << D);
        }
    }
    ntt16s(x, g.sm, g.gmask, g.t);
    store16_chunks(reinterpret_cast<int32_t *>(rows + (size_t)it * pitch + C::PK_T1 + (size_t)i * C::POLY), x, g.t);
}

// ------------------------------------------------------------------ per-batch prologue

// Messages live in one device buffer at 8-byte aligned offsets.  order[] lists the items longest
// first so a warp's messages have similar lengths (nullptr: they already are).
struct MsgRefs {
    const uint8_t *msgs;
    const unsigned long long *offsets;
    const unsigned int *mlens;
    const unsigned int *key_idx;
    const unsigned int *order;
    const uint8_t *rhoprime;  // randomized signing: 64 bytes per item (dense); nullptr = SHAKE256(K || mu)
    unsigned nkeys;           // key-cache rows allocated (bound of key_idx[])
};

// One warp per block, so that the warps holding the longest messages (the order is longest first)
// spread over all SMs.
constexpr int kPrehashBlock = 32;

// Items order[first .. first + count).  Also clears the nclear 16-byte units at `clear` (the staged signer's
// round counters) for the kernels that follow.
template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kPrehashBlock) k_fused_prehash(const uint8_t *cache, size_t cpitch, MsgRefs mr,
                                                                 uint8_t *items, const FusedQueue *q, unsigned first,
                                                                 unsigned count, uint4 *clear, unsigned nclear) {
    using C = Cache<MODE>;
    using Sp = Shake256<PAIR>;
    constexpr unsigned PER = kPrehashBlock / Sp::LANES;  // items of a block
    if (blockIdx.x == 0)
        for (unsigned k = threadIdx.x; k < nclear; k += kPrehashBlock) clear[k] = make_uint4(0u, 0u, 0u, 0u);
    for (unsigned r0 = blockIdx.x * PER; r0 < count; r0 += gridDim.x * PER) {
        const unsigned r = r0 + threadIdx.x / Sp::LANES;
        bool on = r < count;
        const unsigned it = on ? (mr.order ? mr.order[first + r] : first + r) : 0u;
        on = on && bc_ok(it < q->n && mr.key_idx[it] < mr.nkeys, BC_PREHASH_ITEM);
        if (!PAIR && !on) continue;
        const uint8_t *row = cache + (on ? (size_t)mr.key_idx[it] * cpitch : 0);
        const long long ml = on ? (long long)mr.mlens[it] : 0;
        TwoPart src{row + C::SK_TR, 4, mr.msgs + (on ? mr.offsets[it] : 0), ml};
        Sp sp;
        sp.hash(src, SEEDBYTES + ml, on);
        uint8_t *out = items + (size_t)it * C::ITEM_BYTES;
        if (on) sp.template store<8>(out);
        if (q->rho_seeded) {
            if (!on || (PAIR && sp.half())) continue;
            uint32_t seed[8];
#pragma unroll
            for (int w = 0; w < 8; ++w) seed[w] = q->rho_seed[w];
            uint2 rp[8];
            derive_rhoprime(rp, seed, q->rho_counter + it);
#pragma unroll
            for (int w = 0; w < 8; ++w) reinterpret_cast<uint2 *>(out)[8 + w] = rp[w];
            continue;
        }
        if (mr.rhoprime) {
            if (!on || (PAIR && sp.half())) continue;
            const uint8_t *rp = mr.rhoprime + (size_t)it * CRHBYTES;
#pragma unroll 1
            for (int b = 0; b < CRHBYTES; ++b) out[64 + b] = rp[b];
            continue;
        }
        rhoprime_from_mu(sp, row + C::SK_KEY);
        if (on) sp.template store<8>(out + 64);
    }
}

// Resets the queue and the per-item winner state of q->n items (n set by the host copy).
static __global__ void k_fused_init(FusedQueue *q, unsigned *best, unsigned *locks, unsigned *next_nonce,
                                    unsigned *inflight) {
    const unsigned n = q->n;
    for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        best[i] = 0xFFFFFFFFu;
        locks[i] = 0u;
        next_nonce[i] = 0u;
        inflight[i] = 0u;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        q->done_items = 0;
        q->error = 0;
        q->attempts = 0;
        q->intt = 0;
        q->iters = 0;
        for (int i = 0; i < 4; ++i) q->cyc[i] = 0;
        for (int i = 0; i < 12; ++i) q->jobs[i] = 0;
    }
}

// ------------------------------------------------------------------ persistent signer
//
// Work queue.  Block b owns the items b, b + grid, b + 2*grid, ... and schedules them itself, so
// refilling slots touches no shared counter.  Every owned item has a next-nonce counter and an
// in-flight counter; a claim gives pending items (no accepted nonce yet) their next nonce, at most
// D in flight per item, D = spec_slots / pending (1..64).  While a block owning many items has many
// pending, D = 1 and each batch takes half of them, so the two batches in flight hold different
// items and no attempt is wasted (blocks owning fewer than A / 4 items keep D >= 2 so both
// batches stay fed); as pending items run out D grows up to 64, so the last items of a block are
// speculated deeply instead of taking one rejection round after another.
// Nonces of an item are issued in increasing order and every issued attempt completes before the
// block exits, so the winner -- the smallest accepted nonce -- is the deterministic signature.
//
struct FusedSignArgs {
    const uint8_t *cache;
    size_t cpitch;
    const unsigned *key_idx;
    const uint8_t *items;
    uint8_t *sig_out;
    size_t sig_pitch;
    uint8_t *scratch;
    FusedQueue *q;
    unsigned *best, *locks, *next_nonce, *inflight;
    unsigned spec_slots;  // per-block target of attempts in flight (<= 2 * THREADS)
    // bounds of the device-side loops (run-time so that a host can shorten them):
    unsigned nonce_limit;  // nonces an item may use (the 16-bit nonce field allows 65536)
    unsigned lock_spins;   // tries for a per-item publication lock before giving up (error bit 0)
    unsigned idle_polls;   // empty polls before an asynchronous signer block gives up (error bit 2)
    unsigned nkeys;        // key-cache rows allocated (bound of key_idx[])
};

// Sentinel best nonce of an item that used all its nonces without an accepted attempt: below the
// "pending" value 0xFFFFFFFF, above every real nonce, so the item counts as finished (error bit 1).
constexpr unsigned kNonceExhausted = 0xFFFFFFFEu;

template <int MODE, int THREADS>
struct FusedSignSmem {
    using PM = P<MODE>;
    static constexpr int G = THREADS / 16;
    static constexpr size_t CTRL = 4 * THREADS * sizeof(unsigned) + 256;
    static constexpr size_t PH_N = (size_t)G * (PM::L * N * 4 + NTT_SMEM_WORDS * 4);
    static constexpr size_t PH_K = (size_t)THREADS * SIB_WORDS * 4;
    static constexpr size_t BYTES = CTRL + (PH_N > PH_K ? PH_N : PH_K);
};

// default bounds of the signer's loops (FusedSignArgs)
constexpr unsigned kNonceLimit = 1u << 16;
constexpr unsigned kLockSpinLimit = 1u << 22;  // x ~64 ns sleeps

// Copies a staged signature (256-byte aligned words, whole 256-byte units) to its output row with NT
// cooperating threads (t = 0 .. NT-1).  Rows start at any byte (a Dilithium3 or Dilithium5 signature is no whole
// number of words): the row's aligned words are put together from two staged ones, and only the bytes before the
// first and after the last of them are stored singly.  Word stores matter when the output is pinned host memory
// written over PCIe: 20 000 Dilithium3 signatures 44.5 ms with such rows stored byte by byte, 5.1 ms this
// way.  Eight words per thread are in flight before any is stored.
template <int BYTES, int NT>
__device__ __forceinline__ void publish_signature(uint8_t *dst, const uint32_t *src, int t) {
    const unsigned head = (0u - (unsigned)(reinterpret_cast<uintptr_t>(dst))) & 3u;  // bytes before the first aligned word
    const int nfull = (BYTES - (int)head) / 4, tail = (BYTES - (int)head) % 4;
    uint32_t *d = reinterpret_cast<uint32_t *>(dst + head);
    if (head == 0u) {  // (loads of its own: 0.7% of 65 536 Dilithium2 signatures)
#pragma unroll 1
        for (int w0 = 0; w0 < nfull; w0 += 8 * NT) {
            uint32_t v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int w = w0 + t + NT * k;
                v[k] = w < nfull ? src[w] : 0u;
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int w = w0 + t + NT * k;
                if (w < nfull) d[w] = v[k];
            }
        }
    } else {
        // aligned word w holds the signature's bytes head + 4 w ..: the end of staged word w, the start of w + 1
#pragma unroll 1
        for (int w0 = 0; w0 < nfull; w0 += 4 * NT) {
            uint32_t lo[4], hi[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int w = w0 + t + NT * k;
                lo[k] = w < nfull ? src[w] : 0u;
                hi[k] = w < nfull ? src[w + 1] : 0u;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int w = w0 + t + NT * k;
                if (w < nfull) d[w] = __funnelshift_r(lo[k], hi[k], 8u * head);
            }
        }
    }
    const uint8_t *sb = reinterpret_cast<const uint8_t *>(src);
    if (t < (int)head) dst[t] = sb[t];
    if (t < tail) dst[(int)head + 4 * nfull + t] = sb[(int)head + 4 * nfull + t];
}

template <int MODE, int THREADS>
__global__ void __launch_bounds__(THREADS, 512 / THREADS) k_fused_sign(FusedSignArgs arg) {
    using PM = P<MODE>;
    using C = Cache<MODE>;
    constexpr int K = PM::K, L = PM::L, OMEGA = PM::OMEGA, A = THREADS;
    enum { CT_PEND = 0, CT_KJOB, CT_NJOB, CT_NA0, CT_NA1 };
    extern __shared__ __align__(16) uint8_t fs_smem[];
    unsigned *s_item = reinterpret_cast<unsigned *>(fs_smem);   // [2][A]
    unsigned *s_nonce = s_item + 2 * A;                          // [2][A]
    unsigned *s_ctl = s_nonce + 2 * A;                           // CT_* and per-warp counts
    uint8_t *ph = fs_smem + FusedSignSmem<MODE, THREADS>::CTRL;
    FusedQueue *q = arg.q;
    const int tid = threadIdx.x, gi = tid >> 4, lane = tid & 31, lane_off = lane & 16;
    const unsigned n = q->n;
    uint8_t *my_slots = arg.scratch + (size_t)blockIdx.x * 2 * A * C::SLOT;
    auto slot_of = [&](int buf, int a) { return my_slots + ((size_t)buf * A + a) * C::SLOT; };

    Group g;
    g.t = tid & 15;
    g.gmask = 0xFFFFu << lane_off;
    // Dilithium2's signer holds the inlined transforms in its register budget without spilling, so
    // loads issued before a transform overlap it; the larger parameter sets call the out-of-line
    // copies, which keep register use and code size down.
    auto fwd = [&](int32_t (&x)[16]) {
        if constexpr (MODE == 2)
            ntt16s(x, g.sm, g.gmask, g.t);
        else
            ntt16_ool(x, g.sm, g.gmask, g.t);
    };
    auto inv = [&](int32_t (&x)[16]) {
        if constexpr (MODE == 2)
            intt16s(x, g.sm, g.gmask, g.t);
        else
            intt16_ool(x, g.sm, g.gmask, g.t);
    };

    // ---------------- claim: fill batch `buf` with up to A attempts of this block's items
    // (block-collective; warp 0 scans the owned items, one item per lane per pass)
    const unsigned grid = gridDim.x, b0 = blockIdx.x;
    const unsigned n_own = (b0 < n) ? (n - b0 + grid - 1) / grid : 0u;
    auto claim = [&](int buf) {
        if (tid < 32) {
            const unsigned pend = s_ctl[CT_PEND];
            unsigned D = 0;
            if (pend) {
                // depth 1 (alternating halves) needs enough owned items to fill both batches
                const unsigned dmin = (n_own >= (unsigned)A / 4u) ? 1u : 2u;
                const unsigned t = arg.spec_slots / pend;
                D = t < dmin ? dmin : (t > 64u ? 64u : t);
            }
            // With one attempt per item (D == 1) a batch takes at most half of the pending items, so
            // the two batches in flight hold different items and no attempt is speculative.
            const unsigned cap = (D == 1u) ? ((pend + 1u) / 2u < (unsigned)A ? (pend + 1u) / 2u : (unsigned)A) : (unsigned)A;
            unsigned filled = 0;
            // An item with f attempts in flight gets D - f more (none when f >= D).  When all of
            // them fit the batch (D * pend <= cap), one scan hands each item its attempts with one
            // atomic on its nonce counter; otherwise pass p gives one more attempt to the items
            // with at most p in flight, so a full batch spreads its slots over the items.
            const bool one_scan = D >= 2u && D * pend <= cap;
            unsigned issued = 0;  // this lane's attempts
            auto place = [&](unsigned pos, unsigned i, unsigned nn) {
                s_item[buf * A + pos] = i;
                if (nn < arg.nonce_limit) {
                    s_nonce[buf * A + pos] = nn;
                    ++issued;
                } else {
                    // every nonce used without acceptance (never for honest keys at the default
                    // limit): the slot becomes a no-op, and the first lane to get here marks the
                    // item finished so that the block can exit
                    s_nonce[buf * A + pos] = 0xFFFFFFFFu;
                    if (atomicCAS(arg.best + i, 0xFFFFFFFFu, kNonceExhausted) == 0xFFFFFFFFu) {
                        atomicOr(&q->error, 2u);
                        atomicSub(&s_ctl[CT_PEND], 1u);
                    }
                }
            };
#pragma unroll 1
            for (unsigned k0 = 0; one_scan && k0 < n_own; k0 += 32) {
                const unsigned k = k0 + lane, i = b0 + k * grid;
                unsigned want = 0;
                if (k < n_own) {
                    const unsigned bi = __ldcg(arg.best + i), fi = __ldcg(arg.inflight + i);
                    want = (bi == 0xFFFFFFFFu && fi < D) ? D - fi : 0u;
                }
                unsigned incl = want;  // inclusive prefix sum over the warp
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const unsigned v = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                    if (lane >= o) incl += v;
                }
                const unsigned pos0 = filled + incl - want;
                // (D * pend <= cap keeps every position below cap; the clamp only guards the bound)
                const unsigned take = pos0 >= cap ? 0u : (want < cap - pos0 ? want : cap - pos0);
                if (take) {
                    const unsigned nn = atomicAdd(arg.next_nonce + i, take);
                    atomicAdd(arg.inflight + i, take);
#pragma unroll 1
                    for (unsigned r = 0; r < take; ++r) place(pos0 + r, i, nn + r);
                }
                filled += __shfl_sync(0xFFFFFFFFu, incl, 31);
                if (filled > cap) filled = cap;
            }
#pragma unroll 1
            for (unsigned pass = 0; !one_scan && pass < D && filled < cap; ++pass) {
#pragma unroll 1
                for (unsigned k0 = 0; k0 < n_own && filled < cap; k0 += 32) {
                    const unsigned k = k0 + lane, i = b0 + k * grid;
                    bool ok = false;
                    if (k < n_own) {
                        // both loads issued together (one round trip, not two dependent ones)
                        const unsigned bi = __ldcg(arg.best + i), fi = __ldcg(arg.inflight + i);
                        ok = bi == 0xFFFFFFFFu && fi <= pass;
                    }
                    const unsigned bal = __ballot_sync(0xFFFFFFFFu, ok);
                    const unsigned pos = filled + __popc(bal & ((1u << lane) - 1u));
                    if (ok && pos < cap) {
                        const unsigned nn = atomicAdd(arg.next_nonce + i, 1u);
                        atomicAdd(arg.inflight + i, 1u);
                        place(pos, i, nn);
                    }
                    filled += __popc(bal);
                    if (filled > cap) filled = cap;
                }
            }
            issued = __reduce_add_sync(0xFFFFFFFFu, issued);
            if (lane == 0) {
                s_ctl[CT_NA0 + buf] = filled;
                s_ctl[CT_KJOB] = 0;
                s_ctl[CT_NJOB] = 0;
                if (issued) atomicAdd(&q->attempts, (unsigned long long)issued);
            }
        }
        __syncthreads();
    };

    // ---------------- Keccak phase: challenge of batch cb (jobs < na_c), ExpandMask of batch nb
    auto keccak_phase = [&](int cb, int na_c, int nb, int na_n) {
        uint32_t *sib = reinterpret_cast<uint32_t *>(ph);
        const uint32_t *mask = sib_result<THREADS>(sib, tid);
        // ExpandMask jobs start at a multiple of 32, so no warp holds both job types (a warp runs
        // divergent branches one after the other: a mixed warp would take 8 + 5 permutations)
        const int cpad = (na_c + 31) & ~31;
        const int total = cpad + na_n * L;
        // a warp takes 32 consecutive jobs at a time, so its lanes run the same job type together
#pragma unroll 1
        for (;;) {
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(&s_ctl[CT_KJOB], 32u);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if ((int)base >= total) break;
            const int job = (int)base + lane;
            // attempts above an already accepted nonce of their item are skipped (they cannot win)
            if (job < na_c) {
                const unsigned item = bc_ok(job < A, BC_SIGN_SLOT) ? s_item[cb * A + job] : 0xFFFFFFFFu;
                if (bc_ok(item < n, BC_SIGN_SLOT) && !(__ldcg(arg.best + item) < s_nonce[cb * A + job])) {
                    uint8_t *slot = slot_of(cb, job);
                    uint32_t al[25], ah[25];
                    TwoPart src{arg.items + (size_t)item * C::ITEM_BYTES, 8, slot + C::SL_W1P, PM::W1PACKED_BYTES};
                    shake_absorb<SHAKE256_RATE>(al, ah, src, CRHBYTES + PM::W1PACKED_BYTES);
                    keccak_f1600(al, ah);
                    uint2 ct[4];
#pragma unroll
                    for (int w = 0; w < 4; ++w) ct[w] = make_uint2(al[w], ah[w]);
                    uint2 *sg = reinterpret_cast<uint2 *>(slot + C::SL_SIG);
#pragma unroll
                    for (int w = 0; w < 4; ++w) sg[w] = ct[w];
                    sample_in_ball<PM::TAU, THREADS>(ct, sib, tid);
                    uint4 *mo = reinterpret_cast<uint4 *>(slot + C::SL_CM);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        mo[k] = make_uint4(mask[(4 * k) * THREADS], mask[(4 * k + 1) * THREADS], mask[(4 * k + 2) * THREADS],
                                           mask[(4 * k + 3) * THREADS]);
                }
            } else if (job >= cpad && job < total) {
                const int idx = job - cpad, a = idx / L, j = idx % L;
                const bool slot_ok = bc_ok(a < A, BC_SIGN_SLOT);
                const unsigned item = slot_ok ? s_item[nb * A + a] : 0xFFFFFFFFu, nonce = slot_ok ? s_nonce[nb * A + a] : 0u;
                if (bc_ok(item < n, BC_SIGN_SLOT) && !(__ldcg(arg.best + item) < nonce)) {
                    uint2 rhop[8];
                    ld_lanes(rhop, arg.items + (size_t)item * C::ITEM_BYTES + 64);
                    expand_mask_stream<MODE>(slot_of(nb, a) + C::SL_Y + (size_t)j * PM::POLYZ_PACKED, rhop,
                                             (uint32_t)(L * nonce + j));
                }
            }
            __syncwarp();  // every lane runs the same grab / sync sequence
        }
    };

    // rejection checks, hints and publication of one attempt (warp-collective).  The two groups
    // of the warp take the attempt's polynomials in pairs (poly 2p + half), so they follow the same
    // control flow: a rejection ends the job for the whole warp, and no group waits for another
    // group's longer attempt.
    auto reject_job = [&](int cb, int a) {
        // (range checks of the bounds-checked build: every value is the same across the warp)
        if (!bc_ok(a < A, BC_SIGN_SLOT)) return;
        const unsigned item = s_item[cb * A + a], nonce = s_nonce[cb * A + a];
        if (!bc_ok(item < n, BC_SIGN_SLOT)) return;
        // one decision per warp: out-of-range nonce, or a smaller nonce of the item already accepted
        bool skip = nonce > 0xFFFFu || __ldcg(arg.best + item) < nonce;
        skip = __shfl_sync(0xFFFFFFFFu, skip, 0);
        const unsigned key = arg.key_idx[item];
        if (skip || !bc_ok(key < arg.nkeys, BC_SIGN_KEY)) {
            if (lane == 0) atomicSub(arg.inflight + item, 1u);
            return;
        }
        uint8_t *slot = slot_of(cb, a);
        const uint8_t *row = arg.cache + (size_t)key * arg.cpitch;
        g.sm = reinterpret_cast<int32_t *>(ph) + (size_t)gi * (L * N + NTT_SMEM_WORDS) + L * N;
        uint32_t masks[16];
        {
            const uint4 *mi = reinterpret_cast<const uint4 *>(slot + C::SL_CM);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint4 v = mi[k];
                masks[4 * k] = v.x;
                masks[4 * k + 1] = v.y;
                masks[4 * k + 2] = v.z;
                masks[4 * k + 3] = v.w;
            }
        }
        // both groups transform c (same data, same instructions)
        int32_t ch[16];
        challenge_strided(ch, masks, g.t);
        fwd(ch);
#pragma unroll
        for (int m = 0; m < 16; ++m) ch[m] = scale_f(ch[m]);
        const int32_t *s1 = reinterpret_cast<const int32_t *>(row + C::SK_S1);
        const int32_t *s2 = reinterpret_cast<const int32_t *>(row + C::SK_S2);
        const int32_t *t0 = reinterpret_cast<const int32_t *>(row + C::SK_T0);
        uint8_t *hs = slot + C::SL_SIG + PM::SIG_H;
        const int half = lane_off >> 4;
        bool rejected = false;
        int n_intt = 0, cnt = 0;
        // Acceptance needs every check to pass, so the checks run most selective first: pair steps
        // of the r0_i (r0 replaces w0 in the slot, for the hints), then of the z_j, then of the
        // ct0_i with the hints.  K is even for every parameter set; L is odd for two of them, so
        // the last z pair may leave the second group without a polynomial (it transforms zeros
        // and stores nothing).  While one step transforms, the next step's key rows and (inlined
        // transforms) this step's slot data are in flight.
        constexpr int PR = K / 2, PZ = (L + 1) / 2, NSTEP = 2 * PR + PZ;
        auto operand = [&](int step) -> const int32_t * {
            if (step < PR) return s2 + (size_t)(2 * step + half) * N;
            if (step < PR + PZ) {
                const int j = 2 * (step - PR) + half;
                return s1 + (size_t)(j < L ? j : L - 1) * N;
            }
            return t0 + (size_t)(2 * (step - PR - PZ) + half) * N;
        };
        int32_t nx[16];
        load16_chunks(nx, operand(0), g.t);
#pragma unroll 1
        for (int step = 0; step < NSTEP; ++step) {
            const bool is_r0 = step < PR, is_z = !is_r0 && step < PR + PZ;
            const int k = 2 * (is_r0 ? step : (is_z ? step - PR : step - PR - PZ)) + half;  // i, or j for z
            const bool act = !is_z || k < L;
            int32_t x[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) x[m] = act ? montmul(ch[m], nx[m]) : 0;
            if (step + 1 < NSTEP) load16_chunks(nx, operand(step + 1), g.t);
            int32_t *w0 = reinterpret_cast<int32_t *>(slot + C::SL_W0) + (size_t)(is_z ? 0 : k) * N;
            const uint8_t *yp = slot + C::SL_Y + (size_t)(act ? k : 0) * PM::POLYZ_PACKED;
            int32_t pre[16];
            // the slot data of the step: with the inlined transform it is in flight across it; the
            // out-of-line transform would spill a load held across the call, so there it is read
            // afterwards
            auto load_pre = [&] {
                if (is_z) {
                    unpack_z_strided<MODE>(pre, yp, g.t);
#pragma unroll
                    for (int m = 0; m < 16; ++m) pre[m] = act ? pre[m] : 0;
                } else {
                    load16_strided(pre, w0, g.t);
                }
            };
            if constexpr (MODE == 2) load_pre();
            inv(x);
            n_intt += act ? 1 : 0;
            if constexpr (MODE != 2) load_pre();
            bool bad = false;
            if (is_z) {
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    x[m] = reduce32(x[m] + pre[m]);
                    bad |= act && exceeds(x[m], PM::GAMMA1 - PM::BETA);
                }
                if (__ballot_sync(0xFFFFFFFFu, bad)) {
                    rejected = true;
                    break;
                }
                int32_t zc[16];
                strided_to_contig(g, x, zc);
                if (act) {
                    uint32_t v[16];
#pragma unroll
                    for (int m = 0; m < 16; ++m) v[m] = (uint32_t)(PM::GAMMA1 - zc[m]);
                    pack16_words<PM::Z_BITS>(
                        reinterpret_cast<uint32_t *>(slot + C::SL_SIG + PM::SIG_Z + (size_t)k * PM::POLYZ_PACKED + g.t * 2 * PM::Z_BITS), v);
                }
            } else if (is_r0) {
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    pre[m] = reduce32(pre[m] - x[m]);
                    bad |= exceeds(pre[m], PM::GAMMA2 - PM::BETA);
                }
                if (__ballot_sync(0xFFFFFFFFu, bad)) {
                    rejected = true;
                    break;
                }
                store16_strided(w0, pre, g.t);
            } else {
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    x[m] = reduce32(x[m]);
                    bad |= exceeds(x[m], PM::GAMMA2);
                }
                if (__ballot_sync(0xFFFFFFFFu, bad)) {
                    rejected = true;
                    break;
                }
                // hint bits of poly k: bit m of hb = hint of coefficient t + 16 m
                const uint8_t *w1p = slot + C::SL_W1P + (size_t)k * PM::POLYW1_PACKED;
                unsigned hb = 0;
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    const int32_t w1 = (int32_t)get_bits(w1p, (g.t + 16 * m) * PM::W1_BITS, PM::W1_BITS);
                    hb |= make_hint<MODE>(pre[m] + x[m], w1) << m;
                }
                // hint counts of both polynomials of the pair (sums over each group), then the
                // positions in ascending coefficient order: poly 2p first, then poly 2p + 1
                int tot = __popc(hb);
#pragma unroll
                for (int o = 8; o >= 1; o >>= 1) tot += __shfl_xor_sync(0xFFFFFFFFu, tot, o);
                const int tot0 = __shfl_sync(0xFFFFFFFFu, tot, 0), tot1 = __shfl_sync(0xFFFFFFFFu, tot, 16);
                if (cnt + tot0 + tot1 > OMEGA) {
                    rejected = true;
                    break;
                }
                int idx = cnt + (half ? tot0 : 0);
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    const unsigned bit = (hb >> m) & 1u;
                    const unsigned bal = (__ballot_sync(0xFFFFFFFFu, bit) >> lane_off) & 0xFFFFu;
                    if (bit) hs[idx + __popc(bal & ((1u << g.t) - 1u))] = (uint8_t)(g.t + 16 * m);
                    idx += __popc(bal);
                }
                if (g.t == 0) hs[OMEGA + k] = (uint8_t)(cnt + (half ? tot0 + tot1 : tot0));
                cnt += tot0 + tot1;
            }
        }
        n_intt += __shfl_down_sync(0xFFFFFFFFu, n_intt, 16);  // lane 0: both groups
        if (lane == 0) {
            atomicAdd(&q->intt, (unsigned long long)n_intt);
            atomicSub(arg.inflight + item, 1u);
        }
        if (rejected) return;
        for (int qq = cnt + lane; qq < OMEGA; qq += 32) hs[qq] = 0;
        __syncwarp();
        // accepted: lower the item's best nonce; publish if this attempt holds the minimum
        unsigned old = 0;
        if (lane == 0) old = atomicMin(arg.best + item, nonce);
        old = __shfl_sync(0xFFFFFFFFu, old, 0);
        if (nonce >= old) return;
        if (lane == 0 && old == 0xFFFFFFFFu) {
            atomicAdd(&q->done_items, 1u);
            atomicSub(&s_ctl[CT_PEND], 1u);
        }
        // (old == kNonceExhausted: the item was already counted as finished; a late acceptance
        // below the limit still publishes its signature)
        int got = 0;
        if (lane == 0) {
            for (unsigned spin = 0; spin < arg.lock_spins; ++spin) {
                if (atomicCAS(arg.locks + item, 0u, 1u) == 0u) {
                    got = 1;
                    break;
                }
                __nanosleep(64);
            }
            if (!got) atomicOr(&q->error, 1u);
        }
        got = __shfl_sync(0xFFFFFFFFu, got, 0);
        if (!got) return;
        __threadfence();
        unsigned cur = 0;
        if (lane == 0) cur = *reinterpret_cast<volatile unsigned *>(arg.best + item);
        cur = __shfl_sync(0xFFFFFFFFu, cur, 0);
        if (cur == nonce) {
            publish_signature<PM::SIG_BYTES, 32>(arg.sig_out + (size_t)item * arg.sig_pitch,
                                                 reinterpret_cast<const uint32_t *>(slot + C::SL_SIG), lane);
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) atomicExch(arg.locks + item, 0u);
    };

    // w = invNTT(A_hat * NTT(y)), Decompose, pack w1 of one attempt (group-collective)
    auto w_job = [&](int nb, int a) {
        if (!bc_ok(a < A, BC_SIGN_SLOT)) return;
        const unsigned item = s_item[nb * A + a];
        if (!bc_ok(item < n, BC_SIGN_SLOT)) return;
        bool skip = __ldcg(arg.best + item) < s_nonce[nb * A + a];
        skip = __shfl_sync(g.gmask, skip, lane_off);
        const unsigned key = arg.key_idx[item];
        if (skip || !bc_ok(key < arg.nkeys, BC_SIGN_KEY)) return;
        uint8_t *slot = slot_of(nb, a);
        const uint8_t *row = arg.cache + (size_t)key * arg.cpitch;
        int32_t *yh = reinterpret_cast<int32_t *>(ph) + (size_t)gi * (L * N + NTT_SMEM_WORDS);
        g.sm = yh + L * N;
#pragma unroll 1
        for (int j = 0; j < L; ++j) {
            int32_t x[16];
            unpack_z_strided<MODE>(x, slot + C::SL_Y + (size_t)j * PM::POLYZ_PACKED, g.t);
            fwd(x);
            store16_smem(yh + j * N, x, g.t);
        }
        __syncwarp(g.gmask);
        const int32_t *mat0 = reinterpret_cast<const int32_t *>(row + C::SK_MAT);
#pragma unroll 1
        for (int i = 0; i < K; ++i) {
            int32_t acc[16];
            dot16<L, (L + 1) / 2>(acc, yh, g.t, [&](int j) { return mat0 + ((size_t)i * L + j) * N; });
            inv(acc);
            int32_t *w0 = reinterpret_cast<int32_t *>(slot + C::SL_W0) + (size_t)i * N;
            int32_t w1[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                int32_t a0;
                w1[m] = decompose<MODE>(a0, caddq(reduce32(acc[m])));
                w0[g.t + 16 * m] = a0;
            }
            int32_t w1c[16];
            strided_to_contig(g, w1, w1c);
            uint32_t v[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) v[m] = (uint32_t)w1c[m];
            pack16_words<PM::W1_BITS>(
                reinterpret_cast<uint32_t *>(slot + C::SL_W1P + (size_t)i * PM::POLYW1_PACKED + g.t * 2 * PM::W1_BITS), v);
        }
        __syncwarp(g.gmask);
    };

    // ---------------- NTT phase: rejection of batch cb, w = A y of batch nb
    auto ntt_phase = [&](int cb, int na_c, int nb, int na_n) {
        // a warp takes one unit at a time: a rejection unit is one attempt for the whole warp, a w
        // unit two attempts, one per 16-thread group (w jobs have no data-dependent control flow,
        // so the two groups run in lockstep)
        const int total = na_c + (na_n + 1) / 2;
#pragma unroll 1
        for (;;) {
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(&s_ctl[CT_NJOB], 1u);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if ((int)base >= total) break;
            if ((int)base < na_c) {
                reject_job(cb, (int)base);
            } else {
                const int a = 2 * ((int)base - na_c) + (lane_off ? 1 : 0);
                if (a < na_n) w_job(nb, a);
            }
            __syncwarp();  // both groups back together before the next full-warp grab
        }
    };

    // ---------------- main loop (thread 0 accumulates per-phase cycles for the work counters)
    long long t_claim = 0, t_kec = 0, t_ntt = 0, t_start = clock64(), t0;
    unsigned iters = 0;
    // owned items still pending: all of them after k_fused_init, those the staged rounds left otherwise
    if (tid == 0) s_ctl[CT_PEND] = 0;
    __syncthreads();
    unsigned mine = 0;
    for (unsigned k = tid; k < n_own; k += THREADS) mine += __ldcg(arg.best + b0 + k * grid) == 0xFFFFFFFFu ? 1u : 0u;
    if (mine) atomicAdd(&s_ctl[CT_PEND], mine);
    // The block leaves as a whole: every thread gets the barrier's own result.  (The count itself may already
    // have been lowered when a late warp reads it: the claim that follows marks items that are out of nonces.)
    if (!__syncthreads_or(mine != 0u)) return;
    claim(0);
    keccak_phase(0, 0, 0, (int)s_ctl[CT_NA0]);
    __syncthreads();
    ntt_phase(0, 0, 0, (int)s_ctl[CT_NA0]);
    __syncthreads();
    int cur = 0;
#pragma unroll 1
    for (;;) {
        const int nxt = cur ^ 1;
        t0 = clock64();
        claim(nxt);
        t_claim += clock64() - t0;
        const int na_c = (int)s_ctl[CT_NA0 + cur], na_n = (int)s_ctl[CT_NA0 + nxt];
        // nothing in flight and nothing claimable: every owned item has its winner
        if (na_c == 0 && na_n == 0) break;
        ++iters;
        t0 = clock64();
        keccak_phase(cur, na_c, nxt, na_n);
        __syncthreads();
        t_kec += clock64() - t0;
        t0 = clock64();
        ntt_phase(cur, na_c, nxt, na_n);
        __syncthreads();
        t_ntt += clock64() - t0;
        cur = nxt;
    }
    if (tid == 0) {
        atomicAdd(&q->cyc[0], (unsigned long long)t_claim);
        atomicAdd(&q->cyc[1], (unsigned long long)t_kec);
        atomicAdd(&q->cyc[2], (unsigned long long)t_ntt);
        atomicAdd(&q->cyc[3], (unsigned long long)(clock64() - t_start));
        atomicAdd(&q->iters, iters);
    }
}

}  // namespace cudil
