// Staged signer: the same work queue as k_fused_sign (per-item next nonce, smallest accepted nonce
// wins), run round by round over the whole GPU instead of block by block.
//
// A round is five kernels over the round's attempts, each in the shape its stage needs:
//   k_st_claim      publishes the previous round's winners, compacts the pending items and gives each its
//                   next D nonces, D = target / pending, at most kStagedMaxDepth
//   k_st_mask       ExpandMask, one thread (few streams: a pair) per (attempt, j) stream
//   k_st_w          w = A y, Decompose, w1 packing: one warp per attempt, its two 16-thread groups on
//                   different polynomials
//   k_st_challenge  c~ = H(mu || w1) and SampleInBall, one thread per attempt
//   k_st_reject     rejection checks and hints, one warp per attempt; an accepted attempt lowers its
//                   item's best nonce
// The host enqueues as many rounds as the acceptance rate calls for (EngineImpl::sign_staged) without
// waiting for any of them; the counts stay on the device, and a round that finds nothing pending returns
// at once.  k_fused_sign runs last and finishes the items, if any, that the enqueued rounds left.
//
// Why rounds over the whole GPU: the persistent kernels bind an item to a block.  A block's rounds then
// keep costing the latency of their dependent permutations long after most of its items are signed, and
// one register and shared-memory budget serves every stage.  Here a round's attempts spread over all SMs
// whatever items they belong to, and every stage runs at its own occupancy.
#pragma once

#include "fused_kernels.cuh"

namespace cudil {

// Counters of one round; the prehash kernel clears them.
struct StagedRound {
    unsigned npend;     // pending items listed
    unsigned depth;     // attempts of each; the first `extra` listed have one more
    unsigned extra;
    unsigned limit;     // attempts of the round at most
    unsigned accepted;  // items whose first accepted nonce came in this round
    unsigned pad[3];
};

struct StagedAttempt {
    unsigned item, nonce;  // nonce 0xFFFFFFFF: none (the item's nonces ran out)
    unsigned accepted;
    unsigned pad;
};

constexpr int kStagedMaxRounds = 40;
constexpr size_t kStagedRoundBytes = kStagedMaxRounds * sizeof(StagedRound);  // of one part
constexpr unsigned kStagedMaxDepth = 64;
constexpr unsigned kStagedPending = 0xFFFFFFFFu, kStagedNoNonce = 0xFFFFFFFFu;

template <int MODE>
struct StagedSlot {
    using PM = P<MODE>;
    static constexpr int K = PM::K, L = PM::L;
    static constexpr size_t POLY = N * sizeof(int32_t);
    static constexpr size_t Y = 0;                                          // packed y (y_word order)
    static constexpr size_t W0 = align256((size_t)L * PM::POLYZ_PACKED);    // [K][4 chunks][16 positions] int4
    static constexpr size_t W1P = W0 + (size_t)K * POLY;                    // packed w1
    static constexpr size_t W1B = W1P + align256(PM::W1PACKED_BYTES);       // [K][16 positions][16] w1 bytes
    static constexpr size_t CM = W1B + (size_t)K * 256;                     // challenge masks
    static constexpr size_t SIG = CM + 256;                                 // staged signature
    static constexpr size_t SIZE = SIG + align256(PM::SIG_BYTES);
    // shared memory of one warp of k_st_w (y_hat and two transposes) and of k_st_reject
    static constexpr size_t WARP_W = (size_t)L * POLY + 2 * NTT_SMEM_WORDS * 4;
    static constexpr size_t WARP_R = 2 * POLY + 2 * NTT_SMEM_WORDS * 4;  // c_hat of two attempts, two transposes
};

struct StagedArgs {
    const uint8_t *cache;
    size_t cpitch;
    const unsigned *key_idx;
    const uint8_t *items;
    uint8_t *sig_out;
    size_t sig_pitch;
    uint8_t *slots;
    StagedAttempt *att[2];  // by round parity: a claim writes one while it publishes from the other
    unsigned *pend[2];
    StagedRound *rounds;
    FusedQueue *q;
    unsigned *best, *locks, *next_nonce, *inflight;
    const unsigned *order;  // longest message first (nullptr: item order)
    unsigned n;             // items of the batch
    unsigned first, count;  // this part's items: order[first .. first + count)
    unsigned cap;           // attempt slots
    unsigned target;     // attempts a round aims at once fewer items than that are pending
    unsigned quantum;    // attempts whose ExpandMask streams fill every sub-partition's lanes evenly
    unsigned nonce_limit;
    unsigned nkeys;
};

__device__ __forceinline__ unsigned staged_attempts(const StagedArgs &a, int r) {
    const StagedRound &rd = a.rounds[r];
    const unsigned long long v = (unsigned long long)rd.npend * rd.depth + (rd.npend < rd.extra ? rd.npend : rd.extra);
    return v < rd.limit ? (unsigned)v : rd.limit;
}

// Round r's claim (claim = false: only the publication of round r - 1).  Positions in the pending list
// come from an atomic counter, so the list's order varies from run to run; which nonces an item tries, and
// so its signature, does not depend on it.
template <int MODE>
__global__ void __launch_bounds__(256) k_st_claim(StagedArgs a, int r, bool claim) {
    using PM = P<MODE>;
    using S = StagedSlot<MODE>;
    const int lane = threadIdx.x & 31;
    const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x, nthreads = gridDim.x * blockDim.x;
    if (claim) {
        const unsigned nprev = r ? a.rounds[r - 1].npend : a.count;
        const unsigned pending = r ? nprev - a.rounds[r - 1].accepted : a.count;
        // target attempts, spread evenly; with more items pending than that, one attempt each to as many as
        // make whole quanta (the others wait a round: a partly filled last layer of the ExpandMask streams
        // would cost as much as a full one)
        unsigned depth = 1, extra = 0, limit = a.target;
        if (pending >= a.target) {
            limit = pending < a.cap ? pending : a.cap;
            if (limit > a.quantum && limit < 4u * a.quantum) limit = limit / a.quantum * a.quantum;
        } else if (pending) {
            depth = a.target / pending;
            extra = a.target - depth * pending;
            if (depth >= kStagedMaxDepth) {
                depth = kStagedMaxDepth;
                extra = 0;
            }
        }
        if (tid == 0) {
            a.rounds[r].depth = depth;
            a.rounds[r].extra = extra;
            a.rounds[r].limit = limit;
            if (pending) atomicAdd(&a.q->iters, 1u);
        }
        const unsigned *prev = a.pend[(r + 1) & 1];
        unsigned *next = a.pend[r & 1];
        StagedAttempt *att = a.att[r & 1];
        for (unsigned k0 = tid - lane; k0 < nprev; k0 += nthreads) {
            const unsigned k = k0 + lane;
            unsigned item = 0, nn = 0;
            bool ok = k < nprev;
            if (ok) {
                if (r == 0) {
                    item = a.order ? a.order[a.first + k] : a.first + k;
                    ok = bc_ok(item < a.n, BC_SIGN_SLOT);
                    if (ok) {
                        a.best[item] = kStagedPending;
                        a.locks[item] = 0u;
                        a.inflight[item] = 0u;
                    }
                } else {
                    item = prev[k];
                    ok = bc_ok(item < a.n, BC_SIGN_SLOT) && a.best[item] == kStagedPending;
                    if (ok) nn = a.next_nonce[item];
                    if (ok && nn >= a.nonce_limit) {
                        // every nonce tried, none accepted: the item is finished (error bit 1)
                        a.best[item] = kNonceExhausted;
                        atomicOr(&a.q->error, 2u);
                        ok = false;
                    }
                }
            }
            const unsigned bal = __ballot_sync(0xFFFFFFFFu, ok);
            unsigned base = 0;
            if (lane == 0 && bal) base = atomicAdd(&a.rounds[r].npend, (unsigned)__popc(bal));
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            unsigned issued = 0;
            if (ok) {
                const unsigned pos = base + __popc(bal & ((1u << lane) - 1u));
                next[pos] = item;
                const unsigned own = depth + (pos < extra ? 1u : 0u);
                const unsigned long long s0 = (unsigned long long)pos * depth + (pos < extra ? pos : extra);
                if (s0 + own <= limit) {
                    for (unsigned d = 0; d < own; ++d) {
                        const bool real = nn + d < a.nonce_limit;
                        att[s0 + d] = StagedAttempt{item, real ? nn + d : kStagedNoNonce, 0u, 0u};
                        issued += real ? 1u : 0u;
                    }
                }
                a.next_nonce[item] = nn + issued;
            }
            issued = __reduce_add_sync(0xFFFFFFFFu, issued);
            if (lane == 0 && issued) atomicAdd(&a.q->attempts, (unsigned long long)issued);
        }
    }
    if (r == 0) return;
    const unsigned na = staged_attempts(a, r - 1);
    const StagedAttempt *att = a.att[(r - 1) & 1];
    for (unsigned s = tid >> 5; s < na; s += nthreads >> 5) {
        const StagedAttempt at = att[s];
        if (!at.accepted || !bc_ok(at.item < a.n, BC_SIGN_SLOT) || a.best[at.item] != at.nonce) continue;
        publish_signature<PM::SIG_BYTES, 32>(a.sig_out + (size_t)at.item * a.sig_pitch,
                                             reinterpret_cast<const uint32_t *>(a.slots + (size_t)s * S::SIZE + S::SIG), lane);
    }
}

// The staged signer keeps a packed y polynomial (ExpandMask's output, gamma1 - y in Z_BITS-bit fields) in the
// order its readers load it.  Sixteen fields are YW = Z_BITS / 2 words; word k of each sixteen, for four
// consecutive sixteens, makes a 16-byte chunk, and the chunks of four sixteens follow one another: word
// YW i + k of the stream is at y_word(i, k).  Position t's fields t + 16 i sit in words k and k + 1 of every
// sixteen, k = Z_BITS t / 32: eight 128-bit loads read a position's sixteen fields instead of 32 word loads.
template <int MODE>
__host__ __device__ constexpr int y_word(int i, int k) {
    return ((i >> 2) * (P<MODE>::Z_BITS / 2) + k) * 4 + (i & 3);
}

template <int MODE>
__device__ __forceinline__ void unpack_y(int32_t (&x)[16], const uint8_t *poly, int t) {
    constexpr int ZB = P<MODE>::Z_BITS, YW = ZB / 2;
    const unsigned bit = (unsigned)(ZB * t), k = bit >> 5, sh = bit & 31u;
    const int4 *q = reinterpret_cast<const int4 *>(poly) + k;
    const int second = sh + ZB > 32u ? 1 : 0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const int4 lo = q[c * YW], hi = q[c * YW + second];
        auto field = [&](int l, int h) {
            return Params<MODE>::GAMMA1 - (int32_t)(__funnelshift_r((uint32_t)l, (uint32_t)h, sh) & ((1u << ZB) - 1u));
        };
        x[4 * c] = field(lo.x, hi.x);
        x[4 * c + 1] = field(lo.y, hi.y);
        x[4 * c + 2] = field(lo.z, hi.z);
        x[4 * c + 3] = field(lo.w, hi.w);
    }
}

template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kBlock) k_st_mask(StagedArgs a, int r) {
    using PM = P<MODE>;
    using S = StagedSlot<MODE>;
    constexpr int L = PM::L, YW = PM::Z_BITS / 2, RL = SHAKE256_RATE / 8, LANES = PAIR ? 2 : 1;
    const unsigned total = staged_attempts(a, r) * L, per = blockDim.x / LANES;
    const StagedAttempt *att = a.att[r & 1];
    // (the whole block strides together: in pair form every lane of a warp takes part in the shuffles)
    for (unsigned u0 = blockIdx.x * per; u0 < total; u0 += gridDim.x * per) {
        const unsigned u = u0 + threadIdx.x / LANES;
        bool on = u < total;
        const unsigned s = on ? u / L : 0u, j = u % L, item = on ? att[s].item : 0u, nonce = on ? att[s].nonce : kStagedNoNonce;
        on = nonce != kStagedNoNonce && bc_ok(item < a.n, BC_SIGN_SLOT);
        if (!PAIR && !on) continue;
        const uint8_t *rhop = a.items + (size_t)(on ? item : 0u) * Cache<MODE>::ITEM_BYTES + 64;
        uint32_t *o = reinterpret_cast<uint32_t *>(a.slots + (size_t)s * S::SIZE + S::Y + (size_t)j * PM::POLYZ_PACKED);
        const uint32_t kappa = (L * nonce + j) & 0xFFFFu;
        // SHAKE256(rho' || kappa): the words' places are constants, so the blocks are unrolled
        if constexpr (PAIR) {
            const int half = threadIdx.x & 1;
            uint32_t st[25];
#pragma unroll
            for (int w = 0; w < 25; ++w) st[w] = w < 8 ? reinterpret_cast<const uint32_t *>(rhop)[2 * w + half] : 0u;
            st[8] = half ? 0u : (kappa | (0x1Fu << 16));
            st[RL - 1] ^= half ? 0x80000000u : 0u;
#pragma unroll
            for (int blk = 0; blk < PM::MASK_BLOCKS; ++blk) {
                keccak_f1600_pair(st, half);
#pragma unroll
                for (int w = 0; w < RL; ++w) {
                    const int g = 2 * (RL * blk + w);  // the pair's words g and g + 1
                    if (g < 16 * YW && on) o[half ? y_word<MODE>((g + 1) / YW, (g + 1) % YW) : y_word<MODE>(g / YW, g % YW)] = st[w];
                }
            }
        } else {
            uint2 rp[8];
            ld_lanes(rp, rhop);
            uint32_t al[25], ah[25];
            shake_absorb_seed_nonce<SHAKE256_RATE, 8>(al, ah, rp, kappa);
#pragma unroll
            for (int blk = 0; blk < PM::MASK_BLOCKS; ++blk) {
                keccak_f1600(al, ah);
#pragma unroll
                for (int w = 0; w < 2 * RL; ++w) {
                    const int g = 2 * RL * blk + w;
                    if (g < 16 * YW) o[y_word<MODE>(g / YW, g % YW)] = (w & 1) ? ah[w >> 1] : al[w >> 1];
                }
            }
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(kBlock, 6) k_st_w(StagedArgs a, int r) {
    using PM = P<MODE>;
    using C = Cache<MODE>;
    using S = StagedSlot<MODE>;
    constexpr int K = PM::K, L = PM::L;
    extern __shared__ __align__(16) uint8_t st_smem[];
    const int lane = threadIdx.x & 31, half = lane >> 4, warp = threadIdx.x >> 5;
    int32_t *yh = reinterpret_cast<int32_t *>(st_smem + (size_t)warp * S::WARP_W);
    Group g;
    g.t = lane & 15;
    g.gmask = 0xFFFFu << (lane & 16);
    g.sm = yh + L * N + half * NTT_SMEM_WORDS;
    const unsigned na = staged_attempts(a, r), nwarps = gridDim.x * (blockDim.x >> 5);
    const StagedAttempt *att = a.att[r & 1];
    for (unsigned s = blockIdx.x * (blockDim.x >> 5) + warp; s < na; s += nwarps) {
        const unsigned item = att[s].item;
        if (att[s].nonce == kStagedNoNonce || !bc_ok(item < a.n, BC_SIGN_SLOT)) continue;
        const unsigned key = a.key_idx[item];
        if (!bc_ok(key < a.nkeys, BC_SIGN_KEY)) continue;
        uint8_t *slot = a.slots + (size_t)s * S::SIZE;
        __syncwarp();  // the previous attempt's y_hat has been read
#pragma unroll 1
        for (int j = half; j < L; j += 2) {
            int32_t x[16];
            unpack_y<MODE>(x, slot + S::Y + (size_t)j * PM::POLYZ_PACKED, g.t);
            ntt16s(x, g.sm, g.gmask, g.t);
            store16_smem(yh + j * N, x, g.t);
        }
        __syncwarp();
        const int32_t *mat = reinterpret_cast<const int32_t *>(a.cache + (size_t)key * a.cpitch + C::SK_MAT);
#pragma unroll 1
        for (int i = half; i < K; i += 2) {  // K is even
            int32_t acc[16];
            dot16<L, (L + 1) / 2>(acc, yh, g.t, [&](int j) { return mat + ((size_t)i * L + j) * N; });
            intt16s(acc, g.sm, g.gmask, g.t);
            int4 *w0 = reinterpret_cast<int4 *>(slot + S::W0 + (size_t)i * S::POLY);
            uint32_t b[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                int32_t a0[4], w1[4];
#pragma unroll
                for (int m = 0; m < 4; ++m) w1[m] = decompose<MODE>(a0[m], caddq(reduce32(acc[4 * c + m])));
                w0[16 * c + g.t] = make_int4(a0[0], a0[1], a0[2], a0[3]);
                b[c] = (uint32_t)w1[0] | (uint32_t)w1[1] << 8 | (uint32_t)w1[2] << 16 | (uint32_t)w1[3] << 24;
            }
            *reinterpret_cast<uint4 *>(slot + S::W1B + (size_t)i * 256 + 16 * g.t) = make_uint4(b[0], b[1], b[2], b[3]);
            pack_strided_bytes<PM::W1_BITS>(reinterpret_cast<uint32_t *>(slot + S::W1P + (size_t)i * PM::POLYW1_PACKED), b, g.t, g.gmask);
        }
    }
}

template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kItemBlock) k_st_challenge(StagedArgs a, int r) {
    using PM = P<MODE>;
    using S = StagedSlot<MODE>;
    using Sp = Shake256<PAIR>;
    constexpr unsigned PER = kItemBlock / Sp::LANES;  // attempts of a block
    __shared__ uint32_t s_sib[SIB_WORDS * kItemBlock];
    const unsigned na = staged_attempts(a, r);
    const StagedAttempt *att = a.att[r & 1];
    for (unsigned s0 = blockIdx.x * PER; s0 < na; s0 += gridDim.x * PER) {
        const unsigned s = s0 + threadIdx.x / Sp::LANES;
        bool on = s < na && att[s].nonce != kStagedNoNonce;
        const unsigned item = on ? att[s].item : 0u;
        on = on && bc_ok(item < a.n, BC_SIGN_SLOT);
        if (!PAIR && !on) continue;
        uint8_t *slot = a.slots + (size_t)(on ? s : 0u) * S::SIZE;
        TwoPart src{a.items + (size_t)item * Cache<MODE>::ITEM_BYTES, 8, slot + S::W1P, PM::W1PACKED_BYTES};
        Sp sp;
        sp.hash(src, CRHBYTES + PM::W1PACKED_BYTES, on);
        if (on) sp.template store<4>(slot + S::SIG);
        sample_in_ball<PM::TAU, kItemBlock, PAIR>(sp, s_sib, threadIdx.x);
        if (on && (!PAIR || sp.half() == 0)) sib_store<kItemBlock>(slot + S::CM, s_sib, threadIdx.x);
        if constexpr (PAIR) __syncwarp();
    }
}

// The checks run most selective first, a polynomial pair (2 p + half) at a time, as in k_fused_sign's
// rejection job: r0 pairs (r0 replaces w0 in the slot, for the hints), z pairs, ct0 pairs with the hints.
// Both groups of the warp follow the same control flow, and a rejection ends the attempt.
//
// A one-warp block takes `per` attempts (up to NSTEP = 6, 9 or 12 steps each).  per = 2: each group transforms one
// attempt's c, once for both groups; per = 1, in rounds with fewer attempts than resident warps: both groups
// transform the same c.  c_hat waits in shared memory, which leaves the registers to hold a step's w0 in
// flight across its transform.  Resident blocks that draw tickets measured slower in rounds of one or two
// layers of attempts (10 000 items 1.80 against 1.77 ms), blocks of four warps too (a block's slot is free
// only when its longest attempt ends).
template <int MODE>
__global__ void __launch_bounds__(32, 16) k_st_reject(StagedArgs a, int r, unsigned per) {
    using PM = P<MODE>;
    using C = Cache<MODE>;
    using S = StagedSlot<MODE>;
    constexpr int K = PM::K, L = PM::L, OMEGA = PM::OMEGA;
    constexpr unsigned FULL = 0xFFFFFFFFu;
    __shared__ __align__(16) uint8_t st_smem[S::WARP_R];
    const int lane = threadIdx.x & 31, lane_off = lane & 16, half = lane >> 4;
    int32_t *s_c = reinterpret_cast<int32_t *>(st_smem);  // [2][N]
    Group g;
    g.t = lane & 15;
    g.gmask = 0xFFFFu << lane_off;
    g.sm = s_c + 2 * N + half * NTT_SMEM_WORDS;
    const unsigned na = staged_attempts(a, r);
    StagedAttempt *att = a.att[r & 1];
    for (unsigned s0 = blockIdx.x * per; s0 < na; s0 += gridDim.x * per) {
        {
            const unsigned sg = s0 + (per == 2u ? half : 0);
            uint32_t fld[16];
            const uint4 *mi = reinterpret_cast<const uint4 *>(a.slots + (size_t)(sg < na ? sg : s0) * S::SIZE + S::CM);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint4 v = mi[k];
                fld[4 * k] = v.x;
                fld[4 * k + 1] = v.y;
                fld[4 * k + 2] = v.z;
                fld[4 * k + 3] = v.w;
            }
            int32_t x[16];
            challenge_strided(x, fld, g.t);
            ntt16s(x, g.sm, g.gmask, g.t);
#pragma unroll
            for (int m = 0; m < 16; ++m) x[m] = scale_f(x[m]);
            __syncwarp();
            store16_smem(s_c + half * N, x, g.t);
            __syncwarp();
        }
#pragma unroll 1
        for (unsigned s = s0; s < s0 + per && s < na; ++s) {
            const unsigned item = att[s].item, nonce = att[s].nonce;
            if (nonce == kStagedNoNonce || !bc_ok(item < a.n, BC_SIGN_SLOT)) continue;
            const unsigned key = a.key_idx[item];
            if (!bc_ok(key < a.nkeys, BC_SIGN_KEY)) continue;
            // a smaller nonce of the item was accepted: this one cannot win (one decision per warp)
            if (__shfl_sync(FULL, __ldcg(a.best + item) < nonce, 0)) continue;
            uint8_t *slot = a.slots + (size_t)s * S::SIZE;
            const uint8_t *row = a.cache + (size_t)key * a.cpitch;
            const int32_t *chat = s_c + (s - s0) * N;
            const int32_t *s1 = reinterpret_cast<const int32_t *>(row + C::SK_S1);
            const int32_t *s2 = reinterpret_cast<const int32_t *>(row + C::SK_S2);
            const int32_t *t0 = reinterpret_cast<const int32_t *>(row + C::SK_T0);
            uint8_t *hs = slot + S::SIG + PM::SIG_H;
            // K is even; L is odd for two parameter sets: the second group of the last z pair then repeats the
            // first one's polynomial (and stores nothing)
            constexpr int PR = K / 2, PZ = (L + 1) / 2, NSTEP = 2 * PR + PZ;
            auto operand = [&](int step) -> const int32_t * {
                if (step < PR) return s2 + (size_t)(2 * step + half) * N;
                if (step < PR + PZ) {
                    const int j = 2 * (step - PR) + half;
                    return s1 + (size_t)(j < L ? j : L - 1) * N;
                }
                return t0 + (size_t)(2 * (step - PR - PZ) + half) * N;
            };
            bool rejected = false;
            int n_intt = 0, cnt = 0;
            int32_t nx[16];
            load16_chunks(nx, operand(0), g.t);
#pragma unroll 1
            for (int step = 0; step < NSTEP; ++step) {
                const bool is_r0 = step < PR, is_z = !is_r0 && step < PR + PZ;
                int k = 2 * (is_r0 ? step : (is_z ? step - PR : step - PR - PZ)) + half;  // i, or j for z
                const bool act = L % 2 == 0 || !is_z || k < L;
                if (!act) k = L - 1;
                int32_t x[16];
                load16_smem(x, chat, g.t);
#pragma unroll
                for (int m = 0; m < 16; ++m) x[m] = montmul(x[m], nx[m]);
                // the next step's key row and this one's w0 (r0) are in flight during the transform
                if (step + 1 < NSTEP) load16_chunks(nx, operand(step + 1), g.t);
                int4 *w0 = reinterpret_cast<int4 *>(slot + S::W0 + (size_t)k * S::POLY);
                int32_t r0[16];
                if (!is_z) load16_chunks(r0, reinterpret_cast<const int32_t *>(w0), g.t);
                intt16s(x, g.sm, g.gmask, g.t);
                n_intt += act ? 1 : 0;
                bool bad = false;
                if (is_z) {
                    int32_t y[16];
                    unpack_y<MODE>(y, slot + S::Y + (size_t)k * PM::POLYZ_PACKED, g.t);
#pragma unroll
                    for (int m = 0; m < 16; ++m) {
                        x[m] = reduce32(x[m] + y[m]);
                        bad |= exceeds(x[m], PM::GAMMA1 - PM::BETA);
                    }
                    if (__ballot_sync(FULL, bad)) {
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
                            reinterpret_cast<uint32_t *>(slot + S::SIG + PM::SIG_Z + (size_t)k * PM::POLYZ_PACKED + g.t * 2 * PM::Z_BITS), v);
                    }
                    continue;
                }
                if (is_r0) {
#pragma unroll
                    for (int m = 0; m < 16; ++m) {
                        r0[m] = reduce32(r0[m] - x[m]);
                        bad |= exceeds(r0[m], PM::GAMMA2 - PM::BETA);
                    }
                    if (__ballot_sync(FULL, bad)) {
                        rejected = true;
                        break;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) w0[16 * c + g.t] = make_int4(r0[4 * c], r0[4 * c + 1], r0[4 * c + 2], r0[4 * c + 3]);
                    continue;
                }
                const uint4 w1v = *reinterpret_cast<const uint4 *>(slot + S::W1B + (size_t)k * 256 + 16 * g.t);
                const uint32_t w1w[4] = {w1v.x, w1v.y, w1v.z, w1v.w};
                unsigned hb = 0;  // bit m = hint of coefficient t + 16 m
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    x[m] = reduce32(x[m]);
                    bad |= exceeds(x[m], PM::GAMMA2);
                    hb |= make_hint<MODE>(r0[m] + x[m], (int32_t)((w1w[m >> 2] >> (8 * (m & 3))) & 0xFFu)) << m;
                }
                if (__ballot_sync(FULL, bad)) {
                    rejected = true;
                    break;
                }
                // hint counts of both polynomials of the pair, then the positions in ascending coefficient
                // order: poly 2p first, then poly 2p + 1
                int tot = __popc(hb);
#pragma unroll
                for (int o = 8; o >= 1; o >>= 1) tot += __shfl_xor_sync(FULL, tot, o);
                const int tot0 = __shfl_sync(FULL, tot, 0), tot1 = __shfl_sync(FULL, tot, 16);
                if (cnt + tot0 + tot1 > OMEGA) {
                    rejected = true;
                    break;
                }
                int idx = cnt + (half ? tot0 : 0);
#pragma unroll
                for (int m = 0; m < 16; ++m) {
                    const unsigned bit = (hb >> m) & 1u;
                    const unsigned bal = (__ballot_sync(FULL, bit) >> lane_off) & 0xFFFFu;
                    if (bit) hs[idx + __popc(bal & ((1u << g.t) - 1u))] = (uint8_t)(g.t + 16 * m);
                    idx += __popc(bal);
                }
                if (g.t == 0) hs[OMEGA + k] = (uint8_t)(cnt + (half ? tot0 + tot1 : tot0));
                cnt += tot0 + tot1;
            }
            n_intt += __shfl_down_sync(FULL, n_intt, 16);  // lane 0: both groups
            if (lane == 0) atomicAdd(&a.q->intt, (unsigned long long)n_intt);
            if (rejected) continue;
            for (int p = cnt + lane; p < OMEGA; p += 32) hs[p] = 0;
            if (lane == 0) {
                att[s].accepted = 1u;
                // the next claim publishes the attempt whose nonce is still the item's smallest
                if (atomicMin(a.best + item, nonce) == kStagedPending) {
                    atomicAdd(&a.rounds[r].accepted, 1u);
                    atomicAdd(&a.q->done_items, 1u);
                }
            }
        }
    }
}

}  // namespace cudil
