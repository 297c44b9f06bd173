// Verification of a batch against the resident public rows (no ExpandA / H(pk) per signature), one kernel
// per parallel shape:
//   k_fv_challenge  one thread (few signatures: a pair) per signature, longest message first:
//                   mu = H(tr || m), c = SampleInBall(c~)
//   k_fv_w          one warp per signature, its two 16-thread groups on different polynomials: hint encoding
//                   and z range checks, w' = A_hat NTT(z) - NTT(c) t1_hat, UseHint, packing
//   k_fv_final      one thread or pair per signature: c~' = H(mu || w1') and comparison
//
// One persistent kernel did the three before, a block's 30 to 200 signatures at a time: its hashing phases
// kept a few of the block's warps busy, and a signature's polynomials went one after the other through one
// group.  65 536 Dilithium5 signatures over 256 resident keys: 1.37 ms, 1.00 ms in these kernels; 10 000
// Dilithium2 signatures with as many fresh keys 537 us (key caches included), 459 us; 33 Dilithium3
// signatures 118 us, 99 us.
#pragma once

#include "fused_kernels.cuh"

namespace cudil {

template <int MODE>
struct VerifyRow {
    // per-signature scratch between k_fv_w and k_fv_final
    static constexpr size_t W1 = align256(P<MODE>::W1PACKED_BYTES);
    // shared memory of one warp of k_fv_w: z_hat_0..L-1, -c_hat, two transposes, two hint bitmaps
    static constexpr size_t WARP = (size_t)(Params<MODE>::L + 1) * N * 4 + 2 * NTT_SMEM_WORDS * 4 + 2 * 8 * 4;
};

struct VerifyArgs {
    const uint8_t *cache;
    size_t cpitch;
    MsgRefs mr;
    const uint8_t *sig;
    size_t sig_pitch;
    uint8_t *items;    // mu | challenge (two-bit fields)
    uint8_t *w1;       // VerifyRow::W1 bytes per signature
    unsigned *status;  // 0 = no check failed
    int *ret;
    unsigned n;             // signatures
    unsigned first, count;  // those of one launch of k_fv_w and k_fv_final, first's w1 at the scratch's start
};

// Signatures whose packed w1' the scratch holds at a time (200 MB for Dilithium2, 270 MB for the others); a
// larger batch runs k_fv_w and k_fv_final in turns.  The bound keeps an engine's memory per item from
// growing by the size of a w1' (768 or 1024 bytes to the 164 an item takes); turns of this size are hundreds
// of waves of blocks, so their ends cost nothing.
constexpr size_t kVerifyTurn = size_t(1) << 18;

// Word w (0..7) of the 32 bytes of c~ at s, which may start at any byte.
__device__ __forceinline__ uint32_t ctilde_word(const uint8_t *s, int w) {
    if ((reinterpret_cast<uintptr_t>(s) & 3u) == 0u) return reinterpret_cast<const uint32_t *>(s)[w];
    return load_lane_bytes(s + 4 * w, 4).x;
}

template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kPrehashBlock) k_fv_challenge(VerifyArgs a) {
    using PM = P<MODE>;
    using C = Cache<MODE>;
    using Sp = Shake256<PAIR>;
    constexpr unsigned PER = kPrehashBlock / Sp::LANES;
    __shared__ uint32_t s_sib[SIB_WORDS * kPrehashBlock];
    for (unsigned r0 = blockIdx.x * PER; r0 < a.n; r0 += gridDim.x * PER) {
        const unsigned r = r0 + threadIdx.x / Sp::LANES;
        bool on = r < a.n;
        const unsigned it = on ? (a.mr.order ? a.mr.order[r] : r) : 0u;
        on = on && bc_ok(it < a.n && a.mr.key_idx[it] < a.mr.nkeys, BC_PREHASH_ITEM);
        if (!PAIR && !on) continue;
        const uint8_t *row = a.cache + (on ? (size_t)a.mr.key_idx[it] * a.cpitch : 0);
        const long long ml = on ? (long long)a.mr.mlens[it] : 0;
        TwoPart src{row + C::PK_TR, 4, a.mr.msgs + (on ? a.mr.offsets[it] : 0), ml};
        Sp sp;
        sp.hash(src, SEEDBYTES + ml, on);
        uint8_t *out = a.items + (size_t)it * C::ITEM_BYTES;
        if (on) sp.template store<8>(out);
        const uint8_t *s = a.sig + (size_t)it * a.sig_pitch;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            if constexpr (PAIR) {
                sp.dlo[w] = ctilde_word(s, 2 * w + sp.half());
            } else {
                sp.dlo[w] = ctilde_word(s, 2 * w);
                sp.dhi[w] = ctilde_word(s, 2 * w + 1);
            }
        }
        sample_in_ball<PM::TAU, kPrehashBlock, PAIR>(sp, s_sib, threadIdx.x);
        if (on && (!PAIR || sp.half() == 0)) sib_store<kPrehashBlock>(out + 64, s_sib, threadIdx.x);
        if constexpr (PAIR) __syncwarp();
    }
}

template <int MODE>
__global__ void __launch_bounds__(kBlock, MODE == 5 ? 5 : 6) k_fv_w(VerifyArgs a) {
    using PM = P<MODE>;
    using C = Cache<MODE>;
    using V = VerifyRow<MODE>;
    constexpr int K = PM::K, L = PM::L, OMEGA = PM::OMEGA;
    constexpr unsigned FULL = 0xFFFFFFFFu;
    extern __shared__ __align__(16) uint8_t fv_smem[];
    const int lane = threadIdx.x & 31, half = lane >> 4, warp = threadIdx.x >> 5;
    int32_t *zh = reinterpret_cast<int32_t *>(fv_smem + (size_t)warp * V::WARP);
    Group g;
    g.t = lane & 15;
    g.gmask = 0xFFFFu << (lane & 16);
    g.sm = zh + (L + 1) * N + half * NTT_SMEM_WORDS;
    uint32_t *hbits = reinterpret_cast<uint32_t *>(zh + (L + 1) * N + 2 * NTT_SMEM_WORDS) + 8 * half;
    const unsigned nwarps = gridDim.x * (blockDim.x >> 5);
    for (unsigned u = blockIdx.x * (blockDim.x >> 5) + warp; u < a.count; u += nwarps) {
        const unsigned it = a.first + u;
        const unsigned key = a.mr.key_idx[it];
        const bool key_ok = bc_ok(key < a.mr.nkeys, BC_VERIFY_KEY);
        const uint8_t *row = a.cache + (size_t)(key_ok ? key : 0u) * a.cpitch;
        const uint8_t *s = a.sig + (size_t)it * a.sig_pitch, *h = s + PM::SIG_H;
        bool bad = !key_ok;
        // hint encoding: per-poly ends non-decreasing and at most OMEGA, positions strictly increasing
        // inside each poly, unused positions zero; lane j checks positions j, j + 32, ...
        {
            const int end = lane < K ? h[OMEGA + lane] : 0;
            const int before = __shfl_up_sync(FULL, end, 1);
            bad |= lane < K && (end > OMEGA || (lane > 0 && end < before));
            const int used = __shfl_sync(FULL, end, K - 1);
#pragma unroll
            for (int j0 = 0; j0 < OMEGA; j0 += 32) {
                const int j = j0 + lane;
                bool starts = j == 0;  // j is the first position of a poly
#pragma unroll
                for (int i = 0; i < K - 1; ++i) starts |= j == __shfl_sync(FULL, end, i);
                if (j < OMEGA) bad |= j >= used ? h[j] != 0 : (!starts && h[j] <= h[j - 1]);
            }
        }
        __syncwarp();  // the previous signature's vectors have been read
#pragma unroll 1
        for (int j = half; j <= L; j += 2) {
            int32_t x[16];
            if (j < L) {
                unpack_z_strided<MODE>(x, s + PM::SIG_Z + (size_t)j * PM::POLYZ_PACKED, g.t);
#pragma unroll
                for (int m = 0; m < 16; ++m) bad |= exceeds(x[m], PM::GAMMA1 - PM::BETA);
            } else {
                uint32_t fld[16];
                const uint4 *mi = reinterpret_cast<const uint4 *>(a.items + (size_t)it * C::ITEM_BYTES + 64);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint4 v = mi[k];
                    fld[4 * k] = v.x;
                    fld[4 * k + 1] = v.y;
                    fld[4 * k + 2] = v.z;
                    fld[4 * k + 3] = v.w;
                }
                challenge_strided(x, fld, g.t);
            }
            ntt16s(x, g.sm, g.gmask, g.t);
            if (j == L) {  // -c_hat with the inverse transform's factor (A_hat carries it already)
#pragma unroll
                for (int m = 0; m < 16; ++m) x[m] = -scale_f(x[m]);
            }
            store16_smem(zh + j * N, x, g.t);
        }
        __syncwarp();
        bad = __any_sync(FULL, bad);
        if (lane == 0) a.status[it] = bad ? 1u : 0u;
        if (bad) continue;  // rejected whatever the hash says
        const int32_t *mat = reinterpret_cast<const int32_t *>(row + C::PK_MAT), *t1 = reinterpret_cast<const int32_t *>(row + C::PK_T1);
        uint8_t *w1out = a.w1 + (size_t)u * V::W1;
#pragma unroll 1
        for (int i = half; i < K; i += 2) {  // K is even
            // the poly's hint bitmap (positions were checked above)
            if (g.t < 8) hbits[g.t] = 0u;
            __syncwarp(g.gmask);
            const int from = i ? h[OMEGA + i - 1] : 0, to = h[OMEGA + i];
            for (int j = from + g.t; j < to; j += 16) atomicOr(&hbits[h[j] >> 5], 1u << (h[j] & 31));
            __syncwarp(g.gmask);
            // sum_j A_ij z_j - c t1_i: t1_i is operand L, whose shared-memory vector is -c_hat
            int32_t acc[16];
            dot16<L + 1, (L + 2) / 2>(acc, zh, g.t, [&](int j) { return j < L ? mat + ((size_t)i * L + j) * N : t1 + (size_t)i * N; });
            intt16s(acc, g.sm, g.gmask, g.t);
            uint32_t b[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                b[c] = 0u;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    // coefficient t + 16 (4 c + m)
                    const unsigned hint = (hbits[2 * c + (m >> 1)] >> (g.t + 16 * (m & 1))) & 1u;
                    b[c] |= (uint32_t)use_hint<MODE>(caddq(reduce32(acc[4 * c + m])), hint) << (8 * m);
                }
            }
            pack_strided_bytes<PM::W1_BITS>(reinterpret_cast<uint32_t *>(w1out + (size_t)i * PM::POLYW1_PACKED), b, g.t, g.gmask);
            __syncwarp(g.gmask);
        }
    }
}

template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kPrehashBlock) k_fv_final(VerifyArgs a) {
    using PM = P<MODE>;
    using C = Cache<MODE>;
    using V = VerifyRow<MODE>;
    using Sp = Shake256<PAIR>;
    constexpr unsigned PER = kPrehashBlock / Sp::LANES;
    for (unsigned u0 = blockIdx.x * PER; u0 < a.count; u0 += gridDim.x * PER) {
        const unsigned u = u0 + threadIdx.x / Sp::LANES;
        const bool on = u < a.count;
        if (!PAIR && !on) continue;
        const unsigned it = a.first + (on ? u : 0u);
        const uint8_t *s = a.sig + (size_t)it * a.sig_pitch;
        TwoPart src{a.items + (size_t)it * C::ITEM_BYTES, 8, a.w1 + (size_t)(it - a.first) * V::W1, PM::W1PACKED_BYTES};
        Sp sp;
        sp.hash(src, CRHBYTES + PM::W1PACKED_BYTES, on);
        bool eq = true;
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            if constexpr (PAIR)
                eq &= sp.dlo[w] == ctilde_word(s, 2 * w + sp.half());
            else
                eq &= sp.dlo[w] == ctilde_word(s, 2 * w) && sp.dhi[w] == ctilde_word(s, 2 * w + 1);
        }
        if constexpr (PAIR) eq = __shfl_xor_sync(0xFFFFFFFFu, eq, 1) && eq;
        if (on) a.ret[it] = (eq && a.status[it] == 0u) ? 0 : -1;
    }
}

}  // namespace cudil
