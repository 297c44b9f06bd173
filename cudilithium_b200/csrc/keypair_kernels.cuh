// Batched key generation (reference: gpu_keypair, src/keypair.cu:35-311, one warp per key), one kernel
// per parallel shape so that every Keccak stage has all its threads on streams:
//   k_kp_seed  one thread per key: seed (from the counter scheme of src/keypair.cu:53-59 or
//              caller-provided) -> (rho, rho', K) = SHAKE256(seed, 128)
//   k_kp_s     one thread per secret polynomial: ExpandS stream, eta fields packed into sk as sampled
//   k_kp_s1    16-thread group per s1 polynomial: s1_hat = NTT(s1), with the inverse transform's factor
//   k_kp_t     one thread per ExpandA entry, products A_ij * s1_hat_j summed into the block's rows of
//              t_hat in shared memory (no A matrix is stored), then per row invNTT, + s2, Power2Round,
//              t1/t0 packing
//   k_kp_tr    one thread or thread pair per key: tr = SHAKE256(pk, 32)
#pragma once

#include "sign_kernels.cuh"

namespace cudil {

template <int MODE>
__global__ void __launch_bounds__(kBlock) k_kp_seed(uint8_t *pool, size_t pitch, int n, unsigned long long rand_index,
                                                    int seeds_given) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    const int it = blockIdx.x * blockDim.x + threadIdx.x;
    if (it >= n) return;
    uint8_t *row = pool + (size_t)it * pitch;
    uint32_t al[25], ah[25];
    uint2 seed[4];
    if (seeds_given) {
        // caller seed parked in sk's tr slot (written last by k_kp_tr)
        ld_lanes(seed, row + LY::KP_SK + PM::SK_TR);
    } else {
        const unsigned long long ctr = rand_index + 2ull * (unsigned long long)it + 1ull;
        keccak_zero(al, ah);
        al[0] = (uint32_t)ctr;
        ah[0] = (uint32_t)(ctr >> 32);
        al[1] = 0x1Fu;
        ah[20] ^= 0x80000000u;  // SHAKE128 rate 168 -> last lane 20
        keccak_f1600(al, ah);
#pragma unroll
        for (int w = 0; w < 4; ++w) seed[w] = make_uint2(al[w], ah[w]);
    }
    keccak_zero(al, ah);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        al[w] = seed[w].x;
        ah[w] = seed[w].y;
    }
    al[4] = 0x1Fu;
    ah[16] ^= 0x80000000u;
    keccak_f1600(al, ah);
    uint2 *pk = reinterpret_cast<uint2 *>(row + LY::KP_PK);
    uint2 *sk = reinterpret_cast<uint2 *>(row + LY::KP_SK);
    uint2 *rhop = reinterpret_cast<uint2 *>(row + LY::KP_RHOP);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const uint2 v = make_uint2(al[w], ah[w]);
        pk[w] = v;
        sk[w] = v;
        sk[4 + w] = make_uint2(al[12 + w], ah[12 + w]);  // K
    }
#pragma unroll
    for (int w = 0; w < 8; ++w) rhop[w] = make_uint2(al[4 + w], ah[4 + w]);
}

// 16 bits-per-unit packing of 16 consecutive values of BITS bits (BITS halfwords).
template <int BITS>
__device__ __forceinline__ void pack16_halves(uint16_t *out, const uint32_t (&v)[16]) {
    uint32_t w[BITS];
#pragma unroll
    for (int i = 0; i < BITS; ++i) w[i] = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int bit = i * BITS, wi = bit >> 4, sh = bit & 15;
        const uint32_t sv = v[i] << sh;  // at most BITS + 15 <= 28 bits
        w[wi] |= sv & 0xFFFFu;
        if (wi + 1 < BITS) w[wi + 1] |= (sv >> 16) & 0xFFFFu;
    }
#pragma unroll
    for (int i = 0; i < BITS; ++i) out[i] = (uint16_t)w[i];
}

// ExpandS (src/keypair.cu:84-114): s1 (nonces 0..L-1) then s2 (nonces L..L+K-1), one thread per
// polynomial, SHAKE256(rho' || nonce); nibbles, low one first, below 15 (eta 2) or 9 (eta 4) are
// accepted.  The fields go straight into sk: a table of the 256 byte values gives a byte's accepted
// fields, already packed, and their bits, so two nibbles cost one lookup and one append.
template <int MODE>
__global__ void __launch_bounds__(kBlock) k_kp_s(uint8_t *pool, size_t pitch, int n) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    constexpr int NP = PM::L + PM::K, EB = PM::ETA_BITS, NW = N * EB / 32;
    __shared__ uint32_t lut[256];  // fields | bits << 8
    for (int v = threadIdx.x; v < 256; v += kBlock) {
        uint32_t f = 0, nb = 0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t t = (uint32_t)(v >> (4 * h)) & 15u;
            if (PM::ETA == 2 ? t < 15u : t < 9u) {
                f |= (PM::ETA == 2 ? t % 5u : t) << nb;
                nb += EB;
            }
        }
        lut[v] = f | nb << 8;
    }
    __syncthreads();
    const int u = blockIdx.x * blockDim.x + threadIdx.x, it = u / NP, p = u % NP;
    if (it >= n) return;
    uint8_t *row = pool + (size_t)it * pitch;
    uint2 rhop[8];
    ld_lanes(rhop, row + LY::KP_RHOP);
    uint32_t *dst = reinterpret_cast<uint32_t *>(row + LY::KP_SK + PM::SK_S1 + (size_t)p * PM::POLYETA_PACKED);
    uint32_t al[25], ah[25];
    shake_absorb_seed_nonce<SHAKE256_RATE, 8>(al, ah, rhop, (uint32_t)p);
    uint32_t w = 0, nb = 0;
    int words = 0;
    while (words < NW) {
        keccak_f1600(al, ah);
#pragma unroll
        for (int k = 0; k < 2 * (SHAKE256_RATE / 8); ++k) {
            const uint32_t word = (k & 1) ? ah[k >> 1] : al[k >> 1];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const uint32_t e = lut[(word >> (8 * b)) & 0xFFu], f = e & 0xFFu;
                w |= f << nb;
                const uint32_t nn = nb + (e >> 8);
                if (nn >= 32u) {
                    // the field bits past the word; fields past the last word are dropped
                    if (words < NW) dst[words] = w;
                    ++words;
                    w = f >> (32u - nb);
                }
                nb = nn & 31u;
            }
        }
    }
}

// The eta field of coefficient c of a packed secret polynomial.
template <int MODE>
__device__ __forceinline__ int32_t eta_coef(const uint8_t *poly, int c) {
    constexpr int EB = P<MODE>::ETA_BITS;
    const int bit = EB * c, byte = bit >> 3, sh = bit & 7;
    uint32_t v = poly[byte];
    if (sh + EB > 8) v |= (uint32_t)poly[byte + 1] << 8;
    return Params<MODE>::ETA - (int32_t)((v >> sh) & ((1u << EB) - 1u));
}

template <int MODE>
__global__ void __launch_bounds__(kBlock) k_kp_s1(uint8_t *pool, size_t pitch, int n) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    __shared__ int32_t sm[kGroupsPerBlock * NTT_SMEM_WORDS];
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) >> 4, it = gid / PM::L, j = gid % PM::L;
    if (it >= n) return;
    Group g = make_group(sm, threadIdx.x >> 4);
    uint8_t *row = pool + (size_t)it * pitch;
    const uint8_t *src = row + LY::KP_SK + PM::SK_S1 + (size_t)j * PM::POLYETA_PACKED;
    int32_t x[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) x[m] = eta_coef<MODE>(src, g.t + 16 * m);
    ntt16s(x, g.sm, g.gmask, g.t);
#pragma unroll
    for (int m = 0; m < 16; ++m) x[m] = scale_f(x[m]);
    // natural order: k_kp_t's threads walk it coefficient by coefficient
    store16_contig(reinterpret_cast<int32_t *>(row + LY::KP_S1H) + (size_t)j * N + 16 * g.t, x);
}

// A block takes kBlock / L consecutive rows (key, i) of t_hat, one thread per entry A_ij of them, and
// sums the products in shared memory.  Rows are 257 words apart: the lanes of a warp -- the same j of
// different rows -- then add to the same coefficient in different banks.
//
// Every candidate goes the same way: eight acceptances give eight offsets, then the loads of s1_hat, the
// products and the predicated additions follow without a branch.  (A wide path for aligned groups beside a
// path for the others was executed twice by nearly every warp: a lane that has rejected a candidate, one in
// five by the end of its stream, is no longer aligned.)
//
// Bound: the ALU pipe (K L 5 permutations a key).  10 000 Dilithium2 key pairs, this stage: sums by
// shared-memory atomics with a row's L entries in neighbouring lanes (L-way collisions) 316 us; entries
// kept in shared memory and summed by the groups (128 KiB per 128 threads, too few warps) 372 us; wide and
// narrow paths 321 us; this form 283 us (186 us of permutations at the ALU rate).
constexpr int KP_ROW = N + 1;

template <int MODE>
__global__ void __launch_bounds__(kBlock) k_kp_t(uint8_t *pool, size_t pitch, int n) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    constexpr int K = PM::K, L = PM::L, ROWS = kBlock / L;
    __shared__ int32_t acc[ROWS * KP_ROW];
    __shared__ int32_t sm[kGroupsPerBlock * NTT_SMEM_WORDS];
    const long long row0 = (long long)blockIdx.x * ROWS, nrows = (long long)n * K;
    for (int q = threadIdx.x; q < ROWS * KP_ROW; q += kBlock) acc[q] = 0;
    __syncthreads();
    {
        const int j = threadIdx.x / ROWS, r = threadIdx.x % ROWS;
        const long long gr = row0 + r;
        if (j < L && gr < nrows) {
            const int it = (int)(gr / K), i = (int)(gr % K);
            const uint8_t *row = pool + (size_t)it * pitch;
            uint2 rho[4];
            ld_lanes(rho, row + LY::KP_PK);
            const int32_t *sh = reinterpret_cast<const int32_t *>(row + LY::KP_S1H) + (size_t)j * N;
            int32_t *ac = acc + r * KP_ROW;
            uint32_t al[25], ah[25];
            shake_absorb_seed_nonce<SHAKE128_RATE, 4>(al, ah, rho, (uint32_t)((i << 8) | j));
            int ctr = 0;
            // four blocks give at most 224 coefficients: no candidate is one too many
#pragma unroll 1
            for (int blk = 0; blk < 4; ++blk) {
                keccak_f1600(al, ah);
#pragma unroll
                for (int gq = 0; gq < 7; ++gq) {
                    uint32_t c[8];
                    int32_t sv[8];
                    int at[8], o = ctr;
                    expand_a_candidates(c, al, ah, gq);
#pragma unroll
                    for (int m = 0; m < 8; ++m) {
                        at[m] = o;
                        o += c[m] < (uint32_t)Q ? 1 : 0;
                    }
#pragma unroll
                    for (int m = 0; m < 8; ++m) sv[m] = sh[at[m]];
#pragma unroll
                    for (int m = 0; m < 8; ++m)
                        if (c[m] < (uint32_t)Q) atomicAdd(ac + at[m], montmul((int32_t)c[m], sv[m]));
                    ctr = o;
                }
            }
#pragma unroll 1
            while (ctr < N) {
                keccak_f1600(al, ah);
#pragma unroll
                for (int gq = 0; gq < 7; ++gq) {
                    uint32_t c[8];
                    expand_a_candidates(c, al, ah, gq);
#pragma unroll
                    for (int m = 0; m < 8; ++m)
                        if (c[m] < (uint32_t)Q && ctr < N) {
                            atomicAdd(ac + ctr, montmul((int32_t)c[m], sh[ctr]));
                            ++ctr;
                        }
                }
            }
        }
    }
    __syncthreads();

    // t = invNTT(t_hat) + s2; Power2Round; pack t1 (pk) and t0 (sk)
    const int gi = threadIdx.x >> 4;
    Group g = make_group(sm, gi);
    for (int r = gi; r < ROWS; r += kGroupsPerBlock) {
        const long long gr = row0 + r;
        if (gr >= nrows) break;
        const int it = (int)(gr / K), i = (int)(gr % K);
        uint8_t *row = pool + (size_t)it * pitch;
        int32_t x[16];
        {
            int32_t y[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) y[m] = reduce32(acc[r * KP_ROW + g.t + 16 * m]);
            strided_to_contig(g, y, x);
        }
        intt16s(x, g.sm, g.gmask, g.t);
        const uint8_t *s2 = row + LY::KP_SK + PM::SK_S2 + (size_t)i * PM::POLYETA_PACKED;
        int32_t t1[16], t0[16];
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int32_t v = caddq(reduce32(x[m] + eta_coef<MODE>(s2, g.t + 16 * m)));
            t1[m] = power2round(t0[m], v);
        }
        int32_t c1[16], c0[16];
        strided_to_contig(g, t1, c1);
        strided_to_contig(g, t0, c0);
        uint32_t v1[16], v0[16];
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            v1[m] = (uint32_t)c1[m];
            v0[m] = (uint32_t)((1 << (D - 1)) - c0[m]);
        }
        pack16_words<10>(reinterpret_cast<uint32_t *>(row + LY::KP_PK + SEEDBYTES + (size_t)i * POLYT1_PACKED + 20 * g.t), v1);
        pack16_halves<13>(reinterpret_cast<uint16_t *>(row + LY::KP_SK + PM::SK_T0 + (size_t)i * POLYT0_PACKED + 26 * g.t), v0);
    }
}

template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kBlock) k_kp_tr(uint8_t *pool, size_t pitch, int n) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    using Sp = Shake256<PAIR>;
    const int it = (blockIdx.x * blockDim.x + threadIdx.x) / Sp::LANES;
    const bool on = it < n;
    if (!PAIR && !on) return;
    uint8_t *row = pool + (size_t)(on ? it : 0) * pitch;
    AlignedBytes pk{row + LY::KP_PK, PM::PK_BYTES};
    Sp sp;
    sp.hash(pk, PM::PK_BYTES, on);
    if (on) sp.template store<4>(row + LY::KP_SK + PM::SK_TR);
}

// Packed keys of one row to dense device arrays (word-aligned): one launch for both keys, where two pitched
// copies took about 49 us for 10 000 Dilithium2 pairs (21 us now).
template <int MODE>
__global__ void __launch_bounds__(kBlock) k_kp_out(const uint8_t *pool, size_t pitch, uint8_t *pk, uint8_t *sk) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    constexpr int PW = PM::PK_BYTES / 4, SW = PM::SK_BYTES / 4;
    static_assert(PM::PK_BYTES % 4 == 0 && PM::SK_BYTES % 4 == 0, "whole words");
    const uint8_t *row = pool + (size_t)blockIdx.x * pitch;
    const uint32_t *ps = reinterpret_cast<const uint32_t *>(row + LY::KP_PK), *ss = reinterpret_cast<const uint32_t *>(row + LY::KP_SK);
    uint32_t *po = reinterpret_cast<uint32_t *>(pk) + (size_t)blockIdx.x * PW, *so = reinterpret_cast<uint32_t *>(sk) + (size_t)blockIdx.x * SW;
#pragma unroll 4
    for (int i = threadIdx.x; i < PW + SW; i += kBlock) {
        if (i < PW)
            po[i] = ps[i];
        else
            so[i - PW] = ss[i - PW];
    }
}

}  // namespace cudil
