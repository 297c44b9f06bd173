// Device routines shared by the keypair / sign / verify kernels: SHAKE-stream samplers run by one
// thread per stream, and 16-thread-group polynomial helpers.
#pragma once

#include <cstdint>

#include "arith.cuh"
#include "bounds.cuh"
#include "keccak.cuh"
#include "ntt.cuh"
#include "params.cuh"

namespace cudil {

__device__ __forceinline__ uint2 ld_lane(const uint8_t *p) { return *reinterpret_cast<const uint2 *>(p); }

template <int NL>
__device__ __forceinline__ void ld_lanes(uint2 (&v)[NL], const uint8_t *p) {
#pragma unroll
    for (int i = 0; i < NL; ++i) v[i] = ld_lane(p + 8 * i);
}

// The eight 23-bit little-endian candidates of three lanes of an ExpandA block.
__device__ __forceinline__ void expand_a_candidates(uint32_t (&c)[8], const uint32_t (&al)[25], const uint32_t (&ah)[25], int g) {
    const uint32_t w0 = al[3 * g], w1 = ah[3 * g], w2 = al[3 * g + 1];
    const uint32_t w3 = ah[3 * g + 1], w4 = al[3 * g + 2], w5 = ah[3 * g + 2];
    c[0] = w0;
    c[1] = __funnelshift_r(w0, w1, 24);
    c[2] = __funnelshift_r(w1, w2, 16);
    c[3] = w2 >> 8;
    c[4] = w3;
    c[5] = __funnelshift_r(w3, w4, 24);
    c[6] = __funnelshift_r(w4, w5, 16);
    c[7] = w5 >> 8;
#pragma unroll
    for (int m = 0; m < 8; ++m) c[m] &= 0x7FFFFFu;
}

// ExpandA entry A[i][j] (NTT domain), times the inverse transform's factor f (scale_f), written to the
// polynomial out in the storage order of NTT-domain polynomials: SHAKE128(rho || j || i), 23-bit
// little-endian candidates accepted below q (src/sign.cu:98-163, src/keypair.cu:139-190; the stream is
// extended until 256 coefficients are accepted, as benches/bench_rej_sampling.cu:571-593 does).  out is
// 16-byte aligned (pool rows and key-cache rows are).
//
// A block's accepted candidates go to the thread's row of shared memory (stage, EA_STAGE words) one after
// the other, predicated and without a branch; then the whole groups of four leave it as 16-byte stores and
// up to three values stay for the next block.  The rows are 60 words apart: 16-byte accesses of eight lanes
// do not collide, single words four ways.  (Storing aligned groups of eight directly and the others word by
// word ran both paths in nearly every warp, since one lane in five has rejected a candidate by the end of
// its stream: four streamed batches of 10 000 Dilithium2 signatures with fresh keys 5.86 ms, 5.80 ms this way.)
constexpr int EA_STAGE = 60;

__device__ __forceinline__ void expand_a_row(const uint2 (&rho)[4], int i, int j, int32_t *out, uint32_t *stage) {
    uint32_t al[25], ah[25];
    shake_absorb_seed_nonce<SHAKE128_RATE, 4>(al, ah, rho, (uint32_t)((i << 8) | j));
    int fill = 0, done = 0;  // words waiting in stage, groups of four written
#pragma unroll 1
    while (done < N / 4) {
        keccak_f1600(al, ah);
        // 21 lanes = 7 groups of 3 lanes = 7 x 8 candidates of 3 bytes
        int o = fill;
#pragma unroll
        for (int g = 0; g < 7; ++g) {
            uint32_t c[8];
            expand_a_candidates(c, al, ah, g);
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                if (c[m] < (uint32_t)Q) stage[o] = c[m];
                o += c[m] < (uint32_t)Q ? 1 : 0;
            }
        }
        const int nv = min(o >> 2, N / 4 - done);
#pragma unroll
        for (int v = 0; v < EA_STAGE / 4 - 1; ++v) {
            if (v < nv) {
                const int4 w = reinterpret_cast<const int4 *>(stage)[v];
                *reinterpret_cast<int4 *>(out + ntt_at4(4 * (done + v))) =
                    make_int4(scale_f(w.x), scale_f(w.y), scale_f(w.z), scale_f(w.w));
            }
        }
        reinterpret_cast<int4 *>(stage)[0] = reinterpret_cast<const int4 *>(stage)[nv];
        fill = o - 4 * nv;
        done += nv;
    }
}

// ExpandMask entry y_j: SHAKE256(rho' || kappa) with kappa = L*nonce + j (src/sign.cu:488-499);
// the first POLYZ_PACKED bytes are stored verbatim (gamma1 - y packing), `out` 8-byte aligned.
template <int MODE>
__device__ __forceinline__ void expand_mask_stream(uint8_t *out, const uint2 (&rhoprime)[8], uint32_t kappa) {
    constexpr int LANES = P<MODE>::POLYZ_PACKED / 8;  // 72 or 80
    uint32_t al[25], ah[25];
    shake_absorb_seed_nonce<SHAKE256_RATE, 8>(al, ah, rhoprime, kappa & 0xFFFFu);
    uint2 *o = reinterpret_cast<uint2 *>(out);
#pragma unroll 1
    for (int blk = 0; blk < 5; ++blk) {
        keccak_f1600(al, ah);
#pragma unroll
        for (int w = 0; w < 17; ++w) {
            const int g = blk * 17 + w;
            if (g < LANES) o[g] = make_uint2(al[w], ah[w]);
        }
    }
}

// Bit field of `bits` bits (<= 20) starting at bit offset `bitpos` of a little-endian byte string.
__device__ __forceinline__ uint32_t get_bits(const uint8_t *p, int bitpos, int bits) {
    const int byte = bitpos >> 3, sh = bitpos & 7;
    uint32_t v = (uint32_t)p[byte] | ((uint32_t)p[byte + 1] << 8) | ((uint32_t)p[byte + 2] << 16);
    if (sh + bits > 24) v |= (uint32_t)p[byte + 3] << 24;
    return (v >> sh) & ((1u << bits) - 1u);
}

// Pack 16 consecutive values of BITS bits (16*BITS/8 bytes, a multiple of 4) into 32-bit words.
template <int BITS>
__device__ __forceinline__ void pack16_words(uint32_t *out_words, const uint32_t (&v)[16]) {
    constexpr int NW = 16 * BITS / 32;
    uint32_t w[NW];
#pragma unroll
    for (int i = 0; i < NW; ++i) w[i] = 0;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int bit = i * BITS, wi = bit >> 5, sh = bit & 31;
        w[wi] |= v[i] << sh;
        if (sh + BITS > 32) w[wi + 1] |= v[i] >> (32 - sh);
    }
#pragma unroll
    for (int i = 0; i < NW; ++i) out_words[i] = w[i];
}

// Packs the sixteen values below 2^BITS of every position of a 16-thread group -- byte m of b = coefficient
// t + 16 m -- in coefficient order: position t writes the words of coefficients 16 t .. 16 t + 15.  The
// 16 x 16 byte transpose is four exchange steps of two shuffles, where the way through shared memory takes
// 32 accesses.
template <int BITS>
__device__ __forceinline__ void pack_strided_bytes(uint32_t *poly_words, uint32_t (&b)[4], int t, unsigned gmask) {
    static_assert(BITS == 4 || BITS == 6, "w1 fields");
    {
        const bool hi = t & 8;
        const uint32_t r0 = __shfl_xor_sync(gmask, hi ? b[0] : b[2], 8), r1 = __shfl_xor_sync(gmask, hi ? b[1] : b[3], 8);
        if (hi) {
            b[0] = r0;
            b[1] = r1;
        } else {
            b[2] = r0;
            b[3] = r1;
        }
    }
    {
        const bool hi = t & 4;
        const uint32_t r0 = __shfl_xor_sync(gmask, hi ? b[0] : b[1], 4), r1 = __shfl_xor_sync(gmask, hi ? b[2] : b[3], 4);
        if (hi) {
            b[0] = r0;
            b[2] = r1;
        } else {
            b[1] = r0;
            b[3] = r1;
        }
    }
#pragma unroll
    for (int p = 0; p < 4; p += 2) {  // halfwords of a word pair
        const bool hi = t & 2;
        const uint32_t r = __shfl_xor_sync(gmask, __byte_perm(b[p], b[p + 1], hi ? 0x5410 : 0x7632), 2);
        b[p] = hi ? __byte_perm(r, b[p], 0x7610) : __byte_perm(b[p], r, 0x5410);
        b[p + 1] = hi ? __byte_perm(r, b[p + 1], 0x7632) : __byte_perm(b[p + 1], r, 0x7610);
    }
#pragma unroll
    for (int p = 0; p < 4; p += 2) {  // bytes of a word pair
        const bool hi = t & 1;
        const uint32_t r = __shfl_xor_sync(gmask, __byte_perm(b[p], b[p + 1], hi ? 0x6420 : 0x7531), 1);
        b[p] = __byte_perm(b[p], r, hi ? 0x3514 : 0x5240);
        b[p + 1] = __byte_perm(b[p + 1], r, hi ? 0x3716 : 0x7260);
    }
    uint32_t z[4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        if constexpr (BITS == 4) {
            const uint32_t y = (b[w] | (b[w] >> 4)) & 0x00FF00FFu;
            z[w] = (y | (y >> 8)) & 0xFFFFu;
        } else {
            const uint32_t y = (b[w] & 0x003F003Fu) | ((b[w] & 0x3F003F00u) >> 2);
            z[w] = (y & 0xFFFu) | ((y >> 4) & 0xFFF000u);
        }
    }
    if constexpr (BITS == 4) {
        uint2 *o = reinterpret_cast<uint2 *>(poly_words) + t;
        *o = make_uint2(z[0] | z[1] << 16, z[2] | z[3] << 16);
    } else {
        uint32_t *o = poly_words + 3 * t;
        o[0] = z[0] | z[1] << 24;
        o[1] = (z[1] >> 8) | z[2] << 16;
        o[2] = (z[2] >> 16) | z[3] << 8;
    }
}

// Group helpers: 16 threads, t = position, gmask = lanes of the group.
struct Group {
    int t;
    unsigned gmask;
    int32_t *sm;  // NTT_SMEM_WORDS words
};

__device__ __forceinline__ Group make_group(int32_t *smem_base, int group_in_block) {
    Group g;
    const int lane = threadIdx.x & 31;
    g.t = lane & 15;
    g.gmask = 0xFFFFu << (lane & 16);
    g.sm = smem_base + group_in_block * NTT_SMEM_WORDS;
    return g;
}

// true if any thread of the group has `pred`.
__device__ __forceinline__ bool group_any(const Group &g, bool pred) {
    return __ballot_sync(g.gmask, pred) != 0u;
}

// Reorders the group's strided slice x[i] = a[t + 16 i] into consecutive order
// y[i] = a[16 t + i] through the group's shared memory (for bit packing).
__device__ __forceinline__ void strided_to_contig(const Group &g, const int32_t (&x)[16], int32_t (&y)[16]) {
#pragma unroll
    for (int i = 0; i < 16; ++i) g.sm[g.t + 17 * i] = x[i];
    __syncwarp(g.gmask);
#pragma unroll
    for (int i = 0; i < 16; ++i) y[i] = g.sm[17 * g.t + i];
    __syncwarp(g.gmask);
}

// Fields t + 16 i (i = 0..15) of a packed array of BITS-bit fields, BITS even: sixteen fields are
// BITS / 2 whole words, so all the fields of position t sit at the same shift in words BITS / 2 apart,
// and two word loads and a funnel shift read one (three or four byte loads, shifts and ORs before).
// The array may start at any byte: the words are the aligned ones that hold it.  A word is read only if
// it holds bits of the field, so nothing past the array's last aligned word is touched.
template <int BITS>
__device__ __forceinline__ void unpack_strided(uint32_t (&v)[16], const uint8_t *packed, int t) {
    static_assert(BITS % 2 == 0 && BITS <= 20, "whole words every sixteen fields");
    const unsigned mis = (unsigned)(reinterpret_cast<uintptr_t>(packed) & 3u);
    const unsigned bit = 8u * mis + (unsigned)(BITS * t), sh = bit & 31u;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(packed - mis) + (bit >> 5);
    const int second = sh + BITS > 32u ? 1 : 0;
#pragma unroll
    for (int i = 0; i < 16; ++i)
        v[i] = __funnelshift_r(w[(BITS / 2) * i], w[(BITS / 2) * i + second], sh) & ((1u << BITS) - 1u);
}

// The same for BITS odd and a word-aligned array: sixteen fields are BITS / 2 words and a half, so the even
// i share one word and shift and the odd i another.
template <int BITS>
__device__ __forceinline__ void unpack_strided_odd(uint32_t (&v)[16], const uint8_t *packed, int t) {
    static_assert(BITS % 2 == 1 && BITS <= 17, "a word and a half every sixteen fields");
    const uint32_t *w = reinterpret_cast<const uint32_t *>(packed);
#pragma unroll
    for (int odd = 0; odd < 2; ++odd) {
        const unsigned bit = (unsigned)(BITS * (t + 16 * odd)), sh = bit & 31u;
        const uint32_t *p = w + (bit >> 5);
        const int second = sh + BITS > 32u ? 1 : 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[2 * i + odd] = __funnelshift_r(p[BITS * i], p[BITS * i + second], sh) & ((1u << BITS) - 1u);
    }
}

// z coefficients a[t + 16 i] from a packed (gamma1 - z) polynomial.
template <int MODE>
__device__ __forceinline__ void unpack_z_strided(int32_t (&x)[16], const uint8_t *packed, int t) {
    uint32_t v[16];
    unpack_strided<P<MODE>::Z_BITS>(v, packed, t);
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = Params<MODE>::GAMMA1 - (int32_t)v[i];
}

// z coefficients a[16 t + i] (the contiguous slice of group thread t) from a packed (gamma1 - z)
// polynomial whose start is 4-byte aligned: the slice is 16 * Z_BITS / 32 whole words, read as
// 32-bit loads and split with funnel shifts.
template <int MODE>
__device__ __forceinline__ void unpack_z_contig(int32_t (&x)[16], const uint8_t *packed, int t) {
    constexpr int ZB = P<MODE>::Z_BITS, NWD = ZB / 2;
    const uint32_t *w = reinterpret_cast<const uint32_t *>(packed) + NWD * t;
    uint32_t v[NWD + 1];
#pragma unroll
    for (int k = 0; k < NWD; ++k) v[k] = w[k];
    v[NWD] = 0u;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int bit = i * ZB, wi = bit >> 5, sh = bit & 31;
        const uint32_t r = __funnelshift_r(v[wi], v[wi + 1], sh) & ((1u << ZB) - 1u);
        x[i] = Params<MODE>::GAMMA1 - (int32_t)r;
    }
}

// c coefficients a[t + 16 i] from the challenge's 16 words of two-bit fields (sample_in_ball): field t of
// word i, sign-extended.
__device__ __forceinline__ void challenge_strided(int32_t (&x)[16], const uint32_t *fld, int t) {
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = (int32_t)(fld[i] << (30 - 2 * t)) >> 30;
}

}  // namespace cudil
