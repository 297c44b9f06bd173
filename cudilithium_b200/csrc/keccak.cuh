// Register-resident Keccak-f[1600] for one state per thread, plus SHAKE absorb helpers.
//
// The reference spreads one state over 25 lanes of a warp and exchanges lanes with
// __shfl_sync (include/fips202/fips202.cuh:23-69, :104-147).  Here every thread owns a whole
// state as 50 32-bit registers (lo/hi halves of the 25 lanes): theta/chi become 3-input LOP3
// operations and every 64-bit rotation two funnel shifts, with no shuffles and no idle lanes,
// so independent SHAKE streams (ExpandA's k*l entries, ExpandMask's l entries, one challenge
// hash per attempt) map one-to-one onto threads.
//
// Round constants and rotation offsets are derived from FIPS 202 (the LFSR of Algorithm 5 and
// the (t+1)(t+2)/2 rule of Algorithm 2) at compile time.
#pragma once

#include <cstdint>

#include "params.cuh"

namespace cudil {

struct KeccakTables {
    uint32_t rc_lo[24];
    uint32_t rc_hi[24];
    int rho[25];     // rotation of lane x + 5y
    int pi_src[25];  // B[dst] = rot(A[pi_src[dst]])
};

__host__ __device__ constexpr int keccak_rc_bit(unsigned t) {
    unsigned r = 1;
    if (t % 255 == 0) return 1;
    for (unsigned i = 1; i <= t % 255; i++) {
        r <<= 1;
        if (r & 0x100) r ^= 0x171;
    }
    return (int)(r & 1);
}

__host__ __device__ constexpr KeccakTables make_keccak_tables() {
    KeccakTables k{};
    for (unsigned ir = 0; ir < 24; ir++) {
        uint64_t rc = 0;
        for (unsigned j = 0; j <= 6; j++)
            if (keccak_rc_bit(j + 7 * ir)) rc |= 1ull << ((1u << j) - 1);
        k.rc_lo[ir] = (uint32_t)rc;
        k.rc_hi[ir] = (uint32_t)(rc >> 32);
    }
    for (int i = 0; i < 25; i++) k.rho[i] = 0;
    unsigned x = 1, y = 0;
    for (unsigned t = 0; t < 24; t++) {
        unsigned nx = y, ny = (2 * x + 3 * y) % 5;
        k.rho[x + 5 * y] = (int)(((t + 1) * (t + 2) / 2) % 64);
        x = nx;
        y = ny;
    }
    for (unsigned yy = 0; yy < 5; yy++)
        for (unsigned xx = 0; xx < 5; xx++) k.pi_src[xx + 5 * yy] = (int)(((xx + 3 * yy) % 5) + 5 * xx);
    return k;
}

constexpr KeccakTables kKeccak = make_keccak_tables();
static_assert(kKeccak.rc_lo[0] == 1u && kKeccak.rc_hi[0] == 0u, "keccak rc");
static_assert(kKeccak.rc_lo[23] == 0x80008008u && kKeccak.rc_hi[23] == 0x80000000u, "keccak rc");
static_assert(kKeccak.rho[1] == 1 && kKeccak.rho[24] == 14, "keccak rho");

static __constant__ KeccakTables c_keccak = make_keccak_tables();
// Compile-time copy for device code (rotation amounts and lane permutation fold to immediates).
static constexpr __device__ KeccakTables kKeccakDev = make_keccak_tables();

// 64-bit rotate-left of (h:l) by a compile-time amount (after unrolling), two funnel shifts.
__device__ __forceinline__ void rotl64(uint32_t &ol, uint32_t &oh, uint32_t l, uint32_t h, int n) {
    if (n == 0) {
        ol = l;
        oh = h;
    } else if (n < 32) {
        oh = __funnelshift_l(l, h, n);
        ol = __funnelshift_l(h, l, n);
    } else if (n == 32) {
        ol = h;
        oh = l;
    } else {
        oh = __funnelshift_l(h, l, n - 32);
        ol = __funnelshift_l(l, h, n - 32);
    }
}

// a ^ b ^ c as one LOP3.
__device__ __forceinline__ uint32_t xor3(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x96;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
    return r;
}

// Keccak-f[1600] on a state held as lo/hi 32-bit halves.  Every array index is static after
// unrolling, so the state stays in registers.
//
// Bound: the ALU pipe (LOP3 and funnel shifts, 64 a clock and SM), which one warp a sub-partition
// already fills.  theta folds D into the state as a three-input XOR of the column's two parities, so
// D itself is never formed: 180 instead of 190 operations a round.  Measured on a B200, microseconds
// for one permutation of one warp on every sub-partition, full load: 4.73 before, 4.44 now (180
// operations at the pipe's rate: 4.40).  Rotations moved to the idle FMA pipe (wide multiplies by
// powers of two) measured slower in every mix from one lane (4.46) to all of them (5.31).
__device__ __forceinline__ void keccak_f1600(uint32_t (&al)[25], uint32_t (&ah)[25]) {
#pragma unroll 1
    for (int r = 0; r < 24; ++r) {
        uint32_t cl[5], ch[5], bl[25], bh[25];
#pragma unroll
        for (int x = 0; x < 5; ++x) {
            cl[x] = xor3(xor3(al[x], al[x + 5], al[x + 10]), al[x + 15], al[x + 20]);
            ch[x] = xor3(xor3(ah[x], ah[x + 5], ah[x + 10]), ah[x + 15], ah[x + 20]);
        }
#pragma unroll
        for (int x = 0; x < 5; ++x) {
            uint32_t rl, rh;
            rotl64(rl, rh, cl[(x + 1) % 5], ch[(x + 1) % 5], 1);
#pragma unroll
            for (int y = 0; y < 5; ++y) {
                al[x + 5 * y] = xor3(al[x + 5 * y], cl[(x + 4) % 5], rl);
                ah[x + 5 * y] = xor3(ah[x + 5 * y], ch[(x + 4) % 5], rh);
            }
        }
#pragma unroll
        for (int i = 0; i < 25; ++i) {
            const int s = kKeccakDev.pi_src[i];
            rotl64(bl[i], bh[i], al[s], ah[s], kKeccakDev.rho[s]);
        }
#pragma unroll
        for (int y = 0; y < 5; ++y) {
#pragma unroll
            for (int x = 0; x < 5; ++x) {
                al[x + 5 * y] = bl[x + 5 * y] ^ (~bl[(x + 1) % 5 + 5 * y] & bl[(x + 2) % 5 + 5 * y]);
                ah[x + 5 * y] = bh[x + 5 * y] ^ (~bh[(x + 1) % 5 + 5 * y] & bh[(x + 2) % 5 + 5 * y]);
            }
        }
        al[0] ^= c_keccak.rc_lo[r];
        ah[0] ^= c_keccak.rc_hi[r];
    }
}

// rotl64 of a lane held by two neighbouring threads (own = this thread's half, the low half in the even
// thread): one shuffle and one funnel shift.
__device__ __forceinline__ uint32_t rotl64_pair(uint32_t own, int n) {
    if (n == 0) return own;
    const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, own, 1);
    return n < 32 ? __funnelshift_l(other, own, n) : (n == 32 ? other : __funnelshift_l(own, other, n - 32));
}

// Keccak-f[1600] of one state per pair of threads (half = lane & 1: 0 the low, 1 the high 32 bits of every
// lane).  All 32 lanes of the warp take part.  Half the ALU operations of a thread and 29 shuffles a round:
// a permutation of a warp alone on its sub-partition takes 3.47 us instead of 4.60, and the throughput of a
// full GPU is 10% lower (3.83 against 4.27 G permutations/s).  So it serves kernels whose states are too
// few to give every sub-partition a warp of 32 of them (keccak_pairs).
__device__ __forceinline__ void keccak_f1600_pair(uint32_t (&a)[25], int half) {
#pragma unroll 1
    for (int r = 0; r < 24; ++r) {
        uint32_t c[5], rc[5], b[25];
#pragma unroll
        for (int x = 0; x < 5; ++x) c[x] = xor3(xor3(a[x], a[x + 5], a[x + 10]), a[x + 15], a[x + 20]);
#pragma unroll
        for (int x = 0; x < 5; ++x) rc[x] = rotl64_pair(c[x], 1);
#pragma unroll
        for (int x = 0; x < 5; ++x)
#pragma unroll
            for (int y = 0; y < 5; ++y) a[x + 5 * y] = xor3(a[x + 5 * y], c[(x + 4) % 5], rc[(x + 1) % 5]);
#pragma unroll
        for (int i = 0; i < 25; ++i) {
            const int s = kKeccakDev.pi_src[i];
            b[i] = rotl64_pair(a[s], kKeccakDev.rho[s]);
        }
#pragma unroll
        for (int y = 0; y < 5; ++y)
#pragma unroll
            for (int x = 0; x < 5; ++x)
                a[x + 5 * y] = b[x + 5 * y] ^ (~b[(x + 1) % 5 + 5 * y] & b[(x + 2) % 5 + 5 * y]);
        a[0] ^= half ? c_keccak.rc_hi[r] : c_keccak.rc_lo[r];
    }
}

__device__ __forceinline__ void keccak_zero(uint32_t (&al)[25], uint32_t (&ah)[25]) {
#pragma unroll
    for (int i = 0; i < 25; ++i) al[i] = ah[i] = 0;
}

// Little-endian 8-byte lane from an arbitrary byte pointer; bytes at or beyond `avail` read
// as zero (avail may be >= 8 for a full lane).
__device__ __forceinline__ uint2 load_lane_bytes(const uint8_t *p, int avail) {
    uint32_t lo = 0, hi = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
        if (b < avail) lo |= (uint32_t)p[b] << (8 * b);
#pragma unroll
    for (int b = 0; b < 4; ++b)
        if (b + 4 < avail) hi |= (uint32_t)p[b + 4] << (8 * b);
    return make_uint2(lo, hi);
}

// Lane source for a byte string whose start is 8-byte aligned.
struct AlignedBytes {
    const uint8_t *p;
    long long len;
    __device__ __forceinline__ uint2 lane(long long g) const {
        long long off = g * 8;
        if (off + 8 <= len) return *reinterpret_cast<const uint2 *>(p + off);
        return load_lane_bytes(p + off, (int)(len - off));
    }
    // 32-bit half h of lane g
    __device__ __forceinline__ uint32_t word(long long g, int h) const {
        const long long off = g * 8 + 4 * h;
        if (off + 4 <= len) return *reinterpret_cast<const uint32_t *>(p + off);
        return off < len ? load_lane_bytes(p + off, (int)(len - off)).x : 0u;
    }
};

// Lane source for the concatenation of two 8-byte aligned strings whose first part is a whole
// number of lanes (tr||m, mu||w1, rho'||kappa ...).
struct TwoPart {
    const uint8_t *a;
    int a_lanes;
    const uint8_t *b;
    long long b_len;
    __device__ __forceinline__ uint2 lane(long long g) const {
        if (g < a_lanes) return *reinterpret_cast<const uint2 *>(a + g * 8);
        long long off = (g - a_lanes) * 8;
        if (off + 8 <= b_len) return *reinterpret_cast<const uint2 *>(b + off);
        return load_lane_bytes(b + off, (int)(b_len - off));
    }
    __device__ __forceinline__ uint32_t word(long long g, int h) const {
        if (g < a_lanes) return *reinterpret_cast<const uint32_t *>(a + g * 8 + 4 * h);
        const long long off = (g - a_lanes) * 8 + 4 * h;
        if (off + 4 <= b_len) return *reinterpret_cast<const uint32_t *>(b + off);
        return off < b_len ? load_lane_bytes(b + off, (int)(b_len - off)).x : 0u;
    }
};

// SHAKE absorb of `total_bytes` bytes (lanes from `src`) into a zero state, with the 0x1F / 0x80
// padding applied.  The caller permutes before reading each output block.
template <int RATE, typename Src>
__device__ __forceinline__ void shake_absorb(uint32_t (&al)[25], uint32_t (&ah)[25], const Src &src,
                                             long long total_bytes) {
    constexpr int RL = RATE / 8;
    keccak_zero(al, ah);
    long long nfull = total_bytes / RATE;
    long long g = 0;
    for (long long blk = 0; blk < nfull; ++blk) {
#pragma unroll
        for (int w = 0; w < RL; ++w) {
            uint2 v = src.lane(g + w);
            al[w] ^= v.x;
            ah[w] ^= v.y;
        }
        g += RL;
        keccak_f1600(al, ah);
    }
    const int rem = (int)(total_bytes - nfull * RATE);
#pragma unroll
    for (int w = 0; w < RL; ++w) {
        uint2 v = make_uint2(0u, 0u);
        if (8 * w < rem) v = src.lane(g + w);
        if (8 * w <= rem && rem < 8 * w + 8) {
            const int sh = 8 * (rem - 8 * w);
            if (sh < 32)
                v.x ^= 0x1Fu << sh;
            else
                v.y ^= 0x1Fu << (sh - 32);
        }
        if (w == RL - 1) v.y ^= 0x80000000u;
        al[w] ^= v.x;
        ah[w] ^= v.y;
    }
}

// shake_absorb for long inputs read from global memory: the next block's lanes are loaded before
// the current block is permuted, so their latency overlaps the permutation instead of preceding
// the next one (RATE / 4 more registers live across the permutation; for kernels whose register
// budget allows it, such as the message hashes of the prehash kernels).
template <int RATE, typename Src>
__device__ __forceinline__ void shake_absorb_prefetch(uint32_t (&al)[25], uint32_t (&ah)[25], const Src &src,
                                                      long long total_bytes) {
    constexpr int RL = RATE / 8;
    keccak_zero(al, ah);
    const long long nfull = total_bytes / RATE;
    uint2 nxt[RL];
    if (nfull > 0) {
#pragma unroll
        for (int w = 0; w < RL; ++w) nxt[w] = src.lane(w);
    }
    long long g = 0;
#pragma unroll 1
    for (long long blk = 0; blk < nfull; ++blk) {
#pragma unroll
        for (int w = 0; w < RL; ++w) {
            al[w] ^= nxt[w].x;
            ah[w] ^= nxt[w].y;
        }
        g += RL;
        if (blk + 1 < nfull) {
#pragma unroll
            for (int w = 0; w < RL; ++w) nxt[w] = src.lane(g + w);
        }
        keccak_f1600(al, ah);
    }
    const int rem = (int)(total_bytes - nfull * RATE);
#pragma unroll
    for (int w = 0; w < RL; ++w) {
        uint2 v = make_uint2(0u, 0u);
        if (8 * w < rem) v = src.lane(g + w);
        if (8 * w <= rem && rem < 8 * w + 8) {
            const int sh = 8 * (rem - 8 * w);
            if (sh < 32)
                v.x ^= 0x1Fu << sh;
            else
                v.y ^= 0x1Fu << (sh - 32);
        }
        if (w == RL - 1) v.y ^= 0x80000000u;
        al[w] ^= v.x;
        ah[w] ^= v.y;
    }
}

// SHAKE256 of one message per thread (PAIR = false) or per pair of threads (PAIR = true), for the kernels
// that hash one message per item.  In pair form every lane of the warp calls hash(), with on = false where
// there is no item: the warp runs as many permutations as its longest message takes.
template <bool PAIR>
struct Shake256 {
    static constexpr int LANES = PAIR ? 2 : 1;  // threads per message
    static constexpr int RL = SHAKE256_RATE / 8;
    uint32_t lo[25], hi[PAIR ? 1 : 25];  // the state (PAIR: this thread's halves in lo)
    uint32_t dlo[8], dhi[PAIR ? 1 : 8];  // the first eight lanes of the digest block

    __device__ __forceinline__ int half() const { return (int)(threadIdx.x & 1u); }

    __device__ __forceinline__ void permute() {
        if constexpr (PAIR)
            keccak_f1600_pair(lo, half());
        else
            keccak_f1600(lo, hi);
    }

    // dlo / dhi = the digest's first 64 bytes; the state is left where squeezing can go on (PAIR: only
    // if every message of the warp has as many blocks)
    template <typename Src>
    __device__ __forceinline__ void hash(const Src &src, long long bytes, bool on = true) {
        if constexpr (!PAIR) {
            shake_absorb_prefetch<SHAKE256_RATE>(lo, hi, src, bytes);
            permute();
#pragma unroll
            for (int w = 0; w < 8; ++w) {
                dlo[w] = lo[w];
                dhi[w] = hi[w];
            }
        } else {
            const int h = half();
            const int nfull = on ? (int)(bytes / SHAKE256_RATE) : 0, rem = on ? (int)(bytes - (long long)nfull * SHAKE256_RATE) : 0;
            const int most = (int)__reduce_max_sync(0xFFFFFFFFu, (unsigned)nfull);
#pragma unroll
            for (int i = 0; i < 25; ++i) lo[i] = 0u;
            // block k's words are loaded before block k - 1 is permuted
            uint32_t nxt[RL];
            auto load = [&](int k) {
                if (k < nfull) {
#pragma unroll
                    for (int w = 0; w < RL; ++w) nxt[w] = src.word((long long)k * RL + w, h);
                } else {
                    // the message's rest, 0x1F behind it, 0x80 at the block's end; nothing after that
                    const bool last = k == nfull && on;
#pragma unroll
                    for (int w = 0; w < RL; ++w) {
                        const int at = 8 * w + 4 * h;
                        uint32_t v = 0u;
                        if (last && at < rem) v = src.word((long long)k * RL + w, h);
                        if (last && at <= rem && rem < at + 4) v ^= 0x1Fu << (8 * (rem - at));
                        nxt[w] = v;
                    }
                    if (last && h) nxt[RL - 1] ^= 0x80000000u;
                }
            };
            load(0);
#pragma unroll 1
            for (int k = 0; k <= most; ++k) {
#pragma unroll
                for (int w = 0; w < RL; ++w) lo[w] ^= nxt[w];
                if (k < most) load(k + 1);
                permute();
                if (k == nfull) {
#pragma unroll
                    for (int w = 0; w < 8; ++w) dlo[w] = lo[w];
                }
            }
        }
    }

    // the digest's first NL lanes to p (8-byte aligned)
    template <int NL>
    __device__ __forceinline__ void store(uint8_t *p) const {
#pragma unroll
        for (int w = 0; w < NL; ++w) {
            if constexpr (PAIR)
                reinterpret_cast<uint32_t *>(p)[2 * w + half()] = dlo[w];
            else
                reinterpret_cast<uint2 *>(p)[w] = make_uint2(dlo[w], dhi[w]);
        }
    }

    // the state after absorbing one block made of NL lanes (PAIR: their halves) and the padding, permuted
    template <int NL>
    __device__ __forceinline__ void one_block(const uint32_t (&blo)[NL], const uint32_t (&bhi)[PAIR ? 1 : NL]) {
        static_assert(NL < RL, "one block");
#pragma unroll
        for (int i = 0; i < 25; ++i) {
            lo[i] = i < NL ? blo[i] : 0u;
            if constexpr (!PAIR) hi[i] = i < NL ? bhi[i] : 0u;
        }
        if constexpr (PAIR) {
            if (half())
                lo[RL - 1] ^= 0x80000000u;
            else
                lo[NL] = 0x1Fu;
        } else {
            lo[NL] = 0x1Fu;
            hi[RL - 1] ^= 0x80000000u;
        }
        permute();
    }
};

// Seeded randomized signing: rho' = SHAKE256(seed || le64(ctr), 64), 40 bytes in one SHAKE256 block
// (seed as eight little-endian 32-bit words).
__device__ __forceinline__ void derive_rhoprime(uint2 (&out)[8], const uint32_t (&seed)[8], unsigned long long ctr) {
    uint32_t al[25], ah[25];
    keccak_zero(al, ah);
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        al[w] = seed[2 * w];
        ah[w] = seed[2 * w + 1];
    }
    al[4] = (uint32_t)ctr;
    ah[4] = (uint32_t)(ctr >> 32);
    al[5] = 0x1Fu;
    ah[SHAKE256_RATE / 8 - 1] ^= 0x80000000u;
    keccak_f1600(al, ah);
#pragma unroll
    for (int w = 0; w < 8; ++w) out[w] = make_uint2(al[w], ah[w]);
}

// Absorb of a short input of IN_LANES whole lanes plus an extra 16-bit little-endian nonce
// (seed || nonce, as ExpandA/ExpandS/ExpandMask use); the input must fit one block.
template <int RATE, int IN_LANES>
__device__ __forceinline__ void shake_absorb_seed_nonce(uint32_t (&al)[25], uint32_t (&ah)[25], const uint2 (&seed)[IN_LANES],
                                                        uint32_t nonce16) {
    static_assert(IN_LANES * 8 + 2 < RATE, "single block");
    keccak_zero(al, ah);
#pragma unroll
    for (int w = 0; w < IN_LANES; ++w) {
        al[w] = seed[w].x;
        ah[w] = seed[w].y;
    }
    // bytes 8*IN_LANES, +1 = nonce, +2 = 0x1F
    al[IN_LANES] = (nonce16 & 0xFFFFu) | (0x1Fu << 16);
    ah[RATE / 8 - 1] ^= 0x80000000u;
}

}  // namespace cudil
