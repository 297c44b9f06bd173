// Batched signing kernels (stage-by-stage).  Each kernel maps its stage onto the GPU in the shape
// that stage needs: SHAKE streams one per thread, polynomial arithmetic one per 16-thread group.
//
// Stage list (reference kernel each one replaces):
//   k_sign_setup       mu = H(tr||m), rho' = H(K||mu)     notmp_shake_new_kernel, src/api.cu:137-152
//     (its other blocks) A_hat = ExpandA(rho)               polyvec_matrix_expand_opt_kernel, src/sign.cu:98-163
//   k_sign_unpack_ntt  s1_hat, s2_hat, t0_hat             unpack_fuse_ntt_radix2_opt_kernel, src/sign.cu:306-403
//   k_sign_expand_mask y = ExpandMask(rho', L*nonce + j)  compute_y_opt_kernel, src/sign.cu:463-526
//   k_sign_compute_w   w = invNTT(A_hat NTT(y)); w0, w1   compute_w_128t_kernel, src/sign.cu:605-685
//   k_sign_challenge   c~ = H(mu||w1), c = SampleInBall   compute_cp_kernel, src/sign.cu:687-735
//   k_sign_reject      z, r0, ct0 checks, hints, packing  rej_loop_128t_kernel, src/sign.cu:986-1196
//   k_sig_copy         move the winning attempt           sig_copy_kernel, src/sign.cu:1198-1207
#pragma once

#include "device.cuh"
#include "layout.cuh"

namespace cudil {

constexpr int kBlock = 128;             // threads per block for the SHAKE-stream kernels
constexpr int kGroupsPerBlock = 8;      // 16-thread groups per 128-thread block
constexpr int kItemBlock = 32;          // threads per block for thread-per-item kernels

// rho' = SHAKE256(K || mu, 64) into sp's digest, mu being its digest so far (96 bytes, one block).
template <bool PAIR>
__device__ __forceinline__ void rhoprime_from_mu(Shake256<PAIR> &sp, const uint8_t *key) {
    uint32_t bl[12], bh[PAIR ? 1 : 12];
#pragma unroll
    for (int w = 0; w < 12; ++w) {
        if constexpr (PAIR) {
            bl[w] = w < 4 ? reinterpret_cast<const uint32_t *>(key)[2 * w + sp.half()] : sp.dlo[w < 4 ? 0 : w - 4];
        } else {
            const uint2 k = w < 4 ? ld_lane(key + 8 * w) : make_uint2(sp.dlo[w < 4 ? 0 : w - 4], sp.dhi[w < 4 ? 0 : w - 4]);
            bl[w] = k.x;
            bh[w] = k.y;
        }
    }
    sp.template one_block<12>(bl, bh);
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        sp.dlo[w] = sp.lo[w];
        if constexpr (!PAIR) sp.dhi[w] = sp.hi[w];
    }
}

// ------------------------------------------------------------------ per-item setup

// Fewer items than this fill every sub-partition with one warp of 16 pairs but not with one of 32 states:
// kernels that hash one message per item then use two threads per state (keccak_f1600_pair).
inline bool keccak_pairs(size_t items, int sm_count) { return items <= (size_t)sm_count * 4 * 16; }

// rhop_given: rho' was placed in the row by the caller (randomized signing), only mu is computed.
template <int MODE, bool PAIR>
__device__ __forceinline__ void sign_prehash(uint8_t *pool, size_t pitch, size_t mlen, const uint32_t *mlens, int n, int rhop_given,
                                             int block) {
    using LY = Layout<MODE>;
    using Sp = Shake256<PAIR>;
    const int it = (block * (int)blockDim.x + (int)threadIdx.x) / Sp::LANES;
    const bool on = it < n;
    if (!PAIR && !on) return;
    uint8_t *row = pool + (size_t)(on ? it : 0) * pitch;
    const size_t ml = mlens ? (size_t)mlens[on ? it : 0] : mlen;  // per-item length (<= mlen) when given
    TwoPart src{row + LY::SG_SK + P<MODE>::SK_TR, 4, row + LY::SG_MSG, (long long)ml};
    Sp sp;
    sp.hash(src, (long long)(SEEDBYTES + ml), on);
    if (on) sp.template store<8>(row + LY::SG_MU);
    if (rhop_given) return;
    rhoprime_from_mu(sp, row + LY::SG_SK + P<MODE>::SK_KEY);
    if (on) sp.template store<8>(row + LY::SG_RHOP);
}

// One thread per ExpandA entry; rho at row+rho_off, A_hat (K*L polys) at row+mat_off.
template <int MODE>
__device__ __forceinline__ void expand_a_entry(uint8_t *pool, size_t pitch, size_t rho_off, size_t mat_off, int n, int block,
                                               uint32_t *stage) {
    constexpr int K = Params<MODE>::K, L = Params<MODE>::L, KL = K * L;
    const int s = block * (int)blockDim.x + (int)threadIdx.x;
    if (s >= n * KL) return;
    const int it = s / KL, ij = s % KL;
    uint8_t *row = pool + (size_t)it * pitch;
    uint2 rho[4];
    ld_lanes(rho, row + rho_off);
    int32_t *out = reinterpret_cast<int32_t *>(row + mat_off) + (size_t)ij * N;
    expand_a_row(rho, ij / L, ij % L, out, stage + threadIdx.x * EA_STAGE);
}

// Blocks [0, hash_blocks) hash the messages, the others run ExpandA: neither needs the other, and the hash
// chains of a small batch would leave most of the GPU idle in a launch of their own.  (1024 Dilithium3 items:
// prehash and ExpandA 21 + 73 us apart; verification's prepare and ExpandA 96 + 73 us.)
template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kItemBlock) k_sign_setup(uint8_t *pool, size_t pitch, size_t mlen, const uint32_t *mlens, int n,
                                                           int rhop_given, unsigned hash_blocks) {
    using LY = Layout<MODE>;
    __shared__ __align__(16) uint32_t s_stage[kItemBlock * EA_STAGE];
    if (blockIdx.x < hash_blocks)
        sign_prehash<MODE, PAIR>(pool, pitch, mlen, mlens, n, rhop_given, (int)blockIdx.x);
    else
        expand_a_entry<MODE>(pool, pitch, LY::SG_SK + P<MODE>::SK_RHO, LY::sg_mat(mlen), n, (int)(blockIdx.x - hash_blocks), s_stage);
}

// The same with rho read from the packed keys (key i at keys + i * key_bytes, rho = its first 32
// bytes), so the build of a cache row's Â needs no other part of the row.  One warp per block: a few thousand
// entries then spread evenly over the SMs (public-key caches of 2048 Dilithium2 keys 96 us with four warps a
// block, 78 with one; of 10 000 keys 294 and 275).
template <int MODE>
__global__ void __launch_bounds__(kItemBlock) k_expand_a_keys(const uint8_t *keys, size_t key_bytes, uint8_t *rows, size_t pitch,
                                                          size_t mat_off, int n) {
    constexpr int K = Params<MODE>::K, L = Params<MODE>::L, KL = K * L;
    __shared__ __align__(16) uint32_t s_stage[kItemBlock * EA_STAGE];
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n * KL) return;
    const int it = s / KL, ij = s % KL;
    const uint8_t *key = keys + (size_t)it * key_bytes;
    uint2 rho[4];
    if ((reinterpret_cast<uintptr_t>(key) & 7u) == 0u) {
        ld_lanes(rho, key);
    } else {
#pragma unroll
        for (int w = 0; w < 4; ++w) rho[w] = load_lane_bytes(key + 8 * w, 8);
    }
    int32_t *out = reinterpret_cast<int32_t *>(rows + (size_t)it * pitch + mat_off) + (size_t)ij * N;
    expand_a_row(rho, ij / L, ij % L, out, s_stage + threadIdx.x * EA_STAGE);
}

// Coefficients a[t + 16 i] of secret polynomial p of a packed key: s1 (p < L), s2 (p < L + K), then t0.
template <int MODE>
__device__ __forceinline__ void unpack_secret(int32_t (&x)[16], const uint8_t *sk, int p, int t) {
    using PM = P<MODE>;
    constexpr int K = PM::K, L = PM::L;
    const bool eta = p < L + K;
    const uint8_t *src = sk + (eta ? PM::SK_S1 + (size_t)p * PM::POLYETA_PACKED : PM::SK_T0 + (size_t)(p - L - K) * POLYT0_PACKED);
    const int32_t top = eta ? PM::ETA : 1 << (D - 1);
    uint32_t v[16];
    if ((reinterpret_cast<uintptr_t>(sk) & 3u) == 0u) {
        if (!eta) {
            unpack_strided_odd<13>(v, src, t);
        } else if constexpr (PM::ETA_BITS == 3) {
            unpack_strided_odd<3>(v, src, t);
        } else {
            unpack_strided<4>(v, src, t);
        }
    } else {
        // packed keys at any byte: three byte loads, two where the field ends with the key's last byte
        const int bits = eta ? PM::ETA_BITS : 13;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int bit = (t + 16 * i) * bits, byte = bit >> 3, sh = bit & 7;
            uint32_t w = src[byte];
            if (sh + bits > 8) w |= (uint32_t)src[byte + 1] << 8;
            if (sh + bits > 16) w |= (uint32_t)src[byte + 2] << 16;
            v[i] = (w >> sh) & ((1u << bits) - 1u);
        }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = top - (int32_t)v[i];
}

// One 16-thread group per secret polynomial: unpack (eta / 13-bit) and forward NTT.
template <int MODE>
__global__ void __launch_bounds__(kBlock) k_sign_unpack_ntt(uint8_t *pool, size_t pitch, size_t mlen, int n) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    constexpr int K = PM::K, L = PM::L, NP = L + 2 * K;
    __shared__ int32_t sm[kGroupsPerBlock * NTT_SMEM_WORDS];
    const int gid = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const int it = gid / NP, p = gid % NP;
    if (it >= n) return;
    Group g = make_group(sm, threadIdx.x >> 4);
    uint8_t *row = pool + (size_t)it * pitch;
    int32_t x[16];
    unpack_secret<MODE>(x, row + LY::SG_SK, p, g.t);
    const size_t dst = p < L ? LY::sg_s1(mlen) + (size_t)p * LY::POLY
                             : (p < L + K ? LY::sg_s2(mlen) + (size_t)(p - L) * LY::POLY : LY::sg_t0(mlen) + (size_t)(p - L - K) * LY::POLY);
    ntt16s(x, g.sm, g.gmask, g.t);
    store16_chunks(reinterpret_cast<int32_t *>(row + dst), x, g.t);
}

// ------------------------------------------------------------------ per-attempt stages

// exec_lut entry = (item << 16) | nonce, as the reference's task_lut (src/api.cu:221-230).
template <int MODE>
__global__ void __launch_bounds__(kBlock) k_sign_expand_mask(const uint8_t *sign_pool, size_t sp, uint8_t *temp_pool,
                                                             size_t tp, const uint32_t *exec_lut, int nexec, int nitems) {
    using LY = Layout<MODE>;
    constexpr int L = Params<MODE>::L;
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= nexec * L) return;
    const int e = s / L, j = s % L;
    const uint32_t info = exec_lut[e];
    const uint32_t item = info >> 16, nonce = info & 0xFFFFu;
    if (!bc_ok(item < (uint32_t)nitems, BC_STAGE_ITEM)) return;
    uint2 rhop[8];
    ld_lanes(rhop, sign_pool + (size_t)item * sp + LY::SG_RHOP);
    expand_mask_stream<MODE>(temp_pool + (size_t)e * tp + LY::TP_Y + (size_t)j * P<MODE>::POLYZ_PACKED, rhop,
                             (uint32_t)(L * nonce + j));
}

// AW attempts per 128-thread block: NTT(y_j) into shared memory, then one group per row i
// computes w_i = invNTT(sum_j A_ij * y_hat_j), Decompose, w0 and packed w1.
template <int MODE, int AW>
__global__ void __launch_bounds__(kBlock) k_sign_compute_w(const uint8_t *sign_pool, size_t sp, size_t mlen, uint8_t *temp_pool,
                                                           size_t tp, const uint32_t *exec_lut, int nexec, int nitems) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    constexpr int K = PM::K, L = PM::L;
    __shared__ __align__(16) int32_t s_yhat[AW][L][N];
    __shared__ int32_t sm[kGroupsPerBlock * NTT_SMEM_WORDS];
    const int gi = threadIdx.x >> 4;
    Group g = make_group(sm, gi);
    const int e0 = blockIdx.x * AW;
    for (int u = gi; u < AW * L; u += kGroupsPerBlock) {
        const int a = u / L, j = u % L, e = e0 + a;
        if (e >= nexec) continue;
        int32_t x[16];
        unpack_z_strided<MODE>(x, temp_pool + (size_t)e * tp + LY::TP_Y + (size_t)j * PM::POLYZ_PACKED, g.t);
        ntt16s(x, g.sm, g.gmask, g.t);
        store16_smem(&s_yhat[a][j][0], x, g.t);
    }
    __syncthreads();
    for (int u = gi; u < AW * K; u += kGroupsPerBlock) {
        const int a = u / K, i = u % K, e = e0 + a;
        if (e >= nexec) continue;
        const uint32_t item = exec_lut[e] >> 16;
        if (!bc_ok(item < (uint32_t)nitems, BC_STAGE_ITEM)) continue;
        const int32_t *mat = reinterpret_cast<const int32_t *>(sign_pool + (size_t)item * sp + LY::sg_mat(mlen)) + (size_t)i * L * N;
        int32_t acc[16];
        dot16<L, (L + 1) / 2>(acc, &s_yhat[a][0][0], g.t, [&](int j) { return mat + (size_t)j * N; });
        intt16s(acc, g.sm, g.gmask, g.t);
        uint8_t *trow = temp_pool + (size_t)e * tp;
        int32_t *w0 = reinterpret_cast<int32_t *>(trow + LY::TP_W0) + (size_t)i * N;
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
        pack16_words<PM::W1_BITS>(reinterpret_cast<uint32_t *>(trow + LY::TP_W1P + (size_t)i * PM::POLYW1_PACKED + g.t * 2 * PM::W1_BITS), v);
    }
}

// SampleInBall(c~) (src/sign.cu:767-787), one thread per challenge: thread `self` of STRIDE threads that
// share the scratch, SIB_WORDS words per thread.  The result is 16 words, two bits per coefficient (0, 1 or
// 3 = -1; coefficient p in bits 2 (p % 16) of word p / 16), word k of a thread at fld[k * STRIDE] so that
// the dynamically indexed accesses of neighbouring threads hit distinct banks; sib_result gives fld.  The
// drawn positions are bytes of 17 words (an odd number: no two lanes' same byte in one bank).
//
// Two passes.  The first draws the TAU positions from the squeezed block in registers: a byte is stored
// and the count advanced by its comparison, with no load on the way.  The second moves the coefficients,
// c[i] = c[b], c[b] = sign, with one dependent read of the result per position (c[i] takes an atomic OR
// that nothing waits for: coefficient i is 0 until step i).  Drawing from shared memory and moving position
// by position on separate occupancy and sign masks took about 650 cycles a position: a challenge kernel
// of one warp per sub-partition (8 permutations, Dilithium2) took 54 us.
constexpr int SIB_POS_WORDS = 17, SIB_WORDS = SIB_POS_WORDS + 16;

template <int STRIDE>
__device__ __forceinline__ uint32_t *sib_result(uint32_t *scratch, int self) {
    return scratch + SIB_POS_WORDS * STRIDE + self;
}

template <int TAU, int STRIDE, bool PAIR = false>
__device__ __forceinline__ void sample_in_ball(Shake256<PAIR> &sp, uint32_t *scratch, int self) {
    static_assert(TAU <= 4 * SIB_POS_WORDS, "positions");
    uint32_t *pos = scratch + SIB_POS_WORDS * self, *fld = sib_result<STRIDE>(scratch, self);
    // the block c~ (the digest's first four lanes), then SHAKE256 of it
    uint32_t cl[4], ch[PAIR ? 1 : 4];
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        cl[w] = sp.dlo[w];
        if constexpr (!PAIR) ch[w] = sp.dhi[w];
    }
    sp.template one_block<4>(cl, ch);
    // (pair form: the even thread draws; its odd neighbour hands it the high halves)
    const bool draws = !PAIR || sp.half() == 0;
    if (draws) {
#pragma unroll
        for (int k = 0; k < 16; ++k) fld[k * STRIDE] = 0;
    }
    uint32_t sl = 0, sh = 0, i = draws ? N - TAU : N;
    uint8_t *out = reinterpret_cast<uint8_t *>(pos);
    bool first = true;  // the first block's first lane holds the signs
#pragma unroll 1
    for (;;) {
#pragma unroll
        for (int w = 0; w < 2 * (SHAKE256_RATE / 8); ++w) {
            uint32_t word;
            if constexpr (PAIR)
                word = (w & 1) ? __shfl_xor_sync(0xFFFFFFFFu, sp.lo[w >> 1], 1) : sp.lo[w >> 1];
            else
                word = (w & 1) ? sp.hi[w >> 1] : sp.lo[w >> 1];
            if (first && w == 0) sl = word;
            if (first && w == 1) sh = word;
            if ((w < 2 && first) || i >= (uint32_t)N) continue;
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                const uint32_t b = (word >> (8 * m)) & 0xFFu;
                if (b <= i && i < (uint32_t)N) {
                    *out++ = (uint8_t)b;
                    ++i;
                }
            }
        }
        first = false;
        if constexpr (PAIR) {
            if (!__any_sync(0xFFFFFFFFu, i < (uint32_t)N)) break;
        } else {
            if (i >= (uint32_t)N) break;
        }
        sp.permute();
    }
    if (!draws) return;
#pragma unroll 1
    for (int k0 = 0; k0 < TAU; k0 += 4) {
        uint32_t pw = pos[k0 >> 2];
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            if (k0 + m >= TAU) break;
            const uint32_t b = pw & 0xFFu, p = (uint32_t)(N - TAU + k0 + m), at = 2u * (b & 15u);
            pw >>= 8;
            uint32_t *wb = fld + (b >> 4) * STRIDE;
            const uint32_t v = *wb, c = (v >> at) & 3u;
            *wb = (v & ~(3u << at)) | (((sl & 1u) ? 3u : 1u) << at);
            if (c) atomicOr(fld + (p >> 4) * STRIDE, c << (2u * (p & 15u)));
            sl = __funnelshift_r(sl, sh, 1);
            sh >>= 1;
        }
    }
}

// The same from the 32 bytes of c~ in four lanes, one thread per challenge.
template <int TAU, int STRIDE>
__device__ __forceinline__ void sample_in_ball(const uint2 (&ct)[4], uint32_t *scratch, int self) {
    Shake256<false> sp;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        sp.dlo[w] = ct[w].x;
        sp.dhi[w] = ct[w].y;
    }
    sample_in_ball<TAU, STRIDE, false>(sp, scratch, self);
}

// Copies a challenge's result (16 words) to 64 bytes at p.
template <int STRIDE>
__device__ __forceinline__ void sib_store(uint8_t *p, const uint32_t *scratch, int self) {
    const uint32_t *f = scratch + SIB_POS_WORDS * STRIDE + self;
    uint4 *o = reinterpret_cast<uint4 *>(p);
#pragma unroll
    for (int k = 0; k < 4; ++k)
        o[k] = make_uint4(f[(4 * k) * STRIDE], f[(4 * k + 1) * STRIDE], f[(4 * k + 2) * STRIDE], f[(4 * k + 3) * STRIDE]);
}

// Thread-per-item kernels run TB = kItemBlock threads per block so that batches of a few thousand
// items still spread over every SM.
template <int MODE, bool PAIR, int TB = kItemBlock>
__global__ void __launch_bounds__(TB) k_sign_challenge(const uint8_t *sign_pool, size_t sp, uint8_t *temp_pool, size_t tp,
                                                       const uint32_t *exec_lut, int nexec, int nitems) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    using Sp = Shake256<PAIR>;
    __shared__ uint32_t s_sib[SIB_WORDS * TB];
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) / Sp::LANES;
    bool on = e < nexec;
    const uint32_t item = on ? exec_lut[e] >> 16 : 0u;
    on = on && bc_ok(item < (uint32_t)nitems, BC_STAGE_ITEM);
    if (!PAIR && !on) return;
    uint8_t *trow = temp_pool + (size_t)(on ? e : 0) * tp;
    TwoPart src{sign_pool + (size_t)(on ? item : 0u) * sp + LY::SG_MU, 8, trow + LY::TP_W1P, PM::W1PACKED_BYTES};
    Sp sh;
    sh.hash(src, CRHBYTES + PM::W1PACKED_BYTES, on);
    if (on) sh.template store<4>(trow + LY::TP_SIG);
    sample_in_ball<PM::TAU, TB, PAIR>(sh, s_sib, threadIdx.x);
    if (on && (!PAIR || sh.half() == 0)) sib_store<TB>(trow + LY::TP_CMASK, s_sib, threadIdx.x);
}

// One warp (a block of its own: attempts end after different numbers of steps) per attempt: c_hat = NTT(c); r0 = w0 - c*s2, z = y + c*s1 and c*t0 (norm checks);
// MakeHint (at most OMEGA, positions in ascending order).  The two 16-thread groups of the warp
// take the attempt's polynomials in pairs (poly 2p + half), so they follow the same control flow
// and a rejection ends the attempt for the whole warp.  On acceptance the temp row holds the
// complete signature and done[e] = 1 (src/sign.cu:1010-1195).
template <int MODE>
__global__ void __launch_bounds__(32, 16) k_sign_reject(const uint8_t *sign_pool, size_t sp, size_t mlen, uint8_t *temp_pool,
                                                        size_t tp, const uint32_t *exec_lut, uint8_t *done, int nexec,
                                                        int nitems) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    constexpr int K = PM::K, L = PM::L, OMEGA = PM::OMEGA;
    __shared__ int32_t sm[2 * NTT_SMEM_WORDS];
    const int e = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (e >= nexec) return;  // (the same for the whole warp)
    Group g = make_group(sm, threadIdx.x >> 4);
    const int lane = threadIdx.x & 31, lane_off = lane & 16, half = lane_off >> 4;
    const uint32_t item = exec_lut[e] >> 16;
    if (!bc_ok(item < (uint32_t)nitems, BC_STAGE_ITEM)) return;
    const uint8_t *srow = sign_pool + (size_t)item * sp;
    uint8_t *trow = temp_pool + (size_t)e * tp;

    uint32_t masks[16];
    {
        const uint4 *mi = reinterpret_cast<const uint4 *>(trow + LY::TP_CMASK);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            uint4 v = mi[k];
            masks[4 * k] = v.x;
            masks[4 * k + 1] = v.y;
            masks[4 * k + 2] = v.z;
            masks[4 * k + 3] = v.w;
        }
    }
    // both groups transform c (same data, same instructions)
    int32_t ch[16];
    challenge_strided(ch, masks, g.t);
    ntt16s(ch, g.sm, g.gmask, g.t);
#pragma unroll
    for (int m = 0; m < 16; ++m) ch[m] = scale_f(ch[m]);

    // Acceptance needs every check to pass (src/sign.cu:1026-1144 checks z, then r0, then ct0);
    // here the most selective runs first: pair steps of the r0_i (r0 replaces w0 in the temp row,
    // for the hints), then of the z_j, then of the ct0_i with the hints.  K is even for every
    // parameter set; L is odd for two of them, so the last z pair may leave the second group
    // without a polynomial (it transforms zeros and stores nothing).  One inverse-NTT call site;
    // the next step's key rows load while the current one transforms.
    const int32_t *s1 = reinterpret_cast<const int32_t *>(srow + LY::sg_s1(mlen));
    const int32_t *s2 = reinterpret_cast<const int32_t *>(srow + LY::sg_s2(mlen));
    const int32_t *t0 = reinterpret_cast<const int32_t *>(srow + LY::sg_t0(mlen));
    constexpr int PR = K / 2, PZ = (L + 1) / 2, NSTEP = 2 * PR + PZ;
    auto operand = [&](int step) -> const int32_t * {
        if (step < PR) return s2 + (size_t)(2 * step + half) * N;
        if (step < PR + PZ) {
            const int j = 2 * (step - PR) + half;
            return s1 + (size_t)(j < L ? j : L - 1) * N;
        }
        return t0 + (size_t)(2 * (step - PR - PZ) + half) * N;
    };
    uint8_t *hs = trow + LY::TP_SIG + PM::SIG_H;
    int cnt = 0;
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
        intt16s(x, g.sm, g.gmask, g.t);
        bool bad = false;
        if (is_z) {
            int32_t y[16];
            unpack_z_strided<MODE>(y, trow + LY::TP_Y + (size_t)(act ? k : 0) * PM::POLYZ_PACKED, g.t);
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                x[m] = reduce32(x[m] + (act ? y[m] : 0));
                bad |= act && exceeds(x[m], PM::GAMMA1 - PM::BETA);
            }
            if (__ballot_sync(0xFFFFFFFFu, bad)) return;
            int32_t zc[16];
            strided_to_contig(g, x, zc);
            if (act) {
                uint32_t v[16];
#pragma unroll
                for (int m = 0; m < 16; ++m) v[m] = (uint32_t)(PM::GAMMA1 - zc[m]);
                pack16_words<PM::Z_BITS>(
                    reinterpret_cast<uint32_t *>(trow + LY::TP_SIG + PM::SIG_Z + (size_t)k * PM::POLYZ_PACKED + g.t * 2 * PM::Z_BITS), v);
            }
        } else if (is_r0) {
            int32_t *w0 = reinterpret_cast<int32_t *>(trow + LY::TP_W0) + (size_t)k * N;
            int32_t r0[16];
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                r0[m] = reduce32(w0[g.t + 16 * m] - x[m]);
                bad |= exceeds(r0[m], PM::GAMMA2 - PM::BETA);
            }
            if (__ballot_sync(0xFFFFFFFFu, bad)) return;
#pragma unroll
            for (int m = 0; m < 16; ++m) w0[g.t + 16 * m] = r0[m];
        } else {
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                x[m] = reduce32(x[m]);
                bad |= exceeds(x[m], PM::GAMMA2);
            }
            if (__ballot_sync(0xFFFFFFFFu, bad)) return;
            const int32_t *r0 = reinterpret_cast<const int32_t *>(trow + LY::TP_W0) + (size_t)k * N;
            const uint8_t *w1p = trow + LY::TP_W1P + (size_t)k * PM::POLYW1_PACKED;
            // hint bits of poly k: bit m of hb = hint of coefficient t + 16 m
            unsigned hb = 0;
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                const int32_t w1 = (int32_t)get_bits(w1p, (g.t + 16 * m) * PM::W1_BITS, PM::W1_BITS);
                hb |= make_hint<MODE>(r0[g.t + 16 * m] + x[m], w1) << m;
            }
            // hint counts of both polynomials of the pair, then the positions in ascending
            // coefficient order: poly 2p first, then poly 2p + 1
            int tot = __popc(hb);
#pragma unroll
            for (int o = 8; o >= 1; o >>= 1) tot += __shfl_xor_sync(0xFFFFFFFFu, tot, o);
            const int tot0 = __shfl_sync(0xFFFFFFFFu, tot, 0), tot1 = __shfl_sync(0xFFFFFFFFu, tot, 16);
            if (cnt + tot0 + tot1 > OMEGA) return;
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
    for (int q = cnt + lane; q < OMEGA; q += 32) hs[q] = 0;
    if (lane == 0) done[e] = 1;
}

struct CopyEntry {
    size_t exec_idx;
    size_t sign_idx;
};

template <int MODE>
__global__ void k_sig_copy(uint8_t *sign_pool, size_t sp, const uint8_t *temp_pool, size_t tp, const CopyEntry *lut,
                           size_t nexec, size_t nitems) {
    const CopyEntry e = lut[blockIdx.x];
    if (!bc_ok(e.exec_idx < nexec && e.sign_idx < nitems, BC_COPY_ENTRY)) return;
    const uint8_t *src = temp_pool + e.exec_idx * tp + Layout<MODE>::TP_SIG;
    uint8_t *dst = sign_pool + e.sign_idx * sp + Layout<MODE>::SG_SIG;
    // (both start at a multiple of 16 bytes and their areas are whole 256-byte units)
    for (int i = threadIdx.x; i < (P<MODE>::SIG_BYTES + 15) / 16; i += blockDim.x)
        reinterpret_cast<uint4 *>(dst)[i] = reinterpret_cast<const uint4 *>(src)[i];
}

}  // namespace cudil
