// Batched verification kernels (reference: gpu_verify, src/verify.cu:28-325, one warp per
// signature).  Split by stage shape:
//   k_verify_setup    one thread or pair per signature: hint-encoding checks (src/verify.cu:51-93),
//                     tr' = H(pk), mu = H(tr'||m), c = SampleInBall(c~)
//                     and, in blocks of its own, one thread per ExpandA entry
//   k_verify_w        16-thread groups: z norm check + NTT(z), NTT(c), A z - c t1 2^d, invNTT,
//                     UseHint, pack w1'
//   k_verify_final    one thread per signature: c~' = H(mu||w1') and compare
#pragma once

#include "sign_kernels.cuh"

namespace cudil {

template <int MODE, bool PAIR, int TB>
__device__ __forceinline__ void verify_prepare(uint8_t *pool, size_t pitch, size_t mlen, const uint32_t *mlens, int n, int block,
                                               uint32_t *s_sib) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    using Sp = Shake256<PAIR>;
    constexpr int K = PM::K, OMEGA = PM::OMEGA;
    const int it = (block * TB + (int)threadIdx.x) / Sp::LANES;
    const bool on = it < n;
    if (!PAIR && !on) return;
    uint8_t *row = pool + (size_t)(on ? it : 0) * pitch;
    uint8_t *aux = row + LY::vf_aux(mlen);
    Sp sp;

    // hint encoding: per-poly counts non-decreasing and <= OMEGA, positions strictly increasing
    // inside each poly, unused slots zero
    int status = 0;
    if (on && (!PAIR || sp.half() == 0)) {
        const uint8_t *h = row + LY::VF_SIG + PM::SIG_H;
        int k = 0;
        for (int i = 0; i < K && !status; ++i) {
            const int end = h[OMEGA + i];
            if (end < k || end > OMEGA) {
                status = 1;
                break;
            }
            for (int j = k + 1; j < end; ++j)
                if (h[j] <= h[j - 1]) status = 1;
            k = end;
        }
        if (!status)
            for (int j = k; j < OMEGA; ++j)
                if (h[j]) status = 1;
        reinterpret_cast<int *>(aux + 64)[0] = status;
    }
    __syncwarp();

    // tr' = SHAKE256(pk, 32) -> row + VF_TRM (m follows it)
    AlignedBytes pk{row + LY::VF_PK, PM::PK_BYTES};
    sp.hash(pk, PM::PK_BYTES, on);
    if (on) sp.template store<4>(row + LY::VF_TRM);
    __syncwarp();  // (pair form: each thread wrote its halves)
    // mu = SHAKE256(tr' || m, 64); per-item length (<= mlen) when given
    const size_t ml = mlens ? (size_t)mlens[on ? it : 0] : mlen;
    AlignedBytes tm{row + LY::VF_TRM, (long long)(SEEDBYTES + ml)};
    sp.hash(tm, (long long)(SEEDBYTES + ml), on);
    if (on) sp.template store<8>(row + LY::vf_mu(mlen));

#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const uint2 v = ld_lane(row + LY::VF_SIG + 8 * w);
        if constexpr (PAIR) {
            sp.dlo[w] = sp.half() ? v.y : v.x;
        } else {
            sp.dlo[w] = v.x;
            sp.dhi[w] = v.y;
        }
    }
    sample_in_ball<PM::TAU, TB, PAIR>(sp, s_sib, threadIdx.x);
    if (on && (!PAIR || sp.half() == 0)) sib_store<TB>(aux, s_sib, threadIdx.x);
}

// Blocks [0, prep_blocks) prepare the signatures, the others run ExpandA (as k_sign_setup).
template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kItemBlock) k_verify_setup(uint8_t *pool, size_t pitch, size_t mlen, const uint32_t *mlens, int n,
                                                             unsigned prep_blocks) {
    using LY = Layout<MODE>;
    // SampleInBall scratch or ExpandA rows
    __shared__ __align__(16) uint32_t s_words[kItemBlock * (EA_STAGE > SIB_WORDS ? EA_STAGE : SIB_WORDS)];
    if (blockIdx.x < prep_blocks)
        verify_prepare<MODE, PAIR, kItemBlock>(pool, pitch, mlen, mlens, n, (int)blockIdx.x, s_words);
    else
        expand_a_entry<MODE>(pool, pitch, LY::VF_PK, LY::vf_mat(mlen), n, (int)(blockIdx.x - prep_blocks), s_words);
}

// AV signatures per 128-thread block.  Phase 1 units: (sig, j<L) -> z_hat_j, (sig, L) -> c_hat.
// Phase 2 units: (sig, i<K) -> w1'_i packed.
template <int MODE, int AV>
__global__ void __launch_bounds__(kBlock) k_verify_w(uint8_t *pool, size_t pitch, size_t mlen, int n) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    constexpr int K = PM::K, L = PM::L, OMEGA = PM::OMEGA;
    __shared__ __align__(16) int32_t s_hat[AV][L + 1][N];
    __shared__ uint32_t s_hint[AV][K][8];
    __shared__ int32_t sm[kGroupsPerBlock * NTT_SMEM_WORDS];
    const int gi = threadIdx.x >> 4;
    Group g = make_group(sm, gi);
    const int i0 = blockIdx.x * AV;

    for (int q = threadIdx.x; q < AV * K * 8; q += blockDim.x) (&s_hint[0][0][0])[q] = 0;
    __syncthreads();
    // hint bitmaps (positions are validated by k_verify_setup; a bad encoding only needs to not
    // index out of range here, which byte positions < 256 guarantee)
    for (int q = threadIdx.x; q < AV * K; q += blockDim.x) {
        const int a = q / K, i = q % K, it = i0 + a;
        if (it >= n) continue;
        const uint8_t *h = pool + (size_t)it * pitch + LY::VF_SIG + PM::SIG_H;
        const int start = (i == 0) ? 0 : h[OMEGA + i - 1];
        int end = h[OMEGA + i];
        if (end > OMEGA) end = OMEGA;
        for (int j = start; j < end; ++j) atomicOr(&s_hint[a][i][h[j] >> 5], 1u << (h[j] & 31));
    }

    for (int u = gi; u < AV * (L + 1); u += kGroupsPerBlock) {
        const int a = u / (L + 1), j = u % (L + 1), it = i0 + a;
        if (it >= n) continue;
        uint8_t *row = pool + (size_t)it * pitch;
        int32_t x[16];
        if (j < L) {
            unpack_z_strided<MODE>(x, row + LY::VF_SIG + PM::SIG_Z + (size_t)j * PM::POLYZ_PACKED, g.t);
            bool bad = false;
#pragma unroll
            for (int m = 0; m < 16; ++m) bad |= exceeds(x[m], PM::GAMMA1 - PM::BETA);
            if (group_any(g, bad) && g.t == 0) atomicOr(reinterpret_cast<int *>(row + LY::vf_aux(mlen) + 64), 2);
        } else {
            uint32_t masks[16];
            const uint4 *mi = reinterpret_cast<const uint4 *>(row + LY::vf_aux(mlen));
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                uint4 v = mi[k];
                masks[4 * k] = v.x;
                masks[4 * k + 1] = v.y;
                masks[4 * k + 2] = v.z;
                masks[4 * k + 3] = v.w;
            }
            challenge_strided(x, masks, g.t);
        }
        ntt16s(x, g.sm, g.gmask, g.t);
        if (j == L) {  // -c_hat with the inverse transform's factor (A_hat carries it already)
#pragma unroll
            for (int m = 0; m < 16; ++m) x[m] = -scale_f(x[m]);
        }
        store16_smem(&s_hat[a][j][0], x, g.t);
    }
    __syncthreads();

    for (int u = gi; u < AV * K; u += kGroupsPerBlock) {
        const int a = u / K, i = u % K, it = i0 + a;
        if (it >= n) continue;
        uint8_t *row = pool + (size_t)it * pitch;
        // t1_i * 2^d, NTT
        int32_t t1[16];
        {
            uint32_t v[16];
            unpack_strided<10>(v, row + LY::VF_PK + SEEDBYTES + (size_t)i * POLYT1_PACKED, g.t);
#pragma unroll
            for (int m = 0; m < 16; ++m) t1[m] = (int32_t)(v[m] << D);
        }
        ntt16s(t1, g.sm, g.gmask, g.t);
        const int32_t *mat = reinterpret_cast<const int32_t *>(row + LY::vf_mat(mlen)) + (size_t)i * L * N;
        int32_t acc[16];
        dot16<L, (L + 1) / 2>(acc, &s_hat[a][0][0], g.t, [&](int j) { return mat + (size_t)j * N; });
        int32_t cv[16];
        load16_smem(cv, &s_hat[a][L][0], g.t);
        // + (-c) t1: |sum| < 1.2 q, reduced below q for the inverse transform
#pragma unroll
        for (int m = 0; m < 16; ++m) acc[m] = reduce32(acc[m] + montmul(cv[m], t1[m]));
        intt16s(acc, g.sm, g.gmask, g.t);
        int32_t w1[16];
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            const int c = g.t + 16 * m;
            const unsigned hb = (s_hint[a][i][c >> 5] >> (c & 31)) & 1u;
            w1[m] = use_hint<MODE>(caddq(reduce32(acc[m])), hb);
        }
        int32_t w1c[16];
        strided_to_contig(g, w1, w1c);
        uint32_t v[16];
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = (uint32_t)w1c[m];
        pack16_words<PM::W1_BITS>(
            reinterpret_cast<uint32_t *>(row + LY::vf_mu(mlen) + CRHBYTES + (size_t)i * PM::POLYW1_PACKED + g.t * 2 * PM::W1_BITS), v);
    }
}

template <int MODE, bool PAIR>
__global__ void __launch_bounds__(kBlock) k_verify_final(uint8_t *pool, size_t pitch, size_t mlen, int n) {
    using PM = P<MODE>;
    using LY = Layout<MODE>;
    using Sp = Shake256<PAIR>;
    const int it = (blockIdx.x * blockDim.x + threadIdx.x) / Sp::LANES;
    const bool on = it < n;
    if (!PAIR && !on) return;
    uint8_t *row = pool + (size_t)(on ? it : 0) * pitch;
    uint8_t *aux = row + LY::vf_aux(mlen);
    AlignedBytes src{row + LY::vf_mu(mlen), CRHBYTES + PM::W1PACKED_BYTES};
    Sp sp;
    sp.hash(src, CRHBYTES + PM::W1PACKED_BYTES, on);
    bool eq = true;
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const uint2 v = ld_lane(row + LY::VF_SIG + 8 * w);
        if constexpr (PAIR)
            eq &= sp.dlo[w] == (sp.half() ? v.y : v.x);
        else
            eq &= (v.x == sp.dlo[w]) && (v.y == sp.dhi[w]);
    }
    if constexpr (PAIR) eq = __shfl_xor_sync(0xFFFFFFFFu, eq, 1) && eq;
    if (!on) return;
    const int status = reinterpret_cast<const int *>(aux + 64)[0];
    reinterpret_cast<int *>(aux + 68)[0] = (eq && status == 0) ? 0 : -1;
}

}  // namespace cudil
