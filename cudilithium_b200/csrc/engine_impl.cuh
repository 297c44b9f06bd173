// Host side of the fused engine: device buffers sized once at creation, per-key caches, and the kernels
// of a whole signing or verification batch, enqueued without waiting for any of them:
//   sign    rounds of the staged signer (fused_sign_staged.cuh) after k_fused_prehash, then k_fused_sign
//           for what they left; or k_fused_init, k_fused_prehash and one persistent signer
//   verify  k_fv_challenge, k_fv_w, k_fv_final (fused_verify.cuh)
// The batch's metadata -- queue block, message offsets and lengths, key indices, longest-first order -- go
// up in one copy.  Buffers are kernel arguments, so a call with new buffers costs what a repeated one does.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>

#include <cuda_runtime.h>

#include "fused_kernels.cuh"
#include "fused_sign_async.cuh"
#include "fused_sign_staged.cuh"
#include "fused_verify.cuh"
#include "host_impl.cuh"
#include "length_order.cuh"
#include "profiling.cuh"

namespace cudil {

struct EngineBase {
    int mode = 0, threads = 0, device = 0, sm_count = 0;
    size_t max_keys = 0, max_items = 0;
    size_t n_sk = 0, n_pk = 0;
    uint8_t *sk_cache = nullptr, *pk_cache = nullptr;
    size_t sk_pitch = 0, pk_pitch = 0;
    uint8_t *items = nullptr;       // max_items * 128
    unsigned *best = nullptr, *locks = nullptr, *next_nonce = nullptr, *inflight = nullptr;
    unsigned spec_slots = 0;  // signer's target of attempts in flight (0 = default for the grid)
    // bounds of the signer's device-side loops (FusedSignArgs)
    unsigned nonce_limit = kNonceLimit, lock_spins = kLockSpinLimit, idle_polls = kAsyncIdleLimit;
    size_t last_n = 0;  // items of the last signing batch
    // a batch's metadata (device, the queue block first) and its pinned staging:
    // [FusedQueue | off | key | mlen | order], each array as long as the batch
    uint8_t *d_meta = nullptr, *h_stage = nullptr;
    unsigned *h_order = nullptr;    // second array of the ordering by length
    FusedQueue *q = nullptr;  // = d_meta
    FusedQueue *h_status = nullptr; // D2H copy of the queue after a batch
    cudaEvent_t stage_ev = nullptr; // recorded after a batch's metadata upload from h_stage
    // key-cache builds run their independent kernels on a side stream too (fork / join events)
    cudaStream_t side = nullptr;
    cudaEvent_t fork_ev = nullptr, join_ev = nullptr;
    bool stage_pending = false;
    uint8_t *scratch = nullptr;
    size_t scratch_bytes = 0;
    int sign_grid = 0, verify_grid = 0, reject_grid = 0;
    size_t sign_smem = 0;
    // signer kernel: 0 = staged rounds, finished by the phased k_fused_sign (block-wide Keccak / NTT
    // phases, the engine's block size) on what they leave; 1..4 = asynchronous k_fused_sign_async with (threads, slots) per block of
    // (256, 64), (512, 128), (640, 160), (768, 192); 5 = phased with one wide block per SM (512
    // threads, 384 for Dilithium5, whose wider phase buffers allow no more)
    int sign_kernel = 0;
    static constexpr int kAsyncVariants = 4;  // (threads, slots) = (256, 64), (512, 128), (640, 160), (768, 192)
    static constexpr int kWideVariant = kAsyncVariants + 1;
    int async_grid[kAsyncVariants] = {0, 0, 0, 0};
    size_t async_smem[kAsyncVariants] = {0, 0, 0, 0};
    int wide_grid = 0;
    size_t wide_smem = 0;
    // Batches of at least large_min_items items (0 = never) sign with large_kernel / large_spec; smaller
    // ones with sign_kernel / spec_slots.
    size_t large_min_items = 0;
    int large_kernel = 0;
    unsigned large_spec = 0;
    size_t device_bytes = 0;
    bool owns_cache = true;  // false when the key caches belong to another engine (attach_keys)
    const EngineBase *key_src = nullptr;  // that engine: its key rows are read as they stand at each call
    virtual ~EngineBase() = default;
};

template <int MODE>
struct EngineImpl : EngineBase {
    using PM = P<MODE>;
    using C = Cache<MODE>;

    static constexpr int L = PM::L;
    // the queue block, padded for the arrays behind it
    static constexpr size_t kStageHead = (sizeof(FusedQueue) + 63) / 64 * 64;
    static size_t stage_bytes(size_t max_items) {
        return kStageHead + max_items * (3 * sizeof(unsigned) + sizeof(unsigned long long));
    }

    template <int T>
    static int grid_for(const void *fn, size_t smem, int sm_count) {
        int per_sm = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, T, smem) != cudaSuccess || per_sm < 1) return 0;
        return per_sm * sm_count;
    }

    // Device bytes the engine needs (the admission budget checks this before allocating).
    size_t required_bytes(size_t max_keys, size_t max_items) const {
        return max_keys * (align256(C::SK_ROW) + align256(C::PK_ROW)) + max_items * (C::ITEM_BYTES + 4 * sizeof(unsigned)) +
               stage_bytes(max_items) + scratch_for(max_items);
    }
    // attempt slots of the largest signer variant, or the packed w1' of a verification turn
    size_t scratch_for(size_t max_items) const {
        if (max_items == 0) return 0;
        size_t b = std::max((size_t)sign_grid * 2 * threads * C::SLOT, std::min(max_items, kVerifyTurn) * VerifyRow<MODE>::W1);
        static constexpr int slots[kAsyncVariants] = {64, 128, 160, 192};
        for (int v = 0; v < kAsyncVariants; ++v) b = std::max(b, (size_t)async_grid[v] * slots[v] * C::SLOT);
        b = std::max(b, (size_t)wide_grid * 2 * kWideThreads * C::SLOT);
        return b;
    }

    static constexpr int kWideThreads = (MODE == 5) ? 384 : 512;

    int configure_wide() {
        wide_smem = FusedSignSmem<MODE, kWideThreads>::BYTES;
        if (cudaFuncSetAttribute(k_fused_sign<MODE, kWideThreads>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)wide_smem) != cudaSuccess)
            return ::cudil::cudil_record_cuda_error(cudaGetLastError(), __FILE__, __LINE__);
        wide_grid = grid_for<kWideThreads>((const void *)k_fused_sign<MODE, kWideThreads>, wide_smem, sm_count);
        return wide_grid > 0 ? CUDIL_OK : cudil_record_cuda_error(cudaErrorInvalidConfiguration, __FILE__, __LINE__);
    }

    template <int T, int S>
    int configure_async_one(int v) {
        async_smem[v] = AsyncSignSmem<MODE, T, S>::BYTES;
        if (cudaFuncSetAttribute(k_fused_sign_async<MODE, T, S>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)async_smem[v]) != cudaSuccess)
            return ::cudil::cudil_record_cuda_error(cudaGetLastError(), __FILE__, __LINE__);
        async_grid[v] = grid_for<T>((const void *)k_fused_sign_async<MODE, T, S>, async_smem[v], sm_count);
        return async_grid[v] > 0 ? CUDIL_OK : cudil_record_cuda_error(cudaErrorInvalidConfiguration, __FILE__, __LINE__);
    }

    int configure_async() {
        int rc = configure_async_one<256, 64>(0);
        if (!rc) rc = configure_async_one<512, 128>(1);
        if (!rc) rc = configure_async_one<640, 160>(2);
        if (!rc) rc = configure_async_one<768, 192>(3);
        return rc;
    }

    // The kernels of a key-cache build run side by side, on one SM too, so they ask for the same split of its
    // memory between L1 and shared memory.  An SM changes the split only while it is idle: with the driver's
    // choice, which follows each kernel's own shared memory, ExpandA and the transforms waited for one another:
    // secret rows of 1024 Dilithium2 keys 151 us, 75 us with one split; public rows of 2048 keys 182 and 96 us.
    // Three quarters of the memory hold the 24 ExpandA warps that the registers allow; with all of it
    // verification of 10 000 signatures with fresh keys takes 451 instead of 447 us.
    static constexpr int kCacheSplit = 75;  // percent
    int configure_caches() {
        const void *fns[] = {(const void *)k_cache_sk<MODE>, (const void *)k_expand_a_keys<MODE>, (const void *)k_cache_pk_t1<MODE>,
                             (const void *)k_cache_pk_tr<MODE, false>, (const void *)k_cache_pk_tr<MODE, true>};
        for (const void *fn : fns)
            CUDIL_CK(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, kCacheSplit));
        return CUDIL_OK;
    }

    template <int T>
    int configure() {
        sign_smem = FusedSignSmem<MODE, T>::BYTES;
        if (cudaFuncSetAttribute(k_fused_sign<MODE, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sign_smem) != cudaSuccess)
            return ::cudil::cudil_record_cuda_error(cudaGetLastError(), __FILE__, __LINE__);
        sign_grid = grid_for<T>((const void *)k_fused_sign<MODE, T>, sign_smem, sm_count);
        reject_grid = grid_for<32>((const void *)k_st_reject<MODE>, 0, sm_count);
        verify_grid = grid_for<kBlock>((const void *)k_fv_w<MODE>, 4 * VerifyRow<MODE>::WARP, sm_count);
        return (sign_grid > 0 && verify_grid > 0 && reject_grid > 0) ? CUDIL_OK : cudil_record_cuda_error(cudaErrorInvalidConfiguration, __FILE__, __LINE__);
    }

    int create(size_t mk, size_t mi, int thr, size_t budget) {
        mode = MODE;
        max_keys = mk;
        max_items = mi;
        threads = thr;
        // mk == 0: caches attached later; mi == 0: a cache-only engine other engines attach to
        if ((mi == 0 && mk == 0) || mi > (1u << 24)) return CUDIL_ERR_INVALID;
        CUDIL_CK(cudaGetDevice(&device));
        CUDIL_CK(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, device));
        int rc = (threads == 128) ? configure<128>() : (threads == 256 ? configure<256>() : CUDIL_ERR_INVALID);
        if (rc) return rc;
        rc = configure_async();
        if (rc) return rc;
        rc = configure_wide();
        if (rc) return rc;
        rc = configure_caches();
        if (rc) return rc;
        device_bytes = required_bytes(mk, mi);
        if (budget && device_bytes > budget) return CUDIL_ERR_BUDGET;
        sk_pitch = align256(C::SK_ROW);
        pk_pitch = align256(C::PK_ROW);
        scratch_bytes = scratch_for(mi);
        spec_slots = (unsigned)threads;
        if ((mk && (cudaMalloc(&sk_cache, mk * sk_pitch) != cudaSuccess || cudaMalloc(&pk_cache, mk * pk_pitch) != cudaSuccess)) ||
            (mi && (cudaMalloc(&items, mi * C::ITEM_BYTES) != cudaSuccess || cudaMalloc(&best, mi * sizeof(unsigned)) != cudaSuccess ||
                    cudaMalloc(&locks, mi * sizeof(unsigned)) != cudaSuccess ||
                    cudaMalloc(&next_nonce, mi * sizeof(unsigned)) != cudaSuccess ||
                    cudaMalloc(&inflight, mi * sizeof(unsigned)) != cudaSuccess ||
                    cudaMalloc(&scratch, scratch_bytes) != cudaSuccess)) ||
            cudaMalloc(&d_meta, stage_bytes(mi)) != cudaSuccess || cudaMallocHost(&h_stage, stage_bytes(mi)) != cudaSuccess ||
            cudaMallocHost(&h_status, sizeof(FusedQueue)) != cudaSuccess)
            return ::cudil::cudil_record_cuda_error(cudaGetLastError(), __FILE__, __LINE__);
        if (mi && !(h_order = new (std::nothrow) unsigned[mi])) return CUDIL_ERR_INVALID;
        std::memset(h_status, 0, sizeof(FusedQueue));
        CUDIL_CK(cudaEventCreateWithFlags(&stage_ev, cudaEventDisableTiming));
        CUDIL_CK(cudaEventCreateWithFlags(&fork_ev, cudaEventDisableTiming));
        CUDIL_CK(cudaEventCreateWithFlags(&join_ev, cudaEventDisableTiming));
        CUDIL_CK(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
        q = reinterpret_cast<FusedQueue *>(d_meta);
        CUDIL_CK(cudaMemset(q, 0, sizeof(FusedQueue)));
        return CUDIL_OK;
    }

    ~EngineImpl() override {
        if (owns_cache) {
            cudaFree(sk_cache);
            cudaFree(pk_cache);
        }
        cudaFree(items);
        cudaFree(best);
        cudaFree(locks);
        cudaFree(next_nonce);
        cudaFree(inflight);
        cudaFree(d_meta);
        cudaFree(scratch);
        delete[] h_order;
        if (h_stage) cudaFreeHost(h_stage);
        if (h_status) cudaFreeHost(h_status);
        if (stage_ev) cudaEventDestroy(stage_ev);
        if (fork_ev) cudaEventDestroy(fork_ev);
        if (join_ev) cudaEventDestroy(join_ev);
        if (side) cudaStreamDestroy(side);
    }

    // ------------------------------------------------------------ key caches
    // Use another engine's key caches (same parameter set); its caches must outlive this engine.
    int attach_keys(const EngineBase *src) {
        if (!src || src->mode != MODE || src == this) return CUDIL_ERR_INVALID;
        if (owns_cache) {
            cudaFree(sk_cache);
            cudaFree(pk_cache);
        }
        owns_cache = false;
        key_src = src->key_src ? src->key_src : src;  // the engine that owns the caches
        sk_cache = src->sk_cache;
        pk_cache = src->pk_cache;
        n_sk = src->n_sk;
        n_pk = src->n_pk;
        max_keys = src->max_keys;
        return CUDIL_OK;
    }

    int set_secret_keys(const uint8_t *d_sk, size_t nkeys, cudaStream_t st) {
        if (!d_sk || nkeys == 0 || nkeys > max_keys || !owns_cache) return CUDIL_ERR_INVALID;
        const int rc = build_sk_rows(d_sk, 0, nkeys, st);
        if (rc == CUDIL_OK) n_sk = nkeys;
        return rc;
    }

    // Cache rows [first, first + nkeys); first <= the number of rows built so far, so the built rows
    // stay one contiguous prefix.
    int update_secret_keys(const uint8_t *d_sk, size_t first, size_t nkeys, cudaStream_t st) {
        if (!d_sk || nkeys == 0 || first > n_sk || first > max_keys || nkeys > max_keys - first || !owns_cache)
            return CUDIL_ERR_INVALID;
        const int rc = build_sk_rows(d_sk, first, nkeys, st);
        if (rc == CUDIL_OK) n_sk = std::max(n_sk, first + nkeys);
        return rc;
    }

    // The unpack / transform of s1, s2, t0 and ExpandA (rho read from the packed keys) are independent: the
    // transforms go to the side stream, beside ExpandA, and the caller's stream waits for both.  Between 4 and 48
    // of the transforms' blocks per SM the two follow one another instead.  Side by side ExpandA's few warps
    // then start behind the transforms, and unevenly: 1024 Dilithium2 keys 75 us, one after the other 54, 4096
    // keys 166 and 144.  Below that the transforms leave the SMs free (repeated builds of 100 keys 37 against
    // 41 us), above it ExpandA is long enough to even out (6000 keys 199 against 205).
    int build_sk_rows(const uint8_t *d_sk, size_t first, size_t nkeys, cudaStream_t st) {
        const int nn = (int)nkeys;
        uint8_t *rows = sk_cache + first * sk_pitch;
        const unsigned blocks = blocks_for(nkeys * (PM::L + 2 * PM::K + 1) * 16);
        const bool beside = blocks <= 4u * (unsigned)sm_count || blocks > 48u * (unsigned)sm_count;
        cudaStream_t ts = beside ? side : st;
        if (beside) {
            CUDIL_CK(cudaEventRecord(fork_ev, st));
            CUDIL_CK(cudaStreamWaitEvent(side, fork_ev, 0));
        }
        CUDIL_LAUNCH(KID_CACHE_SK, ts, k_cache_sk<MODE><<<blocks, kBlock, 0, ts>>>(d_sk, rows, sk_pitch, nn));
        CUDIL_CK_LAUNCH();
        CUDIL_LAUNCH(KID_EXPAND_A, st,
                     k_expand_a_keys<MODE><<<blocks_for(nkeys * PM::K * PM::L, kItemBlock), kItemBlock, 0, st>>>(d_sk, PM::SK_BYTES, rows, sk_pitch,
                                                                                             C::SK_MAT, nn));
        CUDIL_CK_LAUNCH();
        if (beside) {
            CUDIL_CK(cudaEventRecord(join_ev, side));
            CUDIL_CK(cudaStreamWaitEvent(st, join_ev, 0));
        }
        return CUDIL_OK;
    }

    int set_public_keys(const uint8_t *d_pk, size_t nkeys, cudaStream_t st) {
        if (!d_pk || nkeys == 0 || nkeys > max_keys || !owns_cache) return CUDIL_ERR_INVALID;
        const int nn = (int)nkeys;
        // tr = H(pk) and t1_hat (side stream) run concurrently with ExpandA (rho from the packed keys)
        CUDIL_CK(cudaEventRecord(fork_ev, st));
        CUDIL_CK(cudaStreamWaitEvent(side, fork_ev, 0));
        CUDIL_LAUNCH(KID_CACHE_PK, side, CUDIL_PAIRED_ON(nkeys, sm_count, k_cache_pk_tr<MODE, PAIR><<<blocks_for(nkeys * LANES, kItemBlock), kItemBlock, 0, side>>>(d_pk, pk_cache, pk_pitch, nn)));
        CUDIL_CK_LAUNCH();
        CUDIL_LAUNCH(KID_CACHE_PK, side,
                     k_cache_pk_t1<MODE><<<blocks_for(nkeys * PM::K * 16), kBlock, 0, side>>>(d_pk, pk_cache, pk_pitch, nn));
        CUDIL_CK_LAUNCH();
        CUDIL_LAUNCH(KID_EXPAND_A, st,
                     k_expand_a_keys<MODE><<<blocks_for(nkeys * PM::K * PM::L, kItemBlock), kItemBlock, 0, st>>>(d_pk, PM::PK_BYTES, pk_cache, pk_pitch,
                                                                                             C::PK_MAT, nn));
        CUDIL_CK_LAUNCH();
        CUDIL_CK(cudaEventRecord(join_ev, side));
        CUDIL_CK(cudaStreamWaitEvent(st, join_ev, 0));
        n_pk = nkeys;
        return CUDIL_OK;
    }

    // A batch's metadata goes up from the engine's staging buffer, which the next call rewrites: a batch in a
    // captured graph would read some later call's lengths and key indices at its replay.
    static int refuse_capture(cudaStream_t st) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        CUDIL_CK(cudaStreamIsCapturing(st, &cs));
        return cs == cudaStreamCaptureStatusNone ? CUDIL_OK : CUDIL_ERR_INVALID;
    }

    // ------------------------------------------------------------ metadata upload
    // Checks the batch's metadata and queues its upload; m gets the device arrays (and the caller's
    // buffers).  An order that is the identity -- every batch of equal lengths -- does not travel.
    int upload_meta(MsgRefs &m, const unsigned long long *off, const unsigned *mlen, const unsigned *key, size_t n, size_t nkeys,
                    size_t msgs_bytes, cudaStream_t st, const uint8_t *rho_seed = nullptr, unsigned long long rho_counter = 0) {
        // the previous batch's copy out of the staging buffer must have completed (only that: work the
        // caller queued on the stream, such as input copies or cache builds, keeps running while this
        // batch is prepared)
        if (stage_pending) CUDIL_CK(cudaEventSynchronize(stage_ev));
        FusedQueue *hq = reinterpret_cast<FusedQueue *>(h_stage);
        std::memset(h_stage, 0, kStageHead);
        hq->n = (unsigned)n;
        if (rho_seed) {
            hq->rho_seeded = 1u;
            hq->rho_counter = rho_counter;
            std::memcpy(hq->rho_seed, rho_seed, sizeof hq->rho_seed);
        }
        unsigned long long *hoff = reinterpret_cast<unsigned long long *>(h_stage + kStageHead);
        unsigned *hk = reinterpret_cast<unsigned *>(hoff + n), *hm = hk + n, *ho = hm + n;
        bool descending = true;  // already longest first (every batch of equal lengths is)
        for (size_t i = 0; i < n; ++i) {
            if (key[i] >= nkeys || (off[i] & 7u) || off[i] > msgs_bytes || mlen[i] > msgs_bytes - off[i])
                return CUDIL_ERR_INVALID;
            hk[i] = key[i];
            hm[i] = mlen[i];
            hoff[i] = off[i];
            if (i && mlen[i] > mlen[i - 1]) descending = false;
        }
        size_t bytes = kStageHead + n * (sizeof(unsigned long long) + 2 * sizeof(unsigned));
        if (!descending) {
            order_longest_first(ho, h_order, hm, n);
            bytes += n * sizeof(unsigned);
        }
        CUDIL_CK(cudaMemcpyAsync(d_meta, h_stage, bytes, cudaMemcpyHostToDevice, st));
        CUDIL_CK(cudaEventRecord(stage_ev, st));
        stage_pending = true;
        m.offsets = reinterpret_cast<const unsigned long long *>(d_meta + kStageHead);
        m.key_idx = reinterpret_cast<const unsigned *>(m.offsets + n);
        m.mlens = m.key_idx + n;
        m.order = descending ? nullptr : m.mlens + n;
        m.nkeys = (unsigned)max_keys;
        return CUDIL_OK;
    }

    // ------------------------------------------------------------ signers
    // one of the persistent signers, on what is pending in best[] (after k_fused_init: everything)
    void launch_persistent(const FusedSignArgs &a, int variant, cudaStream_t st) {
        if (variant == 1)
            k_fused_sign_async<MODE, 256, 64><<<async_grid[0], 256, async_smem[0], st>>>(a);
        else if (variant == 2)
            k_fused_sign_async<MODE, 512, 128><<<async_grid[1], 512, async_smem[1], st>>>(a);
        else if (variant == 3)
            k_fused_sign_async<MODE, 640, 160><<<async_grid[2], 640, async_smem[2], st>>>(a);
        else if (variant == 4)
            k_fused_sign_async<MODE, 768, 192><<<async_grid[3], 768, async_smem[3], st>>>(a);
        else if (variant == kWideVariant)
            k_fused_sign<MODE, kWideThreads><<<wide_grid, kWideThreads, wide_smem, st>>>(a);
        else if (threads == 128)
            k_fused_sign<MODE, 128><<<sign_grid, 128, sign_smem, st>>>(a);
        else
            k_fused_sign<MODE, 256><<<sign_grid, 256, sign_smem, st>>>(a);
    }

    // Where the staged signer's attempt slots start in the scratch: behind two lists of pending items and the
    // round counters of both parts.
    size_t staged_lists() const { return 2 * align256(max_items * sizeof(unsigned)) + align256(2 * kStagedRoundBytes); }
    // Attempt slots the scratch holds behind them.
    size_t staged_cap() const {
        const size_t lists = staged_lists();
        if (scratch_bytes <= lists) return 0;
        return (scratch_bytes - lists) / (StagedSlot<MODE>::SIZE + 2 * sizeof(StagedAttempt));
    }

    // Acceptance probability of an attempt, a little below the parameter set's average since it varies by
    // key (used only to size the enqueued rounds).
    static constexpr double kAccept = MODE == 2 ? 0.21 : (MODE == 3 ? 0.175 : 0.23);

    // The rounds of one part of the batch (0 or 1) on its stream.
    struct StagedPart {
        StagedArgs a;
        cudaStream_t st;
        double p;             // expected pending items
        unsigned prev_slots;  // attempts the previous round's kernels were launched for
        int r;
        bool done() const { return r >= kStagedMaxRounds || p <= 0.01; }
    };

    // Kernels of stage 0..3 (claim and ExpandMask, w, challenge, rejection) of the part's current round.
    void staged_stage(StagedPart &t, int stage) {
        using S = StagedSlot<MODE>;
        const unsigned sms = (unsigned)sm_count;
        StagedArgs &a = t.a;
        cudaStream_t st = t.st;
        // enough blocks for a pending count four standard deviations above the expected one (kernels
        // stride over what exceeds it)
        const double hi = std::min((double)a.count, t.p + 4.0 * std::sqrt(t.p) + 4.0);
        // (attempts at most: whole quanta where the claim rounds down to them)
        const double most = hi > a.quantum && hi < 4.0 * a.quantum ? std::floor(hi / a.quantum) * a.quantum : hi;
        const unsigned slots = (unsigned)std::min((double)a.cap, std::max(most, std::min((double)a.target, hi * kStagedMaxDepth)));
        if (stage == 0) {
            const unsigned cb = std::max(blocks_for((size_t)hi + 1, 256), std::min(blocks_for(t.prev_slots, 8), 8u * sms));
            CUDIL_LAUNCH(KID_ST_CLAIM, st, k_st_claim<MODE><<<cb, 256, 0, st>>>(a, t.r, true));
            const unsigned mb = (size_t)slots * L <= (size_t)sms * 128 ? 32u : (unsigned)kBlock;
            CUDIL_LAUNCH(KID_ST_MASK, st, CUDIL_PAIRED_ON((size_t)slots * L, sm_count, k_st_mask<MODE, PAIR><<<blocks_for((size_t)slots * L * LANES, mb), mb, 0, st>>>(a, t.r)));
        } else if (stage == 1) {
            const unsigned wb = slots <= 8u * sms ? 1u : 4u;  // warps per block
            CUDIL_LAUNCH(KID_ST_W, st, k_st_w<MODE><<<blocks_for(slots, wb), 32 * wb, wb * S::WARP_W, st>>>(a, t.r));
        } else if (stage == 2) {
            CUDIL_LAUNCH(KID_ST_CHALLENGE, st,
                         CUDIL_PAIRED_ON(slots, sm_count, k_st_challenge<MODE, PAIR><<<blocks_for((size_t)slots * LANES, kItemBlock), kItemBlock, 0, st>>>(a, t.r)));
        } else {
            const unsigned per = slots <= (unsigned)reject_grid ? 1u : 2u;  // attempts per warp
            CUDIL_LAUNCH(KID_ST_REJECT, st, k_st_reject<MODE><<<blocks_for(slots, per), 32, 0, st>>>(a, t.r, per));
            t.prev_slots = slots;
            if (t.p >= a.target)
                t.p -= kAccept * (t.p > a.quantum && t.p < 4.0 * a.quantum ? std::floor(t.p / a.quantum) * a.quantum : std::min(t.p, (double)a.cap));
            else
                t.p *= std::pow(1.0 - kAccept, std::min((double)kStagedMaxDepth, a.target / std::max(t.p, 1.0)));
            ++t.r;
        }
    }

    void staged_finish(StagedPart &t) {
        const unsigned cb = std::max(1u, std::min(blocks_for(t.prev_slots, 8), 8u * (unsigned)sm_count));
        CUDIL_LAUNCH(KID_ST_CLAIM, t.st, k_st_claim<MODE><<<cb, 256, 0, t.st>>>(t.a, t.r, false));
    }

    // Items of the batch's first part (longest messages first), 0 = the batch stays whole.
    //
    // A batch of mixed lengths waits for its longest message: its blocks are one thread pair's chain (3.5 us
    // each), and nothing is signed before.  In two parts the shorter messages are signed on a second stream
    // while the longest are still being hashed.  The split is the eighth of the batch that ends soonest by
    // this model: hashing as above, signing 0.3 ms (rounds' latency) and kSignUs per item.
    // 16 384 Dilithium3 messages of 32 B..64 KiB: 5.78 ms whole, 4.50 ms in two parts.  A batch without an
    // order array stays whole.  That is every batch of equal lengths -- two halves on two streams gained 5%
    // alone and lost 4% where batches already run on two engines' streams -- and also a mixed one that arrives
    // longest first, which the two parts would serve too.
    size_t staged_split(const MsgRefs &mr, const unsigned *mlen, size_t n) const {
        if (!mr.order) return 0;
        constexpr double kSignUs = MODE == 2 ? 0.10 : (MODE == 3 ? 0.18 : 0.25), kRoundsUs = 300.0, kBlockUs = 3.5;
        const unsigned *ho = reinterpret_cast<const unsigned *>(h_stage + ((const uint8_t *)mr.order - d_meta));
        auto hash = [&](size_t r) { return kBlockUs * ((double)mlen[ho[r]] / SHAKE256_RATE + 2.0); };
        const double whole = hash(0) + kRoundsUs + (double)n * kSignUs;
        double best = 0.95 * whole;
        size_t split = 0;
        for (size_t e = 1; e <= 4; ++e) {
            const size_t k = n * e / 8;
            if (k == 0) continue;
            const double t = std::max(hash(0), hash(k) + kRoundsUs + (double)(n - k) * kSignUs) + kRoundsUs + (double)k * kSignUs;
            if (t < best) {
                best = t;
                split = k;
            }
        }
        return split;
    }

    int sign_staged(const MsgRefs &mr, uint8_t *out, size_t n, size_t split, unsigned target, cudaStream_t st) {
        using S = StagedSlot<MODE>;
        const int parts = split ? 2 : 1;
        const size_t cap = std::min<size_t>(staged_cap(), 0x7FFFFFFFu) / parts;
        unsigned *pend = reinterpret_cast<unsigned *>(scratch);
        StagedRound *rounds = reinterpret_cast<StagedRound *>(scratch + 2 * align256(max_items * sizeof(unsigned)));
        uint8_t *slots = scratch + staged_lists();
        StagedAttempt *att = reinterpret_cast<StagedAttempt *>(slots + cap * parts * S::SIZE);
        unsigned first = 0;
        StagedPart part[2];
        for (int k = 0; k < parts; ++k) {
            StagedArgs &a = part[k].a;
            a = StagedArgs{};
            a.cache = sk_cache;
            a.cpitch = sk_pitch;
            a.key_idx = mr.key_idx;
            a.items = items;
            a.sig_out = out;
            a.sig_pitch = (size_t)PM::SIG_BYTES;
            a.first = first;
            a.count = k == 0 && split ? (unsigned)split : (unsigned)n - first;
            a.order = mr.order;
            a.n = (unsigned)n;
            a.cap = (unsigned)cap;
            a.slots = slots + k * cap * S::SIZE;
            a.att[0] = att + 2 * k * cap;
            a.att[1] = a.att[0] + cap;
            a.pend[0] = pend + first;
            a.pend[1] = reinterpret_cast<unsigned *>(scratch + align256(max_items * sizeof(unsigned))) + first;
            a.rounds = rounds + k * kStagedMaxRounds;
            a.q = q;
            a.best = best;
            a.locks = locks;
            a.next_nonce = next_nonce;
            a.inflight = inflight;
            // two layers of 32 streams on every sub-partition
            a.quantum = (unsigned)(sm_count * 4 * 32 * 2 / L);
            a.target = (unsigned)std::min<size_t>(std::max(1u, target / parts), cap);
            if (a.target > a.quantum) a.target = a.target / a.quantum * a.quantum;
            a.nonce_limit = nonce_limit;
            a.nkeys = (unsigned)max_keys;
            part[k].st = k ? side : st;
            part[k].p = (double)a.count;
            part[k].prev_slots = 0;
            part[k].r = 0;
            first += a.count;
        }
        if (parts == 2) {
            CUDIL_CK(cudaEventRecord(fork_ev, st));
            CUDIL_CK(cudaStreamWaitEvent(side, fork_ev, 0));
        }
        for (int k = 0; k < parts; ++k) {
            const StagedArgs &a = part[k].a;
            CUDIL_LAUNCH(KID_ST_PREHASH, part[k].st,
                         CUDIL_PAIRED_ON(a.count, sm_count, k_fused_prehash<MODE, PAIR><<<prehash_blocks(a.count * LANES), kPrehashBlock, 0, part[k].st>>>(sk_cache, sk_pitch, mr, items, q, a.first, a.count, reinterpret_cast<uint4 *>(a.rounds), (unsigned)(kStagedRoundBytes / sizeof(uint4)))));
        }
        for (bool more = true; more;) {
            more = false;
            for (int k = 0; k < parts; ++k) {
                if (part[k].done()) continue;
                for (int stage = 0; stage < 4; ++stage) staged_stage(part[k], stage);
                more = true;
            }
        }
        for (int k = 0; k < parts; ++k) staged_finish(part[k]);
        if (parts == 2) {
            CUDIL_CK(cudaEventRecord(join_ev, side));
            CUDIL_CK(cudaStreamWaitEvent(st, join_ev, 0));
        }
        CUDIL_CK_LAUNCH();
        return CUDIL_OK;
    }

    unsigned prehash_blocks(size_t n) const { return (unsigned)std::min<size_t>(blocks_for(n, kPrehashBlock), (size_t)sm_count * 32); }

    // d_rhop: randomized signing seeds, 64 bytes per item (dense, device); nullptr = deterministic
    // rho_seed (host, 32 bytes): seeded randomized signing, rho' of item i derived on the device from
    // (rho_seed, rho_counter + i); it goes up with the batch metadata
    int sign(uint8_t *d_sig, const uint8_t *d_msgs, size_t msgs_bytes, const unsigned long long *off, const unsigned *mlen,
             const unsigned *key, size_t n, cudaStream_t st, const uint8_t *d_rhop = nullptr,
             const uint8_t *rho_seed = nullptr, unsigned long long rho_counter = 0) {
        if (n == 0) return CUDIL_OK;
        if (key_src) n_sk = key_src->n_sk;  // rows the owning engine has built by now
        if (!d_sig || !off || !mlen || !key || n > max_items || n_sk == 0) return CUDIL_ERR_INVALID;
        if (!d_msgs) {
            for (size_t i = 0; i < n; ++i)
                if (mlen[i]) return CUDIL_ERR_INVALID;
            d_msgs = reinterpret_cast<const uint8_t *>(items);  // any aligned pointer; never read
        }
        if (((uintptr_t)d_msgs) & 7u) return CUDIL_ERR_INVALID;
        // The signature rows may be device memory or pinned host memory (written by the signer over
        // PCIe); pageable host memory is refused before anything is queued.
        uint8_t *out = d_sig;
        cudaPointerAttributes pa{};
        if (cudaPointerGetAttributes(&pa, d_sig) != cudaSuccess) {
            cudaGetLastError();
            return CUDIL_ERR_INVALID;
        }
        if (pa.type == cudaMemoryTypeUnregistered) return CUDIL_ERR_INVALID;
        if (pa.type == cudaMemoryTypeHost) {
            if (!pa.devicePointer) return CUDIL_ERR_INVALID;
            out = static_cast<uint8_t *>(pa.devicePointer);
        }
        MsgRefs mr{};
        int rc = refuse_capture(st);
        if (!rc) rc = upload_meta(mr, off, mlen, key, n, n_sk, msgs_bytes, st, rho_seed, rho_counter);
        if (rc) return rc;
        mr.msgs = d_msgs;
        mr.rhoprime = d_rhop;
        const bool large = large_min_items && n >= large_min_items;
        int variant = large ? large_kernel : sign_kernel;
        unsigned spec = large ? large_spec : spec_slots;
        // variant 0: staged rounds, then the phased kernel on what they left.  A caller that shortened the
        // publication lock's bound gets the kernel that has that lock; more items than attempt slots go
        // to the wide phased kernel.
        const bool staged = variant == 0 && lock_spins == kLockSpinLimit && n <= staged_cap();
        if (variant == 0 && lock_spins == kLockSpinLimit && !staged) {
            variant = kWideVariant;
            spec = std::min<unsigned>(128u, 2u * (unsigned)threads);
        }
        FusedSignArgs a{sk_cache, sk_pitch, mr.key_idx, items, out, (size_t)PM::SIG_BYTES, scratch, q, best, locks, next_nonce,
                        inflight, spec, nonce_limit, lock_spins, idle_polls, (unsigned)max_keys};
        cudaEvent_t ev = Profiler::get().before(st);
        if (staged) {
            // the target is a count per block of a four-blocks-per-SM grid, as tuned for the phased kernel
            rc = sign_staged(mr, out, n, staged_split(mr, mlen, n), spec * 4u * (unsigned)sm_count, st);
            if (rc) return rc;
        } else {
            k_fused_init<<<std::max(1, sm_count * 2), 256, 0, st>>>(q, best, locks, next_nonce, inflight);
            CUDIL_LAUNCH(KID_ST_PREHASH, st, CUDIL_PAIRED_ON(n, sm_count, k_fused_prehash<MODE, PAIR><<<prehash_blocks(n * LANES), kPrehashBlock, 0, st>>>(sk_cache, sk_pitch, mr, items, q, 0u, (unsigned)n, nullptr, 0u)));
        }
        launch_persistent(a, variant, st);
        CUDIL_CK_LAUNCH();
        Profiler::get().after(KID_FUSED_SIGN, ev, st);
        CUDIL_CK(cudaMemcpyAsync(h_status, q, sizeof(FusedQueue), cudaMemcpyDeviceToHost, st));
        last_n = n;
        return CUDIL_OK;
    }

    // Winning nonce per item of the last signing batch (kNonceExhausted: no accepted nonce below the
    // limit), copied into out (host or device memory) on st; returns after the copy completed.
    int last_nonces(unsigned *out, size_t n, cudaStream_t st) {
        if (!out || n > last_n || !best) return CUDIL_ERR_INVALID;
        if (n == 0) return CUDIL_OK;
        CUDIL_CK(cudaMemcpyAsync(out, best, n * sizeof(unsigned), cudaMemcpyDefault, st));
        CUDIL_CK(cudaStreamSynchronize(st));
        return CUDIL_OK;
    }

    // Bounds of the signer's loops, from the next batch on.
    int set_limits(unsigned nonces, unsigned spins, unsigned polls) {
        if (nonces == 0 || nonces > kNonceLimit) return CUDIL_ERR_INVALID;
        nonce_limit = nonces;
        lock_spins = spins;
        idle_polls = polls;
        return CUDIL_OK;
    }

    int verify(int *d_ret, const uint8_t *d_sig, const uint8_t *d_msgs, size_t msgs_bytes, const unsigned long long *off,
               const unsigned *mlen, const unsigned *key, size_t n, cudaStream_t st) {
        if (n == 0) return CUDIL_OK;
        if (key_src) n_pk = key_src->n_pk;
        if (!d_ret || !d_sig || !off || !mlen || !key || n > max_items || n_pk == 0) return CUDIL_ERR_INVALID;
        if (!d_msgs) {
            for (size_t i = 0; i < n; ++i)
                if (mlen[i]) return CUDIL_ERR_INVALID;
            d_msgs = reinterpret_cast<const uint8_t *>(items);
        }
        if (((uintptr_t)d_msgs) & 7u) return CUDIL_ERR_INVALID;
        MsgRefs mr{};
        int rc = refuse_capture(st);
        if (!rc) rc = upload_meta(mr, off, mlen, key, n, n_pk, msgs_bytes, st);
        if (rc) return rc;
        mr.msgs = d_msgs;
        cudaEvent_t ev = Profiler::get().before(st);
        VerifyArgs a{pk_cache, pk_pitch, mr, d_sig, (size_t)PM::SIG_BYTES, items, scratch, locks, d_ret, (unsigned)n, 0u, 0u};  // (best[] keeps the last signing batch's nonces)
        CUDIL_LAUNCH(KID_FV_CHALLENGE, st, CUDIL_PAIRED_ON(n, sm_count, k_fv_challenge<MODE, PAIR><<<prehash_blocks(n * LANES), kPrehashBlock, 0, st>>>(a)));
        for (size_t first = 0; first < n; first += kVerifyTurn) {
            const size_t count = std::min(n - first, kVerifyTurn);
            a.first = (unsigned)first;
            a.count = (unsigned)count;
            const unsigned wb = count <= 8u * (size_t)sm_count ? 1u : 4u;  // warps per block
            CUDIL_LAUNCH(KID_FV_W, st, k_fv_w<MODE><<<blocks_for(count, wb), 32 * wb, wb * VerifyRow<MODE>::WARP, st>>>(a));
            CUDIL_LAUNCH(KID_FV_FINAL, st, CUDIL_PAIRED_ON(count, sm_count, k_fv_final<MODE, PAIR><<<blocks_for(count * LANES, kPrehashBlock), kPrehashBlock, 0, st>>>(a)));
        }
        CUDIL_CK_LAUNCH();
        Profiler::get().after(KID_FUSED_VERIFY, ev, st);
        CUDIL_CK(cudaMemcpyAsync(h_status, q, sizeof(FusedQueue), cudaMemcpyDeviceToHost, st));
        return CUDIL_OK;
    }

    // Signer variant and target of signing attempts in flight, from the next batch on.
    int set_sign_kernel(int v) {
        if (v < 0 || v > kWideVariant) return CUDIL_ERR_INVALID;
        sign_kernel = v;
        return CUDIL_OK;
    }

    int set_spec_slots(unsigned v) {
        spec_slots = v ? std::min<unsigned>(v, 2u * (unsigned)threads) : (unsigned)threads;
        return CUDIL_OK;
    }

    int set_large_batch(size_t min_items, int variant, unsigned spec) {
        if (variant < 0 || variant > kWideVariant) return CUDIL_ERR_INVALID;
        large_min_items = min_items;
        large_kernel = variant;
        large_spec = spec ? std::min<unsigned>(spec, 2u * (unsigned)threads) : (unsigned)threads;
        return CUDIL_OK;
    }
};

}  // namespace cudil
