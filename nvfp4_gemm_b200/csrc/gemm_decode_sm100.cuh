// NVFP4 GEMM for few rows of activations (decode; up to 128, more with K split):  C[M,N] (fp16) = (A x SFA) . (B x SFB)^T.
//
// Operands are swapped on the tensor core: the weights B are the M operand (128 of their rows = output
// columns per CTA), the activations A the N operand, BT = 32, 64 or 128 of them.  D[column, token]
// lands with one output column per TMEM lane.
//
// Why swapped.  These shapes stream the weights once; the kernel is bound by HBM when enough bytes
// are in flight, and what an SM can take in is 65 bytes a cycle (its TMA unit).  As the M
// operand the activations took 16 KB of every 36 KB stage whatever the batch (128-row tile,
// zero-filled beyond M); as the N operand they take 128 bytes a row of a batch rounded up to 32, so
// that the ring holds more stages, and MMAs and epilogue shrink with the batch.  Measured (us, replays of 24
// launches over rotating inputs beyond L2, both kernels in turn in one process; the 128-row-tile kernels -> this one):
// 17 x 7168 x 2048 5.8 -> 4.2, 17 x 7168 x 16384 15.3 -> 12.5 (5.3 TB/s), 1 x 28672 x 4096 20.6 -> 13.0, 40 x 4096 x 7168
// 9.1 -> 6.6, 128 x 7168 x 16384 15.9 -> 14.9 (replays of 200: 16.7 -> 15.2-15.6), 128 x 4096 x 7168 9.3 -> 8.0.  For 65 to 128
// rows without a split the 128-row-tile kernels stay ahead (128 x 28672 x 4096: 14.6 against 17.3).
//
// K is split over the KS ranks of a cluster, so that there are enough CTAs to pull at HBM's rate.
// Rank r finalises tokens [r, r + 1) * BT / KS of the tile.  The accumulator is turned round in
// shared memory (in [token][column] order a thread gets 16 or 32 neighbouring columns of one token,
// which the fp16 rows and the NVFP4 scale blocks both want), and that staging is also what a bulk
// copy sends to the peers, 32 tokens at a time so that the copies, the drain of the next columns and
// the sums overlap.  The landing area is not part of the operand ring: a rank may send as soon as it
// is done, without asking whether its peers are.  The older exchange took K = 4096 to 9.1-10.1 us on
// 7168 columns; this one 5.8 (17 rows) and 7.4 (128).
// Tried and not kept, on 128 x 7168 x 16384, each against this kernel in the same session: CTA pairs that halve the
// activations' bytes again (15.1 us, this one 14.5-15.2: the ring is not what binds, and the pair meets before its
// first load); prefetching weights into L2 further ahead than the ring (17.9, 15.1: the TMA unit serves prefetches
// like loads); eight epilogue warps (14.9, 14.5).
//
// Warp roles as in gemm_sm100.cuh: warp 0 TMA producer, warp 1 MMA issuer, one thread each; warps
// 2..5 epilogue.  Every wait is bounded.  No load uses cluster multicast.
#pragma once
#include "gemm_sm100.cuh"

namespace nvfp4 {

constexpr int kDecodeThreads = 192;

template <int BT, int STAGES, int KS>
struct DecodeSmem {
    static constexpr uint32_t kWBytes = kBM * kBKBytes;               // weights: 128 rows of 256 e2m1
    static constexpr uint32_t kXBytes = BT * kBKBytes;                // activations: BT rows
    static constexpr uint32_t kSfBytes = kMmaPerStage * kSfAtomBytes; // scales of 128 rows, for either operand
    static constexpr uint32_t kStageBytes = kWBytes + kXBytes + 2 * kSfBytes;
    static constexpr int kPieceTokens = BT / KS;                      // tokens a rank finalises
    static constexpr int kChunkTokens = kPieceTokens < 32 ? kPieceTokens : 32;
    static constexpr int kChunks = kPieceTokens / kChunkTokens;
    static constexpr uint32_t kChunkBytes = kChunkTokens * kBM * 4;   // [token][128 columns] fp32
    static constexpr uint32_t kPieceBytes = kChunks * kChunkBytes;
    static constexpr uint32_t kLandOff = STAGES * kStageBytes;        // the other ranks' sums of this CTA's piece
    static constexpr uint32_t kBarOff = kLandOff + (KS - 1) * kPieceBytes;
    // full[STAGES] empty[STAGES] accumulator landed[kChunks] | tmem slot | abort
    static constexpr uint32_t kNumBars = 2 * STAGES + 1 + kChunks;
    static constexpr uint32_t kBytes = kBarOff + kNumBars * 8 + 16;
    static constexpr uint32_t kDynamicBytes = kBytes + 1024;          // slack for manual 1024-byte alignment
    static_assert(kStageBytes % 1024 == 0 && kPieceBytes % 1024 == 0, "tiles must keep 1024-byte alignment");
    static_assert(KS * kPieceBytes <= STAGES * kStageBytes, "the idle ring must hold the whole accumulator");
    static_assert(kDynamicBytes <= 232448, "exceeds the 227 KB of shared memory one CTA may use");
};

// Scale buffers behind the accumulator's BT columns; the double buffers of the two operands.
constexpr int kDecodeSfwCol = 128, kDecodeSfxCol = 160, kDecodeTmemCols = 256;

template <int BT, int STAGES, int KS, bool EPI_EX>
__global__ void __launch_bounds__(kDecodeThreads, 1) gemm_decode_kernel(const __grid_constant__ GemmParams p) {
    using S = DecodeSmem<BT, STAGES, KS>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - ptx::smem_u32(smem_raw));
    const uint32_t bar_full = smem_base + S::kBarOff;
    const uint32_t bar_empty = bar_full + STAGES * 8;
    const uint32_t bar_acc = bar_empty + STAGES * 8;
    const uint32_t bar_land = bar_acc + 8;
    const uint32_t tmem_slot = bar_land + S::kChunks * 8;
    volatile uint32_t* tmem_slot_gen = reinterpret_cast<volatile uint32_t*>(smem_gen + S::kBarOff + S::kNumBars * 8);
    volatile uint32_t* abort_flag = tmem_slot_gen + 1;

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int ks_rank = KS > 1 ? static_cast<int>(ptx::cluster_ctarank()) : 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(bar_full + s * 8, 1);
            ptx::mbar_init(bar_empty + s * 8, 1);
        }
        ptx::mbar_init(bar_acc, 1);
        for (int c = 0; c < S::kChunks; ++c) ptx::mbar_init(bar_land + c * 8, 1);
        *abort_flag = 0u;
        ptx::fence_mbar_init();
        // what will land is known now, so that nobody has to ask before sending
        if (KS > 1)
            for (int c = 0; c < S::kChunks; ++c) ptx::mbar_expect_tx(bar_land + c * 8, (KS - 1) * S::kChunkBytes);
        ptx::prefetch_tensormap(&p.tma_a);
        ptx::prefetch_tensormap(&p.tma_b);
        ptx::prefetch_tensormap(&p.tma_sfa);
        ptx::prefetch_tensormap(&p.tma_sfb);
    }
    __syncthreads();
    if constexpr (KS > 1) ptx::cluster_arrive();   // peers are written to in the exchange only: the wait is there
    bool cluster_waited = KS == 1;
    uint32_t tmem_base = 0;
    if (warp == 1) {
        ptx::tmem_alloc<1>(tmem_slot, kDecodeTmemCols);
        ptx::tmem_relinquish<1>();
        ptx::tc_fence_before();
    }
    const int KT = p.k_tiles;
    const int tile = static_cast<int>(blockIdx.x) / KS;
    // (the token tiles that share a block of weights are neighbours, so that it comes from HBM once)
    const int mt = tile % p.tiles_m;                 // token tile
    const int l = tile / p.tiles_m / p.tiles_n;
    const int nb = tile / p.tiles_m - l * p.tiles_n; // 128-row block of the weights
    const int k0 = (ks_rank * KT) / KS, k1 = ((ks_rank + 1) * KT) / KS;
    const uint64_t timeout = p.timeout_cycles;
    // the first operands are asked into L2 ahead of the dependency wait (see gemm_sm100.cuh)
    if (warp == 0) {
        if (ptx::elect_one()) {
            for (int kt = k0; kt < min(k1, k0 + kPrefetchStages); ++kt) {
                ptx::tma_prefetch_3d(&p.tma_b, kt * kBKBytes, nb * kBM, l);
                ptx::tma_prefetch_4d(&p.tma_sfb, 0, kt * kMmaPerStage, nb, l);
                ptx::tma_prefetch_3d(&p.tma_a, kt * kBKBytes, mt * BT, l);
                ptx::tma_prefetch_4d(&p.tma_sfa, 0, kt * kMmaPerStage, mt, l);
            }
        }
        __syncwarp();
    }
    ptx::grid_dependency_launch_dependents();
    ptx::grid_dependency_wait();
    if (warp != 0) {
        ptx::named_bar_sync(3, kDecodeThreads - 32);
        ptx::tc_fence_after();
        tmem_base = *tmem_slot_gen;
    }

    if (warp == 0) {
        // ------------------------------------------------------------ producer
        const uint64_t pol_x = ptx::policy_evict_last();     // re-read by every weight block
        const uint64_t pol_w = p.tiles_m > 1 ? ptx::policy_evict_last() : ptx::policy_evict_first();   // read once per token tile
        if (ptx::elect_one()) {
            uint32_t stage = 0, phase = 0;
            for (int kt = k0; kt < k1; ++kt) {
                if (!ptx::mbar_wait_bounded(bar_empty + stage * 8, phase ^ 1u, abort_flag, timeout)) break;
                const uint32_t sw = smem_base + stage * S::kStageBytes;
                const uint32_t sx = sw + S::kWBytes;
                const uint32_t ssfw = sx + S::kXBytes, ssfx = ssfw + S::kSfBytes;
                const uint32_t full = bar_full + stage * 8;
                ptx::mbar_expect_tx(full, S::kStageBytes);
                ptx::tma_load_3d(sw, &p.tma_b, kt * kBKBytes, nb * kBM, l, full, pol_w);
                ptx::tma_load_4d(ssfw, &p.tma_sfb, 0, kt * kMmaPerStage, nb, l, full);
                ptx::tma_load_3d(sx, &p.tma_a, kt * kBKBytes, mt * BT, l, full, pol_x);
                ptx::tma_load_4d(ssfx, &p.tma_sfa, 0, kt * kMmaPerStage, mt, l, full);
                if (++stage == STAGES) { stage = 0; phase ^= 1u; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------ MMA issuer (one thread, see gemm_sm100.cuh)
        constexpr uint32_t idesc = ptx::idesc_nvf4(kBM, BT);
        const uint64_t desc_ab0 = ptx::smem_desc_sw128(smem_base);
        const uint64_t desc_sf0 = ptx::smem_desc_sf(smem_base + S::kWBytes + S::kXBytes);
        const uint32_t ab_lo0 = static_cast<uint32_t>(desc_ab0), ab_hi = static_cast<uint32_t>(desc_ab0 >> 32);
        const uint32_t sf_lo0 = static_cast<uint32_t>(desc_sf0), sf_hi = static_cast<uint32_t>(desc_sf0 >> 32);
        if (ptx::elect_one()) {
            uint32_t stage = 0, phase = 0;
            for (int kt = k0; kt < k1; ++kt) {
                if (!ptx::mbar_wait_bounded(bar_full + stage * 8, phase, abort_flag, timeout)) break;
                ptx::tc_fence_after();
                const uint32_t slot_off = stage * (S::kStageBytes >> 4);
                const uint32_t w_lo = ab_lo0 + slot_off, x_lo = w_lo + (S::kWBytes >> 4);
                const uint32_t sfw_lo = sf_lo0 + slot_off, sfx_lo = sfw_lo + (S::kSfBytes >> 4);
                const uint32_t sf_buf = static_cast<uint32_t>(kt - k0) & 1u;
                const uint32_t t_sfw = tmem_base + kDecodeSfwCol + sf_buf * 16;
                const uint32_t t_sfx = tmem_base + kDecodeSfxCol + sf_buf * 16;
#pragma unroll
                for (int kb = 0; kb < kMmaPerStage; ++kb) {
                    ptx::tc_cp_sf<1>(t_sfw + kb * 4, sfw_lo + kb * (kSfAtomBytes >> 4), sf_hi);
                    ptx::tc_cp_sf<1>(t_sfx + kb * 4, sfx_lo + kb * (kSfAtomBytes >> 4), sf_hi);
                }
#pragma unroll
                for (int kb = 0; kb < kMmaPerStage; ++kb)
                    ptx::tc_mma_nvf4<1>(tmem_base, w_lo + 2 * kb, x_lo + 2 * kb, ab_hi, idesc, t_sfw + kb * 4, t_sfx + kb * 4,
                                         (kt > k0 || kb > 0) ? 1u : 0u);
                ptx::tc_commit(bar_empty + stage * 8);
                if (kt + 1 == k1) ptx::tc_commit(bar_acc);
                if (++stage == STAGES) { stage = 0; phase ^= 1u; }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------ epilogue
        const int quad = warp & 3;             // TMEM lane quadrant this warp may read
        const int col = quad * 32 + lane;      // output column of this thread's TMEM lane, in the 128-wide block
        const int tid = threadIdx.x - 64;      // 0..127
        // Staging and landing areas hold [token][128 columns] fp32 chunks, the 16-byte units of a
        // token's row permuted inside groups of eight so that neither the writers (a warp: 32
        // neighbouring columns of a token) nor the readers (16-byte units, below) meet in a bank.
        auto unit_at = [](int token, int unit) { return (unit & ~7) | ((unit ^ (4 * (token & 1) + (unit >> 3))) & 7); };
        float* const stage_gen = reinterpret_cast<float*>(smem_gen);        // the ring, idle once the accumulator is complete
        const float* const land_gen = reinterpret_cast<const float*>(smem_gen + S::kLandOff);
        if (!cluster_waited) { ptx::cluster_wait(); cluster_waited = true; }
        bool ok = ptx::mbar_wait_bounded(bar_acc, 0u, abort_flag, timeout);
        if (ptx::named_bar_and(2, 128, ok)) {
            ptx::tc_fence_after();
            const uint32_t t_acc = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
            // Blocks of 32 tokens are turned round into the staging area (token t at row t of it), the own
            // piece last.  When a block is complete in shared memory, one thread sends what it holds of
            // other ranks' pieces.
            constexpr int kBlocks = BT / 32;
            constexpr int kPiecesPerBlock = 32 / S::kChunkTokens;              // pieces that a block holds, when they are that small
            const int first_block = (kPiecesPerBlock > 1) ? 0 : (ks_rank + 1) % KS * S::kChunks;
#pragma unroll 1
            for (int i = 0; i < kBlocks; ++i) {
                const int b = (first_block + i) % kBlocks;
                uint32_t v[32];
                ptx::tc_ld_32cols(t_acc + b * 32, v);
                ptx::tc_wait_ld();
#pragma unroll
                for (int t = 0; t < 32; ++t) stage_gen[(b * 32 + t) * kBM + unit_at(t, col >> 2) * 4 + (col & 3)] = __uint_as_float(v[t]);
                if constexpr (KS > 1) {
                    ptx::fence_proxy_async_smem();      // read by the bulk copies (async proxy)
                    ptx::named_bar_sync(1, 128);
                    if (tid == 0) {
#pragma unroll 1
                        for (int h = 0; h < kPiecesPerBlock; ++h) {
                            const int token = b * 32 + h * S::kChunkTokens;
                            const int q = token / S::kPieceTokens;                     // the rank that finalises them
                            const int c = (token % S::kPieceTokens) / S::kChunkTokens;
                            const int slot = ks_rank - (ks_rank > q ? 1 : 0);          // q keeps the foreign pieces in rank order
                            if (q != ks_rank)
                                ptx::bulk_copy_to_cluster(ptx::mapa_u32(smem_base + S::kLandOff + slot * S::kPieceBytes + c * S::kChunkBytes, q),
                                                          smem_base + token * (kBM * 4), S::kChunkBytes, ptx::mapa_u32(bar_land + c * 8, q));
                        }
                    }
                    __syncwarp();
                }
            }
            if constexpr (KS == 1) ptx::named_bar_sync(1, 128);
            // Sum and store: a thread takes kCols neighbouring columns of one token at a time.
            constexpr int kCols = S::kChunkTokens < 16 ? 16 : S::kChunkTokens;
            constexpr int kParts = kBM / kCols;                                 // threads per token
            const int t_in_chunk = tid / kParts, c0 = (tid % kParts) * kCols;
            const int gcol = nb * kBM + c0;
#pragma unroll 1
            for (int c = 0; c < S::kChunks; ++c) {
                if constexpr (KS > 1) {
                    ok = ptx::mbar_wait_bounded<true>(bar_land + c * 8, 0u, abort_flag, timeout);
                    if (!ptx::named_bar_and(2, 128, ok)) break;
                }
                const int token = ks_rank * S::kPieceTokens + c * S::kChunkTokens + t_in_chunk;   // in the tile
                const int row = mt * BT + token;
                if (t_in_chunk < S::kChunkTokens && row < p.M) {
                    // (the extended epilogue's code exists once, for 16 columns a turn: it is fetched cold)
                    constexpr int kUnroll = EPI_EX ? 1 : kCols / 16;
#pragma unroll kUnroll
                    for (int h = 0; h < kCols; h += 16) {
                        float s[16];
#pragma unroll
                        for (int i = 0; i < 16; ++i) s[i] = 0.f;
#pragma unroll
                        for (int r = 0; r < KS; ++r) {   // ascending rank: the same sum whoever finalises
                            const float* src = (r == ks_rank) ? stage_gen + token * kBM
                                                              : land_gen + (r - (r > ks_rank ? 1 : 0)) * (S::kPieceBytes / 4) + (c * S::kChunkTokens + t_in_chunk) * kBM;
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const float4 t = *reinterpret_cast<const float4*>(src + unit_at(token, (c0 + h) / 4 + j) * 4);
                                s[4 * j] += t.x; s[4 * j + 1] += t.y; s[4 * j + 2] += t.z; s[4 * j + 3] += t.w;
                            }
                        }
                        if constexpr (EPI_EX) bias_act16(p, gcol + h, s);
                        if (!EPI_EX || !p.out_nvfp4) {
                            __half* dst = p.c + l * p.c_batch_stride + static_cast<long long>(row) * p.c_row_stride + gcol + h;
                            *reinterpret_cast<uint4*>(dst) = pack8_fp16(&s[0]);
                            *reinterpret_cast<uint4*>(dst + 8) = pack8_fp16(&s[8]);
                        } else {
                            float v[16];
#pragma unroll
                            for (int i = 0; i < 8; ++i) {   // the fp16-rounded values are quantised, as in gemm_sm100.cuh
                                const float2 f = __half22float2(__floats2half2_rn(s[2 * i], s[2 * i + 1]));
                                v[2 * i] = f.x;
                                v[2 * i + 1] = f.y;
                            }
                            uint32_t o[2];
                            const uint8_t sf = quantize_block16(v, o);
                            const int blk = (gcol + h) / 16;
                            *reinterpret_cast<uint2*>(p.out_packed + l * p.out_packed_batch_stride + static_cast<long long>(row) * p.out_packed_row_stride +
                                                      blk * 8) = make_uint2(o[0], o[1]);
                            if (p.out_sf != nullptr) p.out_sf[l * p.out_sf_batch_stride + static_cast<long long>(row) * p.out_sf_row_stride + blk] = sf;
                            if (p.out_sf_perm != nullptr)   // (more than one token tile: of 128, a row block each)
                                p.out_sf_perm[l * p.out_sf_perm_batch_stride + mt * p.out_sf_perm_block_stride + (blk / 4) * 512 + (token % 32) * 16 + (token / 32) * 4 + blk % 4] = sf;
                        }
                    }
                }
                __syncwarp();
            }
            if constexpr (EPI_EX) {
                // rows of the 128-row scale block that do not exist read as zero scales: eight blocks = two words per row
                if (p.out_nvfp4 && p.out_sf_perm != nullptr && ks_rank == 0 && mt * BT + tid >= p.M) {
                    uint8_t* dst = p.out_sf_perm + l * p.out_sf_perm_batch_stride + mt * p.out_sf_perm_block_stride + nb * 2 * 512 + (tid % 32) * 16 + (tid / 32) * 4;
                    *reinterpret_cast<uint32_t*>(dst) = 0u;
                    *reinterpret_cast<uint32_t*>(dst + 512) = 0u;
                }
            }
            __syncwarp();
        }
    }

    // ---------------------------------------------------------------- teardown
    if (!cluster_waited) ptx::cluster_wait();
    ptx::tc_fence_before();
    __syncthreads();
    meet_cluster<KS>(abort_flag, tmem_slot + 4, p.status);
    const bool gave_up = KS > 1 && *abort_flag;
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc<1>(tmem_base, kDecodeTmemCols);
    }
    if constexpr (KS > 1) leave_cluster(gave_up);
}

}  // namespace nvfp4
