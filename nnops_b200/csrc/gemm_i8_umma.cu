// int8 GEMM for prefill-sized problems on sm_100a: out = epilogue(A[M,K] * W[N,K]^T).
//
// Replaces the reference's mma.sync tile engine (i8_gemm_kernel,
// src/backend/cuda/matmul/matmul_i8_ptx.cu:22-385) with a design native to Blackwell:
//
//   * persistent CTAs (one per SM), each walking 128 x BN output tiles in an L2-friendly
//     grouped order;
//   * warp 0 streams A and W tiles (128 bytes of K per stage) into a shared-memory ring with
//     TMA, 128-byte swizzle, out-of-range rows/columns zero-filled by the hardware;
//   * warp 1 issues tcgen05.mma kind::i8 (M128 x N=BN x K32) into one of two TMEM
//     accumulators and frees ring slots with tcgen05.commit;
//   * the other warps -- sixteen for 8-bit destinations, eight for the rest, four in the sharded
//     form (see sixteen_warps) -- drain the other accumulator with tcgen05.ld and apply the fused
//     epilogue (zero-point compensation, int32 bias, Relu, requantisation / dequantisation) in
//     registers, so the epilogue of tile i overlaps the main loop of tile i+1.
//
// Sharded form (template flag PEERS): the epilogue of an 8-bit destination stages 32 rows x 128
// columns per warp in shared memory (128-byte swizzle) and hands each such tile to TMA, once per
// destination: this GPU's output and the same window of every peer GPU's output (peer memory
// over NVLink).  The all-gather is thereby fused into the GEMM's write-back, tile by tile, as
// asynchronous bulk stores; the epilogue warps only wait for a staging buffer to be read out.
// Loads never touch peer memory.
//
// Both operands are already K-major in memory ([M,K] and [N,K]), which is the layout the
// UMMA shared-memory descriptors want, so no transposes or repacking happen anywhere.
// Every barrier wait is bounded; a wait that runs out records an error code and the CTA
// tears down cleanly.

#include <cuda_fp16.h>

#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <mutex>

#include "internal.cuh"
#include "gemm_i8_umma_tile.cuh"
#include "ptx.cuh"
#include "ptx_pair.cuh"

namespace nnb200 {

namespace {

// ---- CTA-pair form ---------------------------------------------------------------------------
// Two CTAs (a cluster of two, on neighbouring SMs) share one 256 x BN output tile: each loads its
// own 128 rows of A and HALF of the tile's W rows, the pair leader issues tcgen05.mma with
// cta_group::2 (M = 256 over both SMs' tensor cores and TMEM), and each CTA drains its own 128
// accumulator rows through the same epilogue.  Per multiply-add the pair moves two thirds of the
// operand bytes through L2 and shared memory, which under the power cap is worth clock.
//
// What the form lives or dies by is how often the tensor pipe is interrupted: every commit is a
// point the pipe drains to, and every barrier wait a round trip for the issuing thread.  With one
// 128-byte k-block per barrier slot (4 MMAs between commits, one commit per destination CTA) the
// pipe was busy 75 % of the cycles and the form LOST to the single-CTA kernel; with two k-blocks
// per slot (SUB = 2: 8 MMAs between commits) and one commit instruction that arrives on both
// CTAs' barriers (MC) it is busy about 89 % and wins by 8-9 %.  Three k-blocks per slot leave a
// ring of two slots, too coarse to hide the loads, and lose again.
//
// Signalling: TMA loads of both CTAs report their bytes to the LEADER's full barrier; the
// leader's commits arrive on BOTH CTAs' empty / accumulator-full barriers; the epilogue warps of
// both CTAs arrive on the leader's accumulator-empty barrier.  A cluster barrier brackets the
// kernel so neither CTA initialises late or exits early.
template <int BN>
struct PairTileConfig {
    static constexpr int kATileBytes = kBlockM * kBlockKBytes;   // this CTA's 128 rows of A
    static constexpr int kBTileBytes = (BN / 2) * kBlockKBytes;  // this CTA's half of the W rows
    static constexpr int kStageBytes = kATileBytes + kBTileBytes;
    static constexpr int kHalf0 = first_half_cols(BN, 0);
    static constexpr int kColParamBytes = epilogue_warps(0) * 4 * kHalf0 * 4;
    static constexpr int kStages = (208 * 1024 - kColParamBytes) / kStageBytes;  // 256: 6, 224: 6, 192: 7
    static constexpr int kTmemCols = 512;
    static constexpr int kBarrierBytes = (2 * kStages + 4) * 8 + 16;
    static constexpr int kSmemBytes = 1024 + kStages * kStageBytes + kColParamBytes + kBarrierBytes;
};

template <int BN, int KIND, int SUB, bool MC, bool CONV = false, int POSE = 0>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kMaxThreads, 1)
gemm_i8_umma_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                         const I8Epilogue ep, const int m_total, const int n_total, const int k_total,
                         const uint32_t idesc, const int vec_ok, const int group_m, const int k_rot,
                         int32_t* error_word, const ConvTile conv)
{
    using Cfg = PairTileConfig<BN>;
    // SUB consecutive 128-byte k-blocks share one pair of barriers (a "slot"): one wait, one
    // expect-tx and one pair of commits per SUB x 4 MMAs.
    constexpr int kStages = Cfg::kStages / SUB;           // slots in the ring
    constexpr int kSlotBytes = SUB * Cfg::kStageBytes;
    constexpr int kPairM = 2 * kBlockM;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* stage_base = smem;
    int32_t* col_params = reinterpret_cast<int32_t*>(smem + Cfg::kStages * Cfg::kStageBytes);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(col_params + Cfg::kColParamBytes / 4);
    uint64_t* empty_bar = full_bar + Cfg::kStages;
    uint64_t* acc_full_bar = empty_bar + Cfg::kStages;
    uint64_t* acc_empty_bar = acc_full_bar + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty_bar + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int role = warp_uniform(warp);   // the same, warp-uniform to the compiler too
    const int lane = threadIdx.x & 31;
    const uint32_t rank = cluster_cta_rank();  // 0 = pair leader
    const int pair = static_cast<int>(blockIdx.x >> 1);
    const int num_pairs = static_cast<int>(gridDim.x >> 1);
    const int num_m = (m_total + kPairM - 1) / kPairM;
    const int num_n = (n_total + BN - 1) / BN;
    const int num_tiles = num_m * num_n;
    const int num_kb = (k_total + kBlockKBytes - 1) / kBlockKBytes;
    const TileWalk walk(num_m, num_n, group_m);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full_bar[s], 1);   // the leader's: its own expect-tx arrival; bytes come from both CTAs
            mbar_init(&empty_bar[s], 1);  // one commit from the leader
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full_bar[a], 1);
            mbar_init(&acc_empty_bar[a], 2 * epilogue_warps(0));  // the leader's: the epilogue warps of both CTAs
        }
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == 0 && lane == 0) {
        tma_prefetch_desc(&map_a);
        tma_prefetch_desc(&map_w);
    }
    if (warp == 1) {
        tmem_alloc_pair(tmem_slot, Cfg::kTmemCols);
        tmem_relinquish_pair();
    }
    tc_fence_before_sync();
    cluster_sync_all();  // both CTAs' barriers and TMEM exist before anything is signalled across
    tc_fence_after_sync();
    previous_kernel_done();
    const uint32_t tmem_base = *tmem_slot;

    // In both issuing roles the whole warp walks the loop, one elected lane issues, and no branch depends on
    // what a wait returned (see mbar_wait_converged).
    uint32_t failed = 0;   // this role's first failed wait, see mbar_wait_converged
    int stage = 0;
    uint32_t phase = 0;
    if (role == 0) {
        // ---------------- TMA producer (each CTA loads its own halves) ----------------
        for (int tile = pair; tile < num_tiles; tile += num_pairs) {
            const TileCoord tc = walk(tile);
            const int m0 = warp_uniform(tc.m_blk * kPairM + static_cast<int>(rank) * kBlockM);
            const int n0 = warp_uniform(tc.n_blk * BN + static_cast<int>(rank) * (BN / 2));
            const int rot = warp_uniform(k_rotation(tile, k_rot, num_kb));
            int patch_w = 0, patch_h = 0, patch_img = 0, tap_a = 0, tap_b = 0, tap_c = 0;   // CONV
            (void)patch_w; (void)patch_h; (void)patch_img; (void)tap_a; (void)tap_b; (void)tap_c;
            if constexpr (CONV) {
                // This CTA's patch of the pair (2 * m_blk + rank), shifted by the k-block's tap.
                const ConvPatch pt = conv_patch(conv, 2 * tc.m_blk + static_cast<int>(rank));
                patch_w = warp_uniform((pt.tw << conv.bw_log2) * conv.sw - conv.pw);
                patch_h = warp_uniform(pt.th * conv.bh * conv.sh - conv.ph);
                patch_img = warp_uniform(pt.img);
                const int tap = rot / conv.kb_per_tap;
                tap_c = warp_uniform(rot - tap * conv.kb_per_tap);
                tap_a = warp_uniform(tap / conv.kw);
                tap_b = warp_uniform(tap - tap_a * conv.kw);
            }
            int kx = rot;
            for (int kb = 0; kb < num_kb; kb += SUB) {
                mbar_wait_converged_cluster<kErrProducerWait>(&empty_bar[stage], phase ^ 1u, abort_flag, failed);
                const int nsub = (num_kb - kb) < SUB ? (num_kb - kb) : SUB;
                const uint32_t leader_full = map_to_cta(smem_u32(&full_bar[stage]), 0);
                const bool issue = elect_one() && !wait_failed(failed);
                if (issue && rank == 0) {
                    mbar_expect_tx(&full_bar[stage], 2 * nsub * Cfg::kStageBytes);
                }
#pragma unroll
                for (int j = 0; j < SUB; ++j) {
                    if (j < nsub) {
                        uint8_t* a_dst = stage_base + stage * kSlotBytes + j * Cfg::kStageBytes;
                        uint8_t* b_dst = a_dst + Cfg::kATileBytes;
                        if (issue) {
                            if constexpr (CONV) {
                                tma_load_4d_pair(a_dst, &map_a, leader_full, conv.c_base + tap_c * kBlockKBytes,
                                                 patch_w + tap_b * conv.dw, patch_h + tap_a * conv.dh, patch_img);
                            } else if constexpr ((POSE & 1) != 0) {
                                // A stored [K][M]: 128 k-rows of this CTA's 128 m-bytes.
                                tma_load_2d_pair(a_dst, &map_a, leader_full, m0, kx * kBlockKBytes);
                            } else {
                                tma_load_2d_pair(a_dst, &map_a, leader_full, kx * kBlockKBytes, m0);
                            }
                            if constexpr ((POSE & 2) != 0) {
                                // W stored [K][N]: 128 k-rows of this CTA's 128 n-bytes (BN = 256).
                                tma_load_2d_pair(b_dst, &map_w, leader_full, n0, kx * kBlockKBytes);
                            } else {
                                tma_load_2d_pair(b_dst, &map_w, leader_full, kx * kBlockKBytes, n0);
                            }
                        }
                        __syncwarp();
                        if constexpr (CONV) {
                            if (++tap_c == conv.kb_per_tap) {
                                tap_c = 0;
                                if (++tap_b == conv.kw) {
                                    tap_b = 0;
                                    if (++tap_a == conv.kh) {
                                        tap_a = 0;
                                    }
                                }
                            }
                        }
                        if (++kx == num_kb) {
                            kx = 0;
                        }
                    }
                }
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        }
        let_next_kernel_start();
        if (const uint32_t code = warp_failure(failed); code != 0 && lane == 0) {
            atomicCAS(error_word, 0, static_cast<int32_t>(code));
        }
        __syncwarp();
    } else if (role == 1) {
        // ---------------- MMA issuer (pair leader only) ----------------
        const uint32_t tmem = warp_uniform(tmem_base);
        // MN-major tiles (POSE bits): 32 k-rows of 128 bytes per K step instead of 32 bytes along the row, as in
        // the single-CTA kernel.  The ring's descriptors advance by addition.
        const uint32_t ring = smem_u32(stage_base);
        const uint64_t a_first = (POSE & 1) ? umma_desc_sw128_mnmajor(ring, 128 * kBlockKBytes) : umma_desc_sw128_kmajor(ring);
        const uint64_t b_first = (POSE & 2) ? umma_desc_sw128_mnmajor(ring + Cfg::kATileBytes, 128 * kBlockKBytes)
                                            : umma_desc_sw128_kmajor(ring + Cfg::kATileBytes);
        constexpr uint64_t a_step = (POSE & 1) ? 256u : 2u;
        constexpr uint64_t b_step = (POSE & 2) ? 256u : 2u;
        uint64_t a_desc = a_first, b_desc = b_first;
        int local_tile = 0;
        for (int tile = pair; rank == 0 && tile < num_tiles; tile += num_pairs, ++local_tile) {
            const int acc = local_tile & 1;
            const uint32_t acc_phase = (local_tile >> 1) & 1u;
            mbar_wait_converged_cluster<kErrAccumWait>(&acc_empty_bar[acc], acc_phase ^ 1u, abort_flag, failed);
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem + static_cast<uint32_t>(acc * 256);
            uint32_t accumulate = 0;
            for (int kb = 0; kb < num_kb; kb += SUB) {
                mbar_wait_converged_cluster<kErrMmaWait>(&full_bar[stage], phase, abort_flag, failed);
                tc_fence_after_sync();
                const int nsub = (num_kb - kb) < SUB ? (num_kb - kb) : SUB;
                if (elect_one()) {
#pragma unroll
                    for (int j = 0; j < SUB; ++j) {
                        if (j < nsub) {
#pragma unroll
                            for (int ks = 0; ks < kBlockKBytes / kUmmaK; ++ks) {
                                umma_i8_pair(d_tmem, a_desc + static_cast<uint64_t>(j * (Cfg::kStageBytes / 16)) + static_cast<uint64_t>(ks) * a_step,
                                             b_desc + static_cast<uint64_t>(j * (Cfg::kStageBytes / 16)) + static_cast<uint64_t>(ks) * b_step,
                                             idesc, (j > 0 || ks > 0) ? 1u : accumulate);
                            }
                        }
                    }
                    // The slot is free in BOTH CTAs once these MMAs have read it.
                    if constexpr (MC) {
                        umma_commit_pair_mask(&empty_bar[stage], 3);
                    } else {
                        const uint32_t e = smem_u32(&empty_bar[stage]);
                        umma_commit_pair(map_to_cta(e, 0));
                        umma_commit_pair(map_to_cta(e, 1));
                    }
                }
                __syncwarp();
                accumulate = 1;
                a_desc += kSlotBytes / 16;
                b_desc += kSlotBytes / 16;
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                    a_desc = a_first;
                    b_desc = b_first;
                }
            }
            if (elect_one()) {
                if constexpr (MC) {
                    umma_commit_pair_mask_unless(&acc_full_bar[acc], 3, failed);
                } else {
                    const uint32_t f = smem_u32(&acc_full_bar[acc]);
                    umma_commit_pair_unless(map_to_cta(f, 0), failed);
                    umma_commit_pair_unless(map_to_cta(f, 1), failed);
                }
            }
            __syncwarp();
        }
        if (const uint32_t code = warp_failure(failed); code != 0) {
            if (lane == 0) {
                atomicCAS(error_word, 0, static_cast<int32_t>(code));
            }
            umma_settle_after_failure();
        }
        __syncwarp();
    } else {
        // ---------------- epilogue warps (each CTA drains its own 128 rows) ----------------
        const int quarter = warp & 3;
        const bool fold_scale = KIND != NNB200_OUT_S32 && ep.scale_a == nullptr;
        const float folded_row_k = (KIND == NNB200_OUT_S8 || KIND == NNB200_OUT_U8)
                                       ? __fdiv_rn(ep.scale_a_scalar, ep.out_scale) : ep.scale_a_scalar;
        const bool fold_comp = (KIND == NNB200_OUT_S8 || KIND == NNB200_OUT_U8) && ep.compensate != 0 &&
                               ep.zp_a == nullptr && ep.r_a == nullptr;
        constexpr int kTermIters = (Cfg::kHalf0 + 31) / 32;   // 4 for 256-wide tiles
        ColTerms next_terms[kTermIters];
        constexpr int kHalf0 = Cfg::kHalf0;
        const int half = (warp - 2) >> 2;   // two warps per lane quarter, half of the columns each
        const int col0 = half * kHalf0;
        const int ncols = half ? BN - kHalf0 : kHalf0;
        float* cs = reinterpret_cast<float*>(col_params + (warp - 2) * 4 * kHalf0);
        int32_t* cb = reinterpret_cast<int32_t*>(cs) + kHalf0;
        int32_t* cr = cb + kHalf0;
        int32_t* cz = cr + kHalf0;
        int local_tile = 0;
        for (int tile = pair; tile < num_tiles; tile += num_pairs, ++local_tile) {
            const TileCoord tc = walk(tile);
            const int acc = local_tile & 1;
            const uint32_t acc_phase = (local_tile >> 1) & 1u;
            const int n_base = tc.n_blk * BN + col0;   // first column this warp drains

            // This tile's per-column terms: fetched while the previous tile was being drained, or
            // (first tile) now, hidden behind the tile's main loop.
            __syncwarp();
#pragma unroll
            for (int i = 0; i < kTermIters; ++i) {
                const int j = lane + i * 32;
                if (j < ncols) {
                    const ColTerms ct = finish_col_terms<KIND>(
                        ep, local_tile > 0 ? next_terms[i] : load_col_terms<KIND>(ep, n_base + j, n_total), fold_scale,
                        folded_row_k, fold_comp);
                    cs[j] = ct.scale;
                    cb[j] = ct.bias;
                    cr[j] = ct.rw;
                    cz[j] = ct.zpw;
                }
            }
            __syncwarp();

            int64_t m = static_cast<int64_t>(tc.m_blk) * kPairM + static_cast<int64_t>(rank) * kBlockM +
                        quarter * 32 + lane;
            bool row_ok = m < m_total;
            uint32_t bad_h = 0, bad_w = 0;   // CONV: the row's border class along each axis
            if constexpr (CONV) {
                const ConvRow cr_ = conv_row(conv, 2 * tc.m_blk + static_cast<int>(rank), quarter * 32 + lane);
                m = cr_.m;
                row_ok = cr_.ok;
                bad_h = cr_.bad_h;
                bad_w = cr_.bad_w;
            }
            I8RowTerms rt;
            rt.zpa = 0;
            rt.ra = 0;
            rt.s_a = 1.0f;
            rt.row_k = 1.0f;
            if (row_ok) {
                rt = i8_row_terms(ep, m);
            }

            int ok = 1;
            if (lane == 0) {
                ok = mbar_wait_cluster(&acc_full_bar[acc], acc_phase, abort_flag) ? 1 : 0;
            }
            ok = __shfl_sync(0xFFFFFFFFu, ok, 0);
            if (!ok) {
                atomicCAS(error_word, 0, kErrEpilogueWait);
                break;
            }
            tc_fence_after_sync();

            {
                // The next tile's column terms, in flight while this tile is drained.
                const int next = tile + num_pairs;
                if (next < num_tiles) {
                    const int next_base = walk(next).n_blk * BN + col0;
#pragma unroll
                    for (int i = 0; i < kTermIters; ++i) {
                        next_terms[i] = load_col_terms<KIND>(ep, next_base + lane + i * 32, n_total);
                    }
                }
            }

            const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                   static_cast<uint32_t>(acc * 256 + col0);
            // Chunks of 32 columns, two register sets: the load of the next chunk is in flight while
            // this one is requantised and stored.
            const int left = n_total - n_base;
            const int nch = left <= 0 ? 0 : min(ncols / 32, (left + 31) / 32);   // uniform across the warp
            const auto finish = [&](int c, uint32_t (&v)[32]) {
                const int n0 = n_base + c * 32;
                if constexpr (CONV) {
                    conv_border_fix(conv, v, bad_h, bad_w, n0, n_total);
                }
                epilogue_chunk<KIND>(ep, rt, v, m, row_ok, n0, n_total, cs + c * 32, cb + c * 32, cr + c * 32,
                                     cz + c * 32, vec_ok, fold_scale, fold_comp);
            };
            uint32_t va[32], vb[32];
            if (nch > 0) {
                tmem_ld_32x32(t_row, va);
            }
#pragma unroll 1
            for (int c = 0; c < nch; c += 2) {
                tmem_ld_wait();
                if (c + 1 < nch) {
                    tmem_ld_32x32(t_row + static_cast<uint32_t>((c + 1) * 32), vb);
                }
                finish(c, va);
                if (c + 1 < nch) {
                    tmem_ld_wait();
                    if (c + 2 < nch) {
                        tmem_ld_32x32(t_row + static_cast<uint32_t>((c + 2) * 32), va);
                    }
                    finish(c + 1, vb);
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive_cluster(map_to_cta(smem_u32(&acc_empty_bar[acc]), 0));
            }
        }
        if (ep.direct_peers > 0) {
            __threadfence_system();  // stores into the other rank's copy are performed before the kernel completes
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before_sync();
    cluster_sync_all();  // the peer has stopped signalling into / reading from this CTA
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc_pair(tmem_base, Cfg::kTmemCols);
    }
}

// CTA-pair launch: 256 x BN tiles, two CTAs per tile.  NNB200_UNSUPPORTED when the device cannot
// co-schedule a single pair (the caller then uses the single-CTA form).
// Step of the per-tile K rotation (see k_rotation).  Default: 5 blocks per tile index where the
// weight has at most 4096 rows -- few column tiles, so many CTAs of a wave share each W tile
// (measured +3..10 % there, -2 % at 8192 rows); knob I8_K_ROTATE sets it, 0 = every tile starts
// at block 0.
inline int k_rotation_step(int n)
{
    const int kn = knob(NNB200_KNOB_I8_K_ROTATE);
    return kn >= 0 ? kn : (n <= 4096 ? 5 : 0);
}

template <int BN, int KIND, int SUB = 1, bool MC = false, int POSE = 0>
int launch_pair_variant(const I8Problem& p, const I8Epilogue& ep, int m, int n, int k, uint32_t a_fmt, int vec_ok,
                        const DeviceInfo& dev, cudaStream_t stream)
{
    static_assert(POSE == 0 || BN == 256, "an MN-major W half is one 128-column block");
    using Cfg = PairTileConfig<BN>;
    auto kernel = gemm_i8_umma_pair_kernel<BN, KIND, SUB, MC, false, POSE>;
    static std::once_flag once[kMaxDevices];
    static cudaError_t attr_err[kMaxDevices];
    static int max_pairs[kMaxDevices];
    std::call_once(once[dev.device], [&] {
        attr_err[dev.device] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
        max_pairs[dev.device] = 0;
        if (attr_err[dev.device] == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(static_cast<unsigned>(dev.sm_count & ~1));
            cfg.blockDim = dim3(num_threads(0));
            cfg.dynamicSmemBytes = Cfg::kSmemBytes;
            int count = 0;
            if (cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) == cudaSuccess) {
                max_pairs[dev.device] = count;
            }
        }
    });
    if (attr_err[dev.device] != cudaSuccess) {
        return NNB200_INTERNAL;
    }
    if (max_pairs[dev.device] < 1) {
        return NNB200_UNSUPPORTED;
    }
    CUtensorMap map_a, map_w;
    const bool map_a_ok =
        (POSE & 1) ? make_tma_2d(&map_a, p.a, 1, static_cast<uint64_t>(m), static_cast<uint64_t>(k),
                                 static_cast<uint64_t>(p.a_stride_k), kBlockM, kBlockKBytes)
                   : make_tma_2d(&map_a, p.a, 1, static_cast<uint64_t>(k), static_cast<uint64_t>(m),
                                 static_cast<uint64_t>(p.a_stride_m), kBlockKBytes, kBlockM);
    const bool map_w_ok =
        (POSE & 2) ? make_tma_2d(&map_w, p.w, 1, static_cast<uint64_t>(n), static_cast<uint64_t>(k),
                                 static_cast<uint64_t>(p.w_stride_k), 128, kBlockKBytes)
                   : make_tma_2d(&map_w, p.w, 1, static_cast<uint64_t>(k), static_cast<uint64_t>(n),
                                 static_cast<uint64_t>(p.w_stride_n), kBlockKBytes, BN / 2);
    if (!map_a_ok || !map_w_ok) {
        return NNB200_INTERNAL;
    }
    const int num_tiles = ((m + 2 * kBlockM - 1) / (2 * kBlockM)) * ((n + BN - 1) / BN);
    const int pairs = num_tiles < max_pairs[dev.device] ? num_tiles : max_pairs[dev.device];
    int group_m = static_cast<int>((40ll << 20) / (static_cast<int64_t>(2 * kBlockM) * (k > 0 ? k : 1)));
    group_m = group_m < 2 ? 2 : group_m;
    constexpr uint32_t major_bits = ((POSE & 1) ? kUmmaAMajorMN : 0u) | ((POSE & 2) ? kUmmaBMajorMN : 0u);
    const cudaError_t launched = launch_overlapping(kernel, dim3(static_cast<unsigned>(2 * pairs)), dim3(num_threads(0)), Cfg::kSmemBytes, stream, 1,
                                                    map_a, map_w, ep, m, n, k, umma_idesc(2, a_fmt, 1, 2 * kBlockM, BN) | major_bits, vec_ok, group_m, k_rotation_step(n), dev.error_word, ConvTile{});
    note_launch();
    return cuda_status(launched);
}

template <int BN, int SUB = 1, bool MC = false, int POSE = 0>
int launch_pair_bn(const I8Problem& p, const I8Epilogue& ep, int m, int n, int k, uint32_t a_fmt, int vec_ok,
                   const DeviceInfo& dev, cudaStream_t stream)
{
    switch (ep.out_kind) {
    case NNB200_OUT_S32: return launch_pair_variant<BN, NNB200_OUT_S32, SUB, MC, POSE>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream);
    case NNB200_OUT_S8: return launch_pair_variant<BN, NNB200_OUT_S8, SUB, MC, POSE>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream);
    case NNB200_OUT_U8: return launch_pair_variant<BN, NNB200_OUT_U8, SUB, MC, POSE>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream);
    case NNB200_OUT_F32: return launch_pair_variant<BN, NNB200_OUT_F32, SUB, MC, POSE>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream);
    case NNB200_OUT_F16: return launch_pair_variant<BN, NNB200_OUT_F16, SUB, MC, POSE>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream);
    default: return NNB200_UNSUPPORTED;
    }
}

template <int BN, int KIND, int PEERS>
int launch_variant(const CUtensorMap& map_a, const CUtensorMap& map_w, const I8Epilogue& ep, int m, int n, int k,
                   uint32_t idesc, int vec_ok, const DeviceInfo& dev, cudaStream_t stream)
{
    using Cfg = TileConfig<BN, PEERS, KIND>;
    auto kernel = gemm_i8_umma_kernel<BN, KIND, PEERS>;
    constexpr int kSmem = Cfg::kSmemBytes;
    PeerMaps maps;
    std::memset(&maps, 0, sizeof(maps));
    if constexpr (PEERS) {
        // Output windows as 2-D byte tensors [m][n] with the caller's pitch; 128 x 32 boxes.
        for (int d = 0; d <= ep.num_peers; ++d) {
            const void* base = d == 0 ? ep.out : ep.peer_out[d - 1];
            if (!make_tma_2d(&maps.m[d], base, 1, static_cast<uint64_t>(n), static_cast<uint64_t>(m),
                             static_cast<uint64_t>(ep.ldc), Cfg::kStageGroupCols, 32)) {
                return NNB200_INTERNAL;
            }
        }
    }
    static std::once_flag once[kMaxDevices];
    static cudaError_t attr_err[kMaxDevices];
    std::call_once(once[dev.device], [&] {
        attr_err[dev.device] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
    });
    if (attr_err[dev.device] != cudaSuccess) {
        return NNB200_INTERNAL;
    }
    const int num_tiles = ((m + kBlockM - 1) / kBlockM) * ((n + BN - 1) / BN);
    const int grid = num_tiles < dev.sm_count ? num_tiles : dev.sm_count;
    // Raster group: as many m-blocks as keep the group's band of A within about a third of L2
    // (126 MB on B200), so that W is read from DRAM once per group.
    int group_m = static_cast<int>((40ll << 20) / (static_cast<int64_t>(kBlockM) * (k > 0 ? k : 1)));
    group_m = group_m < 4 ? 4 : group_m;
    if (knob(NNB200_KNOB_GROUP_M) > 0) {
        group_m = knob(NNB200_KNOB_GROUP_M);
    }
    const cudaError_t launched = launch_overlapping(kernel, dim3(static_cast<unsigned>(grid)), dim3(tile_threads(KIND, PEERS)), kSmem, stream, 1,
                                                    map_a, map_w, maps, ep, m, n, k, idesc, vec_ok, group_m, k_rotation_step(n), dev.error_word, ConvTile{});
    note_launch();
    return cuda_status(launched);
}

template <int BN>
int launch_bn(int kind, const CUtensorMap& map_a, const CUtensorMap& map_w, const I8Epilogue& ep, int m, int n, int k,
              uint32_t idesc, int vec_ok, const DeviceInfo& dev, cudaStream_t stream)
{
    if (ep.num_peers > 0 || ep.mc_out != nullptr) {
        // Sharded write-back exists for the 8-bit destinations: 256- and 128-wide tiles, and --
        // multicast stores only, whose pieces need not be whole 128-byte boxes -- 224-wide ones.
        // knob I8_PEER_STAGING = 1 / 2 forces the staging depth (measurement aid).
        // One staging tile per warp and the fourth ring stage it leaves room for: measured faster than
        // two tiles and three stages at every size (per step, one / three / seven peers:
        // 0.380 -> 0.346, 0.262 -> 0.237 and 0.255 -> 0.238 ms).  Multicast stores leave the SM as
        // ordinary stores: one staging tile per warp is all they need.
        bool single = true;
        if (const int staging = knob(NNB200_KNOB_I8_PEER_STAGING); staging == 1 || staging == 2) {
            single = staging == 1;
        }
        if constexpr (BN == 256 || BN == 128) {
            if (kind == NNB200_OUT_S8) {
                return single
                           ? launch_variant<BN, NNB200_OUT_S8, 1>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream)
                           : launch_variant<BN, NNB200_OUT_S8, 2>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream);
            }
            if (kind == NNB200_OUT_U8) {
                return single
                           ? launch_variant<BN, NNB200_OUT_U8, 1>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream)
                           : launch_variant<BN, NNB200_OUT_U8, 2>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream);
            }
        }
        if constexpr (BN == 224) {
            if (ep.mc_out != nullptr && kind == NNB200_OUT_S8) {
                return launch_variant<BN, NNB200_OUT_S8, 1>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream);
            }
            if (ep.mc_out != nullptr && kind == NNB200_OUT_U8) {
                return launch_variant<BN, NNB200_OUT_U8, 1>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream);
            }
        }
        return NNB200_UNSUPPORTED;
    }
    switch (kind) {
    case NNB200_OUT_S32: return launch_variant<BN, NNB200_OUT_S32, 0>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream);
    case NNB200_OUT_S8: return launch_variant<BN, NNB200_OUT_S8, 0>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream);
    case NNB200_OUT_U8: return launch_variant<BN, NNB200_OUT_U8, 0>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream);
    case NNB200_OUT_F32: return launch_variant<BN, NNB200_OUT_F32, 0>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream);
    case NNB200_OUT_F16: return launch_variant<BN, NNB200_OUT_F16, 0>(map_a, map_w, ep, m, n, k, idesc, vec_ok, dev, stream);
    default: return NNB200_UNSUPPORTED;
    }
}

}  // namespace

namespace {

template <int BN, int KIND>
int launch_conv_variant(const CUtensorMap& map_a, const CUtensorMap& map_w, const I8Epilogue& ep, int m_tiles, int n,
                        int k, uint32_t idesc, int vec_ok, const ConvTile& conv, const DeviceInfo& dev,
                        cudaStream_t stream)
{
    using Cfg = TileConfig<BN, 0, KIND>;
    auto kernel = gemm_i8_umma_kernel<BN, KIND, 0, true>;
    static std::once_flag once[kMaxDevices];
    static cudaError_t attr_err[kMaxDevices];
    std::call_once(once[dev.device], [&] {
        attr_err[dev.device] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    });
    if (attr_err[dev.device] != cudaSuccess) {
        return NNB200_INTERNAL;
    }
    PeerMaps maps;
    std::memset(&maps, 0, sizeof(maps));
    const int num_tiles = m_tiles * ((n + BN - 1) / BN);
    const int grid = num_tiles < dev.sm_count ? num_tiles : dev.sm_count;
    int group_m = static_cast<int>((40ll << 20) / (static_cast<int64_t>(kBlockM) * (k > 0 ? k : 1)));
    group_m = group_m < 4 ? 4 : group_m;
    const cudaError_t launched = launch_overlapping(kernel, dim3(static_cast<unsigned>(grid)), dim3(tile_threads(KIND, 0)), Cfg::kSmemBytes, stream, 1,
                                                    map_a, map_w, maps, ep, m_tiles * kBlockM, n, k, idesc, vec_ok, group_m, k_rotation_step(n), dev.error_word, conv);
    note_launch();
    return cuda_status(launched);
}

// The CTA-pair form of the same: two patches per 256 x 256 tile, each CTA loading its own patch
// and half of the filter rows.  NNB200_UNSUPPORTED when the device cannot co-schedule a pair.
template <int KIND>
int launch_conv_pair_variant(const CUtensorMap& map_a, const CUtensorMap& map_w, const I8Epilogue& ep, int m_tiles, int n,
                             int k, uint32_t a_fmt, int vec_ok, const ConvTile& conv, const DeviceInfo& dev,
                             cudaStream_t stream)
{
    constexpr int BN = 256;
    using Cfg = PairTileConfig<BN>;
    auto kernel = gemm_i8_umma_pair_kernel<BN, KIND, 2, true, true>;
    static std::once_flag once[kMaxDevices];
    static cudaError_t attr_err[kMaxDevices];
    static int max_pairs[kMaxDevices];
    std::call_once(once[dev.device], [&] {
        attr_err[dev.device] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
        max_pairs[dev.device] = 0;
        if (attr_err[dev.device] == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(static_cast<unsigned>(dev.sm_count & ~1));
            cfg.blockDim = dim3(num_threads(0));
            cfg.dynamicSmemBytes = Cfg::kSmemBytes;
            int count = 0;
            if (cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) == cudaSuccess) {
                max_pairs[dev.device] = count;
            }
        }
    });
    if (attr_err[dev.device] != cudaSuccess) {
        return NNB200_INTERNAL;
    }
    if (max_pairs[dev.device] < 1) {
        return NNB200_UNSUPPORTED;
    }
    const int num_tiles = ((m_tiles + 1) / 2) * ((n + BN - 1) / BN);
    const int pairs = num_tiles < max_pairs[dev.device] ? num_tiles : max_pairs[dev.device];
    int group_m = static_cast<int>((40ll << 20) / (static_cast<int64_t>(2 * kBlockM) * (k > 0 ? k : 1)));
    group_m = group_m < 2 ? 2 : group_m;
    const cudaError_t launched = launch_overlapping(kernel, dim3(static_cast<unsigned>(2 * pairs)), dim3(num_threads(0)), Cfg::kSmemBytes, stream, 1,
                                                    map_a, map_w, ep, m_tiles * kBlockM, n, k, umma_idesc(2, a_fmt, 1, 2 * kBlockM, BN), vec_ok, group_m, k_rotation_step(n), dev.error_word, conv);
    note_launch();
    return cuda_status(launched);
}

int launch_conv_pair(const CUtensorMap& map_a, const CUtensorMap& map_w, const I8Epilogue& ep, int m_tiles, int n, int k,
                     uint32_t a_fmt, int vec_ok, const ConvTile& conv, const DeviceInfo& dev, cudaStream_t stream)
{
    switch (ep.out_kind) {
    case NNB200_OUT_S8: return launch_conv_pair_variant<NNB200_OUT_S8>(map_a, map_w, ep, m_tiles, n, k, a_fmt, vec_ok, conv, dev, stream);
    case NNB200_OUT_U8: return launch_conv_pair_variant<NNB200_OUT_U8>(map_a, map_w, ep, m_tiles, n, k, a_fmt, vec_ok, conv, dev, stream);
    case NNB200_OUT_F32: return launch_conv_pair_variant<NNB200_OUT_F32>(map_a, map_w, ep, m_tiles, n, k, a_fmt, vec_ok, conv, dev, stream);
    case NNB200_OUT_F16: return launch_conv_pair_variant<NNB200_OUT_F16>(map_a, map_w, ep, m_tiles, n, k, a_fmt, vec_ok, conv, dev, stream);
    default: return NNB200_UNSUPPORTED;
    }
}

template <int BN>
int launch_conv_bn(const CUtensorMap& map_a, const CUtensorMap& map_w, const I8Epilogue& ep, int m_tiles, int n, int k,
                   uint32_t idesc, int vec_ok, const ConvTile& conv, const DeviceInfo& dev, cudaStream_t stream)
{
    switch (ep.out_kind) {
    case NNB200_OUT_S8: return launch_conv_variant<BN, NNB200_OUT_S8>(map_a, map_w, ep, m_tiles, n, k, idesc, vec_ok, conv, dev, stream);
    case NNB200_OUT_U8: return launch_conv_variant<BN, NNB200_OUT_U8>(map_a, map_w, ep, m_tiles, n, k, idesc, vec_ok, conv, dev, stream);
    case NNB200_OUT_F32: return launch_conv_variant<BN, NNB200_OUT_F32>(map_a, map_w, ep, m_tiles, n, k, idesc, vec_ok, conv, dev, stream);
    case NNB200_OUT_F16: return launch_conv_variant<BN, NNB200_OUT_F16>(map_a, map_w, ep, m_tiles, n, k, idesc, vec_ok, conv, dev, stream);
    default: return NNB200_UNSUPPORTED;
    }
}

}  // namespace

// Implicit-GEMM convolution of one group: output pixels are tiled in patches of 128 (bh rows x
// bw columns of one image, bw a power of two chosen for the least padding), the activation is
// read through a 4-D tensor map {c, w, h, n} whose boxes are those patches shifted by the tap.
int launch_conv_i8_umma(const ConvUmmaArgs& c, const I8Epilogue& ep, const DeviceInfo& dev, cudaStream_t stream)
{
    ConvTile t;
    std::memset(&t, 0, sizeof(t));
    const int best = conv_patch_log2(c.oh, c.ow, nullptr);
    t.oh = c.oh; t.ow = c.ow; t.ih = c.ih; t.iw = c.iw;
    t.kh = c.kh; t.kw = c.kw; t.dh = c.dh; t.dw = c.dw; t.ph = c.ph; t.pw = c.pw;
    t.sh = c.sh; t.sw = c.sw;
    t.bw_log2 = best;
    t.bh = 128 >> best;
    t.tiles_w = (c.ow + (1 << best) - 1) >> best;
    t.tiles_h = (c.oh + t.bh - 1) / t.bh;
    t.c_base = c.c_base;
    t.kb_per_tap = c.icg / kBlockKBytes;
    t.zp_x = c.zp_x;
    t.wtap_ld = c.wtap_ld;
    t.nh = c.nh;
    t.nw = c.nw;
    for (int q = 0; q < 8; ++q) {
        t.mask_h[q] = c.mask_h[q];
        t.mask_w[q] = c.mask_w[q];
    }
    t.border = c.border;
    const int64_t m_tiles64 = static_cast<int64_t>(c.batch) * t.tiles_h * t.tiles_w;
    if (m_tiles64 > (INT32_MAX / kBlockM)) {
        return NNB200_UNSUPPORTED;
    }
    const int m_tiles = static_cast<int>(m_tiles64);
    t.m_tiles = m_tiles;
    const int n = c.ocg, k = c.k;
    int bn = 256;
    if (static_cast<int64_t>(m_tiles) * ((n + 255) / 256) < dev.sm_count || n <= 128) {
        bn = 128;
        if (static_cast<int64_t>(m_tiles) * ((n + 127) / 128) < dev.sm_count || n <= 64) {
            bn = 64;
        }
    }
    CUtensorMap map_a, map_w;
    if (!make_tma_nhwc_u8(&map_a, c.x, static_cast<uint64_t>(c.ic_total), static_cast<uint64_t>(c.iw),
                          static_cast<uint64_t>(c.ih), static_cast<uint64_t>(c.batch), static_cast<uint64_t>(c.in_w),
                          static_cast<uint64_t>(c.in_h), static_cast<uint64_t>(c.in_n), kBlockKBytes, 1u << best,
                          static_cast<uint32_t>(t.bh), static_cast<uint32_t>(c.sw), static_cast<uint32_t>(c.sh)) ||
        !make_tma_2d(&map_w, c.wt, 1, static_cast<uint64_t>(k), static_cast<uint64_t>(n), static_cast<uint64_t>(c.ldw),
                     kBlockKBytes, static_cast<uint32_t>(bn))) {
        return NNB200_INTERNAL;
    }
    const int elem = ep.out_kind == NNB200_OUT_S32 || ep.out_kind == NNB200_OUT_F32 ? 4 : (ep.out_kind == NNB200_OUT_F16 ? 2 : 1);
    const uint64_t pitch_bytes = static_cast<uint64_t>(ep.ldc) * elem;
    const int vec_ok = (((reinterpret_cast<uintptr_t>(ep.out) & 15u) == 0 && (pitch_bytes & 15u) == 0) ? 1 : 0) |
                       (((reinterpret_cast<uintptr_t>(ep.out) & 31u) == 0 && (pitch_bytes & 31u) == 0) ? 2 : 0);
    // CTA pairs (two patches per tile, half of the filter rows per CTA) where there are enough
    // pair tiles to fill the device: a single CTA's 128 x 256 tile asks its SM for more operand
    // bytes per clock than the L2 delivers to one SM, the pair's halves do not.  Knob I8_PAIR = 0
    // keeps the single-CTA form.
    if (bn == 256 && knob(NNB200_KNOB_I8_PAIR) != 0 &&
        static_cast<int64_t>((m_tiles + 1) / 2) * ((n + 255) / 256) >= dev.sm_count / 2) {
        CUtensorMap map_wh;
        if (!make_tma_2d(&map_wh, c.wt, 1, static_cast<uint64_t>(k), static_cast<uint64_t>(n), static_cast<uint64_t>(c.ldw),
                         kBlockKBytes, 128u)) {
            return NNB200_INTERNAL;
        }
        const int st = launch_conv_pair(map_a, map_wh, ep, m_tiles, n, k, c.a_unsigned ? 0u : 1u, vec_ok, t, dev, stream);
        if (st != NNB200_UNSUPPORTED) {
            return st;
        }
    }
    const uint32_t idesc = umma_idesc(2, c.a_unsigned ? 0u : 1u, 1, kBlockM, bn);
    switch (bn) {
    case 256: return launch_conv_bn<256>(map_a, map_w, ep, m_tiles, n, k, idesc, vec_ok, t, dev, stream);
    case 128: return launch_conv_bn<128>(map_a, map_w, ep, m_tiles, n, k, idesc, vec_ok, t, dev, stream);
    default: return launch_conv_bn<64>(map_a, map_w, ep, m_tiles, n, k, idesc, vec_ok, t, dev, stream);
    }
}

bool umma_i8_supported(const I8Problem& p)
{
    if (p.m < 1 || p.n < 1 || p.k < 1 || p.m > INT32_MAX || p.n > INT32_MAX || p.k > INT32_MAX) {
        return false;
    }
    // Each operand in either pose, as long as TMA can address it: the contiguous index has
    // stride 1, the other a pitch that is a multiple of 16 bytes and covers a row; 16-byte base.
    const auto aligned16 = [](uint64_t v) { return (v & 15u) == 0; };
    const auto operand_ok = [&](const void* base, int64_t stride_mn, int64_t stride_k, int64_t mn, int64_t k) {
        if (!aligned16(reinterpret_cast<uintptr_t>(base))) {
            return false;
        }
        if (stride_k == 1) {   // K-major: rows of k bytes
            return aligned16(static_cast<uint64_t>(stride_mn)) && stride_mn >= k;
        }
        return stride_mn == 1 && aligned16(static_cast<uint64_t>(stride_k)) && stride_k >= mn;   // MN-major
    };
    return operand_ok(p.a, p.a_stride_m, p.a_stride_k, p.m, p.k) && operand_ok(p.w, p.w_stride_n, p.w_stride_k, p.n, p.k);
}

int launch_gemm_i8_umma(const I8Problem& p, const I8Epilogue& ep_in, const DeviceInfo& dev, cudaStream_t stream)
{
    const int m = static_cast<int>(p.m);
    const int n = static_cast<int>(p.n);
    const int k = static_cast<int>(p.k);

    // A shard with ONE peer (two ranks) is bound by its GEMM, not by the link: it runs the
    // ordinary kernels -- the CTA-pair form where that applies -- whose epilogue stores each
    // 32-byte sector a second time, into the peer's copy, instead of the staged bulk stores of
    // the sharded form.  Needs whole 32-column chunks and 32-byte aligned destinations.
    I8Epilogue ep = ep_in;
    {
        const auto mis32 = [](const void* q) { return (reinterpret_cast<uintptr_t>(q) & 31u) != 0; };
        const uint64_t pitch = static_cast<uint64_t>(ep.ldc);   // 8-bit destinations: bytes
        if (ep.num_peers == 1 && ep.mc_out == nullptr && knob(NNB200_KNOB_I8_PEER_STAGING) <= 0 &&
            (ep.out_kind == NNB200_OUT_S8 || ep.out_kind == NNB200_OUT_U8) && p.a_stride_k == 1 && p.w_stride_k == 1 &&
            m >= 4 * kBlockM && k >= 2048 && n % 32 == 0 && pitch % 32 == 0 && !mis32(ep.out) && !mis32(ep.peer_out[0])) {
            ep.direct_peers = 1;
            ep.num_peers = 0;
        }
    }

    // Tile width.  When even the widest tile gives every SM work, take the width with the least
    // padded work over whole waves (waves x width; ties to the wider tile); narrow problems
    // trade arithmetic intensity for parallelism.
    const int num_m = (m + kBlockM - 1) / kBlockM;
    const bool sharded = ep.num_peers > 0 || ep.mc_out != nullptr;
    int bn = 256;
    if (static_cast<int64_t>(num_m) * ((n + 255) / 256) < dev.sm_count) {
        bn = 128;
        if (static_cast<int64_t>(num_m) * ((n + 127) / 128) < dev.sm_count && !sharded) {
            bn = 64;
        }
    } else if (sharded) {
        // A shard of a wide layer often ends a little past a whole number of waves (N / 8 = 3584:
        // 448 tiles of 256 columns on 148 SMs = 3.03 waves).  With multicast stores the 224-wide
        // tile is available: 512 tiles = 3.46 waves, an eighth less padded work.
        const auto padded_work = [&](int width) {
            const int64_t tiles = static_cast<int64_t>(num_m) * ((n + width - 1) / width);
            return (tiles + dev.sm_count - 1) / dev.sm_count * width;
        };
        if (ep.mc_out != nullptr && padded_work(224) * 100 < padded_work(256) * 92) {
            bn = 224;
        }
    } else {
        const auto padded_work = [&](int width) {
            const int64_t tiles = static_cast<int64_t>(num_m) * ((n + width - 1) / width);
            return (tiles + dev.sm_count - 1) / dev.sm_count * width;
        };
        int64_t best_cost = padded_work(256);
        for (const int cand : {224, 192}) {
            // A narrower tile moves more operand bytes per multiply-add (measured: about 8 % slower
            // per unit of work at 224): it has to save more than that.
            if (padded_work(cand) * 100 < best_cost * 92) {
                best_cost = padded_work(cand);
                bn = cand;
            }
        }
        // Single-wave form: when the problem needs a second, mostly empty wave, a tile wide enough
        // to give every CTA exactly one tile (two MMAs of BN / 2 columns per k-step) ends sooner.
        for (const int wide : {320, 384, 448, 512}) {
            const int64_t tiles = static_cast<int64_t>(num_m) * ((n + wide - 1) / wide);
            if (tiles <= dev.sm_count) {
                if (static_cast<int64_t>(wide) * 100 < best_cost * 92) {
                    best_cost = wide;
                    bn = wide;
                }
                break;  // wider ones only add padding
            }
        }
    }
    if (const int v = knob(NNB200_KNOB_I8_BN); v > 0) {  // measurement aid
        if (v == 512 || v == 448 || v == 384 || v == 320 || v == 256 || v == 224 || v == 192 || v == 128 || v == 64) {
            bn = v;
        }
    }
    // Operand poses: MN-major means the operand's M / N index is the contiguous one in memory
    // (MatMul's transpose_a, and its default [K, N] weights).  An MN-major W tile is brought in as
    // whole 128-column blocks, so its width is 256 or 128.
    const bool a_mn = p.a_stride_k != 1;
    const bool w_mn = p.w_stride_k != 1;
    if (w_mn && bn != 256 && bn != 128) {
        bn = (bn > 256 || static_cast<int64_t>(num_m) * ((n + 255) / 256) >= dev.sm_count) ? 256 : 128;
    }
    const uint32_t major_bits = (a_mn ? kUmmaAMajorMN : 0u) | (w_mn ? kUmmaBMajorMN : 0u);
    const auto idesc_of = [&](int mma_n) { return umma_idesc(2, p.a_unsigned ? 0u : 1u, 1, kBlockM, mma_n) | major_bits; };

    CUtensorMap map_a, map_w;
    const bool map_a_ok =
        a_mn ? make_tma_2d(&map_a, p.a, 1, static_cast<uint64_t>(m), static_cast<uint64_t>(k),
                           static_cast<uint64_t>(p.a_stride_k), kBlockM, kBlockKBytes)
             : make_tma_2d(&map_a, p.a, 1, static_cast<uint64_t>(k), static_cast<uint64_t>(m),
                           static_cast<uint64_t>(p.a_stride_m), kBlockKBytes, kBlockM);
    const bool map_w_ok =
        w_mn ? make_tma_2d(&map_w, p.w, 1, static_cast<uint64_t>(n), static_cast<uint64_t>(k),
                           static_cast<uint64_t>(p.w_stride_k), 128, kBlockKBytes)
             : make_tma_2d(&map_w, p.w, 1, static_cast<uint64_t>(k), static_cast<uint64_t>(n),
                           static_cast<uint64_t>(p.w_stride_n), kBlockKBytes, static_cast<uint32_t>(bn > 256 ? bn / 2 : bn));
    if (!map_a_ok || !map_w_ok) {
        return NNB200_INTERNAL;
    }

    // Destination vector stores need a 16-byte aligned base and row pitch.
    const int elem = (ep.out_kind == NNB200_OUT_S32 || ep.out_kind == NNB200_OUT_F32) ? 4
                     : (ep.out_kind == NNB200_OUT_F16)                                ? 2
                                                                                      : 1;
    // Destination vector stores: bit 0 = 16-byte aligned base and row pitch, bit 1 = 32-byte.
    const uint64_t pitch_bytes = static_cast<uint64_t>(ep.ldc) * static_cast<uint64_t>(elem);
    const int vec_ok = (((reinterpret_cast<uintptr_t>(ep.out) & 15u) == 0 && (pitch_bytes & 15u) == 0) ? 1 : 0) |
                       (((reinterpret_cast<uintptr_t>(ep.out) & 31u) == 0 && (pitch_bytes & 31u) == 0) ? 2 : 0) |
                       (a_mn ? 16 : 0) | (w_mn ? 32 : 0);   // bits 4-5: operand poses, read by the kernel

    const uint32_t a_fmt = p.a_unsigned ? 0u : 1u;

    // CTA-pair form from 256 rows up, with a K of 2048 or more (below that single CTAs are level or
    // ahead: 22.3 against 23.7 us at 4096 x 4096 x 1024, 35.6 against 37.4 at 8192 x 4096 x 1024) and at
    // least 24 tiles of 256 x 256.  CUDA-graph timings, single / pair: 512 x 4096 x 4096 (32 tiles)
    // 24.9 / 16.6 us, 256 x 8192 x 8192 (32) 45.3 / 26.1, 384 x 8192 x 4096 (64) 26.9 / 17.0, 512 x 4096 x 11008
    // (32) 58.3 / 31.9; with 16 tiles or fewer they are level or single CTAs ahead (256 x 4096 x 4096:
    // 14.9 / 16.3).  With more tiles than SM pairs, where the single-CTA form would pick a narrower
    // tile to fill its waves, the pairs' own waves must be at least three quarters full
    // (2048 x 8192 x 2048, 256 tiles on 74 pairs: 30.9 / 28.5; not 640 x 8192 x 4096, 96 tiles: 22.5 / 27.2;
    // not M = 512, N = 11008, 86 tiles: 22.3 / 27.3).
    // Knob I8_PAIR: 0 = never; 2 = the pair form whatever the shape, or an error; 1 / 3 = older
    // forms kept for comparison (one k-block per barrier slot; two k-blocks but one commit per
    // destination CTA), forced likewise.
    {
        const int pair_knob = knob(NNB200_KNOB_I8_PAIR);
        const int64_t pair_tiles = static_cast<int64_t>((m + 2 * kBlockM - 1) / (2 * kBlockM)) * ((n + 255) / 256);
        const bool forced = pair_knob >= 1 && pair_knob <= 3;   // 1, 2, 3: a pair form or an error
        const int64_t pairs = dev.sm_count / 2 > 0 ? dev.sm_count / 2 : 1;
        const bool pair_waves_full = pair_tiles * 4 >= ((pair_tiles + pairs - 1) / pairs) * pairs * 3;
        const bool mn = a_mn || w_mn;   // MN-major operands: the default pair form only (knob 1 / 3: K-major)
        if (forced && (sharded || (mn && pair_knob != 2))) {
            return NNB200_UNSUPPORTED;
        }
        if (pair_knob != 0 && !sharded &&
            (forced || (m >= 2 * kBlockM && k >= 2048 && pair_tiles >= 24 &&
                        (pair_tiles <= pairs || bn == 256 || pair_waves_full)))) {
            const int pose = (a_mn ? 1 : 0) | (w_mn ? 2 : 0);
            const int st = pair_knob == 1   ? launch_pair_bn<256, 1, false>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream)
                           : pair_knob == 3 ? launch_pair_bn<256, 2, false>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream)
                           : pose == 1      ? launch_pair_bn<256, 2, true, 1>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream)
                           : pose == 2      ? launch_pair_bn<256, 2, true, 2>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream)
                           : pose == 3      ? launch_pair_bn<256, 2, true, 3>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream)
                                            : launch_pair_bn<256, 2, true>(p, ep, m, n, k, a_fmt, vec_ok, dev, stream);
            if (st != NNB200_UNSUPPORTED || forced) {
                return st;
            }
        }
    }
    switch (bn) {
    case 512:
        return launch_bn<512>(ep.out_kind, map_a, map_w, ep, m, n, k, idesc_of(256), vec_ok,
                              dev, stream);
    case 448:
        return launch_bn<448>(ep.out_kind, map_a, map_w, ep, m, n, k, idesc_of(224), vec_ok,
                              dev, stream);
    case 384:
        return launch_bn<384>(ep.out_kind, map_a, map_w, ep, m, n, k, idesc_of(192), vec_ok,
                              dev, stream);
    case 320:
        return launch_bn<320>(ep.out_kind, map_a, map_w, ep, m, n, k, idesc_of(160), vec_ok,
                              dev, stream);
    case 256:
        return launch_bn<256>(ep.out_kind, map_a, map_w, ep, m, n, k, idesc_of(256), vec_ok,
                              dev, stream);
    case 224:
        return launch_bn<224>(ep.out_kind, map_a, map_w, ep, m, n, k, idesc_of(224), vec_ok,
                              dev, stream);
    case 192:
        return launch_bn<192>(ep.out_kind, map_a, map_w, ep, m, n, k, idesc_of(192), vec_ok,
                              dev, stream);
    case 128:
        return launch_bn<128>(ep.out_kind, map_a, map_w, ep, m, n, k, idesc_of(128), vec_ok,
                              dev, stream);
    default:
        return launch_bn<64>(ep.out_kind, map_a, map_w, ep, m, n, k, idesc_of(64), vec_ok,
                             dev, stream);
    }
}

}  // namespace nnb200
