// Q4_1 product for a few to 128 activation rows, weights as the 128-row operand in tensor memory:
//   out[M,N] = act(alpha * A[M,K] * dequant(W)[N,K]^T + bias), f32 accumulation.
//
// What the other forms pay here: the GEMM with the activations as the 128-row operand pads 16 rows
// to 128 and writes every expanded weight to shared memory and reads it back for the tensor core
// (4 bytes of shared-memory traffic per weight: at the HBM rate an SM decodes about 38 weights per
// clock, more than its shared memory carries); the warp-MMA GEMV walks the weights once per 8 rows
// and spends more instructions on fragments and MMAs than on decoding.
//
//   * A CTA owns a tile of up to 128 output channels; the channel is the row of the MMA and the lane
//     of tensor memory.  A thread decodes a unit (256 k) of ITS channel at a time -- nibbles to f16
//     with one rounding per weight, exactly as the other forms do -- and stores the pairs with
//     tcgen05.st into a tensor-memory stage, which tcgen05.mma reads as its A operand.  Expanded
//     weights never touch shared memory.
//   * The activations are the MMA's N operand (16 to 128 rows, padded with zeros by TMA), loaded a
//     unit at a time by one warp, 128-byte swizzle.
//   * The raw weight rows come in by 16-byte cp.async, each warp its own 32 channels, two units
//     ahead.  (TMA and bulk copies sustain about one short row per 17-24 clocks and SM.)
//   * Three warpgroups, a stage each, take the units in turn, so decoding, the stores to tensor
//     memory and the MMAs of different units overlap.
//   * Few channels: `split` CTAs (a cluster) share a tile's K and add up their accumulators
//     through distributed shared memory in a fixed order -- the result does not depend on timing.
//   * Launched with programmatic stream serialization: barriers and tensor memory are set up before
//     griddepcontrol.wait, and with NNB200_Q4_FLAG_OVERLAP_PREVIOUS the first units' weights fetched;
//     activations are read (by TMA, never through L1) and outputs written after it.
//   * f32 activations are given as two f16 rows each, high part and remainder; the epilogue adds the
//     two accumulator columns (see split_f32_to_f16_kernel).
//
// What bounds it: instruction issue.  16 rows of 28672 x 8192 issue 4.5 warp instructions for 32 weights
// (decoding, stores to tensor memory, copies, polls), 64 % of the issue slots of the active cycles, the
// integer pipe 52 %; the tensor pipe is busy 9 %, DRAM 34 % of peak.  What the MMAs cost is latency: 35 clocks
// each to issue (A = 128 x 16 from tensor memory, whatever the rows) and some hundred to drain for a commit.
// 16 rows of 14336 x 4096 take 16.0 us (50.5 before; the weights' HBM time is 5.7), 28672 x 8192 46.8
// (186), 4096 x 4096 9.0 (49.3).
//
// Every wait is bounded (see ptx.cuh).

#include <cstring>
#include <mutex>
#include <type_traits>

#include "internal.cuh"
#include "ptx.cuh"
#include "ptx_pair.cuh"
#include "q4_1_common.cuh"
#include "q4_1_rows_umma.cuh"

namespace nnb200 {

namespace {

constexpr int kTileRows = 128;                    // lanes of tensor memory
constexpr int kGroups = 3;                        // warpgroups that decode in turn, one stage each
constexpr int kWarps = kGroups * 4;
constexpr int kThreads = (kWarps + 2) * 32;
constexpr int kAccCols = 128;                     // accumulator columns = most activation rows
constexpr int kTmemCols = 512;
constexpr int kSlotK = 64;                        // k of one 128-byte swizzle row of activations
constexpr int kMaxSplit = 8;

// A unit is what a warpgroup decodes per turn: 8 blocks (256 k) of every row, or 4 when more than 64
// activation rows would make three stages of them too large for shared memory.
template <int BLOCKS>
struct RowsConfig {
    static constexpr int kUnitK = BLOCKS * kQ4BlockElems;
    static constexpr int kUnitBytes = BLOCKS * kQ4BlockBytes;     // 160 or 80 bytes of a row
    static constexpr int kWarpUnitBytes = 32 * kUnitBytes;
    static constexpr int kDepth = BLOCKS == 8 ? 2 : 4;            // units of raw rows on their way per warp
    static constexpr int kRawBytes = kWarps * kDepth * kWarpUnitBytes;   // 122 880 either way
    static constexpr int kUnitCols = kUnitK / 2;                  // tensor-memory columns: two f16 each
    static constexpr int kMaxRows = BLOCKS == 8 ? 64 : 128;
    static constexpr int kRingBytes = kGroups * kMaxRows * kUnitK * 2;   // 98 304 either way
    static constexpr int kBarrierBytes = (2 * kGroups + 2) * 8 + 16;
    static constexpr int kSmemBytes = 1024 + kRingBytes + kRawBytes + kBarrierBytes;
    static_assert(kAccCols * kTileRows * 4 <= kRawBytes, "partial sums reuse the raw buffers");
    static_assert(kAccCols + kGroups * kUnitCols <= kTmemCols, "tensor memory");
    static_assert(kSmemBytes <= 227 * 1024, "shared memory");
};

// D[tmem] (+)= A[tmem] * B[smem], issued by one thread.
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                            uint32_t accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// Warp-wide: 32 lanes x 16 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
          "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

__device__ __forceinline__ void tmem_st_wait()
{
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void tmem_ld_32x1(uint32_t taddr, uint32_t& v)
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(taddr) : "memory");
}

__device__ __forceinline__ float ld_shared_cluster_f32(uint32_t cluster_addr)
{
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
    return v;
}

// Asynchronous copy of N bytes, those past `src_bytes` as zeros.
template <int N>
__device__ __forceinline__ void cp_async(void* smem_dst, const void* gmem_src, uint32_t src_bytes)
{
    if constexpr (N == 16) {
        cp_async_16(smem_dst, gmem_src, src_bytes);
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(smem_u32(smem_dst)), "l"(gmem_src), "n"(N), "r"(src_bytes)
                     : "memory");
    }
}

// One block of a row, {d | m, four words of nibbles} -> its 32 weights as 16 f16 pairs in k order.
// A word's bytes carry k = 4wi .. 4wi+3 in their low and 16 + the same in their high nibbles:
// byte | 0x6400 = 1024 + q, (byte & 0xF0) | 0x5400 = 64 + q; the bias goes out exactly and d * q + m
// is rounded once.
__device__ __forceinline__ void decode_block(const uint32_t (&b)[5], uint32_t (&v)[16])
{
    const uint32_t d = __byte_perm(b[0], b[0], 0x1010);
    const uint32_t m = __byte_perm(b[0], b[0], 0x3232);
    const auto scale = [&](uint32_t biased, uint32_t bias) {
        uint32_t q, r;
        asm("sub.f16x2 %0, %1, %2;" : "=r"(q) : "r"(biased), "r"(bias));
        asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(q), "r"(d), "r"(m));
        return r;
    };
#pragma unroll
    for (int wi = 0; wi < 4; ++wi) {
        const uint32_t lo = b[1 + wi] & 0x0F0F0F0Fu;
        const uint32_t hi = b[1 + wi] & 0xF0F0F0F0u;
        v[2 * wi] = scale(__byte_perm(lo, 0x64646464u, 0x4140), 0x64006400u);
        v[2 * wi + 1] = scale(__byte_perm(lo, 0x64646464u, 0x4342), 0x64006400u);
        v[8 + 2 * wi] = scale(__byte_perm(hi, 0x54545454u, 0x4140), 0x54005400u);
        v[9 + 2 * wi] = scale(__byte_perm(hi, 0x54545454u, 0x4342), 0x54005400u);
    }
}

// hi_lo: activation row m is the MMA's rows 2 m and 2 m + 1; nb: the MMA's rows padded to a multiple
// of 16.  Clusters take the tiles in turn; with split > 1 each has one tile.
//
// One barrier pair per stage: "full" counts the four decoding warps of its group and the bytes of the
// unit's activations, "empty" one commit.  A commit interrupts the tensor pipe and costs the issuing
// thread some hundred cycles with its wait, so there are few: with a pair per 64 k (and barriers of
// their own for the activations) a call at 16 x 14336 x 4096 took 34.6 us, with one per 128 k 18.6, as
// here 16.0.  (Two issuing warps with an accumulator each: 17.8.)
//
// PIECE: bytes of one copy, the most (16, 8 or 4) that the weight rows' alignment allows.
template <bool OUT_F16, int BLOCKS, int PIECE>
__global__ void __launch_bounds__(kThreads, 1)
q4_1_rows_umma_kernel(const __grid_constant__ CUtensorMap map_a, const uint8_t* w,
                      const int64_t w_pitch_bytes, void* __restrict__ out, const int64_t ldc, const int m_total,
                      const int hi_lo, const int nb, const int n_total, const int k_total, const int tile_rows,
                      const int split, const FpEpilogue ep, const uint32_t idesc, int32_t* error_word, const int early)
{
    using Cfg = RowsConfig<BLOCKS>;
    constexpr int kUnitK = Cfg::kUnitK;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* ring = smem;
    uint8_t* raw = smem + Cfg::kRingBytes;
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(raw + Cfg::kRawBytes);
    uint64_t* empty_bar = full_bar + kGroups;
    uint64_t* acc_full = empty_bar + kGroups;
    uint64_t* acc_empty = acc_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = __shfl_sync(0xFFFFFFFFu, static_cast<int>(threadIdx.x >> 5), 0);   // warp-uniform to the compiler too
    const int lane = threadIdx.x & 31;
    const int rank = split > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
    const int cluster = static_cast<int>(blockIdx.x) / split;
    const int clusters = static_cast<int>(gridDim.x) / split;
    const int num_tiles = (n_total + tile_rows - 1) / tile_rows;
    // This CTA's units; the row's last unit of 256 k may hold 128.  K is padded to a multiple of 128:
    // blocks past a row's end are zeros in shared memory, activations past K zeros from TMA.
    const int k_pad = (k_total + 127) / 128 * 128;
    const int row_bytes = (k_total + kQ4BlockElems - 1) / kQ4BlockElems * kQ4BlockBytes;
    const int units_total = (k_pad + kUnitK - 1) / kUnitK;
    const int u0 = units_total * rank / split;
    const int units = units_total * (rank + 1) / split - u0;
    const int slab_bytes = nb * 128;               // 64 k of the activations
    const int stage_bytes = nb * kUnitK * 2;
    const auto slabs_of = [&](int u) { return min(kUnitK, k_pad - (u0 + u) * kUnitK) / kSlotK; };   // 4 or 2

    if (threadIdx.x == 0) {
        for (int g = 0; g < kGroups; ++g) {
            mbar_init(&full_bar[g], 5);   // four decoding warps and the producer's expect-tx
            mbar_init(&empty_bar[g], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, kWarps);
        *abort_flag = 0;
        mbar_init_fence();
    }
    if (warp == kWarps && lane == 0) {
        tma_prefetch_desc(&map_a);
    }

    // The decoding warps start their weight rows before the barriers exist: nothing but the weights
    // is touched.  Warp w of group g owns lanes 32 * (w % 4) and takes steps g, g + 3, ... of the
    // CTA's (tile, unit) sequence.
    const int group = warp >> 2;
    const int quarter = warp & 3;
    uint8_t* my_raw = raw + warp * (Cfg::kDepth * Cfg::kWarpUnitBytes);
    // The pieces of a unit's row, over the lanes: several rows at once, or several lanes' worth of one.
    constexpr int kPieces = Cfg::kUnitBytes / PIECE;
    constexpr int kRowsAtOnce = kPieces <= 32 ? 32 / kPieces : 1;
    const int copy_row = kPieces <= 32 ? lane / kPieces : 0;
    const int copy_piece = lane - copy_row * kPieces;
    int next_tile = cluster, next_u = group, next_buf = 0;   // of the next unit to copy
    const auto issue_unit = [&]() {
        while (next_u >= units) {
            next_u -= units;
            next_tile += clusters;
        }
        if (next_tile < num_tiles) {
            const int row0 = next_tile * tile_rows + quarter * 32;
            const int rows = min(min(32, tile_rows - quarter * 32), n_total - row0);
            const int64_t step = kRowsAtOnce * w_pitch_bytes;
#pragma unroll
            for (int p = copy_piece; p < kPieces; p += 32) {
                const int at = (u0 + next_u) * Cfg::kUnitBytes + p * PIECE;   // within the row
                const int bytes = max(0, min(PIECE, row_bytes - at));         // the rest of the piece becomes zeros
                const uint8_t* src = w + (row0 + copy_row) * w_pitch_bytes + (bytes > 0 ? at : 0);
                uint8_t* dst = my_raw + next_buf * Cfg::kWarpUnitBytes + copy_row * Cfg::kUnitBytes + p * PIECE;
                // A unit of half the k ends before the pieces do.
                const bool live = copy_row < kRowsAtOnce && p * PIECE < slabs_of(next_u) * (2 * kQ4BlockBytes);
#pragma unroll
                for (int i = 0; i * kRowsAtOnce < 32; ++i) {
                    if (live && copy_row + i * kRowsAtOnce < rows) {
                        cp_async<PIECE>(dst + i * (kRowsAtOnce * Cfg::kUnitBytes), src, static_cast<uint32_t>(bytes));
                    }
                    src += step;
                }
                if (kPieces <= 32) {
                    break;
                }
            }
        }
        cp_async_commit();   // one group a call, empty or not: the waits count groups
        next_u += kGroups;
        next_buf = next_buf + 1 == Cfg::kDepth ? 0 : next_buf + 1;
    };
    // Nothing but weights is touched before the previous kernel has completed, and those only where the
    // caller says that no kernel before this one writes them (early).
    if (warp < kWarps) {
        if (!early) {
            previous_kernel_done();
        }
#pragma unroll 1
        for (int s = 0; s < Cfg::kDepth; ++s) {
            issue_unit();
        }
    } else if (warp == kWarps + 1) {
        tmem_alloc(tmem_slot, kTmemCols);
        tmem_relinquish();
    }
    previous_kernel_done();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t a_col0 = tmem_base + kAccCols;

    if (warp == kWarps) {
        // ---------------- activations: TMA producer ----------------
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0, armed = 0, armed_phase = 0;
            bool ok = true;
            for (int tile = cluster; ok && tile < num_tiles; tile += clusters) {
                for (int u = 0; u < units; ++u) {
                    if (!mbar_wait(&empty_bar[stage], phase ^ 1u, abort_flag)) {
                        atomicCAS(error_word, 0, kErrProducerWait);
                        ok = false;
                        break;
                    }
                    const int slabs = slabs_of(u);
                    mbar_expect_tx(&full_bar[stage], static_cast<uint32_t>(slabs * slab_bytes));
                    for (int i = 0; i < slabs; ++i) {
                        tma_load_2d(ring + stage * stage_bytes + i * slab_bytes, &map_a, &full_bar[stage],
                                    (u0 + u) * kUnitK + i * kSlotK, 0);
                    }
                    armed |= 1u << stage;
                    armed_phase = (armed_phase & ~(1u << stage)) | (phase << stage);
                    if (++stage == kGroups) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
            if (!ok) {
                // Copies in flight land before the CTA exits (a stage whose decoding warps gave up
                // never completes: the wait is bounded and the copies are long done by then).
                const long long t0 = clock64();
                for (int s = 0; s < kGroups; ++s) {
                    while (((armed >> s) & 1u) && !mbar_try_wait(&full_bar[s], (armed_phase >> s) & 1u)) {
                        if (clock64() - t0 > kWaitLimitCycles / 64) {
                            break;
                        }
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == kWarps + 1) {
        // ---------------- MMA issuer ----------------
        // The whole warp walks the loop and one elected lane issues: addresses and descriptors are then
        // warp-uniform to the compiler, which is how the MMA takes its operands.  From a loop run by one
        // lane an MMA took 93 clocks to issue, 35 this way (the call 23.6 us, then 17.8).  The waits keep
        // it so (see mbar_wait_converged).
        const uint32_t d_tmem = warp_uniform(tmem_base);
        const uint64_t ring_desc = umma_desc_sw128_kmajor(smem_u32(ring));
        const uint64_t slab_step = static_cast<uint64_t>(slab_bytes >> 4);
        const int my_units = warp_uniform(units);
        uint32_t failed = 0;
        int stage = 0;
        uint32_t phase = 0, acc_phase = 1;
        for (int tile = warp_uniform(cluster); tile < num_tiles; tile += warp_uniform(clusters)) {
            mbar_wait_converged<kErrAccumWait>(acc_empty, acc_phase, abort_flag, failed);
            tc_fence_after_sync();
            acc_phase ^= 1u;
            uint32_t accumulate = 0;
            for (int u = 0; u < my_units; ++u) {
                mbar_wait_converged<kErrMmaWait>(&full_bar[stage], phase, abort_flag, failed);
                tc_fence_after_sync();
                const uint64_t b_desc = ring_desc + static_cast<uint64_t>((stage * stage_bytes) >> 4);
                const uint32_t a_tmem = d_tmem + static_cast<uint32_t>(kAccCols + stage * Cfg::kUnitCols);
                const int slabs = warp_uniform(slabs_of(u));
                if (elect_one()) {
#pragma unroll
                    for (int i = 0; i < kUnitK / kSlotK; ++i) {
                        if (i < slabs) {
#pragma unroll
                            for (int ks = 0; ks < kSlotK / 16; ++ks) {
                                umma_f16_ts(d_tmem, a_tmem + i * (kSlotK / 2) + ks * 8,
                                            b_desc + i * slab_step + static_cast<uint64_t>(ks * 2), idesc,
                                            (i > 0 || ks > 0) ? 1u : accumulate);
                            }
                        }
                    }
                    umma_commit(&empty_bar[stage]);
                }
                __syncwarp();
                accumulate = 1;
                if (++stage == kGroups) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            if (elect_one()) {
                umma_commit_unless(acc_full, failed);
            }
            __syncwarp();
        }
        let_next_kernel_start();
        if (const uint32_t code = warp_failure(failed); code != 0) {
            if (lane == 0) {
                atomicCAS(error_word, 0, static_cast<int32_t>(code));
            }
            umma_settle_after_failure();
        }
        __syncwarp();
    } else {
        // ---------------- decoding warps, then the epilogue of each tile ----------------
        const uint32_t lane_bits = static_cast<uint32_t>(quarter * 32) << 16;
        const int row = quarter * 32 + lane;
        float* part = reinterpret_cast<float*>(raw) + row;   // [accumulator column][128 rows]
        int u = group, buf = 0;
        uint32_t phase = 1, acc_phase = 0;
        bool ok = true;
        for (int tile = cluster; ok && tile < num_tiles; tile += clusters) {
            for (; u < units; u += kGroups) {
                const int halves = slabs_of(u) / 2;   // 4 blocks, 128 k each
                cp_async_wait_group<Cfg::kDepth - 1>();
                __syncwarp();   // every lane's pieces have landed
                const uint4* mine = reinterpret_cast<const uint4*>(my_raw + buf * Cfg::kWarpUnitBytes + lane * Cfg::kUnitBytes);
                buf = buf + 1 == Cfg::kDepth ? 0 : buf + 1;
                const uint32_t st_col = a_col0 + lane_bits + static_cast<uint32_t>(group * Cfg::kUnitCols);
                // The stage is free once the MMAs of the group's previous unit have read it.
                if (!mbar_wait_warp(&empty_bar[group], phase, abort_flag)) {
                    if (lane == 0) {
                        atomicCAS(error_word, 0, kErrDequantWait);
                    }
                    ok = false;
                    break;
                }
                phase ^= 1u;
                tc_fence_after_sync();
#pragma unroll
                for (int h = 0; h < BLOCKS / 4; ++h) {
                    if (h < halves) {
                        uint4 q[5];
#pragma unroll
                        for (int j = 0; j < 5; ++j) {
                            q[j] = mine[5 * h + j];
                        }
                        const uint32_t words[20] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w, q[2].x, q[2].y,
                                                    q[2].z, q[2].w, q[3].x, q[3].y, q[3].z, q[3].w, q[4].x, q[4].y, q[4].z, q[4].w};
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            const uint32_t blk[5] = {words[5 * b], words[5 * b + 1], words[5 * b + 2], words[5 * b + 3], words[5 * b + 4]};
                            uint32_t v[16];
                            decode_block(blk, v);
                            tmem_st_32x16(st_col + static_cast<uint32_t>((h * 4 + b) * 16), v);
                        }
                    }
                }
                tmem_st_wait();
                tc_fence_before_sync();
                __syncwarp();   // every lane has stored its weights and read its row
                if (lane == 0) {
                    mbar_arrive(&full_bar[group]);
                }
                issue_unit();   // refills the buffer just read, while the MMAs run
            }
            if (!ok) {
                break;
            }
            u -= units;
            if (!mbar_wait_warp(acc_full, acc_phase, abort_flag)) {
                if (lane == 0) {
                    atomicCAS(error_word, 0, kErrEpilogueWait);
                }
                ok = false;
                break;
            }
            acc_phase ^= 1u;
            tc_fence_after_sync();
            const int n = tile * tile_rows + row;
            const bool row_ok = row < tile_rows && n < n_total;
            const int cols = m_total << hi_lo;
            const uint32_t acc_row = tmem_base + lane_bits;
            const auto store = [&](int m, float x) {
                if constexpr (OUT_F16) {
                    static_cast<__half*>(out)[m * ldc + n] = __float2half_rn(x);
                } else {
                    static_cast<float*>(out)[m * ldc + n] = x;
                }
            };
            if (split == 1 && ep.activation != NNB200_ACT_NONE && ep.activation != NNB200_ACT_RELU) {
                // One copy of the activation's code (unrolled, fetching it cold cost more than the
                // arithmetic): a row at a time, the next one's sums on their way.
                const int step = kGroups << hi_lo;
                uint32_t hi = 0, lo = 0;
                int c = group << hi_lo;
                if (c < cols) {
                    tmem_ld_32x1(acc_row + static_cast<uint32_t>(c), hi);
                    if (hi_lo) {
                        tmem_ld_32x1(acc_row + static_cast<uint32_t>(c + 1), lo);
                    }
                }
#pragma unroll 1
                for (; c < cols; c += step) {
                    tmem_ld_wait();
                    const float x = __uint_as_float(hi) + __uint_as_float(lo);
                    if (c + step < cols) {
                        tmem_ld_32x1(acc_row + static_cast<uint32_t>(c + step), hi);
                        if (hi_lo) {
                            tmem_ld_32x1(acc_row + static_cast<uint32_t>(c + step + 1), lo);
                        }
                    }
                    if (row_ok) {
                        store(c >> hi_lo, fp_epilogue_value<OUT_F16>(ep, x, n));
                    }
                }
            } else {
                // 16 columns at a time, the groups in turn.
                float bias = -0.0f;   // x + -0.0f is x for every x
                if (ep.bias != nullptr && row_ok) {
                    bias = OUT_F16 ? __half2float(static_cast<const __half*>(ep.bias)[n]) : static_cast<const float*>(ep.bias)[n];
                }
#pragma unroll 1
                for (int c = group * 16; c < cols; c += kGroups * 16) {
                    uint32_t v[16];
                    tmem_ld_32x16(acc_row + static_cast<uint32_t>(c), v);
                    tmem_ld_wait();
                    if (split > 1) {
                        // One tile per cluster: nothing is left to read in the raw buffers (acc_full
                        // reports MMAs that came after every read of them).
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            part[(c + j) * kTileRows] = __uint_as_float(v[j]);
                        }
                        continue;
                    }
                    if (hi_lo) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            v[j] = __float_as_uint(__uint_as_float(v[2 * j]) + __uint_as_float(v[2 * j + 1]));
                        }
                    }
                    const int m0 = c >> hi_lo;
                    const int count = row_ok ? min(16 >> hi_lo, m_total - m0) : 0;
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (j < count) {
                            float x = __fadd_rn(__fmul_rn(__uint_as_float(v[j]), ep.alpha), bias);
                            x = fminf(fmaxf(x, ep.min_clip), ep.max_clip);
                            store(m0 + j, ep.activation == NNB200_ACT_RELU ? fmaxf(x, 0.0f) : x);
                        }
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(acc_empty);
            }
        }
        cp_async_wait_group<0>();
    }

    if (split > 1) {
        // Each CTA of the cluster finishes every split-th activation row of the tile.
        cluster_sync_all();
        if (warp < kWarps) {
            const int row = quarter * 32 + lane;
            const int n = cluster * tile_rows + row;
            if (row < tile_rows && n < n_total) {
                const uint32_t base = smem_u32(raw) + static_cast<uint32_t>(row * 4);
#pragma unroll 1
                for (int m = rank + split * group; m < m_total; m += split * kGroups) {
                    const uint32_t at = base + static_cast<uint32_t>((m << hi_lo) * kTileRows * 4);
                    float hi[kMaxSplit], lo[kMaxSplit];
#pragma unroll
                    for (int s = 0; s < kMaxSplit; ++s) {
                        hi[s] = lo[s] = 0.0f;
                        if (s < split) {
                            const uint32_t there = map_to_cta(at, static_cast<uint32_t>(s));
                            hi[s] = ld_shared_cluster_f32(there);
                            lo[s] = hi_lo ? ld_shared_cluster_f32(there + kTileRows * 4) : 0.0f;
                        }
                    }
                    float x = hi[0], y = lo[0];
#pragma unroll
                    for (int s = 1; s < kMaxSplit; ++s) {
                        x += hi[s];   // + 0.0f past the last part
                        y += lo[s];
                    }
                    x = fp_epilogue_value<OUT_F16>(ep, x + y, n);
                    if constexpr (OUT_F16) {
                        static_cast<__half*>(out)[m * ldc + n] = __float2half_rn(x);
                    } else {
                        static_cast<float*>(out)[m * ldc + n] = x;
                    }
                }
            }
        }
        cluster_sync_all();   // nobody leaves while its partial sums may still be read
    }

    // ---------------- teardown ----------------
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kWarps + 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// `split`: the most CTAs that may share a tile.
template <bool OUT_F16, int BLOCKS, int PIECE>
int launch_variant(const CUtensorMap& map_a, const Q4RowsCall& c, int nb, int tile_rows, int split, int tiles,
                   const FpEpilogue& ep, const DeviceInfo& dev, cudaStream_t stream)
{
    using Cfg = RowsConfig<BLOCKS>;
    auto kernel = q4_1_rows_umma_kernel<OUT_F16, BLOCKS, PIECE>;
    static std::once_flag once[kMaxDevices];
    static cudaError_t attr_err[kMaxDevices];
    static int resident[kMaxDevices][kMaxSplit + 1];   // clusters of that many CTAs the device holds at once
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    std::call_once(once[dev.device], [&] {
        attr_err[dev.device] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
        for (int s = 2; s <= kMaxSplit && attr_err[dev.device] == cudaSuccess; ++s) {
            attr[0].val.clusterDim.x = static_cast<unsigned>(s);
            cfg.gridDim = dim3(static_cast<unsigned>(dev.sm_count / s * s));
            int count = 0;
            if (cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) == cudaSuccess) {
                resident[dev.device][s] = count;
            } else {
                (void)cudaGetLastError();   // no clusters of that many: the launch takes a smaller one
            }
        }
    });
    if (attr_err[dev.device] != cudaSuccess) {
        return NNB200_INTERNAL;
    }
    // Clusters live within a group of SMs, so fewer of them fit than the SMs would hold: sixteen of eight do
    // not, and a second turn for the last ones costs more than all (2048 channels, K = 4096: 4 f32 rows 14.3 ->
    // 9.6 us; K = 1024: 128 f16 rows 17.5 -> 10.5).
    while (split > 1 && resident[dev.device][split] < tiles) {
        --split;
    }
    const int ctas = split > 1 ? tiles * split : (tiles < dev.sm_count ? tiles : dev.sm_count);
    attr[0].val.clusterDim.x = static_cast<unsigned>(split);
    cfg.gridDim = dim3(static_cast<unsigned>(ctas));
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, map_a, static_cast<const uint8_t*>(c.q->w_blocks),
                                             c.q->ldw_blocks * kQ4BlockBytes, c.q->out, c.q->ldc, static_cast<int>(c.q->m),
                                             c.hi_lo ? 1 : 0, nb, static_cast<int>(c.q->n), static_cast<int>(c.q->k), tile_rows,
                                             split, ep, umma_idesc(1, 0, 0, kTileRows, static_cast<uint32_t>(nb)), dev.error_word,
                                             (c.q->flags & NNB200_Q4_FLAG_OVERLAP_PREVIOUS) != 0 ? 1 : 0);
    note_launch();
    return cuda_status(e);
}

}  // namespace

bool q4_1_rows_umma_supported(const nnb200_q4_1_args& q)
{
    // Raw weight rows (4-byte aligned by the format), activations addressable by TMA; f32
    // activations come as a scratch copy that always is.
    const int64_t b_rows = q.a_f16 != 0 ? q.m : 2 * q.m;
    const bool a_ok = q.a_f16 == 0 || ((reinterpret_cast<uintptr_t>(q.a) & 15u) == 0 && (q.lda % 8) == 0);
    return a_ok && q.m >= 1 && b_rows <= kAccCols && q.n >= 1 && q.n <= INT32_MAX / 2 && q.k >= 1 && q.k <= INT32_MAX / 2 &&
           q.w_dm == nullptr && (reinterpret_cast<uintptr_t>(q.w_blocks) & 3u) == 0;
}

int launch_q4_1_rows_umma(const Q4RowsCall& c, const DeviceInfo& dev, cudaStream_t stream)
{
    const nnb200_q4_1_args& q = *c.q;
    FpEpilogue ep;
    ep.alpha = q.alpha;
    ep.bias = q.bias;
    ep.activation = q.activation;
    ep.act_alpha = q.act_alpha;
    ep.act_beta = q.act_beta;
    ep.min_clip = q.min_clip;
    ep.max_clip = q.max_clip;

    const int b_rows = static_cast<int>(c.hi_lo ? 2 * q.m : q.m);
    const int nb = (b_rows + 15) / 16 * 16;
    const int n = static_cast<int>(q.n);
    const bool wide = nb > RowsConfig<8>::kMaxRows;   // units of 128 k instead of 256
    const int unit_k = wide ? RowsConfig<4>::kUnitK : RowsConfig<8>::kUnitK;
    const int units = static_cast<int>(((q.k + 127) / 128 * 128 + unit_k - 1) / unit_k);
    // Every SM gets the same share of the channels: with at least half as many 128-channel tiles as
    // SMs, whole waves of equal, narrower tiles (a lane without a channel costs nothing that is
    // scarce: the weight stream is); below that, clusters that share K.
    const int tiles128 = (n + kTileRows - 1) / kTileRows;
    int split = 1, tiles = tiles128;
    if (tiles128 * 2 > dev.sm_count) {
        tiles = (tiles128 + dev.sm_count - 1) / dev.sm_count * dev.sm_count;
    } else {
        split = dev.sm_count / tiles128;
        split = split > kMaxSplit ? kMaxSplit : split;
        split = split > units ? units : split;
    }
    int tile_rows = (n + tiles - 1) / tiles;
    tile_rows = tile_rows > kTileRows ? kTileRows : tile_rows;
    tiles = (n + tile_rows - 1) / tile_rows;

    CUtensorMap map_a;
    if (!make_tma_2d(&map_a, c.a, 2, static_cast<uint64_t>(q.k), static_cast<uint64_t>(b_rows),
                     static_cast<uint64_t>(c.lda) * 2, kSlotK, static_cast<uint32_t>(nb))) {
        return NNB200_INTERNAL;
    }
    const uint64_t row_bits = reinterpret_cast<uintptr_t>(q.w_blocks) | static_cast<uint64_t>(q.ldw_blocks * kQ4BlockBytes);
    const auto launch = [&](auto piece) {
        constexpr int P = decltype(piece)::value;
        if (wide) {
            return q.out_f16 ? launch_variant<true, 4, P>(map_a, c, nb, tile_rows, split, tiles, ep, dev, stream)
                             : launch_variant<false, 4, P>(map_a, c, nb, tile_rows, split, tiles, ep, dev, stream);
        }
        return q.out_f16 ? launch_variant<true, 8, P>(map_a, c, nb, tile_rows, split, tiles, ep, dev, stream)
                         : launch_variant<false, 8, P>(map_a, c, nb, tile_rows, split, tiles, ep, dev, stream);
    };
    if ((row_bits & 15u) == 0) {
        return launch(std::integral_constant<int, 16>{});
    }
    return (row_bits & 7u) == 0 ? launch(std::integral_constant<int, 8>{}) : launch(std::integral_constant<int, 4>{});
}

}  // namespace nnb200
