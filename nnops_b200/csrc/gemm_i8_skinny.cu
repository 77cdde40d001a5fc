// int8 GEMM for a handful of activation rows (up to 128: decode, batched decode, short prefills).
//
// With so few rows the whole cost is streaming W once, and the square-tile engine
// (gemm_i8_umma.cu) is a poor fit: it pads the activations to a 128-row MMA operand, re-reads
// that mostly empty tile for every 256 channels and, on mid-sized layers, has fewer tiles than
// the GPU has SMs.  Here the roles of the operands are swapped:
//
//   * the WEIGHTS are the 128-row operand of tcgen05.mma (M = 128 channels per tile), the
//     activations its N operand, padded only to MP = 32 / 64 / 128 rows;
//   * one tile = 128 channels x all activation rows: a stage is 16 KB of weights plus MP x 128
//     bytes of activations, so nearly all ring traffic is the weight stream itself, and N / 128
//     tiles keep more SMs busy than N / 256;
//   * the accumulator comes out transposed (TMEM lane = channel, column = activation row):
//     a thread owns ONE channel, loads that channel's scale / bias / zero point / row sum once
//     per tile into registers, and for each activation row the warp stores 32 consecutive
//     channels of that output row.
//
// Same pipeline skeleton as the square engine (TMA warp, MMA warp, epilogue warps, two TMEM
// accumulators, bounded waits) except that each accumulator has its own four epilogue warps;
// same epilogue arithmetic (epilogue.cuh): results are bit-identical to every other int8 engine.
//
// What bounds it: the weight stream once several hundred KB a CTA are on their way (28672 x 8192, 24 rows:
// 41.7 us = 0.89 of measured HBM); below that the start -- 0.6 us to the first load, 2 us to the first weights
// with every SM asking at once -- and the tail.  A K block of 128 bytes takes the issuing warps 200 to 250 cycles
// (525 while their waits branched, see mbar_wait_converged): 24 rows of 11008 x 4096 15.6 -> 10.8 us, 64 rows
// 18.8 -> 11.7, 128 rows 24.8 -> 14.0.
//
// Tiles need not be 128 channels high: without shared K a layer of several waves of tiles is cut into
// equal ones (N = 28672 on 148 SMs: 296 tiles of 97 channels instead of 224 of 128), so that every SM
// streams the same bytes; the rows of the MMA past a tile's channels hold whatever the ring held
// before, and nobody reads their accumulators.
//
// Work split.  The unit of work is one 128-byte K block of one tile; tile t owns units
// [t * num_kb, (t + 1) * num_kb).  Every CTA takes one contiguous range of units:
//   * with so few tiles that two or more CTAs a tile find an SM each: clusters of up to eight CTAs share a
//     tile's K; their sums meet through distributed shared memory, each CTA finishing its share of the
//     rows (4096 x 4096, 24 rows: 15.3 us with whole tiles, 17.4 on the square engine -> 6.9);
//   * whole tiles only (CTA c gets an equal run of them) when no scratch is given;
//   * an equal share of ALL units (CTA c gets [c U / G, (c + 1) U / G)) when the caller gave
//     scratch: a range then starts and ends in the middle of tiles, so that every SM streams
//     the same number of weight bytes whatever N / 128 is (224 tiles on 148 SMs would otherwise
//     run as two waves, the second half empty).  A CTA that holds only part of a tile's K range
//     writes its int32 partial sums to its own slot of the scratch and counts itself in on the
//     tile's counter; whichever warp counts in last adds the other parts to its own and runs
//     the epilogue.  Nobody waits for anybody, and integer addition makes the result
//     independent of who came last.  The protocol runs per warp (a warp owns 32 channels of the
//     tile in every CTA), so it needs no CTA-wide barrier.

#include <atomic>
#include <chrono>
#include <cstdlib>
#include <mutex>
#include <type_traits>

#include "internal.cuh"
#include "ptx.cuh"
#include "ptx_pair.cuh"

namespace nnb200 {

namespace {

constexpr int kBlockN = 128;       // channels per tile = rows of the MMA's 128-row operand
constexpr int kBlockKBytes = 128;  // one 128-byte swizzle row of K per stage
constexpr int kUmmaK = 32;
// TMA warp, MMA warp and two groups of four epilogue warps.  Group g drains accumulator g, i.e.
// every second piece of the CTA's range, so the drains (and, with shared K, the exchanges of
// partial sums, each a chain of L2 round trips) of consecutive pieces run side by side.
constexpr int kNumThreads = 320;
constexpr int kEpilogueThreads = 128;  // per group
constexpr int kMaxParts = 8;           // CTAs of a cluster that share a tile's K

template <int MP>
struct SkinnyConfig {
    static constexpr int kWTileBytes = kBlockN * kBlockKBytes;  // 16 KB
    static constexpr int kATileBytes = MP * kBlockKBytes;       // 4 / 8 / 16 KB
    static constexpr int kStageBytes = kWTileBytes + kATileBytes;
    static constexpr int kStages = (192 * 1024) / kStageBytes > 10 ? 10 : (192 * 1024) / kStageBytes;
    static constexpr int kTmemCols = 2 * MP < 32 ? 32 : 2 * MP;  // two accumulators of MP columns
    static constexpr int kRowTerms = 136;                         // I8RowTerms of up to 128 activation rows, groups of rows read past the last
    static constexpr int kRowTermBytes = kRowTerms * 16;
    static constexpr int kBarrierBytes = (2 * kStages + 4) * 8 + 16;
    static constexpr int kSmemBytes = 1024 + kStages * kStageBytes + kRowTermBytes + kBarrierBytes;
};

// First unit of CTA c's range (c = G gives the end of the last range).  The launcher keeps the number of
// units below 2^31.
__device__ __forceinline__ int range_begin(int c, int grid, int num_tiles, int num_kb)
{
    // floor(c * total / grid) without a 64-bit division (some hundred cycles each at the kernel's start).
    const int total = num_tiles * num_kb;
    const int q = total / grid, r = total - q * grid;
    return c * q + static_cast<int>(static_cast<unsigned>(c) * static_cast<unsigned>(r) / static_cast<unsigned>(grid));
}

// The CTA whose range contains unit u under the equal-share split.
__device__ __forceinline__ int cta_of_unit(int64_t u, int grid, int64_t total_units)
{
    return static_cast<int>(((u + 1) * grid - 1) / total_units);
}

// Bytes of the per-tile, per-warp arrival words at the head of the split scratch.
__host__ __device__ inline size_t split_counter_bytes(int num_tiles)
{
    return (static_cast<size_t>(num_tiles) * 4 * sizeof(unsigned long long) + 255) & ~size_t(255);
}

// One piece of a CTA's range: K blocks [kb0, kb1) of `tile`.
struct Segment {
    int tile, kb0, kb1;
};

// A CTA's range [u_begin, u_end) cut at tile boundaries, in the order it is worked through:
// the part of a tile that somebody else started (head), the part of a tile that somebody else
// finishes (tail), then the whole tiles.  Parts go first so that they are published early and
// the exchange with the neighbours hides behind the whole tiles that follow.
struct SegmentList {
    int head0, head1, tail0, tail1;
    int tile0, tile1;
    int num_kb;

    __device__ __forceinline__ SegmentList(int u_begin, int u_end, int nkb) : num_kb(nkb)
    {
        const int first_full = (u_begin + nkb - 1) / nkb * nkb;
        const int last_full_end = u_end / nkb * nkb;
        head0 = u_begin;
        head1 = first_full < u_end ? first_full : u_end;
        if (last_full_end >= first_full && last_full_end < u_end) {
            tail0 = last_full_end;
            tail1 = u_end;
        } else {
            tail0 = tail1 = 0;
        }
        tile0 = first_full / nkb;
        tile1 = last_full_end > first_full ? last_full_end / nkb : tile0;
    }
    // Whole tiles [t0, t1); no division at the kernel's start.
    struct Whole {
        int t0, t1;
    };
    __device__ __forceinline__ SegmentList(Whole w, int nkb) : num_kb(nkb)
    {
        head0 = head1 = tail0 = tail1 = 0;
        tile0 = w.t0;
        tile1 = w.t1;
    }
    __device__ __forceinline__ int count() const
    {
        return (head1 > head0 ? 1 : 0) + (tail1 > tail0 ? 1 : 0) + (tile1 - tile0);
    }
    __device__ __forceinline__ Segment at(int i) const
    {
        Segment s;
        if (head1 > head0) {
            if (i == 0) {
                s.tile = head0 / num_kb;
                s.kb0 = head0 - s.tile * num_kb;
                s.kb1 = s.kb0 + (head1 - head0);
                return s;
            }
            --i;
        }
        if (tail1 > tail0) {
            if (i == 0) {
                s.tile = tail0 / num_kb;
                s.kb0 = 0;
                s.kb1 = tail1 - tail0;
                return s;
            }
            --i;
        }
        s.tile = tile0 + i;
        s.kb0 = 0;
        s.kb1 = num_kb;
        return s;
    }
    // For loops that issue MMAs or copies: warp-uniform to the compiler as well.
    __device__ __forceinline__ Segment uniform_at(int i) const
    {
        Segment s = at(i);
        s.tile = warp_uniform(s.tile);
        s.kb0 = warp_uniform(s.kb0);
        s.kb1 = warp_uniform(s.kb1);
        return s;
    }
};

// Arrival words.  The scratch arrives with arbitrary contents and nothing clears it: a word is
// (call tag << 8) | count, the tag unique to this launch, and a word carrying any other tag
// counts as zero.  The warp that finishes a tile writes (tag << 8) | 0 back, so that a replay of
// a captured launch -- same tag -- starts from zero as well.
__device__ __forceinline__ unsigned long long ld_acquire_gpu_u64(const unsigned long long* p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ int arrivals_of(unsigned long long word, unsigned long long tag)
{
    return (word >> 8) == tag ? static_cast<int>(word & 0xFFu) : 0;
}

// Count this part in, starting from the word as last seen; returns how many parts had arrived
// before it (-1 if the bounded retry ran out).
__device__ __forceinline__ int arrive(unsigned long long* p, unsigned long long tag, unsigned long long old)
{
    for (int tries = 0; tries < 1024; ++tries) {
        const int before = arrivals_of(old, tag);
        const unsigned long long prev = atomicCAS(p, old, (tag << 8) | static_cast<unsigned long long>(before + 1));
        if (prev == old) {
            return before;
        }
        old = prev;
    }
    return -1;
}

// Sum over the other CTAs' published parts of one tile, rows [row0, row0 + 32) of this thread's
// channel.  All loads of a part are issued before any is used: one L2 round trip per part.
__device__ __forceinline__ void collect_parts(int32_t (&sum)[32], const int32_t* split_slots, size_t slot_elems, int ch,
                                              int first_cta, int last_cta, int self, int row0, int m_total)
{
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        sum[j] = 0;
    }
    for (int other = first_cta; other <= last_cta; ++other) {
        if (other == self) {
            continue;
        }
        const int32_t* theirs = split_slots + (2 * static_cast<size_t>(other) + (other == first_cta ? 1u : 0u)) * slot_elems + ch;
        int32_t part[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            part[j] = (row0 + j < m_total) ? __ldcg(theirs + static_cast<size_t>(row0 + j) * kBlockN) : 0;
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            sum[j] += part[j];
        }
    }
}

// One channel's epilogue terms, held by the thread that finishes its sums.
struct ChannelTerms {
    int32_t zpw, rw, bias_i;
    float s_w, bias_f;
};

template <int KIND>
__device__ __forceinline__ ChannelTerms channel_terms(const I8Epilogue& ep, int64_t n, bool n_ok)
{
    ChannelTerms c;
    c.zpw = (n_ok && ep.zp_w != nullptr) ? ep.zp_w[n] : ep.zp_w_scalar;
    c.rw = (n_ok && ep.compensate && ep.r_w != nullptr) ? ep.r_w[n] : 0;
    c.s_w = (n_ok && ep.scale_w != nullptr) ? ep.scale_w[n] : ep.scale_w_scalar;
    c.bias_i = 0;
    c.bias_f = 0.0f;
    if (n_ok && ep.bias != nullptr) {
        if constexpr (KIND <= NNB200_OUT_U8) {
            c.bias_i = static_cast<const int32_t*>(ep.bias)[n];
        } else if constexpr (KIND == NNB200_OUT_F32) {
            c.bias_f = static_cast<const float*>(ep.bias)[n];
        } else {
            c.bias_f = __half2float(static_cast<const __half*>(ep.bias)[n]);
        }
    }
    return c;
}

// Epilogue and store of one channel's sums for activation rows [m0, m0 + ROWS), clipped at m_end.  A few rows
// at a time in a loop, with every switch taken once per group and none per element: one element after
// the other, each behind its own branches, cost 200 cycles a row (64 rows into f16: 27.0 us a call of
// which 13 were this), and the 32 unrolled copies were mostly fetched cold.
template <int KIND, int ROWS>
__device__ __forceinline__ void finish_rows(const I8Epilogue& ep, const I8RowTerms* row_terms, const uint32_t (&acc)[ROWS],
                                            int m0, int m_end, int64_t n, bool n_ok, const ChannelTerms& ct)
{
    I8RowTerms t[ROWS];
    int32_t v[ROWS];
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
        t[j] = row_terms[m0 + j];   // the table has entries past the last row
        v[j] = static_cast<int32_t>(acc[j]);
    }
    if (ep.compensate) {
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            v[j] = i8_compensate(v[j], t[j].zpa, ct.zpw, t[j].ra, ct.rw, ep.k);
        }
    }
    const int64_t idx = static_cast<int64_t>(m0) * ep.ldc + n;
    if constexpr (KIND <= NNB200_OUT_U8) {
        const int32_t relu_lo = ep.relu ? 0 : INT32_MIN;
        const float zpf = static_cast<float>(ep.out_zp);
        const float lo = (KIND == NNB200_OUT_S8 ? -128.0f : 0.0f) - zpf;
        const float hi = (KIND == NNB200_OUT_S8 ? 127.0f : 255.0f) - zpf;
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            v[j] = max(static_cast<int32_t>(static_cast<uint32_t>(v[j]) + static_cast<uint32_t>(ct.bias_i)), relu_lo);
            if constexpr (KIND != NNB200_OUT_S32) {
                v[j] = i8_requant(v[j], __fmul_rn(t[j].row_k, ct.s_w), lo, hi, ep.out_zp);
            }
        }
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            if (m0 + j < m_end && n_ok) {
                if constexpr (KIND == NNB200_OUT_S32) {
                    static_cast<int32_t*>(ep.out)[idx + j * ep.ldc] = v[j];
                } else {
                    static_cast<uint8_t*>(ep.out)[idx + j * ep.ldc] = static_cast<uint8_t>(v[j]);
                }
            }
        }
    } else {
        float f[ROWS];
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            f[j] = __fmul_rn(__int2float_rn(v[j]), __fmul_rn(t[j].s_a, ct.s_w));
            const float fb = __fadd_rn(f[j], ct.bias_f);
            f[j] = ct.bias_f != 0.0f ? fb : f[j];   // a zero bias is not added (-0 stays -0)
            f[j] = fminf(fmaxf(f[j], ep.min_clip), ep.max_clip);
        }
        const auto activate = [&](auto act) {
#pragma unroll
            for (int j = 0; j < ROWS; ++j) {
                f[j] = act_apply(decltype(act)::value, ep.act_alpha, ep.act_beta, f[j]);
            }
        };
        switch (ep.activation) {
        case NNB200_ACT_RELU: activate(std::integral_constant<int, NNB200_ACT_RELU>{}); break;
        case NNB200_ACT_RELU6: activate(std::integral_constant<int, NNB200_ACT_RELU6>{}); break;
        case NNB200_ACT_LEAKY_RELU: activate(std::integral_constant<int, NNB200_ACT_LEAKY_RELU>{}); break;
        case NNB200_ACT_SIGMOID: activate(std::integral_constant<int, NNB200_ACT_SIGMOID>{}); break;
        case NNB200_ACT_TANH: activate(std::integral_constant<int, NNB200_ACT_TANH>{}); break;
        case NNB200_ACT_GELU: activate(std::integral_constant<int, NNB200_ACT_GELU>{}); break;
        case NNB200_ACT_SILU: activate(std::integral_constant<int, NNB200_ACT_SILU>{}); break;
        case NNB200_ACT_HARD_SWISH: activate(std::integral_constant<int, NNB200_ACT_HARD_SWISH>{}); break;
        case NNB200_ACT_ELU: activate(std::integral_constant<int, NNB200_ACT_ELU>{}); break;
        default: break;
        }
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
            if (m0 + j < m_end && n_ok) {
                if constexpr (KIND == NNB200_OUT_F32) {
                    static_cast<float*>(ep.out)[idx + j * ep.ldc] = f[j];
                } else {
                    static_cast<__half*>(ep.out)[idx + j * ep.ldc] = __float2half_rn(f[j]);
                }
            }
        }
    }
}

__device__ __forceinline__ uint32_t ld_shared_cluster_u32(uint32_t cluster_addr)
{
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(cluster_addr) : "memory");
    return v;
}

__device__ __forceinline__ void st_shared_cluster_u32(uint32_t cluster_addr, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}

// How whole tiles are dealt to CTAs, or with parts > 1 the K blocks of a tile to the CTAs of a cluster: per_cta
// each, one more for the first `longer`.
struct Shares {
    int parts, per_cta, longer;
};

template <int MP, int KIND>
__global__ void __launch_bounds__(kNumThreads, 1)
gemm_i8_skinny_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a,
                      const I8Epilogue ep, const int m_total, const int n_total, const int k_total,
                      const uint32_t idesc, int32_t* error_word, unsigned long long* split_counters,
                      int32_t* split_slots, const unsigned long long split_tag, const int tile_rows, const int num_tiles, const Shares shares)
{
    using Cfg = SkinnyConfig<MP>;
    constexpr int kStages = Cfg::kStages;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* stage_base = smem;
    I8RowTerms* row_terms = reinterpret_cast<I8RowTerms*>(smem + kStages * Cfg::kStageBytes);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(reinterpret_cast<uint8_t*>(row_terms) + Cfg::kRowTermBytes);
    uint64_t* empty_bar = full_bar + kStages;
    uint64_t* acc_full_bar = empty_bar + kStages;
    uint64_t* acc_empty_bar = acc_full_bar + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty_bar + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int role = __shfl_sync(0xFFFFFFFFu, warp, 0);   // the same, warp-uniform to the compiler too
    const int lane = threadIdx.x & 31;
    const int num_kb = (k_total + kBlockKBytes - 1) / kBlockKBytes;
    const bool split = split_counters != nullptr;
    const int grid = static_cast<int>(gridDim.x);
    const int cta = static_cast<int>(blockIdx.x);
    // shares.parts > 1: a cluster of that many CTAs works one tile, each on its share of the K blocks.
    const int parts = shares.parts;
    const int rank = parts > 1 ? static_cast<int>(cluster_cta_rank()) : 0;
    const int cluster = parts > 1 ? static_cast<int>(cluster_id()) : 0;
    const SegmentList segments =
        split ? SegmentList(range_begin(cta, grid, num_tiles, num_kb), range_begin(cta + 1, grid, num_tiles, num_kb), num_kb)
              : SegmentList(SegmentList::Whole{cta * shares.per_cta + min(cta, shares.longer),
                                               (cta + 1) * shares.per_cta + min(cta + 1, shares.longer)}, num_kb);
    const int num_segments = parts > 1 ? 1 : warp_uniform(segments.count());
    const auto segment_at = [&](int i) {
        if (parts > 1) {
            return Segment{cluster, rank * shares.per_cta + min(rank, shares.longer),
                           (rank + 1) * shares.per_cta + min(rank + 1, shares.longer)};
        }
        return segments.uniform_at(i);
    };

    // ---------------- TMA producer (warp 0) ----------------
    // Like the MMA warp below: the whole warp walks the loop, one elected lane issues, and no branch
    // depends on what a wait returned.  Its loads need no barrier but the ring's, which it sets up itself, and
    // start before the CTA has met.
    uint32_t failed = 0;   // this role's first failed wait, see mbar_wait_converged
    int stage = 0;
    uint32_t phase = 0;
    if (role == 0) {
        if (lane == 0) {
            for (int s = 0; s < kStages; ++s) {
                mbar_init(&full_bar[s], 1);
                mbar_init(&empty_bar[s], 1);
            }
            for (int a = 0; a < 2; ++a) {
                mbar_init(&acc_full_bar[a], 1);
                mbar_init(&acc_empty_bar[a], kEpilogueThreads / 32);
            }
            *abort_flag = 0;
            mbar_init_fence();
        }
        __syncwarp();
        named_barrier_arrive(1, kNumThreads);   // the others meet below; this warp needs nothing of theirs
        previous_kernel_done();
    } else if (warp == 1) {
        tmem_alloc(tmem_slot, Cfg::kTmemCols);
        tmem_relinquish();
        named_barrier_arrive(2, 64);   // the producer, before it lets the next kernel start
    }
    // Per-row epilogue terms of every activation row, once per CTA (the rows are the same for all tiles).
    else {
        previous_kernel_done();
        const int t = threadIdx.x - 64;
        if (t < Cfg::kRowTerms) {
            row_terms[t] = i8_row_terms(ep, t < m_total ? t : 0);
        }
    }
    if (role != 0) {
        tc_fence_before_sync();
        named_barrier_sync(1, kNumThreads);
        tc_fence_after_sync();
    }
    const uint32_t tmem_base = *tmem_slot;

    if (role == 0) {
        uint32_t issued = 0;   // by this lane
        for (int si = 0; si < num_segments; ++si) {
            const Segment seg = segment_at(si);
            const int row = seg.tile * tile_rows;
            for (int kb = seg.kb0; kb < seg.kb1; ++kb) {
                mbar_wait_converged<kErrProducerWait>(&empty_bar[stage], phase ^ 1u, abort_flag, failed);
                if (elect_one() && !wait_failed(failed)) {
                    uint8_t* w_dst = stage_base + stage * Cfg::kStageBytes;
                    mbar_expect_tx(&full_bar[stage], static_cast<uint32_t>(tile_rows * kBlockKBytes + Cfg::kATileBytes));
                    ++issued;
                    tma_load_2d(w_dst, &map_w, &full_bar[stage], kb * kBlockKBytes, row);
                    tma_load_2d(w_dst + Cfg::kWTileBytes, &map_a, &full_bar[stage], kb * kBlockKBytes, 0);
                }
                __syncwarp();
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        }
        const uint32_t all_issued = __reduce_add_sync(0xFFFFFFFFu, issued);   // one lane has counted
        named_barrier_sync(2, 64);   // tensor memory is allocated
        let_next_kernel_start();
        if (const uint32_t code = warp_failure(failed); code != 0 && lane == 0) {
            atomicCAS(error_word, 0, static_cast<int32_t>(code));
            if (!drain_ring(full_bar, kStages, all_issued)) {
                atomicCAS(error_word, 0, kErrDrainWait);
            }
        }
        __syncwarp();
        if (parts > 1) {
            cluster_sync_all();
            cluster_sync_all_relaxed();
        }
    } else if (role == 1) {
        // ---------------- MMA issuer ----------------
        // The whole warp walks the loop and one elected lane issues: tensor-memory addresses and
        // descriptors are then warp-uniform to the compiler, which is how the MMA takes its operands.
        // The waits keep it so (see mbar_wait_converged): a K block of four MMAs takes 160 to 256 cycles
        // of tensor pipe, and the loop took 525 cycles a block while its waits branched.
        const uint32_t tmem = warp_uniform(tmem_base);
        // The ring's descriptors advance by addition; the activations' tile lies behind the weights'.
        const uint64_t first_desc = umma_desc_sw128_kmajor(smem_u32(stage_base));
        uint64_t w_desc = first_desc;   // the MMA's 128-row operand
        for (int local_seg = 0; local_seg < num_segments; ++local_seg) {
            const Segment seg = segment_at(local_seg);
            const int acc = local_seg & 1;
            const uint32_t acc_phase = (local_seg >> 1) & 1u;
            mbar_wait_converged<kErrAccumWait>(&acc_empty_bar[acc], acc_phase ^ 1u, abort_flag, failed);
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem + static_cast<uint32_t>(acc * MP);
            uint32_t accumulate = 0;
            for (int kb = seg.kb0; kb < seg.kb1; ++kb) {
                mbar_wait_converged<kErrMmaWait>(&full_bar[stage], phase, abort_flag, failed);
                tc_fence_after_sync();
                const uint64_t a_desc = w_desc + Cfg::kWTileBytes / 16;  // its N operand: MP activation rows
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < kBlockKBytes / kUmmaK; ++ks) {
                        umma_i8(d_tmem, w_desc + static_cast<uint64_t>(ks * 2), a_desc + static_cast<uint64_t>(ks * 2),
                                idesc, ks > 0 ? 1u : accumulate);
                    }
                    umma_commit(&empty_bar[stage]);
                }
                __syncwarp();
                accumulate = 1;
                w_desc += Cfg::kStageBytes / 16;
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                    w_desc = first_desc;
                }
            }
            if (elect_one()) {
                umma_commit_unless(&acc_full_bar[acc], failed);
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
        if (parts > 1) {
            cluster_sync_all();
            cluster_sync_all_relaxed();
        }
    } else {
        // ---------------- epilogue warps: one channel per thread ----------------
        const int quarter = warp & 3;
        const int ch = quarter * 32 + lane;  // this thread's channel within the tile
        const int64_t total_units = static_cast<int64_t>(num_tiles) * num_kb;
        const size_t slot_elems = static_cast<size_t>(kBlockN) * static_cast<size_t>(m_total);
        const int group = (warp - 2) >> 2;
        if (parts > 1) {
            // Each CTA of the cluster finishes its share of the tile's rows, four at a time per warp, from
            // everybody's sums.  The first pass stores nothing: it brings the instructions in while the weights
            // stream (cold, they took longer than the work itself).
            const int64_t n = static_cast<int64_t>(cluster) * tile_rows + ch;
            const bool n_ok = ch < tile_rows && n < n_total;
            const ChannelTerms ct = channel_terms<KIND>(ep, n, n_ok);
            uint32_t* mine = reinterpret_cast<uint32_t*>(stage_base) + ch;
            const bool all_ok = __all_sync(0xFFFFFFFFu, n_ok);
            const uint32_t never = static_cast<uint32_t>(parts) >> 16;   // 0, which the compiler does not know
            int row = 0, row_end = 1, store_end = 0, part = rank, part_step = 0;   // first pass: its own sums only, the others' CTAs may not have begun
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass) {
                if (pass == 1) {
                    part_step = 1;
                    if (mbar_wait_warp(&acc_full_bar[0], 0, abort_flag)) {
                        tc_fence_after_sync();
                        const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
                        // This CTA's sums, [row][channel], where the ring was: all its loads have been consumed.
#pragma unroll 1
                        for (int r = group * 8; r < m_total; r += 16) {
                            uint32_t v[8];
                            tmem_ld_32x8(t_row + static_cast<uint32_t>(r), v);
                            tmem_ld_wait();
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
                                mine[(r + j) * kBlockN] = v[j];
                            }
                        }
                    } else {
                        // This CTA has no sums (a role that gives up commits none): nobody in the cluster stores.
                        if (lane == 0) {
                            atomicCAS(error_word, 0, kErrEpilogueWait);
                        }
                        if (lane < parts) {
                            st_shared_cluster_u32(map_to_cta(smem_u32(const_cast<const int*>(abort_flag)), static_cast<uint32_t>(lane)), 1u);
                        }
                    }
                    __syncwarp();
                    cluster_sync_all();
                    row = rank * m_total / parts + group * 4;
                    store_end = row_end = *abort_flag != 0 ? row : (rank + 1) * m_total / parts;
                    part = 0;
                }
#pragma unroll 1
                for (int r = row; r < row_end; r += 8) {
                    // All loads before any sum: one round trip to the other SMs.
                    uint32_t theirs[kMaxParts][4];
#pragma unroll
                    for (int p = 0; p < kMaxParts; ++p) {
                        if (p < parts) {
                            const uint32_t from = map_to_cta(smem_u32(mine), static_cast<uint32_t>(part + p * part_step));
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                theirs[p][j] = ld_shared_cluster_u32(from + static_cast<uint32_t>((r + j) * kBlockN) * 4);
                            }
                        }
                    }
                    uint32_t v[4] = {0, 0, 0, 0};
#pragma unroll
                    for (int p = 0; p < kMaxParts; ++p) {
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            v[j] += p < parts ? theirs[p][j] : 0u;
                        }
                    }
                    finish_rows<KIND, 4>(ep, row_terms, v, r, store_end, n, n_ok, ct);
                    if (r + 4 > row_end || !all_ok) {
                        // Rows or channels that are not stored: nothing else waits for their loads, and the CTA they come
                        // from may leave after the barrier below.  Once the warp has met here they have come.
                        const uint32_t seen = v[0] | v[1] | v[2] | v[3];
                        row_end = __any_sync(0xFFFFFFFFu, (seen & never) != 0) ? 0 : row_end;
                    }
                }
            }
            __syncwarp();
            cluster_sync_all_relaxed();   // nobody leaves while its sums may still be read
        }
        // A CTA that holds one piece has both groups work on it, eight rows in turn.
        const bool shared = num_segments == 1 && !split;
        for (int local_seg = shared ? 0 : group; parts == 1 && local_seg < num_segments; local_seg += 2) {
            const Segment seg = segment_at(local_seg);
            const int tile = seg.tile;
            const int acc = local_seg & 1;
            const uint32_t acc_phase = (local_seg >> 1) & 1u;
            const bool partial = split && (seg.kb0 != 0 || seg.kb1 != num_kb);
            const int64_t n = static_cast<int64_t>(tile) * tile_rows + ch;
            const bool n_ok = ch < tile_rows && n < n_total;
            // This channel's terms, in registers for the whole tile.
            const ChannelTerms ct = channel_terms<KIND>(ep, n, n_ok);

            // Part of a tile.  While this piece's MMAs are still running, look whether everybody else
            // has published already; if so this warp will finish the tile and fetches the others'
            // sums for the first 32 rows now, off the critical path.
            int first_cta = 0, last_cta = -1;
            bool early = false;
            int32_t early_sum[32];
            if (partial) {
                first_cta = cta_of_unit(static_cast<int64_t>(tile) * num_kb, grid, total_units);
                last_cta = cta_of_unit(static_cast<int64_t>(tile + 1) * num_kb - 1, grid, total_units);
                int seen = 0;
                if (MP == 32 && lane == 0) {
                    seen = arrivals_of(ld_acquire_gpu_u64(&split_counters[tile * 4 + quarter]), split_tag);
                }
                seen = __shfl_sync(0xFFFFFFFFu, seen, 0);
                // Only where 32 rows are all there is: with more rows the early fetch covers a part of
                // the work and measured slower than none.
                early = MP == 32 && seen == last_cta - first_cta;
                if (early) {
                    __threadfence();  // every lane's reads of the others' slots come after lane 0's look
                    collect_parts(early_sum, split_slots, slot_elems, ch, first_cta, last_cta, static_cast<int>(blockIdx.x),
                                  0, m_total);
                }
            }

            const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                   static_cast<uint32_t>(acc * MP);
            if (!partial) {
                // A whole tile.  The first of the CTA's starts with a pass that stores nothing: it brings the
                // instructions in while the weights stream (cold, they took longer than the work itself).
                bool ok = true;
#pragma unroll 1
                for (int pass = local_seg < 2 ? 0 : 1; pass < 2; ++pass) {
                    int row = 0, row_end = 1;
                    if (pass == 1) {
                        ok = mbar_wait_warp(&acc_full_bar[acc], acc_phase, abort_flag);
                        if (!ok) {
                            break;
                        }
                        tc_fence_after_sync();
                        row = shared ? group * 8 : 0;
                        row_end = m_total;
                    }
#pragma unroll 1
                    for (int r = row; r < row_end; r += shared ? 16 : 8) {
                        uint32_t v[8];
                        tmem_ld_32x8(t_row + static_cast<uint32_t>(r), v);
                        tmem_ld_wait();
                        finish_rows<KIND, 8>(ep, row_terms, v, r, pass == 1 ? row_end : 0, n, n_ok, ct);
                    }
                }
                if (!ok) {
                    atomicCAS(error_word, 0, kErrEpilogueWait);
                    break;
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&acc_empty_bar[acc]);
                }
                continue;
            }
            if (!mbar_wait_warp(&acc_full_bar[acc], acc_phase, abort_flag)) {
                atomicCAS(error_word, 0, kErrEpilogueWait);
                break;
            }
            tc_fence_after_sync();
            // Otherwise: publish this warp's 32 channels, count in, and carry on only if every other
            // part of the tile has been published by then.
            bool finish = true;
            bool publish = partial && !early;
            unsigned long long seen_word = 0;  // lane 0's last look at the tile's arrival word
            if (publish) {
                // Everybody else in by now?  Then this warp finishes the tile and has nothing to publish.
                int seen = 0;
                if (lane == 0) {
                    seen_word = ld_acquire_gpu_u64(&split_counters[tile * 4 + quarter]);
                    seen = arrivals_of(seen_word, split_tag);
                }
                seen = __shfl_sync(0xFFFFFFFFu, seen, 0);
                publish = seen != last_cta - first_cta;
                if (!publish) {
                    __threadfence();  // every lane's reads of the others' slots come after lane 0's look
                }
            }
            if (publish) {
                int32_t* mine = split_slots +
                                (2 * static_cast<size_t>(blockIdx.x) + (seg.kb0 == 0 ? 1u : 0u)) * slot_elems + ch;
#pragma unroll 1
                for (int c = 0; c < MP / 32; ++c) {
                    if (c * 32 >= m_total) {
                        break;  // uniform
                    }
                    uint32_t v[32];
                    tmem_ld_32x32(t_row + static_cast<uint32_t>(c * 32), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        if (c * 32 + j < m_total) {
                            __stcg(mine + static_cast<size_t>(c * 32 + j) * kBlockN, static_cast<int32_t>(v[j]));
                        }
                    }
                }
                __threadfence();
                __syncwarp();
                int ticket = 0;
                if (lane == 0) {
                    ticket = arrive(&split_counters[tile * 4 + quarter], split_tag, seen_word);
                }
                ticket = __shfl_sync(0xFFFFFFFFu, ticket, 0);
                if (ticket < 0) {
                    atomicCAS(error_word, 0, kErrEpilogueWait);  // cannot happen with at most 148 parts per word
                }
                finish = ticket == last_cta - first_cta;
                if (finish) {
                    __threadfence();
                }
            }
            if (partial && finish && lane == 0) {
                split_counters[tile * 4 + quarter] = split_tag << 8;  // nobody else touches it in this launch
            }
#pragma unroll 1
            for (int c = 0; c < MP / 32; ++c) {
                if (c * 32 >= m_total || !finish) {
                    break;  // uniform
                }
                if (!(early && c == 0)) {
                    collect_parts(early_sum, split_slots, slot_elems, ch, first_cta, last_cta,
                                  static_cast<int>(blockIdx.x), c * 32, m_total);
                }
#pragma unroll
                for (int r = 0; r < 32; r += 8) {
                    uint32_t v[8];
                    tmem_ld_32x8(t_row + static_cast<uint32_t>(c * 32 + r), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        v[j] += static_cast<uint32_t>(early_sum[r + j]);
                    }
                    if (c * 32 + r < m_total) {
                        finish_rows<KIND, 8>(ep, row_terms, v, c * 32 + r, m_total, n, n_ok, ct);
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&acc_empty_bar[acc]);
            }
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before_sync();
    __syncwarp();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

// A 56-bit tag no earlier launch of this process has used, never zero; the sequence starts at
// a point derived from the clock so that words left in recycled memory by another process do
// not match either.
unsigned long long next_split_tag()
{
    static std::atomic<unsigned long long> counter{
        static_cast<unsigned long long>(std::chrono::steady_clock::now().time_since_epoch().count()) * 0x9E3779B97F4A7C15ull};
    unsigned long long t;
    do {
        t = counter.fetch_add(1, std::memory_order_relaxed) & ((1ull << 56) - 1);
    } while (t == 0);
    return t;
}

// Clusters of `parts` CTAs that the device holds at once; 0 where it cannot say.  Every variant of the kernel takes an
// SM to itself, so one stands for all.
int resident_clusters(const DeviceInfo& dev, int parts)
{
    static std::once_flag once[kMaxDevices];
    static int resident[kMaxDevices][kMaxParts + 1];
    std::call_once(once[dev.device], [&] {
        auto kernel = gemm_i8_skinny_kernel<128, NNB200_OUT_F32>;
        cudaLaunchConfig_t cfg = {};
        cfg.blockDim = dim3(kNumThreads);
        cfg.dynamicSmemBytes = SkinnyConfig<128>::kSmemBytes;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SkinnyConfig<128>::kSmemBytes) == cudaSuccess;
        for (int c = 2; c <= kMaxParts && ok; ++c) {
            attr.val.clusterDim.x = static_cast<unsigned>(c);
            cfg.gridDim = dim3(static_cast<unsigned>(dev.sm_count / c * c));
            int count = 0;
            if (cudaOccupancyMaxActiveClusters(&count, kernel, &cfg) == cudaSuccess) {
                resident[dev.device][c] = count;
            } else {
                (void)cudaGetLastError();   // no clusters of that many: the launch takes a smaller one
            }
        }
    });
    return resident[dev.device][parts];
}

// CTAs that share a tile's K, by way of their cluster: as many as leave every tile's cluster an SM per CTA.
int cluster_parts(const I8Problem& p, const DeviceInfo& dev)
{
    const int64_t tiles = (p.n + kBlockN - 1) / kBlockN;
    const int64_t num_kb = (p.k + kBlockKBytes - 1) / kBlockKBytes;
    int64_t parts = dev.sm_count / tiles;
    parts = parts > kMaxParts ? kMaxParts : parts;
    parts = parts > num_kb / 4 ? num_kb / 4 : parts;
    while (parts > 1 && resident_clusters(dev, static_cast<int>(parts)) < tiles) {
        --parts;
    }
    return parts > 1 ? static_cast<int>(parts) : 1;
}

template <int MP, int KIND>
int launch_skinny_variant(const I8Problem& p, const I8Epilogue& ep, const DeviceInfo& dev, void* split_scratch,
                          cudaStream_t stream)
{
    using Cfg = SkinnyConfig<MP>;
    auto kernel = gemm_i8_skinny_kernel<MP, KIND>;
    static std::once_flag once[kMaxDevices];
    static cudaError_t attr_err[kMaxDevices];
    std::call_once(once[dev.device], [&] {
        attr_err[dev.device] = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    });
    if (attr_err[dev.device] != cudaSuccess) {
        return NNB200_INTERNAL;
    }
    const int m = static_cast<int>(p.m), n = static_cast<int>(p.n), k = static_cast<int>(p.k);
    // Whole tiles over several waves: as many waves as 128-channel tiles need, cut into equal tiles (24
    // rows, 128-channel tiles / equal ones: N = 28672, K = 8192 51.8 / 45.4 us, N = 19456, K = 4096 28.1 / 24.8).
    // A caller that brings the scratch for shared K gets that on the first of the two: 45.7.
    // A single wave of whole tiles is cut likewise up to 32 rows (N = 11008, K = 4096: 16 rows 10.7 / 9.7, 24 rows
    // 10.3 / 10.0); with more, the activations that more CTAs load eat what the even weight stream gives (64 and
    // 128 rows lost 3 and 8 %).  Shared K evens the SMs out itself, and its scratch is laid out for 128.
    int tile_rows = kBlockN;
    int parts = split_scratch != nullptr ? 1 : cluster_parts(p, dev);   // the scratch is offered where clusters do not serve
    const int waves = ((n + kBlockN - 1) / kBlockN + dev.sm_count - 1) / dev.sm_count;
    if (split_scratch == nullptr && parts == 1 && (waves > 1 || p.m <= 32)) {
        tile_rows = (n + waves * dev.sm_count - 1) / (waves * dev.sm_count);
    }
    CUtensorMap map_w, map_a;
    if (!make_tma_2d(&map_w, p.w, 1, static_cast<uint64_t>(k), static_cast<uint64_t>(n),
                     static_cast<uint64_t>(p.w_stride_n), kBlockKBytes, static_cast<uint32_t>(tile_rows)) ||
        !make_tma_2d(&map_a, p.a, 1, static_cast<uint64_t>(k), static_cast<uint64_t>(m),
                     static_cast<uint64_t>(p.a_stride_m), kBlockKBytes, MP)) {
        return NNB200_INTERNAL;
    }
    const int num_tiles = (n + tile_rows - 1) / tile_rows;
    int grid = num_tiles < dev.sm_count ? num_tiles : dev.sm_count;
    unsigned long long* counters = nullptr;
    int32_t* slots = nullptr;
    unsigned long long tag = 0;
    if (parts > 1) {
        grid = num_tiles * parts;
    } else if (split_scratch != nullptr) {
        // Equal shares of all K blocks over every SM.
        grid = dev.sm_count;
        counters = static_cast<unsigned long long*>(split_scratch);
        slots = reinterpret_cast<int32_t*>(static_cast<uint8_t*>(split_scratch) + split_counter_bytes(num_tiles));
        tag = next_split_tag();
    }
    // 128-row operand = weights (s8), N operand = activations (s8 or u8).
    const uint32_t idesc = umma_idesc(2, 1, p.a_unsigned ? 0u : 1u, kBlockN, MP);
    Shares shares{parts, 0, 0};
    const int dealt = parts > 1 ? (k + kBlockKBytes - 1) / kBlockKBytes : num_tiles, hands = parts > 1 ? parts : grid;
    shares.per_cta = dealt / hands;
    shares.longer = dealt % hands;
    const cudaError_t launched = launch_overlapping(kernel, dim3(static_cast<unsigned>(grid)), dim3(kNumThreads), Cfg::kSmemBytes, stream, parts, map_w, map_a, ep, m, n, k, idesc, dev.error_word, counters, slots,
                                                    tag, tile_rows, num_tiles, shares);
    note_launch();
    return cuda_status(launched);
}

template <int MP>
int launch_skinny_mp(const I8Problem& p, const I8Epilogue& ep, const DeviceInfo& dev, void* split_scratch,
                     cudaStream_t stream)
{
    switch (ep.out_kind) {
    case NNB200_OUT_S32: return launch_skinny_variant<MP, NNB200_OUT_S32>(p, ep, dev, split_scratch, stream);
    case NNB200_OUT_S8: return launch_skinny_variant<MP, NNB200_OUT_S8>(p, ep, dev, split_scratch, stream);
    case NNB200_OUT_U8: return launch_skinny_variant<MP, NNB200_OUT_U8>(p, ep, dev, split_scratch, stream);
    case NNB200_OUT_F32: return launch_skinny_variant<MP, NNB200_OUT_F32>(p, ep, dev, split_scratch, stream);
    case NNB200_OUT_F16: return launch_skinny_variant<MP, NNB200_OUT_F16>(p, ep, dev, split_scratch, stream);
    default: return NNB200_UNSUPPORTED;
    }
}

}  // namespace

// The square tensor-core engine's operands with k contiguous in both (its tensor maps know no other
// pose: a [K, N] weight runs on the square engine), at most 128 activation rows.
bool skinny_i8_supported(const I8Problem& p)
{
    return p.m >= 1 && p.m <= 128 && p.a_stride_k == 1 && p.w_stride_k == 1 && umma_i8_supported(p) &&
           (p.n / kBlockN + 1) * (p.k / kBlockKBytes + 1) < (int64_t{1} << 29);   // units are counted in 32 bits
}

// Whether the busiest SM of a single wave of tiles sheds enough K blocks when all SMs share K: at least 30, plus 0.7 per
// row above 12 (see skinny_i8_split_bytes).
static bool sharing_sheds_enough(const I8Problem& p, int64_t sms)
{
    const int64_t tiles = (p.n + kBlockN - 1) / kBlockN;
    const int64_t num_kb = (p.k + kBlockKBytes - 1) / kBlockKBytes;
    const int64_t share = (tiles * num_kb + sms - 1) / sms;
    const int64_t rows_over = p.m > 12 ? p.m - 12 : 0;
    return (num_kb - share) * 10 >= 300 + 7 * rows_over;
}

// Whether a call that the square engine or the streaming engine (up to 16 rows) would get by its number of
// rows and channels is better off here, on clusters that share K.  CUDA-graph timings, weights beyond L2,
// here / square engine, us:
//   rows   N = 1024                                4096                                8192
//     32   K = 512 4.2 / 4.5, 4096 5.1 / 8.6       512 4.4 / 5.1, 4096 7.2 / 9.6       4096 9.8 / 10.5, 8192 14.4 / 16.8
//     64   512 4.9 / 4.6, 2048 5.4 / 6.2           512 5.0 / 4.8, 4096 8.1 / 9.5       2048 8.4 / 7.8, 8192 15.4 / 16.7
//    128   2048 6.7 / 6.4, 4096 7.2 / 8.8          2048 8.1 / 7.3, 4096 9.5 / 9.9      4096 13.2 / 10.6
// and here / streaming engine:
//     16   2048 3.6 / 3.4, 4096 4.1 / 5.1          2048 4.5 / 4.7, 4096 5.8 / 7.3      512 3.3 / 5.4, 2048 5.7 / 8.2
//      4   2048 3.4 / 3.0, 4096 3.7 / 4.0          2048 4.5 / 4.3, 4096 5.8 / 5.9      512 3.5 / 5.2, 8192 12.9 / 16.8
//      1   2048 3.4 / 2.5, 8192 4.5 / 6.4          4096 5.6 / 5.4, 16384 12.6 / 14.2   512 3.4 / 4.1, 2048 5.6 / 6.7
//   N = 64, 8192: 16 rows 4.2 / 5.7, 4 rows 3.9 / 4.3, one 3.5 / 3.8; N = 6144, 4096: 16 rows 7.4 / 8.1, 4 rows 7.7 / 6.8;
//   N = 28672, 8192: 16 rows 40.0 / 56.8, one 38.0 / 40.9; 28672, 1024: one 7.7 / 12.3.  The one place past 6272
//   channels where one row is better off there: too many tiles for clusters and too few for the SMs, with a
//   long K (N = 11008: K = 1024 4.8 / 5.9, 4096 11.3 / 10.4; N = 14336, 4096 12.3 / 13.6).
bool skinny_i8_preferred(const I8Problem& p, bool over_streaming, int64_t sms)
{
    if (!skinny_i8_supported(p)) {
        return false;
    }
    const int64_t tiles = (p.n + kBlockN - 1) / kBlockN;
    if (over_streaming) {
        const bool sparse = p.m == 1 && p.k > 2048 && tiles * 2 > sms && tiles * 4 <= sms * 3;
        return (tiles * 3 > sms && !sparse) || p.k >= 8192 || (p.m > 8 && p.n >= 1024 && p.k >= 4096);
    }
    if (p.m <= 32) {
        return true;
    }
    if (p.m <= 64) {
        return tiles * 3 <= sms ? p.k >= 2048 : p.k >= 8192;
    }
    // Past the middle only where K is long for the rows (clusters / square engine: 72 x 6400 x 16384 25.0 / 27.1, 72 x
    // 9472 x 16384 32.4 / 32.9, 66 x 6400 x 12288 19.5 / 20.3).
    return (tiles * 4 <= sms && p.k >= 4096) || (tiles * 2 <= sms && sharing_sheds_enough(p, sms));
}

// Scratch for the equal-share split of K over all SMs, or 0 when it would not pay.  Publishing a
// part, counting in and collecting the others' parts is a chain of L2 round trips at the end of
// the kernel, each well over a microsecond while every SM is streaming: about 6 us in all plus
// ~0.1 us per activation row, against the K blocks that the busiest CTA no longer has to stream.  Measured, shared K /
// without, 24 and 64 rows (us):
//   one wave of tiles:
//         N=9600,K=8192 20.4 / 17.2, 24.8 / 18.5          N=9600,K=16384 36.6 / 30.8, 41.8 / 33.2
//         N=11008,K=8192 22.4 / 19.1, 27.1 / 20.7         N=11008,K=16384 36.8 / 33.7, 42.6 / 36.4
//         N=12288,K=28672 61.5 / 56.6, 67.4 / 59.6        N=16384,K=16384 49.5 / 44.8, 54.8 / 47.8
//   several, where the alternative is equal tiles, by waves of 128-channel tiles:
//   1.03  N=19456,K=8192 33.0 / 31.5, 37.5 / 35.3         1.16  N=22016,K=8192 35.3 / 33.6, 39.4 / 37.5
//   1.30  N=24576,K=8192 38.4 / 36.7, 42.7 / 40.4         1.51  N=28672,K=8192 43.4 / 40.8, 48.2 / 44.5
//   1.51  N=28672,K=4096 25.3 / 22.9, 29.5 / 25.2         1.51  N=28672,K=16384 77.8 / 74.5, 82.6 / 80.0
//   1.69  N=32000,K=8192 47.6 / 44.9, 52.2 / 48.9         2.27  N=43008,K=8192 59.3 / 58.8, 63.7 / 63.0
// So none of these gains.  The lines below are older: they were drawn when a K block took the issuing warps 525 cycles
// (0.3 us for the busiest CTA; N=8192, K=8192 25.3 / 22.2 the other way round) and have not been drawn again.
// With one wave, share when the busiest CTA sheds at least 30 K blocks, plus 0.7 per row
// above 12; with several waves, when the last one is less than 9/10 full, a share is at least 48
// K blocks and there are at most 64 rows.
// None where clusters share K (4096 x 14336, 24 rows: 21.3 us on the scratch, 13.3 in clusters).
// Knob I8_SHARE_K = 0 turns this split off; 2 offers it from 8 K blocks per SM and prefers it (measurement, tests).
size_t skinny_i8_split_bytes(const I8Problem& p, const DeviceInfo& dev)
{
    if (!skinny_i8_supported(p)) {
        return 0;
    }
    const int share_knob = knob(NNB200_KNOB_I8_SHARE_K);
    const char mode = share_knob < 0 ? '1' : static_cast<char>('0' + (share_knob > 2 ? 1 : share_knob));
    if (mode == '0') {
        return 0;
    }
    const int64_t tiles = (p.n + kBlockN - 1) / kBlockN;
    const int64_t num_kb = (p.k + kBlockKBytes - 1) / kBlockKBytes;
    const int64_t sms = dev.sm_count;
    const int64_t waves = (tiles + sms - 1) / sms;
    const int64_t share = (tiles * num_kb + sms - 1) / sms;
    if (tiles * 10 >= waves * sms * 9 || share < 8) {
        return 0;  // whole tiles already fill the SMs, or there is next to nothing to share
    }
    if (mode != '2') {
        if (cluster_parts(p, dev) > 1) {
            return 0;
        }
        if (waves == 1) {
            if (!sharing_sheds_enough(p, sms)) {
                return 0;
            }
        } else if (share < 48 || p.m > 64) {
            return 0;
        }
    }
    // Two slots per CTA (the tile it finishes for someone and the tile it leaves to someone),
    // each 128 channels x m int32.
    return split_counter_bytes(static_cast<int>(tiles)) +
           2 * static_cast<size_t>(sms) * kBlockN * static_cast<size_t>(p.m) * sizeof(int32_t);
}

int launch_gemm_i8_skinny(const I8Problem& p, const I8Epilogue& ep, const DeviceInfo& dev, void* split_scratch,
                          cudaStream_t stream)
{
    if (p.m <= 32) {
        return launch_skinny_mp<32>(p, ep, dev, split_scratch, stream);
    }
    if (p.m <= 64) {
        return launch_skinny_mp<64>(p, ep, dev, split_scratch, stream);
    }
    return launch_skinny_mp<128>(p, ep, dev, split_scratch, stream);
}

}  // namespace nnb200
