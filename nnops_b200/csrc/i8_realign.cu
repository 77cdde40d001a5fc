// Realigned copies of 8-bit operands for the tensor-core engines.
//
// TMA addresses a matrix whose base and row pitch are multiples of 16 bytes; a K (or, for an
// operand stored the other way round, an M or N) that 16 does not divide breaks the rule for the
// whole matrix.  Such calls used to run on the generic CUDA-core engine, whose cost grows with
// M * N * K; copying the operands once into rows of a 16-byte pitch grows with (M + N) * K, and
// everything behind the copy is the ordinary engine choice.
//
// Bound by memory: a row is read once and written once.  One warp per row -- or one block, where the
// rows are few and long -- each thread one 16-byte piece of the destination at a time, assembled from
// five aligned words with funnel shifts (the source row starts at any byte).  A word that reaches past the row's first or last byte is
// gathered byte by byte instead, so nothing outside the operand is read.  The row sums that a
// zero point on the other operand calls for ride along (rows along k only): a separate sweep
// would read the operand again.  Bytes past the row's end, up to the pitch, are zeros.

#include "internal.cuh"
#include "ptx.cuh"
#include "i8_realign.cuh"

namespace nnb200 {

namespace {

constexpr int kWarps = 8;

// The four bytes at row[at .. at+3], an address that is a multiple of four; what lies outside [0, cols)
// reads as zero.
__device__ __forceinline__ uint32_t load_word(const uint8_t* row, int64_t at, int64_t cols)
{
    if (at >= 0 && at + 4 <= cols) {
        return *reinterpret_cast<const uint32_t*>(row + at);
    }
    uint32_t v = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        if (at + b >= 0 && at + b < cols) {
            v |= static_cast<uint32_t>(row[at + b]) << (8 * b);
        }
    }
    return v;
}

// TEAM: threads on a row, a warp's or a block's.
template <int TEAM>
__global__ void __launch_bounds__(kWarps * 32) i8_realign_kernel(const I8RealignJob a, const I8RealignJob w)
{
    previous_kernel_done();
    constexpr int kTeams = kWarps * 32 / TEAM;
    __shared__ int32_t part[kWarps];
    const int lane = threadIdx.x % TEAM;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * kTeams;
    const int64_t a_rows = a.rows * a.batch;
    const int64_t total = a_rows + w.rows * w.batch;
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * kTeams + threadIdx.x / TEAM; i < total; i += stride) {
        const bool is_a = i < a_rows;
        const I8RealignJob& j = is_a ? a : w;
        const int64_t at = is_a ? i : i - a_rows;
        const int64_t b = j.batch > 1 ? at / j.rows : 0;
        const int64_t r = at - b * j.rows;
        const uint8_t* row = j.src + b * j.src_batch + r * j.src_pitch;
        uint8_t* dst = j.dst + at * j.dst_pitch;
        const int shift = static_cast<int>(reinterpret_cast<uintptr_t>(row) & 3u);
        int32_t sum = 0;
        for (int64_t c = lane * 16; c < j.dst_pitch; c += TEAM * 16) {
            uint32_t q[5];
#pragma unroll
            for (int t = 0; t < 5; ++t) {
                q[t] = (t < 4 || shift != 0) ? load_word(row, c - shift + 4 * t, j.cols) : 0u;
            }
            uint4 v;
            v.x = __funnelshift_r(q[0], q[1], 8 * shift);
            v.y = __funnelshift_r(q[1], q[2], 8 * shift);
            v.z = __funnelshift_r(q[2], q[3], 8 * shift);
            v.w = __funnelshift_r(q[3], q[4], 8 * shift);
            *reinterpret_cast<uint4*>(dst + c) = v;
            if (j.sums != nullptr) {
                const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    sum = j.is_unsigned ? static_cast<int32_t>(__dp4a(words[t], 0x01010101u, static_cast<uint32_t>(sum)))
                                        : __dp4a(static_cast<int32_t>(words[t]), 0x01010101, sum);
                }
            }
        }
        if (j.sums != nullptr) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
            }
            if constexpr (TEAM > 32) {
                // The whole block is on this row and takes the same turns.
                if ((threadIdx.x & 31) == 0) {
                    part[threadIdx.x >> 5] = sum;
                }
                __syncthreads();
                sum = 0;
#pragma unroll
                for (int o = 0; o < kWarps; ++o) {
                    sum += part[o];
                }
                __syncthreads();
            }
            if (lane == 0) {
                *reinterpret_cast<int32_t*>(j.sums + b * j.sums_batch + r * 4) = sum;
            }
        }
    }
}

}  // namespace

int launch_i8_realign(const I8RealignJob& a, const I8RealignJob& w, const DeviceInfo& dev, cudaStream_t stream)
{
    const int64_t rows = a.rows * a.batch + w.rows * w.batch;
    if (rows == 0) {
        return NNB200_OK;
    }
    const int64_t most = static_cast<int64_t>(dev.sm_count) * 8 * 4;   // eight resident blocks an SM, four turns
    // A warp copies 512 bytes a turn, and a turn is a round trip to memory.  Rows of more than four turns, no
    // more of them than resident blocks, get a block each.  Copies and product, us, a warp / a block: weight
    // [K, N] of 300 x 200001 x 256 474 / 262, 300 x 10001 x 256 31.2 / 25.4; k-contiguous 300 x 300 x 9001
    // 34.1 / 29.5, 1 x 512 x 100001 170 / 64; with more rows the blocks' fewer turns do not pay for their
    // barrier (1 x 4700 x 2100 17.0 / 20.2).
    const int64_t pitch = a.rows > 0 && (w.rows == 0 || a.dst_pitch > w.dst_pitch) ? a.dst_pitch : w.dst_pitch;
    const bool wide = rows <= static_cast<int64_t>(dev.sm_count) * 8 && pitch > 4 * 512;
    const int64_t blocks = wide ? rows : (rows + kWarps - 1) / kWarps;
    const unsigned grid = static_cast<unsigned>(blocks < most ? blocks : most);
    cudaError_t launched;
    if (wide) {
        launched = launch_overlapping(i8_realign_kernel<kWarps * 32>, dim3(grid), dim3(kWarps * 32), 0, stream, 1, a, w);
    } else {
        launched = launch_overlapping(i8_realign_kernel<32>, dim3(grid), dim3(kWarps * 32), 0, stream, 1, a, w);
    }
    note_launch();
    return cuda_status(launched);
}

}  // namespace nnb200
