// Copies of 8-bit matrices into rows of a 16-byte pitch (i8_realign.cu).
#pragma once

#include <cstdint>

#include "internal.cuh"

namespace nnb200 {

// `rows` rows of `cols` contiguous bytes, `batch` times.  rows == 0: nothing to copy.
struct I8RealignJob {
    const uint8_t* src;
    int64_t rows, cols, src_pitch, src_batch, batch;
    uint8_t* dst;           // [batch][rows][dst_pitch], 16-byte aligned
    int64_t dst_pitch;      // cols rounded up to a multiple of 16
    uint8_t* sums;          // int32 sum of each row, at sums + b * sums_batch + 4 * row; or null
    int64_t sums_batch;     // bytes
    int32_t is_unsigned;
};

int launch_i8_realign(const I8RealignJob& a, const I8RealignJob& w, const DeviceInfo& dev, cudaStream_t stream);

}  // namespace nnb200
