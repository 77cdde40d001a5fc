// A batch of equal int8 products in one launch (gemm_i8_umma_batched.cu).
#pragma once

#include <cstdint>

#include "internal.cuh"

namespace nnb200 {

struct I8Batch {
    int64_t count;
    int64_t a_stride, w_stride;    // bytes between problems; 0 = shared by all
    int64_t out_stride;            // elements
    int32_t ra_step, rw_step;      // int32 entries between one problem's sums and the next's; 0 = shared
};

bool umma_i8_batched_supported(const I8Problem& p, const I8Batch& b, const DeviceInfo& dev);
int launch_gemm_i8_umma_batched(const I8Problem& p, const I8Batch& b, const I8Epilogue& ep, const DeviceInfo& dev,
                                cudaStream_t stream);

}  // namespace nnb200
