// Q4_1 product with the weights as the 128-row operand in tensor memory (q4_1_rows_umma.cu).
#pragma once

#include "internal.cuh"

namespace nnb200 {

struct Q4RowsCall {
    const nnb200_q4_1_args* q;
    const void* a;      // f16 rows of the MMA: the activations, or (hi, lo) rows of f32 ones
    int64_t lda;        // elements between those rows
    bool hi_lo;
};

// Halves between the (hi, lo) rows of f32 activations: 16-byte rows.
inline int64_t q4_1_rows_split_pitch(int64_t k) { return (k + 7) / 8 * 8; }
bool q4_1_rows_umma_supported(const nnb200_q4_1_args& q);
// [m][k] f32 rows -> rows of 2 kp halves, the f16 parts followed by the f16 remainders (zeros past k);
// with kp == k that is 2 m rows of k halves, part and remainder in turn.
int launch_split_f32_to_f16(const float* a, int64_t lda, int64_t m, int64_t k, int64_t kp, void* out, const DeviceInfo& dev,
                            cudaStream_t stream);
int launch_q4_1_rows_umma(const Q4RowsCall& c, const DeviceInfo& dev, cudaStream_t stream);

}  // namespace nnb200
