// A batch of int8 products of one shape in one launch of the tile kernel (MatMul over heads).
//
// One launch per product left a problem of a few tiles alone on the device: 32 heads of
// 512 x 128 x 512 were 32 launches of 8 tiles each, on 148 SMs.  Here the persistent tile walk
// runs through the tiles of every product, and the operands are read through tensor maps with the
// batch as their third axis (the four-axis map of the convolution, its last axis 1); an operand
// that all products share has a batch axis of 1 and is always read at 0.

#include <cstring>
#include <mutex>

#include "gemm_i8_umma_batched.cuh"
#include "gemm_i8_umma_tile.cuh"

namespace nnb200 {

namespace {

template <int BN, int KIND>
int launch_batched_variant(const CUtensorMap& map_a, const CUtensorMap& map_w, const I8Epilogue& ep, int m, int n, int k,
                           uint32_t idesc, int vec_ok, const BatchTile& batch, const DeviceInfo& dev, cudaStream_t stream)
{
    using Cfg = TileConfig<BN, 0, KIND>;
    auto kernel = gemm_i8_umma_kernel<BN, KIND, 0, false, true>;
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
    const int num_m = (m + kBlockM - 1) / kBlockM;
    const int64_t num_tiles = static_cast<int64_t>(batch.count) * num_m * ((n + BN - 1) / BN);
    const int grid = num_tiles < dev.sm_count ? static_cast<int>(num_tiles) : dev.sm_count;
    const cudaError_t launched = launch_overlapping(kernel, dim3(static_cast<unsigned>(grid)), dim3(tile_threads(KIND, 0)), Cfg::kSmemBytes, stream, 1,
                                                    map_a, map_w, maps, ep, m, n, k, idesc, vec_ok, num_m, 0, dev.error_word, batch);
    note_launch();
    return cuda_status(launched);
}

template <int BN>
int launch_batched_bn(const CUtensorMap& map_a, const CUtensorMap& map_w, const I8Epilogue& ep, int m, int n, int k,
                      uint32_t idesc, int vec_ok, const BatchTile& b, const DeviceInfo& dev, cudaStream_t stream)
{
    switch (ep.out_kind) {
    case NNB200_OUT_S32: return launch_batched_variant<BN, NNB200_OUT_S32>(map_a, map_w, ep, m, n, k, idesc, vec_ok, b, dev, stream);
    case NNB200_OUT_S8: return launch_batched_variant<BN, NNB200_OUT_S8>(map_a, map_w, ep, m, n, k, idesc, vec_ok, b, dev, stream);
    case NNB200_OUT_U8: return launch_batched_variant<BN, NNB200_OUT_U8>(map_a, map_w, ep, m, n, k, idesc, vec_ok, b, dev, stream);
    case NNB200_OUT_F32: return launch_batched_variant<BN, NNB200_OUT_F32>(map_a, map_w, ep, m, n, k, idesc, vec_ok, b, dev, stream);
    case NNB200_OUT_F16: return launch_batched_variant<BN, NNB200_OUT_F16>(map_a, map_w, ep, m, n, k, idesc, vec_ok, b, dev, stream);
    default: return NNB200_UNSUPPORTED;
    }
}

// {contiguous index, the other index, batch, 1} of one operand.
bool make_operand_map(CUtensorMap* map, const void* base, int64_t contiguous, int64_t rows, int64_t pitch, int64_t count,
                      int64_t batch_stride, uint32_t box_rows)
{
    const uint64_t z = batch_stride != 0 ? static_cast<uint64_t>(count) : 1u;
    // The step of an axis of one entry is never taken; any multiple of 16 will do.
    const uint64_t step_z = z > 1 ? static_cast<uint64_t>(batch_stride) : static_cast<uint64_t>(pitch);
    return make_tma_nhwc_u8(map, base, static_cast<uint64_t>(contiguous), static_cast<uint64_t>(rows), z, 1,
                            static_cast<uint64_t>(pitch), step_z, step_z, kBlockKBytes, box_rows, 1);
}

}  // namespace

bool umma_i8_batched_supported(const I8Problem& p, const I8Batch& b, const DeviceInfo& dev)
{
    if (!umma_i8_supported(p) || b.count < 2 || b.count > INT32_MAX || b.a_stride < 0 || b.w_stride < 0 ||
        (b.a_stride & 15) != 0 || (b.w_stride & 15) != 0) {
        return false;
    }
    // A tensor map's strides stay below 2^40 bytes.
    constexpr int64_t kMostStride = int64_t{1} << 40;
    if (b.a_stride >= kMostStride || b.w_stride >= kMostStride) {
        return false;
    }
    // Few rows against a large weight: each product is a stream of its own that the engines for few
    // rows spread over all SMs, and long enough to pay for its launch.
    if (p.m <= kBlockM && p.n * p.k >= (int64_t{8} << 20)) {
        return false;
    }
    // One problem that fills the device by itself has more to gain from the forms for large
    // problems (CTA pairs, wider tiles) than from sharing a launch.  Below that the shared launch is
    // never the slower one, pairs or not (us, one launch a product / one for all: 2 x 1280 x 3584 x 4096 36.9 /
    // 32.4, 4 of them 81.4 / 63.5, 2 x 4096 x 1024 x 8192 58.0 / 58.2, 2 x 640 x 7168 x 16384 176 / 118).
    const int64_t tiles = ((p.m + kBlockM - 1) / kBlockM) * ((p.n + 255) / 256);
    return tiles < dev.sm_count && tiles * 4 * b.count < INT32_MAX;
}

int launch_gemm_i8_umma_batched(const I8Problem& p, const I8Batch& b, const I8Epilogue& ep, const DeviceInfo& dev,
                                cudaStream_t stream)
{
    const int m = static_cast<int>(p.m);
    const int n = static_cast<int>(p.n);
    const int k = static_cast<int>(p.k);
    const bool a_mn = p.a_stride_k != 1;
    const bool w_mn = p.w_stride_k != 1;
    // Tile width: the least time over whole waves, a tile costing its columns plus about 64 more for
    // its share of the main loop's start and the walk.  An MN-major W tile is whole 128-column blocks.
    int bn = 256;
    int64_t best = -1;
    for (const int width : {256, 128, 64}) {
        if (width == 64 && w_mn) {
            continue;
        }
        const int64_t tiles = b.count * ((m + kBlockM - 1) / kBlockM) * ((n + width - 1) / width);
        const int64_t cost = (tiles + dev.sm_count - 1) / dev.sm_count * (width + 64);
        if (best < 0 || cost < best) {
            best = cost;
            bn = width;
        }
    }
    CUtensorMap map_a, map_w;
    const bool ok = (a_mn ? make_operand_map(&map_a, p.a, m, k, p.a_stride_k, b.count, b.a_stride, kBlockKBytes)
                          : make_operand_map(&map_a, p.a, k, m, p.a_stride_m, b.count, b.a_stride, kBlockM)) &&
                    (w_mn ? make_operand_map(&map_w, p.w, n, k, p.w_stride_k, b.count, b.w_stride, kBlockKBytes)
                          : make_operand_map(&map_w, p.w, k, n, p.w_stride_n, b.count, b.w_stride, static_cast<uint32_t>(bn)));
    if (!ok) {
        return NNB200_INTERNAL;
    }
    const int elem = (ep.out_kind == NNB200_OUT_S32 || ep.out_kind == NNB200_OUT_F32) ? 4 : (ep.out_kind == NNB200_OUT_F16 ? 2 : 1);
    BatchTile t;
    t.count = static_cast<int32_t>(b.count);
    t.a_step = b.a_stride != 0 ? 1 : 0;
    t.w_step = b.w_stride != 0 ? 1 : 0;
    t.ra_step = b.ra_step;
    t.rw_step = b.rw_step;
    t.out_step = b.out_stride * elem;
    // Destination vector stores: bit 0 = 16-byte aligned base, row pitch and batch step, bit 1 = 32-byte;
    // bits 4-5: operand poses, read by the kernel.
    const uint64_t out_bits = reinterpret_cast<uintptr_t>(ep.out) | (static_cast<uint64_t>(ep.ldc) * elem) |
                              static_cast<uint64_t>(t.out_step);
    const int vec_ok = ((out_bits & 15u) == 0 ? 1 : 0) | ((out_bits & 31u) == 0 ? 2 : 0) | (a_mn ? 16 : 0) | (w_mn ? 32 : 0);
    const uint32_t idesc = umma_idesc(2, p.a_unsigned ? 0u : 1u, 1, kBlockM, bn) | (a_mn ? kUmmaAMajorMN : 0u) |
                           (w_mn ? kUmmaBMajorMN : 0u);
    switch (bn) {
    case 256: return launch_batched_bn<256>(map_a, map_w, ep, m, n, k, idesc, vec_ok, t, dev, stream);
    case 128: return launch_batched_bn<128>(map_a, map_w, ep, m, n, k, idesc, vec_ok, t, dev, stream);
    default: return launch_batched_bn<64>(map_a, map_w, ep, m, n, k, idesc, vec_ok, t, dev, stream);
    }
}

}  // namespace nnb200
