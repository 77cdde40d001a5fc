// The int8 Linear when device memory is short: a weight off the 16-byte rule asks for scratch as large as
// itself; if that cannot be had the call goes out with the least it needs, and only if that fails too is
// the failure the caller's.  The library calls that need a GPU are faked here (the program's own
// definitions come before the shared library's); sizes come from the real ones.

#include "nnops_b200/nnops_api.hpp"
#include "nnb200.h"

#include <cstdio>
#include <cstdlib>
#include <vector>

using namespace nnops;

static size_t g_limit = 0;                 // largest allocation that succeeds
static std::vector<size_t> g_asked;
static nnb200_gemm_i8_args g_seen;
static int g_calls = 0;

extern "C" int nnb200_scratch_alloc_async(void** out, size_t bytes, void*)
{
    g_asked.push_back(bytes);
    *out = bytes <= g_limit ? std::aligned_alloc(256, (bytes + 255) / 256 * 256) : nullptr;
    return *out != nullptr ? NNB200_OK : NNB200_OUT_OF_MEMORY;
}

extern "C" int nnb200_scratch_free_async(void* p, void*)
{
    std::free(p);
    return NNB200_OK;
}

extern "C" int nnb200_is_device_pointer(const void*) { return 1; }

extern "C" int nnb200_gemm_i8(const nnb200_gemm_i8_args* a, void*)
{
    g_seen = *a;
    ++g_calls;
    return NNB200_OK;
}

static int g_failed = 0;
#define EXPECT(cond)                                                  \
    do {                                                              \
        if (!(cond)) {                                                \
            ++g_failed;                                               \
            std::printf("line %d: %s\n", __LINE__, #cond);            \
        }                                                             \
    } while (0)

static Status run(int32_t zero_point)
{
    constexpr int64_t m = 3, n = 5000, k = 2049;
    static std::vector<int8_t> a(m * k + 64), w(n * k + 64);
    static std::vector<int32_t> c(m * n);
    const int64_t as[] = {m, k}, ws[] = {n, k}, cs[] = {m, n};
    QuantParams qa;
    qa.scale = 0.5f;
    qa.zero_point = zero_point;
    qa.granularity = QuantGranularity::PerTensor;
    TensorView va(as, DataType::s8, a.data(), TensorLayout::Dense, qa);
    TensorView vw(ws, DataType::s8, w.data(), TensorLayout::Dense);
    TensorView vc(cs, DataType::s32, c.data(), TensorLayout::Dense);
    LinearAttributes attrs;
    attrs.output_dtype = DataType::s32;
    const auto op = Linear::create(attrs, Backend::CUDA);
    const TensorView in[] = {va, vw};
    g_asked.clear();
    g_calls = 0;
    return op->compute(vc, in);
}

int main()
{
    for (const int32_t zp : {0, 7}) {
        const size_t least = zp != 0 ? 256 + (5000 * 4 + 255) / 256 * 256 : 0;
        g_limit = size_t(1) << 40;
        EXPECT(run(zp) == Status::ok && g_calls == 1);
        EXPECT(g_seen.workspace_bytes > size_t(5000) * 2049);
        g_limit = size_t(1) << 20;
        EXPECT(run(zp) == Status::ok && g_calls == 1);
        EXPECT(g_seen.workspace_bytes == least && (g_seen.workspace != nullptr) == (least > 0));
        EXPECT(g_asked.size() == (least > 0 ? 2u : 1u));
    }
    g_limit = 0;
    EXPECT(run(7) != Status::ok && g_calls == 0);
    std::printf(g_failed == 0 ? "PASS\n" : "FAIL\n");
    return g_failed == 0 ? 0 : 1;
}
