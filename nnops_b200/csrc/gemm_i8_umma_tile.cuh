// The tile kernel of the int8 GEMM: its geometry, its fused epilogue and the single-CTA kernel with
// its sharded, convolution and batched forms.  Included by the translation units that launch it;
// the overview stands at the top of gemm_i8_umma.cu.
#pragma once

#include <cuda_fp16.h>

#include <type_traits>

#include "internal.cuh"
#include "ptx.cuh"

namespace nnb200 {

namespace {

constexpr int kBlockM = 128;
constexpr int kBlockKBytes = 128;  // one 128-byte swizzle row of K per stage
constexpr int kUmmaK = 32;         // K per tcgen05.mma for 8-bit operands
// TMA warp, MMA warp, then the epilogue warps.  The sharded form has four, whose staging tiles are per
// warp; elsewhere there are two per TMEM lane quarter, each draining half of the tile's columns: one
// warp per scheduler issues an instruction every ~4 cycles on the epilogue's dependent chains, and
// with four warps a 128 x 256 tile took ~17k cycles to drain, which hid behind the main loop only
// from K = 4096 up.
constexpr int kMaxThreads = 320;
__host__ __device__ constexpr int epilogue_warps(int peers) { return peers ? 4 : 8; }
__host__ __device__ constexpr int num_threads(int peers) { return (2 + epilogue_warps(peers)) * 32; }
// The single-CTA kernel's 8-bit destinations have sixteen.  Up to 256 columns they form two groups, each
// with an accumulator of its own, that take the tiles in turn: of the ~6600 cycles eight warps needed
// for a 128 x 256 tile, ~2300 passed between two tiles (column terms, row terms, barriers) with nothing
// to issue, and the drain itself kept the schedulers less than two thirds busy.  A wider tile, the only
// one of its CTA, is drained by four warps per lane quarter.  100352 x 1024 x 256 77.5 -> 63.6 us,
// 32768 x 4096 x 256 97.2 -> 78.8, 8192 x 4096 x 1024 33.8 -> 31.3, 512 x 11008 x 4096 (320 wide) 24.6 -> 24.0.
// The floating destinations hold twice the values per chunk in registers and keep eight.
__host__ __device__ constexpr bool sixteen_warps(int kind, int peers)
{
    return peers == 0 && (kind == NNB200_OUT_S8 || kind == NNB200_OUT_U8);
}
__host__ __device__ constexpr int tile_epilogue_warps(int kind, int peers) { return sixteen_warps(kind, peers) ? 16 : epilogue_warps(peers); }
__host__ __device__ constexpr int tile_threads(int kind, int peers) { return (2 + tile_epilogue_warps(kind, peers)) * 32; }
// Columns drained by the first of the two warps of a lane quarter (whole 32-column chunks).
__host__ __device__ constexpr int first_half_cols(int bn, int peers) { return peers ? bn : ((bn / 32 + 1) / 2) * 32; }

// TMA descriptors of the output windows the sharded form writes: [0] this GPU's, then the peers'.
struct alignas(64) PeerMaps {
    CUtensorMap m[8];
};

// Geometry of the implicit-GEMM convolution (CONV kernels): an M tile is a patch of bh x bw
// output pixels of one image, its A operand for the k-block (tap, 128 channels) one 4-D TMA
// box of the NHWC activation shifted by the tap -- what lies outside the image is filled with
// zeros, and rows whose window overhangs get the zero point's share added back in the epilogue.
struct ConvTile {
    int32_t oh, ow, ih, iw;
    int32_t kh, kw, dh, dw, ph, pw;
    int32_t sh, sw;                // window strides (1 or 2): the tensor map's element strides along h and w
    int32_t bw_log2, bh;           // patch: bh rows x (1 << bw_log2) columns, 128 pixels
    int32_t tiles_w, tiles_h;      // patches per image
    int32_t c_base;                // first channel of this group in the activation
    int32_t kb_per_tap;            // 128-channel k-blocks per tap
    int32_t zp_x;                  // activation zero point (0: no correction)
    int32_t wtap_ld;               // output channels of the whole filter (row length of the tables)
    // Border classes: the distinct masks of out-of-image taps along each axis (at most eight
    // each); class (i, j) -- i, j = 1 + index of the row's masks, 0 = none -- has a table row
    // holding the sum of the per-tap channel sums of the filter over the taps it loses.
    int32_t nh, nw;
    uint32_t mask_h[8], mask_w[8];
    const int32_t* border;         // [(nh + 1) * (nw + 1)][wtap_ld], at this group's first column
    int32_t m_tiles;               // patches in all (batch * tiles_h * tiles_w)
};

// Patch m_blk = (image, th, tw); a patch index past m_tiles (the second half of an odd pair)
// decodes to an image past the batch: its loads are all fill, its rows are not stored.
struct ConvPatch {
    int img, th, tw;
};

__device__ __forceinline__ ConvPatch conv_patch(const ConvTile& conv, int m_blk)
{
    ConvPatch p;
    p.tw = m_blk % conv.tiles_w;
    const int t2 = m_blk / conv.tiles_w;
    p.th = t2 % conv.tiles_h;
    p.img = t2 / conv.tiles_h;
    return p;
}

// Row r of a patch: its output pixel's flat index, whether it exists, and -- with a non-zero
// activation zero point -- the row's border class along each axis (0: every tap inside).
struct ConvRow {
    int64_t m;
    bool ok;
    uint32_t bad_h, bad_w;
};

__device__ __forceinline__ ConvRow conv_row(const ConvTile& conv, int m_blk, int r)
{
    const ConvPatch p = conv_patch(conv, m_blk);
    const int y = p.th * conv.bh + (r >> conv.bw_log2);
    const int x = (p.tw << conv.bw_log2) + (r & ((1 << conv.bw_log2) - 1));
    ConvRow o;
    o.ok = m_blk < conv.m_tiles && y < conv.oh && x < conv.ow;
    o.m = (static_cast<int64_t>(p.img) * conv.oh + y) * conv.ow + x;
    o.bad_h = 0;
    o.bad_w = 0;
    if (conv.zp_x != 0 && o.ok) {
        uint32_t lost_h = 0, lost_w = 0;
        for (int a = 0; a < conv.kh; ++a) {
            const int iy = y * conv.sh - conv.ph + a * conv.dh;
            lost_h |= (iy < 0 || iy >= conv.ih) ? (1u << a) : 0u;
        }
        for (int b = 0; b < conv.kw; ++b) {
            const int ix = x * conv.sw - conv.pw + b * conv.dw;
            lost_w |= (ix < 0 || ix >= conv.iw) ? (1u << b) : 0u;
        }
        // 1 + index of the mask among the axis's classes (0 = no tap lost).
        for (int q = 0; q < conv.nh; ++q) {
            o.bad_h = (lost_h != 0 && conv.mask_h[q] == lost_h) ? static_cast<uint32_t>(q + 1) : o.bad_h;
        }
        for (int q = 0; q < conv.nw; ++q) {
            o.bad_w = (lost_w != 0 && conv.mask_w[q] == lost_w) ? static_cast<uint32_t>(q + 1) : o.bad_w;
        }
    }
    return o;
}

// A tap outside the image was loaded as 0 where the reference's gather holds the zero point:
// add zp_x * (that tap's channel sum of the filter) back, from the row's class in the table.
__device__ __forceinline__ void conv_border_fix(const ConvTile& conv, uint32_t (&v)[32], uint32_t bad_h, uint32_t bad_w,
                                                int n0, int n_total)
{
    if ((bad_h | bad_w) == 0) {
        return;
    }
    const int32_t* tb = conv.border + static_cast<int64_t>(bad_h * (conv.nw + 1) + bad_w) * conv.wtap_ld + n0;
    if (n0 + 32 <= n_total && (reinterpret_cast<uintptr_t>(tb) & 15u) == 0) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
            const int4 t4 = *reinterpret_cast<const int4*>(tb + j);
            v[j] += static_cast<uint32_t>(conv.zp_x) * static_cast<uint32_t>(t4.x);
            v[j + 1] += static_cast<uint32_t>(conv.zp_x) * static_cast<uint32_t>(t4.y);
            v[j + 2] += static_cast<uint32_t>(conv.zp_x) * static_cast<uint32_t>(t4.z);
            v[j + 3] += static_cast<uint32_t>(conv.zp_x) * static_cast<uint32_t>(t4.w);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            if (n0 + j < n_total) {
                v[j] += static_cast<uint32_t>(conv.zp_x) * static_cast<uint32_t>(tb[j]);
            }
        }
    }
}

template <int BN, int PEERS = 0, int KIND = NNB200_OUT_S32>
struct TileConfig {
    static constexpr int kEpilogueWarps = tile_epilogue_warps(KIND, PEERS);
    static constexpr int kGroups = (kEpilogueWarps == 16 && BN <= 256) ? 2 : 1;   // groups that take the tiles in turn
    static constexpr int kColParts = kEpilogueWarps / 4 / kGroups;                 // warps per lane quarter and group
    // Tiles wider than 256 columns (single-wave form, see launch_gemm_i8_umma) are issued as two
    // MMAs of BN / 2 columns over one A tile and keep ONE accumulator: a CTA owns exactly one tile.
    static constexpr int kNSplit = BN > 256 ? 2 : 1;
    static constexpr int kMmaN = BN / kNSplit;
    static constexpr int kATileBytes = kBlockM * kBlockKBytes;
    static constexpr int kBTileBytes = BN * kBlockKBytes;
    static constexpr int kStageBytes = kATileBytes + kBTileBytes;
    // Ring depth: as many stages as fit beside the epilogue staging in ~200 KB.
    static constexpr int kStages = PEERS ? ((BN == 256) ? (PEERS == 1 ? 4 : 3) : (BN == 224 ? 4 : 5))
                                   : (BN > 256) ? (BN > 384 ? 2 : 3)
                                                : ((BN > 128) ? 4 : (BN == 128 ? 6 : 8));
    // Two accumulators BN columns apart (one when BN > 256); a power of two of at least that.
    static constexpr int kTmemCols = BN > 128 ? 512 : 2 * BN;
    // Per epilogue warp {scale, bias, r_w, zp_w} of the columns it drains, 4 B each.
    static constexpr int kPartCols = (BN / 32 + kColParts - 1) / kColParts * 32;   // the last part may be narrower
    static constexpr int kColParamBytes = kEpilogueWarps * 4 * kPartCols * 4;
    static constexpr int kBarrierBytes = (2 * kStages + 4) * 8 + 16;
    // Sharded form (PEERS = 2): two staging tiles of 32 rows x 128 B per epilogue warp, one being
    // filled while the other is being stored.  With few peers (PEERS = 1, used up to three) the
    // stores are not what saturates first and the main loop decides: one staging tile per warp,
    // and the shared memory that frees keeps the ring at four stages.
    // (Rows of 256 bytes per bulk store from a plain 32 x 256 tile were tried: no change on four
    // GPUs at the same ring depth.)
    static constexpr int kStageTiles = PEERS == 2 ? 2 : 1;
    static constexpr int kStageGroupCols = 128;   // columns per staging tile
    static constexpr int kPeerStageBytes = PEERS ? 4 * kStageTiles * 32 * kStageGroupCols : 0;
    static constexpr int kSmemBytes =
        1024 /*alignment slack*/ + kStages * kStageBytes + kPeerStageBytes + kColParamBytes + kBarrierBytes;
    static_assert(kSmemBytes <= 227 * 1024, "shared memory");
};

// A batch of equal problems in one launch (BATCH kernels).  Steps are 0 where the operand is shared.
struct BatchTile {
    int32_t count;
    int32_t a_step, w_step;        // 1, or 0 for an operand that every problem shares
    int32_t ra_step, rw_step;      // int32 entries between the sums of one problem and the next
    int64_t out_step;              // bytes between outputs
};

struct TileCoord {
    int m_blk;
    int n_blk;
};

// Where a tile's walk over the K blocks starts.  Integer accumulation does not depend on the order
// of the K blocks, so each tile may start somewhere else: CTAs that share an operand tile (every
// CTA of a wave when N is one tile wide, as in a convolution's GEMM) then ask the L2 for
// different lines at any one time instead of all for the same ones.  k_rot == 0 keeps 0.
__device__ __forceinline__ int k_rotation(int tile, int k_rot, int num_kb)
{
    return k_rot == 0 ? 0 : static_cast<int>((static_cast<unsigned>(tile) * static_cast<unsigned>(k_rot)) % static_cast<unsigned>(num_kb));
}

// Division of a number below 2^31 by a fixed divisor as a multiply and a shift (the GPU has no
// integer divider: a plain `/` is a chain of some thirty dependent instructions, and the tile
// walk below needs three of them per tile in every role's loop).
struct FastDiv {
    uint32_t mul, shift;
    __device__ __forceinline__ void init(uint32_t d)
    {
        shift = d > 1 ? 32u - static_cast<uint32_t>(__clz(static_cast<int>(d - 1))) : 0u;
        mul = static_cast<uint32_t>(((static_cast<uint64_t>(1) << 32) * ((static_cast<uint64_t>(1) << shift) - d)) / d + 1);
    }
    __device__ __forceinline__ uint32_t div(uint32_t n) const { return (__umulhi(n, mul) + n) >> shift; }
};

// Tiles are walked m-fastest inside groups of `group_m` m-blocks, groups n-fastest: the CTAs of
// one wave then share a band of A (kept in L2 for the whole pass over N) while W streams by once
// per group.  The last group may hold fewer m-blocks.
struct TileWalk {
    int num_m, group_m, group_size, last_gm;
    FastDiv by_group, by_gm, by_last_gm;
    __device__ __forceinline__ TileWalk(int num_m_, int num_n, int group_m_)
    {
        num_m = num_m_;
        group_m = group_m_ < num_m_ ? group_m_ : (num_m_ > 0 ? num_m_ : 1);
        group_size = group_m * num_n;
        const int groups = (num_m + group_m - 1) / group_m;
        last_gm = num_m - (groups - 1) * group_m;
        last_gm = last_gm > 0 ? last_gm : 1;
        by_group.init(static_cast<uint32_t>(group_size > 0 ? group_size : 1));
        by_gm.init(static_cast<uint32_t>(group_m));
        by_last_gm.init(static_cast<uint32_t>(last_gm));
    }
    __device__ __forceinline__ TileCoord operator()(int tile) const
    {
        const int group = static_cast<int>(by_group.div(static_cast<uint32_t>(tile)));
        const int first_m = group * group_m;
        const int in_group = tile - group * group_size;
        const bool last = num_m - first_m < group_m;
        const int gm = last ? last_gm : group_m;
        TileCoord c;
        c.n_blk = static_cast<int>(last ? by_last_gm.div(static_cast<uint32_t>(in_group))
                                        : by_gm.div(static_cast<uint32_t>(in_group)));
        c.m_blk = first_m + in_group - c.n_blk * gm;
        return c;
    }
};

// The per-column terms of the epilogue as one epilogue warp stages them in shared memory.
struct ColTerms {
    float scale;     // s_w[n], or (s_a / s_out) * s_w[n] when the row factor is folded in
    int32_t bias;    // int32 bias (integer destinations) or the fp bias as bits; with fold_comp also -zp_a * R_w[n]
    int32_t rw;      // R_w[n] when compensation is live
    int32_t zpw;     // zp_w[n]
};

// The loads only, so that they can be issued a tile ahead: nothing here depends on a loaded
// value (an f16 bias stays as its 16 bits).  finish_col_terms() does the arithmetic when the
// terms are staged.
template <int KIND>
__device__ __forceinline__ ColTerms load_col_terms(const I8Epilogue& ep, int n, int n_total)
{
    ColTerms c;
    const bool in = n < n_total;
    c.scale = ep.scale_w_scalar;
    if (in && ep.scale_w != nullptr) {
        c.scale = ep.scale_w[n];
    }
    c.bias = 0;
    if (in && ep.bias != nullptr) {
        if constexpr (KIND <= NNB200_OUT_U8) {
            c.bias = static_cast<const int32_t*>(ep.bias)[n];
        } else if constexpr (KIND == NNB200_OUT_F32) {
            c.bias = __float_as_int(static_cast<const float*>(ep.bias)[n]);
        } else {
            c.bias = static_cast<int32_t>(static_cast<const uint16_t*>(ep.bias)[n]);
        }
    }
    c.rw = 0;
    if (in && ep.compensate && ep.r_w != nullptr) {
        c.rw = ep.r_w[n];
    }
    c.zpw = ep.zp_w_scalar;
    if (in && ep.zp_w != nullptr) {
        c.zpw = ep.zp_w[n];
    }
    return c;
}

// fold_scale: the per-tensor row factor s_a / s_out goes into the column scale.
// fold_comp: a per-tensor activation zero point against weights whose zero points are all 0 -- the
// only live compensation term is -zp_a * R_w[n], a column constant, and goes into the bias.
template <int KIND>
__device__ __forceinline__ ColTerms finish_col_terms(const I8Epilogue& ep, ColTerms c, bool fold_scale, float folded_row_k,
                                                     bool fold_comp)
{
    if (fold_scale) {
        c.scale = __fmul_rn(folded_row_k, c.scale);
    }
    if constexpr (KIND == NNB200_OUT_F16) {
        c.bias = __float_as_int(__half2float(__ushort_as_half(static_cast<unsigned short>(c.bias))));
    }
    if (fold_comp) {
        c.bias = static_cast<int32_t>(static_cast<uint32_t>(c.bias) -
                                      static_cast<uint32_t>(ep.zp_a_scalar) * static_cast<uint32_t>(c.rw));
    }
    return c;
}

// Four requantised 8-bit values in one word, first value in the low byte.  Same bytes as four
// i8_requant() calls, with fewer instructions: that routine clamps x = float(v) * req to
// [lo - zp, hi - zp], rounds half away from zero as trunc(x + copysign(0.5, x)) and adds zp;
// the bounds are integers, so clamping before the rounding or saturating after it (and after
// the zero-point add) gives the same value.  Here the 8-bit saturation rides the packing
// instruction; with a non-zero zero point x is first kept inside +-32000 so that the add cannot
// overflow, with ZP0 (out_zp == 0, the usual s8 destination) not even that is needed.
template <bool U8, bool ZP0>
__device__ __forceinline__ uint32_t requant_pack4(const int32_t (&v)[4], const float (&req)[4], int32_t zp)
{
    int32_t r[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        float x = __fmul_rn(__int2float_rn(v[b]), req[b]);
        if constexpr (ZP0) {
            // The conversion itself saturates at the int32 range; nothing is added afterwards.
            r[b] = __float2int_rz(__fadd_rn(x, copysignf(0.5f, x)));
        } else {
            x = fminf(fmaxf(x, -32000.0f), 32000.0f);
            r[b] = __float2int_rz(__fadd_rn(x, copysignf(0.5f, x))) + zp;
        }
    }
    uint32_t hi, out;
    if constexpr (U8) {
        asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(r[3]), "r"(r[2]), "r"(0));
        asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(out) : "r"(r[1]), "r"(r[0]), "r"(hi));
    } else {
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(r[3]), "r"(r[2]), "r"(0));
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(out) : "r"(r[1]), "r"(r[0]), "r"(hi));
    }
    return out;
}

// 32 bytes to a destination of any alignment.  Rows whose pitch 16 does not divide used to go out a byte
// at a time, 32 scattered stores a lane and chunk (2000 x 1000 x 128, 8-bit: 25.7 -> 6.7 us).
__device__ __forceinline__ void store_32_bytes_anywhere(uint8_t* dst, const uint32_t (&w)[8])
{
    const uint32_t at = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(dst));
    if ((at & 7u) == 0) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            reinterpret_cast<uint2*>(dst)[j] = make_uint2(w[2 * j], w[2 * j + 1]);
        }
        return;
    }
    // `head` bytes up to the first word boundary, whole words assembled across the seams, the rest.
    const uint32_t head = (4u - (at & 3u)) & 3u;
#pragma unroll
    for (uint32_t b = 0; b < 3; ++b) {
        if (b < head) {
            dst[b] = static_cast<uint8_t>(w[0] >> (8 * b));
        }
    }
    uint32_t* words = reinterpret_cast<uint32_t*>(dst + head);
#pragma unroll
    for (int j = 0; j < 7; ++j) {
        words[j] = __funnelshift_r(w[j], w[j + 1], 8 * head);
    }
    if (head == 0) {
        words[7] = w[7];
    } else {
#pragma unroll
        for (uint32_t b = 1; b < 4; ++b) {
            if (b >= head) {
                dst[28 + b] = static_cast<uint8_t>(w[7] >> (8 * b));
            }
        }
    }
}

// Epilogue of one 32-column chunk of one row.  `acc` holds the raw int32 sums of columns
// n0..n0+31; col_* point at the chunk's staged per-column terms in shared memory.
template <int KIND>
__device__ __forceinline__ void epilogue_chunk(const I8Epilogue& e, const I8RowTerms& t, const uint32_t (&acc)[32],
                                               int64_t m, bool row_ok, int n0, int n_total,
                                               const float* col_scale, const int32_t* col_bias,
                                               const int32_t* col_rw, const int32_t* col_zpw, int vec,
                                               bool scale_folded = false, bool plain = false)
{
    // plain: no per-element compensation terms are needed -- either every zero point is 0, or
    // the only live term (-zp_a * R_w[n], a per-tensor activation zero point against symmetric
    // weights) was folded into the staged column bias.
    // vec: bit 0 = the destination takes 16-byte stores, bit 1 = 32-byte stores as well.
    const bool vec_ok = (vec & 1) != 0;
    const bool vec32 = (vec & 2) != 0;
    const bool full = n0 + 32 <= n_total;
    const float zpf = static_cast<float>(e.out_zp);

    if constexpr (KIND == NNB200_OUT_S32) {
        int32_t o[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
            o[j] = i8_int_value(e, t, static_cast<int32_t>(acc[j]), col_zpw[j], col_rw[j], col_bias[j]);
        }
        if (!row_ok) {
            return;
        }
        int32_t* dst = static_cast<int32_t*>(e.out) + m * e.ldc + n0;
        if (full && vec32) {
            // The lane's 128 bytes as four 256-bit stores (whole 32-byte sectors).
#pragma unroll
            for (int j = 0; j < 32; j += 8) {
                st_global_32(dst + j, static_cast<uint32_t>(o[j]), static_cast<uint32_t>(o[j + 1]), static_cast<uint32_t>(o[j + 2]),
                             static_cast<uint32_t>(o[j + 3]), static_cast<uint32_t>(o[j + 4]), static_cast<uint32_t>(o[j + 5]),
                             static_cast<uint32_t>(o[j + 6]), static_cast<uint32_t>(o[j + 7]));
            }
        } else if (full && vec_ok) {
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                *reinterpret_cast<int4*>(dst + j) = make_int4(o[j], o[j + 1], o[j + 2], o[j + 3]);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (n0 + j < n_total) {
                    dst[j] = o[j];
                }
            }
        }
    } else if constexpr (KIND == NNB200_OUT_S8 || KIND == NNB200_OUT_U8) {
        const float lo = (KIND == NNB200_OUT_S8 ? -128.0f : 0.0f) - zpf;
        const float hi = (KIND == NNB200_OUT_S8 ? 127.0f : 255.0f) - zpf;
        uint32_t packed[8];
        if (!e.compensate || plain) {
            // Common case: with a per-tensor activation scale the staged column scales already
            // carry (s_a / s_out) * s_w[n].  The column terms are read four at a time.
            (void)lo;
            (void)hi;
            // Branch-free per element: the run-time switches become operands (a lower bound for
            // the ReLU, a row factor of exactly 1 when the scale is already folded -- x * 1.0f is
            // x), and the zero-point variant is chosen once per chunk.
            const int32_t relu_lo = e.relu ? 0 : INT32_MIN;
            const float row_k = scale_folded ? 1.0f : t.row_k;
            const auto body = [&](auto zp0_tag) {
                constexpr bool kZp0 = decltype(zp0_tag)::value;
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    const int4 b4 = *reinterpret_cast<const int4*>(col_bias + j);
                    const float4 s4 = *reinterpret_cast<const float4*>(col_scale + j);
                    const int32_t bias4[4] = {b4.x, b4.y, b4.z, b4.w};
                    const float scale4[4] = {s4.x, s4.y, s4.z, s4.w};
                    int32_t v[4];
                    float req[4];
#pragma unroll
                    for (int b = 0; b < 4; ++b) {
                        v[b] = max(static_cast<int32_t>(static_cast<uint32_t>(acc[j + b]) + static_cast<uint32_t>(bias4[b])),
                                   relu_lo);
                        req[b] = __fmul_rn(row_k, scale4[b]);
                    }
                    packed[j / 4] = requant_pack4<KIND == NNB200_OUT_U8, kZp0>(v, req, e.out_zp);
                }
            };
            if (e.out_zp == 0) {
                body(std::true_type{});
            } else {
                body(std::false_type{});
            }
        } else {
            // Compensation live (zero points on both sides, or per-row ones): the integer terms, then
            // the same packed requantisation, one loop for every zero point (more code here slows
            // the common path above measurably).
            (void)lo;
            (void)hi;
            const int32_t relu_lo = e.relu ? 0 : INT32_MIN;
            const float row_k = scale_folded ? 1.0f : t.row_k;
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                int32_t v[4];
                float req[4];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int32_t c = i8_compensate(static_cast<int32_t>(acc[j + b]), t.zpa, col_zpw[j + b], t.ra,
                                                    col_rw[j + b], e.k);
                    v[b] = max(static_cast<int32_t>(static_cast<uint32_t>(c) + static_cast<uint32_t>(col_bias[j + b])),
                               relu_lo);
                    req[b] = __fmul_rn(row_k, col_scale[j + b]);
                }
                packed[j / 4] = requant_pack4<KIND == NNB200_OUT_U8, false>(v, req, e.out_zp);
            }
        }
        if (!row_ok) {
            return;
        }
        uint8_t* dst = static_cast<uint8_t*>(e.out) + m * e.ldc + n0;
        if (full && vec32) {
            // The lane's 32 values are exactly one 32-byte sector of its row.
            st_global_32(dst, packed[0], packed[1], packed[2], packed[3], packed[4], packed[5], packed[6], packed[7]);
            // Two-rank shards: the same sector into the other rank's copy, over the link (the
            // launcher has checked that every chunk is full and every pointer 32-byte aligned).
            for (int d = 0; d < e.direct_peers; ++d) {
                st_global_32(static_cast<uint8_t*>(e.peer_out[d]) + m * e.ldc + n0, packed[0], packed[1], packed[2],
                             packed[3], packed[4], packed[5], packed[6], packed[7]);
            }
        } else if (full && vec_ok) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            *reinterpret_cast<uint4*>(dst + 16) = make_uint4(packed[4], packed[5], packed[6], packed[7]);
        } else if (full) {
            store_32_bytes_anywhere(dst, packed);
        } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                if (n0 + j < n_total) {
                    dst[j] = static_cast<uint8_t>(packed[j / 4] >> (8 * (j % 4)));
                }
            }
        }
    } else {  // F32 / F16
        // One loop per (compensation live?, activation class): the run-time switches are taken
        // once per chunk, not once per element.  With a per-tensor activation scale the staged
        // column scale already carries s_a * s_w[n] (row factor exactly 1: x * 1.0f is x).
        const float row_s = scale_folded ? 1.0f : t.s_a;
        float o[32];
        const auto body = [&](auto comp_tag, auto act_tag) {
            constexpr bool kComp = decltype(comp_tag)::value;
            constexpr int kAct = decltype(act_tag)::value;   // 0 none, 1 Relu, 2 any other, 3 Gelu
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
                const int4 b4 = *reinterpret_cast<const int4*>(col_bias + j);
                const float4 s4 = *reinterpret_cast<const float4*>(col_scale + j);
                const float bias4[4] = {__int_as_float(b4.x), __int_as_float(b4.y), __int_as_float(b4.z), __int_as_float(b4.w)};
                const float scale4[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    int32_t v = static_cast<int32_t>(acc[j + b]);
                    if constexpr (kComp) {
                        v = i8_compensate(v, t.zpa, col_zpw[j + b], t.ra, col_rw[j + b], e.k);
                    }
                    float f = __fmul_rn(__int2float_rn(v), __fmul_rn(row_s, scale4[b]));
                    const float fb = __fadd_rn(f, bias4[b]);
                    f = bias4[b] != 0.0f ? fb : f;   // a zero bias is not added (-0 stays -0)
                    f = fminf(fmaxf(f, e.min_clip), e.max_clip);
                    if constexpr (kAct == 1) {
                        f = fmaxf(f, 0.0f);
                    } else if constexpr (kAct == 2) {
                        f = act_apply(e.activation, e.act_alpha, e.act_beta, f);
                    } else if constexpr (kAct == 3) {
                        f = act_apply(NNB200_ACT_GELU, e.act_alpha, e.act_beta, f);   // the switch folds away
                    }
                    o[j + b] = f;
                }
            }
        };
        // Gelu (the usual partner of a Linear) gets a loop of its own; the remaining activations
        // share one with the switch inside.
        const int act_class = e.activation == NNB200_ACT_NONE ? 0
                              : e.activation == NNB200_ACT_RELU ? 1
                              : e.activation == NNB200_ACT_GELU ? 3 : 2;
        if (e.compensate) {
            if (act_class == 0) {
                body(std::true_type{}, std::integral_constant<int, 0>{});
            } else if (act_class == 1) {
                body(std::true_type{}, std::integral_constant<int, 1>{});
            } else {
                body(std::true_type{}, std::integral_constant<int, 2>{});
            }
        } else {
            if (act_class == 0) {
                body(std::false_type{}, std::integral_constant<int, 0>{});
            } else if (act_class == 1) {
                body(std::false_type{}, std::integral_constant<int, 1>{});
            } else if (act_class == 3) {
                body(std::false_type{}, std::integral_constant<int, 3>{});
            } else {
                body(std::false_type{}, std::integral_constant<int, 2>{});
            }
        }
        if (!row_ok) {
            return;
        }
        if constexpr (KIND == NNB200_OUT_F32) {
            float* dst = static_cast<float*>(e.out) + m * e.ldc + n0;
            if (full && vec32) {
#pragma unroll
                for (int j = 0; j < 32; j += 8) {
                    st_global_32(dst + j, __float_as_uint(o[j]), __float_as_uint(o[j + 1]), __float_as_uint(o[j + 2]),
                                 __float_as_uint(o[j + 3]), __float_as_uint(o[j + 4]), __float_as_uint(o[j + 5]),
                                 __float_as_uint(o[j + 6]), __float_as_uint(o[j + 7]));
                }
            } else if (full && vec_ok) {
#pragma unroll
                for (int j = 0; j < 32; j += 4) {
                    *reinterpret_cast<float4*>(dst + j) = make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]);
                }
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    if (n0 + j < n_total) {
                        dst[j] = o[j];
                    }
                }
            }
        } else {
            uint32_t packed[16];
#pragma unroll
            for (int j = 0; j < 32; j += 2) {
                packed[j / 2] = static_cast<uint32_t>(__half_as_ushort(__float2half_rn(o[j]))) |
                                (static_cast<uint32_t>(__half_as_ushort(__float2half_rn(o[j + 1]))) << 16);
            }
            uint16_t* dst = static_cast<uint16_t*>(e.out) + m * e.ldc + n0;
            if (full && vec32) {
                st_global_32(dst, packed[0], packed[1], packed[2], packed[3], packed[4], packed[5], packed[6], packed[7]);
                st_global_32(dst + 16, packed[8], packed[9], packed[10], packed[11], packed[12], packed[13], packed[14],
                             packed[15]);
            } else if (full && vec_ok) {
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    *reinterpret_cast<uint4*>(dst + 2 * j) =
                        make_uint4(packed[j], packed[j + 1], packed[j + 2], packed[j + 3]);
                }
            } else if (full) {
                uint32_t half[2][8];
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    half[j / 8][j % 8] = packed[j];
                }
                store_32_bytes_anywhere(reinterpret_cast<uint8_t*>(dst), half[0]);
                store_32_bytes_anywhere(reinterpret_cast<uint8_t*>(dst + 16), half[1]);
            } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) {
                    if (n0 + j < n_total) {
                        dst[j] = static_cast<uint16_t>(packed[j / 2] >> (16 * (j % 2)));
                    }
                }
            }
        }
    }
}

// BATCH: one launch for a batch of equal problems (BatchTile in the last parameter); the persistent
// tile walk runs through all of them and the operands are read through maps with a batch axis.
template <int BN, int KIND, int PEERS, bool CONV = false, bool BATCH = false>
__global__ void __launch_bounds__(tile_threads(KIND, PEERS), 1)
gemm_i8_umma_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w,
                    const __grid_constant__ PeerMaps peer_maps, const I8Epilogue ep_all, const int m_total,
                    const int n_total, const int k_total, const uint32_t idesc, const int vec_ok, const int group_m, const int k_rot,
                    int32_t* error_word, const std::conditional_t<BATCH, BatchTile, ConvTile> conv)
{
    static_assert(!CONV || PEERS == 0, "the convolution form has no sharded epilogue");
    static_assert(!BATCH || (!CONV && PEERS == 0), "the batched form is a plain product");
    using Cfg = TileConfig<BN, PEERS, KIND>;
    constexpr int kStages = Cfg::kStages;
    extern __shared__ uint8_t smem_raw[];
    // The swizzled tiles must start on a 1024-byte boundary.
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* stage_base = smem;
    // Per-column epilogue terms, one private copy per epilogue warp (no cross-warp barrier).
    uint8_t* peer_stage = smem + kStages * Cfg::kStageBytes;  // 1024-byte aligned (PEERS only)
    int32_t* col_params = reinterpret_cast<int32_t*>(peer_stage + Cfg::kPeerStageBytes);
    uint64_t* full_bar = reinterpret_cast<uint64_t*>(col_params + Cfg::kColParamBytes / 4);
    uint64_t* empty_bar = full_bar + kStages;
    uint64_t* acc_full_bar = empty_bar + kStages;
    uint64_t* acc_empty_bar = acc_full_bar + 2;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty_bar + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int warp = threadIdx.x >> 5;
    const int role = warp_uniform(warp);   // the same, warp-uniform to the compiler too
    const int lane = threadIdx.x & 31;
    // Operand poses ride in bits 4-5 of vec_ok: bit 4 = A stored [K][M], bit 5 = W stored [K][N]
    // (MN-major operands: the tensor maps, the descriptors and the K step change, nothing else).
    const int pose = (vec_ok >> 4) & 3;

    const int num_m = (m_total + kBlockM - 1) / kBlockM;
    const int num_n = (n_total + BN - 1) / BN;
    const int elem_tiles = num_m * num_n;   // tiles of one problem
    int num_tiles = elem_tiles;
    FastDiv by_elem{};
    if constexpr (BATCH) {
        num_tiles *= conv.count;
        by_elem.init(static_cast<uint32_t>(elem_tiles));
    }
    const int num_kb = (k_total + kBlockKBytes - 1) / kBlockKBytes;
    const TileWalk walk(num_m, num_n, group_m);
    // Which problem of the batch a tile belongs to, and its place in it.
    const auto batch_of = [&](int tile) { return BATCH ? static_cast<int>(by_elem.div(static_cast<uint32_t>(tile))) : 0; };
    const auto coord_of = [&](int tile) { return walk(BATCH ? tile - batch_of(tile) * elem_tiles : tile); };

    // The producer warp sets the barriers up and starts to load at once: it needs nothing of the others, who
    // meet at a barrier of their own.
    constexpr uint32_t kThreads = tile_threads(KIND, PEERS);
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
                mbar_init(&acc_empty_bar[a], Cfg::kEpilogueWarps / Cfg::kGroups);
            }
            *abort_flag = 0;
            mbar_init_fence();
        }
        __syncwarp();
        named_barrier_arrive(1, kThreads);
        previous_kernel_done();
    } else {
        if (role == 1) {
            if (lane == 0) {
                tma_prefetch_desc(&map_a);
                tma_prefetch_desc(&map_w);
            }
            __syncwarp();
            tmem_alloc(tmem_slot, Cfg::kTmemCols);
            tmem_relinquish();
            named_barrier_arrive(2, 64);   // the producer, before it lets the next kernel start
        } else {
            previous_kernel_done();
        }
        tc_fence_before_sync();
        named_barrier_sync(1, kThreads);
        tc_fence_after_sync();
    }
    const uint32_t tmem_base = *tmem_slot;   // not the producer's

    if (role == 0) {
        // ---------------- TMA producer ----------------
        // The whole warp walks the loop, one elected lane issues, and no branch depends on what a wait
        // returned (see mbar_wait_converged); the same in the MMA warp.
        uint32_t issued = 0;   // by this lane
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
            const TileCoord at = coord_of(tile);
            const int m_blk = warp_uniform(at.m_blk), n_blk = warp_uniform(at.n_blk);
            const int bat = warp_uniform(batch_of(tile));
            (void)bat;
            const int rot = warp_uniform(k_rotation(tile, k_rot, num_kb));
            int patch_w = 0, patch_h = 0, patch_img = 0, tap_a = 0, tap_b = 0, tap_c = 0;   // CONV
            (void)patch_w; (void)patch_h; (void)patch_img; (void)tap_a; (void)tap_b; (void)tap_c;
            if constexpr (CONV) {
                const ConvPatch pt = conv_patch(conv, m_blk);
                patch_w = warp_uniform((pt.tw << conv.bw_log2) * conv.sw - conv.pw);
                patch_h = warp_uniform(pt.th * conv.bh * conv.sh - conv.ph);
                patch_img = warp_uniform(pt.img);
                const int tap = rot / conv.kb_per_tap;
                tap_c = warp_uniform(rot - tap * conv.kb_per_tap);
                tap_a = warp_uniform(tap / conv.kw);
                tap_b = warp_uniform(tap - tap_a * conv.kw);
            }
            int kb = rot;
            for (int step = 0; step < num_kb; ++step) {
                mbar_wait_converged<kErrProducerWait>(&empty_bar[stage], phase ^ 1u, abort_flag, failed);
                if (elect_one() && !wait_failed(failed)) {
                    uint8_t* a_dst = stage_base + stage * Cfg::kStageBytes;
                    uint8_t* b_dst = a_dst + Cfg::kATileBytes;
                    mbar_expect_tx(&full_bar[stage], Cfg::kStageBytes);
                    ++issued;
                    if constexpr (CONV) {
                        // Patch (image, th, tw) shifted by the k-block's tap; 128 channels of it.
                        tma_load_4d(a_dst, &map_a, &full_bar[stage], conv.c_base + tap_c * kBlockKBytes,
                                    patch_w + tap_b * conv.dw, patch_h + tap_a * conv.dh, patch_img);
                    } else if constexpr (BATCH) {
                        // Either pose through a map {contiguous index, the other, batch, 1}.
                        const int az = bat * conv.a_step;
                        if (pose & 1) {
                            tma_load_4d(a_dst, &map_a, &full_bar[stage], m_blk * kBlockM, kb * kBlockKBytes, az, 0);
                        } else {
                            tma_load_4d(a_dst, &map_a, &full_bar[stage], kb * kBlockKBytes, m_blk * kBlockM, az, 0);
                        }
                    } else if (pose & 1) {
                        // A stored [K][M]: the box is 128 k-rows of 128 m-bytes.
                        tma_load_2d(a_dst, &map_a, &full_bar[stage], m_blk * kBlockM, kb * kBlockKBytes);
                    } else {
                        tma_load_2d(a_dst, &map_a, &full_bar[stage], kb * kBlockKBytes, m_blk * kBlockM);
                    }
                    if constexpr (BATCH) {
                        const int wz = bat * conv.w_step;
                        if (pose & 2) {
#pragma unroll
                            for (int blk = 0; blk < BN / 128; ++blk) {
                                tma_load_4d(b_dst + blk * (128 * kBlockKBytes), &map_w, &full_bar[stage],
                                            n_blk * BN + blk * 128, kb * kBlockKBytes, wz, 0);
                            }
                        } else {
                            tma_load_4d(b_dst, &map_w, &full_bar[stage], kb * kBlockKBytes, n_blk * BN, wz, 0);
                        }
                    } else if (pose & 2) {
                        // W stored [K][N]: one box of 128 k-rows x 128 n-bytes per 128 columns of the tile.
#pragma unroll
                        for (int blk = 0; blk < BN / 128; ++blk) {
                            tma_load_2d(b_dst + blk * (128 * kBlockKBytes), &map_w, &full_bar[stage],
                                        n_blk * BN + blk * 128, kb * kBlockKBytes);
                        }
                    } else {
#pragma unroll
                        for (int h = 0; h < Cfg::kNSplit; ++h) {  // TMA boxes hold at most 256 rows
                            tma_load_2d(b_dst + h * Cfg::kMmaN * kBlockKBytes, &map_w, &full_bar[stage], kb * kBlockKBytes,
                                        n_blk * BN + h * Cfg::kMmaN);
                        }
                    }
                }
                __syncwarp();
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                }
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
                if (++kb == num_kb) {
                    kb = 0;
                }
            }
        }
        const uint32_t all_issued = __reduce_add_sync(0xFFFFFFFFu, issued);   // one lane has counted
        named_barrier_sync(2, 64);   // tensor memory is allocated
        let_next_kernel_start();
        if (const uint32_t code = warp_failure(failed); code != 0 && lane == 0) {
            atomicCAS(error_word, 0, static_cast<int32_t>(code));
            // Copies already issued still land in shared memory: the CTA must not exit underneath them.
            if (!drain_ring(full_bar, kStages, all_issued)) {
                atomicCAS(error_word, 0, kErrDrainWait);
            }
        }
        __syncwarp();
    } else if (role == 1) {
        // ---------------- MMA issuer ----------------
        const uint32_t tmem = warp_uniform(tmem_base);
        // K-major tiles step 32 bytes along their 128-byte rows per MMA (+2 in the descriptor's 16-byte
        // units); MN-major tiles step 32 k-rows of 128 bytes (+256).  The ring's descriptors advance by addition.
        const uint32_t ring = smem_u32(stage_base);
        const uint64_t a_first = (pose & 1) ? umma_desc_sw128_mnmajor(ring, 128 * kBlockKBytes) : umma_desc_sw128_kmajor(ring);
        const uint64_t b_first = (pose & 2) ? umma_desc_sw128_mnmajor(ring + Cfg::kATileBytes, 128 * kBlockKBytes)
                                            : umma_desc_sw128_kmajor(ring + Cfg::kATileBytes);
        const uint64_t a_step = (pose & 1) ? 256u : 2u;
        const uint64_t b_step = (pose & 2) ? 256u : 2u;
        uint64_t a_desc = a_first, b_desc = b_first;
        int local_tile = 0;
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++local_tile) {
            const int acc = Cfg::kNSplit > 1 ? 0 : (local_tile & 1);
            const uint32_t acc_phase = Cfg::kNSplit > 1 ? (local_tile & 1u) : ((local_tile >> 1) & 1u);
            mbar_wait_converged<kErrAccumWait>(&acc_empty_bar[acc], acc_phase ^ 1u, abort_flag, failed);
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem + static_cast<uint32_t>(acc * BN);
            uint32_t accumulate = 0;
            for (int kb = 0; kb < num_kb; ++kb) {
                mbar_wait_converged<kErrMmaWait>(&full_bar[stage], phase, abort_flag, failed);
                tc_fence_after_sync();
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < kBlockKBytes / kUmmaK; ++ks) {
#pragma unroll
                        for (int h = 0; h < Cfg::kNSplit; ++h) {
                            // Second half of a wide tile: kMmaN rows further down the W tile (16-byte
                            // descriptor units), kMmaN columns further along the accumulator.
                            umma_i8(d_tmem + static_cast<uint32_t>(h * Cfg::kMmaN), a_desc + static_cast<uint64_t>(ks) * a_step,
                                    b_desc + static_cast<uint64_t>(ks) * b_step +
                                        static_cast<uint64_t>(h * (Cfg::kMmaN * kBlockKBytes / 16)),
                                    idesc, ks > 0 ? 1u : accumulate);
                        }
                    }
                    umma_commit(&empty_bar[stage]);  // slot is free once these MMAs have read it
                }
                __syncwarp();
                accumulate = 1;
                a_desc += Cfg::kStageBytes / 16;
                b_desc += Cfg::kStageBytes / 16;
                if (++stage == kStages) {
                    stage = 0;
                    phase ^= 1u;
                    a_desc = a_first;
                    b_desc = b_first;
                }
            }
            if (elect_one()) {
                umma_commit_unless(&acc_full_bar[acc], failed);  // accumulator complete
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
        // ---------------- epilogue warps ----------------
        const int quarter = warp & 3;  // the TMEM lane quarter this warp may read
        // 8-bit destinations with a per-tensor activation scale: the row factor s_a / s_out is the
        // same for every row, so it is folded into the staged column scales (same two roundings,
        // once per column instead of once per element).  The sharded form keeps the plain scales.
        // fp destinations: the row factor is s_a itself.
        const bool fold_scale = !PEERS && KIND != NNB200_OUT_S32 && ep_all.scale_a == nullptr;
        const float folded_row_k = (KIND == NNB200_OUT_S8 || KIND == NNB200_OUT_U8)
                                       ? __fdiv_rn(ep_all.scale_a_scalar, ep_all.out_scale) : ep_all.scale_a_scalar;
        const bool fold_comp = !PEERS && (KIND == NNB200_OUT_S8 || KIND == NNB200_OUT_U8) && ep_all.compensate != 0 &&
                               ep_all.zp_a == nullptr && ep_all.r_a == nullptr;
        // The next tile's column terms are loaded into registers before this tile is drained,
        // so their latency is not paid between tiles (up to four per lane and term).
        constexpr int kTermIters = (Cfg::kPartCols + 31) / 32;
        constexpr bool kPrefetch = !PEERS && kTermIters <= 4 && Cfg::kEpilogueWarps < 16;
        ColTerms next_terms[kPrefetch ? kTermIters : 1];
        // The warps of a lane quarter share out the tile's columns.
        constexpr int kPartCols = Cfg::kPartCols;
        const int part = ((warp - 2) >> 2) % Cfg::kColParts;
        const int group = ((warp - 2) >> 2) / Cfg::kColParts;
        const int col0 = part * kPartCols;
        const int ncols = min(kPartCols, BN - col0);
        float* cs = reinterpret_cast<float*>(col_params + (warp - 2) * 4 * kPartCols);
        int32_t* cb = reinterpret_cast<int32_t*>(cs) + kPartCols;
        int32_t* cr = cb + kPartCols;
        int32_t* cz = cr + kPartCols;
        int stage_turn = 0;  // sharded form: which of the warp's two staging tiles is next
        (void)stage_turn;
        // The epilogue block of one problem of the batch: its output and its operands' sums.
        const auto epilogue_of = [&](int bat) -> std::conditional_t<BATCH, I8Epilogue, const I8Epilogue&> {
            if constexpr (BATCH) {
                I8Epilogue e = ep_all;
                e.out = static_cast<uint8_t*>(e.out) + bat * conv.out_step;
                if (e.compensate) {
                    e.r_a = e.r_a != nullptr ? e.r_a + static_cast<int64_t>(bat) * conv.ra_step : nullptr;
                    e.r_w = e.r_w != nullptr ? e.r_w + static_cast<int64_t>(bat) * conv.rw_step : nullptr;
                }
                return e;
            } else {
                return ep_all;
            }
        };
        int staged_base = 0;
        int local_tile = 0;
        for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x, ++local_tile) {
            if (Cfg::kGroups > 1 && (local_tile & 1) != group) {
                continue;
            }
            const TileCoord tc = coord_of(tile);
            const int acc = Cfg::kNSplit > 1 ? 0 : (local_tile & 1);
            const uint32_t acc_phase = Cfg::kNSplit > 1 ? (local_tile & 1u) : ((local_tile >> 1) & 1u);
            decltype(auto) ep = epilogue_of(batch_of(tile));
            const int n_base = tc.n_blk * BN + col0;   // first column this warp drains

            // This tile's per-column terms: fetched while the previous tile was being drained
            // (kPrefetch), or now, hidden behind the tile's main loop.
            // Tiles that follow one another in a CTA mostly share their columns: then the terms are there already, and
            // no round trip to the L2 stands between two tiles (1x1 convolution 256 -> 1024 71.8 -> 62.8 us).
            const bool stage_terms = BATCH || n_base != staged_base || local_tile < Cfg::kGroups;
            staged_base = n_base;
            __syncwarp();  // previous tile's reads of the staging are done
#pragma unroll
            for (int i = 0; i < kTermIters; ++i) {
                const int j = lane + i * 32;
                if (stage_terms && j < ncols) {
                    const ColTerms ct = finish_col_terms<KIND>(
                        ep, (kPrefetch && local_tile > 0) ? next_terms[kPrefetch ? i : 0] : load_col_terms<KIND>(ep, n_base + j, n_total),
                        fold_scale, folded_row_k, fold_comp);
                    cs[j] = ct.scale;
                    cb[j] = ct.bias;
                    cr[j] = ct.rw;
                    cz[j] = ct.zpw;
                }
            }
            __syncwarp();

            int64_t m = static_cast<int64_t>(tc.m_blk) * kBlockM + quarter * 32 + lane;
            bool row_ok = m < m_total;
            uint32_t bad_h = 0, bad_w = 0;   // CONV: the row's border class along each axis (0: every tap inside)
            if constexpr (CONV) {
                const ConvRow cr_ = conv_row(conv, tc.m_blk, quarter * 32 + lane);
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

            // Warp-uniform outcome, so no lane is left behind at a later warp sync.
            if (!__all_sync(0xFFFFFFFFu, mbar_wait(&acc_full_bar[acc], acc_phase, abort_flag))) {
                atomicCAS(error_word, 0, kErrEpilogueWait);
                break;
            }
            tc_fence_after_sync();

            if constexpr (kPrefetch) {
                const int next = tile + static_cast<int>(gridDim.x);
                if (next < num_tiles) {
                    const int next_base = coord_of(next).n_blk * BN + col0;
                    decltype(auto) next_ep = epilogue_of(batch_of(next));
#pragma unroll
                    for (int i = 0; i < kTermIters; ++i) {
                        next_terms[i] = load_col_terms<KIND>(next_ep, next_base + lane + i * 32, n_total);
                    }
                }
            }

            const uint32_t t_row = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                   static_cast<uint32_t>(acc * BN + col0);
            if constexpr (PEERS && (KIND == NNB200_OUT_S8 || KIND == NNB200_OUT_U8)) {
                // Sharded write-back: 128 columns at a time through a per-warp staging tile.
                const float zpf = static_cast<float>(ep.out_zp);
                const float lo = (KIND == NNB200_OUT_S8 ? -128.0f : 0.0f) - zpf;
                const float hi = (KIND == NNB200_OUT_S8 ? 127.0f : 255.0f) - zpf;
                (void)lo;
                (void)hi;
                const int row0 = tc.m_blk * kBlockM + quarter * 32;
                const int num_dst = 1 + ep.num_peers;
                const bool multicast = ep.mc_out != nullptr;
                constexpr int kGroupCols = Cfg::kStageGroupCols;       // 128 (swizzled tile) or 256 (plain tile)
                constexpr int kGroupChunks = kGroupCols / 32;
#pragma unroll 1
                for (int c4 = 0; c4 < (BN + kGroupCols - 1) / kGroupCols; ++c4) {
                    const int n128 = n_base + c4 * kGroupCols;
                    if (n128 >= n_total) {
                        break;  // uniform across the warp
                    }
                    // Two staging tiles per warp, used alternately: before refilling one, its
                    // previous bulk stores must have finished READING it (they may still be in flight
                    // on the wire).  Only lane 0 issues bulk stores, so only lane 0 has groups to wait on.
                    uint8_t* stage = peer_stage + ((warp - 2) * Cfg::kStageTiles + (stage_turn % Cfg::kStageTiles)) *
                                                      (32 * kGroupCols);
                    ++stage_turn;
                    if (lane == 0) {
                        bulk_wait_group_read<Cfg::kStageTiles - 1>();
                    }
                    __syncwarp();
#pragma unroll 1
                    for (int cc = 0; cc < kGroupChunks; ++cc) {
                        const int c = c4 * kGroupChunks + cc;
                        if (c >= BN / 32) {
                            break;  // a 224-wide tile ends inside its second 128-column group
                        }
                        uint32_t v[32];
                        tmem_ld_32x32(t_row + static_cast<uint32_t>(c * 32), v);
                        tmem_ld_wait();
                        // No branch per element: the ReLU is a lower bound, compensation is chosen
                        // once per chunk, saturation rides the packing instruction.
                        uint32_t packed[8];
                        const int32_t relu_lo = ep.relu ? 0 : INT32_MIN;
                        if (ep.compensate) {
#pragma unroll
                            for (int j = 0; j < 32; j += 4) {
                                int32_t vv[4];
                                float rq[4];
#pragma unroll
                                for (int b = 0; b < 4; ++b) {
                                    const int col = c * 32 + j + b;
                                    const int32_t x = i8_compensate(static_cast<int32_t>(v[j + b]), rt.zpa, cz[col], rt.ra,
                                                                    cr[col], ep.k);
                                    vv[b] = max(static_cast<int32_t>(static_cast<uint32_t>(x) + static_cast<uint32_t>(cb[col])),
                                                relu_lo);
                                    rq[b] = __fmul_rn(rt.row_k, cs[col]);
                                }
                                packed[j / 4] = requant_pack4<KIND == NNB200_OUT_U8, false>(vv, rq, ep.out_zp);
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; j += 4) {
                                int32_t vv[4];
                                float rq[4];
#pragma unroll
                                for (int b = 0; b < 4; ++b) {
                                    const int col = c * 32 + j + b;
                                    vv[b] = max(static_cast<int32_t>(v[j + b] + static_cast<uint32_t>(cb[col])), relu_lo);
                                    rq[b] = __fmul_rn(rt.row_k, cs[col]);
                                }
                                packed[j / 4] = requant_pack4<KIND == NNB200_OUT_U8, false>(vv, rq, ep.out_zp);
                            }
                        }
                        // This lane's row of the tile: 16-byte pieces 2cc and 2cc+1 (swizzled in the 128-byte form).
                        uint4* srow = reinterpret_cast<uint4*>(stage + lane * kGroupCols);
                        const int sw = lane & 7;
                        srow[(2 * cc) ^ sw] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
                        srow[(2 * cc + 1) ^ sw] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
                    }
                    if (multicast) {
                        // One store per tile for all ranks: the staged rows go out as 16-byte
                        // multimem stores, eight lanes covering one 128-byte row, four rows per
                        // pass, and the switch replicates them into every rank's copy.
                        __syncwarp();
                        const int piece = lane & 7;
                        const int cols_here = min(min(128, BN - c4 * 128), n_total - n128);
#pragma unroll 1
                        for (int pass = 0; pass < 8; ++pass) {
                            const int r = pass * 4 + (lane >> 3);
                            const int64_t grow = static_cast<int64_t>(row0) + r;
                            if (grow < m_total && piece * 16 < cols_here) {
                                const uint4 q = *reinterpret_cast<const uint4*>(stage + r * 128 + ((piece ^ (r & 7)) * 16));
                                multimem_st_16(static_cast<uint8_t*>(ep.mc_out) + grow * ep.ldc + n128 + piece * 16, q);
                            }
                        }
                        __syncwarp();  // the staging tile may be refilled
                        continue;
                    }
                    fence_proxy_async_smem();  // generic-proxy writes -> visible to the TMA engine
                    __syncwarp();
                    if (lane == 0) {
                        // One bulk store per destination; rows past M and columns past N are clipped
                        // by the descriptor.
                        for (int d = 0; d < num_dst; ++d) {
                            tma_store_2d(&peer_maps.m[d], stage, n128, row0);
                        }
                        bulk_commit_group();
                    }
                }
            } else {
                // Chunks of 32 columns, two register sets: the load of the next chunk is in flight
                // while this one is requantised and stored.
                const int left = n_total - n_base;   // columns of the matrix from this warp's first one
                const int nch = left <= 0 ? 0 : min(ncols / 32, (left + 31) / 32);   // uniform across the warp
                const auto finish = [&](int c, uint32_t (&v)[32]) {
                    const int n0 = n_base + c * 32;
                    if constexpr (CONV) {
                        conv_border_fix(conv, v, bad_h, bad_w, n0, n_total);
                    }
                    epilogue_chunk<KIND>(ep, rt, v, m, row_ok, n0, n_total, cs + c * 32, cb + c * 32, cr + c * 32,
                                         cz + c * 32, vec_ok, fold_scale, fold_comp);
                };
                if constexpr (Cfg::kEpilogueWarps == 16) {
                    // Enough warps to cover a load's latency; one register set keeps them resident.
                    uint32_t v[32];
#pragma unroll 1
                    for (int c = 0; c < nch; ++c) {
                        tmem_ld_32x32(t_row + static_cast<uint32_t>(c * 32), v);
                        tmem_ld_wait();
                        finish(c, v);
                    }
                } else {
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
                }
            }
            // Accumulator drained: hand it back to the MMA warp.
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&acc_empty_bar[acc]);
            }
        }
        if (!PEERS && ep_all.direct_peers > 0) {
            __threadfence_system();  // this warp's stores into the peer's copy are performed before the kernel completes
        }
        if constexpr (PEERS) {
            if (ep_all.mc_out != nullptr) {
                __threadfence_system();  // this warp's multicast stores are performed before the kernel completes
            }
            if (lane == 0) {
                bulk_wait_group<0>();  // every bulk store of this warp has completed before the CTA exits
            }
            __syncwarp();
        }
    }

    // ---------------- teardown ----------------
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, Cfg::kTmemCols);
    }
}

}  // namespace
}  // namespace nnb200
