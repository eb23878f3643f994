// The prepared form of the 3xTF32 families: D = alpha A B + beta C from operands split into FP16 pairs.
//
// A TF32 number and an FP16 number have the same 11 significant bits, and the tensor cores multiply
// FP16 at twice the rate. With the operands scaled (gemm_fp16x3_split.cu, which also says
// when that is exact enough and leaves the launch to the TF32 kernel when it is not),
//   a b = a_hi b_hi + (a_lo b_hi + a_hi b_lo) / 2^11,     a = a_hi + a_lo / 2^11, b likewise,
// is three tcgen05.mma.kind::f16 products in half the tensor time of three TF32 ones, with less
// rounding in the low parts (2^-23 at most, to nearest, against a truncation at 2^-21). And because the operands arrive
// split, no warp converts anything here: the conversion, which every CTA of the TF32 kernel repeats
// for every tile, is paid once per operand element, and the tensor cores wait for TMA alone.
//
// A pair of CTAs (tcgen05 cta_group::2, a cluster of two) shares an output tile of 256 rows and up to
// 256 columns, K walked in blocks of 64. Each CTA brings its 128 rows of A and half of the tile's rows
// of B (B is K-major here whatever the caller's orientation), high and low parts, in two TMA copies:
// at most 64 KiB a stage, three stages.
//
//   warp 0       TMA producer (one thread, in both CTAs; the bytes of both count on the first CTA's barrier)
//   warps 1, 2   MMA issuers (one thread each, in the first CTA, for both CTAs' tensor cores)
//   warps 4-11   drain / epilogue, 32 rows x half of the columns each
//
// Tensor memory holds two accumulators, 512 columns in all: X, the two cross products, issued by warp 1, and H, a_hi b_hi,
// issued by warp 2. Both are read at the end of every slab of K (768, the split's unit of scaling), multiplied by
// the slab's powers of two (addScaled) and added up in registers, to nearest. The tensor core's own FP32
// additions truncate, so below K = 22500 H is read more often than that (chunkBlocks); X is 2^11 times smaller
// in effect. A reading of H leaves the tensor pipe idle for about 1000 cycles, nearly all of it the way through the barriers:
// without loads or additions in the drain it costs the same (timing build, 4096^3: 349 us with one per slab, 374 with three, 367
// with three empty ones). Holding the cross products' issuer back so that H's last products of a sum go first gave 1 %, or lost. With an issuer each, one accumulator is read while products go to the other, and what a single thread does
// between two K blocks -- barriers, descriptors -- no longer leaves the tensor pipe idle (one issuer for both:
// 440 us instead of 388 at 4096^3, 187 instead of 154 at 2048 x 4096 x 3072, each with one reading per slab). Rings of their own for the high and
// the low parts, with H held one block behind X, were not faster (398 to 421 us).
//
// Shared memory is the resource next to the tensor pipe: operand fetches and TMA writes take 106 of its 128 bytes a
// cycle. So the drain takes nothing from there -- B's scales are common to 16 columns and sit in registers -- and
// the results go to memory straight from registers, 32 bytes a thread and store: 9400 cycles a tile, 15000 in pieces of
// 16 bytes, 12000 turned in shared memory first (and the MMAs slower meanwhile).
//
// Measured, the whole launch with its split, TF32 form / this one in microseconds: 16384 x 4096 x 14336 9000 / 5100 (398
// to 415 TFLOP/s in bursts; power-limited), 8192 x 4096 x 8192 2530 / 1440, 4096^3 640 / 426, 2048^3 132 / 70, 1024 x 1024 x 4096 76 / 40.
//
// Every wait is bounded, as in the other kernels (ptx.cuh).
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "fp16x3.hpp"
#include "gemm_kernels.hpp"
#include "ptx.cuh"
#include "tf32x3_common.cuh"

namespace ftcuda {
namespace {

using fp16x3::kBlockBytes;
using fp16x3::kBlockK;
using fp16x3::kMaxTileN;
using fp16x3::kSlabBlocks;
using fp16x3::kSlabK;
using fp16x3::kTileM;

constexpr int kStages     = 3;
constexpr int kThreads    = 384;
constexpr int kABytes     = 128 * static_cast<int>(kBlockBytes);  // a CTA's A tile: high | low, 16 KiB each
constexpr int kStageBytes = kABytes + kMaxTileN / 2 * static_cast<int>(kBlockBytes);  // ... and its half of B's
constexpr int kBarrierOffset = kStages * kStageBytes;
constexpr int kSmemBytes     = kBarrierOffset + 256 + 1024;
static_assert(kSmemBytes <= 232448, "shared memory of one CTA");

constexpr int kRegsLight = 72;   // producer, issuer (warpgroup 0)
constexpr int kRegsDrain = 216;  // drain / epilogue (warpgroups 1, 2)
static_assert(128 * kRegsLight + 256 * kRegsDrain <= 168 * kThreads, "the CTA's register pool is what it was launched with");
constexpr int kProducerWarp  = 0;
constexpr int kCrossWarp     = 1;
constexpr int kHighWarp      = 2;
constexpr int kFirstEpilogue = 4;
constexpr std::uint32_t kTmemColumns = 512;
constexpr std::uint32_t kHColumn     = 256;  // X at 0

struct Barriers {
    std::uint64_t full[kStages];  // used in the pair's first CTA
    std::uint64_t empty[kStages];
    std::uint64_t x_full, h_full;
    std::uint64_t x_empty, h_empty;  // used in the pair's first CTA
    std::uint64_t flush_x, flush_h;
    std::uint32_t tmem_base;
    int abort_flag;
    std::uint32_t fallback;
};
static_assert(sizeof(Barriers) <= 256, "barrier block");

struct Fp16Params {
    const float* c;
    float* d;
    std::int64_t c_row_stride, c_col_stride;
    std::int64_t d_row_stride, d_col_stride;
    std::uint32_t m, n;
    std::uint32_t k, k_blocks, blocks_per_split, splits;
    std::uint32_t tiles_m, tiles_n, tile_n, band_m_tiles;
    std::uint32_t chunk_blocks;
    float alpha, beta;
    float* partials;  // non-null: the K slices' sums, [split][m][n]
    const float* inverse_a;  // [slab][inverse_pitch_a]
    const float* inverse_b;
    std::uint64_t inverse_pitch_a, inverse_pitch_b;
    const std::uint32_t* verdicts;        // of the split's CTAs: first A's, then B's, slab by slab
    std::uint32_t verdicts_per_slab[2];
    std::uint32_t slabs;
    std::uint32_t* use_fallback;    // the decision, for the kernels behind this one
    std::uint32_t vector;  // consecutive columns of the output and C that one aligned access takes: 8, 4, or 0 (any strides)
    int* status;
};

struct Item {
    std::uint32_t row, col, split, first_block, blocks;
};

__device__ __forceinline__ Item decode(const Fp16Params& p, std::uint32_t item) {
    const std::uint32_t tiles = p.tiles_m * p.tiles_n;
    Item w;
    w.split                   = item / tiles;
    const std::uint32_t tile  = item - w.split * tiles;
    const std::uint32_t band  = tile / (p.band_m_tiles * p.tiles_n);
    const std::uint32_t first = band * p.band_m_tiles;
    const std::uint32_t rows  = min(p.band_m_tiles, p.tiles_m - first);
    const std::uint32_t rest  = tile - band * p.band_m_tiles * p.tiles_n;
    w.row                     = (first + rest % rows) * kTileM;
    w.col                     = rest / rows * p.tile_n;
    w.first_block             = w.split * p.blocks_per_split;
    w.blocks                  = min(p.k_blocks - w.first_block, p.blocks_per_split);
    return w;
}

// Position in a ring of slots: the slot, and how often the ring has been gone round.
struct Ring {
    std::uint32_t slots, slot = 0, round = 0;
    __device__ __forceinline__ explicit Ring(std::uint32_t n) : slots(n) {}
    __device__ __forceinline__ void next() {
        if (++slot == slots) {
            slot = 0;
            ++round;
        }
    }
};

// K blocks of an item from `block` on that lie in one slab. (A K slice may begin and end inside one.)
__device__ __forceinline__ std::uint32_t blocksInSlab(const Item& w, std::uint32_t block) {
    return min(kSlabBlocks - (w.first_block + block) % kSlabBlocks, w.blocks - block);
}

// Writes 32 consecutive columns of one row, held by one thread.
__device__ __forceinline__ void writePiece(const Fp16Params& p, const Item& w, std::uint32_t row, std::uint32_t col, const float2* values) {
    const std::uint32_t end       = min(p.n, w.col + p.tile_n);  // of the tile's columns
    const bool partial            = p.partials != nullptr;
    float* const out              = partial ? p.partials + static_cast<std::uint64_t>(w.split) * p.m * p.n : p.d;
    const std::int64_t row_stride = partial ? p.n : p.d_row_stride;
    const float* const c          = partial ? nullptr : p.c;
    const float alpha             = partial ? 1.0F : p.alpha;
    if (p.vector == 8) {
        // 32 bytes, a whole sector, per thread and store: half the passes through the L1 that 16 take.
        float* const at = out + static_cast<std::int64_t>(row) * row_stride + col;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float addend[2][8];
            if (c != nullptr) {
                // C's values are asked for before the stores: C may be D, so the compiler moves no load past a store by itself.
                const float* const from = c + static_cast<std::int64_t>(row) * p.c_row_stride + col + 16 * half;
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (col + 16 * half + 8 * j < end) { loadGlobal8(from + 8 * j, addend[j]); }
                }
            }
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                if (col + 16 * half + 8 * j >= end) { continue; }
                float o[8];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    o[2 * i]     = alpha * values[8 * half + 4 * j + i].x;
                    o[2 * i + 1] = alpha * values[8 * half + 4 * j + i].y;
                }
                if (c != nullptr) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) { o[i] += p.beta * addend[j][i]; }
                }
                storeGlobal8(at + 16 * half + 8 * j, o);
            }
        }
        return;
    }
    if (p.vector == 4) {
        float* const at         = out + static_cast<std::int64_t>(row) * row_stride + col;
        const float* const from = c != nullptr ? c + static_cast<std::int64_t>(row) * p.c_row_stride + col : nullptr;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (col + 4 * j >= end) { continue; }
            const float2 low = values[2 * j], high = values[2 * j + 1];
            float4 o = make_float4(alpha * low.x, alpha * low.y, alpha * high.x, alpha * high.y);
            if (c != nullptr) {
                const float4 addend = *reinterpret_cast<const float4*>(from + 4 * j);
                o.x += p.beta * addend.x;
                o.y += p.beta * addend.y;
                o.z += p.beta * addend.z;
                o.w += p.beta * addend.w;
            }
            *reinterpret_cast<float4*>(at + 4 * j) = o;
        }
        return;
    }
    const std::int64_t col_stride = partial ? 1 : p.d_col_stride;
    float* const at = out + static_cast<std::int64_t>(row) * row_stride + static_cast<std::int64_t>(col) * col_stride;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
        if (col + j >= end) { continue; }
        float value = alpha * (j % 2 == 0 ? values[j / 2].x : values[j / 2].y);
        if (c != nullptr) {
            value += p.beta * c[static_cast<std::int64_t>(row) * p.c_row_stride + static_cast<std::int64_t>(col + j) * p.c_col_stride];
        }
        at[j * col_stride] = value;
    }
}

// acc += row_scale * scale of the 16 columns * accumulator, for up to four pieces of 32 columns at `tmem`. The scales are powers
// of two. As long as their product is one that FP32 has (not under 2^-149), it scales exactly and the addition is the only
// rounding. Operands may be as small as 2^-100 each, so it need not be: then (kApart) the row's scale, which alone is at least
// 2^-125, is applied first. What that rounds off is under 2^-150 / 2^-125 of one in units of the accumulator, whose
// products reach up to 2^28. Twice the arithmetic, so only where it is needed.
template<bool kApart>
__device__ __forceinline__ void addScaled(std::uint32_t tmem, std::uint32_t pieces, float row_scale, const float (&scales)[8],
                                          float2 (&acc)[64]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        if (static_cast<std::uint32_t>(q) < pieces) {
            float v[32];
            tmemLoad32(tmem + q * 32, v);
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                const float scale = kApart ? scales[2 * q + g] : row_scale * scales[2 * q + g];
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float2& sum  = acc[q * 16 + g * 8 + j];
                    float2 value = make_float2(v[g * 16 + 2 * j], v[g * 16 + 2 * j + 1]);
                    if (kApart) { value = multiply2(make_float2(row_scale, row_scale), value); }
                    sum = multiplyAdd2(make_float2(scale, scale), value, sum);
                }
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(2, 1, 1)
tensorGemm3xFp16(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Fp16Params p,
                 std::uint32_t num_items) {
    extern __shared__ unsigned char smem_raw[];
    const std::uint32_t align_offset = (1024 - (smemAddress(smem_raw) & 1023)) & 1023;
    unsigned char* smem              = smem_raw + align_offset;
    Barriers* bars                   = reinterpret_cast<Barriers*>(smem + kBarrierOffset);
    volatile int* abort_flag         = &bars->abort_flag;
    const int warp                   = threadIdx.x >> 5;
    const int lane                   = threadIdx.x & 31;
    const std::uint32_t rank         = clusterCtaRank();
    const std::uint32_t pair         = blockIdx.x >> 1;
    const std::uint32_t pairs        = gridDim.x >> 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbarrierInit(&bars->full[s], 1);
            mbarrierInit(&bars->empty[s], 2);  // both issuers
        }
        mbarrierInit(&bars->x_full, 1);
        mbarrierInit(&bars->h_full, 1);
        mbarrierInit(&bars->x_empty, 16);
        mbarrierInit(&bars->h_empty, 16);
        mbarrierInit(&bars->flush_x, 1);
        mbarrierInit(&bars->flush_h, 1);
        bars->abort_flag = 0;
        bars->fallback   = 0;
        fenceBarrierInit();
        prefetchTensorMap(&map_a);
        prefetchTensorMap(&map_b);
    }
    if (warp == kCrossWarp) { tmemAllocatePair(&bars->tmem_base, kTmemColumns); }
    tcgen05FenceBeforeSync();
    __syncthreads();
    clusterBarrierArrive();
    clusterBarrierWait();
    tcgen05FenceAfterSync();
    const std::uint32_t tmem_base = bars->tmem_base;

    // Launched with programmatic stream serialization: what is above overlaps the split's tail.
    gridDependencyWait();
    gridDependencyLaunchDependents();
    // Every CTA comes to the same decision. Left to the fallback, there are no items.
    {
        // A warp takes a slab at a time: a gray element only concerns its own.
        for (std::uint32_t slab = warp; slab < p.slabs; slab += kThreads / 32) {
            const std::uint32_t length = min(kSlabK, p.k - slab * kSlabK);
            std::uint32_t small[2][3]  = {{0, 0, 0}, {0, 0, 0}}, state = fp16x3::kAllCovered;
#pragma unroll
            for (int which = 0; which < 2; ++which) {
                const std::uint32_t count           = p.verdicts_per_slab[which];
                const std::uint32_t* const verdicts = p.verdicts + (which != 0 ? p.slabs * p.verdicts_per_slab[0] : 0) + slab * count;
#pragma unroll 1
                for (std::uint32_t at = lane; at < count; at += 32 * 8) {
                    std::uint32_t v[8];
#pragma unroll
                    for (std::uint32_t i = 0; i < 8; ++i) { v[i] = at + 32 * i < count ? __ldcg(verdicts + at + 32 * i) : 0; }
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        state = max(state, v[i] >> fp16x3::kVerdictState);
#pragma unroll
                        for (int t = 0; t < 3; ++t) { small[which][t] = max(small[which][t], v[i] >> (10 * t) & fp16x3::kVerdictSmall); }
                    }
                }
#pragma unroll
                for (int t = 0; t < 3; ++t) { small[which][t] = __reduce_max_sync(0xFFFFFFFFU, small[which][t]); }
            }
            state = __reduce_max_sync(0xFFFFFFFFU, state);
            // F_a + F_b - L >= (g_a + g_b) / 128 for any pair of thresholds whose exponents add up to 18.
            const std::uint32_t common = state == fp16x3::kManyGray ? (2 * length + 127) / 128 : 1;
            const auto enough          = [&](int a, int b) { return small[0][a] + small[1][b] + common <= length; };
            if (state == fp16x3::kOutOfRange || (state != fp16x3::kAllCovered && !enough(0, 2) && !enough(1, 1) && !enough(2, 0))) {
                if (lane == 0) { bars->fallback = 1; }
            }
        }
        __syncthreads();
        const bool fallback = bars->fallback != 0;
        if (blockIdx.x == 0 && threadIdx.x == 0) { *p.use_fallback = fallback ? 1U : 0U; }
        if (fallback) { num_items = 0; }
    }

    if (warp >= kFirstEpilogue) {
        registersGrow<kRegsDrain>();
        const int e                   = warp - kFirstEpilogue;                    // 0..7
        const std::uint32_t in_tile   = static_cast<std::uint32_t>(32 * (warp & 3));  // the tensor-memory lanes a warp can read
        const std::uint32_t tmem_row  = tmem_base + (in_tile << 16);
        const std::uint32_t pieces    = (p.tile_n + 31) / 32;
        const std::uint32_t first     = (e >> 2) != 0 ? (pieces + 1) / 2 : 0;  // this warp's pieces of 32 columns
        const std::uint32_t mine      = (e >> 2) != 0 ? pieces / 2 : (pieces + 1) / 2;
        const std::uint32_t x_empty   = mapToRank(&bars->x_empty, 0);
        const std::uint32_t h_empty   = mapToRank(&bars->h_empty, 0);
        std::uint32_t slabs = 0, chunks = 0;
        bool ok = true;
        for (std::uint32_t item = pair; item < num_items && ok; item += pairs) {
            const Item w             = decode(p, item);
            const std::uint32_t row0 = w.row + rank * 128 + in_tile;
            const std::uint32_t mine_at = w.col + first * 32;
            float2 acc[64];
#pragma unroll
            for (int j = 0; j < 64; ++j) { acc[j] = make_float2(0.0F, 0.0F); }
            for (std::uint32_t block = 0, in_slab; block < w.blocks && ok; block += in_slab, ++slabs) {
                in_slab = blocksInSlab(w, block);
                // The slab's scales: of this thread's row, and of this warp's groups of 16 columns (1 beyond the last).
                const std::uint32_t slab = (w.first_block + block) / kSlabBlocks;
                const float row_scale    = row0 + lane < p.m ? p.inverse_a[slab * p.inverse_pitch_a + row0 + lane] : 1.0F;
                const float* const groups = p.inverse_b + slab * p.inverse_pitch_b + mine_at / fp16x3::kColumnGroup;
                float scales[8];
#pragma unroll
                for (std::uint32_t g = 0; g < 8; ++g) { scales[g] = mine_at + g * fp16x3::kColumnGroup < p.n ? groups[g] : 1.0F; }
                const float smallest = fminf(fminf(fminf(scales[0], scales[1]), fminf(scales[2], scales[3])),
                                             fminf(fminf(scales[4], scales[5]), fminf(scales[6], scales[7])));
                const bool apart     = __any_sync(0xFFFFFFFFU, row_scale * 0x1p-11F * smallest == 0.0F);
                const std::uint32_t num_chunks = (in_slab + p.chunk_blocks - 1) / p.chunk_blocks;
                for (std::uint32_t chunk = 0; chunk < num_chunks && ok; ++chunk, ++chunks) {
                    // X once per slab, ahead of the last reading of H.
                    if (chunk + 1 == num_chunks) {
                        ok = mbarrierWait(&bars->x_full, slabs & 1, abort_flag);
                        if (!ok) { break; }
                        tcgen05FenceAfterSync();
                        if (apart) {
                            addScaled<true>(tmem_row + first * 32, mine, row_scale * 0x1p-11F, scales, acc);
                        } else {
                            addScaled<false>(tmem_row + first * 32, mine, row_scale * 0x1p-11F, scales, acc);
                        }
                        tcgen05FenceBeforeSync();
                        __syncwarp();
                        if (lane == 0) { mbarrierArriveCluster(x_empty); }
                    }
                    ok = mbarrierWait(&bars->h_full, chunks & 1, abort_flag);
                    if (!ok) { break; }
                    tcgen05FenceAfterSync();
                    if (apart) {
                        addScaled<true>(tmem_row + kHColumn + first * 32, mine, row_scale, scales, acc);
                    } else {
                        addScaled<false>(tmem_row + kHColumn + first * 32, mine, row_scale, scales, acc);
                    }
                    tcgen05FenceBeforeSync();
                    __syncwarp();
                    if (lane == 0) { mbarrierArriveCluster(h_empty); }
                }
            }
            if (!ok) { break; }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const std::uint32_t col = mine_at + q * 32;
                if (static_cast<std::uint32_t>(q) < mine && col < p.n && row0 + lane < p.m) {
                    writePiece(p, w, row0 + lane, col, acc + q * 16);
                }
            }
        }
        if (!ok) { *abort_flag = 1; }
    } else {
        registersShrink<kRegsLight>();
        if (warp == kProducerWarp) {
            bool ok = true;
            if (lane == 0) {
                const std::uint32_t stage_bytes = kABytes + p.tile_n / 2 * static_cast<std::uint32_t>(kBlockBytes);
                Ring ring(kStages);
                std::uint32_t filled = 0;
                for (std::uint32_t item = pair; item < num_items && ok; item += pairs) {
                    const Item w = decode(p, item);
                    const std::int32_t row_a = static_cast<std::int32_t>(w.row + rank * 128);
                    const std::int32_t row_b = static_cast<std::int32_t>(w.col + rank * (p.tile_n / 2));
                    for (std::uint32_t kb = 0; kb < w.blocks; ++kb, ++filled, ring.next()) {
                        ok = mbarrierWait(&bars->empty[ring.slot], (ring.round & 1) ^ 1, abort_flag);
                        if (!ok) { break; }
                        // The bytes of both CTAs count on the first CTA's barrier, which that CTA arms. (The other's
                        // may land first: the phase cannot complete before it has been armed.)
                        if (rank == 0) { mbarrierArriveExpectTx(&bars->full[ring.slot], 2 * stage_bytes); }
                        const std::uint32_t full  = mapToRank(&bars->full[ring.slot], 0);
                        unsigned char* const slot = smem + ring.slot * kStageBytes;
                        const std::int32_t z      = static_cast<std::int32_t>((w.first_block + kb) * 2);
                        tmaLoad3dPair(slot, &map_a, full, 0, row_a, z);
                        tmaLoad3dPair(slot + kABytes, &map_b, full, 0, row_b, z);
                    }
                }
                // Neither CTA leaves before the last commits have arrived on its barriers.
                for (std::uint32_t i = 0; i < kStages && i < filled && ok; ++i) {
                    const std::uint32_t use = filled - 1 - i;
                    ok = mbarrierWait(&bars->empty[use % kStages], (use / kStages) & 1, abort_flag);
                }
                if (!ok) { *abort_flag = 1; }
            }
            __syncwarp();
        } else if ((warp == kCrossWarp || warp == kHighWarp) && rank == 0) {
            if (lane == 0) {
                const bool cross                = warp == kCrossWarp;
                const std::uint32_t instruction = umaInstructionF16(kTileM, p.tile_n);
                // Operand descriptors of the first stage, and their distance to the next, in units of 16 bytes.
                const std::uint64_t stage_step = kStageBytes >> 4;
                const std::uint64_t a_hi0 = umaDescriptorK128(smemAddress(smem)), a_lo0 = a_hi0 + (128 * 128 >> 4);
                const std::uint64_t b_hi0 = a_hi0 + (kABytes >> 4), b_lo0 = b_hi0 + (p.tile_n / 2 * 128 >> 4);
                std::uint64_t* const sum_full  = cross ? &bars->x_full : &bars->h_full;
                std::uint64_t* const sum_empty = cross ? &bars->x_empty : &bars->h_empty;
                Ring ring(kStages);
                std::uint32_t sums = 0;
                bool ok            = true;
                for (std::uint32_t item = pair; item < num_items && ok; item += pairs) {
                    const Item w = decode(p, item);
                    // K blocks left in the slab, and in the sum that goes to the drain warps next.
                    std::uint32_t in_slab = 0, in_sum = 0;
                    for (std::uint32_t kb = 0; kb < w.blocks; ++kb, ring.next()) {
                        if (in_slab == 0) { in_slab = blocksInSlab(w, kb); }
                        const bool fresh = in_sum == 0;
                        if (fresh) {
                            in_sum = cross ? in_slab : min(in_slab, p.chunk_blocks);
                            ok     = mbarrierWait(sum_empty, (sums & 1) ^ 1, abort_flag);
                            if (!ok) { break; }
                            ++sums;
                        }
                        ok = mbarrierWait(&bars->full[ring.slot], ring.round & 1, abort_flag);
                        if (!ok) { break; }
                        tcgen05FenceAfterSync();
                        const std::uint64_t a_hi = a_hi0 + ring.slot * stage_step, b_hi = b_hi0 + ring.slot * stage_step;
                        if (cross) {
                            const std::uint64_t a_lo = a_lo0 + ring.slot * stage_step, b_lo = b_lo0 + ring.slot * stage_step;
#pragma unroll
                            for (std::uint32_t step = 0; step < kBlockK / 16; ++step) {  // 32 bytes along K = two descriptor units
                                umaF16Pair(tmem_base, a_lo + 2 * step, b_hi + 2 * step, instruction, !fresh || step != 0 ? 1U : 0U);
                                umaF16Pair(tmem_base, a_hi + 2 * step, b_lo + 2 * step, instruction, 1U);
                            }
                        } else {
#pragma unroll
                            for (std::uint32_t step = 0; step < kBlockK / 16; ++step) {
                                umaF16Pair(tmem_base + kHColumn, a_hi + 2 * step, b_hi + 2 * step, instruction, !fresh || step != 0 ? 1U : 0U);
                            }
                        }
                        umaCommitPair(&bars->empty[ring.slot]);
                        --in_slab;
                        if (--in_sum == 0) { umaCommitPair(sum_full); }
                    }
                }
                if (!ok) {
                    *abort_flag = 1;
                    // Let MMAs already issued finish before tensor memory is freed.
                    std::uint64_t* const flush = cross ? &bars->flush_x : &bars->flush_h;
                    umaCommitPair(flush);
                    int never = 0;
                    mbarrierWait(flush, 0, &never);
                }
            }
            __syncwarp();
        }
    }

    __syncthreads();
    if (*abort_flag != 0) {
        if (threadIdx.x == 0) {
            if (p.status != nullptr) { *p.status = 2; }
            // Copies that were armed but never consumed may still be landing (their bytes count on the
            // first CTA's barriers; the second waits for the first below).
            int never = 0;
            for (int s = 0; s < kStages && rank == 0; ++s) {
                mbarrierWait(&bars->full[s], 0, &never);
                mbarrierWait(&bars->full[s], 1, &never);
            }
        }
        __syncthreads();
    }
    tcgen05FenceBeforeSync();
    clusterBarrierArrive();
    clusterBarrierWait();
    if (warp == kCrossWarp) {
        tcgen05FenceAfterSync();
        tmemFreePair(tmem_base, kTmemColumns);
    }
}

// K blocks (of 64) accumulated into H between two drains: the largest divisor of the slab's that is at most the TF32 kernel's
// interval of blocks of 32. The tensor core cuts every product off at a few bits below the last one of the sum so far; with
// products of one sign that adds up to a bias in proportion to the products in a chain, whatever the width of its MMAs. So a
// chain may be twice as deep as the TF32 kernel's, which takes the small products into the same sum, and no deeper. Error against 64 bits,
// |N(0,1)| operands, K = 512 / 1024 / 2048 / 4096 / 8192: 2.1e-7 / 5.1e-7 / 7.8e-7 / 1.2e-6 / 1.7e-6 (TF32 form 2.3e-7 / 5.2e-7 / 7.8e-7 /
// 1.5e-6 / 2.1e-6); with chains three times as long 5.1e-7 / 1.7e-6 / 1.8e-6 / 3.9e-6 / 3.6e-6, for 4 to 7 % of the time.
std::uint32_t chunkBlocks(std::uint64_t k) {
    const std::uint32_t interval = tf32x3::drainInterval(k);
    std::uint32_t blocks         = kSlabBlocks;
    while (blocks > interval || kSlabBlocks % blocks != 0) { --blocks; }
    return blocks;
}

std::uint64_t roundUp(std::uint64_t x, std::uint64_t unit) { return (x + unit - 1) / unit * unit; }

// A's rows and B's columns as the split sees them.
void describeOperands(const FtcudaGemmDesc& desc, fp16x3::SplitOperand (&operands)[2]) {
    operands[0]            = {};
    operands[0].source     = desc.a;
    operands[0].row_stride = desc.a_row_stride;
    operands[0].k_stride   = desc.a_col_stride;
    operands[0].rows       = static_cast<std::uint32_t>(desc.m);
    operands[1]            = {};
    operands[1].source     = desc.b;
    operands[1].row_stride = desc.b_col_stride;
    operands[1].k_stride   = desc.b_row_stride;
    operands[1].rows       = static_cast<std::uint32_t>(desc.n);
    operands[1].grouped    = 1;
}

}  // namespace

const char* supportsPrepared(const FtcudaGemmDesc& desc) {
    if (desc.m * desc.n == 0 || desc.k < 256) { return "too small or too shallow to be worth splitting the operands"; }
    if (desc.m >= (1ULL << 24) || desc.n >= (1ULL << 24) || desc.k >= (1ULL << 24)) { return "an extent is too large for the prepared form"; }
    if (desc.a == nullptr || desc.b == nullptr) { return "an operand has no address"; }
    if (ceilDiv(desc.m, 8) * ceilDiv(desc.k, 1024) >= (1ULL << 30) || ceilDiv(desc.n, 8) * ceilDiv(desc.k, 1024) >= (1ULL << 30)) {
        return "too many blocks for the prepared form";
    }
    return nullptr;
}

int configurePrepared(LaunchState& state, const FtcudaGemmDesc& desc, char* message, std::size_t capacity) {
    int sms = 0;
    if (!deviceSmCount(desc.device, &sms, message, capacity)) { return 1; }
    PreparedState& prepared = state.prepared;
    prepared.desc           = desc;
    const std::uint64_t k_blocks = ceilDiv(desc.k, kBlockK);
    const std::uint64_t pairs    = static_cast<std::uint64_t>(sms) / 2;
    const fp16x3::Geometry geometry = fp16x3::chooseGeometry(desc.m, desc.n, k_blocks, pairs);
    prepared.tile_n              = geometry.tile_n;
    prepared.splits              = geometry.splits;
    prepared.blocks_per_split    = geometry.blocks_per_split;
    prepared.chunk_blocks        = chunkBlocks(desc.k);
    const std::uint64_t items    = ceilDiv(desc.m, kTileM) * ceilDiv(desc.n, geometry.tile_n) * geometry.splits;
    prepared.grid                = static_cast<std::uint32_t>(2 * (items < pairs ? items : pairs));

    const std::uint64_t rows[2] = {desc.m, desc.n};
    const std::uint64_t slabs   = ceilDiv(k_blocks, kSlabBlocks);
    fp16x3::SplitOperand operands[2];
    describeOperands(desc, operands);
    for (fp16x3::SplitOperand& operand : operands) { fp16x3::planSplit(operand, static_cast<std::uint32_t>(slabs)); }
    std::uint64_t at            = 256;  // the decision
    prepared.verdicts_at        = at;
    at += roundUp((static_cast<std::uint64_t>(operands[0].blocks) + operands[1].blocks) * 4, 256);
    for (int i = 0; i < 2; ++i) {
        prepared.inverse_pitch[i] = roundUp(ceilDiv(rows[i], i == 0 ? 1 : fp16x3::kColumnGroup), 4);
        prepared.inverse_at[i]    = at;
        at += roundUp(slabs * prepared.inverse_pitch[i] * 4, 256);
    }
    for (int i = 0; i < 2; ++i) {
        prepared.split_at[i] = at;
        at += roundUp(rows[i] * k_blocks * kBlockBytes, 256);
    }
    prepared.partials_at = at;
    if (prepared.splits > 1) { at += static_cast<std::uint64_t>(prepared.splits) * desc.m * desc.n * sizeof(float); }
    // The fallback's own workspace lies over all of this but the decision: it runs when none of it is needed any more.
    const std::uint64_t fallback = 256 + state.workspace_bytes;
    state.workspace_bytes        = (at > fallback ? at : fallback) + 256;

    // Encoded for a stand-in address; re-pointed at the workspace in front of every launch.
    const void* stand_in = reinterpret_cast<const void*>(std::uintptr_t{256});
    if (!encodeSplitMap(&prepared.map_a, stand_in, desc.m, k_blocks, 128, message, capacity) ||
        !encodeSplitMap(&prepared.map_b, stand_in, desc.n, k_blocks, prepared.tile_n / 2, message, capacity)) {
        return 1;
    }
    cudaError_t error = cudaFuncSetAttribute(tensorGemm3xFp16, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (error == cudaSuccess) { error = fp16x3::configureSplit(); }
    if (error != cudaSuccess) { return fail(message, capacity, 1, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(error)); }
    return 0;
}

cudaError_t launchPrepared(const LaunchState& state, void* workspace, cudaStream_t stream, char* message, std::size_t capacity) {
    const PreparedState& prepared = state.prepared;
    const FtcudaGemmDesc& desc    = prepared.desc;
    unsigned char* const base     = reinterpret_cast<unsigned char*>((reinterpret_cast<std::uintptr_t>(workspace) + 255) & ~std::uintptr_t{255});
    std::uint32_t* const decision = reinterpret_cast<std::uint32_t*>(base);
    std::uint32_t* const verdicts = reinterpret_cast<std::uint32_t*>(base + prepared.verdicts_at);

    fp16x3::SplitParams split{};
    split.k        = static_cast<std::uint32_t>(desc.k);
    split.k_blocks = static_cast<std::uint32_t>(ceilDiv(desc.k, kBlockK));
    split.slabs    = static_cast<std::uint32_t>(ceilDiv(split.k_blocks, kSlabBlocks));
    describeOperands(desc, split.operand);
    for (int i = 0; i < 2; ++i) {
        fp16x3::SplitOperand& o = split.operand[i];
        o.split                 = base + prepared.split_at[i];
        o.inverse               = reinterpret_cast<float*>(base + prepared.inverse_at[i]);
        o.pitch                 = prepared.inverse_pitch[i];
        fp16x3::planSplit(o, split.slabs);
        o.verdicts = verdicts + (i == 0 ? 0 : split.operand[0].blocks);
    }
    cudaError_t error = fp16x3::launchSplit(split, stream);
    if (error != cudaSuccess) { return error; }

    CUtensorMap map_a = prepared.map_a, map_b = prepared.map_b;
    if (!replaceMapAddress(&map_a, split.operand[0].split) || !replaceMapAddress(&map_b, split.operand[1].split)) {
        fail(message, capacity, 1, "cuTensorMapReplaceAddress failed");
        return cudaErrorInvalidValue;
    }
    Fp16Params p{};
    p.c                = desc.c;
    p.d                = desc.d;
    p.c_row_stride     = desc.c_row_stride;
    p.c_col_stride     = desc.c_col_stride;
    p.d_row_stride     = desc.d_row_stride;
    p.d_col_stride     = desc.d_col_stride;
    p.m                = static_cast<std::uint32_t>(desc.m);
    p.n                = static_cast<std::uint32_t>(desc.n);
    p.k                = split.k;
    p.k_blocks         = split.k_blocks;
    p.blocks_per_split = prepared.blocks_per_split;
    p.splits           = prepared.splits;
    p.tiles_m          = static_cast<std::uint32_t>(ceilDiv(desc.m, kTileM));
    p.tiles_n          = static_cast<std::uint32_t>(ceilDiv(desc.n, prepared.tile_n));
    p.tile_n           = prepared.tile_n;
    p.band_m_tiles     = 8;
    p.chunk_blocks     = prepared.chunk_blocks;
    p.alpha            = desc.alpha;
    p.beta             = desc.beta;
    p.partials         = prepared.splits > 1 ? reinterpret_cast<float*>(base + prepared.partials_at) : nullptr;
    p.inverse_a        = split.operand[0].inverse;
    p.inverse_b        = split.operand[1].inverse;
    p.inverse_pitch_a  = prepared.inverse_pitch[0];
    p.inverse_pitch_b  = prepared.inverse_pitch[1];
    p.verdicts         = verdicts;
    p.slabs            = split.slabs;
    for (int i = 0; i < 2; ++i) { p.verdicts_per_slab[i] = split.operand[i].blocks / split.slabs; }
    p.use_fallback     = decision;
    p.status           = state.device_status;
    const auto aligned = [&](std::uint32_t width, const float* at, std::int64_t row_stride, std::int64_t col_stride) {
        return desc.n % width == 0 && col_stride == 1 && row_stride % width == 0 && reinterpret_cast<std::uintptr_t>(at) % (4 * width) == 0;
    };
    for (const std::uint32_t width : {8U, 4U}) {
        const bool fits = p.partials != nullptr ? aligned(width, p.partials, static_cast<std::int64_t>(desc.n), 1)
                                                : aligned(width, desc.d, desc.d_row_stride, desc.d_col_stride) &&
                                                      (desc.c == nullptr || aligned(width, desc.c, desc.c_row_stride, desc.c_col_stride));
        if (fits) {
            p.vector = width;
            break;
        }
    }
    const std::uint32_t items = p.tiles_m * p.tiles_n * p.splits;
    cudaLaunchConfig_t config{};
    config.gridDim          = dim3(prepared.grid, 1, 1);
    config.blockDim         = dim3(kThreads, 1, 1);
    config.dynamicSmemBytes = kSmemBytes;
    config.stream           = stream;
    cudaLaunchAttribute attribute{};
    attribute.id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs                                         = &attribute;
    config.numAttrs                                      = 1;
    error = cudaLaunchKernelEx(&config, tensorGemm3xFp16, map_a, map_b, p, items);
    if (error != cudaSuccess) { return error; }
    countLaunches(1);
    if (prepared.splits > 1) {
        error = launchSplitKReduce(desc, p.partials, prepared.splits, stream, decision, false);
        if (error != cudaSuccess) { return error; }
        countLaunches(1);
    }
    LaunchState fallback = state;
    fallback.kernel      = prepared.fallback_kernel;
    fallback.run_if      = decision;
    return launchTensorStaged(fallback, base + 256, stream, message, capacity);
}

}  // namespace ftcuda
