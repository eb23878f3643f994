// The prepared form of the 3xTF32 families: D = alpha A B + beta C from operands split into FP16 pairs.
//
// A TF32 number and an FP16 number have the same 11 significant bits, and the tensor cores multiply
// FP16 at twice the rate. With the operands scaled row by row (gemm_fp16x3_split.cu, which also says
// when that is exact enough and leaves the launch to the TF32 kernel when it is not),
//   a b = a_hi b_hi + (a_lo b_hi + a_hi b_lo) / 2^11,     a = a_hi + a_lo / 2^11, b likewise,
// is three tcgen05.mma.kind::f16 products in half the tensor time of three TF32 ones, with less
// rounding in the low parts (2^-24 against a truncation at 2^-21). And because the operands arrive
// split, no warp converts anything here: the conversion, which every CTA of the TF32 kernel repeats
// for every tile, is paid once per operand element, and the tensor cores wait for TMA alone.
//
// A pair of CTAs (tcgen05 cta_group::2, a cluster of two) shares an output tile of 256 rows and up to
// 256 columns, K walked in blocks of 64. Each CTA brings its 128 rows of A and half of the tile's rows
// of B (B is K-major here whatever the caller's orientation), high and low parts, in two TMA copies:
// at most 64 KiB a stage, three stages. One thread of the pair's first CTA issues the MMAs of both.
//
//   warp 0       TMA producer (one thread, in both CTAs; the bytes of both count on the first CTA's barrier)
//   warp 1       MMA issuer (one thread of the first CTA)
//   warps 4-11   drain / epilogue, 32 rows x half of the columns each
//
// Tensor memory holds two accumulators, 512 columns in all: H (a_hi b_hi) and X (the two cross products).
// The tensor core's FP32 additions truncate, so H is drained into registers every `chunk_blocks` K blocks
// and added up there to nearest (see drainInterval in tf32x3_common.cuh); X, 2^11 times smaller in
// effect, is read once per tile. In a K block the cross products are issued first: while the drain
// warps read H, the tensor core works on the next block's eight MMAs into X, and at the end of a tile
// X is read behind the last block's H products. The drain so costs the tensor pipe nothing; it cost
// the TF32 kernel 4 %.
//
// The epilogue turns each warp's 32 x 32 pieces in shared memory so that a row's 128 bytes are written
// (and C's read) by eight neighbouring lanes, and undoes the scaling with the rows' and columns' powers
// of two, exactly.
//
// Measured, the whole launch with its split: 16384 x 4096 x 14336 8.81 -> 4.52 ms (218 -> 426 TFLOP/s; this kernel alone
// 499, three times that in FP16 products, 0.91 of the measured dense BF16 rate: what bounds it is the power limit),
// 4096^3 688 -> 471 us.
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

using fp16x3::Control;
using fp16x3::kBlockBytes;
using fp16x3::kBlockK;

constexpr int kTileM      = 256;  // of a CTA pair
constexpr int kMaxTileN   = 256;
constexpr int kStages     = 3;
constexpr int kThreads    = 384;
constexpr int kABytes     = 128 * static_cast<int>(kBlockBytes);          // hi | lo, 16 KiB each
constexpr int kStageBytes = kABytes + kMaxTileN / 2 * static_cast<int>(kBlockBytes);
constexpr int kTurnOffset = kStages * kStageBytes;                        // 4 KiB per epilogue warp
constexpr int kBarrierOffset = kTurnOffset + 8 * 4096;
constexpr int kSmemBytes     = kBarrierOffset + 256 + 1024;
static_assert(kSmemBytes <= 232448, "shared memory of one CTA");

constexpr int kRegsLight = 72;   // producer, issuer (warpgroup 0)
constexpr int kRegsDrain = 216;  // drain / epilogue (warpgroups 1, 2)
static_assert(128 * kRegsLight + 256 * kRegsDrain <= 168 * kThreads, "the CTA's register pool is what it was launched with");
constexpr int kProducerWarp  = 0;
constexpr int kMmaWarp       = 1;
constexpr int kFirstEpilogue = 4;
constexpr std::uint32_t kTmemColumns = 512;
constexpr std::uint32_t kHColumn     = 256;  // X at 0

struct Barriers {
    std::uint64_t full[kStages];   // used in the pair's first CTA
    std::uint64_t empty[kStages];
    std::uint64_t x_full, h_full;
    std::uint64_t x_empty, h_empty;  // used in the pair's first CTA
    std::uint64_t flush;
    std::uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(Barriers) <= 256, "barrier block");

struct Fp16Params {
    const float* c;
    float* d;
    std::int64_t c_row_stride, c_col_stride;
    std::int64_t d_row_stride, d_col_stride;
    std::uint32_t m, n;
    std::uint32_t k_blocks, blocks_per_split, splits;
    std::uint32_t tiles_m, tiles_n, tile_n, band_m_tiles;
    std::uint32_t chunk_blocks;
    float alpha, beta;
    float* partials;  // non-null: unscaled sums of the K slices, [split][m][n]
    const float* inverse_a;
    const float* inverse_b;
    const Control* control;
    std::uint32_t vector;  // 16-byte accesses to the output and to C are aligned
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

// Rows and columns of one warp's share, written 32 columns at a time.
__device__ __forceinline__ void writePiece(const Fp16Params& p, const Item& w, std::uint32_t row0, std::uint32_t col0,
                                           unsigned char* turn, int lane, const float* values) {
    // A thread holds 32 columns of its row; 16-byte chunks are stored XOR-ed with the row so that
    // neither side of the turn has bank conflicts.
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        *reinterpret_cast<float4*>(turn + lane * 128 + ((c ^ (lane & 7)) << 4)) =
            make_float4(values[4 * c], values[4 * c + 1], values[4 * c + 2], values[4 * c + 3]);
    }
    __syncwarp();
    const std::uint32_t col = col0 + (lane & 7) * 4;
    float cs[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) { cs[j] = col + j < p.n ? p.inverse_b[col + j] : 0.0F; }
    const bool partial = p.partials != nullptr;
    float* const out   = partial ? p.partials + static_cast<std::uint64_t>(w.split) * p.m * p.n : p.d;
    const std::int64_t row_stride = partial ? p.n : p.d_row_stride;
    const std::int64_t col_stride = partial ? 1 : p.d_col_stride;
    const float* const c          = partial ? nullptr : p.c;
    const float alpha             = partial ? 1.0F : p.alpha;
    const bool vector             = p.vector != 0 && col + 4 <= p.n;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r             = i * 4 + (lane >> 3);
        const std::uint32_t row = row0 + r;
        const float4 v = *reinterpret_cast<const float4*>(turn + r * 128 + (((lane & 7) ^ (r & 7)) << 4));
        if (row >= p.m) { continue; }
        float o[4] = {v.x * cs[0] * alpha, v.y * cs[1] * alpha, v.z * cs[2] * alpha, v.w * cs[3] * alpha};
        float* const at = out + static_cast<std::int64_t>(row) * row_stride + static_cast<std::int64_t>(col) * col_stride;
        if (vector) {
            if (c != nullptr) {
                const float4 addend = *reinterpret_cast<const float4*>(c + static_cast<std::int64_t>(row) * p.c_row_stride + col);
                o[0] += p.beta * addend.x;
                o[1] += p.beta * addend.y;
                o[2] += p.beta * addend.z;
                o[3] += p.beta * addend.w;
            }
            *reinterpret_cast<float4*>(at) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (col + j >= p.n) { continue; }
                if (c != nullptr) {
                    o[j] += p.beta * c[static_cast<std::int64_t>(row) * p.c_row_stride + static_cast<std::int64_t>(col + j) * p.c_col_stride];
                }
                at[j * col_stride] = o[j];
            }
        }
    }
    __syncwarp();
}

__global__ void __launch_bounds__(kThreads, 1) __cluster_dims__(2, 1, 1)
tensorGemm3xFp16(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b, const Fp16Params p,
                 const std::uint32_t num_items) {
    extern __shared__ unsigned char smem_raw[];
    // The decision of the split: every CTA leaves together.
    if (p.control->use_fallback != 0) { return; }
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
            mbarrierInit(&bars->empty[s], 1);
        }
        mbarrierInit(&bars->x_full, 1);
        mbarrierInit(&bars->h_full, 1);
        mbarrierInit(&bars->x_empty, 16);
        mbarrierInit(&bars->h_empty, 16);
        mbarrierInit(&bars->flush, 1);
        bars->abort_flag = 0;
        fenceBarrierInit();
        prefetchTensorMap(&map_a);
        prefetchTensorMap(&map_b);
    }
    if (warp == kMmaWarp) { tmemAllocatePair(&bars->tmem_base, kTmemColumns); }
    tcgen05FenceBeforeSync();
    __syncthreads();
    clusterBarrierArrive();
    clusterBarrierWait();
    tcgen05FenceAfterSync();
    const std::uint32_t tmem_base = bars->tmem_base;

    if (warp >= kFirstEpilogue) {
        registersGrow<kRegsDrain>();
        const int e                   = warp - kFirstEpilogue;  // 0..7; warp % 4 is the tensor-memory lane quadrant
        const std::uint32_t in_tile   = static_cast<std::uint32_t>(32 * (e & 3));
        const std::uint32_t tmem_row  = tmem_base + (in_tile << 16);
        const std::uint32_t pieces    = p.tile_n / 32;
        const std::uint32_t first     = (e >> 2) != 0 ? (pieces + 1) / 2 : 0;  // this warp's pieces of 32 columns
        const std::uint32_t mine      = (e >> 2) != 0 ? pieces / 2 : (pieces + 1) / 2;
        unsigned char* turn           = smem + kTurnOffset + e * 4096;
        const std::uint32_t x_empty   = mapToRank(&bars->x_empty, 0);
        const std::uint32_t h_empty   = mapToRank(&bars->h_empty, 0);
        std::uint32_t items = 0, chunks = 0;
        bool ok = true;
        for (std::uint32_t item = pair; item < num_items && ok; item += pairs, ++items) {
            const Item w                   = decode(p, item);
            const std::uint32_t num_chunks = (w.blocks + p.chunk_blocks - 1) / p.chunk_blocks;
            float acc[128];
#pragma unroll
            for (int j = 0; j < 128; ++j) { acc[j] = 0.0F; }
            for (std::uint32_t chunk = 0; chunk < num_chunks && ok; ++chunk, ++chunks) {
                if (chunk + 1 == num_chunks) {
                    ok = mbarrierWait(&bars->x_full, items & 1, abort_flag);
                    if (!ok) { break; }
                    tcgen05FenceAfterSync();
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        if (static_cast<std::uint32_t>(q) < mine) {
                            float x[32];
                            tmemLoad32(tmem_row + (first + q) * 32, x);
#pragma unroll
                            for (int j = 0; j < 32; ++j) { acc[q * 32 + j] += x[j] * 0x1p-11F; }
                        }
                    }
                    tcgen05FenceBeforeSync();
                    __syncwarp();
                    if (lane == 0) { mbarrierArriveCluster(x_empty); }
                }
                ok = mbarrierWait(&bars->h_full, chunks & 1, abort_flag);
                if (!ok) { break; }
                tcgen05FenceAfterSync();
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if (static_cast<std::uint32_t>(q) < mine) {
                        float h[32];
                        tmemLoad32(tmem_row + kHColumn + (first + q) * 32, h);
#pragma unroll
                        for (int j = 0; j < 32; ++j) { acc[q * 32 + j] += h[j]; }
                    }
                }
                tcgen05FenceBeforeSync();
                __syncwarp();
                if (lane == 0) { mbarrierArriveCluster(h_empty); }
            }
            if (!ok) { break; }
            const std::uint32_t row0 = w.row + rank * 128 + in_tile;
            const std::uint32_t row  = row0 + lane;
            const float row_scale    = row < p.m ? p.inverse_a[row] : 0.0F;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const std::uint32_t col0 = w.col + (first + q) * 32;
                if (static_cast<std::uint32_t>(q) < mine && col0 < p.n && row0 < p.m) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) { acc[q * 32 + j] *= row_scale; }
                    writePiece(p, w, row0, col0, turn, lane, acc + q * 32);
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
                std::uint32_t s = 0, parity = 1;
                std::uint32_t filled = 0;
                for (std::uint32_t item = pair; item < num_items && ok; item += pairs) {
                    const Item w = decode(p, item);
                    const std::int32_t row_a = static_cast<std::int32_t>(w.row + rank * 128);
                    const std::int32_t row_b = static_cast<std::int32_t>(w.col + rank * (p.tile_n / 2));
                    for (std::uint32_t kb = 0; kb < w.blocks; ++kb) {
                        ok = mbarrierWait(&bars->empty[s], parity, abort_flag);
                        if (!ok) { break; }
                        // The bytes of both CTAs count on the first CTA's barrier, which that CTA arms. (The other's
                        // may land first: the phase cannot complete before it has been armed.)
                        if (rank == 0) { mbarrierArriveExpectTx(&bars->full[s], 2 * stage_bytes); }
                        const std::uint32_t full  = mapToRank(&bars->full[s], 0);
                        unsigned char* const slot = smem + s * kStageBytes;
                        const std::int32_t z      = static_cast<std::int32_t>((w.first_block + kb) * 2);
                        tmaLoad3dPair(slot, &map_a, full, 0, row_a, z);
                        tmaLoad3dPair(slot + kABytes, &map_b, full, 0, row_b, z);
                        ++filled;
                        if (++s == kStages) {
                            s = 0;
                            parity ^= 1;
                        }
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
        } else if (warp == kMmaWarp && rank == 0) {
            if (lane == 0) {
                const std::uint32_t instruction = umaInstructionF16(kTileM, p.tile_n);
                const std::uint32_t b_low       = p.tile_n / 2 * 128;  // bytes of B's high part in a stage
                std::uint32_t s = 0, parity = 0;
                std::uint32_t items = 0, chunks = 0;
                bool ok = true;
                for (std::uint32_t item = pair; item < num_items && ok; item += pairs, ++items) {
                    const Item w           = decode(p, item);
                    std::uint32_t in_chunk = 0;
                    for (std::uint32_t kb = 0; kb < w.blocks; ++kb) {
                        const bool last = kb + 1 == w.blocks;
                        if (kb == 0) { ok = mbarrierWait(&bars->x_empty, (items & 1) ^ 1, abort_flag); }
                        ok = ok && mbarrierWait(&bars->full[s], parity, abort_flag);
                        if (!ok) { break; }
                        tcgen05FenceAfterSync();
                        const std::uint32_t slot  = smemAddress(smem + s * kStageBytes);
                        const std::uint64_t a_hi  = umaDescriptorK128(slot);
                        const std::uint64_t a_lo  = umaDescriptorK128(slot + 128 * 128);
                        const std::uint64_t b_hi  = umaDescriptorK128(slot + kABytes);
                        const std::uint64_t b_lo  = umaDescriptorK128(slot + kABytes + b_low);
#pragma unroll
                        for (std::uint32_t step = 0; step < kBlockK / 16; ++step) {  // 32 bytes along K = two descriptor units
                            umaF16Pair(tmem_base, a_lo + 2 * step, b_hi + 2 * step, instruction, kb != 0 || step != 0 ? 1U : 0U);
                            umaF16Pair(tmem_base, a_hi + 2 * step, b_lo + 2 * step, instruction, 1U);
                        }
                        if (last) { umaCommitPair(&bars->x_full); }
                        if (in_chunk == 0) {
                            ok = mbarrierWait(&bars->h_empty, (chunks & 1) ^ 1, abort_flag);
                            if (!ok) { break; }
                            tcgen05FenceAfterSync();
                            ++chunks;
                        }
#pragma unroll
                        for (std::uint32_t step = 0; step < kBlockK / 16; ++step) {
                            umaF16Pair(tmem_base + kHColumn, a_hi + 2 * step, b_hi + 2 * step, instruction,
                                       in_chunk != 0 || step != 0 ? 1U : 0U);
                        }
                        umaCommitPair(&bars->empty[s]);
                        if (++in_chunk == p.chunk_blocks || last) {
                            umaCommitPair(&bars->h_full);
                            in_chunk = 0;
                        }
                        if (++s == kStages) {
                            s = 0;
                            parity ^= 1;
                        }
                    }
                }
                if (!ok) {
                    *abort_flag = 1;
                    // Let MMAs already issued finish before tensor memory is freed.
                    umaCommitPair(&bars->flush);
                    int never = 0;
                    mbarrierWait(&bars->flush, 0, &never);
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
    if (warp == kMmaWarp) {
        tcgen05FenceAfterSync();
        tmemFreePair(tmem_base, kTmemColumns);
    }
}

// K blocks (of 64) accumulated into H between two drains. A block is four truncating additions where the TF32 kernel
// makes twelve for half of the depth. Relative error against float64 at K = 4096: 4.3e-7 with a drain every 5
// blocks, 7.8e-7 every 10 (the choice there), 1.14e-6 every 15, 4.9e-6 never; the TF32 kernel 1.13e-6. The time
// does not depend on it (447, 445, 462, 428 us).
std::uint32_t preparedChunkBlocks(std::uint64_t k) {
    return 2 * tf32x3::drainInterval(k);
}

std::uint64_t roundUp(std::uint64_t x, std::uint64_t unit) { return (x + unit - 1) / unit * unit; }

// Tile width and K slices. Modelled cost in SM cycles: a K step of 16 is three MMAs of tile_n / 2 cycles each, or the
// shared-memory traffic behind them (operand fetches and TMA writes at 128 bytes a cycle) where that is longer, which it is
// under 192 columns; a tile costs about 4000 more (pipeline fill, last drain, output); K slices cost a second
// kernel and their sums' way through memory.
struct Geometry {
    std::uint32_t tile_n, splits, blocks_per_split;
    double cycles;
};

Geometry chooseGeometry(std::uint64_t m, std::uint64_t n, std::uint64_t k_blocks, std::uint64_t pairs) {
    Geometry best{kMaxTileN, 1, static_cast<std::uint32_t>(k_blocks), 0.0};
    for (std::uint32_t width = kMaxTileN; width >= 64; width -= 32) {
        const std::uint64_t tiles = ceilDiv(m, kTileM) * ceilDiv(n, width);
        const double mma          = 1.5 * width;
        const double smem         = 160.0 + 0.625 * width;
        const double block_cycles = 4.0 * (mma > smem ? mma : smem);
        for (std::uint32_t splits = 1; splits <= 32; ++splits) {
            const std::uint64_t per_split = ceilDiv(k_blocks, splits);
            if (splits > 1 && (per_split < 4 || ceilDiv(k_blocks, per_split) != splits)) { continue; }
            if (tiles * splits >= (1ULL << 31)) { break; }
            double cycles = static_cast<double>(ceilDiv(tiles * splits, pairs)) * (static_cast<double>(per_split) * block_cycles + 4000.0);
            if (splits > 1) { cycles += 8000.0 + static_cast<double>(m) * static_cast<double>(n) * (8.0 * splits + 4.0) / 3500.0; }
            if (best.cycles == 0.0 || cycles < best.cycles) {
                best = Geometry{width, splits, static_cast<std::uint32_t>(per_split), cycles};
            }
        }
    }
    return best;
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
    const Geometry geometry      = chooseGeometry(desc.m, desc.n, k_blocks, pairs);
    prepared.tile_n              = geometry.tile_n;
    prepared.splits              = geometry.splits;
    prepared.blocks_per_split    = geometry.blocks_per_split;
    prepared.chunk_blocks        = preparedChunkBlocks(desc.k);
    const std::uint64_t items    = ceilDiv(desc.m, kTileM) * ceilDiv(desc.n, geometry.tile_n) * geometry.splits;
    prepared.grid                = static_cast<std::uint32_t>(2 * (items < pairs ? items : pairs));

    const std::uint64_t rows[2] = {desc.m, desc.n};
    std::uint64_t at            = 256;  // Control
    for (int i = 0; i < 2; ++i) {
        prepared.max_at[i] = at;
        at += roundUp(rows[i] * 4, 256);
        prepared.few_at[i] = at;
        at += roundUp(rows[i] * 4, 256);
    }
    prepared.cleared_bytes = at;
    for (int i = 0; i < 2; ++i) {
        prepared.inverse_at[i] = at;
        at += roundUp(rows[i] * 4, 256);
    }
    const std::uint64_t control_bytes = at;
    for (int i = 0; i < 2; ++i) {
        prepared.split_at[i] = at;
        at += roundUp(rows[i] * k_blocks * kBlockBytes, 256);
    }
    prepared.partials_at = at;
    if (prepared.splits > 1) { at += static_cast<std::uint64_t>(prepared.splits) * desc.m * desc.n * sizeof(float); }
    // The fallback's own workspace lies over the split operands, which it does not need.
    const std::uint64_t fallback = control_bytes + state.workspace_bytes;
    state.workspace_bytes        = (at > fallback ? at : fallback) + 256;

    // Encoded for a stand-in address; re-pointed at the workspace in front of every launch.
    const void* stand_in = reinterpret_cast<const void*>(std::uintptr_t{256});
    if (!encodeSplitMap(&prepared.map_a, stand_in, desc.m, k_blocks, 128, message, capacity) ||
        !encodeSplitMap(&prepared.map_b, stand_in, desc.n, k_blocks, prepared.tile_n / 2, message, capacity)) {
        return 1;
    }
    const cudaError_t error = cudaFuncSetAttribute(tensorGemm3xFp16, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes);
    if (error != cudaSuccess) { return fail(message, capacity, 1, "cudaFuncSetAttribute failed: %s", cudaGetErrorString(error)); }
    return 0;
}

cudaError_t launchPrepared(const LaunchState& state, void* workspace, cudaStream_t stream, char* message, std::size_t capacity) {
    const PreparedState& prepared = state.prepared;
    const FtcudaGemmDesc& desc    = prepared.desc;
    unsigned char* const base     = reinterpret_cast<unsigned char*>((reinterpret_cast<std::uintptr_t>(workspace) + 255) & ~std::uintptr_t{255});
    Control* const control        = reinterpret_cast<Control*>(base);
    cudaError_t error             = cudaMemsetAsync(base, 0, prepared.cleared_bytes, stream);
    if (error != cudaSuccess) { return error; }

    fp16x3::SplitParams split{};
    split.k        = static_cast<std::uint32_t>(desc.k);
    split.k_blocks = static_cast<std::uint32_t>(ceilDiv(desc.k, kBlockK));
    split.control  = control;
    const struct {
        const float* source;
        std::int64_t row_stride, k_stride;
        std::uint64_t rows;
    } sources[2] = {{desc.a, desc.a_row_stride, desc.a_col_stride, desc.m}, {desc.b, desc.b_col_stride, desc.b_row_stride, desc.n}};
    for (int i = 0; i < 2; ++i) {
        fp16x3::SplitOperand& o = split.operand[i];
        o.source                = sources[i].source;
        o.row_stride            = sources[i].row_stride;
        o.k_stride              = sources[i].k_stride;
        o.rows                  = static_cast<std::uint32_t>(sources[i].rows);
        o.split                 = base + prepared.split_at[i];
        o.row_max               = reinterpret_cast<std::uint32_t*>(base + prepared.max_at[i]);
        o.few                   = reinterpret_cast<std::uint32_t*>(base + prepared.few_at[i]);
        o.inverse               = reinterpret_cast<float*>(base + prepared.inverse_at[i]);
        fp16x3::planSplit(o, split.k);
    }
    error = fp16x3::launchSplit(split, stream);
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
    p.control          = control;
    p.status           = state.device_status;
    const auto aligned = [](const float* at, std::int64_t row_stride, std::int64_t col_stride) {
        return col_stride == 1 && row_stride % 4 == 0 && reinterpret_cast<std::uintptr_t>(at) % 16 == 0;
    };
    p.vector = p.partials != nullptr ? (desc.n % 4 == 0 ? 1U : 0U)
               : aligned(desc.d, desc.d_row_stride, desc.d_col_stride) && (desc.c == nullptr || aligned(desc.c, desc.c_row_stride, desc.c_col_stride))
                   ? 1U
                   : 0U;
    const std::uint32_t items = p.tiles_m * p.tiles_n * p.splits;
    tensorGemm3xFp16<<<prepared.grid, kThreads, kSmemBytes, stream>>>(map_a, map_b, p, items);
    error = cudaGetLastError();
    if (error != cudaSuccess) { return error; }
    countLaunches(1);
    if (prepared.splits > 1) {
        error = launchSplitKReduce(desc, p.partials, prepared.splits, stream, &control->use_fallback, false);
        if (error != cudaSuccess) { return error; }
        countLaunches(1);
    }
    LaunchState fallback = state;
    fallback.kernel      = prepared.fallback_kernel;
    fallback.run_if      = &control->use_fallback;
    return launchTensorStaged(fallback, base + prepared.split_at[0], stream, message, capacity);
}

}  // namespace ftcuda
