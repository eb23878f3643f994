// Splits A and B into pairs of FP16 numbers for gemm_fp16x3.cu.
//
// Every row of A and every column of B ("row" below, for both) is scaled by a power of two that
// brings its largest magnitude to [2^14, 2^15), and every scaled element x becomes
//   hi = fp16(x),  lo = fp16((x - hi) * 2^11)      (both to nearest even)
// so that x = hi + lo / 2^11 to within 2^-24 |x| as long as |x| >= 2^-12, i.e. for every element within
// 2^26 of its row's largest; below that ("gray" elements) to within 2^-36, which is 2^-50 of the largest.
//
// When that is enough. An element's error e contributes e * |b| to the result. For gray elements of a row of A
// the bound is 2^-50 max|a| max|b| each. If at least F_a elements of every row of A, and F_b of every
// column of B, reach 2^-8 of their row's largest, then any row and column have F_a + F_b - K positions
// where both do, so sum |a||b| >= (F_a + F_b - K) 2^-16 max|a| max|b|. With F_a + F_b - K >= K / 64 all
// gray elements of both together add at most 2 K 2^-50 against (K / 64) 2^-16: 2^-27 of sum |a||b| -- below
// the rounding of an FP32 product. Otherwise, or when a row's largest magnitude is outside
// [2^-60, 2^60], infinite or NaN, the launch is left to the TF32 kernel, which splits without
// scaling. No gray element at all needs no such count. The last CTA decides, on the device, for the
// whole launch.
//
// Both kernels are HBM-bound: the first reads the operands once (4 bytes an element), the second
// reads them again (from L2 when they fit) and writes as many bytes. At 16384 x 4096 x 14336 (502 MB of operands) 98 + 217 us,
// 5.1 and 4.6 TB/s.
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "fp16x3.hpp"
#include "gemm_kernels.hpp"

namespace ftcuda {
namespace fp16x3 {
namespace {

constexpr int kThreads           = 256;
constexpr std::uint32_t kMaxK    = 2048;  // row_max, source along K: 8 rows x 2048 K values per CTA
constexpr std::uint32_t kSplitK  = 1024;  // split, source along K: 8 rows x 1024 K values
constexpr std::uint32_t kTileR   = 128;   // source along its rows: 128 rows x ...
constexpr std::uint32_t kMaxTall = 128;   // ... 128 K values (row_max)
constexpr std::uint32_t kSplitTall = 256; // ... 256 K values (split)

constexpr std::uint32_t kLowestExponent  = 127 - 60;
constexpr std::uint32_t kHighestExponent = 127 + 60;

__device__ __forceinline__ std::uint32_t magnitude(float value) { return __float_as_uint(value) & 0x7FFFFFFFU; }

// Four consecutive K values of a row, zeros beyond the end.
__device__ __forceinline__ float4 loadAlongK(const SplitOperand& o, const float* row, std::uint32_t k, std::uint32_t depth) {
    if (o.vector != 0 && k + 4 <= depth) { return *reinterpret_cast<const float4*>(row + k); }
    float4 v = make_float4(0.0F, 0.0F, 0.0F, 0.0F);
    const float* at = row + static_cast<std::int64_t>(k) * o.k_stride;
    if (k < depth) { v.x = at[0]; }
    if (k + 1 < depth) { v.y = at[o.k_stride]; }
    if (k + 2 < depth) { v.z = at[2 * o.k_stride]; }
    if (k + 3 < depth) { v.w = at[3 * o.k_stride]; }
    return v;
}

__global__ void __launch_bounds__(kThreads) splitRowMax(const SplitParams p) {
    const std::uint32_t which = blockIdx.x < p.operand[0].max_blocks ? 0 : 1;
    const SplitOperand& o     = p.operand[which];
    const std::uint32_t block = blockIdx.x - (which != 0 ? p.operand[0].max_blocks : 0);
    const std::uint32_t warp  = threadIdx.x >> 5;
    const std::uint32_t lane  = threadIdx.x & 31;
    if (o.along_k != 0) {
        const std::uint32_t pieces = (p.k + kMaxK - 1) / kMaxK;
        const std::uint32_t row    = block / pieces * 8 + warp;
        const std::uint32_t begin  = block % pieces * kMaxK;
        if (row >= o.rows) { return; }
        const float* source  = o.source + static_cast<std::int64_t>(row) * o.row_stride;
        std::uint32_t most   = 0;
#pragma unroll 8
        for (std::uint32_t i = 0; i < kMaxK / 128; ++i) {
            const float4 v = loadAlongK(o, source, begin + i * 128 + lane * 4, p.k);
            most = max(max(max(most, magnitude(v.x)), max(magnitude(v.y), magnitude(v.z))), magnitude(v.w));
        }
        most = __reduce_max_sync(0xFFFFFFFFU, most);
        if (lane == 0 && most != 0) { atomicMax(o.row_max + row, most); }
        return;
    }
    // Along the rows: 32 consecutive rows per load, a warp takes 16 of the 128 K values.
    __shared__ std::uint32_t most_of[8][kTileR];
    const std::uint32_t pieces = (p.k + kMaxTall - 1) / kMaxTall;
    const std::uint32_t row0   = block / pieces * kTileR;
    const std::uint32_t begin  = block % pieces * kMaxTall + warp * (kMaxTall / 8);
    std::uint32_t most[4]      = {0, 0, 0, 0};
#pragma unroll 4
    for (std::uint32_t i = 0; i < kMaxTall / 8; ++i) {
        const std::uint32_t k = begin + i;
        const float* source   = o.source + static_cast<std::int64_t>(k) * o.k_stride;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const std::uint32_t row = row0 + lane + 32 * j;
            if (k < p.k && row < o.rows) { most[j] = max(most[j], magnitude(source[static_cast<std::int64_t>(row) * o.row_stride])); }
        }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) { most_of[warp][lane + 32 * j] = most[j]; }
    __syncthreads();
    if (threadIdx.x < kTileR && row0 + threadIdx.x < o.rows) {
        std::uint32_t all = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) { all = max(all, most_of[w][threadIdx.x]); }
        if (all != 0) { atomicMax(o.row_max + row0 + threadIdx.x, all); }
    }
}

// What a row's largest magnitude says about its scaling.
struct RowScale {
    float scale, inverse;
    bool covered;  // false: the row's magnitudes are out of range (the scale is then 1)
};
__device__ __forceinline__ RowScale rowScale(std::uint32_t most) {
    const std::uint32_t exponent = most >> 23;
    if (most == 0) { return {1.0F, 1.0F, true}; }
    if (exponent < kLowestExponent || exponent > kHighestExponent) { return {1.0F, 1.0F, false}; }
    // 2^(14 - (exponent - 127)) and its reciprocal, both normal numbers.
    return {__uint_as_float((268 - exponent) << 23), __uint_as_float((exponent - 14) << 23), true};
}

// hi | lo of one scaled element; counts what the decision needs.
__device__ __forceinline__ void splitElement(float x, __half& hi, __half& lo, std::uint32_t& few, bool& gray) {
    hi = __float2half_rn(x);
    lo = __float2half_rn((x - __half2float(hi)) * 2048.0F);
    const float size = fabsf(x);
    few += size < 128.0F ? 1U : 0U;              // 2^-8 of 2^15, the largest a row can hold
    gray = gray || (size < 0x1p-12F && x != 0.0F);
}

__device__ __forceinline__ std::uint32_t packed(__half a, __half b) {
    return static_cast<std::uint32_t>(__half_as_ushort(a)) | (static_cast<std::uint32_t>(__half_as_ushort(b)) << 16);
}

// Called by every thread of the CTA once its part is done. The last CTA of the grid decides.
__device__ __forceinline__ void finishSplit(const SplitParams& p) {
    __shared__ std::uint32_t last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) { last = atomicAdd(&p.control->blocks_done, 1U) + 1 == gridDim.x ? 1U : 0U; }
    __syncthreads();
    if (last == 0) { return; }
    __threadfence();
    const volatile Control* control = p.control;
    bool fallback                   = control->out_of_range != 0;
    if (!fallback && control->gray != 0) {
        // The largest number of small elements in a row, per operand.
        __shared__ std::uint32_t worst[2];
        if (threadIdx.x < 2) { worst[threadIdx.x] = 0; }
        __syncthreads();
        for (int which = 0; which < 2; ++which) {
            const SplitOperand& o = p.operand[which];
            std::uint32_t most    = 0;
#pragma unroll 8
            for (std::uint32_t row = threadIdx.x; row < o.rows; row += kThreads) { most = max(most, __ldcg(o.few + row)); }
            most = __reduce_max_sync(0xFFFFFFFFU, most);
            if ((threadIdx.x & 31) == 0) { atomicMax(&worst[which], most); }
        }
        __syncthreads();
        // F_a + F_b - K = K - worst_a - worst_b.
        fallback = static_cast<std::uint64_t>(worst[0]) + worst[1] + p.k / 64 + 1 > p.k;
    }
    if (threadIdx.x == 0) { p.control->use_fallback = fallback ? 1U : 0U; }
}

__global__ void __launch_bounds__(kThreads) splitOperands(const SplitParams p) {
    const std::uint32_t which = blockIdx.x < p.operand[0].split_blocks ? 0 : 1;
    const SplitOperand& o     = p.operand[which];
    const std::uint32_t block = blockIdx.x - (which != 0 ? p.operand[0].split_blocks : 0);
    const std::uint32_t warp  = threadIdx.x >> 5;
    const std::uint32_t lane  = threadIdx.x & 31;
    const std::uint64_t pitch = p.k_blocks * kBlockBytes;
    bool gray                 = false;
    bool covered              = true;
    if (o.along_k != 0) {
        const std::uint32_t pieces = (p.k + kSplitK - 1) / kSplitK;
        const std::uint32_t row    = block / pieces * 8 + warp;
        const std::uint32_t begin  = block % pieces * kSplitK;
        if (row < o.rows) {
            const RowScale scaling = rowScale(o.row_max[row]);
            const bool zero_row    = o.row_max[row] == 0;
            covered                = scaling.covered;
            const float* source    = o.source + static_cast<std::int64_t>(row) * o.row_stride;
            unsigned char* target  = o.split + row * pitch;
            std::uint32_t few      = 0;
            const std::uint32_t k_end = p.k_blocks * kBlockK;
            float4 v[kSplitK / 128];
#pragma unroll
            for (std::uint32_t i = 0; i < kSplitK / 128; ++i) { v[i] = loadAlongK(o, source, begin + i * 128 + lane * 4, p.k); }
#pragma unroll
            for (std::uint32_t i = 0; i < kSplitK / 128; ++i) {
                const std::uint32_t k = begin + i * 128 + lane * 4;
                if (k >= k_end) { continue; }
                __half hi[4], lo[4];
                splitElement(v[i].x * scaling.scale, hi[0], lo[0], few, gray);
                splitElement(v[i].y * scaling.scale, hi[1], lo[1], few, gray);
                splitElement(v[i].z * scaling.scale, hi[2], lo[2], few, gray);
                splitElement(v[i].w * scaling.scale, hi[3], lo[3], few, gray);
                // The zeros that fill up the last K block are not elements.
                if (k + 4 > p.k) { few -= k >= p.k ? 4U : k + 4 - p.k; }
                unsigned char* at = target + k / kBlockK * kBlockBytes + k % kBlockK * 2;
                *reinterpret_cast<uint2*>(at)               = make_uint2(packed(hi[0], hi[1]), packed(hi[2], hi[3]));
                *reinterpret_cast<uint2*>(at + 2 * kBlockK) = make_uint2(packed(lo[0], lo[1]), packed(lo[2], lo[3]));
            }
            few = __reduce_add_sync(0xFFFFFFFFU, few);
            if (lane == 0) {
                if (few != 0 && !zero_row) { atomicAdd(o.few + row, few); }
                if (begin == 0) { o.inverse[row] = scaling.inverse; }
            }
        }
    } else {
        // The tile is turned in shared memory: read along the rows, written along K. An odd pitch keeps
        // both sides within two accesses to a bank.
        __shared__ float tile[kBlockK][kTileR + 1];
        const std::uint32_t pieces = (p.k + kSplitTall - 1) / kSplitTall;
        const std::uint32_t row0   = block / pieces * kTileR;
        const std::uint32_t begin  = block % pieces * kSplitTall;
        const std::uint32_t eighth = lane & 7;  // this thread's 8 K values of a block
        std::uint32_t few[4]       = {0, 0, 0, 0};
        RowScale scaling[4];
        bool zero_row[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const std::uint32_t row  = row0 + warp * 16 + j * 4 + lane / 8;
            const std::uint32_t most = row < o.rows ? o.row_max[row] : 0;
            scaling[j]               = rowScale(most);
            zero_row[j]              = most == 0;
            covered                  = covered && scaling[j].covered;
            if (begin == 0 && eighth == 0 && row < o.rows) { o.inverse[row] = scaling[j].inverse; }
        }
        for (std::uint32_t k0 = begin; k0 < begin + kSplitTall && k0 < p.k; k0 += kBlockK) {
            float v[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const std::uint32_t k = k0 + warp * 8 + i;
                const float* source   = o.source + static_cast<std::int64_t>(k) * o.k_stride;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const std::uint32_t row = row0 + lane + 32 * j;
                    v[i][j] = k < p.k && row < o.rows ? source[static_cast<std::int64_t>(row) * o.row_stride] : 0.0F;
                }
            }
            __syncthreads();  // the previous block's tile has been read
#pragma unroll
            for (int i = 0; i < 8; ++i) {
#pragma unroll
                for (int j = 0; j < 4; ++j) { tile[warp * 8 + i][lane + 32 * j] = v[i][j]; }
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const std::uint32_t in_tile = warp * 16 + j * 4 + lane / 8;
                const std::uint32_t row     = row0 + in_tile;
                __half hi[8], lo[8];
                std::uint32_t small = 0;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    splitElement(tile[eighth * 8 + i][in_tile] * scaling[j].scale, hi[i], lo[i], small, gray);
                }
                const std::uint32_t k = k0 + eighth * 8;
                if (k + 8 > p.k) { small -= k >= p.k ? 8U : k + 8 - p.k; }
                few[j] += small;
                if (row < o.rows) {
                    unsigned char* at = o.split + row * pitch + k0 / kBlockK * kBlockBytes + eighth * 16;
                    *reinterpret_cast<uint4*>(at) = make_uint4(packed(hi[0], hi[1]), packed(hi[2], hi[3]), packed(hi[4], hi[5]), packed(hi[6], hi[7]));
                    *reinterpret_cast<uint4*>(at + 2 * kBlockK) =
                        make_uint4(packed(lo[0], lo[1]), packed(lo[2], lo[3]), packed(lo[4], lo[5]), packed(lo[6], lo[7]));
                }
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const std::uint32_t row = row0 + warp * 16 + j * 4 + lane / 8;
            std::uint32_t all       = few[j];
            all += __shfl_xor_sync(0xFFFFFFFFU, all, 1);
            all += __shfl_xor_sync(0xFFFFFFFFU, all, 2);
            all += __shfl_xor_sync(0xFFFFFFFFU, all, 4);
            if (eighth == 0 && row < o.rows && all != 0 && !zero_row[j]) { atomicAdd(o.few + row, all); }
        }
    }
    if (__any_sync(0xFFFFFFFFU, gray) && lane == 0) { p.control->gray = 1; }
    if (!__all_sync(0xFFFFFFFFU, covered) && lane == 0) { p.control->out_of_range = 1; }
    finishSplit(p);
}

}  // namespace

void planSplit(SplitOperand& o, std::uint32_t k) {
    const auto size = [](std::int64_t stride) { return stride < 0 ? -stride : stride; };
    o.along_k       = size(o.k_stride) <= size(o.row_stride) ? 1U : 0U;
    o.vector        = o.k_stride == 1 && o.row_stride % 4 == 0 && reinterpret_cast<std::uintptr_t>(o.source) % 16 == 0 ? 1U : 0U;
    const std::uint64_t rows8 = ceilDiv(o.rows, 8), tiles = ceilDiv(o.rows, kTileR);
    o.max_blocks   = static_cast<std::uint32_t>(o.along_k != 0 ? rows8 * ceilDiv(k, kMaxK) : tiles * ceilDiv(k, kMaxTall));
    o.split_blocks = static_cast<std::uint32_t>(o.along_k != 0 ? rows8 * ceilDiv(k, kSplitK) : tiles * ceilDiv(k, kSplitTall));
}

cudaError_t launchSplit(const SplitParams& p, cudaStream_t stream) {
    splitRowMax<<<p.operand[0].max_blocks + p.operand[1].max_blocks, kThreads, 0, stream>>>(p);
    cudaError_t error = cudaGetLastError();
    if (error != cudaSuccess) { return error; }
    splitOperands<<<p.operand[0].split_blocks + p.operand[1].split_blocks, kThreads, 0, stream>>>(p);
    error = cudaGetLastError();
    countLaunches(2);
    return error;
}

}  // namespace fp16x3
}  // namespace ftcuda
