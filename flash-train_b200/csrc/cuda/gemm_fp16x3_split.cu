// Splits A and B into pairs of FP16 numbers for gemm_fp16x3.cu.
//
// A "row" below is a row of A or a column of B. K is cut into slabs of 768. In each slab every row of A, and
// every 16 columns of B together, are scaled by a power of two that brings their largest magnitude there to
// [2^14, 2^15), and every scaled element x becomes
//   hi = fp16(x),  lo = fp16((x - hi) * 2^11)      (both to nearest even)
// so that x = hi + lo / 2^11 to within 2^-23 |x| as long as |x| >= 2^-12, i.e. for every element within
// 2^26 of the largest (1 + 2^-12 + 2^-23 is that far off: the low part is a tie); below that ("gray" elements) to within 2^-36, which is 2^-50 of the largest.
//
// When that is enough. An element's error e contributes e * |b| to the result: for a gray element of A at most
// 2^-50 M_a M_b, with M the largest magnitude that either scale allows for, and with g_a gray elements in a row of A and g_b in
// a column of B at most (g_a + g_b) 2^-50 M_a M_b in all. If at least F_a elements of every nonzero row of A
// reach 2^-s M_a and F_b of every nonzero column of B reach 2^-t M_b, any row and column have F_a + F_b - L of the slab's L
// positions where both do, so sum |a||b| over the slab is at least (F_a + F_b - L) 2^-(s+t) M_a M_b. With
// s + t = 18 and F_a + F_b - L >= (g_a + g_b) / 128, the gray elements add at most
// 2^-25 of sum |a||b|, below the rounding of an FP32 product. The elements are counted for s (and t) of 5, 9 and 13, so
// that an operand with a few very large elements -- outliers of activations -- is made up for by an even one; of the gray ones it
// is only told whether a row has up to 64 of them (two such rows need one position in common) or more (counted as L each). No
// gray element at all needs no count. All of this concerns one slab: a gray element here is no reason to mind a row that is
// nearly empty there. Where it is not enough, or a largest magnitude is outside [2^-100, 2^61), infinite or
// NaN, the launch is left to the TF32 kernel, which splits without scaling. Every CTA leaves a verdict; the
// multiplying kernel decides slab by slab and then for the whole launch.
//
// The scales belong to slabs, and not to whole rows, so that one pass is enough: a CTA holds a slab of
// some rows, takes their largest magnitudes, and converts. HBM-bound: 4 bytes read and 4 written an element.
// At 4096 x 4096 for each operand (134 MB read, as many written; 41 us at the copy rate) 49 us with both sources along K,
// 56 with both along their rows. (A pass over the operands for whole rows' maxima and a second one that
// converted took 31 + 65 us, and 4 us more in launches.)
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "fp16x3.hpp"
#include "gemm_kernels.hpp"
#include "ptx.cuh"

namespace ftcuda {
namespace fp16x3 {
namespace {

constexpr int kThreads = 512;
constexpr int kWarps   = kThreads / 32;
static_assert(kWarps == 2 * kSplitRows / 4 && kSlabBlocks % 2 == 0, "a warp takes four rows, half of the K blocks");
static_assert(kSplitRowsAlongK == kWarps && kSplitRowsAlongK == kColumnGroup, "a warp takes a row, a CTA a group of columns");
// A slab of 32 rows, [k][row]: the odd pitch keeps the stores free of bank conflicts and the loads along K within two
// accesses to a bank.
constexpr int kTilePitch = static_cast<int>(kSplitRows) + 1;
constexpr int kTileBytes = static_cast<int>(kSlabK) * kTilePitch * 4;

constexpr std::uint32_t kLowestExponent  = 127 - 100;
constexpr std::uint32_t kHighestExponent = 127 + 60;

// The larger magnitude; a NaN stays.
__device__ __forceinline__ float largerMagnitude(float a, float b) {
    float result;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(result) : "f"(a), "f"(fabsf(b)));
    return result;
}
__device__ __forceinline__ std::uint32_t warpMax(float magnitude) { return __reduce_max_sync(0xFFFFFFFFU, __float_as_uint(magnitude)); }

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

// What a row's largest magnitude (its bit pattern) says about its scaling.
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

__device__ __forceinline__ std::uint32_t grayElement(float x, float scale) { return x != 0.0F && fabsf(x * scale) < 0x1p-12F ? 1U : 0U; }

// Splits pairs of elements of one row and keeps what the verdict needs: how many reach each threshold (in the scaled
// numbers, whose largest is below 2^15), and the smallest nonzero magnitude. Gray elements are rare: they are only counted,
// in another pass over what the CTA still holds, where there are any.
struct PairSplitter {
    float2 scale;
    __half2 large[3];                  // counts, in halves: at most 2048 each
    std::uint32_t least = 0xFFFFFFFFU; // twice the bit pattern of a magnitude, less one

    __device__ __forceinline__ explicit PairSplitter(float s) : scale(make_float2(s, s)) {
#pragma unroll
        for (int t = 0; t < 3; ++t) { large[t] = __half2half2(__ushort_as_half(0)); }
    }
    __device__ __forceinline__ void split(float a, float b, std::uint32_t& hi, std::uint32_t& lo) {
        least = min(least, min(__float_as_uint(a) * 2U - 1U, __float_as_uint(b) * 2U - 1U));  // zero: the largest number
        const float2 x   = multiply2(make_float2(a, b), scale);
        const __half2 h  = __float22half2_rn(x);
        const float2 up  = multiply2(x, make_float2(2048.0F, 2048.0F));
        const float2 low = multiplyAdd2(__half22float2(h), make_float2(-2048.0F, -2048.0F), up);  // exact
        const __half2 l  = __float22half2_rn(low);
        const __half2 m  = __habs2(h);
        large[0] = __hadd2(large[0], __hge2(m, __float2half2_rn(0x1p10F)));
        large[1] = __hadd2(large[1], __hge2(m, __float2half2_rn(0x1p6F)));
        large[2] = __hadd2(large[2], __hge2(m, __float2half2_rn(0x1p2F)));
        hi       = *reinterpret_cast<const std::uint32_t*>(&h);
        lo       = *reinterpret_cast<const std::uint32_t*>(&l);
    }
    // The three counts, ten bits each (a slab of one row has at most 768).
    __device__ __forceinline__ std::uint32_t largeElements() const {
        std::uint32_t all = 0;
#pragma unroll
        for (int t = 0; t < 3; ++t) { all |= static_cast<std::uint32_t>(__low2float(large[t]) + __high2float(large[t])) << (10 * t); }
        return all;
    }
    __device__ __forceinline__ bool sawGray() const {
        return least != 0xFFFFFFFFU && __uint_as_float((least + 1U) / 2U) * scale.x < 0x1p-12F;
    }
};

// For each threshold the larger number of small elements, of `length`, given counts of large ones.
__device__ __forceinline__ void worstCounts(std::uint32_t (&worst)[3], std::uint32_t large, std::uint32_t length) {
#pragma unroll
    for (int t = 0; t < 3; ++t) { worst[t] = max(worst[t], length - (large >> (10 * t) & 0x3FFU)); }
}

__global__ void __launch_bounds__(kThreads, 2) splitOperands(const SplitParams p) {
    extern __shared__ float tile[];
    __shared__ std::uint32_t most_of[kWarps][kSplitRows];
    __shared__ std::uint32_t large_of[kSplitRows], gray_of[kSplitRows];
    __shared__ float scale_of[kSplitRows];
    __shared__ std::uint32_t worst_of[kWarps][3], state_of[kWarps];
    const std::uint32_t which = blockIdx.x < p.operand[0].blocks ? 0 : 1;
    const SplitOperand& o     = p.operand[which];
    const std::uint32_t block = blockIdx.x - (which != 0 ? p.operand[0].blocks : 0);
    const std::uint32_t warp  = threadIdx.x >> 5;
    const std::uint32_t lane  = threadIdx.x & 31;
    const std::uint64_t pitch = p.k_blocks * kBlockBytes;
    std::uint32_t state       = kAllCovered;
    std::uint32_t worst[3]    = {0, 0, 0};  // small elements of the worst row this thread knows
    gridDependencyWait();
    gridDependencyLaunchDependents();
    const std::uint32_t row_blocks = o.blocks / p.slabs;
    std::uint32_t slab, row_block, row0;
    if (o.along_k != 0) {  // neighbouring CTAs take neighbouring pieces of memory
        slab      = block % p.slabs;
        row_block = block / p.slabs;
        row0      = row_block * kSplitRowsAlongK;
    } else {
        slab      = block / row_blocks;
        row_block = block % row_blocks;
        row0      = row_block * kSplitRows;
    }
    const std::uint32_t begin  = slab * kSlabK;
    const std::uint32_t depth  = min(p.k, begin + kSlabK);
    const std::uint32_t length = depth - begin;
    const std::uint32_t k_end  = min(p.k_blocks * kBlockK, begin + kSlabK);
    if (o.along_k != 0) {
        // A warp takes a row, 128 K values per load.
        const std::uint32_t row = row0 + warp;
        const float* source     = o.source + static_cast<std::int64_t>(row) * o.row_stride;
        float4 v[kSlabK / 128];
#pragma unroll
        for (std::uint32_t i = 0; i < kSlabK / 128; ++i) {
            v[i] = row < o.rows ? loadAlongK(o, source, begin + i * 128 + lane * 4, depth) : make_float4(0.0F, 0.0F, 0.0F, 0.0F);
        }
        float magnitude = 0.0F;
#pragma unroll
        for (std::uint32_t i = 0; i < kSlabK / 128; ++i) {
            magnitude = largerMagnitude(largerMagnitude(magnitude, v[i].x), v[i].y);
            magnitude = largerMagnitude(largerMagnitude(magnitude, v[i].z), v[i].w);
        }
        const std::uint32_t most = warpMax(magnitude);
        std::uint32_t of_group   = most;
        if (o.grouped != 0) {
            if (lane == 0) { large_of[warp] = most; }
            __syncthreads();
            of_group = __reduce_max_sync(0xFFFFFFFFU, large_of[lane % kWarps]);
        }
        const RowScale scaling = rowScale(of_group);
        if (!scaling.covered) { state = kOutOfRange; }
        if (row < o.rows) {
            unsigned char* target = o.split + row * pitch + begin / kBlockK * kBlockBytes + lane / 16 * kBlockBytes + lane % 16 * 8;
            PairSplitter splitter(scaling.scale);
#pragma unroll
            for (std::uint32_t i = 0; i < kSlabK / 128; ++i) {
                uint2 hi, lo;
                splitter.split(v[i].x, v[i].y, hi.x, lo.x);
                splitter.split(v[i].z, v[i].w, hi.y, lo.y);
                if (begin + i * 128 + lane * 4 < k_end) {
                    *reinterpret_cast<uint2*>(target + i * 2 * kBlockBytes)               = hi;
                    *reinterpret_cast<uint2*>(target + i * 2 * kBlockBytes + 2 * kBlockK) = lo;
                }
            }
            if (__any_sync(0xFFFFFFFFU, splitter.sawGray())) {
                std::uint32_t gray = 0;
#pragma unroll
                for (std::uint32_t i = 0; i < kSlabK / 128; ++i) {
                    gray += grayElement(v[i].x, scaling.scale) + grayElement(v[i].y, scaling.scale) +
                            grayElement(v[i].z, scaling.scale) + grayElement(v[i].w, scaling.scale);
                }
                gray  = __reduce_add_sync(0xFFFFFFFFU, gray);
                state = max(state, gray > kFewGrayElements ? kManyGray : kFewGray);
            }
            const std::uint32_t large = __reduce_add_sync(0xFFFFFFFFU, splitter.largeElements());
            if (most != 0) { worstCounts(worst, large, length); }
            if (lane == 0) { o.inverse[slab * o.pitch + (o.grouped != 0 ? row / kColumnGroup : row)] = scaling.inverse; }
        }
    } else {
        // The slab is turned in shared memory: read along the rows, written along K.
        if (threadIdx.x < kSplitRows) { large_of[threadIdx.x] = gray_of[threadIdx.x] = 0; }
        if (o.vector != 0) {
            // 16-byte loads: a warp takes 4 K values of all 32 rows.
            const std::uint32_t at_row = lane % 8 * 4;
            const std::uint32_t row    = row0 + at_row;
            const bool whole           = row + 4 <= o.rows;
            float most[4]              = {0.0F, 0.0F, 0.0F, 0.0F};
#pragma unroll
            for (int batch = 0; batch < 2; ++batch) {
                float4 v[6];
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                    const std::uint32_t k = begin + (batch * 6 + i) * 64 + warp * 4 + lane / 8;
                    const float* source   = o.source + static_cast<std::int64_t>(k) * o.k_stride + row;
                    v[i]                  = make_float4(0.0F, 0.0F, 0.0F, 0.0F);
                    if (k < depth) {
                        if (whole) {
                            v[i] = *reinterpret_cast<const float4*>(source);
                        } else {
                            if (row < o.rows) { v[i].x = source[0]; }
                            if (row + 1 < o.rows) { v[i].y = source[1]; }
                            if (row + 2 < o.rows) { v[i].z = source[2]; }
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                    float* to = tile + ((batch * 6 + i) * 64 + warp * 4 + lane / 8) * kTilePitch + at_row;
                    to[0] = v[i].x, to[1] = v[i].y, to[2] = v[i].z, to[3] = v[i].w;
                    most[0] = largerMagnitude(most[0], v[i].x);
                    most[1] = largerMagnitude(most[1], v[i].y);
                    most[2] = largerMagnitude(most[2], v[i].z);
                    most[3] = largerMagnitude(most[3], v[i].w);
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                std::uint32_t bits = __float_as_uint(most[j]);
                bits = max(bits, __shfl_xor_sync(0xFFFFFFFFU, bits, 8));
                bits = max(bits, __shfl_xor_sync(0xFFFFFFFFU, bits, 16));
                if (lane < 8) { most_of[warp][at_row + j] = bits; }
            }
        } else {
            const std::uint32_t row = row0 + lane;
            float most              = 0.0F;
#pragma unroll 1
            for (int batch = 0; batch < 3; ++batch) {
                float v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const std::uint32_t k = begin + (batch * 16 + i) * 16 + warp;
                    v[i] = k < depth && row < o.rows
                               ? o.source[static_cast<std::int64_t>(k) * o.k_stride + static_cast<std::int64_t>(row) * o.row_stride]
                               : 0.0F;
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    tile[((batch * 16 + i) * 16 + warp) * kTilePitch + lane] = v[i];
                    most = largerMagnitude(most, v[i]);
                }
            }
            most_of[warp][lane] = __float_as_uint(most);
        }
        __syncthreads();
        std::uint32_t most = 0;
        if (threadIdx.x < kSplitRows) {
#pragma unroll
            for (int w = 0; w < kWarps; ++w) { most = max(most, most_of[w][threadIdx.x]); }
            std::uint32_t of_group = most;
            if (o.grouped != 0) {
                of_group = max(of_group, __shfl_xor_sync(0xFFFFFFFFU, of_group, 1));
                of_group = max(of_group, __shfl_xor_sync(0xFFFFFFFFU, of_group, 2));
                of_group = max(of_group, __shfl_xor_sync(0xFFFFFFFFU, of_group, 4));
                of_group = max(of_group, __shfl_xor_sync(0xFFFFFFFFU, of_group, 8));
            }
            const RowScale scaling  = rowScale(of_group);
            const std::uint32_t row = row0 + threadIdx.x;
            if (!scaling.covered) { state = kOutOfRange; }
            scale_of[threadIdx.x]   = scaling.scale;
            if (row < o.rows) { o.inverse[slab * o.pitch + (o.grouped != 0 ? row / kColumnGroup : row)] = scaling.inverse; }
        }
        __syncthreads();
        // A warp takes four rows, half of the K blocks; a thread 8 K values of each block.
        constexpr std::uint32_t kGroups = kSplitRows / 4;
        const std::uint32_t at_row      = warp % kGroups * 4 + lane / 8;
        const std::uint32_t first       = warp / kGroups * (kSlabBlocks / 2);
        const bool inside               = row0 + at_row < o.rows;
        unsigned char* at = o.split + (row0 + at_row) * pitch + (begin / kBlockK + first) * kBlockBytes + lane % 8 * 16;
        const float* from = tile + (first * kBlockK + lane % 8 * 8) * kTilePitch + at_row;
        PairSplitter splitter(scale_of[at_row]);
#pragma unroll 2
        for (std::uint32_t i = 0; i < kSlabBlocks / 2; ++i, at += kBlockBytes, from += kBlockK * kTilePitch) {
            if (begin + (first + i) * kBlockK >= k_end) { break; }
            uint4 hi, lo;
            splitter.split(from[0], from[kTilePitch], hi.x, lo.x);
            splitter.split(from[2 * kTilePitch], from[3 * kTilePitch], hi.y, lo.y);
            splitter.split(from[4 * kTilePitch], from[5 * kTilePitch], hi.z, lo.z);
            splitter.split(from[6 * kTilePitch], from[7 * kTilePitch], hi.w, lo.w);
            if (inside) {
                *reinterpret_cast<uint4*>(at)               = hi;
                *reinterpret_cast<uint4*>(at + 2 * kBlockK) = lo;
            }
        }
        if (splitter.sawGray()) {
            std::uint32_t gray = 0;
            from               = tile + (first * kBlockK + lane % 8 * 8) * kTilePitch + at_row;
#pragma unroll 1
            for (std::uint32_t i = 0; i < kSlabBlocks / 2; ++i, from += kBlockK * kTilePitch) {
                for (int j = 0; j < 8; ++j) { gray += grayElement(from[j * kTilePitch], scale_of[at_row]); }
            }
            atomicAdd(&gray_of[at_row], gray);
        }
        std::uint32_t large = splitter.largeElements();
        large += __shfl_xor_sync(0xFFFFFFFFU, large, 1);
        large += __shfl_xor_sync(0xFFFFFFFFU, large, 2);
        large += __shfl_xor_sync(0xFFFFFFFFU, large, 4);
        if (lane % 8 == 0) { atomicAdd(&large_of[at_row], large); }
        __syncthreads();
        if (threadIdx.x < kSplitRows && most != 0) {
            worstCounts(worst, large_of[threadIdx.x], length);
            const std::uint32_t gray = gray_of[threadIdx.x];
            if (gray != 0) { state = max(state, gray > kFewGrayElements ? kManyGray : kFewGray); }
        }
    }
    state = __reduce_max_sync(0xFFFFFFFFU, state);
#pragma unroll
    for (int t = 0; t < 3; ++t) { worst[t] = __reduce_max_sync(0xFFFFFFFFU, worst[t]); }
    if (lane == 0) {
#pragma unroll
        for (int t = 0; t < 3; ++t) { worst_of[warp][t] = worst[t]; }
        state_of[warp] = state;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        std::uint32_t small[3] = {0, 0, 0}, worst_state = kAllCovered;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            worst_state = max(worst_state, state_of[w]);
#pragma unroll
            for (int t = 0; t < 3; ++t) { small[t] = max(small[t], worst_of[w][t]); }
        }
        o.verdicts[slab * row_blocks + row_block] = worst_state << kVerdictState | small[0] | small[1] << 10 | small[2] << 20;
    }
}

}  // namespace

void planSplit(SplitOperand& o, std::uint32_t slabs) {
    const auto size = [](std::int64_t stride) { return stride < 0 ? -stride : stride; };
    o.along_k       = size(o.k_stride) <= size(o.row_stride) ? 1U : 0U;
    const std::int64_t fast = o.along_k != 0 ? o.k_stride : o.row_stride, slow = o.along_k != 0 ? o.row_stride : o.k_stride;
    o.vector = fast == 1 && slow % 4 == 0 && reinterpret_cast<std::uintptr_t>(o.source) % 16 == 0 ? 1U : 0U;
    o.blocks = static_cast<std::uint32_t>(ceilDiv(o.rows, o.along_k != 0 ? kSplitRowsAlongK : kSplitRows) * slabs);
}

cudaError_t configureSplit() {
    return cudaFuncSetAttribute(splitOperands, cudaFuncAttributeMaxDynamicSharedMemorySize, kTileBytes);
}

cudaError_t launchSplit(const SplitParams& p, cudaStream_t stream) {
    cudaLaunchConfig_t config{};
    config.gridDim          = dim3(p.operand[0].blocks + p.operand[1].blocks, 1, 1);
    config.blockDim         = dim3(kThreads, 1, 1);
    config.dynamicSmemBytes = p.operand[0].along_k != 0 && p.operand[1].along_k != 0 ? 0 : kTileBytes;
    config.stream           = stream;
    cudaLaunchAttribute attribute{};
    attribute.id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute.val.programmaticStreamSerializationAllowed = 1;
    config.attrs                                         = &attribute;
    config.numAttrs                                      = 1;
    countLaunches(1);
    return cudaLaunchKernelEx(&config, splitOperands, p);
}

}  // namespace fp16x3
}  // namespace ftcuda
