// The prepared form of the 3xTF32 families: operands split once per launch into FP16 pairs
// (gemm_fp16x3_split.cu), multiplied by CTA pairs on the tensor cores (gemm_fp16x3.cu).
#ifndef FTCUDA_FP16X3_HPP_
#define FTCUDA_FP16X3_HPP_

#include <cuda_runtime_api.h>

#include <cstdint>

#include "fp16x3_geometry.hpp"

namespace ftcuda {
namespace fp16x3 {

constexpr std::uint32_t kSlabBlocks = 12;   // K blocks with scales of their own
constexpr std::uint32_t kSlabK      = kSlabBlocks * kBlockK;

// A split operand in the workspace: [rows][K blocks][high 64 | low 64] FP16, K-major whatever the
// source's orientation, the last K block filled up with zeros.
constexpr std::uint64_t kBlockBytes = 2 * kBlockK * 2;

// Rows of the operand that one CTA of the split takes, for one slab of K: source along K, or along the rows.
constexpr std::uint32_t kSplitRowsAlongK = 16;
constexpr std::uint32_t kSplitRows       = 32;

constexpr std::uint32_t kColumnGroup = 16;  // columns of B that share a scale

// What one CTA of the split found, a word for each slab and group of rows: how many nonzero rows' elements are below 2^-5, 2^-9
// and 2^-13 of the largest the row's scale allows for (the worst row; ten bits each), and what else there is to mind.
constexpr std::uint32_t kVerdictSmall = 0x3FF;
constexpr int kVerdictState           = 30;
enum VerdictState : std::uint32_t {
    kAllCovered  = 0,
    kFewGray     = 1,  // elements far below that, up to kFewGrayElements in a row
    kManyGray    = 2,
    kOutOfRange  = 3,  // a row whose magnitudes the scaling does not cover
};
constexpr std::uint32_t kFewGrayElements = 64;

struct SplitOperand {
    const float* source;
    std::int64_t row_stride;  // between rows of A, or between columns of B
    std::int64_t k_stride;
    std::uint32_t rows;       // rows of A, or columns of B
    std::uint32_t grouped;    // kColumnGroup rows share a scale, and `inverse` has one entry for each group
    std::uint32_t along_k;    // the source runs faster along K than along its rows
    std::uint32_t vector;     // 16-byte loads in that direction are aligned
    std::uint32_t blocks;     // CTAs
    unsigned char* split;
    float* inverse;           // [slab][pitch]: 1 / (scale of the row or group in the slab), a power of two
    std::uint64_t pitch;
    std::uint32_t* verdicts;  // [slab][blocks / slabs]
};

struct SplitParams {
    SplitOperand operand[2];
    std::uint32_t k, k_blocks, slabs;
};

// Fills along_k, vector and blocks from the source, its strides and the rows.
void planSplit(SplitOperand& operand, std::uint32_t slabs);
cudaError_t launchSplit(const SplitParams& params, cudaStream_t stream);
// To be called once per process and device before launches (shared-memory size of the kernel).
cudaError_t configureSplit();

}  // namespace fp16x3
}  // namespace ftcuda

#endif
