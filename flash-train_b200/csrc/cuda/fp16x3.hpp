// The prepared form of the 3xTF32 families: operands split once per launch into FP16 pairs
// (gemm_fp16x3_split.cu), multiplied by CTA pairs on the tensor cores (gemm_fp16x3.cu).
#ifndef FTCUDA_FP16X3_HPP_
#define FTCUDA_FP16X3_HPP_

#include <cuda_runtime_api.h>

#include <cstdint>

namespace ftcuda {
namespace fp16x3 {

constexpr std::uint32_t kBlockK = 64;  // K elements of one block: 128 bytes of FP16, one swizzle row

// A split operand in the workspace: [rows][K blocks][high 64 | low 64] FP16, K-major whatever the
// source's orientation, the last K block filled up with zeros.
constexpr std::uint64_t kBlockBytes = 2 * kBlockK * 2;

// Words at the head of the workspace, cleared in front of every launch.
struct Control {
    std::uint32_t use_fallback;  // the decision: 1 = this launch's operands go through the TF32 kernel
    std::uint32_t out_of_range;  // a row or column whose largest magnitude the scaling does not cover
    std::uint32_t gray;          // an element far below its row's (column's) largest was seen
    std::uint32_t blocks_done;
};

struct SplitOperand {
    const float* source;
    std::int64_t row_stride;  // between rows of A, or between columns of B
    std::int64_t k_stride;
    std::uint32_t rows;       // rows of A, or columns of B
    std::uint32_t along_k;    // the source runs faster along K than along its rows
    std::uint32_t vector;     // 16-byte loads along K are aligned
    std::uint32_t max_blocks, split_blocks;  // CTAs of the two kernels that work on this operand
    unsigned char* split;
    std::uint32_t* row_max;   // bit pattern of the largest magnitude of each row
    std::uint32_t* few;       // elements of each row that are small against its largest
    float* inverse;           // 1 / (scale of each row), a power of two
};

struct SplitParams {
    SplitOperand operand[2];
    std::uint32_t k, k_blocks;
    Control* control;
};

// CTAs of the two kernels for one operand.
void planSplit(SplitOperand& operand, std::uint32_t k);
cudaError_t launchSplit(const SplitParams& params, cudaStream_t stream);

}  // namespace fp16x3
}  // namespace ftcuda

#endif
