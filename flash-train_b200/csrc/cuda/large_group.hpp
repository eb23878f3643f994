// Which groups of a grouped GEMM take the prepared form. Pure arithmetic, shared by the host pipeline (which asks the
// platform for that form only where a group has use for it) and the platform.
#ifndef FTCUDA_LARGE_GROUP_HPP_
#define FTCUDA_LARGE_GROUP_HPP_

#include "ftcuda/ftcuda.h"

namespace ftcuda {

// Whether a group runs faster by itself in the prepared form than inside the one TF32 launch over all groups,
// which works at about 190 TFLOP/s whatever the groups are. Measured alone: 2048 x 1024 x 2048 226 TFLOP/s,
// 4096 x 1024 x 1024 204, 2048 x 4096 x 1024 212, 1024 x 4096 x 4096 262; but 1024 x 2048 x 1024 110, 512 x 4096 x 4096 179.
inline bool largeGroup(const FtcudaGemmDesc& desc) {
    if (desc.m * desc.n == 0 || desc.k < 512) { return false; }
    const double m = static_cast<double>(desc.m), n = static_cast<double>(desc.n);
    return m * n >= 600.0 * (m + n) && m * n * static_cast<double>(desc.k) >= 4e9;
}

}  // namespace ftcuda

#endif
