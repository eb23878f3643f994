// Which groups of a grouped GEMM take the prepared form, and when. Pure arithmetic, shared by the host pipeline (which asks the
// platform for that form only where it pays) and the platform.
#ifndef FTCUDA_LARGE_GROUP_HPP_
#define FTCUDA_LARGE_GROUP_HPP_

#include <cstdint>

#include "fp16x3_geometry.hpp"
#include "ftcuda/ftcuda.h"

namespace ftcuda {

// Whether a group, taken alone, is of a size for the prepared form. (Measured alone, against about 190 TFLOP/s of the one TF32
// launch over many groups: 2048 x 1024 x 2048 226 TFLOP/s, 4096 x 1024 x 1024 204, 2048 x 4096 x 1024 212,
// 1024 x 4096 x 4096 262; but 1024 x 2048 x 1024 110, 512 x 4096 x 4096 179.)
inline bool largeGroup(const FtcudaGemmDesc& desc) {
    if (desc.m * desc.n == 0 || desc.k < 512) { return false; }
    const double m = static_cast<double>(desc.m), n = static_cast<double>(desc.n);
    return m * n >= 600.0 * (m + n) && m * n * static_cast<double>(desc.k) >= 4e9;
}

// Microseconds of the one TF32 launch over groups: whole waves of tiles of 128 x 192, each 15 and 0.81 for every K block of 32.
// Within 12 % of what was measured on 80 mixes of 1 to 16 groups, K from 512 to 4096.
struct OneLaunchEstimate {
    double tiles = 0.0, work = 0.0, longest = 0.0;
    void add(const FtcudaGemmDesc& desc) {
        const double count = static_cast<double>(fp16x3::divideUp(desc.m, 128) * fp16x3::divideUp(desc.n, 192));
        const double each  = 15.0 + 0.81 * static_cast<double>(fp16x3::divideUp(desc.k, 32));
        tiles += count;
        work += count * each;
        longest = each > longest ? each : longest;
    }
    double microseconds(std::uint32_t sms) const {
        if (tiles == 0.0) { return 0.0; }
        const double waves = static_cast<double>(fp16x3::divideUp(static_cast<std::uint64_t>(tiles), sms)) * work / tiles;
        return 7.0 + (waves > longest ? waves : longest);
    }
};

// ... and of one group's launches in the prepared form, behind those of others. 8 % off in the mean (root mean square) over the same mixes.
inline double preparedEstimate(const FtcudaGemmDesc& desc, std::uint32_t sms) {
    const std::uint64_t pairs  = sms / 2 != 0 ? sms / 2 : 1;
    const fp16x3::Geometry g   = fp16x3::chooseGeometry(desc.m, desc.n, fp16x3::divideUp(desc.k, fp16x3::kBlockK), pairs);
    const std::uint64_t items  = fp16x3::divideUp(desc.m, fp16x3::kTileM) * fp16x3::divideUp(desc.n, g.tile_n) * g.splits;
    const double waves         = static_cast<double>(fp16x3::divideUp(items, pairs));
    const double operand_bytes = 4.0 * static_cast<double>(desc.m + desc.n) * static_cast<double>(desc.k);  // read, and as many written
    return 9.3 + waves * (9.1 + 0.75e-3 * g.blocks_per_split * fp16x3::blockCycles(g.tile_n)) + 0.444e-6 * operand_bytes;
}

// Whether the large groups one after another in the prepared form, and the others in one TF32 launch, are faster than all of
// them in that launch. What decides is how the tiles fill whole waves, of each large group and of the one launch, and whether
// the others need a launch of their own. Measured (us, prepared / one launch): 4 x (1500 x 2048 x 2048) 238 / 290,
// 8 x (2048 x 1024 x 2048) 362 / 386, 7 of 372 to 1861 x 4096 x 4096 1228 / 1436, but 4 x (1200 x 2816 x 1200) 228 / 170,
// 8 x (1100 x 4096 x 1536) 669 / 496, 1500 and 130 x 2048 x 1536 115 / 72. The choice costs at most 10 % on 72 mixes, 6 % but for one.
inline bool preparedGroupsPay(const FtcudaGemmDesc* groups, std::uint32_t count, std::uint32_t sms) {
    OneLaunchEstimate all, others;
    double prepared = 0.0;
    bool any        = false;
    for (std::uint32_t g = 0; g < count; ++g) {
        if (groups[g].m * groups[g].n == 0) { continue; }
        all.add(groups[g]);
        if (largeGroup(groups[g])) {
            prepared += preparedEstimate(groups[g], sms);
            any = true;
        } else {
            others.add(groups[g]);
        }
    }
    return any && prepared + others.microseconds(sms) < all.microseconds(sms);
}

}  // namespace ftcuda

#endif
