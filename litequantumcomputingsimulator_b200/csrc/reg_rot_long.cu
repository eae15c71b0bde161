// reg_rot_long.cu — register tile passes in rotation form with more than kRotShort records.
#include "reg_rot.cuh"

namespace lqcs_b200 {

void launch_rot_long(const LaunchCtx& ctx, double2* st, uint32_t batch, const RegPass& p, size_t smem,
                     const RegOp* ops, const RegLayout* d_layouts, const double2* d_mats) {
    launch_rot_records<kRegMaxRecords>(ctx, st, batch, p, smem, ops, d_layouts, d_mats);
}

}  // namespace lqcs_b200
