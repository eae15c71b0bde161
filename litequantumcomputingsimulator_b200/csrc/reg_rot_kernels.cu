// reg_rot_kernels.cu — launch of register tile passes in rotation form (reg_rot.cuh).
#include "reg_rot.cuh"

namespace lqcs_b200 {

// reg_rot_long.cu
void launch_rot_long(const LaunchCtx& ctx, double2* st, uint32_t batch, const RegPass& p, size_t smem,
                     const RegOp* ops, const RegLayout* d_layouts, const double2* d_mats);

// A launch copies its parameters, and the records are one: 8 KiB for the most a pass may have cost
// 0.5 to 0.8 us a launch more than 2 KiB for 64 (one layer of 16-qubit brickwork 37.7 against 36.1
// us), which all but the fullest passes keep to (20 to 40 records on 20 to 30 qubits, up to 140
// where a pass holds a whole 12-qubit circuit).
constexpr uint32_t kRotShort = 64;

void launch_rot_pass(const LaunchCtx& ctx, double2* st, uint32_t n, uint32_t batch,
                     const RegPass& pass, const RegOp* ops, const RegLayout* d_layouts,
                     const double2* d_mats) {
    RegPass p = pass;
    p.batch_stride = uint64_t{1} << n;
    p.n_tiles = (uint64_t{1} << n) >> p.m;
    if (!d_layouts || !d_mats) throw std::logic_error("register tile pass: a table is not on the device");
    const size_t smem = reg_smem_bytes(p);
    if (smem > kTileMaxSmem || p.m < kRegMinBits || p.m > kRegMaxBits || p.h > kTileMaxHigh ||
        p.n_layouts < 1 || p.n_ops > kRegMaxRecords || p.n_mat > kRegMaxMatrix ||
        p.n_dyn > kRegMaxDyn || p.dyn_entries > kRegMaxDynEntries)
        throw std::logic_error("register tile pass: unsupported shape");
    if (p.n_ops <= kRotShort) launch_rot_records<kRotShort>(ctx, st, batch, p, smem, ops, d_layouts, d_mats);
    else launch_rot_long(ctx, st, batch, p, smem, ops, d_layouts, d_mats);
}

}  // namespace lqcs_b200
