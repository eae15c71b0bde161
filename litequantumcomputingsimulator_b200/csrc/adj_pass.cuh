// adj_pass.cuh — register passes of Pauli rotations for the batched adjoint (adj_kernels.cu) and
// their planning (adj_plan.cpp).
//
// A Pauli rotation pairs index i with i ^ x, so a set of rotations can run on a tile whenever
// the tile is closed under XOR with their x masks: a coset of a linear subspace V of the index
// bits (over GF(2)) that contains them.  A tile of 2^m amplitudes then holds m - 3 rotations
// with any independent x (the other three dimensions are qubits 0..2, which keep global rows of
// 128 bytes), where a tile of m - 3 whole qubits holds those whose X and Y qubits all lie among
// them.  In a layout the x masks of up to kRegs rotations are the basis vectors of the register
// index, so each of these rotations pairs register u with u ^ 2^r in the same thread; a remap
// through shared memory moves the tile to the next layout.
#pragma once

#include <cstdint>
#include <vector>

#include "kernels.cuh"

namespace lqcs_b200 {

constexpr uint32_t kAdjMinBits = 9, kAdjMaxBits = 12;   // tile sizes
constexpr uint32_t kAdjMaxRots = 96, kAdjMaxLayouts = 64;
constexpr uint32_t kAdjFwdRegs = 4, kAdjBwdRegs = 3;    // register-index bits: 16, 2 x 8 amplitudes
constexpr uint32_t kAdjDiag = 4;                        // AdjRot::rbit of a rotation with x = 0

struct AdjRot {
    uint64_t zy;      // Z / Y qubits: their parity with the tile's base gives the tile's sign
    uint32_t param;   // row of the (cos, sin) table
    uint16_t tz;      // thread-index bits whose basis vector has odd parity with zy
    uint8_t rz;       // register-index bits
    uint8_t rbit;     // the register-index bit whose basis vector is x, or kAdjDiag
    uint8_t n_y;      // power of i of the string
    uint8_t layout;
    uint8_t pad[2];
};
struct AdjLayout {    // shared-memory slots of the basis vectors
    uint16_t t[10], r[kAdjFwdRegs];
};
struct AdjPass {
    uint32_t m, n_rots, n_layouts, regs;
    uint32_t pivots[kAdjMaxBits];   // ascending: a tile's base has zeros there
    uint64_t tvec[2][10], rvec[2][kAdjFwdRegs];   // basis vectors at the load and at the store
    AdjLayout lay[kAdjMaxLayouts];
    AdjRot rot[kAdjMaxRots];
};

// A rotation as the planner sees it: the string i^n_y X^x Z^zy (x: X / Y qubits, zy: Z / Y).
struct AdjRotation {
    uint64_t x = 0, zy = 0;
    uint32_t n_y = 0, param = 0;
};

// Passes over rotations in the order given (a rotation may move ahead of others it commutes
// with; of all with any_order), on an n-qubit register, m = min(n, `bits`) >= kAdjMinBits.
std::vector<AdjPass> plan_adjoint_passes(const std::vector<AdjRotation>& rots, uint32_t n,
                                         uint32_t bits, uint32_t regs, bool any_order = false,
                                         uint32_t most = kAdjMaxRots);

// Pauli expectations <psi|P|psi> of terms i^n_y X^x Z^zy on the same tiles: a pass reads the state
// once for every term whose x lies in its tiles' subspace.  param: the term's place in d_out.
constexpr uint32_t kExpectTileBits = 11, kExpectTerms = 20;   // per pass
constexpr uint32_t kExpectThreads = 1u << (kExpectTileBits - 4), kExpectCtas = 512 / kExpectThreads;
constexpr uint32_t kExpectSmall = 14;                         // to here: a block per term
uint32_t expect_blocks(const LaunchCtx& ctx, uint32_t n);      // partials per term, n > kExpectSmall
void launch_expect_pass(const LaunchCtx& ctx, const double2* st, uint32_t n, const AdjPass& p,
                        double* d_partials);
void launch_expect_sum(const LaunchCtx& ctx, uint32_t n, uint32_t n_terms, const double* d_partials,
                       double* d_out);
void launch_expect_small(const LaunchCtx& ctx, const double2* st, uint32_t n,
                         const AdjRotation* d_terms, uint32_t n_terms, double* d_out);

void launch_adj_fwd(const LaunchCtx& ctx, double2* st, uint32_t n, uint32_t nb, const AdjPass& p,
                    const double2* d_cs, uint32_t R);
// Undoes the pass's rotations on psi and lambda; before each, d_grad[state * np + param] =
// Im<lambda|P|psi>.  d_partials: n_rots * nb * 2^(n - m) doubles.
void launch_adj_bwd(const LaunchCtx& ctx, double2* psi, double2* lam, uint32_t n, uint32_t nb,
                    const AdjPass& p, const double2* d_cs, uint32_t R, double* d_partials,
                    double* d_grad, uint64_t np);

}  // namespace lqcs_b200
