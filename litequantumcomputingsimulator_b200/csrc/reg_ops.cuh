// reg_ops.cuh — operations on a tile held in registers, shared by the register pass kernels
// (reg_tile_kernels.cu, reg_rot_kernels.cu): 16 amplitudes per thread, the register index u
// holding the tile bits a RegLayout assigns to it.
#pragma once

#include "tile.cuh"

namespace lqcs_b200 {
namespace {

constexpr int kE = 1 << kRegBits;   // amplitudes per thread
constexpr uint32_t kRegSlotLayouts = 16;   // layouts whose per-thread slots are tabulated

__host__ __device__ constexpr int popc4(int m) {
    return (m & 1) + ((m >> 1) & 1) + ((m >> 2) & 1) + ((m >> 3) & 1);
}

// Member l of a group: the bits of l spread over the set bits of mask, lowest first.
__host__ __device__ constexpr int deposit4(int l, int mask) {
    int out = 0, j = 0;
    for (int b = 0; b < kRegBits; ++b) {
        if ((mask >> b) & 1) {
            if ((l >> j) & 1) out |= 1 << b;
            ++j;
        }
    }
    return out;
}

// Shared-memory load the compiler may not hoist or merge: matrix entries are re-read per
// group so they never occupy registers alongside the 16 amplitudes.
__device__ __forceinline__ double2 lds2(uint32_t saddr) {
    double2 r;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(r.x), "=d"(r.y) : "r"(saddr));
    return r;
}

// Matrix entries of an operation, entry i at 16 * i bytes of shared memory (the helpers
// below take any functor of this shape).
struct SharedMat {
    uint32_t base;   // shared-memory address
    __device__ __forceinline__ double2 operator()(uint32_t i) const { return lds2(base + 16u * i); }
};

// Group base of the g-th group of a target mask: g spread over the bits outside TM.
__host__ __device__ constexpr int group_base(int g, int tm) { return deposit4(g, (kE - 1) & ~tm); }

// Dense operation without register controls: one basic block, so the compiler interleaves
// the groups.  Two-target operations take two groups per matrix read (each entry is loaded
// twice per operation instead of four times).
template <int TM, class MS>
__device__ __forceinline__ void reg_dense_free(double2 (&v)[kE], const MS& mat) {
    constexpr int K = popc4(TM);
    constexpr int D = 1 << K;
    constexpr int G = kE / D;   // groups
    if constexpr (K == 1) {
        const double2 m0 = mat(0), m1 = mat(1), m2 = mat(2), m3 = mat(3);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int b = group_base(g, TM);
            const double2 a0 = v[b], a1 = v[b | TM];
            v[b] = cmad(m1, a1, cmul(m0, a0));
            v[b | TM] = cmad(m3, a1, cmul(m2, a0));
        }
    } else if constexpr (K == 2) {
#pragma unroll
        for (int g = 0; g < G; g += 2) {
            const int b0 = group_base(g, TM), b1 = group_base(g + 1, TM);
            double2 y0[D], y1[D];
#pragma unroll
            for (int r = 0; r < D; ++r) {
                const double2 mr = mat(r * D);
                y0[r] = cmul(mr, v[b0]);
                y1[r] = cmul(mr, v[b1]);
            }
#pragma unroll
            for (int c = 1; c < D; ++c) {
#pragma unroll
                for (int r = 0; r < D; ++r) {
                    const double2 mr = mat(r * D + c);
                    y0[r] = cmad(mr, v[b0 | deposit4(c, TM)], y0[r]);
                    y1[r] = cmad(mr, v[b1 | deposit4(c, TM)], y1[r]);
                }
            }
#pragma unroll
            for (int r = 0; r < D; ++r) {
                v[b0 | deposit4(r, TM)] = y0[r];
                v[b1 | deposit4(r, TM)] = y1[r];
            }
        }
    } else {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int b = group_base(g, TM);
            double2 y[D];
#pragma unroll
            for (int r = 0; r < D; ++r) {
                double2 acc = cmul(mat(r * D), v[b]);
#pragma unroll
                for (int c = 1; c < D; ++c)
                    acc = cmad(mat(r * D + c), v[b | deposit4(c, TM)], acc);
                y[r] = acc;
            }
#pragma unroll
            for (int r = 0; r < D; ++r) v[b | deposit4(r, TM)] = y[r];
        }
    }
}

// Dense operation with register controls: groups whose control bits are not all 1 skip.
template <int TM, class MS>
__device__ __forceinline__ void reg_dense(double2 (&v)[kE], const MS& mat, uint32_t rcmask) {
    constexpr int K = popc4(TM);
    constexpr int D = 1 << K;
    if constexpr (K == 1) {
        const double2 m0 = mat(0), m1 = mat(1), m2 = mat(2), m3 = mat(3);
#pragma unroll
        for (int b = 0; b < kE; ++b) {
            if (b & TM) continue;
            if ((b & rcmask) != rcmask) continue;
            const double2 a0 = v[b], a1 = v[b | TM];
            v[b] = cmad(m1, a1, cmul(m0, a0));
            v[b | TM] = cmad(m3, a1, cmul(m2, a0));
        }
    } else {
#pragma unroll
        for (int b = 0; b < kE; ++b) {
            if (b & TM) continue;
            if ((b & rcmask) != rcmask) continue;
            double2 y[D];
#pragma unroll
            for (int r = 0; r < D; ++r) {
                double2 acc = cmul(mat(r * D), v[b | deposit4(0, TM)]);
#pragma unroll
                for (int c = 1; c < D; ++c)
                    acc = cmad(mat(r * D + c), v[b | deposit4(c, TM)], acc);
                y[r] = acc;
            }
#pragma unroll
            for (int r = 0; r < D; ++r) v[b | deposit4(r, TM)] = y[r];
        }
    }
}

template <int I>
__device__ __forceinline__ void reg_swapx(double2 (&v)[kE], uint32_t rcmask) {
#pragma unroll
    for (int b = 0; b < kE; ++b) {
        if ((b >> I) & 1) continue;
        if ((b & rcmask) != rcmask) continue;
        const double2 a = v[b];
        v[b] = v[b | (1 << I)];
        v[b | (1 << I)] = a;
    }
}

template <class MS>
__device__ __forceinline__ void dispatch_dense(double2 (&v)[kE], uint32_t code, const MS& mat,
                                               uint32_t rcmask) {
    if (rcmask == 0) {
        switch (code) {
            case 1: reg_dense_free<1>(v, mat); break;
            case 2: reg_dense_free<2>(v, mat); break;
            case 3: reg_dense_free<3>(v, mat); break;
            case 4: reg_dense_free<4>(v, mat); break;
            case 5: reg_dense_free<5>(v, mat); break;
            case 6: reg_dense_free<6>(v, mat); break;
            case 7: reg_dense_free<7>(v, mat); break;
            case 8: reg_dense_free<8>(v, mat); break;
            case 9: reg_dense_free<9>(v, mat); break;
            case 10: reg_dense_free<10>(v, mat); break;
            case 11: reg_dense_free<11>(v, mat); break;
            case 12: reg_dense_free<12>(v, mat); break;
            case 13: reg_dense_free<13>(v, mat); break;
            case 14: reg_dense_free<14>(v, mat); break;
            default: break;
        }
        return;
    }
    switch (code) {
        case 1: reg_dense<1>(v, mat, rcmask); break;
        case 2: reg_dense<2>(v, mat, rcmask); break;
        case 3: reg_dense<3>(v, mat, rcmask); break;
        case 4: reg_dense<4>(v, mat, rcmask); break;
        case 5: reg_dense<5>(v, mat, rcmask); break;
        case 6: reg_dense<6>(v, mat, rcmask); break;
        case 7: reg_dense<7>(v, mat, rcmask); break;
        case 8: reg_dense<8>(v, mat, rcmask); break;
        case 9: reg_dense<9>(v, mat, rcmask); break;
        case 10: reg_dense<10>(v, mat, rcmask); break;
        case 11: reg_dense<11>(v, mat, rcmask); break;
        case 12: reg_dense<12>(v, mat, rcmask); break;
        case 13: reg_dense<13>(v, mat, rcmask); break;
        case 14: reg_dense<14>(v, mat, rcmask); break;
        default: break;   // 4-target operations never reach a register pass
    }
}

__device__ __forceinline__ void dispatch_swapx(double2 (&v)[kE], uint32_t code, uint32_t rcmask) {
    switch (code) {
        case 1: reg_swapx<0>(v, rcmask); break;
        case 2: reg_swapx<1>(v, rcmask); break;
        case 4: reg_swapx<2>(v, rcmask); break;
        default: reg_swapx<3>(v, rcmask); break;
    }
}

// Diagonal whose entry bits sit on register-index bits R (and on thread bits, fixed per
// thread in tpart): amplitude u takes entry tpart | e(u & R), so a thread loads each of its
// 2^|R| distinct entries once and multiplies the 16 / 2^|R| amplitudes that share it.
template <int R, class MS>
__device__ __forceinline__ void reg_diag_r(double2 (&v)[kE], const MS& mat, uint32_t rcmask,
                                           uint32_t tpart, uint32_t rb0, uint32_t rb1,
                                           uint32_t rb2, uint32_t rb3) {
#pragma unroll
    for (int pt = 0; pt < kE; ++pt) {
        if ((pt & R) != pt) continue;
        const uint32_t e = tpart | ((pt & 1) ? rb0 : 0u) | ((pt & 2) ? rb1 : 0u) |
                           ((pt & 4) ? rb2 : 0u) | ((pt & 8) ? rb3 : 0u);
        const double2 f = mat(e);
#pragma unroll
        for (int u = 0; u < kE; ++u)
            if ((u & R) == pt && (u & rcmask) == rcmask) v[u] = cmul(f, v[u]);
    }
}

// Entry (tpart | bits picked from u) of a diagonal for every amplitude u.
template <class MS>
__device__ __forceinline__ void reg_diag(double2 (&v)[kE], const RegOp& op, const MS& mat,
                                         uint32_t rcmask) {
    uint32_t tpart = 0, rb0 = 0, rb1 = 0, rb2 = 0, rb3 = 0;   // entry bit of register bit i
    const uint32_t k = op.k;
    for (uint32_t j = 0; j < k; ++j) {
        const uint32_t loc = op.loc[j], bit = 1u << j;
        if (loc & 0x80u) {
            tpart |= ((threadIdx.x >> (loc & 0x7fu)) & 1u) << j;
        } else {
            rb0 |= loc == 0 ? bit : 0u;
            rb1 |= loc == 1 ? bit : 0u;
            rb2 |= loc == 2 ? bit : 0u;
            rb3 |= loc == 3 ? bit : 0u;
        }
    }
    const uint32_t R = (rb0 ? 1u : 0u) | (rb1 ? 2u : 0u) | (rb2 ? 4u : 0u) | (rb3 ? 8u : 0u);
    switch (R) {
#define LQCS_DIAG_CASE(r) \
    case r: reg_diag_r<r>(v, mat, rcmask, tpart, rb0, rb1, rb2, rb3); break;
        LQCS_DIAG_CASE(0) LQCS_DIAG_CASE(1) LQCS_DIAG_CASE(2) LQCS_DIAG_CASE(3)
        LQCS_DIAG_CASE(4) LQCS_DIAG_CASE(5) LQCS_DIAG_CASE(6) LQCS_DIAG_CASE(7)
        LQCS_DIAG_CASE(8) LQCS_DIAG_CASE(9) LQCS_DIAG_CASE(10) LQCS_DIAG_CASE(11)
        LQCS_DIAG_CASE(12) LQCS_DIAG_CASE(13) LQCS_DIAG_CASE(14)
        default: reg_diag_r<15>(v, mat, rcmask, tpart, rb0, rb1, rb2, rb3); break;
#undef LQCS_DIAG_CASE
    }
}

// d += a * b on the FP64 tensor path, one m8n8k4 step: lane l holds a = A[l / 4][l % 4],
// b = B[l % 4][l / 4] and d = D[l / 4][2 (l % 4) + {0, 1}].
__device__ __forceinline__ void mma_f64(double& d0, double& d1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// Two-qubit block on the lane pair (kRegMma), every register index whose control bits are
// all 1.  For register u the warp's 32 amplitudes form A (8 groups on lanes 2..4 x 4 members
// on lanes 0..1), split into real and imaginary parts; the 4 x 4 complex matrix M enters as
// B with column n = 2 j + c holding output member j, part c: B_re[k][n] = c ? Im M[j][k] :
// Re M[j][k], B_im[k][n] = c ? Re M[j][k] : -Im M[j][k].  D = A_re B_re + A_im B_im then
// leaves (Re, Im) of the lane's own new amplitude in its two accumulators.  The whole warp
// runs it (the caller keeps it converged); lane l loads one matrix entry.
__device__ __forceinline__ void reg_mma(double2 (&v)[kE], uint32_t mat, uint32_t rcmask) {
    const uint32_t lane = threadIdx.x & 31u;
    const double2 e = lds2(mat + 16u * (((lane >> 3) << 2) | (lane & 3u)));
    const bool im_col = ((lane >> 2) & 1u) != 0;
    const double b_re = im_col ? e.y : e.x, b_im = im_col ? e.x : -e.y;
    if (rcmask == 0) {
#pragma unroll
        for (int u = 0; u < kE; ++u) {
            double d0 = 0.0, d1 = 0.0;
            mma_f64(d0, d1, v[u].x, b_re);
            mma_f64(d0, d1, v[u].y, b_im);
            v[u] = make_double2(d0, d1);
        }
        return;
    }
#pragma unroll
    for (int u = 0; u < kE; ++u) {
        if ((u & rcmask) != rcmask) continue;   // uniform over the warp
        double d0 = 0.0, d1 = 0.0;
        mma_f64(d0, d1, v[u].x, b_re);
        mma_f64(d0, d1, v[u].y, b_im);
        v[u] = make_double2(d0, d1);
    }
}

// Pauli rotation whose flip is the single register bit XR (kRegPauli after the reduction in
// reg_pauli): amplitude u becomes c a_u + y s_u a_(u ^ XR), s_u = (-1)^parity(u & zr), y
// already carrying the sign of the thread's and the tile's Z-type bits; the partner's sign
// is s_u times (-1)^parity(XR & zr).
template <int XR>
__device__ __forceinline__ void reg_pauli_x(double2 (&v)[kE], double c, double2 y, uint32_t zr) {
    const double sx = (zr & XR) ? -1.0 : 1.0;
#pragma unroll
    for (int u = 0; u < kE; ++u) {
        if (u & XR) continue;
        const double2 a = v[u], b = v[u ^ XR];
        const double su = (__popc(static_cast<uint32_t>(u) & zr) & 1u) ? -1.0 : 1.0;
        const double2 yu = cscale(y, su);
        v[u] = cmad(yu, b, cscale(a, c));
        v[u ^ XR] = cmad(cscale(yu, sx), a, cscale(b, c));
    }
}

// The same with flips on lanes too (lane mask xl): the partner of (u, lane) is (u ^ XR,
// lane ^ xl), fetched by shuffle; XR = 0: flips on lanes only.  Every lane of the warp runs it.
template <int XR>
__device__ __forceinline__ void reg_pauli_xl(double2 (&v)[kE], double c, double2 y, uint32_t zr,
                                             uint32_t xl) {
    const int m = static_cast<int>(xl);
    if constexpr (XR == 0) {
#pragma unroll
        for (int u = 0; u < kE; ++u) {
            const double2 b = shfl_xor_d2(v[u], m);
            const double su = (__popc(static_cast<uint32_t>(u) & zr) & 1u) ? -1.0 : 1.0;
            v[u] = cmad(cscale(y, su), b, cscale(v[u], c));
        }
    } else {
#pragma unroll
        for (int u = 0; u < kE; ++u) {
            if (u & XR) continue;
            const double2 pu = shfl_xor_d2(v[u ^ XR], m), pw = shfl_xor_d2(v[u], m);
            const double su = (__popc(static_cast<uint32_t>(u) & zr) & 1u) ? -1.0 : 1.0;
            const double sw = (__popc(static_cast<uint32_t>(u ^ XR) & zr) & 1u) ? -1.0 : 1.0;
            v[u] = cmad(cscale(y, su), pu, cscale(v[u], c));
            v[u ^ XR] = cmad(cscale(y, sw), pw, cscale(v[u ^ XR], c));
        }
    }
}

// kRegPauli record: matrices (cos, 0), y, out-of-tile Z-type mask (two exact halves).  A flip
// set of several register bits reduces to its lowest bit b: with the register permutation
// U = prod_j CX(b -> b_j) over the other flip bits, U P U has flip bits {b} and Z-type bits
// zr with b toggled once per b_j among them, so the kernel permutes, rotates on one bit and
// permutes back (4 + 4 code paths instead of one per flip set, which at 15 unrolled paths
// made the allocator spill over a kilobyte per thread).
__device__ __forceinline__ void reg_pauli(double2 (&v)[kE], uint32_t mat, uint32_t xr, uint32_t zr,
                                          uint32_t zt, uint32_t xl, uint64_t base) {
    const double c = lds2(mat).x;
    double2 y = lds2(mat + 16u);
    const double2 zd = lds2(mat + 32u);
    const uint64_t zg = static_cast<uint64_t>(zd.x) | (static_cast<uint64_t>(zd.y) << 32);
    if ((__popcll(base & zg) + __popc(threadIdx.x & zt)) & 1) y = make_double2(-y.x, -y.y);
    if (xl != 0 && xr == 0) {   // flips on lanes only
        reg_pauli_xl<0>(v, c, y, zr, xl);
        return;
    }
    if (xr == 0) {   // a Z-type string: the diagonal c + y s_u
        const double2 fp = make_double2(c + y.x, y.y), fm = make_double2(c - y.x, -y.y);
#pragma unroll
        for (int u = 0; u < kE; ++u)
            v[u] = cmul(v[u], (__popc(static_cast<uint32_t>(u) & zr) & 1u) ? fm : fp);
        return;
    }
    const uint32_t b = xr & (0u - xr), rest = xr & ~b;
    for (uint32_t r = rest; r; r &= r - 1) dispatch_swapx(v, r & (0u - r), b);
    const uint32_t zr1 = (__popc(zr & rest) & 1u) ? zr ^ b : zr;
    if (xl != 0) {
        switch (b) {
            case 1: reg_pauli_xl<1>(v, c, y, zr1, xl); break;
            case 2: reg_pauli_xl<2>(v, c, y, zr1, xl); break;
            case 4: reg_pauli_xl<4>(v, c, y, zr1, xl); break;
            default: reg_pauli_xl<8>(v, c, y, zr1, xl); break;
        }
    } else {
        switch (b) {
            case 1: reg_pauli_x<1>(v, c, y, zr1); break;
            case 2: reg_pauli_x<2>(v, c, y, zr1); break;
            case 4: reg_pauli_x<4>(v, c, y, zr1); break;
            default: reg_pauli_x<8>(v, c, y, zr1); break;
        }
    }
    for (uint32_t r = rest; r; r &= r - 1) dispatch_swapx(v, r & (0u - r), b);
}

__device__ __forceinline__ uint32_t thread_slot(const RegLayout& ly, uint32_t tbits) {
    uint32_t s = 0;
    for (uint32_t i = 0; i < tbits; ++i)
        if ((threadIdx.x >> i) & 1u) s ^= ly.tsw[i];
    return s;
}

__device__ __forceinline__ uint64_t thread_goff(const RegLayout& ly, uint32_t tbits,
                                                const uint64_t* gbit) {
    uint64_t g = 0;
    for (uint32_t i = 0; i < tbits; ++i)
        if ((threadIdx.x >> i) & 1u) g |= gbit[ly.tpos[i]];
    return g;
}

}  // namespace
}  // namespace lqcs_b200
