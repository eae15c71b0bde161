// adj_kernels.cu — register passes of Pauli rotations for the batched adjoint (adj_pass.cuh).
//
// One CTA applies a pass to one tile of one state: 16 amplitudes per thread forward, 8 of psi and
// 8 of lambda backward.  A rotation exp(-i theta/2 P) acts as the one-rotation kernel does
// (gate_kernels.cu; the reference's apply_pauli_rotation,
// src/backend/kernels/gate_kernels.cpp:191-225):
//     psi'[i] = cos psi[i] + (-i sin) i^{n_y} (-1)^{popcount((i ^ x) & zy)} psi[i ^ x],
// whose second factor is real or imaginary, so it costs four FP64 operations per amplitude, and
// the partner is another register of the same thread.
//
// What bounds it: HBM (32 bytes per amplitude and pass forward, 64 backward).  In shared memory,
// with one barrier and one read and write of the tile per rotation and tiles of whole qubits,
// the 16-qubit ansatz of 200 rotations took 36 + 46 passes at a third of that rate (256 sets: 7.9 ms
// forward, 16.0 backward; in registers, on tiles of 2^12 and 2^11, 3.1 and 8.2).  A CTA's load,
// rotations and store follow one another (by bytes and instructions each about a third), so the tiles
// are as small as the added passes allow (the sizes are chosen in adjoint.cpp).  The next tile
// prefetched to L2 changed nothing; in 128-byte bulk copies it cost 6 %.
#include <algorithm>
#include <stdexcept>
#include <string>

#include "adj_pass.cuh"
#include "common.cuh"
#include "kernels.cuh"

namespace lqcs_b200 {

namespace {

void check_launch(const char* what) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        throw std::runtime_error(std::string("CUDA launch failed in ") + what + ": " +
                                 cudaGetErrorString(e));
    }
    count_launch();
}

__device__ __forceinline__ double toggle(double x, uint32_t s) {   // bit 31 of s flips the sign
    return __hiloint2double(__double2hiint(x) ^ static_cast<int>(s), __double2loint(x));
}
__device__ __forceinline__ double2 toggle(double2 a, uint32_t s) {
    return make_double2(toggle(a.x, s), toggle(a.y, s));
}

// c a + Y b with Y = w (real) or i w.
template <bool IMAG>
__device__ __forceinline__ double2 mix(double c, double2 a, double w, double2 b) {
    if constexpr (IMAG) return make_double2(fma(-w, b.y, c * a.x), fma(w, b.x, c * a.y));
    else return make_double2(fma(w, b.x, c * a.x), fma(w, b.y, c * a.y));
}

// Sign words of the register indices: bit 31 of sign(u) = parity(u & rz) ^ t.
struct Signs {
    uint32_t t, e[4];
    __device__ __forceinline__ Signs(uint32_t thread, uint32_t rz) : t(thread << 31) {
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = (rz >> i) << 31;
    }
    __device__ __forceinline__ uint32_t operator()(int u) const {
        return t ^ ((u & 1) ? e[0] : 0u) ^ ((u & 2) ? e[1] : 0u) ^ ((u & 4) ? e[2] : 0u) ^
               ((u & 8) ? e[3] : 0u);
    }
};

template <int E, int RB, bool IMAG>
__device__ __forceinline__ void rotate(double2 (&v)[E], double c, double w, const Signs& sg) {
#pragma unroll
    for (int u = 0; u < E; ++u) {
        if ((u >> RB) & 1) continue;
        const int p = u | (1 << RB);
        const double2 a = toggle(v[u], sg(u)), b = toggle(v[p], sg(p));
        v[u] = mix<IMAG>(c, v[u], w, b);
        v[p] = mix<IMAG>(c, v[p], w, a);
    }
}

template <int E>
__device__ __forceinline__ void rotate_diag(double2 (&v)[E], double c, double w, const Signs& sg) {
#pragma unroll
    for (int u = 0; u < E; ++u) v[u] = mix<true>(c, v[u], w, toggle(v[u], sg(u)));
}

// (-i sin) i^{n_y} = i w (n_y even) or w (odd)
__device__ __forceinline__ double second_factor(double sin_h, uint32_t n_y) {
    return (n_y == 1u || n_y == 2u) ? sin_h : -sin_h;
}

template <int E>
__device__ __forceinline__ void dispatch_rotate(double2 (&v)[E], const AdjRot& r, double c, double w,
                                                const Signs& sg) {
    const bool imag = (r.n_y & 1u) == 0;
    switch (r.rbit) {
        case 0: if (imag) rotate<E, 0, true>(v, c, w, sg); else rotate<E, 0, false>(v, c, w, sg); break;
        case 1: if (imag) rotate<E, 1, true>(v, c, w, sg); else rotate<E, 1, false>(v, c, w, sg); break;
        case 2: if (imag) rotate<E, 2, true>(v, c, w, sg); else rotate<E, 2, false>(v, c, w, sg); break;
        case 3:
            if constexpr (E == 16) {
                if (imag) rotate<E, 3, true>(v, c, w, sg);
                else rotate<E, 3, false>(v, c, w, sg);
            }
            break;
        default: rotate_diag<E>(v, c, w, sg);
    }
}

// Re or Im of sum conj(lambda_i) (sign) psi_{i ^ x} over the thread's amplitudes.
template <int E, bool IMAG>
__device__ __forceinline__ double overlap(const double2 (&v)[E], const double2 (&l)[E], uint32_t flip,
                                          const Signs& sg) {
    double acc = 0.0;
#pragma unroll
    for (int u = 0; u < E; ++u) {
        const int p = u ^ static_cast<int>(flip);
        const double2 b = toggle(v[p], sg(p));
        acc = IMAG ? fma(l[u].x, b.y, fma(-l[u].y, b.x, acc)) : fma(l[u].x, b.x, fma(l[u].y, b.y, acc));
    }
    return acc;
}

template <int E, int RB>
__device__ __forceinline__ double undo_at(double2 (&v)[E], double2 (&l)[E], bool imag, double c, double w,
                                          const Signs& sg) {
    double g;
    if (imag) {
        g = overlap<E, true>(v, l, 1u << RB, sg);
        rotate<E, RB, true>(v, c, w, sg);
        rotate<E, RB, true>(l, c, w, sg);
    } else {
        g = overlap<E, false>(v, l, 1u << RB, sg);
        rotate<E, RB, false>(v, c, w, sg);
        rotate<E, RB, false>(l, c, w, sg);
    }
    return g;
}

__device__ __forceinline__ uint64_t tile_base(const AdjPass& p, uint64_t t) {
    for (uint32_t i = 0; i < p.m; ++i) t = insert_zero_bit(t, p.pivots[i]);
    return t;
}

// Global offsets of a thread's amplitudes at the load (e = 0) or the store (1): a thread part,
// and one vector per register bit.
template <int TB>
__device__ __forceinline__ uint64_t thread_offset(const AdjPass& p, int e) {
    uint64_t g = 0;
#pragma unroll
    for (int i = 0; i < TB; ++i)
        if ((threadIdx.x >> i) & 1u) g ^= p.tvec[e][i];
    return g;
}
template <int RB>
__device__ __forceinline__ uint64_t reg_offset(const AdjPass& p, int e, int u) {
    uint64_t g = 0;
#pragma unroll
    for (int i = 0; i < RB; ++i)
        if ((u >> i) & 1) g ^= p.rvec[e][i];
    return g;
}
template <int TB>
__device__ __forceinline__ uint32_t thread_slot(const AdjLayout& l) {
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < TB; ++i)
        if ((threadIdx.x >> i) & 1u) s ^= l.t[i];
    return s;
}
template <int RB>
__device__ __forceinline__ uint32_t reg_slot(const AdjLayout& l, int u) {
    uint32_t s = 0;
#pragma unroll
    for (int i = 0; i < RB; ++i)
        if ((u >> i) & 1) s ^= l.r[i];
    return s;
}

// (cos, sin) of the pass's rotations for this CTA's state.
__device__ __forceinline__ void stage_angles(double2* s_cs, const AdjPass& p,
                                             const double2* __restrict__ cs, uint32_t R) {
    for (uint32_t k = threadIdx.x; k < p.n_rots; k += blockDim.x)
        s_cs[k] = __ldg(cs + static_cast<uint64_t>(p.rot[k].param) * R + blockIdx.y);
}

template <int M>
__global__ void __launch_bounds__(1 << (M - 4), 1 << (13 - M))
k_adj_fwd(double2* __restrict__ st, uint64_t len, const __grid_constant__ AdjPass p,
          const double2* __restrict__ cs, uint32_t R) {
    constexpr int TB = M - 4, E = 16;
    extern __shared__ __align__(16) double2 tile[];
    __shared__ double2 s_cs[kAdjMaxRots];
    stage_angles(s_cs, p, cs, R);
    const uint64_t base = tile_base(p, blockIdx.x);
    double2* s = st + static_cast<uint64_t>(blockIdx.y) * len;
    double2 v[E];
    {
        const uint64_t g = base ^ thread_offset<TB>(p, 0);
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = __ldcs(s + (g ^ reg_offset<4>(p, 0, u)));
    }
    __syncthreads();
    uint32_t cur = 0;
    for (uint32_t k = 0; k < p.n_rots; ++k) {
        const AdjRot& r = p.rot[k];
        while (cur != r.layout) {
            if (cur) __syncthreads();   // the previous remap's reads
            const uint32_t a = thread_slot<TB>(p.lay[cur]);
#pragma unroll
            for (int u = 0; u < E; ++u) tile[a ^ reg_slot<4>(p.lay[cur], u)] = v[u];
            cur = r.layout;
            __syncthreads();
            const uint32_t b = thread_slot<TB>(p.lay[cur]);
#pragma unroll
            for (int u = 0; u < E; ++u) v[u] = tile[b ^ reg_slot<4>(p.lay[cur], u)];
        }
        const double2 csv = s_cs[k];
        const Signs sg(__popcll(base & r.zy) + __popc(threadIdx.x & r.tz), r.rz);
        dispatch_rotate<E>(v, r, csv.x, second_factor(csv.y, r.n_y), sg);
    }
    const uint64_t g = base ^ thread_offset<TB>(p, 1);
#pragma unroll
    for (int u = 0; u < E; ++u) s[g ^ reg_offset<4>(p, 1, u)] = v[u];
}

template <int M>
__global__ void __launch_bounds__(1 << (M - 3), 1 << (12 - M))
k_adj_bwd(double2* __restrict__ psi, double2* __restrict__ lam, uint64_t len,
          const __grid_constant__ AdjPass p, const double2* __restrict__ cs, uint32_t R,
          double* __restrict__ partials) {
    constexpr int TB = M - 3, E = 8, W = 1 << (M - 3 - 5);
    extern __shared__ __align__(16) double2 tile[];   // psi, then lambda
    __shared__ double2 s_cs[kAdjMaxRots];
    __shared__ double red[kAdjMaxRots][W];
    stage_angles(s_cs, p, cs, R);
    const uint64_t base = tile_base(p, blockIdx.x);
    double2* gp = psi + static_cast<uint64_t>(blockIdx.y) * len;
    double2* gl = lam + static_cast<uint64_t>(blockIdx.y) * len;
    double2 v[E], l[E];
    {
        const uint64_t g = base ^ thread_offset<TB>(p, 0);
#pragma unroll
        for (int u = 0; u < E; ++u) {
            v[u] = __ldcs(gp + (g ^ reg_offset<3>(p, 0, u)));
            l[u] = __ldcs(gl + (g ^ reg_offset<3>(p, 0, u)));
        }
    }
    __syncthreads();
    uint32_t cur = 0;
    for (uint32_t k = 0; k < p.n_rots; ++k) {
        const AdjRot& r = p.rot[k];
        while (cur != r.layout) {
            if (cur) __syncthreads();
            const uint32_t a = thread_slot<TB>(p.lay[cur]);
#pragma unroll
            for (int u = 0; u < E; ++u) {
                tile[a ^ reg_slot<3>(p.lay[cur], u)] = v[u];
                tile[(1u << M) + (a ^ reg_slot<3>(p.lay[cur], u))] = l[u];
            }
            cur = r.layout;
            __syncthreads();
            const uint32_t b = thread_slot<TB>(p.lay[cur]);
#pragma unroll
            for (int u = 0; u < E; ++u) {
                v[u] = tile[b ^ reg_slot<3>(p.lay[cur], u)];
                l[u] = tile[(1u << M) + (b ^ reg_slot<3>(p.lay[cur], u))];
            }
        }
        const double2 csv = s_cs[k];
        const Signs sg(__popcll(base & r.zy) + __popc(threadIdx.x & r.tz), r.rz);
        const double c = csv.x, w = second_factor(-csv.y, r.n_y);   // the inverse rotation
        const bool imag = (r.n_y & 1u) == 0;
        double g;
        switch (r.rbit) {
            case 0: g = undo_at<E, 0>(v, l, imag, c, w, sg); break;
            case 1: g = undo_at<E, 1>(v, l, imag, c, w, sg); break;
            case 2: g = undo_at<E, 2>(v, l, imag, c, w, sg); break;
            default:   // x = 0: the string is its own Z signs
                g = imag ? overlap<E, true>(v, l, 0u, sg) : overlap<E, false>(v, l, 0u, sg);
                rotate_diag<E>(v, c, w, sg);
                rotate_diag<E>(l, c, w, sg);
        }
        // Im(i^{n_y} z): Im z, Re z, -Im z, -Re z
        if (r.n_y & 2u) g = -g;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
        if ((threadIdx.x & 31u) == 0) red[k][threadIdx.x >> 5] = g;
    }
    {
        const uint64_t g = base ^ thread_offset<TB>(p, 1);
#pragma unroll
        for (int u = 0; u < E; ++u) {
            gp[g ^ reg_offset<3>(p, 1, u)] = v[u];
            gl[g ^ reg_offset<3>(p, 1, u)] = l[u];
        }
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < p.n_rots; k += blockDim.x) {
        double t = 0.0;
#pragma unroll
        for (int i = 0; i < W; ++i) t += red[k][i];
        partials[(static_cast<uint64_t>(k) * gridDim.y + blockIdx.y) * gridDim.x + blockIdx.x] = t;
    }
}

// grad[state * np + param_k] = sum over tiles of partials[(k * nb + state) * n_tiles + t]: one
// warp per (rotation, state), lanes over the tiles in order, then a butterfly.
__global__ void __launch_bounds__(256) k_adj_grad(const double* __restrict__ partials, uint32_t n_tiles,
                                                  uint32_t nb, const __grid_constant__ AdjPass p,
                                                  double* __restrict__ grad, uint64_t np) {
    const uint32_t k = blockIdx.y, b = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (b >= nb) return;   // whole warps
    const double* row = partials + (static_cast<uint64_t>(k) * nb + b) * n_tiles;
    double v = 0.0;
    for (uint32_t t = lane; t < n_tiles; t += 32) v += row[t];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) grad[static_cast<uint64_t>(b) * np + p.rot[k].param] = v;
}

// ---------------------------------------------------------------- expectations
// Statevector::expectation_value (src/backend/statevector.cpp:39-78):
// <P> = Re( i^{n_y} sum_i s_i a_i conj(a_{i ^ x}) ), s_i = (-1)^{popcount(i & zy)}.
// The terms of i and i ^ x are conjugate up to (-1)^{n_y} (n_y = popcount(x & zy) mod 2), so a
// pair gives twice a real (n_y even) or imaginary (odd) part.

// Sum of s_u |a_u|^2, or of s_u times that part over the pairs of register bit RB.
template <int E, int RB, bool ODD>
__device__ __forceinline__ double pair_sum(const double2 (&v)[E], const Signs& sg) {
    double acc = 0.0;
#pragma unroll
    for (int u = 0; u < E; ++u) {
        if ((u >> RB) & 1) continue;
        const double2 a = v[u], b = v[u | (1 << RB)];
        const double r = ODD ? fma(a.y, b.x, -a.x * b.y) : fma(a.x, b.x, a.y * b.y);
        acc += toggle(r, sg(u));
    }
    return acc;
}
template <int RB>
__device__ __forceinline__ double term_sum(const double2 (&v)[16], uint32_t n_y, const Signs& sg) {
    return (n_y & 1u) ? pair_sum<16, RB, true>(v, sg) : pair_sum<16, RB, false>(v, sg);
}

// The factor of a term's sum: 2 i^{n_y} (n_y even) or 2 i^{n_y + 1} (odd); 1 without pairs.
__device__ __forceinline__ double term_factor(bool pairs, uint32_t n_y) {
    if (!pairs) return 1.0;
    return (n_y == 0u || n_y == 3u) ? 2.0 : -2.0;
}

// Persistent CTAs over the tiles; each thread keeps a sum per term (in shared memory), added up
// tile after tile, and the block's sums go out once.  A read of the state (16 bytes per amplitude)
// serves up to eight independent x masks, where a launch per x mask read it for each.  A CTA loads
// a tile and sums it one after the other, so the CTAs of an SM overlap with each other only: four
// on tiles of 2^11 beat two on 2^12 (nine masks a read) and eight on 2^10.  100 terms on 24 qubits:
// 7.09 ms with a launch per mask, 1.25 with 2^12, 0.95 with 2^11, 1.00 with 2^10, 1.06 with 2^9;
// 150 terms on 26 qubits 6.6 (2^12), 4.8 (2^11); 40 terms on 15 qubits 0.092 both.
__global__ void __launch_bounds__(kExpectThreads, kExpectCtas)
k_expect_pass(const double2* __restrict__ s, uint32_t n_tiles, const __grid_constant__ AdjPass p,
              double* __restrict__ partials) {
    constexpr int M = kExpectTileBits, TB = M - 4, E = 16;
    constexpr uint32_t T = 1u << TB;
    extern __shared__ __align__(16) double2 tile[];
    double* sums = reinterpret_cast<double*>(tile + (1u << M));
    for (uint32_t k = 0; k < p.n_rots; ++k) sums[k * T + threadIdx.x] = 0.0;
    const uint64_t off = thread_offset<TB>(p, 0);
    for (uint32_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
        const uint64_t base = tile_base(p, t);
        double2 v[E];
#pragma unroll
        for (int u = 0; u < E; ++u) v[u] = __ldcs(s + (base ^ off ^ reg_offset<4>(p, 0, u)));
        uint32_t cur = 0;
        for (uint32_t k = 0; k < p.n_rots; ++k) {
            const AdjRot& r = p.rot[k];
            if (cur != r.layout) {
                __syncthreads();   // the previous remap's reads
                const uint32_t a = thread_slot<TB>(p.lay[cur]);
#pragma unroll
                for (int u = 0; u < E; ++u) tile[a ^ reg_slot<4>(p.lay[cur], u)] = v[u];
                cur = r.layout;
                __syncthreads();
                const uint32_t b = thread_slot<TB>(p.lay[cur]);
#pragma unroll
                for (int u = 0; u < E; ++u) v[u] = tile[b ^ reg_slot<4>(p.lay[cur], u)];
            }
            const Signs sg(__popcll(base & r.zy) + __popc(threadIdx.x & r.tz), r.rz);
            double g;
            switch (r.rbit) {
                case 0: g = term_sum<0>(v, r.n_y, sg); break;
                case 1: g = term_sum<1>(v, r.n_y, sg); break;
                case 2: g = term_sum<2>(v, r.n_y, sg); break;
                case 3: g = term_sum<3>(v, r.n_y, sg); break;
                default:
                    g = 0.0;
#pragma unroll
                    for (int u = 0; u < E; ++u) g += toggle(fma(v[u].x, v[u].x, v[u].y * v[u].y), sg(u));
            }
            sums[k * T + threadIdx.x] += g;
        }
    }
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k = threadIdx.x >> 5; k < p.n_rots; k += T / 32) {
        double g = 0.0;
#pragma unroll
        for (uint32_t j = 0; j < T / 32; ++j) g += sums[k * T + j * 32 + lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
        const AdjRot& r = p.rot[k];
        if (lane == 0)
            partials[static_cast<uint64_t>(r.param) * gridDim.x + blockIdx.x] =
                term_factor(r.rbit != kAdjDiag, r.n_y) * g;
    }
}

// out[t] = the sum of term t's partials: one warp, lanes over the blocks in order, a butterfly.
__global__ void __launch_bounds__(256) k_expect_sum(const double* __restrict__ partials, uint32_t blocks,
                                                    uint32_t n_terms, double* __restrict__ out) {
    const uint32_t t = blockIdx.x * 8u + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (t >= n_terms) return;   // whole warps
    double g = 0.0;
    for (uint32_t b = lane; b < blocks; b += 32) g += partials[static_cast<uint64_t>(t) * blocks + b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    if (lane == 0) out[t] = g;
}

// States of up to 2^14 amplitudes: one block per term, the state from L2.
__global__ void __launch_bounds__(256) k_expect_small(const double2* __restrict__ s, uint64_t len,
                                                      const AdjRotation* __restrict__ terms,
                                                      double* __restrict__ out) {
    const AdjRotation r = terms[blockIdx.x];
    double g = 0.0;
    if (r.x == 0) {
        for (uint64_t i = threadIdx.x; i < len; i += blockDim.x) {
            const double2 a = __ldg(s + i);
            g += toggle(fma(a.x, a.x, a.y * a.y), static_cast<uint32_t>(__popcll(i & r.zy)) << 31);
        }
    } else {
        const unsigned hb = 63u - static_cast<unsigned>(__clzll(static_cast<long long>(r.x)));
        for (uint64_t q = threadIdx.x; q < len / 2; q += blockDim.x) {
            const uint64_t i = insert_zero_bit(q, hb);
            const double2 a = __ldg(s + i), b = __ldg(s + (i ^ r.x));
            const double z = (r.n_y & 1u) ? fma(a.y, b.x, -a.x * b.y) : fma(a.x, b.x, a.y * b.y);
            g += toggle(z, static_cast<uint32_t>(__popcll(i & r.zy)) << 31);
        }
    }
    __shared__ double red[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = g;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) t += red[w];
        out[blockIdx.x] = term_factor(r.x != 0, r.n_y & 3u) * t;
    }
}

void check_pass(const AdjPass& p, uint32_t n, uint32_t regs) {
    if (p.m > n || p.m < kAdjMinBits || p.m > kAdjMaxBits || p.regs != regs ||
        p.n_rots > kAdjMaxRots || p.n_rots == 0 || p.n_layouts > kAdjMaxLayouts)
        throw std::logic_error("adjoint pass: unsupported shape");
}

template <int M>
void fwd(const LaunchCtx& ctx, double2* st, uint32_t n, uint32_t nb, const AdjPass& p,
         const double2* d_cs, uint32_t R) {
    const size_t smem = sizeof(double2) << M;
    cuda_check_launch_attr(cudaFuncSetAttribute(k_adj_fwd<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                static_cast<int>(smem)));
    k_adj_fwd<M><<<dim3(1u << (n - M), nb), 1 << (M - 4), smem, ctx.stream>>>(st, uint64_t{1} << n, p, d_cs, R);
    check_launch("adjoint pass (forward)");
}

template <int M>
void bwd(const LaunchCtx& ctx, double2* psi, double2* lam, uint32_t n, uint32_t nb, const AdjPass& p,
         const double2* d_cs, uint32_t R, double* d_partials) {
    const size_t smem = 2 * sizeof(double2) << M;
    cuda_check_launch_attr(cudaFuncSetAttribute(k_adj_bwd<M>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                static_cast<int>(smem)));
    k_adj_bwd<M><<<dim3(1u << (n - M), nb), 1 << (M - 3), smem, ctx.stream>>>(
        psi, lam, uint64_t{1} << n, p, d_cs, R, d_partials);
    check_launch("adjoint pass (backward)");
}

}  // namespace

uint32_t expect_blocks(const LaunchCtx& ctx, uint32_t n) {
    return std::min<uint32_t>(1u << (n - kExpectTileBits), static_cast<uint32_t>(ctx.num_sms) * kExpectCtas);
}

void launch_expect_pass(const LaunchCtx& ctx, const double2* st, uint32_t n, const AdjPass& p,
                        double* d_partials) {
    check_pass(p, n, 4);
    if (p.m != kExpectTileBits || p.n_rots > kExpectTerms) throw std::logic_error("expectation pass: unsupported shape");
    const size_t smem = (sizeof(double2) << kExpectTileBits) + sizeof(double) * p.n_rots * (1u << (kExpectTileBits - 4));
    cuda_check_launch_attr(cudaFuncSetAttribute(k_expect_pass, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                static_cast<int>(smem)));
    k_expect_pass<<<expect_blocks(ctx, n), kExpectThreads, smem, ctx.stream>>>(st, 1u << (n - kExpectTileBits), p, d_partials);
    check_launch("expectation pass");
}

void launch_expect_sum(const LaunchCtx& ctx, uint32_t n, uint32_t n_terms, const double* d_partials,
                       double* d_out) {
    k_expect_sum<<<(n_terms + 7) / 8, 256, 0, ctx.stream>>>(d_partials, expect_blocks(ctx, n), n_terms, d_out);
    check_launch("expectation sum");
}

void launch_expect_small(const LaunchCtx& ctx, const double2* st, uint32_t n,
                         const AdjRotation* d_terms, uint32_t n_terms, double* d_out) {
    k_expect_small<<<n_terms, 256, 0, ctx.stream>>>(st, uint64_t{1} << n, d_terms, d_out);
    check_launch("expectation");
}

void launch_adj_fwd(const LaunchCtx& ctx, double2* st, uint32_t n, uint32_t nb, const AdjPass& p,
                    const double2* d_cs, uint32_t R) {
    check_pass(p, n, kAdjFwdRegs);
    switch (p.m) {
        case 9: fwd<9>(ctx, st, n, nb, p, d_cs, R); break;
        case 10: fwd<10>(ctx, st, n, nb, p, d_cs, R); break;
        case 11: fwd<11>(ctx, st, n, nb, p, d_cs, R); break;
        default: fwd<12>(ctx, st, n, nb, p, d_cs, R); break;
    }
}

void launch_adj_bwd(const LaunchCtx& ctx, double2* psi, double2* lam, uint32_t n, uint32_t nb,
                    const AdjPass& p, const double2* d_cs, uint32_t R, double* d_partials,
                    double* d_grad, uint64_t np) {
    check_pass(p, n, kAdjBwdRegs);
    switch (p.m) {
        case 9: bwd<9>(ctx, psi, lam, n, nb, p, d_cs, R, d_partials); break;
        case 10: bwd<10>(ctx, psi, lam, n, nb, p, d_cs, R, d_partials); break;
        case 11: bwd<11>(ctx, psi, lam, n, nb, p, d_cs, R, d_partials); break;
        default: bwd<12>(ctx, psi, lam, n, nb, p, d_cs, R, d_partials); break;
    }
    k_adj_grad<<<dim3((nb + 7) / 8, p.n_rots), 256, 0, ctx.stream>>>(d_partials, 1u << (n - p.m), nb, p,
                                                                     d_grad, np);
    check_launch("adjoint gradients");
}

}  // namespace lqcs_b200
