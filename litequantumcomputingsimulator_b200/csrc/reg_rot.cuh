// reg_rot.cuh — register tile passes in rotation form: the kernel and its launch, for up to CAP
// records (reg_rot_kernels.cu and reg_rot_long.cu instantiate it).
//
// The passes of reg_tile_kernels.cu (one HBM read and write of the state applies a whole list
// of operations to tiles of 2^M amplitudes, 16 per thread in registers, remaps through
// swizzled shared memory), with the gates factored so that a pass is made of three kinds of
// work: real rotations on register bits (two FP64 FMAs per amplitude and gate),
// diagonal tables (one complex multiply per amplitude for every diagonal factor and controlled
// phase that waits on a table's bits: three thread bits beside the register bits where the entries
// are expanded, any six where they are strided), and signs.  A CZ to a
// qubit outside the tile is a Z on the tile bit in half of the tiles; Z moves through a
// rotation by flipping the sign of x and y, so such gates cost no work per amplitude until one
// sign pass at the end (kRegSign).
//
// What bounds it: with dense 4 x 4 blocks the same passes issued 16 FP64 FMAs per amplitude
// and block and read 32 matrix entries per thread and block from shared memory, and ran at
// half of the FP64 rate; rotation form issues less than half of the FP64 work and a third of
// the shared-memory reads, over fewer passes (an out-of-tile target no longer blocks a CX).
// Measured, dense blocks against rotation form: 30-qubit brickwork of depth 40 857 -> 562 ms (48
// passes at 0.29 of HBM -> 40 at 0.37, 32 TFLOP/s of the gate-by-gate work), QFT(27) 12.9 -> 8.1
// ms (0.57 of HBM), the 26-qubit gate mix 24.7 -> 16.0 ms.  What is left is latency: 16 warps per
// SM at 128 registers, FP64 pipe 41 % busy, the rest on shared-memory loads, remaps (a store of a
// register to shared memory costs a warp 4.7 cycles of the SM) and barriers.  Pauli rotations are
// not the bound: with half of their FP64 work, over twice the code paths, the mix took 16.6 ms.
#pragma once

#include <algorithm>
#include <stdexcept>
#include <string>

#include "kernels.cuh"
#include "reg_ops.cuh"
#include "tile.cuh"

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

// x with its sign bit toggled by bit 31 of s.
__device__ __forceinline__ double toggle(double x, uint32_t s) {
    return __hiloint2double(__double2hiint(x) ^ static_cast<int>(s), __double2loint(x));
}

__device__ __forceinline__ uint64_t mask_at(uint32_t saddr) {
    return static_cast<uint64_t>(__double_as_longlong(lds2(saddr).x));
}

// The tile stays in the registers it is in: every operation overwrites its own operands, so
// that the branches of the record loop agree on where each amplitude is and the compiler does
// not move amplitudes between registers at their joins.
__device__ __forceinline__ void fma_to(double& acc, double a, double b) {
    asm("fma.rn.f64 %0, %1, %2, %0;" : "+d"(acc) : "d"(a), "d"(b));
}
// v *= f
__device__ __forceinline__ void cmul_to(double2& v, double2 f) {
    asm("{\n\t"
        ".reg .f64 t, u;\n\t"
        "mul.rn.f64 t, %3, %1;\n\t"
        "mul.rn.f64 u, %3, %0;\n\t"
        "neg.f64 t, t;\n\t"
        "fma.rn.f64 %0, %2, %0, t;\n\t"
        "fma.rn.f64 %1, %2, %1, u;\n\t"
        "}"
        : "+d"(v.x), "+d"(v.y) : "d"(f.x), "d"(f.y));
}
// v *= f, w *= g: the products of both before the sums, so that no sum waits for its product.
__device__ __forceinline__ void cmul_to(double2& v, double2& w, double2 f, double2 g) {
    asm("{\n\t"
        ".reg .f64 t, u, p, q;\n\t"
        "mul.rn.f64 t, %5, %1;\n\t"
        "mul.rn.f64 u, %5, %0;\n\t"
        "mul.rn.f64 p, %7, %3;\n\t"
        "mul.rn.f64 q, %7, %2;\n\t"
        "neg.f64 t, t;\n\t"
        "neg.f64 p, p;\n\t"
        "fma.rn.f64 %0, %4, %0, t;\n\t"
        "fma.rn.f64 %1, %4, %1, u;\n\t"
        "fma.rn.f64 %2, %6, %2, p;\n\t"
        "fma.rn.f64 %3, %6, %3, q;\n\t"
        "}"
        : "+d"(v.x), "+d"(v.y), "+d"(w.x), "+d"(w.y)
        : "d"(f.x), "d"(f.y), "d"(g.x), "d"(g.y));
}

// a0 += x a1, then a1 += y a0 on register bit TM, both signs toggled by bit 31 of `sign`.  Each
// FMA overwrites its own addend: computing both new halves from the old ones took a register
// move for every FMA.
template <int TM>
__device__ __forceinline__ void rotation(double2 (&v)[kE], double2 xy, uint32_t sign) {
    const double x = toggle(xy.x, sign), y = toggle(xy.y, sign);
#pragma unroll
    for (int b = 0; b < kE; ++b) {
        if (b & TM) continue;
        fma_to(v[b].x, x, v[b | TM].x);
        fma_to(v[b].y, x, v[b | TM].y);
    }
#pragma unroll
    for (int b = 0; b < kE; ++b) {
        if (b & TM) continue;
        fma_to(v[b | TM].x, y, v[b].x);
        fma_to(v[b | TM].y, y, v[b].y);
    }
}

// Rotations on the register bits of `code`, their (x, y) at `mat` in bit order, the first in xy;
// bit j of zb: the j-th one's sign.  Each (x, y) is loaded before the rotation in front of it
// (one entry is read past the last: the layouts lie there).
__device__ __forceinline__ void rotations(double2 (&v)[kE], uint32_t code, uint32_t mat, double2 xy,
                                          uint32_t zb) {
    if (code & 1u) { const double2 c = xy; xy = lds2(mat += 16u); rotation<1>(v, c, zb << 31); zb >>= 1; }
    if (code & 2u) { const double2 c = xy; xy = lds2(mat += 16u); rotation<2>(v, c, zb << 31); zb >>= 1; }
    if (code & 4u) { const double2 c = xy; xy = lds2(mat += 16u); rotation<4>(v, c, zb << 31); zb >>= 1; }
    if (code & 8u) rotation<8>(v, xy, zb << 31);
}

// Diagonal tables.  One code path for every set of register bits: a switch over them (2^r loads
// instead of 16) made the allocator spill 600 bytes per thread, and a load of one entry by a
// whole warp costs 1.2 cycles of the SM, against 2 for the four FMAs it feeds.  Expanded: entry u
// of the thread's sixteen.
__device__ __forceinline__ void table_expanded(double2 (&v)[kE], uint32_t addr) {
    double2 f = lds2(addr), g = lds2(addr + 16u);
#pragma unroll
    for (int u = 0; u < kE; u += 2) {   // the next two entries on their way
        double2 f1, g1;
        if (u + 2 < kE) {
            f1 = lds2(addr + 16u * (u + 2));
            g1 = lds2(addr + 16u * (u + 3));
        }
        cmul_to(v[u], v[u + 1], f, g);
        f = f1;
        g = g1;
    }
}
// Strided: the entry at addr + the strides of u's register bits (zero for bits the table does
// not use).
__device__ __forceinline__ void table_strided(double2 (&v)[kE], uint32_t addr, uint32_t s0, uint32_t s1,
                                              uint32_t s2, uint32_t s3) {
#pragma unroll
    for (int u = 0; u < kE; ++u)
        cmul_to(v[u], lds2(addr + ((u & 1) ? s0 : 0u) + ((u & 2) ? s1 : 0u) + ((u & 4) ? s2 : 0u) +
                           ((u & 8) ? s3 : 0u)));
}

// A pass and its records as a kernel parameter: the record loop then decodes them with
// warp-uniform loads and branches on uniform values.
template <uint32_t CAP>
struct RotPass {
    RegPass pass;
    RegOp ops[CAP];
};

// DENSE: some record is a dense or a controlled diagonal operation; PAULI: some is a Pauli
// rotation.  A kernel carries only the paths its pass uses (registers, instruction cache).
template <int M, int MINB, bool DENSE, bool PAULI, uint32_t CAP>
__global__ void __launch_bounds__(1 << (M - kRegBits), MINB)
k_regrot(double2* __restrict__ st, const __grid_constant__ RotPass<CAP> rp,
         const RegLayout* __restrict__ layouts, const double2* __restrict__ mats) {
    const RegPass& p = rp.pass;
    constexpr uint32_t kT = 1u << (M - kRegBits);
    constexpr uint32_t kTB = M - kRegBits;
    extern __shared__ __align__(16) unsigned char smem[];
    double2* smat = reinterpret_cast<double2*>(smem) + (1u << M);   // behind the tile
    RegLayout* slay = reinterpret_cast<RegLayout*>(smat + p.n_mat);
    double2* sdyn = reinterpret_cast<double2*>(
        (reinterpret_cast<uintptr_t>(slay + p.n_layouts) + 15u) & ~uintptr_t{15});
    __shared__ uint64_t gbit[kRegMaxBits];    // global offset of each tile bit at the load
    __shared__ uint64_t sgbit[kRegMaxBits];   // and at the store (relabelled by SWAPs)
    __shared__ uint32_t shbits[kTileMaxHigh];
    __shared__ uint32_t sdynrec[kRegMaxDyn];
    // per-thread constants of every tile: the global offsets of the thread bits at the load
    // and at the store, each layout's shared-memory slot of the thread
    // (the store's with the bits that end up negated: such a register bit steps down)
    __shared__ uint64_t s_ldg[kT], s_stg[kT];
    __shared__ int64_t s_ldr[kRegBits], s_str[kRegBits];
    __shared__ uint16_t s_tslot[kRegSlotLayouts * kT];
    if (threadIdx.x < kTileMaxHigh) {
#pragma unroll
        for (uint32_t i = 0; i < kTileMaxHigh; ++i)
            if (threadIdx.x == i) shbits[i] = p.hbits[i];   // static indices
    }
    if (threadIdx.x < kRegMaxDyn) {
#pragma unroll
        for (uint32_t i = 0; i < kRegMaxDyn; ++i)
            if (threadIdx.x == i) sdynrec[i] = p.dyn_rec[i];
    }
    if (threadIdx.x < M) {
#pragma unroll
        for (uint32_t b = 0; b < kRegMaxBits; ++b)
            if (threadIdx.x == b) sgbit[b] = uint64_t{1} << p.store_qubit[b];
#pragma unroll
        for (uint32_t i = 0; i < kTileMaxHigh; ++i)
            if (threadIdx.x == p.L + i) gbit[threadIdx.x] = uint64_t{1} << p.hbits[i];
        if (threadIdx.x < p.L) gbit[threadIdx.x] = uint64_t{1} << threadIdx.x;
    }
    {
        const uint4* src4 = reinterpret_cast<const uint4*>(
            mats + static_cast<uint64_t>(blockIdx.y) * p.mat_stride);   // this state's matrices
        uint4* dst4 = reinterpret_cast<uint4*>(smat);
        for (uint32_t w = threadIdx.x; w < p.n_mat; w += kT) dst4[w] = __ldg(src4 + w);
        const uint32_t* src = reinterpret_cast<const uint32_t*>(layouts);
        uint32_t* dst = reinterpret_cast<uint32_t*>(slay);
        for (uint32_t w = threadIdx.x; w < p.n_layouts * (sizeof(RegLayout) / 4); w += kT)
            dst[w] = __ldg(src + w);
    }
    __syncthreads();
    {
        const uint32_t last = p.last_layout;
        s_ldg[threadIdx.x] = thread_goff(slay[0], kTB, gbit);
        const uint64_t undo = static_cast<uint64_t>(__double_as_longlong(smat[0].x));
        s_stg[threadIdx.x] = thread_goff(slay[last], kTB, sgbit) ^ undo;
        for (uint32_t l = 0; l < p.n_layouts && l < kRegSlotLayouts; ++l)
            s_tslot[l * kT + threadIdx.x] = static_cast<uint16_t>(thread_slot(slay[l], kTB));
        if (threadIdx.x < kRegBits) {
            s_ldr[threadIdx.x] = static_cast<int64_t>(gbit[slay[0].rpos[threadIdx.x]]);
            const int64_t g = static_cast<int64_t>(sgbit[slay[last].rpos[threadIdx.x]]);
            s_str[threadIdx.x] = (static_cast<uint64_t>(g) & undo) ? -g : g;
        }
    }
    __syncthreads();
    const bool slot_table = p.n_layouts <= kRegSlotLayouts;   // uniform
    const uint32_t smat_addr = static_cast<uint32_t>(__cvta_generic_to_shared(smat));
    const uint32_t sdyn_addr = static_cast<uint32_t>(__cvta_generic_to_shared(sdyn));
    const uint32_t lane = threadIdx.x & 31u;
    double2* __restrict__ s = st + static_cast<uint64_t>(blockIdx.y) * p.batch_stride;
    // tile t's index bits: t spread over the bits outside the tile (t < 2^28: n <= 40)
    auto tile_base = [&](uint32_t t) {
        for (uint32_t i = 0; i < p.h; ++i) {
            const uint32_t low = (1u << (shbits[i] - p.L)) - 1u;
            t = ((t & ~low) << 1) | (t & low);
        }
        return static_cast<uint64_t>(t) << p.L;
    };
    uint64_t row = 0;   // the tile row this thread prefetches
    for (uint32_t i = 0; i < p.h; ++i)
        if ((threadIdx.x >> i) & 1u) row |= uint64_t{1} << shbits[i];
    const uint32_t n_tiles = static_cast<uint32_t>(p.n_tiles);
    uint32_t parity = 0;
    uint64_t base = tile_base(blockIdx.x), next = 0;
    for (uint32_t tid = blockIdx.x; tid < n_tiles; tid += gridDim.x, parity ^= 1u, base = next) {
        // a warp's shared-memory slots differ between layouts with different warp bits:
        // the previous tile's last remap must be done before this tile's first
        if (p.sync_tiles) __syncthreads();
        double2 v[kE];
        {
            const double2* src = s + (base + s_ldg[threadIdx.x]);
            const int64_t g0 = s_ldr[0], g1 = s_ldr[1], g2 = s_ldr[2], g3 = s_ldr[3];
#pragma unroll
            for (int u = 0; u < kE; ++u)
                v[u] = __ldcs(src + (((u & 1) ? g0 : 0) + ((u & 2) ? g1 : 0) + ((u & 4) ? g2 : 0) +
                                     ((u & 8) ? g3 : 0)));
        }
        // relabelled stores go to places other warps load: all loads before any store
        if (p.load_barrier) __syncthreads();
        // the HBM reads of this CTA's next tile go to L2 while this one computes: thread
        // r < 2^h takes the row of high-bit pattern r, 16 B * 2^L from a 16 B boundary
        if (gridDim.x < n_tiles - tid) {
            next = tile_base(tid + gridDim.x);
            if (threadIdx.x < (1u << p.h))
                asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(s + (next | row)),
                             "r"(16u << p.L)
                             : "memory");
        }
        // Per-tile tables: entry e is its base entry times every gated term whose out-of-tile
        // qubits are all 1 in this tile and whose entry bits e contains.  The barrier after
        // the build also ends the use of the other parity's tables (every warp has finished
        // the previous tile), so the next tile may overwrite them.
        const uint32_t dyn_base = parity * p.dyn_entries;
        if (p.n_dyn) {
            for (uint32_t w = threadIdx.x; w < p.n_dyn * 64u; w += kT) {
                const RegOp& op = rp.ops[sdynrec[w >> 6]];
                const uint32_t e = w & 63u;
                if (e >= (1u << op.k)) continue;
                const double2* src = smat + op.mat_off;
                double2 acc = src[e];
                const double2* term = src + (1u << op.k);
                for (uint32_t t = 0; t < op.nterm; ++t) {
                    const double2 meta = term[2 * t + 1];
                    const uint64_t hi = static_cast<uint64_t>(meta.y);
                    const uint64_t gc = static_cast<uint64_t>(meta.x) | ((hi >> 12) << 32);
                    const uint32_t bits = static_cast<uint32_t>(hi & 63u),
                                   value = static_cast<uint32_t>((hi >> 6) & 63u);
                    if ((base & gc) == gc && (e & bits) == value) acc = cmul(term[2 * t], acc);
                }
                sdyn[dyn_base + (op.kind == kRegStage ? op.dyn_table : op.dyn_off) + e] = acc;
            }
            __syncthreads();
        }
        uint64_t signs = 0;   // of the rotations in this tile (bits from n_signs on are 0)
        if (p.n_signs) {
            const uint32_t at = smat_addr + 16u * p.sign_off;
            bool odd = false;
            if (lane < p.n_signs) odd = (__popcll(base & mask_at(at + 16u * lane)) & 1) != 0;
            signs = __ballot_sync(0xffffffffu, odd);
            if (p.n_signs > 32u) {
                odd = lane + 32u < p.n_signs && (__popcll(base & mask_at(at + 16u * (lane + 32u))) & 1) != 0;
                signs |= static_cast<uint64_t>(__ballot_sync(0xffffffffu, odd)) << 32;
            }
        }
        uint32_t cur = 0;
        for (uint32_t o = 0; o < p.n_ops; ++o) {
            // a = {gcmask, mat_off, kind | code | k | rcmask}, b = {tcmask | loc[0..1],
            // loc[2..5], nsel | selq[0..1] | nterm, dyn_off | table}
            const uint4* rec = reinterpret_cast<const uint4*>(&rp.ops[o]);
            const uint4 a = rec[0], b = rec[1];
            const uint32_t kind = a.w & 0xffu, code = (a.w >> 8) & 0xffu;
            const uint32_t mat = smat_addr + 16u * a.z;
            if (kind == kRegStage) {
                const uint32_t form = (b.w >> 16) & 0xffu;
                const uint32_t at = smat_addr + 16u * (b.w & 0xffffu);
                const double2 xy = lds2(at);   // the first rotation's, if there is one
                if (form) {   // the table
                    const uint32_t t = threadIdx.x;
                    uint32_t e = ((t >> ((b.x >> 16) & 31u)) & 1u) | ((t >> ((b.x >> 24) & 31u)) & 1u) << 1 |
                                 ((t >> (b.y & 31u)) & 1u) << 2;
                    if (form == kRegTableExpanded) {
                        table_expanded(v, mat + 272u * e);
                    } else {
                        e |= ((t >> ((b.y >> 8) & 31u)) & 1u) << 3 | ((t >> ((b.y >> 16) & 31u)) & 1u) << 4 |
                             ((t >> ((b.y >> 24) & 31u)) & 1u) << 5;
                        const uint32_t tab = (b.z >> 24) ? sdyn_addr + 16u * (dyn_base + (a.x & 0xffffu)) : mat;
                        table_strided(v, tab + 16u * e, (b.z & 0xffu) << 4, (b.z >> 4) & 0xff0u,
                                      (b.z >> 12) & 0xff0u, (a.w >> 20) & 0xff0u);
                    }
                }
                if (code) {
                    const uint32_t sg = b.x & 0xffffu;
                    uint32_t zb = static_cast<uint32_t>(signs >> sg);
                    if (sg > kRegSignBits) {   // lane j: the sign of the j-th rotation
                        const uint32_t nr = static_cast<uint32_t>(__popc(code));
                        bool odd = false;
                        if (lane < nr) odd = (__popcll(base & mask_at(at + 16u * (nr + lane))) & 1) != 0;
                        zb = __ballot_sync(0xffffffffu, odd);
                    }
                    rotations(v, code, at, xy, zb);
                }
                continue;
            }
            if (kind == kRegRemap) {
                auto slots = [&](uint32_t& ts, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
                    const RegLayout& ly = slay[cur];
                    ts = 16u * (slot_table ? s_tslot[cur * kT + threadIdx.x] : thread_slot(ly, kTB));
                    r0 = 16u * ly.rsw[0];
                    r1 = 16u * ly.rsw[1];
                    r2 = 16u * ly.rsw[2];
                    r3 = 16u * ly.rsw[3];
                };
                uint32_t ts, r0, r1, r2, r3;   // in bytes
                slots(ts, r0, r1, r2, r3);
#pragma unroll
                for (int u = 0; u < kE; ++u)
                    *reinterpret_cast<double2*>(smem + (ts ^ ((u & 1) ? r0 : 0) ^ ((u & 2) ? r1 : 0) ^
                                                        ((u & 4) ? r2 : 0) ^ ((u & 8) ? r3 : 0))) = v[u];
                cur = code;
                const bool local = ((a.w >> 16) & 0xffu) != 0;   // uniform: warp bits unchanged
                if (local) __syncwarp();
                else __syncthreads();
                slots(ts, r0, r1, r2, r3);
#pragma unroll
                for (int u = 0; u < kE; ++u)
                    v[u] = *reinterpret_cast<const double2*>(
                        smem + (ts ^ ((u & 1) ? r0 : 0) ^ ((u & 2) ? r1 : 0) ^ ((u & 4) ? r2 : 0) ^
                                ((u & 8) ? r3 : 0)));
                if (local) __syncwarp();
                else __syncthreads();
                continue;
            }
            if (kind == kRegSign) {
                // lanes 0..M-1: whether the thread- or register-index bit at their position
                // carries a Z in this tile; lane M: the tile's own sign; the lanes above: whether
                // the outside qubits of a CZ are both 1
                const uint32_t terms = b.z >> 24;
                bool on = false;
                if (lane < terms) {
                    const uint64_t mk = mask_at(mat + 16u * lane);
                    on = lane <= M ? (__popcll(base & mk) & 1) != 0 : (base & mk) == mk;
                }
                const uint32_t z = __ballot_sync(0xffffffffu, on);
                const uint32_t par = __popc(threadIdx.x & z) + __popc(z >> M);   // threadIdx.x < 2^kTB
                const uint32_t zr = z >> kTB;
                const uint32_t s0 = par << 31, b0 = zr << 31, b1 = (zr >> 1) << 31,
                               b2 = (zr >> 2) << 31, b3 = (zr >> 3) << 31;
#pragma unroll
                for (int u = 0; u < kE; ++u) {
                    const uint32_t sg = s0 ^ ((u & 1) ? b0 : 0u) ^ ((u & 2) ? b1 : 0u) ^
                                        ((u & 4) ? b2 : 0u) ^ ((u & 8) ? b3 : 0u);
                    v[u] = make_double2(toggle(v[u].x, sg), toggle(v[u].y, sg));
                }
                continue;
            }
            const uint64_t gc = static_cast<uint64_t>(a.x) | (static_cast<uint64_t>(a.y) << 32);
            if ((base & gc) != gc) continue;   // uniform across the CTA
            const uint32_t rc = a.w >> 24, tc = b.x & 0xffffu;
            if (kind == kRegPauli) {   // rc / tc: its Z-type bits, not controls
                if constexpr (PAULI)
                    reg_pauli(v, mat, code, rc, tc, (b.x >> 16) & 0xffu, base);
                continue;
            }
            if ((threadIdx.x & tc) != tc) continue;
            if (kind == kRegPhase) {
                const double2 f = lds2(mat);
#pragma unroll
                for (int u = 0; u < kE; ++u)
                    if ((u & rc) == rc) cmul_to(v[u], f);
            } else if (kind == kRegSwapX) {
                dispatch_swapx(v, code, rc);
            } else if constexpr (DENSE) {
                uint32_t moff = 0;
                if (const uint32_t nsel = b.z & 0xffu) {   // picked by the tile's selector bits
                    uint32_t sel = static_cast<uint32_t>(base >> ((b.z >> 8) & 63u)) & 1u;
                    if (nsel > 1) sel |= (static_cast<uint32_t>(base >> ((b.z >> 16) & 63u)) & 1u) << 1;
                    const uint32_t k = (a.w >> 16) & 0xffu;
                    moff = sel << (kind == kRegDense ? 2u * k : k);
                }
                if (kind == kRegDense) dispatch_dense(v, code, SharedMat{mat + 16u * moff}, rc);
                else reg_diag(v, rp.ops[o], SharedMat{mat + 16u * moff}, rc);
            }
        }
        {
            double2* dst = s + (base + s_stg[threadIdx.x]);
            const int64_t g0 = s_str[0], g1 = s_str[1], g2 = s_str[2], g3 = s_str[3];
#pragma unroll
            for (int u = 0; u < kE; ++u)
                __stcs(dst + (((u & 1) ? g0 : 0) + ((u & 2) ? g1 : 0) + ((u & 4) ? g2 : 0) +
                              ((u & 8) ? g3 : 0)),
                       v[u]);
        }
    }
}

template <int M, int MINB, bool DENSE, bool PAULI, uint32_t CAP>
void launch_variant(const LaunchCtx& ctx, double2* st, uint32_t batch, const RegPass& p, size_t smem,
                    const RegOp* ops, const RegLayout* d_layouts, const double2* d_mats) {
    constexpr uint32_t kT = 1u << (M - kRegBits);
    auto kern = k_regrot<M, MINB, DENSE, PAULI, CAP>;
    cuda_check_launch_attr(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                static_cast<int>(kTileMaxSmem)));
    static const size_t static_smem = [&] {
        cudaFuncAttributes a{};
        cuda_check_launch_attr(cudaFuncGetAttributes(&a, kern));
        return a.sharedSizeBytes;
    }();
    const uint32_t by_smem = static_cast<uint32_t>(
        std::max<size_t>(1, (227 * 1024) / (smem + static_smem + 1024)));
    const uint64_t want = static_cast<uint64_t>(ctx.num_sms) * std::min<uint32_t>(MINB, by_smem);
    const uint32_t grid = static_cast<uint32_t>(std::max<uint64_t>(1, std::min<uint64_t>(want, p.n_tiles)));
    static_assert(sizeof(RotPass<CAP>) <= 32 * 1024, "kernel parameters");
    RotPass<CAP> rp;
    rp.pass = p;
    std::copy(ops, ops + p.n_ops, rp.ops);
    kern<<<dim3(grid, batch), kT, smem, ctx.stream>>>(st, rp, d_layouts, d_mats);
    check_launch("register tile pass (rotation form)");
}

// Two CTAs of 128 registers per thread and SM at M = 12 (64 KiB tiles), as many 16-warp sets
// at the other sizes.
template <int M, int MINB, uint32_t CAP>
void launch_size(const LaunchCtx& ctx, double2* st, uint32_t batch, const RegPass& p, size_t smem,
                 const RegOp* ops, const RegLayout* d_layouts, const double2* d_mats) {
    if (!p.pauli_ops && !p.fma_dense)
        launch_variant<M, MINB, false, false, CAP>(ctx, st, batch, p, smem, ops, d_layouts, d_mats);
    else if (!p.pauli_ops)
        launch_variant<M, MINB, true, false, CAP>(ctx, st, batch, p, smem, ops, d_layouts, d_mats);
    else if (!p.fma_dense)
        launch_variant<M, MINB, false, true, CAP>(ctx, st, batch, p, smem, ops, d_layouts, d_mats);
    else
        launch_variant<M, MINB, true, true, CAP>(ctx, st, batch, p, smem, ops, d_layouts, d_mats);
}

}  // namespace

// A pass of up to CAP records, its shape checked (launch_rot_pass).
template <uint32_t CAP>
void launch_rot_records(const LaunchCtx& ctx, double2* st, uint32_t batch, const RegPass& p, size_t smem,
                        const RegOp* ops, const RegLayout* d_layouts, const double2* d_mats) {
    switch (p.m) {
        case 9: launch_size<9, 12, CAP>(ctx, st, batch, p, smem, ops, d_layouts, d_mats); break;
        case 10: launch_size<10, 8, CAP>(ctx, st, batch, p, smem, ops, d_layouts, d_mats); break;
        case 11: launch_size<11, 4, CAP>(ctx, st, batch, p, smem, ops, d_layouts, d_mats); break;
        case 12: launch_size<12, 2, CAP>(ctx, st, batch, p, smem, ops, d_layouts, d_mats); break;
        default: launch_size<13, 1, CAP>(ctx, st, batch, p, smem, ops, d_layouts, d_mats); break;
    }
}

}  // namespace lqcs_b200
