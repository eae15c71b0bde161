// reg_tile_kernels.cu — multi-gate passes with the tile held in registers.
//
// Same passes as tile_kernels.cu (one HBM read and write of the state applies a whole list
// of operations), with a different home for the tile: each thread keeps 16 amplitudes in
// registers and shared memory only serves the remaps that change which 4 tile bits are
// register bits (see RegLayout).  Per amplitude and operation the shared-memory kernel
// moves 32 bytes through shared memory; here a dense operation on register bits moves
// none, so the pass runs at the FP64 rate instead of the shared-memory rate.
//
// Operation semantics follow the reference kernels (src/backend/kernels/gate_kernels.cpp):
// a dense operation is a 2^k x 2^k matrix on its targets applied where every control is 1;
// a diagonal operation multiplies by the entry its target bits select; a phase operation
// multiplies the amplitudes whose phase bits are all 1.
#include <algorithm>
#include <cstdlib>
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

// MINB resident CTAs per SM: registers per thread <= 65536 / (MINB * threads).  FMAD: the
// pass has dense records on register bits (FP64 FMAs); MMA: it has tensor-path records.  A
// kernel carries only the paths its pass uses: with both, the register allocation spills
// (364 bytes at 128 registers against 64 for the FMA path alone and 8 for the tensor path
// alone), so each pass runs the variant of its own records.  PAULI: it has Pauli rotations.
template <int M, int MINB, bool FMAD, bool MMA, bool PAULI>
__global__ void __launch_bounds__(1 << (M - kRegBits), MINB)
k_regtile(double2* __restrict__ st, RegPass p, const RegOp* __restrict__ ops,
          const RegLayout* __restrict__ layouts, const double2* __restrict__ mats) {
    constexpr uint32_t kT = 1u << (M - kRegBits);
    constexpr uint32_t kTB = M - kRegBits;
    extern __shared__ __align__(16) unsigned char smem[];
    double2* __restrict__ tile = reinterpret_cast<double2*>(smem);
    double2* smat = tile + (1u << M);
    RegOp* sops = reinterpret_cast<RegOp*>(smat + p.n_mat);
    RegLayout* slay = reinterpret_cast<RegLayout*>(sops + p.n_ops);
    // per-tile diagonal tables, two sets (tile parity) on a 16-byte boundary
    double2* sdyn = reinterpret_cast<double2*>(
        (reinterpret_cast<uintptr_t>(slay + p.n_layouts) + 15u) & ~uintptr_t{15});
    __shared__ uint64_t gbit[kRegMaxBits];    // global offset of each tile bit at the load
    __shared__ uint64_t sgbit[kRegMaxBits];   // and at the store (relabelled by SWAPs)
    __shared__ uint32_t shbits[kTileMaxHigh];
    __shared__ uint32_t sdynrec[kRegMaxDyn];
    // per-thread constants of every tile, computed once: the global offsets of the thread
    // bits at the load (layout 0) and at the store (the last layout), and each layout's
    // shared-memory slot of the thread (the first kRegSlotLayouts layouts); the register
    // bits' offsets are the same for every thread
    __shared__ uint64_t s_ldg[kT], s_stg[kT];
    __shared__ uint64_t s_ldr[kRegBits], s_str[kRegBits];
    __shared__ uint16_t s_tslot[kRegSlotLayouts * kT];
    if (threadIdx.x == 0) {
#pragma unroll
        for (uint32_t i = 0; i < kTileMaxHigh; ++i) shbits[i] = p.hbits[i];   // static indices
#pragma unroll
        for (uint32_t i = 0; i < kRegMaxDyn; ++i) sdynrec[i] = p.dyn_rec[i];
        for (uint32_t b = 0; b < M; ++b)
            gbit[b] = uint64_t{1} << (b < p.L ? b : shbits[b - p.L]);
        if (p.relabel) {
#pragma unroll
            for (uint32_t b = 0; b < kRegMaxBits; ++b)
                if (b < M) sgbit[b] = uint64_t{1} << p.store_qubit[b];
        }
    }
    const uint64_t* __restrict__ stbit = p.relabel ? sgbit : gbit;   // uniform
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(
            mats + static_cast<uint64_t>(blockIdx.y) * p.mat_stride);   // this state's matrices
        uint32_t* dst = reinterpret_cast<uint32_t*>(smat);
        for (uint32_t w = threadIdx.x; w < p.n_mat * 4u; w += kT) dst[w] = src[w];
        src = reinterpret_cast<const uint32_t*>(ops);
        dst = reinterpret_cast<uint32_t*>(sops);
        for (uint32_t w = threadIdx.x; w < p.n_ops * (sizeof(RegOp) / 4); w += kT) dst[w] = src[w];
        src = reinterpret_cast<const uint32_t*>(layouts);
        dst = reinterpret_cast<uint32_t*>(slay);
        for (uint32_t w = threadIdx.x; w < p.n_layouts * (sizeof(RegLayout) / 4); w += kT)
            dst[w] = src[w];
    }
    __syncthreads();
    {
        const uint32_t last = p.last_layout;
        s_ldg[threadIdx.x] = thread_goff(slay[0], kTB, gbit);
        s_stg[threadIdx.x] = thread_goff(slay[last], kTB, stbit);
        for (uint32_t l = 0; l < p.n_layouts && l < kRegSlotLayouts; ++l)
            s_tslot[l * kT + threadIdx.x] = static_cast<uint16_t>(thread_slot(slay[l], kTB));
        if (threadIdx.x < kRegBits) {
            s_ldr[threadIdx.x] = gbit[slay[0].rpos[threadIdx.x]];
            s_str[threadIdx.x] = stbit[slay[last].rpos[threadIdx.x]];
        }
    }
    __syncthreads();
    const bool slot_table = p.n_layouts <= kRegSlotLayouts;   // uniform
    const uint32_t smat_addr = static_cast<uint32_t>(__cvta_generic_to_shared(smat));
    const uint32_t sdyn_addr = static_cast<uint32_t>(__cvta_generic_to_shared(sdyn));
    double2* __restrict__ s = st + static_cast<uint64_t>(blockIdx.y) * p.batch_stride;
    uint32_t parity = 0;
    for (uint64_t tid = blockIdx.x; tid < p.n_tiles; tid += gridDim.x, parity ^= 1u) {
        // a warp's shared-memory slots differ between layouts with different warp bits:
        // the previous tile's last remap must be done before this tile's first
        if (p.sync_tiles) __syncthreads();
        uint64_t base = tid << p.L;
        for (uint32_t i = 0; i < p.h; ++i) base = insert_zero_bit(base, shbits[i]);
        double2 v[kE];
        {
            const uint64_t g = base | s_ldg[threadIdx.x];
            const uint64_t g0 = s_ldr[0], g1 = s_ldr[1], g2 = s_ldr[2], g3 = s_ldr[3];
#pragma unroll
            for (int u = 0; u < kE; ++u)
                v[u] = __ldcs(s + (g | ((u & 1) ? g0 : 0) | ((u & 2) ? g1 : 0) | ((u & 4) ? g2 : 0) |
                                   ((u & 8) ? g3 : 0)));
        }
        // relabelled stores go to places other warps load: all loads before any store
        if (p.load_barrier) __syncthreads();
        // Start the HBM reads of this CTA's next tile into L2 while this one computes, so
        // its loads above hit L2 on the next iteration.  Thread r < 2^h takes the row of
        // high-bit pattern r: 2^L contiguous amplitudes, 16 B * 2^L from a 16 B boundary.
        if (threadIdx.x < (1u << p.h) && tid + gridDim.x < p.n_tiles) {
            uint64_t nb = (tid + gridDim.x) << p.L;
            for (uint32_t i = 0; i < p.h; ++i) {
                nb = insert_zero_bit(nb, shbits[i]);
                if ((threadIdx.x >> i) & 1u) nb |= uint64_t{1} << shbits[i];
            }
            const double2* row = s + nb;
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(row), "r"(16u << p.L)
                         : "memory");
        }
        // Per-tile diagonals: entry e of table d is its base entry times every gated term
        // whose out-of-tile qubits are all 1 in this tile and whose entry bits e contains.
        // The barrier after the build also ends the use of the other parity's tables (every
        // warp has finished the previous tile), so the next tile may overwrite them.
        const uint32_t dyn_base = parity * p.dyn_entries;
        if (p.n_dyn) {
            for (uint32_t w = threadIdx.x; w < p.n_dyn * 64u; w += kT) {
                const RegOp& op = sops[sdynrec[w >> 6]];
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
                sdyn[dyn_base + op.dyn_off + e] = acc;
            }
            __syncthreads();
        }
        uint32_t cur = 0;
        for (uint32_t o = 0; o < p.n_ops; ++o) {
            const RegOp& op = sops[o];
            if ((base & op.gcmask) != op.gcmask) continue;   // uniform across the CTA
            const uint32_t kind = op.kind;
            if (kind == kRegRemap) {
                {
                    const RegLayout& ly = slay[cur];
                    const uint32_t ts = slot_table ? s_tslot[cur * kT + threadIdx.x]
                                                   : thread_slot(ly, kTB);
                    const uint32_t r0 = ly.rsw[0], r1 = ly.rsw[1], r2 = ly.rsw[2], r3 = ly.rsw[3];
#pragma unroll
                    for (int u = 0; u < kE; ++u)
                        tile[ts ^ ((u & 1) ? r0 : 0) ^ ((u & 2) ? r1 : 0) ^ ((u & 4) ? r2 : 0) ^
                             ((u & 8) ? r3 : 0)] = v[u];
                }
                cur = op.code;
                const bool local = op.k != 0;   // uniform: warp bits unchanged
                if (local) __syncwarp();
                else __syncthreads();
                {
                    const RegLayout& ly = slay[cur];
                    const uint32_t ts = slot_table ? s_tslot[cur * kT + threadIdx.x]
                                                   : thread_slot(ly, kTB);
                    const uint32_t r0 = ly.rsw[0], r1 = ly.rsw[1], r2 = ly.rsw[2], r3 = ly.rsw[3];
#pragma unroll
                    for (int u = 0; u < kE; ++u)
                        v[u] = tile[ts ^ ((u & 1) ? r0 : 0) ^ ((u & 2) ? r1 : 0) ^
                                    ((u & 4) ? r2 : 0) ^ ((u & 8) ? r3 : 0)];
                }
                if (local) __syncwarp();
                else __syncthreads();
                continue;
            }
            const uint32_t tc = op.tcmask;
            uint32_t moff = op.mat_off;
            if (const uint32_t nsel = op.nsel) {   // matrix picked by the tile's selector bits
                uint32_t sel = 0;
                for (uint32_t i = 0; i < nsel; ++i)
                    sel |= static_cast<uint32_t>((base >> op.selq[i]) & 1u) << i;
                const uint32_t k2 = kind == kRegDense || kind == kRegMma ? 2u * op.k : op.k;
                moff += sel << k2;
            }
            if (kind == kRegMma) {
                if constexpr (MMA) {
                    // controls on warp bits only: the condition is the same on every lane
                    if ((threadIdx.x & tc & ~31u) != (tc & ~31u)) continue;
                    __syncwarp();
                    reg_mma(v, smat_addr + 16u * moff, op.rcmask);
                }
                continue;
            }
            if (kind == kRegPauli) {   // rcmask / tcmask: its Z-type bits, not controls
                if constexpr (PAULI)
                    reg_pauli(v, smat_addr + 16u * moff, op.code, op.rcmask, tc, op.loc[0], base);
                continue;
            }
            if ((threadIdx.x & tc) != tc) continue;
            const uint32_t rc = op.rcmask;
            const uint32_t mat = kind == kRegDiagDyn ? sdyn_addr + 16u * (dyn_base + op.dyn_off)
                                                     : smat_addr + 16u * moff;
            if (kind == kRegDense) {
                if constexpr (FMAD) dispatch_dense(v, op.code, SharedMat{mat}, rc);
            } else if (kind == kRegPhase) {
                const double2 f = lds2(mat);
#pragma unroll
                for (int u = 0; u < kE; ++u)
                    if ((u & rc) == rc) v[u] = cmul(f, v[u]);
            } else if (kind == kRegSwapX) {
                dispatch_swapx(v, op.code, rc);
            } else {
                reg_diag(v, op, SharedMat{mat}, rc);
            }
        }
        {
            const uint64_t g = base | s_stg[threadIdx.x];
            const uint64_t g0 = s_str[0], g1 = s_str[1], g2 = s_str[2], g3 = s_str[3];
#pragma unroll
            for (int u = 0; u < kE; ++u)
                __stcs(s + (g | ((u & 1) ? g0 : 0) | ((u & 2) ? g1 : 0) | ((u & 4) ? g2 : 0) |
                            ((u & 8) ? g3 : 0)),
                       v[u]);
        }
    }
}

// ------------------------------------------------------------------ double-buffered passes
//
// The same pass with the next tile's HBM read overlapped with this tile's compute: each
// thread issues cp.async copies of 16 of the next tile's amplitudes into the second of two
// shared tile buffers while the CTA works on the first, and waits for them only when it
// reaches that tile.  The tile arrives in shared memory in linear order (position q of the
// tile at index q; thread t copies positions j * T + t, so a warp's copy is one coalesced
// 512-byte row), is read into registers through layout 0, and the same buffer then serves
// the remaps (swizzled slots).  One barrier per tile makes the copies visible, ends every
// warp's use of the previous tile's buffer (which the next copies overwrite) and publishes
// the per-tile diagonal tables.

__device__ __forceinline__ void cp_async16(uint32_t saddr, const void* g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

template <int M, int MINB>
__global__ void __launch_bounds__(1 << (M - kRegBits), MINB)
k_regtile_pipe(double2* __restrict__ st, RegPass p, const RegOp* __restrict__ ops,
               const RegLayout* __restrict__ layouts, const double2* __restrict__ mats) {
    constexpr uint32_t kT = 1u << (M - kRegBits);
    constexpr uint32_t kTB = M - kRegBits;
    constexpr uint32_t kN = 1u << M;
    extern __shared__ __align__(16) unsigned char smem[];
    double2* bufs = reinterpret_cast<double2*>(smem);   // two tiles
    double2* smat = bufs + 2 * kN;
    RegOp* sops = reinterpret_cast<RegOp*>(smat + p.n_mat);
    RegLayout* slay = reinterpret_cast<RegLayout*>(sops + p.n_ops);
    double2* sdyn = reinterpret_cast<double2*>(
        (reinterpret_cast<uintptr_t>(slay + p.n_layouts) + 15u) & ~uintptr_t{15});
    __shared__ uint64_t gbit[kRegMaxBits];
    __shared__ uint64_t sgbit[kRegMaxBits];
    __shared__ uint32_t shbits[kTileMaxHigh];
    __shared__ uint32_t sdynrec[kRegMaxDyn];
    // per-thread constants of every tile, computed once: the global offsets of the thread
    // bits at the load (layout 0) and at the store (the last layout), and each layout's
    // shared-memory slot of the thread (the first kRegSlotLayouts layouts); the register
    // bits' offsets are the same for every thread
    __shared__ uint64_t s_ldg[kT], s_stg[kT];
    __shared__ uint64_t s_ldr[kRegBits], s_str[kRegBits];
    __shared__ uint16_t s_tslot[kRegSlotLayouts * kT];
    if (threadIdx.x == 0) {
#pragma unroll
        for (uint32_t i = 0; i < kTileMaxHigh; ++i) shbits[i] = p.hbits[i];
#pragma unroll
        for (uint32_t i = 0; i < kRegMaxDyn; ++i) sdynrec[i] = p.dyn_rec[i];
        for (uint32_t b = 0; b < M; ++b)
            gbit[b] = uint64_t{1} << (b < p.L ? b : shbits[b - p.L]);
        if (p.relabel) {
#pragma unroll
            for (uint32_t b = 0; b < kRegMaxBits; ++b)
                if (b < M) sgbit[b] = uint64_t{1} << p.store_qubit[b];
        }
    }
    const uint64_t* __restrict__ stbit = p.relabel ? sgbit : gbit;
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(
            mats + static_cast<uint64_t>(blockIdx.y) * p.mat_stride);
        uint32_t* dst = reinterpret_cast<uint32_t*>(smat);
        for (uint32_t w = threadIdx.x; w < p.n_mat * 4u; w += kT) dst[w] = src[w];
        src = reinterpret_cast<const uint32_t*>(ops);
        dst = reinterpret_cast<uint32_t*>(sops);
        for (uint32_t w = threadIdx.x; w < p.n_ops * (sizeof(RegOp) / 4); w += kT) dst[w] = src[w];
        src = reinterpret_cast<const uint32_t*>(layouts);
        dst = reinterpret_cast<uint32_t*>(slay);
        for (uint32_t w = threadIdx.x; w < p.n_layouts * (sizeof(RegLayout) / 4); w += kT)
            dst[w] = src[w];
    }
    __syncthreads();
    {
        const uint32_t last = p.last_layout;
        s_ldg[threadIdx.x] = thread_goff(slay[0], kTB, gbit);
        s_stg[threadIdx.x] = thread_goff(slay[last], kTB, stbit);
        for (uint32_t l = 0; l < p.n_layouts && l < kRegSlotLayouts; ++l)
            s_tslot[l * kT + threadIdx.x] = static_cast<uint16_t>(thread_slot(slay[l], kTB));
        if (threadIdx.x < kRegBits) {
            s_ldr[threadIdx.x] = gbit[slay[0].rpos[threadIdx.x]];
            s_str[threadIdx.x] = stbit[slay[last].rpos[threadIdx.x]];
        }
    }
    __syncthreads();
    const bool slot_table = p.n_layouts <= kRegSlotLayouts;   // uniform
    const uint32_t smat_addr = static_cast<uint32_t>(__cvta_generic_to_shared(smat));
    const uint32_t sdyn_addr = static_cast<uint32_t>(__cvta_generic_to_shared(sdyn));
    const uint32_t bufs_addr = static_cast<uint32_t>(__cvta_generic_to_shared(bufs));
    double2* __restrict__ s = st + static_cast<uint64_t>(blockIdx.y) * p.batch_stride;
    // copy positions q = j * kT + t: tile bits 0..kTB-1 from t, the 4 above from j
    uint64_t toff = 0;
    for (uint32_t b = 0; b < kTB; ++b)
        if ((threadIdx.x >> b) & 1u) toff |= gbit[b];
    const uint64_t jb0 = gbit[kTB], jb1 = gbit[kTB + 1], jb2 = gbit[kTB + 2], jb3 = gbit[kTB + 3];
    auto tile_base = [&](uint64_t tile) {
        uint64_t b = tile << p.L;
        for (uint32_t i = 0; i < p.h; ++i) b = insert_zero_bit(b, shbits[i]);
        return b;
    };
    auto issue = [&](uint64_t tile, uint32_t which) {
        const uint64_t g = tile_base(tile) | toff;
        const uint32_t dst = bufs_addr + 16u * (which * kN + threadIdx.x);
#pragma unroll
        for (int j = 0; j < kE; ++j)
            cp_async16(dst + 16u * kT * j, s + (g | ((j & 1) ? jb0 : 0) | ((j & 2) ? jb1 : 0) |
                                               ((j & 4) ? jb2 : 0) | ((j & 8) ? jb3 : 0)));
        cp_async_commit();
    };
    if (blockIdx.x < p.n_tiles) issue(blockIdx.x, 0);
    uint32_t parity = 0;
    for (uint64_t tid = blockIdx.x; tid < p.n_tiles; tid += gridDim.x, parity ^= 1u) {
        const uint64_t base = tile_base(tid);
        // this tile's diagonal tables: their parity's previous user (two tiles back) is done,
        // since every warp passed the previous tile's barrier
        const uint32_t dyn_base = parity * p.dyn_entries;
        if (p.n_dyn) {
            for (uint32_t w = threadIdx.x; w < p.n_dyn * 64u; w += kT) {
                const RegOp& op = sops[sdynrec[w >> 6]];
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
                sdyn[dyn_base + op.dyn_off + e] = acc;
            }
        }
        cp_async_wait_all();
        __syncthreads();
        if (tid + gridDim.x < p.n_tiles) issue(tid + gridDim.x, parity ^ 1u);
        double2* __restrict__ tile = bufs + parity * kN;
        double2 v[kE];
        {
            const RegLayout& ly = slay[0];
            uint32_t tp = 0;
            for (uint32_t i = 0; i < kTB; ++i)
                if ((threadIdx.x >> i) & 1u) tp |= 1u << ly.tpos[i];
            const uint32_t p0 = 1u << ly.rpos[0], p1 = 1u << ly.rpos[1], p2 = 1u << ly.rpos[2],
                           p3 = 1u << ly.rpos[3];
#pragma unroll
            for (int u = 0; u < kE; ++u)
                v[u] = tile[tp | ((u & 1) ? p0 : 0) | ((u & 2) ? p1 : 0) | ((u & 4) ? p2 : 0) |
                            ((u & 8) ? p3 : 0)];
        }
        __syncwarp();   // every lane's linear read before any lane's first remap write
        uint32_t cur = 0;
        for (uint32_t o = 0; o < p.n_ops; ++o) {
            const RegOp& op = sops[o];
            if ((base & op.gcmask) != op.gcmask) continue;
            const uint32_t kind = op.kind;
            if (kind == kRegRemap) {
                {
                    const RegLayout& ly = slay[cur];
                    const uint32_t ts = slot_table ? s_tslot[cur * kT + threadIdx.x]
                                                   : thread_slot(ly, kTB);
                    const uint32_t r0 = ly.rsw[0], r1 = ly.rsw[1], r2 = ly.rsw[2], r3 = ly.rsw[3];
#pragma unroll
                    for (int u = 0; u < kE; ++u)
                        tile[ts ^ ((u & 1) ? r0 : 0) ^ ((u & 2) ? r1 : 0) ^ ((u & 4) ? r2 : 0) ^
                             ((u & 8) ? r3 : 0)] = v[u];
                }
                cur = op.code;
                const bool local = op.k != 0;
                if (local) __syncwarp();
                else __syncthreads();
                {
                    const RegLayout& ly = slay[cur];
                    const uint32_t ts = slot_table ? s_tslot[cur * kT + threadIdx.x]
                                                   : thread_slot(ly, kTB);
                    const uint32_t r0 = ly.rsw[0], r1 = ly.rsw[1], r2 = ly.rsw[2], r3 = ly.rsw[3];
#pragma unroll
                    for (int u = 0; u < kE; ++u)
                        v[u] = tile[ts ^ ((u & 1) ? r0 : 0) ^ ((u & 2) ? r1 : 0) ^
                                    ((u & 4) ? r2 : 0) ^ ((u & 8) ? r3 : 0)];
                }
                if (local) __syncwarp();
                else __syncthreads();
                continue;
            }
            const uint32_t tc = op.tcmask;
            uint32_t moff = op.mat_off;
            if (const uint32_t nsel = op.nsel) {
                uint32_t sel = 0;
                for (uint32_t i = 0; i < nsel; ++i)
                    sel |= static_cast<uint32_t>((base >> op.selq[i]) & 1u) << i;
                const uint32_t k2 = kind == kRegDense || kind == kRegMma ? 2u * op.k : op.k;
                moff += sel << k2;
            }
            if (kind == kRegMma) {
                if ((threadIdx.x & tc & ~31u) != (tc & ~31u)) continue;   // uniform per warp
                __syncwarp();
                reg_mma(v, smat_addr + 16u * moff, op.rcmask);
                continue;
            }
            if (kind == kRegPauli) {
                reg_pauli(v, smat_addr + 16u * moff, op.code, op.rcmask, tc, op.loc[0], base);
                continue;
            }
            if ((threadIdx.x & tc) != tc) continue;
            const uint32_t rc = op.rcmask;
            const uint32_t mat = kind == kRegDiagDyn ? sdyn_addr + 16u * (dyn_base + op.dyn_off)
                                                     : smat_addr + 16u * moff;
            if (kind == kRegDense) {
                dispatch_dense(v, op.code, SharedMat{mat}, rc);
            } else if (kind == kRegPhase) {
                const double2 f = lds2(mat);
#pragma unroll
                for (int u = 0; u < kE; ++u)
                    if ((u & rc) == rc) v[u] = cmul(f, v[u]);
            } else if (kind == kRegSwapX) {
                dispatch_swapx(v, op.code, rc);
            } else {
                reg_diag(v, op, SharedMat{mat}, rc);
            }
        }
        {
            const uint64_t g = base | s_stg[threadIdx.x];
            const uint64_t g0 = s_str[0], g1 = s_str[1], g2 = s_str[2], g3 = s_str[3];
#pragma unroll
            for (int u = 0; u < kE; ++u)
                __stcs(s + (g | ((u & 1) ? g0 : 0) | ((u & 2) ? g1 : 0) | ((u & 4) ? g2 : 0) |
                            ((u & 8) ? g3 : 0)),
                       v[u]);
        }
    }
    cp_async_wait_all();
}

template <int M, int MINB>
void launch_pipe(const LaunchCtx& ctx, double2* st, uint32_t batch, const RegPass& p, size_t smem,
                 const RegOp* d_ops, const RegLayout* d_layouts, const double2* d_mats) {
    constexpr uint32_t kT = 1u << (M - kRegBits);
    auto kern = k_regtile_pipe<M, MINB>;
    cuda_check_launch_attr(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                static_cast<int>(kRegPipeMaxSmem)));
    const uint32_t by_smem = static_cast<uint32_t>(std::max<size_t>(1, (227 * 1024) / (smem + 1024)));
    const uint64_t want = static_cast<uint64_t>(ctx.num_sms) * std::min<uint32_t>(MINB, by_smem);
    const uint32_t grid = static_cast<uint32_t>(std::max<uint64_t>(1, std::min<uint64_t>(want, p.n_tiles)));
    kern<<<dim3(grid, batch), kT, smem, ctx.stream>>>(st, p, d_ops, d_layouts, d_mats);
    check_launch("register tile pass (double-buffered)");
}

template <int M, int MINB, bool FMAD, bool MMA, bool PAULI>
void launch_mbf(const LaunchCtx& ctx, double2* st, uint32_t batch, const RegPass& p, size_t smem,
                const RegOp* d_ops, const RegLayout* d_layouts, const double2* d_mats) {
    constexpr uint32_t kT = 1u << (M - kRegBits);
    auto kern = k_regtile<M, MINB, FMAD, MMA, PAULI>;
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
    kern<<<dim3(grid, batch), kT, smem, ctx.stream>>>(st, p, d_ops, d_layouts, d_mats);
    check_launch("register tile pass");
}

template <int M, int MINB>
void launch_mb(const LaunchCtx& ctx, double2* st, uint32_t batch, const RegPass& p, size_t smem,
               const RegOp* d_ops, const RegLayout* d_layouts, const double2* d_mats) {
    // four variants: FMA, FMA + Pauli, tensor path, all
    if (!p.mma_ops) {
        if (p.pauli_ops) launch_mbf<M, MINB, true, false, true>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
        else launch_mbf<M, MINB, true, false, false>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
    } else if (!p.fma_dense && !p.pauli_ops) {
        launch_mbf<M, MINB, false, true, false>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
    } else {
        launch_mbf<M, MINB, true, true, true>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
    }
}

// Residency per tile size: about 160 registers per thread keep the dense paths free of
// spills, so M <= 11 run 168-register CTAs (12 warps per SM).  M = 12 runs two CTAs of 128
// registers (a few spilled values; measured faster than one 160-register CTA, which
// LQCS_TILE_OCC=1 selects); M = 13 (512 threads) is capped at 128.
template <int M>
void launch_m(const LaunchCtx& ctx, double2* st, uint32_t batch, const RegPass& p, size_t smem,
              const RegOp* d_ops, const RegLayout* d_layouts, const double2* d_mats) {
    if constexpr (M == 12) {
        static const int occ = [] {
            const char* e = std::getenv("LQCS_TILE_OCC");
            return e ? std::atoi(e) : 2;
        }();
        if (occ >= 2) {
            launch_mb<12, 2>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
            return;
        }
        launch_mb<12, 1>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
    } else if constexpr (M == 13) {
        launch_mb<13, 1>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
    } else if constexpr (M == 11) {
        // three 168-register CTAs per SM by default; LQCS_TILE_OCC=4: four of 128 registers
        static const int occ = [] {
            const char* e = std::getenv("LQCS_TILE_OCC");
            return e ? std::atoi(e) : 3;
        }();
        if (occ >= 4) {
            launch_mb<11, 4>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
            return;
        }
        launch_mb<11, 3>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
    } else {
        constexpr int kMinB = 65536 / ((1 << (M - kRegBits)) * 168);
        launch_mb<M, kMinB>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats);
    }
}

}  // namespace

size_t reg_smem_bytes(const RegPass& pass, uint32_t tiles) {
    const size_t records = sizeof(double2) * ((size_t{tiles} << pass.m) + pass.n_mat) +
                           sizeof(RegOp) * pass.n_ops + sizeof(RegLayout) * pass.n_layouts;
    return pass.n_dyn ? ((records + 15) & ~size_t{15}) + sizeof(double2) * 2 * pass.dyn_entries
                      : records;
}

bool reg_pipe_enabled() {
    static const bool on = [] {
        const char* e = std::getenv("LQCS_REG_PIPE");
        return e != nullptr && std::atoi(e) != 0;
    }();
    return on;
}

void launch_reg_pass(const LaunchCtx& ctx, double2* st, uint32_t n, uint32_t batch,
                     const RegPass& pass, const RegOp* d_ops, const RegLayout* d_layouts,
                     const double2* d_mats) {
    RegPass p = pass;
    p.batch_stride = uint64_t{1} << n;
    p.n_tiles = (uint64_t{1} << n) >> p.m;
    if (p.rot) throw std::logic_error("register tile pass: a pass in rotation form");
    if (!d_layouts || (p.n_ops && !d_ops) || (p.n_mat && !d_mats))
        throw std::logic_error("register tile pass: a table is not on the device");
    if (reg_pipe_enabled() && (p.m == 11 || p.m == 12)) {
        const size_t smem2 = reg_smem_bytes(p, 2);
        if (smem2 <= kRegPipeMaxSmem && p.n_ops <= kRegMaxRecords && p.n_mat <= kRegMaxMatrix &&
            p.n_dyn <= kRegMaxDyn && p.dyn_entries <= kRegMaxDynEntries && p.n_layouts >= 1 &&
            p.h <= kTileMaxHigh) {
            if (p.m == 12) launch_pipe<12, 1>(ctx, st, batch, p, smem2, d_ops, d_layouts, d_mats);
            else launch_pipe<11, 3>(ctx, st, batch, p, smem2, d_ops, d_layouts, d_mats);
            return;
        }
    }
    const size_t smem = reg_smem_bytes(p);
    if (smem > kTileMaxSmem || p.m < kRegMinBits || p.m > kRegMaxBits || p.h > kTileMaxHigh ||
        p.n_layouts < 1 || p.n_ops > kRegMaxRecords || p.n_mat > kRegMaxMatrix ||
        p.n_dyn > kRegMaxDyn || p.dyn_entries > kRegMaxDynEntries)
        throw std::logic_error("register tile pass: unsupported shape");
    switch (p.m) {
        case 9: launch_m<9>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats); break;
        case 10: launch_m<10>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats); break;
        case 11: launch_m<11>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats); break;
        case 12: launch_m<12>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats); break;
        default: launch_m<13>(ctx, st, batch, p, smem, d_ops, d_layouts, d_mats); break;
    }
}

}  // namespace lqcs_b200
