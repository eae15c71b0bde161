// engine.cpp — device runtime: state handles, programs, run paths, expectations.
#include "engine.hpp"

#include "adj_pass.cuh"
#include "block_pool.hpp"
#include "costmodel.hpp"

#include <algorithm>
#include <deque>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <numbers>
#include <optional>
#include <string>

namespace lqcs_b200 {

void cuda_check(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return;
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        throw Error(LQCS_ERR_OUT_OF_MEMORY, std::string(what) + ": " + cudaGetErrorString(e));
    }
    throw Error(LQCS_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

namespace {

// The pool's CUDA calls.  None leaves its error in the thread's last-error slot, which the next
// launch check reads.
struct CudaBlocks {
    struct Current {   // the calling thread's device, put back at the end
        int cur = 0;
        explicit Current(int device) {
            if (cudaGetDevice(&cur) != cudaSuccess) cudaGetLastError();
            if (cur != device && cudaSetDevice(device) != cudaSuccess) cudaGetLastError();
        }
        ~Current() { cudaSetDevice(cur); }
    };
    static void* allocate(int device, size_t bytes) {
        Current on(device);
        void* p = nullptr;
        const cudaError_t e = cudaMalloc(&p, bytes);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            return nullptr;
        }
        cuda_check(e, "cudaMalloc");
        return p;
    }
    static bool free(int device, void* p) {
        Current on(device);
        if (cudaFree(p) == cudaSuccess) return true;
        cudaGetLastError();
        return false;
    }
    // Waits for the stream's work.  False where that is not possible: the stream (or one that the
    // default stream would wait for) is being captured, or the device has failed.
    static bool wait(int device, cudaStream_t stream) {
        Current on(device);
        cudaStreamCaptureStatus c = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(stream, &c) == cudaSuccess &&
            (c != cudaStreamCaptureStatusNone || cudaStreamSynchronize(stream) == cudaSuccess))
            return c == cudaStreamCaptureStatusNone;
        cudaGetLastError();
        return false;
    }
};

BlockPool<CudaBlocks>& blocks() {   // never destroyed: buffers may be freed during process exit
    static auto* p = new BlockPool<CudaBlocks>;
    return *p;
}

}  // namespace

void clear_buffer_pool(bool retire) { blocks().clear(retire); }

void DeviceBuffer::release() {
    if (ptr) release(bytes <= kBlockMax && CudaBlocks::wait(device, stream));
}

void DeviceBuffer::release(bool idle) {
    if (!ptr) return;
    void* p = ptr;
    const size_t b = bytes;
    ptr = nullptr;
    bytes = 0;
    blocks().give(device, p, b, era, idle);
}

void DeviceBuffer::ensure(size_t b) {
    if (b <= bytes) return;
    release();
    cuda_check(cudaGetDevice(&device), "cudaGetDevice");
    ptr = blocks().take(device, b, era);
    if (!ptr) cuda_check(cudaErrorMemoryAllocation, "cudaMalloc");
    bytes = capacity(b);
}

int device_sm_count() {
    static std::mutex mu;
    static std::map<int, int> cache;
    int dev = 0;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    std::lock_guard<std::mutex> lk(mu);
    auto it = cache.find(dev);
    if (it != cache.end()) return it->second;
    int sms = 0;
    cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev),
               "cudaDeviceGetAttribute");
    cache[dev] = sms;
    return sms;
}

LaunchCtx make_ctx(cudaStream_t s) {
    LaunchCtx c;
    c.stream = s;
    c.num_sms = device_sm_count();
    return c;
}

uint32_t default_fusion_width() {
    if (const char* e = std::getenv("LQCS_FUSION_WIDTH")) {
        const int v = std::atoi(e);
        if (v >= 1 && v <= kMaxDense) return static_cast<uint32_t>(v);
    }
    return 4;
}

// ------------------------------------------------------------------ programs

static double2 to_d2(cd z) { return make_double2(z.real(), z.imag()); }

void Program::build(std::vector<DevOp> ops_in, cudaStream_t stream) {
    ops = std::move(ops_in);
    std::vector<double2> mats;
    std::vector<uint32_t> u32;
    mat_off.assign(ops.size(), 0);
    cyc_off.assign(ops.size(), 0);
    len_off.assign(ops.size(), 0);
    for (size_t i = 0; i < ops.size(); ++i) {
        const DevOp& op = ops[i];
        source_gates += op.src_gates;
        if (op.kind == OpKind::DENSE || op.kind == OpKind::DIAG) {
            mat_off[i] = mats.size();
            for (const cd& z : op.mat) mats.push_back(to_d2(z));
        } else if (op.kind == OpKind::PERM) {
            cyc_off[i] = u32.size();
            u32.insert(u32.end(), op.cycles.begin(), op.cycles.end());
            len_off[i] = u32.size();
            u32.insert(u32.end(), op.cycle_len.begin(), op.cycle_len.end());
        }
    }
    if (!mats.empty()) {
        d_mats.ensure(mats.size() * sizeof(double2));
        cuda_check(cudaMemcpyAsync(d_mats.ptr, mats.data(), mats.size() * sizeof(double2),
                                   cudaMemcpyHostToDevice, stream),
                   "upload matrices");
    }
    if (!u32.empty()) {
        d_u32.ensure(u32.size() * sizeof(uint32_t));
        cuda_check(cudaMemcpyAsync(d_u32.ptr, u32.data(), u32.size() * sizeof(uint32_t),
                                   cudaMemcpyHostToDevice, stream),
                   "upload permutation cycles");
    }
    std::vector<double2> tmats;
    for (const cd& z : tile_mats) tmats.push_back(to_d2(z));
    if (!tile_ops.empty()) {
        d_tile_ops.ensure(tile_ops.size() * sizeof(TileOp));
        cuda_check(cudaMemcpyAsync(d_tile_ops.ptr, tile_ops.data(), tile_ops.size() * sizeof(TileOp),
                                   cudaMemcpyHostToDevice, stream),
                   "upload tile operations");
    }
    if (!tmats.empty()) {
        d_tile_mats.ensure(tmats.size() * sizeof(double2));
        cuda_check(cudaMemcpyAsync(d_tile_mats.ptr, tmats.data(), tmats.size() * sizeof(double2),
                                   cudaMemcpyHostToDevice, stream),
                   "upload tile matrices");
    }
    // (the records of passes in rotation form are a kernel parameter)
    const bool reads_ops = std::any_of(reg_passes.begin(), reg_passes.end(),
                                       [](const RegPass& rp) { return !rp.rot; });
    if (reads_ops && !reg_ops.empty()) {
        d_reg_ops.ensure(reg_ops.size() * sizeof(RegOp));
        cuda_check(cudaMemcpyAsync(d_reg_ops.ptr, reg_ops.data(), reg_ops.size() * sizeof(RegOp),
                                   cudaMemcpyHostToDevice, stream),
                   "upload register pass records");
    }
    // (a pass may have no records: X gates alone negate bits at the store)
    if (!reg_layouts.empty()) {
        d_reg_layouts.ensure(reg_layouts.size() * sizeof(RegLayout));
        cuda_check(cudaMemcpyAsync(d_reg_layouts.ptr, reg_layouts.data(),
                                   reg_layouts.size() * sizeof(RegLayout), cudaMemcpyHostToDevice,
                                   stream),
                   "upload register layouts");
    }
    if (!reg_mats.empty()) {
        static_assert(sizeof(cd) == sizeof(double2), "uploaded as they are");
        d_reg_mats.ensure(reg_mats.size() * sizeof(double2));
        cuda_check(cudaMemcpyAsync(d_reg_mats.ptr, reg_mats.data(), reg_mats.size() * sizeof(double2),
                                   cudaMemcpyHostToDevice, stream),
                   "upload register pass matrices");
    }
    // the host vectors die with this scope: make sure the copies have consumed them
    cuda_check(cudaStreamSynchronize(stream), "program upload");
}

void Program::launch_op(size_t i, const LaunchCtx& ctx, double2* st, uint32_t n,
                        uint32_t batch) const {
    const DevOp& op = ops[i];
    switch (op.kind) {
        case OpKind::K1Q: {
            Apply1QOp a{};
            for (int e = 0; e < 4; ++e) a.m[e] = to_d2(op.m1[e]);
            a.t = op.targets[0];
            a.cmask = op.cmask;
            a.diag = op.diag1 ? 1 : 0;
            launch_apply_1q(ctx, st, n, batch, a);
            break;
        }
        case OpKind::PHASE:
            launch_phase(ctx, st, n, batch, op.phase_mask, to_d2(op.phase));
            break;
        case OpKind::DENSE:
            launch_dense(ctx, st, n, batch, op.targets.data(), op.k, op.cmask,
                         d_mats.as<double2>() + mat_off[i]);
            break;
        case OpKind::DIAG:
            launch_diag(ctx, st, n, batch, op.targets.data(), op.k, op.cmask,
                        d_mats.as<double2>() + mat_off[i]);
            break;
        case OpKind::PERM: {
            uint32_t total = 0;
            for (uint32_t l : op.cycle_len) total += l;
            launch_perm(ctx, st, n, batch, op.targets.data(), op.k, op.cmask,
                        d_u32.as<uint32_t>() + cyc_off[i], d_u32.as<uint32_t>() + len_off[i],
                        static_cast<uint32_t>(op.cycle_len.size()), total);
            break;
        }
        case OpKind::PAULI:
            launch_pauli_rotation(ctx, st, n, batch, op.x, op.zy, op.n_y, op.cos_h, op.sin_h);
            break;
        case OpKind::TILE:
            if (op.reg_tile && reg_passes[op.pass_index].rot) {
                launch_rot_pass(ctx, st, n, batch, reg_passes[op.pass_index],
                                reg_ops.data() + reg_op_off[op.pass_index],
                                d_reg_layouts.as<RegLayout>() + reg_lay_off[op.pass_index],
                                d_reg_mats.as<double2>() + reg_mat_off[op.pass_index]);
                break;
            }
            if (op.reg_tile) {
                launch_reg_pass(ctx, st, n, batch, reg_passes[op.pass_index],
                                d_reg_ops.as<RegOp>() + reg_op_off[op.pass_index],
                                d_reg_layouts.as<RegLayout>() + reg_lay_off[op.pass_index],
                                d_reg_mats.as<double2>() + reg_mat_off[op.pass_index]);
                break;
            }
            launch_tile_pass(ctx, st, n, batch, passes[op.pass_index],
                             d_tile_ops.as<TileOp>() + pass_op_off[op.pass_index],
                             d_tile_mats.as<double2>());
            break;
    }
}

void Program::launch(const LaunchCtx& ctx, double2* st, uint32_t n, uint32_t batch) const {
    for (size_t i = 0; i < ops.size(); ++i) launch_op(i, ctx, st, n, batch);
}

std::vector<FusedBlock> plan(const std::vector<GateDesc>& gates, uint32_t n,
                             const FusionConfig& fc) {
    const uint32_t w = fc.max_width ? fc.max_width : default_fusion_width();
    if (w < 1 || w > kMaxDense) invalid("fusion width must be in [1, 6]");
    // Barriers split the circuit into independently fused segments.
    std::vector<FusedBlock> out;
    std::vector<GateDesc> seg;
    std::vector<uint32_t> seg_idx;
    auto flush = [&]() {
        std::vector<FusedBlock> p = plan_greedy(seg, n, w);
        for (FusedBlock& b : p) {
            for (uint32_t& g : b.gates) g = seg_idx[g];
            out.push_back(std::move(b));
        }
        seg.clear();
        seg_idx.clear();
    };
    for (uint32_t i = 0; i < gates.size(); ++i) {
        if (gates[i].type == LQCS_GATE_BARRIER) {
            flush();
            continue;
        }
        if (!gates[i].is_unitary()) continue;
        seg.push_back(gates[i]);
        seg_idx.push_back(i);
    }
    flush();
    return out;
}

static bool use_tiles(uint32_t n, const FusionConfig& fc) {
    if (!fc.fuse) return false;
    if (fc.mode == kFuseTile) return n >= kTileMinBits;
    if (fc.mode == kFuseDefault) return n >= 12 && !std::getenv("LQCS_NO_TILES");
    return false;
}

// Host side of a tile-pass program (ops not yet uploaded).
static Program assemble_tiles(const std::vector<GateDesc>& source, uint32_t n,
                              const TileConfig& cfg, std::vector<DevOp>& ops) {
    Program p;
    const std::vector<GateDesc> gates = uses_rotation_form(cfg) ? rotation_form(source, n) : source;
    for (const PlanItem& it : plan_tiles(gates, n, cfg)) {
        if (!it.is_pass) {
            ops.push_back(lower_gate(gates[it.gate], n));
            ops.back().src_gates = source_gates(it, gates);
            continue;
        }
        DevOp op;
        op.kind = OpKind::TILE;
        op.k = static_cast<uint32_t>(it.hbits.size());
        op.targets = it.hbits;
        op.src_gates = source_gates(it, gates);
        op.alg_fraction = 1.0;
        if (cfg.reg) {
            RegPass rp;
            const size_t o0 = p.reg_ops.size(), l0 = p.reg_layouts.size(), m0 = p.reg_mats.size();
            if (lower_pass_reg(it, gates, cfg, rp, p.reg_ops, p.reg_layouts, p.reg_mats,
                               &op.tile_flops)) {
                p.reg_op_off.push_back(o0);
                p.reg_lay_off.push_back(l0);
                p.reg_mat_off.push_back(m0);
                op.reg_tile = true;
                op.pass_index = static_cast<uint32_t>(p.reg_passes.size());
                p.reg_passes.push_back(rp);
                ops.push_back(std::move(op));
                continue;
            }
        }
        // the shared-memory kernel: its operations have no native Pauli rotation, so the pass
        // splits at each (the rotation runs on its own, the gates between as passes)
        auto smem_pass = [&](const PlanItem& part) {
            DevOp sop = op;
            sop.src_gates = source_gates(part, gates);
            TilePass tp;
            p.pass_op_off.push_back(p.tile_ops.size());
            lower_pass(part, gates, cfg, tp, p.tile_ops, p.tile_mats, &sop.tile_flops);
            sop.pass_index = static_cast<uint32_t>(p.passes.size());
            p.passes.push_back(tp);
            ops.push_back(std::move(sop));
        };
        PlanItem part = it;
        part.gates.clear();
        for (uint32_t gi : it.gates) {
            if (!native_pauli(gates[gi], cfg)) {
                part.gates.push_back(gi);
                continue;
            }
            if (!part.gates.empty()) smem_pass(part);
            part.gates.clear();
            ops.push_back(lower_gate(gates[gi], n));
            ops.back().src_gates = gates[gi].src;
        }
        if (!part.gates.empty()) smem_pass(part);
    }
    if (ops.empty())   // products that are the identity
        for (const GateDesc& g : source) p.source_gates += g.is_unitary() ? 1 : 0;
    return p;
}

static std::vector<DevOp> dense_ops(const std::vector<GateDesc>& gates, uint32_t n, uint32_t width) {
    FusionConfig g;
    g.fuse = true;
    g.max_width = width;
    g.mode = kFuseGreedy;
    return lower_plan(plan(gates, n, g), gates, n);
}

bool compile_slots(const std::vector<GateDesc>& source, uint32_t n,
                   const std::vector<std::vector<std::array<cd, 4>>>& slots, cudaStream_t stream,
                   Program& out) {
    if (n < kRegMinBits) return false;
    const TileConfig cfg = default_tile_config(n);
    const std::vector<GateDesc> gates = uses_rotation_form(cfg) ? rotation_form(source, n) : source;
    Program p;
    std::vector<DevOp> ops;
    for (const PlanItem& it : plan_tiles(gates, n, cfg)) {
        if (!it.is_pass) {
            if (gates[it.gate].slot) return false;
            ops.push_back(lower_gate(gates[it.gate], n));
            continue;
        }
        bool has_slot = false;
        for (uint32_t gi : it.gates) has_slot |= gates[gi].slot;
        DevOp op;
        op.kind = OpKind::TILE;
        op.k = static_cast<uint32_t>(it.hbits.size());
        op.targets = it.hbits;
        op.src_gates = source_gates(it, gates);
        op.alg_fraction = 1.0;
        op.reg_tile = true;
        RegPass rp;
        const size_t o0 = p.reg_ops.size(), l0 = p.reg_layouts.size(), m0 = p.reg_mats.size();
        if (!lower_pass_reg(it, gates, cfg, rp, p.reg_ops, p.reg_layouts, p.reg_mats,
                            &op.tile_flops, has_slot ? &slots : nullptr))
            return false;
        p.reg_op_off.push_back(o0);
        p.reg_lay_off.push_back(l0);
        p.reg_mat_off.push_back(m0);
        op.pass_index = static_cast<uint32_t>(p.reg_passes.size());
        p.reg_passes.push_back(rp);
        ops.push_back(std::move(op));
    }
    p.build(std::move(ops), stream);
    out = std::move(p);
    return true;
}

// ------------------------------------------------------------------ autotuner

static std::vector<TuneCandidate> tune_candidates(uint32_t n) {
    std::vector<TuneCandidate> c;
    if (n >= kRegMinBits) {
        const uint32_t shapes[][3] = {{12, 5, 2}, {12, 5, 3}, {11, 5, 2}, {13, 5, 2}};
        for (const auto& s : shapes) {
            TuneCandidate t;
            t.cfg.m = std::min<uint32_t>(s[0], n);
            t.cfg.L = std::min<uint32_t>(s[1], t.cfg.m);
            t.cfg.inner = s[2];
            bool dup = false;
            for (const TuneCandidate& o : c)
                dup |= o.planner == 0 && o.cfg.m == t.cfg.m && o.cfg.inner == t.cfg.inner;
            if (!dup) c.push_back(t);
        }
        TuneCandidate smem;
        smem.planner = 1;
        smem.cfg.m = std::min<uint32_t>(12, n);
        smem.cfg.reg = false;
        c.push_back(smem);
    }
    for (uint32_t w = 2; w <= kMaxDense && w <= n; ++w) {
        if (n >= kRegMinBits && w < 4) continue;   // narrow greedy blocks never beat tile passes
        TuneCandidate t;
        t.planner = 2;
        t.width = w;
        c.push_back(t);
    }
    return c;
}

static Program compile_candidate(const std::vector<GateDesc>& gates, uint32_t n,
                                 const TuneCandidate& c, cudaStream_t stream) {
    std::vector<DevOp> ops;
    if (c.planner == 2) {
        Program p;
        p.build(dense_ops(gates, n, c.width), stream);
        return p;
    }
    Program p = assemble_tiles(gates, n, c.cfg, ops);
    p.build(std::move(ops), stream);
    return p;
}

// FNV-1a over the gate list: the cache key of a tuned circuit.
static uint64_t circuit_key(const std::vector<GateDesc>& gates, uint32_t n) {
    uint64_t h = 1469598103934665603ull;
    auto mix = [&](const void* p, size_t len) {
        const unsigned char* b = static_cast<const unsigned char*>(p);
        for (size_t i = 0; i < len; ++i) h = (h ^ b[i]) * 1099511628211ull;
    };
    mix(&n, sizeof n);
    for (const GateDesc& g : gates) {
        mix(&g.type, sizeof g.type);
        mix(&g.n_controls, sizeof g.n_controls);
        mix(g.qubits.data(), g.qubits.size() * sizeof(uint32_t));
        mix(g.params.data(), g.params.size() * sizeof(double));
        mix(g.mat.data(), g.mat.size() * sizeof(cd));
        mix(g.perm.data(), g.perm.size() * sizeof(uint64_t));
        mix(g.pauli.data(), g.pauli.size());
    }
    return h;
}

static std::mutex g_tune_mu;
// the learned planner's measured choices, per (circuit, cost-model weights)
static std::map<std::pair<uint64_t, uint64_t>, TuneCandidate> g_learned;
static std::map<uint64_t, TuneCandidate> g_tuned;

void clear_autotune_cache() {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tuned.clear();
    g_learned.clear();
}

// Device milliseconds of one application of each candidate plan on a scratch state (after
// one untimed application); empty when no scratch state fits in free memory.
static std::vector<double> time_candidates(const std::vector<GateDesc>& gates, uint32_t n,
                                           const std::vector<TuneCandidate>& cands,
                                           std::vector<uint64_t>* n_ops = nullptr) {
    std::vector<double> out;
    size_t free_b = 0, total_b = 0;
    cuda_check(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
    const double need = 16.0 * std::ldexp(1.0, static_cast<int>(n)) * 1.1 + (256u << 20);
    if (need > static_cast<double>(free_b)) return out;
    cudaStream_t s = nullptr;
    cuda_check(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking), "cudaStreamCreate");
    struct Guard {
        cudaStream_t s;
        cudaEvent_t a = nullptr, b = nullptr;
        ~Guard() {
            if (a) cudaEventDestroy(a);
            if (b) cudaEventDestroy(b);
            cudaStreamDestroy(s);
        }
    } guard{s};
    cuda_check(cudaEventCreate(&guard.a), "cudaEventCreate");
    cuda_check(cudaEventCreate(&guard.b), "cudaEventCreate");
    auto st = new_state(n, 1, s);
    for (const TuneCandidate& c : cands) {
        Program p = compile_candidate(gates, n, c, s);
        const StreamDrain drain{s};
        p.launch(st->ctx, st->d(), n, 1);   // untimed: first-launch set-up
        cuda_check(cudaEventRecord(guard.a, s), "cudaEventRecord");
        p.launch(st->ctx, st->d(), n, 1);
        cuda_check(cudaEventRecord(guard.b, s), "cudaEventRecord");
        cuda_check(cudaEventSynchronize(guard.b), "cudaEventSynchronize");
        float ms = 0.0f;
        cuda_check(cudaEventElapsedTime(&ms, guard.a, guard.b), "cudaEventElapsedTime");
        out.push_back(ms);
        if (n_ops) n_ops->push_back(p.ops.size());
    }
    return out;
}

std::vector<TuneTiming> autotune(const std::vector<GateDesc>& gates, uint32_t n, size_t* best) {
    const std::vector<TuneCandidate> cands = tune_candidates(n);
    std::vector<uint64_t> n_ops;
    const std::vector<double> ms = time_candidates(gates, n, cands, &n_ops);
    std::vector<TuneTiming> out;
    for (size_t i = 0; i < ms.size(); ++i) out.push_back({cands[i], n_ops[i], ms[i]});
    size_t b = 0;
    for (size_t i = 1; i < out.size(); ++i)
        if (out[i].ms < out[b].ms) b = i;
    if (best) *best = b;
    if (!out.empty()) {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_tuned[circuit_key(gates, n)] = out[b].cand;
    }
    return out;
}

// fusion_mode 5: the plan the autotuner measured fastest for this circuit (tuned now on a
// cache miss); the default plan when no scratch state fits.
static Program compile_autotuned(const std::vector<GateDesc>& gates, uint32_t n,
                                 const FusionConfig& fc, cudaStream_t stream) {
    const uint64_t key = circuit_key(gates, n);
    std::optional<TuneCandidate> c;
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        const auto it = g_tuned.find(key);
        if (it != g_tuned.end()) c = it->second;
    }
    if (!c) {
        size_t best = 0;
        const std::vector<TuneTiming> t = autotune(gates, n, &best);
        if (!t.empty()) c = t[best].cand;
    }
    if (!c) {
        FusionConfig d = fc;
        d.mode = kFuseDefault;
        return compile(gates, n, d, stream);
    }
    return compile_candidate(gates, n, *c, stream);
}

// Learned planning: every candidate plan (greedy dense blocks of width 1..6, tile passes of
// several shapes) is scored by the cost model's predicted device time, and the best few
// (two; LQCS_LEARNED_JUDGE sets how many, 1 = the model's choice alone) are then applied
// once on a scratch state with the default plan: measured wall time judges between the
// model's favourites and the default, which catches the model's ranking errors at a
// fraction of the autotuner's cost.  The choice is kept per
// circuit and set of weights.  Without trained weights the plain greedy plan is used.
static Program compile_learned(const std::vector<GateDesc>& gates, uint32_t n,
                               const FusionConfig& fc, cudaStream_t stream) {
    if (!costmodel_trained()) {
        Program p;
        p.build(dense_ops(gates, n, fc.max_width ? fc.max_width : default_fusion_width()), stream);
        return p;
    }
    const std::pair<uint64_t, uint64_t> key{circuit_key(gates, n), costmodel_version()};
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        const auto it = g_learned.find(key);
        if (it != g_learned.end()) return compile_candidate(gates, n, it->second, stream);
    }
    std::vector<std::pair<double, TuneCandidate>> scored;
    for (uint32_t w = 1; w <= kMaxDense && w <= n; ++w) {
        TuneCandidate t;
        t.planner = 2;
        t.width = w;
        scored.emplace_back(predict_ops_ms(dense_ops(gates, n, w), n), t);
    }
    if (n >= kTileMinBits) {
        const uint32_t shapes[][3] = {{11, 5, 2}, {12, 5, 2}, {12, 5, 3}, {13, 5, 2}, {13, 5, 3}};
        for (const auto& sh : shapes) {
            TuneCandidate t;
            t.cfg.m = std::min<uint32_t>(sh[0], n);
            t.cfg.L = std::min<uint32_t>(sh[1], t.cfg.m);
            t.cfg.inner = sh[2];
            std::vector<DevOp> ops;
            assemble_tiles(gates, n, t.cfg, ops);
            scored.emplace_back(predict_ops_ms(ops, n), t);
        }
    }
    std::stable_sort(scored.begin(), scored.end(),
                     [](const auto& a, const auto& b) { return a.first < b.first; });
    TuneCandidate pick = scored.front().second;
    const char* e = std::getenv("LQCS_LEARNED_JUDGE");
    const size_t judge = e ? static_cast<size_t>(std::max(1, std::atoi(e))) : 2;
    if (judge >= 2 && scored.size() >= 2) {
        std::vector<TuneCandidate> shortlist;
        for (size_t i = 0; i < std::min(judge, scored.size()); ++i) shortlist.push_back(scored[i].second);
        // and the default plan, so the judged choice is never slower than it
        if (n >= kTileMinBits) {
            TuneCandidate d;
            d.cfg = default_tile_config(n);
            bool have = false;
            for (const TuneCandidate& c : shortlist)
                have |= c.planner == 0 && c.cfg.m == d.cfg.m && c.cfg.L == d.cfg.L &&
                        c.cfg.inner == d.cfg.inner;
            if (!have) shortlist.push_back(d);
        }
        const std::vector<double> ms = time_candidates(gates, n, shortlist);
        if (!ms.empty())
            pick = shortlist[std::min_element(ms.begin(), ms.end()) - ms.begin()];
    }
    {
        std::lock_guard<std::mutex> lk(g_tune_mu);
        g_learned[key] = pick;
    }
    return compile_candidate(gates, n, pick, stream);
}

Program compile(const std::vector<GateDesc>& gates, uint32_t n, const FusionConfig& fc,
                cudaStream_t stream) {
    if (fc.fuse && fc.mode == kFuseLearned) return compile_learned(gates, n, fc, stream);
    if (fc.fuse && fc.mode == kFuseAutotune) return compile_autotuned(gates, n, fc, stream);
    std::vector<DevOp> ops;
    if (use_tiles(n, fc)) {
        Program p = assemble_tiles(gates, n, default_tile_config(n), ops);
        p.build(std::move(ops), stream);
        return p;
    }
    Program p;
    if (fc.fuse && fc.mode != kFuseNone) {
        ops = lower_plan(plan(gates, n, fc), gates, n);
    } else {
        for (const GateDesc& g : gates)
            if (g.is_unitary()) ops.push_back(lower_gate(g, n));
    }
    p.build(std::move(ops), stream);
    return p;
}

}  // namespace lqcs_b200

// ------------------------------------------------------------------ state handle

lqcs_state::~lqcs_state() { lqcs_b200::release_state(*this); }

double* lqcs_state::partials(size_t values) {
    const size_t need = (lqcs_b200::kMaxReduceBlocks + 1) * values * 2 * sizeof(double) + 4096;
    scratch.ensure(need);
    return scratch.as<double>();
}

void lqcs_state::sync() const {
    lqcs_b200::cuda_check(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
}

namespace lqcs_b200 {

double rng_uniform(Rng& r) {
    std::uniform_real_distribution<double> dist(0.0, 1.0);
    return dist(r);
}

Rng make_rng(const lqcs_sim_options* opts) {
    if (opts && opts->has_seed) return Rng(opts->seed);
    return Rng(std::random_device{}());
}

uint32_t max_qubits_on_device(uint32_t batch) {
    size_t free_b = 0, total_b = 0;
    cuda_check(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
    uint32_t q = 0;
    while (q < 40 && (uint64_t{16} << (q + 1)) * batch <= free_b) ++q;
    return q;
}

// Freed amplitude buffers of 32 MiB to 1 GiB (a 26-qubit state), kept for the next state of the
// same size on the same device: short runs (sampling loops, small circuits, trajectory
// batches of small states) skip cudaMalloc and cudaFree, which synchronise the device.  At
// most four buffers are kept; lqcs_release_caches frees them.
namespace {

struct PooledBuffer {
    int device;
    size_t bytes;
    void* ptr;
    uint64_t era;
};
// Never destroyed: states may be freed during process exit, after static destructors ran.
std::mutex& pool_mu() {
    static auto* m = new std::mutex;
    return *m;
}
std::vector<PooledBuffer>& pool() {   // oldest first
    static auto* p = new std::vector<PooledBuffer>;
    return *p;
}
constexpr size_t kPoolMaxBytes = size_t{1} << 30;
constexpr size_t kPoolEntries = 4;

// A kept buffer of this size for `b`; false if there is none.
bool pool_take(int device, size_t bytes, DeviceBuffer& b) {
    std::lock_guard<std::mutex> lk(pool_mu());
    for (auto it = pool().begin(); it != pool().end(); ++it) {
        if (it->device == device && it->bytes == bytes) {
            b.ptr = it->ptr;
            b.bytes = bytes;
            b.device = device;
            b.era = it->era;
            pool().erase(it);
            return true;
        }
    }
    return false;
}

}  // namespace

void clear_state_pool() {
    std::vector<PooledBuffer> drop;
    {
        std::lock_guard<std::mutex> lk(pool_mu());
        drop.swap(pool());
    }
    for (const PooledBuffer& b : drop) blocks().give(b.device, b.ptr, b.bytes, b.era, false);
}

// The amplitude buffer goes to the kept ones (smaller buffers are the block pool's).
static void keep_amplitudes(lqcs_state& st) {
    if (st.amps.bytes <= kBlockMax || st.amps.bytes > kPoolMaxBytes) return;
    if (st.amps.era != blocks().era()) return;   // allocated before lqcs_release_caches: not kept
    PooledBuffer evict{};
    {
        std::lock_guard<std::mutex> lk(pool_mu());
        if (pool().size() >= kPoolEntries) {
            evict = pool().front();
            pool().erase(pool().begin());
        }
        pool().push_back({st.device, st.amps.bytes, st.amps.ptr, st.amps.era});
    }
    st.amps.ptr = nullptr;
    st.amps.bytes = 0;
    if (evict.ptr) blocks().give(evict.device, evict.ptr, evict.bytes, evict.era, false);
}

void release_state(lqcs_state& st) {
    if (!st.amps.ptr && !st.scratch.ptr && !st.sample_scratch.ptr) return;
    // the buffers are reused only after this state's work on them has finished
    const bool idle = CudaBlocks::wait(st.device, st.stream);
    if (idle && st.amps.ptr) keep_amplitudes(st);
    for (DeviceBuffer* b : {&st.amps, &st.scratch, &st.sample_scratch}) b->release(idle);
}

std::unique_ptr<lqcs_state> new_state(uint32_t n, uint32_t batch, cudaStream_t stream) {
    if (n == 0) invalid("Statevector: num_qubits must be >= 1");
    if (batch == 0) invalid("state batch must be >= 1");
    auto too_large = [&](uint32_t cap) {
        const double gib = 16.0 * std::ldexp(1.0, static_cast<int>(n) - 30) * batch;
        invalid("Statevector: " + std::to_string(n) + " qubits would need " +
                std::to_string(gib) + " GiB (max " + std::to_string(cap) +
                " qubits on this device)");
    };
    // small states skip the query of free memory (it costs more than their kernels): the
    // allocation itself tells
    const bool small = n <= 40 && (static_cast<double>(batch) * std::ldexp(16.0, static_cast<int>(n))) <=
                                      static_cast<double>(kBlockMax);
    if (!small) {
        uint32_t cap = max_qubits_on_device(batch);
        if (n > cap && n <= 40) {   // once more without what lies idle
            clear_state_pool();
            clear_buffer_pool();
            cap = max_qubits_on_device(batch);
        }
        if (n > cap || n > 40) too_large(cap);
    }
    auto st = std::make_unique<lqcs_state>();
    cuda_check(cudaGetDevice(&st->device), "cudaGetDevice");
    st->n = n;
    st->batch = batch;
    st->stream = st->amps.stream = st->scratch.stream = st->sample_scratch.stream = stream;
    st->ctx = make_ctx(stream);
    const size_t bytes = sizeof(double2) * st->len() * batch;
    if (!pool_take(st->device, bytes, st->amps)) {
        try {
            st->amps.ensure(bytes);
        } catch (const Error& e) {
            if (!small || e.code != LQCS_ERR_OUT_OF_MEMORY) throw;
            too_large(max_qubits_on_device(batch));
        }
    }
    launch_set_basis(st->ctx, st->d(), n, batch, 0);
    return st;
}

// Compiled programs of the most recent circuits, so that running the same circuit again
// (a sampling loop, repeated run_statevector) skips planning and upload.  The key is the
// whole gate list with every compile-time setting it depends on (device, register size,
// fusion options, tile shape, environment overrides); learned and autotuned plans keep their
// own caches and are compiled per call.
namespace {

// Never destroyed (programs free device memory; at process exit the runtime may be gone).
std::mutex& prog_mu() {
    static auto* m = new std::mutex;
    return *m;
}
std::deque<std::pair<std::string, std::shared_ptr<const Program>>>& progs() {   // newest last
    static auto* d = new std::deque<std::pair<std::string, std::shared_ptr<const Program>>>;
    return *d;
}
constexpr size_t kProgramCache = 16;

std::string program_key(const std::vector<GateDesc>& gates, uint32_t n, const FusionConfig& fc) {
    std::string k;
    auto put = [&](const void* p, size_t len) { k.append(static_cast<const char*>(p), len); };
    int dev = 0;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    const TileConfig tc = default_tile_config(n);
    const uint32_t fw = default_fusion_width();
    const uint8_t tiles = use_tiles(n, fc) ? 1 : 0, fuse = fc.fuse ? 1 : 0, reg = tc.reg ? 1 : 0;
    put(&dev, sizeof dev);
    put(&n, sizeof n);
    put(&fuse, 1);
    put(&fc.mode, sizeof fc.mode);
    put(&fc.max_width, sizeof fc.max_width);
    put(&fw, sizeof fw);
    put(&tiles, 1);
    put(&tc.m, sizeof tc.m);
    put(&tc.L, sizeof tc.L);
    put(&tc.inner, sizeof tc.inner);
    put(&reg, 1);
    const uint8_t search = tc.search ? 1 : 0, mma = tc.mma ? 1 : 0;
    put(&search, 1);
    put(&mma, 1);
    for (const GateDesc& g : gates) {
        if (g.type == LQCS_GATE_MEASURE) continue;   // not part of the program
        const uint64_t sizes[5] = {g.qubits.size(), g.params.size(), g.mat.size(), g.perm.size(),
                                   g.pauli.size()};
        put(&g.type, sizeof g.type);
        put(&g.n_controls, sizeof g.n_controls);
        put(sizes, sizeof sizes);
        put(g.qubits.data(), g.qubits.size() * sizeof(uint32_t));
        put(g.params.data(), g.params.size() * sizeof(double));
        put(g.mat.data(), g.mat.size() * sizeof(cd));
        put(g.perm.data(), g.perm.size() * sizeof(uint64_t));
        put(g.pauli.data(), g.pauli.size());
    }
    return k;
}

}  // namespace

std::shared_ptr<const Program> cached_program(const std::vector<GateDesc>& gates, uint32_t n,
                                              const FusionConfig& fc, cudaStream_t stream) {
    auto compiled = [&] {
        std::vector<GateDesc> keep;
        keep.reserve(gates.size());
        for (const GateDesc& g : gates)
            if (g.type != LQCS_GATE_MEASURE) keep.push_back(g);
        return std::make_shared<const Program>(compile(keep, n, fc, stream));
    };
    if (fc.fuse && (fc.mode == kFuseLearned || fc.mode == kFuseAutotune)) return compiled();
    const std::string key = program_key(gates, n, fc);
    {
        std::lock_guard<std::mutex> lk(prog_mu());
        for (auto it = progs().begin(); it != progs().end(); ++it) {
            if (it->first == key) {
                auto hit = *it;
                progs().erase(it);
                progs().push_back(hit);
                return hit.second;
            }
        }
    }
    auto prog = compiled();
    cuda_check(cudaStreamSynchronize(stream), "program upload");   // usable from any stream
    std::lock_guard<std::mutex> lk(prog_mu());
    progs().emplace_back(key, prog);
    if (progs().size() > kProgramCache) progs().pop_front();
    return prog;
}

void clear_program_cache() {
    std::lock_guard<std::mutex> lk(prog_mu());
    progs().clear();
}

void apply_circuit(lqcs_state& st, const std::vector<GateDesc>& gates, const FusionConfig& fc) {
    for (const GateDesc& g : gates) {
        if (g.type == LQCS_GATE_RESET)
            invalid("run_statevector: Reset is non-deterministic; use run() instead");
        if (g.type == LQCS_GATE_KRAUS)
            invalid("run_statevector: noisy simulation is stochastic (one trajectory is "
                    "not the quantum state); use run() or DensityMatrixSimulator");
    }
    const std::shared_ptr<const Program> p = cached_program(gates, st.n, fc, st.stream);
    p->launch(st.ctx, st.d(), st.n, st.batch);
    st.sync();
}

std::unique_ptr<lqcs_program> program_create(uint32_t n, const std::vector<GateDesc>& gates,
                                             const FusionConfig& fc) {
    std::vector<GateDesc> keep;
    for (const GateDesc& g : gates) {
        if (g.type == LQCS_GATE_RESET)
            invalid("run_statevector: Reset is non-deterministic; use run() instead");
        if (g.type == LQCS_GATE_KRAUS)
            invalid("run_statevector: noisy simulation is stochastic (one trajectory is "
                    "not the quantum state); use run() or DensityMatrixSimulator");
        if (g.type == LQCS_GATE_MEASURE) continue;
        keep.push_back(g);
    }
    auto p = std::make_unique<lqcs_program>();
    p->n = n;
    p->prog = compile(keep, n, fc, nullptr);
    return p;
}

void program_profile(lqcs_state& st, const lqcs_program& p, uint64_t cap, lqcs_op_profile* out,
                     uint64_t* n_out) {
    const size_t nops = p.prog.ops.size();
    std::vector<cudaEvent_t> ev(nops + 1);
    for (auto& e : ev) cuda_check(cudaEventCreate(&e), "cudaEventCreate");
    cuda_check(cudaEventRecord(ev[0], st.stream), "cudaEventRecord");
    for (size_t i = 0; i < nops; ++i) {
        p.prog.launch_op(i, st.ctx, st.d(), st.n, st.batch);
        cuda_check(cudaEventRecord(ev[i + 1], st.stream), "cudaEventRecord");
    }
    st.sync();
    for (size_t i = 0; i < nops && i < cap && out; ++i) {
        const DevOp& op = p.prog.ops[i];
        float ms = 0.0f;
        cuda_check(cudaEventElapsedTime(&ms, ev[i], ev[i + 1]), "cudaEventElapsedTime");
        lqcs_op_profile& r = out[i];
        r.kind = profile_kind(op);
        r.n_targets = op.k;
        r.n_gates = op.src_gates;
        r.min_target = op.targets.empty() ? 0 : *std::min_element(op.targets.begin(), op.targets.end());
        r.max_target = op.targets.empty() ? 0 : *std::max_element(op.targets.begin(), op.targets.end());
        r.n_controls = static_cast<uint32_t>(__builtin_popcountll(op.cmask));
        r.device_ms = ms;
        r.alg_bytes = 32.0 * static_cast<double>(st.len()) * op.alg_fraction * st.batch;
        r.alg_flops = op_flops_per_amp(op) * static_cast<double>(st.len()) * st.batch;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    *n_out = nops;
}

// ------------------------------------------------------------------ reductions

static double fetch1(lqcs_state& st, const double* d) {
    double h = 0.0;
    cuda_check(cudaMemcpyAsync(&h, d, sizeof(double), cudaMemcpyDeviceToHost, st.stream), "D2H");
    st.sync();
    return h;
}

double state_norm2(lqcs_state& st) {
    double* part = st.partials(1);
    double* out = part + (kMaxReduceBlocks + 1);
    launch_norm2(st.ctx, st.d(), st.n, part, out);
    return fetch1(st, out);
}

std::vector<double> expectation_terms(lqcs_state& st, const std::vector<PauliMasks>& terms) {
    std::vector<double> vals(terms.size(), 0.0);
    if (terms.empty()) return vals;
    const uint32_t count = static_cast<uint32_t>(terms.size());
    std::vector<AdjRotation> list;
    for (uint32_t t = 0; t < count; ++t) list.push_back({terms[t].x, terms[t].zy, terms[t].n_y & 3u, t});
    if (st.n <= kExpectSmall) {
        st.scratch.ensure((sizeof(AdjRotation) + sizeof(double)) * count);
        AdjRotation* d_terms = st.scratch.as<AdjRotation>();
        double* d_out = reinterpret_cast<double*>(d_terms + count);
        cuda_check(cudaMemcpyAsync(d_terms, list.data(), sizeof(AdjRotation) * count,
                                   cudaMemcpyHostToDevice, st.stream), "H2D terms");
        launch_expect_small(st.ctx, st.d(), st.n, d_terms, count, d_out);
        cuda_check(cudaMemcpyAsync(vals.data(), d_out, sizeof(double) * count,
                                   cudaMemcpyDeviceToHost, st.stream), "D2H expectations");
        st.sync();
        return vals;
    }
    // terms of one x mask side by side: they share a layout
    std::stable_sort(list.begin(), list.end(),
                     [](const AdjRotation& a, const AdjRotation& b) { return a.x < b.x; });
    // A bounded number of terms at a time: planning passes takes (terms) * (passes), and a term's
    // partial sums up to 4.7 KB (a block each on 148 SMs).  The device runs one group while the host
    // plans the next; with all terms in one group, 20000 diagonal ones on 15 qubits took 45 ms
    // instead of 16, 3000 random ones on 24 qubits 33 instead of 28.
    constexpr uint32_t kGroup = 1024;
    const uint32_t blocks = expect_blocks(st.ctx, st.n);
    st.scratch.ensure(sizeof(double) * (count + size_t{blocks} * std::min(count, kGroup)));
    double* d_out = st.scratch.as<double>();   // in the sorted order
    double* part = d_out + count;
    std::vector<AdjRotation> group;
    for (uint32_t first = 0; first < count; first += kGroup) {
        const uint32_t n_terms = std::min(kGroup, count - first);
        group.assign(list.begin() + first, list.begin() + first + n_terms);
        for (uint32_t t = 0; t < n_terms; ++t) group[t].param = t;
        for (const AdjPass& p : plan_adjoint_passes(group, st.n, kExpectTileBits, 4, true, kExpectTerms))
            launch_expect_pass(st.ctx, st.d(), st.n, p, part);
        launch_expect_sum(st.ctx, st.n, n_terms, part, d_out + first);
    }
    std::vector<double> sorted(count);
    cuda_check(cudaMemcpyAsync(sorted.data(), d_out, sizeof(double) * count, cudaMemcpyDeviceToHost,
                               st.stream), "D2H expectations");
    st.sync();
    for (uint32_t t = 0; t < count; ++t) vals[list[t].param] = sorted[t];
    return vals;
}

int collapse(lqcs_state& st, uint32_t q, double u) {
    if (q >= st.n) out_of_range("collapse: qubit index out of range");
    double* part = st.partials(1);
    double* out = part + (kMaxReduceBlocks + 1);
    launch_bitprob(st.ctx, st.d(), st.n, q, part, out);
    const double p1 = fetch1(st, out);
    const int outcome = u < p1 ? 1 : 0;
    const double keep = outcome ? p1 : 1.0 - p1;
    const double scale = 1.0 / std::sqrt(keep);
    launch_project(st.ctx, st.d(), st.n, q, outcome, scale);
    return outcome;
}

void reset_qubit(lqcs_state& st, uint32_t q, double u) {
    if (!collapse(st, q, u)) return;
    launch_move_to_zero(st.ctx, st.d(), st.n, q);
}

double kraus_probability(lqcs_state& st, uint32_t q, const std::array<cd, 4>& k) {
    if (q >= st.n) out_of_range("kraus_probability: qubit index out of range");
    double* part = st.partials(1);
    double* out = part + (kMaxReduceBlocks + 1);
    const double2 kk[4] = {to_d2(k[0]), to_d2(k[1]), to_d2(k[2]), to_d2(k[3])};
    launch_kraus_prob(st.ctx, st.d(), st.n, q, kk, part, out);
    return fetch1(st, out);
}

void sample(lqcs_state& st, const double* u, uint64_t shots, uint64_t* idx, double* min_margin) {
    const uint64_t n_t = scan_thread_count(st.n), n_s = scan_block_count(st.n) + 1;
    st.sample_scratch.ensure(sizeof(double) * (n_t + n_s + 3 * shots));
    double* tpref = st.sample_scratch.as<double>();
    double* seg = tpref + n_t;
    double* du = seg + n_s;
    uint64_t* didx = reinterpret_cast<uint64_t*>(du + shots);
    double* dmargin = du + 2 * shots;
    launch_prob_scan(st.ctx, st.d(), st.n, tpref, seg);
    if (shots == 0) {
        if (min_margin) *min_margin = 1.0;
        st.sync();
        return;
    }
    cuda_check(cudaMemcpyAsync(du, u, sizeof(double) * shots, cudaMemcpyHostToDevice, st.stream),
               "H2D uniforms");
    launch_sample_search(st.ctx, st.d(), st.n, tpref, seg, du, shots, didx, dmargin);
    cuda_check(cudaMemcpyAsync(idx, didx, sizeof(uint64_t) * shots, cudaMemcpyDeviceToHost,
                               st.stream),
               "D2H sample indices");
    std::vector<double> margins;
    if (min_margin) {
        margins.resize(shots);
        cuda_check(cudaMemcpyAsync(margins.data(), dmargin, sizeof(double) * shots,
                                   cudaMemcpyDeviceToHost, st.stream),
                   "D2H margins");
    }
    st.sync();
    if (min_margin) *min_margin = *std::min_element(margins.begin(), margins.end());
}

// ------------------------------------------------------------------ run()

using Kraus = std::array<cd, 4>;
using Channel = std::vector<Kraus>;

std::vector<std::vector<std::array<cd, 4>>> decode_channels(const lqcs_sim_options* opts) {
    std::vector<Channel> out;
    if (!opts || opts->n_channels == 0) return out;
    if (!opts->channels) invalid("NoiseModel: channels pointer is null");
    for (uint64_t c = 0; c < opts->n_channels; ++c) {
        const lqcs_kraus_channel& ch = opts->channels[c];
        if (ch.n_ops == 0 || ch.ops == nullptr) invalid("KrausChannel: needs at least one operator");
        Channel k(ch.n_ops);
        for (uint64_t o = 0; o < ch.n_ops; ++o)
            for (int e = 0; e < 4; ++e) k[o][e] = cd{ch.ops[8 * o + 2 * e], ch.ops[8 * o + 2 * e + 1]};
        out.push_back(std::move(k));
    }
    return out;
}

namespace {

// Emission order of SingleQubitGateFusion (src/transpiler/gate_fusion.cpp:32-67), reduced
// to what run()'s path selection reads from it: true when some unitary is emitted after a
// Measure.  Pending one-qubit products are flushed on any other instruction touching the
// qubit, on Barrier, and at the end; identity products (within 1e-12) are dropped.
bool fused_has_unitary_after_measure(const std::vector<GateDesc>& gates, uint32_t n) {
    using M2 = std::array<cd, 4>;
    std::vector<std::optional<M2>> pending(n);
    bool seen_measure = false, after = false;
    auto is_identity = [](const M2& m) {
        constexpr double tol = 1e-12;
        return std::abs(m[0] - cd{1, 0}) < tol && std::abs(m[1]) < tol && std::abs(m[2]) < tol &&
               std::abs(m[3] - cd{1, 0}) < tol;
    };
    auto emit_unitary = [&]() { if (seen_measure) after = true; };
    auto flush = [&](uint32_t q) {
        if (!pending[q]) return;
        if (!is_identity(*pending[q])) emit_unitary();
        pending[q].reset();
    };
    for (const GateDesc& g : gates) {
        if (g.is_unitary() && g.n_controls == 0 && g.base_qubits() == 1) {
            const std::vector<cd> m = g.base_matrix();
            const M2 a{m[0], m[1], m[2], m[3]};
            const uint32_t q = g.qubits[0];
            if (pending[q]) {
                const M2& b = *pending[q];
                pending[q] = M2{a[0] * b[0] + a[1] * b[2], a[0] * b[1] + a[1] * b[3],
                                a[2] * b[0] + a[3] * b[2], a[2] * b[1] + a[3] * b[3]};
            } else {
                pending[q] = a;
            }
            continue;
        }
        if (g.type == LQCS_GATE_BARRIER) {
            for (uint32_t q = 0; q < n; ++q) flush(q);
        } else {
            for (uint32_t q : g.qubits) flush(q);
        }
        if (g.type == LQCS_GATE_MEASURE) seen_measure = true;
        else if (g.is_unitary()) emit_unitary();
    }
    for (uint32_t q = 0; q < n; ++q) flush(q);
    return after;
}

}  // namespace

void run_shots(uint32_t n, uint32_t n_clbits, const std::vector<GateDesc>& gates,
               uint64_t shots, const lqcs_sim_options* opts, uint64_t* regs) {
    if (shots == 0) invalid("run: shots must be >= 1");
    if (n_clbits > 64) invalid("run: this engine reports at most 64 classical bits");
    const std::vector<Channel> channels = decode_channels(opts);
    const bool noisy = !channels.empty();
    const bool fuse = opts ? (opts->fuse_gates != 0) : true;

    // Path selection of StatevectorSimulator::run (src/backend/statevector_simulator.cpp:241-257),
    // evaluated on the instruction order the reference's fusion pass would emit.
    bool seen_measure = false, per_shot = noisy;
    for (const GateDesc& g : gates) {
        if (g.type == LQCS_GATE_MEASURE) {
            if (g.clbit >= n_clbits) {
                out_of_range("clbit index " + std::to_string(g.clbit) +
                             " out of range (num_clbits = " + std::to_string(n_clbits) + ")");
            }
            seen_measure = true;
        } else if (g.type == LQCS_GATE_RESET || g.type == LQCS_GATE_KRAUS) {
            per_shot = true;
        } else if (seen_measure && g.is_unitary()) {
            per_shot = true;
        }
    }
    if (!per_shot && fuse && !noisy) per_shot = fused_has_unitary_after_measure(gates, n);
    if (!seen_measure) {
        invalid("run: circuit has no measurements; use run_statevector() to inspect the final "
                "state");
    }
    Rng rng = make_rng(opts);
    FusionConfig fc;
    fc.fuse = fuse && !noisy;
    if (opts) {
        fc.max_width = static_cast<uint32_t>(std::max(0, opts->max_fusion_width));
        fc.mode = opts->fusion_mode;
    }
    if (!per_shot) {
        // run_sampling (src/backend/statevector_simulator.cpp:88-119)
        auto st = new_state(n, 1, nullptr);
        apply_circuit(*st, gates, fc);
        std::vector<int64_t> src(n_clbits, -1);
        for (const GateDesc& g : gates)
            if (g.type == LQCS_GATE_MEASURE) src[g.clbit] = g.qubits[0];
        std::vector<double> u(shots);
        if (opts && opts->shot_offset) rng.discard(opts->shot_offset);   // one uniform per shot
        for (uint64_t s = 0; s < shots; ++s) u[s] = rng_uniform(rng);
        std::vector<uint64_t> idx(shots);
        sample(*st, u.data(), shots, idx.data(), nullptr);
        for (uint64_t s = 0; s < shots; ++s) {
            uint64_t reg = 0;
            for (uint32_t c = 0; c < n_clbits; ++c)
                if (src[c] >= 0 && ((idx[s] >> src[c]) & 1u)) reg |= uint64_t{1} << c;
            regs[s] = reg;
        }
        return;
    }

    // run_per_shot (src/backend/statevector_simulator.cpp:156-190), many shots at a time
    std::vector<std::vector<std::array<cd, 4>>> chans;
    for (const Channel& c : channels) chans.emplace_back(c.begin(), c.end());
    const uint32_t resident = opts ? static_cast<uint32_t>(std::max(0, opts->max_resident)) : 0;
    run_per_shot_batched(n, gates, shots, chans, fc, rng, resident, regs,
                         opts ? opts->shot_offset : 0);
}

// ------------------------------------------------------------------ Hamiltonians

Hamiltonian decode_hamiltonian(const lqcs_hamiltonian* h, uint32_t n) {
    if (!h) invalid("hamiltonian is null");
    Hamiltonian out;
    if (h->n_terms > 0 && (!h->coeffs || !h->paulis)) invalid("hamiltonian: null arrays");
    for (uint64_t t = 0; t < h->n_terms; ++t) {
        out.coeffs.push_back(h->coeffs[t]);
        out.terms.push_back(pauli_global_masks(h->paulis[t], n, "expectation_value"));
    }
    return out;
}

double energy(lqcs_state& st, const Hamiltonian& h) {
    // algorithms::expectation (src/algorithms/vqe.cpp:11-17): sum in term order
    const std::vector<double> v = expectation_terms(st, h.terms);
    double e = 0.0;
    for (size_t t = 0; t < v.size(); ++t) e += h.coeffs[t] * v[t];
    return e;
}

std::vector<GateDesc> bind_params(const std::vector<GateDesc>& tmpl,
                                         const std::vector<uint64_t>& param_inst,
                                         const double* values) {
    std::vector<GateDesc> g = tmpl;
    for (size_t p = 0; p < param_inst.size(); ++p) {
        GateDesc& d = g[param_inst[p]];
        if (d.params.empty()) d.params.push_back(0.0);
        d.params[0] = values[p];
    }
    return g;
}

void check_pc(const lqcs_parametric_circuit* pc, std::vector<GateDesc>& tmpl,
                     std::vector<uint64_t>& pinst) {
    if (!pc) invalid("parametric circuit is null");
    tmpl = decode_all(pc->insts, pc->n_insts, pc->n_qubits);
    if (pc->n_params > 0 && !pc->param_inst) invalid("parametric circuit: null param_inst");
    pinst.assign(pc->param_inst, pc->param_inst + pc->n_params);
    for (uint64_t p : pinst) {
        if (p >= tmpl.size()) invalid("parametric circuit: parameter index out of range");
        const GateDesc& g = tmpl[p];
        const bool ok = (g.type == LQCS_GATE_RX || g.type == LQCS_GATE_RY || g.type == LQCS_GATE_RZ ||
                         g.type == LQCS_GATE_PAULI_ROTATION) && g.n_controls == 0;
        if (!ok) invalid("parametric circuit: parameterised gates must be RX, RY, RZ or rp");
    }
}

void parameter_shift(const lqcs_parametric_circuit* pc, const Hamiltonian& h,
                     const double* params, double* grad) {
    // algorithms::parameter_shift_gradient (src/algorithms/vqe.cpp:68-94)
    std::vector<GateDesc> tmpl;
    std::vector<uint64_t> pinst;
    check_pc(pc, tmpl, pinst);
    const size_t np = pinst.size();
    auto st = new_state(pc->n_qubits, 1, nullptr);
    FusionConfig fc;
    std::vector<double> theta(params, params + np);
    auto e_at = [&](const std::vector<double>& th) {
        launch_set_basis(st->ctx, st->d(), st->n, 1, 0);
        apply_circuit(*st, bind_params(tmpl, pinst, th.data()), fc);
        return energy(*st, h);
    };
    constexpr double half_pi = std::numbers::pi / 2;
    for (size_t k = 0; k < np; ++k) {
        const double saved = theta[k];
        theta[k] = saved + half_pi;
        const double ep = e_at(theta);
        theta[k] = saved - half_pi;
        const double em = e_at(theta);
        theta[k] = saved;
        grad[k] = 0.5 * (ep - em);
    }
}

}  // namespace lqcs_b200
