// tile_plan.cpp — planning of shared-memory tile passes.
//
// A pass is a set H of high qubits plus the gates it applies.  First-fit over the gates in
// program order: a gate joins the pass when its targets above bit L fit into H (growing H up
// to h qubits) and none of its qubits is blocked; otherwise it is deferred and its qubits
// become blocked, so every later gate on them is deferred too and program order on each
// qubit is kept.  Controls and phase bits need no tile slot (they are constant over a tile
// or select the amplitudes a phase multiplies).  Inside a pass, neighbouring gates on tile
// qubits are fused into dense operations of at most `inner` qubits.
#include <algorithm>
#include <bit>
#include <cmath>
#include <cstdlib>
#include <deque>
#include <map>
#include <string>
#include <tuple>

#include "tile_plan.hpp"

namespace lqcs_b200 {

namespace {

bool is_phase_gate(const GateDesc& g) {
    if (g.slot || !g.is_unitary() || g.base_qubits() != 1) return false;
    if (g.type == LQCS_GATE_PAULI_ROTATION) return false;
    const std::vector<cd> m = g.base_matrix();
    return m[1] == cd{0, 0} && m[2] == cd{0, 0} && m[0] == cd{1, 0};
}

int env_int(const char* name, int dflt) {
    if (const char* e = std::getenv(name)) return std::atoi(e);
    return dflt;
}

}  // namespace

TileConfig default_tile_config(uint32_t n) {
    TileConfig c;
    c.m = static_cast<uint32_t>(env_int("LQCS_TILE_BITS", 12));
    c.L = static_cast<uint32_t>(env_int("LQCS_TILE_LOW", 5));
    c.inner = static_cast<uint32_t>(env_int("LQCS_TILE_INNER", 2));
    c.reg = env_int("LQCS_TILE_REG", 1) != 0;
    c.search = env_int("LQCS_TILE_SEARCH", 1) != 0;
    c.mma = env_int("LQCS_REG_MMA", 0) != 0;
    c.pauli = env_int("LQCS_TILE_PAULI", 1) != 0;
    c.m = std::max<uint32_t>(kTileMinBits, std::min<uint32_t>(std::min<uint32_t>(c.m, kTileMaxBits), n));
    c.L = std::min<uint32_t>(std::min(c.L, c.m), kTileMinBits);   // column bits come from the thread index
    if (c.m - c.L > kTileMaxHigh) c.L = c.m - kTileMaxHigh;
    c.inner = std::max<uint32_t>(1, std::min<uint32_t>(c.inner, kTileMaxK));
    return c;
}

bool native_pauli(const GateDesc& g, const TileConfig& cfg) {
    if (!cfg.reg || !cfg.pauli || g.type != LQCS_GATE_PAULI_ROTATION || g.n_controls != 0 || g.slot)
        return false;
    uint32_t flips = 0;
    for (char ch : g.pauli) flips += ch == 'X' || ch == 'Y';
    return flips <= kRegPauliMaxFlips;
}

// Qubits a gate needs inside the tile, or false if it cannot run in a tile at all.  A native
// Pauli rotation needs only its X/Y qubits there (its Z-type qubits act through parities).
static bool tile_requirements(const GateDesc& g, const TileConfig& c, std::vector<uint32_t>& need) {
    need.clear();
    if (native_pauli(g, c)) {
        const uint32_t k = g.base_qubits();
        for (uint32_t j = 0; j < k; ++j) {
            const char ch = g.pauli[k - 1 - j];   // local bit j <-> pauli[k-1-j] (Gate::pauli_masks)
            if (ch == 'X' || ch == 'Y') need.push_back(g.targets()[j]);
        }
        return true;
    }
    if (is_phase_gate(g)) return g.qubits.size() <= 8;   // at most 8 local phase bits
    const uint32_t k = g.base_qubits();
    if (k == 0 || k > kTileMaxK) return false;
    if (g.type == LQCS_GATE_PERMUTATION && k > kTileMaxK) return false;
    if (k + g.n_controls > 8) return false;
    for (uint32_t j = 0; j < k; ++j) need.push_back(g.targets()[j]);
    (void)c;
    return true;
}

namespace {

bool is_x_matrix(const std::vector<cd>& m) {
    return m.size() == 4 && m[0] == cd{0, 0} && m[1] == cd{1, 0} && m[2] == cd{1, 0} &&
           m[3] == cd{0, 0};
}

// An uncontrolled one-qubit gate with a matrix of its own.
bool plain_1q(const GateDesc& g) {
    return g.is_unitary() && g.n_controls == 0 && g.type != LQCS_GATE_PAULI_ROTATION &&
           g.type != LQCS_GATE_PERMUTATION && g.type != LQCS_GATE_SWAP && g.base_qubits() == 1;
}

GateDesc simple_gate(int type, std::vector<uint32_t> qubits, uint32_t n_controls,
                     std::vector<double> params = {}) {
    GateDesc g;
    g.type = type;
    g.qubits = std::move(qubits);
    g.n_controls = n_controls;
    g.params = std::move(params);
    return g;
}

}  // namespace

std::vector<GateDesc> rotation_form(const std::vector<GateDesc>& gates, uint32_t n) {
    using M2 = std::array<cl, 4>;
    // What each gate is to its neighbours on a qubit: an X with controls (on its target), a
    // one-qubit gate that is (not) diagonal, a dense two-qubit gate that takes one-qubit
    // factors for free, or anything else.
    enum Role : uint8_t { kOther, kCtrlX, kDiag1, kDense1, kDense2 };
    std::vector<Role> role(gates.size(), kOther);
    std::vector<std::vector<uint32_t>> on(n);   // gates touching each qubit, in order
    std::vector<uint32_t> at(gates.size(), 0);  // index of gate i in its target's list
    std::vector<std::array<cd, 4>> base(gates.size());   // base matrix of one-qubit gates
    for (uint32_t i = 0; i < gates.size(); ++i) {
        const GateDesc& g = gates[i];
        if (g.type == LQCS_GATE_BARRIER) {
            for (auto& v : on) v.push_back(i);
            continue;
        }
        if (g.slot) {
            role[i] = kDense1;
        } else if (g.is_unitary() && g.type != LQCS_GATE_PAULI_ROTATION &&
                   g.type != LQCS_GATE_PERMUTATION) {
            if (g.base_qubits() == 1) {
                const std::vector<cd> m = g.base_matrix();
                std::copy_n(m.begin(), 4, base[i].begin());
                if (g.n_controls == 0)
                    role[i] = m[1] == cd{0, 0} && m[2] == cd{0, 0} ? kDiag1 : kDense1;
                else if (is_x_matrix(m) && g.qubits.size() <= 8)
                    role[i] = kCtrlX;
            } else if (g.base_qubits() == 2 && g.n_controls == 0 && g.type != LQCS_GATE_RZZ &&
                       g.type != LQCS_GATE_SWAP) {
                role[i] = kDense2;
            }
        }
        if (role[i] == kCtrlX) at[i] = static_cast<uint32_t>(on[g.targets()[0]].size());
        for (uint32_t q : g.qubits) on[q].push_back(i);
    }
    // the neighbour of gate i on its target in direction dir takes the H (diagonal one-qubit
    // gates in between merge with it)
    auto absorbs = [&](uint32_t i, int dir) {
        const uint32_t t = gates[i].targets()[0];
        const std::vector<uint32_t>& v = on[t];
        for (int64_t k = static_cast<int64_t>(at[i]) + dir;
             k >= 0 && k < static_cast<int64_t>(v.size()); k += dir) {
            const uint32_t j = v[static_cast<size_t>(k)];
            if (role[j] == kDiag1) continue;
            return role[j] == kDense1 || role[j] == kDense2 ||
                   (role[j] == kCtrlX && gates[j].targets()[0] == t);
        }
        return false;
    };

    std::vector<GateDesc> out;
    uint32_t carry = 0;   // source gates of products that turned out to be the identity
    struct Pending {
        M2 m{};
        uint32_t count = 0, src = 0;
        const GateDesc* one = nullptr;   // the source gate while it is the only one, or what a
        int made = 0;                    // gate of this pass's own is made from (0: an H that is
        double value = 0.0;              // rounded to `value`; RZ, P: their angle)
    };
    std::vector<Pending> pend(n);
    auto push = [&](GateDesc g) {
        g.src += carry;
        carry = 0;
        out.push_back(std::move(g));
    };
    auto multiply = [&](uint32_t q, const M2& a, uint32_t src, const GateDesc* one, int made = 0,
                        double value = 0.0) {
        Pending& p = pend[q];
        if (p.count == 0) {
            p.m = a;
            p.one = one;
            p.made = made;
            p.value = value;
        } else {
            const M2 b = p.m;
            p.m = {wide_mul(a[0], b[0]) + wide_mul(a[1], b[2]),
                   wide_mul(a[0], b[1]) + wide_mul(a[1], b[3]),
                   wide_mul(a[2], b[0]) + wide_mul(a[3], b[2]),
                   wide_mul(a[2], b[1]) + wide_mul(a[3], b[3])};
        }
        ++p.count;
        p.src += src;
    };
    auto flush = [&](uint32_t q) {
        Pending& p = pend[q];
        if (p.count == 0) return;
        constexpr long double tol = 5e-16L;
        if (p.count > 1 && std::abs(p.m[0] - cl{1, 0}) < tol && std::abs(p.m[1]) < tol &&
            std::abs(p.m[2]) < tol && std::abs(p.m[3] - cl{1, 0}) < tol) {
            carry += p.src;   // such as the H H between two exchanged X
        } else {
            GateDesc g;
            if (p.count == 1 && p.one) {
                g = *p.one;
            } else if (p.count == 1 && p.made) {
                g = simple_gate(p.made, {q}, 0, {p.value});
                g.wide.assign(p.m.begin(), p.m.end());
            } else {
                g = simple_gate(LQCS_GATE_UNITARY, {q}, 0);
                if (p.count == 1) g.mat = {p.value, p.value, p.value, -p.value};
                else
                    for (const cl& z : p.m) g.mat.push_back(narrow(z));
                g.wide.assign(p.m.begin(), p.m.end());
            }
            g.src = p.src;
            push(std::move(g));
        }
        p = Pending{};
    };
    auto matrix_of = [&](uint32_t i) {
        M2 a;
        for (int e = 0; e < 4; ++e) a[e] = gates[i].wide.empty() ? cl{base[i][e]} : gates[i].wide[e];
        return a;
    };
    // 1/sqrt(2) rounded up and down (see below)
    const long double root = std::sqrt(0.5L);
    const double nearest = static_cast<double>(root);
    const double other = std::nextafter(nearest, nearest > root ? 0.0 : 1.0);
    for (uint32_t i = 0; i < gates.size(); ++i) {
        const GateDesc& g = gates[i];
        if (g.type == LQCS_GATE_BARRIER) {
            for (uint32_t q = 0; q < n; ++q) flush(q);
            push(g);
            continue;
        }
        if (!g.slot && plain_1q(g)) {
            if (role[i] == kDiag1) {   // a damping factor: between two gates it would leave no
                const std::array<cd, 4>& m = base[i];   // rotation form, in a table it is free
                if (std::abs(std::abs(m[0]) - std::abs(m[3])) > 1e-12) {
                    flush(g.qubits[0]);
                    push(g);
                    continue;
                }
            }
            multiply(g.qubits[0], matrix_of(i), g.src, &g);
            continue;
        }
        if (role[i] == kCtrlX && (absorbs(i, -1) || absorbs(i, 1))) {
            const uint32_t t = g.targets()[0];
            // The H before rounds 1/sqrt(2) up and the H after rounds it down: two of the same
            // would scale the state by 1 + 2e-16 for every exchanged X where they are folded
            // into dense blocks.
            const M2 h = {root, root, root, -root};
            multiply(t, h, 0, nullptr, 0, nearest);
            for (uint32_t q : g.qubits) flush(q);
            GateDesc z = simple_gate(LQCS_GATE_Z, g.qubits, g.n_controls);
            z.src = g.src;
            push(std::move(z));
            multiply(t, h, 0, nullptr, 0, other);
            continue;
        }
        if (g.type == LQCS_GATE_RZZ && g.n_controls == 0) {
            // diag(e^-i, e^i, e^i, e^-i)(theta/2): RZ(theta) on a, P(theta) on b, CP(-2 theta);
            // the one-qubit factors join a pending product, or wait for the next gate
            const uint32_t a = g.qubits[0], b = g.qubits[1];
            const double th = g.params.at(0);
            const uint32_t rz = pend[b].count > 0 && pend[a].count == 0 ? b : a;
            const uint32_t ph = rz == a ? b : a;
            auto unit = [](long double x) { return cl{std::cos(x), std::sin(x)}; };
            const M2 grz = {unit(-0.5L * th), 0.0L, 0.0L, unit(0.5L * th)};
            const M2 gph = {1.0L, 0.0L, 0.0L, unit(th)};
            const bool rz_now = pend[rz].count > 0, ph_now = pend[ph].count > 0;
            if (rz_now) multiply(rz, grz, 0, nullptr, LQCS_GATE_RZ, th);
            if (ph_now) multiply(ph, gph, 0, nullptr, LQCS_GATE_P, th);
            flush(a);
            flush(b);
            GateDesc cp = simple_gate(LQCS_GATE_P, {a, b}, 1, {-2.0 * th});
            cp.src = g.src;
            cp.wide = {1.0L, 0.0L, 0.0L, unit(-2.0L * th)};
            push(std::move(cp));
            if (!rz_now) multiply(rz, grz, 0, nullptr, LQCS_GATE_RZ, th);
            if (!ph_now) multiply(ph, gph, 0, nullptr, LQCS_GATE_P, th);
            continue;
        }
        for (uint32_t q : g.qubits) flush(q);
        push(g);
    }
    for (uint32_t q = 0; q < n; ++q) flush(q);
    if (carry && !out.empty()) out.back().src += carry;
    return out;
}

// First-fit picks the high tile qubits in the order gates ask for them, which is often not
// the set that takes the most gates.  Local search: swap one high qubit of the pass for one
// outside it while that lets the pass take more gates (same rules as the first-fit scan:
// program order per qubit, barriers end the pass, at most kTileMaxOps gates).  On the
// 30-qubit brickwork this cuts 75 passes to about 50.
static void improve_high_bits(const std::vector<GateDesc>& gates, uint32_t n, const TileConfig& cfg,
                              const std::vector<uint32_t>& remaining, std::vector<uint32_t>& hset,
                              std::vector<uint32_t>& taken, std::vector<uint32_t>& deferred) {
    struct G {
        uint64_t qubits, need;   // all qubits; high qubits the gate needs in the tile
        bool ok, barrier;
    };
    std::vector<G> gs;
    gs.reserve(remaining.size());
    std::vector<uint32_t> need;
    for (uint32_t gi : remaining) {
        const GateDesc& g = gates[gi];
        G e{0, 0, false, g.type == LQCS_GATE_BARRIER};
        for (uint32_t q : g.qubits) e.qubits |= uint64_t{1} << q;
        if (!e.barrier && tile_requirements(g, cfg, need)) {
            e.ok = true;
            for (uint32_t q : need)
                if (q >= cfg.L) e.need |= uint64_t{1} << q;
        }
        gs.push_back(e);
    }
    auto count = [&](uint64_t hmask) {
        uint64_t blocked = 0;
        size_t got = 0;
        for (const G& e : gs) {
            if (e.barrier || got >= kTileMaxOps) break;
            if (!(e.qubits & blocked) && e.ok && !(e.need & ~hmask)) ++got;
            else blocked |= e.qubits;
        }
        return got;
    };
    uint64_t hmask = 0;
    for (uint32_t q : hset) hmask |= uint64_t{1} << q;
    // with the padded set fixed the scan takes every gate first-fit took (and maybe more)
    size_t best = count(hmask);
    for (int round = 0; round < 8; ++round) {
        bool better = false;
        for (uint32_t out = cfg.L; out < n; ++out) {
            if (!((hmask >> out) & 1)) continue;
            for (uint32_t in = cfg.L; in < n; ++in) {
                if ((hmask >> in) & 1) continue;
                const uint64_t cand = (hmask & ~(uint64_t{1} << out)) | (uint64_t{1} << in);
                const size_t c = count(cand);
                if (c > best) {
                    best = c;
                    hmask = cand;
                    better = true;
                    break;
                }
            }
        }
        if (!better) break;
    }
    hset.clear();
    for (uint32_t q = cfg.L; q < n; ++q)
        if ((hmask >> q) & 1) hset.push_back(q);
    taken.clear();
    deferred.clear();
    uint64_t blocked = 0;
    bool stop = false;
    for (size_t i = 0; i < gs.size(); ++i) {
        const G& e = gs[i];
        if (stop || e.barrier || taken.size() >= kTileMaxOps) {
            stop = true;
            deferred.push_back(remaining[i]);
            continue;
        }
        if (!(e.qubits & blocked) && e.ok && !(e.need & ~hmask)) {
            taken.push_back(remaining[i]);
        } else {
            deferred.push_back(remaining[i]);
            blocked |= e.qubits;
        }
    }
}

std::vector<PlanItem> plan_tiles(const std::vector<GateDesc>& gates, uint32_t n,
                                 const TileConfig& cfg) {
    std::vector<PlanItem> items;
    const uint32_t h = cfg.m - cfg.L;
    std::vector<uint32_t> remaining;
    for (uint32_t i = 0; i < gates.size(); ++i) {
        if (gates[i].type == LQCS_GATE_BARRIER) {
            remaining.push_back(i);
            continue;
        }
        if (gates[i].is_unitary()) remaining.push_back(i);
    }
    std::vector<uint32_t> need;
    std::vector<char> blocked(n, 0);
    while (!remaining.empty()) {
        // a barrier at the front closes nothing (there is no open pass): drop it
        if (gates[remaining.front()].type == LQCS_GATE_BARRIER) {
            remaining.erase(remaining.begin());
            continue;
        }
        std::vector<uint32_t> hset;
        std::vector<uint32_t> taken, deferred;
        std::fill(blocked.begin(), blocked.end(), 0);
        bool stop = false;
        for (uint32_t gi : remaining) {
            const GateDesc& g = gates[gi];
            if (stop || g.type == LQCS_GATE_BARRIER || taken.size() >= kTileMaxOps) {
                // a barrier ends the pass: everything from here waits for the next one
                stop = true;
                deferred.push_back(gi);
                continue;
            }
            bool blk = false;
            for (uint32_t q : g.qubits) blk |= blocked[q] != 0;
            bool ok = !blk && tile_requirements(g, cfg, need);
            if (ok) {
                std::vector<uint32_t> add;
                for (uint32_t q : need)
                    if (q >= cfg.L && std::find(hset.begin(), hset.end(), q) == hset.end() &&
                        std::find(add.begin(), add.end(), q) == add.end())
                        add.push_back(q);
                ok = hset.size() + add.size() <= h;
                if (ok) hset.insert(hset.end(), add.begin(), add.end());
            }
            if (ok) {
                taken.push_back(gi);
            } else {
                deferred.push_back(gi);
                for (uint32_t q : g.qubits) blocked[q] = 1;
            }
        }
        if (taken.empty()) {
            // the first gate cannot run in a tile: run it on its own
            PlanItem it;
            it.is_pass = false;
            it.gate = remaining.front();
            items.push_back(std::move(it));
            remaining.erase(remaining.begin());
            continue;
        }
        // every pass gets the full tile size: pad H with unused high qubits
        for (uint32_t q = cfg.L; q < n && hset.size() < h; ++q)
            if (std::find(hset.begin(), hset.end(), q) == hset.end()) hset.push_back(q);
        if (cfg.search && n <= 64) improve_high_bits(gates, n, cfg, remaining, hset, taken, deferred);
        PlanItem it;
        it.is_pass = true;
        std::sort(hset.begin(), hset.end());
        it.hbits = hset;
        it.gates = taken;
        items.push_back(std::move(it));
        remaining = std::move(deferred);
    }
    return items;
}

// ------------------------------------------------------------------ lowering

namespace {

struct LocalMap {
    uint32_t L;
    std::vector<uint32_t> hbits;
    // tile bit of qubit q, where a relabelling (virtual SWAP) has moved it; -1: none
    std::vector<std::pair<uint32_t, uint32_t>> moved;
    int home(uint32_t q) const {   // tile bit at load, -1 if outside the tile
        if (q < L) return static_cast<int>(q);
        const auto it = std::find(hbits.begin(), hbits.end(), q);
        return it == hbits.end() ? -1 : static_cast<int>(L + (it - hbits.begin()));
    }
    int local(uint32_t q) const {   // -1 if outside the tile
        for (const auto& [qq, b] : moved)
            if (qq == q) return static_cast<int>(b);
        return home(q);
    }
    void swap_bits(uint32_t a, uint32_t b) {
        const uint32_t la = static_cast<uint32_t>(local(a)), lb = static_cast<uint32_t>(local(b));
        auto set = [&](uint32_t q, uint32_t bit) {
            for (auto& e : moved)
                if (e.first == q) {
                    e.second = bit;
                    return;
                }
            moved.emplace_back(q, bit);
        };
        set(a, lb);
        set(b, la);
    }
};

uint32_t deposit(uint32_t v, const std::vector<uint32_t>& sorted_pos) {
    for (uint32_t p : sorted_pos) {
        const uint32_t low = (1u << p) - 1u;
        v = ((v & ~low) << 1) | (v & low);
    }
    return v;
}

bool is_diagonal(const std::vector<cd>& m, uint64_t dim) {
    for (uint64_t r = 0; r < dim; ++r)
        for (uint64_t c = 0; c < dim; ++c)
            if (r != c && m[r * dim + c] != cd{0, 0}) return false;
    return true;
}

// Dense or diagonal op of matrix m on local targets lt, local controls lcmask.
LocalOp matrix_op(const std::vector<cd>& m, const std::vector<uint32_t>& lt, uint32_t lcmask,
                  uint64_t gcmask, bool variant) {
    LocalOp op;
    const uint64_t dim = uint64_t{1} << lt.size();
    op.lt = lt;
    op.lmask = lcmask;
    op.gcmask = gcmask;
    op.variant = variant;
    if (!variant && is_diagonal(m, dim)) {
        op.kind = kTileDiag;
        for (uint64_t i = 0; i < dim; ++i) op.m.push_back(m[i * dim + i]);
    } else {
        op.kind = kTileDense;
        op.m = m;
    }
    return op;
}

// Group enumeration of an op on a 2^m tile: the positions spread over (ascending), the
// group count, and the per-iteration slot parts sw(deposit(j * threads) | lcmask).
void set_groups(TileOp& op, std::vector<uint32_t> pos, uint32_t lcmask, uint32_t m) {
    std::sort(pos.begin(), pos.end());
    op.n_fixed = static_cast<uint8_t>(pos.size());
    for (size_t i = 0; i < pos.size(); ++i) op.fixed[i] = static_cast<uint8_t>(pos[i]);
    const uint32_t groups = (1u << m) >> pos.size();
    op.n_groups = static_cast<uint16_t>(groups);
    op.iters = static_cast<uint16_t>(std::max<uint32_t>(1, groups / kTileThreads));
    for (uint32_t j = 0; j < op.iters; ++j)
        op.dhi[j] = static_cast<uint16_t>(tile_swizzle(deposit(j * kTileThreads, pos) | lcmask));
}

}  // namespace

double local_op_flops(const LocalOp& o, bool x_free) {
    if (o.kind == kTilePauli) return o.lt.empty() ? 6.0 : 16.0;   // op_flops_per_amp of PAULI
    if (o.kind == kTileRot) return 4.0;
    const double frac = std::ldexp(1.0, -(__builtin_popcount(o.lmask) + __builtin_popcountll(o.gcmask)));
    if (o.kind != kTileDense) return 6.0 * frac;
    if (x_free && !o.variant && o.lt.size() == 1 && o.sel.empty() && is_x_matrix(o.m)) return 0.0;
    return 8.0 * std::ldexp(1.0, static_cast<int>(o.lt.size())) * frac;
}

// Matrix of a 2^k dense op with a one-qubit matrix applied first on its target bit j:
// M' = M (I (x) .. u .. (x) I).  Both sides may carry selector blocks: `ms` / `us` give the
// bit of each op's selector qubit within the merged selector set.
static void fold_into(LocalOp& q, const LocalOp& p, uint32_t j, const std::vector<uint32_t>& sel,
                      bool after = false) {
    const uint32_t k = static_cast<uint32_t>(q.lt.size());
    const uint64_t D = uint64_t{1} << k;
    const uint32_t nsel = static_cast<uint32_t>(sel.size());
    auto index_of = [&](const std::vector<uint32_t>& own, uint32_t sv) {
        uint32_t idx = 0;
        for (size_t i = 0; i < own.size(); ++i) {
            const uint32_t pos = static_cast<uint32_t>(std::find(sel.begin(), sel.end(), own[i]) - sel.begin());
            if ((sv >> pos) & 1) idx |= 1u << i;
        }
        return idx;
    };
    std::vector<cd> out;
    for (uint32_t sv = 0; sv < (1u << nsel); ++sv) {
        const cd* m = q.m.data() + static_cast<size_t>(index_of(q.sel, sv)) * D * D;
        std::array<cd, 4> u{};
        const uint32_t pi = index_of(p.sel, sv);
        if (p.kind == kTileDiag) {
            u = {p.m[2 * pi], cd{0, 0}, cd{0, 0}, p.m[2 * pi + 1]};
        } else {
            for (int e = 0; e < 4; ++e) u[e] = p.m[4 * pi + e];
        }
        for (uint64_t r = 0; r < D; ++r) {
            for (uint64_t c = 0; c < D; ++c) {
                cl acc{0, 0};
                if (after) {
                    // (U M)[r][c] = sum_x U[r_j][x] M[r with bit j = x][c]
                    const uint64_t rj = (r >> j) & 1, r0 = r & ~(uint64_t{1} << j);
                    for (uint64_t xj = 0; xj < 2; ++xj)
                        acc += wide_mul(u[rj * 2 + xj], m[(r0 | xj << j) * D + c]);
                } else {
                    // (M U)[r][c] = sum_x M[r][x] U[x][c]; U acts on bit j only
                    const uint64_t cj = (c >> j) & 1, c0 = c & ~(uint64_t{1} << j);
                    for (uint64_t xj = 0; xj < 2; ++xj)
                        acc += wide_mul(m[r * D + (c0 | xj << j)], u[xj * 2 + cj]);
                }
                out.push_back(narrow(acc));
            }
        }
    }
    q.m = std::move(out);
    q.wide.clear();
    q.sel = sel;
}

// Diagonal form of a phase or diagonal op without local controls: local bits (ascending)
// and the 2^k entries.  A phase multiplies where all its bits are 1.
static bool diagonal_form(const LocalOp& o, std::vector<uint32_t>& bits, std::vector<cd>& d) {
    if (o.variant || !o.sel.empty() || !o.dyn.empty()) return false;
    if (o.kind == kTilePhase) {
        bits.clear();
        for (uint32_t b = 0; b < 32; ++b)
            if ((o.lmask >> b) & 1) bits.push_back(b);
        d.assign(size_t{1} << bits.size(), cd{1, 0});
        d.back() = o.m[0];
        return true;
    }
    if (o.kind != kTileDiag || o.lmask) return false;
    // entries in local order (bit j <-> lt[j]); re-index to ascending bits
    std::vector<uint32_t> order(o.lt.size());
    for (size_t j = 0; j < order.size(); ++j) order[j] = static_cast<uint32_t>(j);
    std::sort(order.begin(), order.end(), [&](uint32_t a, uint32_t b) { return o.lt[a] < o.lt[b]; });
    bits.clear();
    for (uint32_t j : order) bits.push_back(o.lt[j]);
    const size_t D = size_t{1} << bits.size();
    d.assign(D, cd{1, 0});
    for (size_t e = 0; e < D; ++e) {
        size_t src = 0;
        for (size_t q = 0; q < order.size(); ++q)
            if ((e >> q) & 1) src |= size_t{1} << order[q];
        d[e] = o.m[src];
    }
    return true;
}

// Product of two diagonals given over ascending tile bits: the table over the union.
static void mul_tables(std::vector<uint32_t>& bi, std::vector<cd>& di, const std::vector<uint32_t>& bj,
                       const std::vector<cd>& dj) {
    uint32_t uni = 0;
    for (uint32_t b : bi) uni |= 1u << b;
    for (uint32_t b : bj) uni |= 1u << b;
    std::vector<uint32_t> ub;
    for (uint32_t b = 0; b < 32; ++b)
        if ((uni >> b) & 1) ub.push_back(b);
    std::vector<cd> du(size_t{1} << ub.size());
    for (size_t e = 0; e < du.size(); ++e) {
        size_t ei = 0, ej = 0;
        for (size_t q = 0; q < ub.size(); ++q) {
            if (!((e >> q) & 1)) continue;
            const auto pi = std::find(bi.begin(), bi.end(), ub[q]);
            if (pi != bi.end()) ei |= size_t{1} << (pi - bi.begin());
            const auto pj = std::find(bj.begin(), bj.end(), ub[q]);
            if (pj != bj.end()) ej |= size_t{1} << (pj - bj.begin());
        }
        du[e] = di[ei] * dj[ej];
    }
    bi = std::move(ub);
    di = std::move(du);
}

// Runs of diagonal work (phases such as the controlled phases of a QFT, diagonal blocks)
// become one diagonal table over the union of their tile bits: an op joins an earlier
// diagonal op when every op in between commutes with it (no dense target on its bits) and
// the union stays within max_bits.  Ops with the same out-of-tile predicate merge into the
// table itself.  With dyn_terms a phase gated by other out-of-tile qubits joins as a term
// that the kernel multiplies into the table at the start of each tile where those qubits are
// all 1 (a group whose own predicate differs turns into such terms when it is made of phases
// only).  Each merge removes a pass over the tile's amplitudes for a table entry lookup.
static void merge_diagonal_runs(std::vector<LocalOp>& ops, uint32_t max_bits, bool dyn_terms) {
    std::vector<char> dead(ops.size(), 0);
    std::vector<uint32_t> bi, bj;
    std::vector<cd> di, dj;
    uint32_t dyn_groups = 0, dyn_entries = 0;
    auto mask_of = [](const std::vector<uint32_t>& bits) {
        uint32_t mk = 0;
        for (uint32_t b : bits) mk |= 1u << b;
        return mk;
    };
    for (size_t i = 0; i < ops.size(); ++i) {
        if (dead[i] || !diagonal_form(ops[i], bi, di)) continue;
        uint64_t gc = ops[i].gcmask;
        std::vector<DynTerm> dyn;
        std::vector<DynTerm> phases;   // the group as phase terms while it is made of phases
        bool only_phases = ops[i].kind == kTilePhase;
        if (only_phases) phases.push_back({gc, ops[i].lmask, ops[i].m[0]});
        uint32_t merged = 0;
        uint32_t blocked = 0;   // tile bits a dense op between i and j targets
        for (size_t j = i + 1; j < ops.size(); ++j) {
            if (dead[j]) continue;
            const LocalOp& q = ops[j];
            if (diagonal_form(q, bj, dj)) {
                const uint32_t mj = mask_of(bj);
                const uint32_t uni = mask_of(bi) | mj;
                const uint32_t width = static_cast<uint32_t>(__builtin_popcount(uni));
                const bool fits = !(mj & blocked) && width <= max_bits &&
                                  (dyn.empty() || dyn_entries + (1u << width) <= kRegMaxDynEntries);
                if (fits && q.gcmask == gc) {
                    mul_tables(bi, di, bj, dj);
                    if (q.kind == kTilePhase) phases.push_back({q.gcmask, q.lmask, q.m[0]});
                    else only_phases = false;
                    dead[j] = 1;
                    ++merged;
                    continue;
                }
                // a gated phase as a per-tile term (table entries within the pass's budget)
                const bool room = dyn_entries + (1u << width) <= kRegMaxDynEntries &&
                                  (!dyn.empty() || dyn_groups < kRegMaxDyn) &&
                                  dyn.size() + (gc ? phases.size() : 0) < kRegMaxDynTerms;
                if (fits && dyn_terms && q.kind == kTilePhase && room && (gc == 0 || only_phases)) {
                    if (gc != 0) {   // the group so far becomes terms over an identity table
                        dyn = phases;
                        std::fill(di.begin(), di.end(), cd{1, 0});
                        gc = 0;
                    }
                    const std::vector<cd> ones(size_t{1} << bj.size(), cd{1, 0});
                    mul_tables(bi, di, bj, ones);
                    if (q.gcmask) dyn.push_back({q.gcmask, q.lmask, q.m[0]});
                    else mul_tables(bi, di, bj, dj);
                    phases.push_back({q.gcmask, q.lmask, q.m[0]});
                    dead[j] = 1;
                    ++merged;
                    continue;
                }
            }
            // q stays: later diagonal work may pass it only on bits it does not target
            if (q.kind == kTileDense || q.kind == kTilePauli)
                for (uint32_t b : q.lt) blocked |= 1u << b;
        }
        if (!merged) continue;   // a lone op keeps its own (cheaper) form
        LocalOp& o = ops[i];
        o.kind = kTileDiag;
        o.lt = bi;
        o.lmask = 0;
        o.gcmask = gc;
        o.m = di;
        o.dyn = std::move(dyn);
        if (!o.dyn.empty()) {
            ++dyn_groups;
            dyn_entries += 1u << o.lt.size();
        }
    }
    size_t w = 0;
    for (size_t i = 0; i < ops.size(); ++i) {
        if (dead[i]) continue;
        if (w != i) ops[w] = std::move(ops[i]);
        ++w;
    }
    ops.resize(w);
}

// Peephole after inner fusion: a one-qubit dense or diagonal op (no controls) moves into the
// next op touching its qubit — or, failing that, the previous one — when that op is a dense
// block on it without controls (the ops in between do not touch the qubit, so they commute
// with it): the block's matrix absorbs it at no extra cost per amplitude and one operation
// disappears.  A noise slot (per-state matrix) folds too: the block becomes per-state.
// In rotation form a diagonal stays out of one-qubit blocks: it is free in a table, and with a
// damping factor a block would have no rotation form any more (16 flops per amplitude, not 4).
static void fold_single_qubit_ops(std::vector<LocalOp>& ops, uint32_t max_select, bool rot) {
    std::vector<char> dead(ops.size(), 0);
    for (size_t i = 0; i < ops.size(); ++i) {
        // a phase on one tile bit (such as K0 of amplitude damping) folds as the diagonal
        // (1, f); if it does not fold it keeps its phase form
        LocalOp as_diag;
        const bool one_bit_phase = ops[i].kind == kTilePhase && !ops[i].gcmask &&
                                   ops[i].sel.empty() && __builtin_popcount(ops[i].lmask) == 1;
        if (one_bit_phase) {
            as_diag.kind = kTileDiag;
            as_diag.lt = {static_cast<uint32_t>(__builtin_ctz(ops[i].lmask))};
            as_diag.m = {cd{1, 0}, ops[i].m[0]};
        }
        const LocalOp& p = one_bit_phase ? as_diag : ops[i];
        if (p.kind == kTilePhase || p.kind == kTilePauli || p.lt.size() != 1 || p.lmask ||
            p.gcmask || !p.dyn.empty())
            continue;
        const uint32_t a = p.lt[0];
        for (size_t j = i + 1; j < ops.size(); ++j) {
            if (dead[j]) continue;
            LocalOp& q = ops[j];
            const bool touches = ((q.lmask >> a) & 1) ||
                                 std::find(q.lt.begin(), q.lt.end(), a) != q.lt.end();
            if (!touches) continue;
            const auto it = std::find(q.lt.begin(), q.lt.end(), a);
            if (q.kind == kTileDense && it != q.lt.end() && !q.lmask && !q.gcmask &&
                !(rot && q.lt.size() == 1 && p.kind == kTileDiag)) {
                std::vector<uint32_t> sel = q.sel;
                for (uint32_t s : p.sel)
                    if (std::find(sel.begin(), sel.end(), s) == sel.end()) sel.push_back(s);
                std::sort(sel.begin(), sel.end());
                if (sel.size() <= max_select || (p.sel.empty() && q.sel.size() <= max_select)) {
                    fold_into(q, p, static_cast<uint32_t>(it - q.lt.begin()), sel);
                    q.variant = q.variant || p.variant;
                    dead[i] = 1;
                }
            }
            break;   // only the next op on the qubit
        }
        if (dead[i]) continue;
        for (size_t j = i; j-- > 0;) {
            if (dead[j]) continue;
            LocalOp& q = ops[j];
            const bool touches = ((q.lmask >> a) & 1) ||
                                 std::find(q.lt.begin(), q.lt.end(), a) != q.lt.end();
            if (!touches) continue;
            const auto it = std::find(q.lt.begin(), q.lt.end(), a);
            if (q.kind == kTileDense && it != q.lt.end() && !q.lmask && !q.gcmask &&
                !(rot && q.lt.size() == 1 && p.kind == kTileDiag)) {
                std::vector<uint32_t> sel = q.sel;
                for (uint32_t s : p.sel)
                    if (std::find(sel.begin(), sel.end(), s) == sel.end()) sel.push_back(s);
                std::sort(sel.begin(), sel.end());
                if (sel.size() <= max_select || (p.sel.empty() && q.sel.size() <= max_select)) {
                    fold_into(q, p, static_cast<uint32_t>(it - q.lt.begin()), sel, true);
                    q.variant = q.variant || p.variant;
                    dead[i] = 1;
                }
            }
            break;   // only the previous op on the qubit
        }
    }
    size_t w = 0;
    for (size_t i = 0; i < ops.size(); ++i) {
        if (dead[i]) continue;
        if (w != i) ops[w] = std::move(ops[i]);
        ++w;
    }
    ops.resize(w);
}

// M = diag(l0, l1) L diag(1, r1) E with L = [[1, x], [y, 1 + x y]] (a0 += x a1, then
// a1 += y a0) and real x, y; E: the exchange of the two halves where `exchange`, else the
// identity.  Every unitary has this form with |x| <= 1, |y| <= 1/2: up to row scales L is then a
// rotation by at most 45 degrees, so the two FMAs round like one, and L needs no register
// besides the pair.  Real matrices and some others have it too; false for the rest.  l0 and l1
// carry the row norms that rounding x and y would change (a drift of the state's norm, which
// would add up over the gates).
static bool rotation_split(const LocalOp& o, bool& exchange, cl& r1, double& x, double& y, cl& l0,
                           cl& l1) {
    auto entry = [&](int e) { return o.wide.empty() ? cl{o.m[e]} : o.wide[e]; };
    cl a = entry(0), b = entry(1), c = entry(2), d = entry(3);
    exchange = std::max(std::abs(b), std::abs(c)) > std::max(std::abs(a), std::abs(d));
    if (exchange) {
        std::swap(a, b);
        std::swap(c, d);
    }
    const long double ad = std::min(std::abs(a), std::abs(d));
    if (!(ad > 0.0L) || !(std::max(std::abs(b), std::abs(c)) <= 1.001L * ad)) return false;
    l0 = a;
    l1 = d;
    r1 = 1.0L;
    x = y = 0.0;
    if (b == cl{0, 0} && c == cl{0, 0}) return true;
    const cl via_b = b / a, via_c = c / d;   // X r1 and Y / r1 of the rows (1, X), (Y, 1)
    r1 = std::abs(via_b) >= std::abs(via_c) ? via_b / std::abs(via_b)
                                            : std::conj(via_c) / std::abs(via_c);
    const cl xc = wide_mul(via_b, std::conj(r1)), yc = wide_mul(via_c, r1);
    if (std::abs(xc.imag()) > 1e-15L || std::abs(yc.imag()) > 1e-15L) return false;
    const long double X = xc.real(), Y = yc.real(), det = 1.0L - X * Y;
    if (det < 0.25L) return false;   // nearly singular
    x = static_cast<double>(X);
    y = static_cast<double>(Y / det);
    const long double s1 = 1.0L + static_cast<long double>(x) * y;
    l0 *= std::sqrt((1.0L + X * X) / (1.0L + static_cast<long double>(x) * x));
    l1 = wide_mul(d, std::conj(r1)) * std::sqrt((1.0L + Y * Y) / (static_cast<long double>(y) * y + s1 * s1));
    return true;
}

// Uncontrolled one-qubit dense operations as diagonal, real rotation, diagonal.  One whose
// matrix differs per state keeps the same three operations for every state.
static void split_rotations(std::vector<LocalOp>& ops) {
    std::vector<LocalOp> out;
    out.reserve(2 * ops.size());
    const cl one{1, 0};
    for (LocalOp& o : ops) {
        bool ex = false;
        cl r1, l0, l1;
        double x = 0, y = 0;
        if (o.kind != kTileDense || o.lt.size() != 1 || o.lmask || o.gcmask || !o.sel.empty() ||
            (!o.variant && is_x_matrix(o.m)) || !rotation_split(o, ex, r1, x, y, l0, l1)) {
            out.push_back(std::move(o));
            continue;
        }
        LocalOp before, rot, after;
        before.kind = after.kind = kTileDiag;
        rot.kind = kTileRot;
        before.lt = rot.lt = after.lt = o.lt;
        before.variant = rot.variant = after.variant = o.variant;
        // diag(1, r1) E = E diag(r1, 1)
        before.wide = ex ? std::vector<cl>{r1, one} : std::vector<cl>{one, r1};
        rot.m = {cd{x, y}};
        rot.exchange = ex;
        after.wide = {l0, l1};
        for (LocalOp* d : {&before, &after}) d->m = {narrow(d->wide[0]), narrow(d->wide[1])};
        if (o.variant || r1 != one) out.push_back(std::move(before));
        out.push_back(std::move(rot));
        if (o.variant || l0 != one || l1 != one) out.push_back(std::move(after));
    }
    ops = std::move(out);
}

std::vector<LocalOp> pass_local_ops(const PlanItem& item, const std::vector<GateDesc>& gates,
                                    const TileConfig& cfg, uint32_t max_select,
                                    const std::vector<std::array<cd, 4>>* slot_mats,
                                    uint32_t max_diag, bool dyn_terms,
                                    std::vector<uint32_t>* store_qubits, bool native_rotations,
                                    bool rot) {
    LocalMap lm{cfg.L, item.hbits, {}};
    std::vector<LocalOp> out;
    // a noise slot takes this state's matrix (identity when no table is given)
    auto resolved = [&](const GateDesc& g) {
        GateDesc r = g;
        if (g.slot) {
            r.type = LQCS_GATE_UNITARY;
            r.mat.assign(4, cd{0, 0});
            r.mat[0] = r.mat[3] = 1.0;
            if (slot_mats) r.mat.assign((*slot_mats)[g.slot_id].begin(), (*slot_mats)[g.slot_id].end());
        }
        return r;
    };
    // inner fusion: greedy blocks of at most cfg.inner local qubits (targets and local
    // controls) and at most max_select out-of-tile controls; any other gate closes the
    // blocks it touches and is emitted on its own
    struct Open {
        std::vector<uint32_t> qubits;   // local part, global numbering, sorted
        std::vector<uint32_t> sel;      // out-of-tile controls, sorted
        std::vector<uint32_t> gates;
        bool alive = true;
    };
    std::vector<Open> open;
    std::vector<int> owner(64, -1);
    auto emit_single = [&](const GateDesc& g) {
        if (is_phase_gate(g)) {
            LocalOp op;
            op.kind = kTilePhase;
            for (uint32_t q : g.qubits) {
                const int l = lm.local(q);
                if (l >= 0) op.lmask |= 1u << l;
                else op.gcmask |= uint64_t{1} << q;
            }
            op.m.push_back(g.base_matrix()[3]);
            if (!g.wide.empty()) op.wide = {g.wide[3]};
            out.push_back(std::move(op));
            return;
        }
        std::vector<uint32_t> lt;
        for (uint32_t j = 0; j < g.base_qubits(); ++j)
            lt.push_back(static_cast<uint32_t>(lm.local(g.targets()[j])));
        uint32_t lc = 0;
        uint64_t gc = 0;
        for (uint32_t c = 0; c < g.n_controls; ++c) {
            const uint32_t q = g.controls()[c];
            const int l = lm.local(q);
            if (l >= 0) lc |= 1u << l;
            else gc |= uint64_t{1} << q;
        }
        out.push_back(matrix_op(resolved(g).base_matrix(), lt, lc, gc, g.slot));
        if (g.wide.size() == 4) {
            LocalOp& op = out.back();
            if (op.kind == kTileDiag) op.wide = {g.wide[0], g.wide[3]};
            else op.wide = g.wide;
        }
    };
    auto emit_block = [&](Open& b) {
        if (!b.alive) return;
        b.alive = false;
        for (uint32_t q : b.qubits) owner[q] = -1;
        if (b.gates.size() == 1) {   // keeps the cheaper single-gate encodings (controls, X)
            emit_single(gates[b.gates[0]]);
            return;
        }
        std::vector<uint32_t> lt;
        for (uint32_t q : b.qubits) lt.push_back(static_cast<uint32_t>(lm.local(q)));
        FusedBlock fb;
        fb.qubits = b.qubits;
        bool variant = false;
        for (uint32_t gi : b.gates) variant |= gates[gi].slot;
        if (b.sel.empty()) {
            std::vector<GateDesc> res;
            for (uint32_t gi : b.gates) {
                fb.gates.push_back(static_cast<uint32_t>(res.size()));
                res.push_back(resolved(gates[gi]));
            }
            const std::vector<cl> wide = block_matrix_wide(fb, res);
            std::vector<cd> m;
            for (const cl& z : wide) m.push_back(narrow(z));
            out.push_back(matrix_op(m, lt, 0, 0, variant));
            if (lt.size() == 1 && out.back().kind == kTileDense) out.back().wide = wide;
            return;
        }
        // one matrix per value s of the out-of-tile controls (bit i of s = qubit sel[i]): a
        // gate acts, without those controls, where all of its own are 1 and is the identity
        // elsewhere
        const uint32_t c = static_cast<uint32_t>(b.sel.size());
        const uint64_t dim = uint64_t{1} << lt.size();
        std::vector<std::vector<cd>> mats;
        bool diag = true;
        for (uint32_t sv = 0; sv < (1u << c); ++sv) {
            std::vector<GateDesc> red;
            for (uint32_t gi : b.gates) {
                const GateDesc g = resolved(gates[gi]);
                GateDesc r = g;
                r.qubits.clear();
                r.n_controls = 0;
                bool on = true;
                for (uint32_t k = 0; k < g.n_controls; ++k) {
                    const uint32_t q = g.controls()[k];
                    if (lm.local(q) >= 0) {
                        r.qubits.push_back(q);
                        ++r.n_controls;
                    } else {
                        const auto it = std::find(b.sel.begin(), b.sel.end(), q);
                        on &= ((sv >> (it - b.sel.begin())) & 1u) != 0;
                    }
                }
                for (uint32_t j = 0; j < g.base_qubits(); ++j) r.qubits.push_back(g.targets()[j]);
                if (on) red.push_back(std::move(r));
            }
            fb.gates.clear();
            for (uint32_t i = 0; i < red.size(); ++i) fb.gates.push_back(i);
            mats.push_back(block_matrix(fb, red));
            diag &= !variant && is_diagonal(mats.back(), dim);
        }
        LocalOp op;
        op.kind = diag ? kTileDiag : kTileDense;
        op.lt = lt;
        op.sel = b.sel;
        op.variant = variant;
        for (const std::vector<cd>& m : mats) {
            if (diag) {
                for (uint64_t i = 0; i < dim; ++i) op.m.push_back(m[i * dim + i]);
            } else {
                op.m.insert(op.m.end(), m.begin(), m.end());
            }
        }
        out.push_back(std::move(op));
    };

    for (uint32_t gi : item.gates) {
        const GateDesc& g = gates[gi];
        // a native Pauli rotation: closes the blocks on its tile qubits and runs on its own
        if (native_rotations && native_pauli(g, cfg)) {
            for (uint32_t q : g.qubits)
                if (lm.local(q) >= 0 && owner[q] >= 0) emit_block(open[owner[q]]);
            const PauliMasks pm = pauli_local_masks(g.pauli);
            LocalOp op;
            op.kind = kTilePauli;
            uint64_t xg = 0, zg = 0;
            for (uint32_t j = 0; j < g.base_qubits(); ++j) {
                const uint32_t q = g.targets()[j];
                const int l = lm.local(q);
                if ((pm.x >> j) & 1) {
                    if (l < 0) logic("tile lowering: a Pauli rotation flips a qubit outside the tile");
                    op.lt.push_back(static_cast<uint32_t>(l));
                    xg |= uint64_t{1} << q;
                }
                if ((pm.zy >> j) & 1) {
                    zg |= uint64_t{1} << q;
                    if (l >= 0) op.lmask |= 1u << l;
                    else op.pz_out |= uint64_t{1} << q;
                }
            }
            std::sort(op.lt.begin(), op.lt.end());
            // y = (-i sin) i^n_Y, as apply_pauli_rotation forms it, times (-1)^parity(x & zy)
            const double h = g.params.at(0) / 2;
            static const cd kIPow[4] = {{1, 0}, {0, 1}, {-1, 0}, {0, -1}};
            cd y = cd{0.0, -std::sin(h)} * kIPow[pm.n_y % 4];
            if (__builtin_popcountll(xg & zg) & 1) y = -y;
            op.m = {cd{std::cos(h), 0.0}, y};
            out.push_back(std::move(op));
            continue;
        }
        // a SWAP of two tile qubits moves no data: the two tile bits trade qubits for the rest
        // of the pass, and the store writes each tile bit to its qubit's place
        if (store_qubits && g.type == LQCS_GATE_SWAP && g.n_controls == 0 && !g.slot &&
            g.qubits.size() == 2 && lm.local(g.qubits[0]) >= 0 && lm.local(g.qubits[1]) >= 0) {
            for (uint32_t q : g.qubits)
                if (owner[q] >= 0) emit_block(open[owner[q]]);
            lm.swap_bits(g.qubits[0], g.qubits[1]);
            continue;
        }
        std::vector<uint32_t> part, sel;   // local qubits; out-of-tile controls
        for (uint32_t q : g.qubits) (lm.local(q) >= 0 ? part : sel).push_back(q);
        std::sort(part.begin(), part.end());
        std::sort(sel.begin(), sel.end());
        if (cfg.inner < 2 || is_phase_gate(g) || part.size() > cfg.inner || sel.size() > max_select) {
            for (uint32_t q : part)
                if (owner[q] >= 0) emit_block(open[owner[q]]);
            emit_single(g);
            continue;
        }
        std::vector<int> touched;
        for (uint32_t q : part)
            if (owner[q] >= 0 && std::find(touched.begin(), touched.end(), owner[q]) == touched.end())
                touched.push_back(owner[q]);
        std::vector<uint32_t> uni = part, usel = sel;
        for (int b : touched) {
            uni.insert(uni.end(), open[b].qubits.begin(), open[b].qubits.end());
            usel.insert(usel.end(), open[b].sel.begin(), open[b].sel.end());
        }
        std::sort(uni.begin(), uni.end());
        uni.erase(std::unique(uni.begin(), uni.end()), uni.end());
        std::sort(usel.begin(), usel.end());
        usel.erase(std::unique(usel.begin(), usel.end()), usel.end());
        Open nb;
        if (uni.size() > cfg.inner || usel.size() > max_select) {
            for (int b : touched) emit_block(open[b]);
            nb.qubits = part;
            nb.sel = sel;
            nb.gates = {gi};
        } else {
            nb.qubits = uni;
            nb.sel = usel;
            for (int b : touched) {
                nb.gates.insert(nb.gates.end(), open[b].gates.begin(), open[b].gates.end());
                open[b].alive = false;
            }
            std::sort(nb.gates.begin(), nb.gates.end());
            nb.gates.push_back(gi);
        }
        const int id = static_cast<int>(open.size());
        for (uint32_t q : nb.qubits) owner[q] = id;
        open.push_back(std::move(nb));
    }
    for (Open& b : open) emit_block(b);
    // one-qubit ops first go into the dense blocks on their qubits (free); the diagonal
    // work left over then merges into tables
    fold_single_qubit_ops(out, max_select, rot);
    if (rot) split_rotations(out);
    else merge_diagonal_runs(out, max_diag, dyn_terms);
    if (store_qubits) {   // qubit each tile bit holds at the end of the pass
        const uint32_t m = cfg.L + static_cast<uint32_t>(item.hbits.size());
        store_qubits->assign(m, 0);
        for (uint32_t b = 0; b < m; ++b) {
            const uint32_t q = b < cfg.L ? b : item.hbits[b - cfg.L];
            (*store_qubits)[static_cast<uint32_t>(lm.local(q))] = q;
        }
    }
    return out;
}

void lower_pass(const PlanItem& item, const std::vector<GateDesc>& gates, const TileConfig& cfg,
                TilePass& pass, std::vector<TileOp>& ops_out, std::vector<cd>& arena,
                double* flops_per_amp) {
    pass = TilePass{};
    pass.L = cfg.L;
    pass.h = static_cast<uint32_t>(item.hbits.size());
    pass.m = cfg.L + pass.h;
    for (uint32_t i = 0; i < pass.h; ++i) pass.hbits[i] = item.hbits[i];
    const size_t first = ops_out.size();
    double flops = 0.0;
    for (const LocalOp& lo : pass_local_ops(item, gates, cfg, 0)) {
        flops += local_op_flops(lo, false);
        TileOp op{};
        op.kind = lo.kind;
        op.gcmask = lo.gcmask;
        op.mat_off = static_cast<uint32_t>(arena.size());
        arena.insert(arena.end(), lo.m.begin(), lo.m.end());
        if (lo.kind == kTilePhase) {
            std::vector<uint32_t> fixed;
            for (uint32_t b = 0; b < 32; ++b)
                if ((lo.lmask >> b) & 1) fixed.push_back(b);
            set_groups(op, fixed, lo.lmask, pass.m);
        } else {
            const uint32_t k = static_cast<uint32_t>(lo.lt.size());
            op.k = static_cast<uint8_t>(k);
            for (uint32_t l = 0; l < (1u << k); ++l) {
                uint32_t o = 0;
                for (uint32_t j = 0; j < k; ++j)
                    if ((l >> j) & 1) o |= 1u << lo.lt[j];
                op.soff[l] = static_cast<uint16_t>(tile_swizzle(o));
            }
            std::vector<uint32_t> fixed = lo.lt;
            for (uint32_t b = 0; b < 32; ++b)
                if ((lo.lmask >> b) & 1) fixed.push_back(b);
            set_groups(op, fixed, lo.lmask, pass.m);
        }
        ops_out.push_back(op);
    }
    pass.n_ops = static_cast<uint32_t>(ops_out.size() - first);
    if (flops_per_amp) *flops_per_amp = flops;
    pass.kmax = 1;
    for (size_t i = first; i < ops_out.size(); ++i)
        if (ops_out[i].kind != kTilePhase) pass.kmax = std::max<uint32_t>(pass.kmax, ops_out[i].k);
}

// ------------------------------------------------------------------ register passes

namespace {

constexpr uint32_t kLaneBits = 5;

uint32_t target_mask(const LocalOp& o) {
    uint32_t t = 0;
    for (uint32_t b : o.lt) t |= 1u << b;
    return t;
}

bool off_diagonal(const LocalOp& o) {
    return o.kind == kTileDense || o.kind == kTilePauli || o.kind == kTileRot;
}

// Tile bits an op uses off the diagonal (dense targets) and on it (controls, phase bits,
// diagonal targets).  Two ops commute when every bit they share is diagonal in both.
struct Use {
    uint32_t nd = 0, dg = 0;
};
Use op_use(const LocalOp& o) {
    Use u;
    if (off_diagonal(o)) u.nd = target_mask(o);
    else if (o.kind == kTileDiag) u.dg = target_mask(o);
    u.dg |= o.lmask;
    return u;
}

// A layout as the scheduler sees it: register set S, warp bits W and the pair P of tile
// bits on lanes 0 and 1 (0: none), where the two-qubit blocks of a tensor-core pass run.
struct Lay {
    uint32_t S = 0, W = 0, P = 0;
};

// Whether op o runs in layout ly: a dense op on the tensor path (mma) needs its targets
// (two, or one) on the lane pair and its tile controls on register or warp bits (every lane
// of a warp takes part in the instruction); any other dense op needs its targets on
// register bits.
bool fits(const LocalOp& o, bool mma, const Lay& ly) {
    if (o.kind == kTilePauli) return (target_mask(o) & ly.W) == 0;   // flips on registers, lanes
    if (o.kind == kTileRot) return (target_mask(o) & ~ly.S) == 0;
    if (o.kind != kTileDense) return true;
    if (mma) return ly.P != 0 && (target_mask(o) & ~ly.P) == 0 && (o.lmask & ~(ly.S | ly.W)) == 0;
    return (target_mask(o) & ~ly.S) == 0;
}

// Scan of the pending ops under layout ly: every op that commutes with all skipped ops
// before it and fits the layout is applied.  The applied ops move to `emitted` (in order) and
// `pending` keeps the rest.  mma[i]: op i is a tensor-path op.
void scan(const std::vector<LocalOp>& ops, const std::vector<Use>& use,
          const std::vector<uint8_t>& mma, std::vector<uint32_t>& pending, const Lay& ly,
          std::vector<uint32_t>& emitted) {
    uint32_t busy_nd = 0, busy_dg = 0;
    std::vector<uint32_t> rest;
    for (uint32_t i : pending) {
        const Use& u = use[i];
        const bool blocked = (u.nd & (busy_nd | busy_dg)) != 0 || (u.dg & busy_nd) != 0;
        if (!blocked && fits(ops[i], mma[i] != 0, ly)) {
            emitted.push_back(i);
        } else {
            busy_nd |= u.nd;
            busy_dg |= u.dg;
            rest.push_back(i);
        }
    }
    pending = std::move(rest);
}

// Layout of register set S, warp bits W and lane pair P on an m-bit tile.  Thread-index bits
// 0..4 (the lanes) take the tile bits outside S and W, bits 5.. (the warps) take W in
// ascending order.  With a pair, lanes 0 and 1 take its lower and higher bit and lane 2 a
// bit of the third residue mod 3 where one exists; otherwise lanes ascending, except that
// when they are not tile bits 0..4 the first three are picked with distinct residues mod 3:
// tile_swizzle sends 1 << b to slot bit (b mod 3), so then the 8 lanes of a quarter warp hit
// 8 different 16-byte bank groups in a remap.  A remap that keeps W keeps every warp on the
// same tile indices, hence on its own shared-memory slots: it needs only a warp-level
// barrier.
RegLayout make_layout(uint32_t S, uint32_t W, uint32_t m, uint32_t P = 0) {
    RegLayout ly{};
    std::vector<uint32_t> rb, lanes, warps;
    for (uint32_t b = 0; b < m; ++b) {
        if ((S >> b) & 1) rb.push_back(b);
        else if ((W >> b) & 1) warps.push_back(b);
        else if (!((P >> b) & 1)) lanes.push_back(b);
    }
    if (P != 0) {
        const uint32_t p0 = static_cast<uint32_t>(__builtin_ctz(P));
        const uint32_t p1 = 31u - static_cast<uint32_t>(__builtin_clz(P));
        const uint32_t seen = (1u << (p0 % 3)) | (1u << (p1 % 3));
        for (size_t i = 0; i < lanes.size(); ++i)
            if (!((seen >> (lanes[i] % 3)) & 1)) {
                std::rotate(lanes.begin(), lanes.begin() + static_cast<long>(i),
                            lanes.begin() + static_cast<long>(i) + 1);
                break;
            }
        lanes.insert(lanes.begin(), {p0, p1});
    } else if (lanes.size() >= 3 && lanes[0] + lanes.size() - 1 != lanes.back()) {
        std::vector<uint32_t> first, rest;
        uint32_t seen = 0;
        for (uint32_t b : lanes) {
            if (first.size() < 3 && !((seen >> (b % 3)) & 1)) {
                first.push_back(b);
                seen |= 1u << (b % 3);
            } else {
                rest.push_back(b);
            }
        }
        lanes = first;
        lanes.insert(lanes.end(), rest.begin(), rest.end());
    }
    std::vector<uint32_t> tb = lanes;
    tb.insert(tb.end(), warps.begin(), warps.end());
    for (uint32_t i = 0; i < kRegBits; ++i) {
        ly.rpos[i] = static_cast<uint8_t>(rb[i]);
        ly.rsw[i] = static_cast<uint16_t>(tile_swizzle(1u << rb[i]));
    }
    for (uint32_t i = 0; i < tb.size(); ++i) {
        ly.tpos[i] = static_cast<uint8_t>(tb[i]);
        ly.tsw[i] = static_cast<uint16_t>(tile_swizzle(1u << tb[i]));
    }
    return ly;
}

// Whether the tile bits in `lanes` cover all three residues mod 3 (see make_layout).
bool residues_spread(uint32_t lanes) {
    uint32_t seen = 0;
    for (uint32_t b = 0; b < 32; ++b)
        if ((lanes >> b) & 1) seen |= 1u << (b % 3);
    return seen == 7u;
}

// `count` warp bits out of `avail`: the tile bits the pending dense operations target least
// (ties: the higher bit), so that few later operations need a bit that is a warp bit.
uint32_t pick_warp_bits(const std::vector<LocalOp>& ops, const std::vector<uint32_t>& pending,
                        uint32_t avail, uint32_t count, uint32_t pair = 0) {
    uint32_t usage[32] = {};
    for (uint32_t i : pending)
        if (off_diagonal(ops[i]))
            for (uint32_t b : ops[i].lt) ++usage[b];
    uint32_t W = 0;
    for (uint32_t k = 0; k < count; ++k) {
        int best = -1;
        for (int b = 31; b >= 0; --b) {
            if (!((avail >> b) & 1) || ((W >> b) & 1)) continue;
            if (best < 0 || usage[b] < usage[best]) best = b;
        }
        if (best >= 0) W |= 1u << best;
    }
    // lanes (the rest of avail and the lane pair) without a residue mod 3: trade a warp bit
    // for a lane bit as little used
    if (!residues_spread((avail & ~W) | pair)) {
        for (uint32_t w = 0; w < 32; ++w) {
            if (!((W >> w) & 1)) continue;
            for (uint32_t l = 0; l < 32; ++l) {
                const uint32_t W2 = (W & ~(1u << w)) | (1u << l);
                if (((avail & ~W) >> l) & 1 && usage[l] <= usage[w] &&
                    residues_spread((avail & ~W2) | pair))
                    return W2;
            }
        }
    }
    return W;
}

// The register set of size kRegBits inside `allowed` that contains `must` and is best by
// (ops applied now with warp bits W and lane pair P, register-path dense ops covered later — a
// tie-break: later use of a layout —, usable as the final layout, and — when the warp bits are
// known, `lane_pool` being the tile bits outside them — lanes that take all three residues mod 3,
// which keeps the remaps free of bank conflicts).  The first of equals in ascending order.
// Most of the time of planning a new circuit goes into these scans, so they run over masks
// alone, from one table per call, and end where every tile bit is blocked.
uint32_t choose_set(const std::vector<LocalOp>& ops, const std::vector<Use>& use,
                    const std::vector<uint8_t>& mma, const std::vector<uint32_t>& pending,
                    uint32_t must, uint32_t allowed, uint32_t m, bool rot, uint32_t lane_pool = 0,
                    uint32_t P = 0, uint32_t W = 0) {
    struct Row {
        uint32_t nd, dg;   // Use
        uint32_t need;     // bits that must be register bits (all ones: it never fits)
        uint32_t counts;   // rotation form: diagonals cost no layout
    };
    std::vector<Row> rows;
    rows.reserve(pending.size());
    uint32_t single[32] = {};              // register-path dense ops by target, and the targets of
    std::vector<uint32_t> several;         // those with more than one
    for (uint32_t i : pending) {
        const LocalOp& o = ops[i];
        const uint32_t t = target_mask(o);
        const bool off = off_diagonal(o);
        // fits(), for the part that does not depend on the set
        uint32_t need = 0;
        if (o.kind == kTilePauli) need = (t & W) == 0 ? 0u : ~0u;
        else if (o.kind == kTileRot) need = t;
        else if (o.kind == kTileDense && !mma[i]) need = t;
        else if (o.kind == kTileDense) need = P != 0 && (t & ~P) == 0 ? o.lmask & ~W : ~0u;
        rows.push_back({use[i].nd, use[i].dg, need, !rot || off ? 1u : 0u});
        if (!off || mma[i]) continue;
        if (o.lt.size() == 1) ++single[o.lt[0]];
        else several.push_back(t);
    }
    uint32_t best = 0;
    size_t best_now = 0, best_later = 0;
    bool best_final = false, best_spread = false, have = false;
    const uint32_t lanes = (1u << kLaneBits) - 1u, all = (1u << m) - 1u;
    // every set: `must` and `more` of the `free` bits, ascending (the next number with as many ones)
    std::vector<uint32_t> sets;
    const uint32_t free = allowed & ~must & all;
    const int n_free = __builtin_popcount(free), more = static_cast<int>(kRegBits) - __builtin_popcount(must);
    if (more < 0 || more > n_free) return 0;
    for (uint32_t pick = (1u << more) - 1u; pick < (1u << n_free);) {
        uint32_t S = must;
        for (uint32_t f = free, x = pick; x; f &= f - 1, x >>= 1)
            if (x & 1u) S |= f & (~f + 1u);
        sets.push_back(S);
        if (pick == 0) break;   // `must` alone
        const uint32_t low = pick & (~pick + 1u), up = pick + low;
        pick = up | (((pick ^ up) / low) >> 2);
    }
    constexpr size_t kLanes = 16;   // sets scanned side by side (vector instructions)
    for (size_t s0 = 0; s0 < sets.size(); s0 += kLanes) {
        const size_t n_sets = std::min(kLanes, sets.size() - s0);
        uint32_t S[kLanes] = {}, busy_nd[kLanes] = {}, busy_dg[kLanes] = {}, now[kLanes] = {};
        std::copy_n(sets.begin() + static_cast<long>(s0), n_sets, S);
        for (size_t i = 0; i < rows.size(); ++i) {
            const Row r = rows[i];
            for (size_t l = 0; l < kLanes; ++l) {
                const uint32_t clash = (r.nd & (busy_nd[l] | busy_dg[l])) | (r.dg & busy_nd[l]) | (r.need & ~S[l]);
                const uint32_t waits = clash != 0 ? ~0u : 0u;
                now[l] += r.counts & ~waits;
                busy_nd[l] |= r.nd & waits;
                busy_dg[l] |= r.dg & waits;
            }
            if (rot && i % 8 == 7) {   // (what touches no bit does not count there)
                uint32_t blocked = all;
                for (size_t l = 0; l < n_sets; ++l) blocked &= busy_nd[l];
                if (blocked == all) break;
            }
        }
        for (size_t l = 0; l < n_sets; ++l) {
            if (have && now[l] < best_now) continue;
            size_t later = 0;
            for (uint32_t b = S[l]; b; b &= b - 1) later += single[__builtin_ctz(b)];
            for (uint32_t t : several) later += (t & ~S[l]) == 0;
            const bool fin = (S[l] & lanes) == 0;
            const bool spread = lane_pool != 0 && residues_spread(lane_pool & ~S[l]);
            const size_t count = now[l];
            if (!have || std::make_tuple(count, later, fin, spread) >
                             std::make_tuple(best_now, best_later, best_final, best_spread)) {
                have = true;
                best = S[l];
                best_now = count;
                best_later = later;
                best_final = fin;
                best_spread = spread;
            }
        }
    }
    return best;
}

}  // namespace

namespace {

// A term of a per-tile diagonal, for the entries e with (e & bits) == value: the factor, then
// {gcmask low 32 bits, gcmask high 32 bits * 4096 + value * 64 + bits} as exact integers.
void append_term(const cd& f, uint64_t gcmask, uint32_t bits, uint32_t value, std::vector<cd>& mats) {
    mats.push_back(f);
    mats.emplace_back(static_cast<double>(gcmask & 0xffffffffu),
                      static_cast<double>((gcmask >> 32) * 4096u + value * 64u + bits));
}

// Matrix data of op o in layout (ly, S): dense matrices re-indexed so that matrix bit q is
// the q-th lowest register target (one block per selector value), diagonals and phase
// factors as they are.  X operations (swaps) have none.
// A tensor-path op (mma) instead: matrix bit 0 is the tile bit on lane 0, bit 1 the one on
// lane 1.
void append_matrices(const LocalOp& o, const RegLayout& ly, uint32_t S, std::vector<cd>& mats,
                     bool mma = false) {
    if (mma) {
        std::vector<cd> pm(16);
        if (o.lt.size() == 1) {   // one target: the 2 x 2 matrix on its lane, identity on the other
            const uint32_t j = o.lt[0] == ly.tpos[0] ? 0u : 1u;
            for (size_t blk = 0; blk < o.m.size(); blk += 4) {
                for (uint32_t rr = 0; rr < 4; ++rr)
                    for (uint32_t cc = 0; cc < 4; ++cc)
                        pm[rr * 4 + cc] = ((rr ^ cc) >> (1u - j)) & 1u
                                              ? cd{0, 0}
                                              : o.m[blk + ((rr >> j) & 1u) * 2 + ((cc >> j) & 1u)];
                mats.insert(mats.end(), pm.begin(), pm.end());
            }
            return;
        }
        const bool swap = o.lt[0] != ly.tpos[0];   // matrix bit 0 is on lane 1
        auto sw = [&](uint32_t l) { return swap ? ((l & 1u) << 1) | (l >> 1) : l; };
        for (size_t blk = 0; blk < o.m.size(); blk += 16) {
            for (uint32_t rr = 0; rr < 4; ++rr)
                for (uint32_t cc = 0; cc < 4; ++cc) pm[sw(rr) * 4 + sw(cc)] = o.m[blk + rr * 4 + cc];
            mats.insert(mats.end(), pm.begin(), pm.end());
        }
        return;
    }
    if (o.kind == kTilePauli) {   // (cos, 0), y, the out-of-tile Z-type qubits as two halves
        mats.insert(mats.end(), o.m.begin(), o.m.end());
        mats.emplace_back(static_cast<double>(o.pz_out & 0xffffffffu),
                          static_cast<double>(o.pz_out >> 32));
        return;
    }
    if (o.kind == kTilePhase || o.kind == kTileDiag) {
        mats.insert(mats.end(), o.m.begin(), o.m.end());
        for (const DynTerm& t : o.dyn) {
            uint32_t em = 0;
            for (size_t j = 0; j < o.lt.size(); ++j)
                if ((t.lbits >> o.lt[j]) & 1) em |= 1u << j;
            append_term(t.f, t.gcmask, em, em, mats);
        }
        return;
    }
    const uint32_t k = static_cast<uint32_t>(o.lt.size());
    if (k == 1 && !o.variant && o.sel.empty() && is_x_matrix(o.m)) return;
    int ridx[32];
    for (uint32_t i = 0; i < kRegBits; ++i) ridx[ly.rpos[i]] = static_cast<int>(i);
    uint32_t tm = 0;
    for (uint32_t b : o.lt) tm |= 1u << ridx[b];
    (void)S;
    std::vector<uint32_t> pos(k);
    for (uint32_t j = 0; j < k; ++j) {
        const uint32_t rb = static_cast<uint32_t>(ridx[o.lt[j]]);
        pos[j] = static_cast<uint32_t>(__builtin_popcount(tm & ((1u << rb) - 1u)));
    }
    const uint32_t D = 1u << k;
    std::vector<uint32_t> perm(D);
    for (uint32_t l = 0; l < D; ++l) {
        uint32_t p = 0;
        for (uint32_t j = 0; j < k; ++j)
            if ((l >> j) & 1) p |= 1u << pos[j];
        perm[l] = p;
    }
    std::vector<cd> pm(D * D);
    for (size_t blk = 0; blk < o.m.size(); blk += D * D) {   // per selector value
        for (uint32_t rr = 0; rr < D; ++rr)
            for (uint32_t cc = 0; cc < D; ++cc) pm[perm[rr] * D + perm[cc]] = o.m[blk + rr * D + cc];
        mats.insert(mats.end(), pm.begin(), pm.end());
    }
}

// The record of op o in layout (ly, S); its matrices start at mat_off.  mma: a two-qubit
// block on the lane pair (tensor path), its controls on register or warp bits.
RegOp make_record(const LocalOp& o, const RegLayout& ly, uint32_t S, uint32_t m, uint32_t mat_off,
                  bool mma = false) {
    int ridx[32], tidx[32];
    for (uint32_t i = 0; i < kRegBits; ++i) ridx[ly.rpos[i]] = static_cast<int>(i);
    for (uint32_t i = 0; i < m - kRegBits; ++i) tidx[ly.tpos[i]] = static_cast<int>(i);
    RegOp r{};
    r.gcmask = o.gcmask;
    r.mat_off = mat_off;
    r.nsel = static_cast<uint8_t>(o.sel.size());
    for (size_t i = 0; i < o.sel.size(); ++i) r.selq[i] = static_cast<uint8_t>(o.sel[i]);
    for (uint32_t b = 0; b < m; ++b) {
        if (!((o.lmask >> b) & 1)) continue;
        if ((S >> b) & 1) r.rcmask = static_cast<uint8_t>(r.rcmask | (1u << ridx[b]));
        else r.tcmask = static_cast<uint16_t>(r.tcmask | (1u << tidx[b]));
    }
    const uint32_t k = static_cast<uint32_t>(o.lt.size());
    r.k = static_cast<uint8_t>(k);
    if (mma) {
        if (r.tcmask & ((1u << kLaneBits) - 1u))
            logic("register tile lowering: a tensor-path block is controlled by a lane bit");
        r.kind = kRegMma;
        r.k = 2;   // always a 4 x 4 block (a one-target op with the identity on the other lane)
    } else if (o.kind == kTilePauli) {   // Z-type tile bits went to rcmask / tcmask above
        r.kind = kRegPauli;
        r.k = 0;
        for (uint32_t b : o.lt) {
            if ((S >> b) & 1) {
                r.code = static_cast<uint8_t>(r.code | (1u << ridx[b]));
            } else {
                if (tidx[b] >= static_cast<int>(kLaneBits))
                    logic("register tile lowering: a Pauli rotation flips a warp bit");
                r.loc[0] = static_cast<uint8_t>(r.loc[0] | (1u << tidx[b]));
            }
        }
    } else if (o.kind == kTilePhase) {
        r.kind = kRegPhase;
    } else if (o.kind == kTileDiag) {
        r.kind = o.dyn.empty() ? kRegDiag : kRegDiagDyn;
        r.nterm = static_cast<uint8_t>(o.dyn.size());
        for (uint32_t j = 0; j < k; ++j) {
            const uint32_t b = o.lt[j];
            r.loc[j] = static_cast<uint8_t>((S >> b) & 1 ? ridx[b] : (0x80 | tidx[b]));
        }
    } else {
        uint32_t tm = 0;
        for (uint32_t b : o.lt) tm |= 1u << ridx[b];
        r.code = static_cast<uint8_t>(tm);
        r.kind = (k == 1 && !o.variant && o.sel.empty() && is_x_matrix(o.m)) ? kRegSwapX : kRegDense;
    }
    return r;
}

bool same_shape(const LocalOp& a, const LocalOp& b) {
    return a.kind == b.kind && a.lt == b.lt && a.lmask == b.lmask && a.gcmask == b.gcmask &&
           a.sel == b.sel && a.m.size() == b.m.size() && a.variant == b.variant &&
           a.dyn.size() == b.dyn.size() && (a.variant || a.exchange == b.exchange);
}

// The records of a schedule and the matrices of one state.
struct Emitted {
    std::vector<RegOp> rec;
    std::vector<cd> mats;
    std::vector<uint32_t> dyn_rec;   // records of per-tile diagonals, and their table entries
    uint32_t dyn_entries = 0;
    uint32_t sign_off = 0;           // the sign masks among the matrices
    double flops = 0.0;
    // Tile bits stored negated: an X (or the exchange a rotation starts with) costs nothing but
    // a bit in here, which later records are written for and the tile's store undoes.
    uint32_t flipped = 0;
    bool failed = false;             // an operation that cannot be written for a negated bit
    bool per_state = false;          // some matrix, hence `flipped`, differs per state: the
                                     // records may depend on neither

    void remap(uint32_t layout, bool local) {
        close();
        RegOp r{};
        r.kind = kRegRemap;
        r.code = static_cast<uint8_t>(layout);
        r.k = local ? 1 : 0;
        rec.push_back(r);
    }
    void add(const LocalOp& o, const RegLayout& ly, uint32_t S, uint32_t m, bool mma) {
        close();
        push(make_record(o, ly, S, m, static_cast<uint32_t>(mats.size()), mma));
        append_matrices(o, ly, S, mats, mma);
        flops += local_op_flops(o, true);
    }
    void push(RegOp r) {
        if (r.kind == kRegDiagDyn || (r.kind == kRegStage && r.nterm)) {
            (r.kind == kRegStage ? r.dyn_table : r.dyn_off) = static_cast<uint16_t>(dyn_entries);
            dyn_entries += 1u << r.k;
            dyn_rec.push_back(static_cast<uint32_t>(rec.size()));
        }
        rec.push_back(r);
    }
    // Neighbouring rotations on different register bits become one record, with the table that
    // precedes them.  xy: the rotation's two factors; signs: the outside qubits of the Z on its
    // bit.
    void rotate(const LocalOp& o, const RegLayout& ly, const cd& xy, uint64_t signs) {
        uint32_t r = 0;
        while (ly.rpos[r] != o.lt[0]) ++r;
        for (const Rot& x : rots_)
            if (x.bit == r) {
                close();
                break;
            }
        rots_.push_back({r, xy, signs});
        flops += local_op_flops(o, true);
    }
    void close() {
        if (rots_.empty()) return;
        std::sort(rots_.begin(), rots_.end(), [](const Rot& a, const Rot& b) { return a.bit < b.bit; });
        const bool after_table = !rec.empty() && rec.back().kind == kRegStage && rec.back().code == 0;
        if (!after_table) {
            RegOp r{};
            r.kind = kRegStage;
            rec.push_back(r);
        }
        RegOp& r = rec.back();
        r.dyn_off = static_cast<uint16_t>(mats.size());
        bool any = false;
        for (const Rot& x : rots_) {
            r.code = static_cast<uint8_t>(r.code | (1u << x.bit));
            mats.push_back(x.xy);
            any |= x.signs != 0;
        }
        // where the tile's sign words hold this record's signs; too many of them in one pass:
        // the masks follow the factors
        r.tcmask = kRegSignBits;
        if (any && signs.size() + rots_.size() <= kRegSignBits) {
            r.tcmask = static_cast<uint16_t>(signs.size());
            for (const Rot& x : rots_) signs.push_back(x.signs);
        } else if (any) {
            r.tcmask = kRegSignBits + 1;
            for (const Rot& x : rots_) mats.emplace_back(std::bit_cast<double>(x.signs), 0.0);
        }
        rots_.clear();
    }
    std::vector<uint64_t> signs;     // masks of the rotations' signs, in record order

  private:
    struct Rot {
        uint32_t bit;
        cd xy;
        uint64_t signs;
    };
    std::vector<Rot> rots_;
};

// Diagonal work of a pass in rotation form that waits for the next operation which needs it:
// diagonals commute with each other, so each waits until an operation is about to mix one of
// its tile bits, and then goes out in one table with everything else that fits beside it.
class DiagonalPool {
  public:
    // compact: strided tables of at most six bits (64 entries) where an expanded one has up to
    // 136: slower to read (an address per entry), for passes whose matrices would outgrow their
    // stage.
    explicit DiagonalPool(bool compact) : compact_(compact) {}
    static bool takes(const LocalOp& o) {
        if (o.kind == kTilePhase)
            return __builtin_popcount(o.lmask) <= static_cast<int>(kRegMaxDiag);
        return o.kind == kTileDiag && !o.lmask && !o.gcmask && o.sel.empty() && o.dyn.empty() &&
               o.lt.size() <= kRegMaxDiag;
    }
    void put(const LocalOp& o) { items_.push_back({&o, bits_of(o)}); }
    bool touches(uint32_t bits) const {
        for (const Item& it : items_)
            if (it.bits & bits) return true;
        return false;
    }
    // Emits one table that takes waiting operations on bits of `touch`.
    void flush(uint32_t touch, Emitted& e, const RegLayout& ly, uint32_t S, uint32_t m) {
        emit(group(touch, S), e, ly, S, m);
    }
    void flush_all(Emitted& e, const RegLayout& ly, uint32_t S, uint32_t m) {
        while (!items_.empty()) {
            uint32_t touch = 0;
            for (const Item& it : items_) touch |= it.bits;
            emit(touch ? group(touch, S) : 0u, e, ly, S, m);
        }
    }

  private:
    struct Item {
        const LocalOp* op;
        uint32_t bits;
    };
    std::vector<Item> items_;
    bool compact_;

    static uint32_t bits_of(const LocalOp& o) { return o.kind == kTilePhase ? o.lmask : target_mask(o); }
    static int width(uint32_t bits) { return __builtin_popcount(bits); }

    // Bits joined to `from` by waiting operations.
    uint32_t closure(uint32_t from) const {
        uint32_t c = from;
        for (bool grew = true; grew;) {
            grew = false;
            for (const Item& it : items_)
                if ((it.bits & c) && (it.bits & ~c)) {
                    c |= it.bits;
                    grew = true;
                }
        }
        return c;
    }

    // Tile bits of the next table: whole components of joined bits while they fit, first those
    // with a bit of `touch`; if the first is too wide, as much of it as fits.  Fitting: at most
    // three thread bits beside the register bits S (an expanded table); with gated phases about,
    // where nothing fits so, or compact, six bits (a strided one, which a tile may build).
    uint32_t group(uint32_t touch, uint32_t S) const {
        bool gated = compact_;
        for (const Item& it : items_) gated |= it.op->kind == kTilePhase && it.op->gcmask != 0;
        for (int strided = gated ? 1 : 0; strided < 2; ++strided) {
            auto fits = [&](uint32_t bits) {
                return strided ? width(bits) <= static_cast<int>(kRegMaxDiag)
                               : width(bits & ~S) <= static_cast<int>(kRegTableThreadBits);
            };
            uint32_t u = 0;
            for (int round = 0; round < 2; ++round)
                for (const Item& it : items_) {
                    if ((it.bits & u) || (round == 0 && !(it.bits & touch))) continue;
                    const uint32_t c = closure(it.bits);
                    if (!(c & u) && fits(u | c)) u |= c;
                }
            if (u & touch) return u;
            u = 0;
            for (int round = 0; round < 2; ++round)   // what touches, then what is joined to that
                for (const Item& it : items_)
                    if ((it.bits & (round ? u : touch)) && fits(u | it.bits)) u |= it.bits;
            if (u & touch) return u;
        }
        logic("register tile lowering: a diagonal too wide for a table");
    }

    // One table over the tile bits `u`: the product of every waiting operation within them,
    // formed in extended precision.  Its entry bits go lanes first (then warp bits, then
    // register bits), so that the lanes of a warp read neighbouring entries.
    void emit(uint32_t u, Emitted& e, const RegLayout& ly, uint32_t S, uint32_t m) {
        RegOp r{};
        std::vector<uint32_t> bits;
        const bool narrow_enough = !compact_ && width(u & ~S) <= static_cast<int>(kRegTableThreadBits);
        for (uint8_t& l : r.loc) l = 31;
        for (uint32_t i = 0; i < m - kRegBits; ++i)
            if ((u >> ly.tpos[i]) & 1) {
                r.loc[bits.size()] = static_cast<uint8_t>(i);
                bits.push_back(ly.tpos[i]);
            }
        uint8_t* const reg_offset[kRegBits] = {&r.nsel, &r.selq[0], &r.selq[1], &r.rcmask};
        for (uint32_t i = 0; i < kRegBits; ++i)
            if ((u >> ly.rpos[i]) & 1) {
                *reg_offset[i] = static_cast<uint8_t>(1u << bits.size());
                bits.push_back(ly.rpos[i]);
            }
        const uint32_t k = static_cast<uint32_t>(bits.size()), size = 1u << k;
        r.k = static_cast<uint8_t>(k);
        uint32_t entry_bit[32] = {};
        for (uint32_t j = 0; j < k; ++j) entry_bit[bits[j]] = 1u << j;
        auto entry_mask = [&](uint32_t from) {
            uint32_t x = 0;
            for (uint32_t b = from; b; b &= b - 1) x |= entry_bit[__builtin_ctz(b)];
            return x;
        };
        const bool dyn_room = e.dyn_rec.size() < kRegMaxDyn && e.dyn_entries + size <= kRegMaxDynEntries;
        std::vector<const LocalOp*> members, gated, alone;
        size_t w = 0;
        for (const Item& it : items_) {
            if (it.bits & ~u) {
                items_[w++] = it;
                continue;
            }
            if (it.op->kind != kTilePhase || it.op->gcmask == 0) members.push_back(it.op);
            else if (dyn_room && gated.size() < kRegMaxDynTerms)
                gated.push_back(it.op);
            else alone.push_back(it.op);
        }
        items_.resize(w);
        // a lone phase is cheaper on its own
        if (members.size() + gated.size() == 1 && !e.per_state && !(u & e.flipped) &&
            (members.empty() ? gated : members)[0]->kind == kTilePhase) {
            alone.insert(alone.end(), members.begin(), members.end());
            alone.insert(alone.end(), gated.begin(), gated.end());
            members.clear();
            gated.clear();
        }
        if (!members.empty() || !gated.empty()) {
            const cl one{1, 0};
            cl bit[kRegBits + kRegMaxDiag][2];
            for (uint32_t j = 0; j < k; ++j) bit[j][0] = bit[j][1] = one;
            for (const LocalOp* o : members) {   // one-bit factors first: a product per bit
                if (o->kind == kTileDiag && o->lt.size() == 1) {
                    const uint32_t j = static_cast<uint32_t>(__builtin_ctz(entry_bit[o->lt[0]]));
                    for (int x = 0; x < 2; ++x)
                        bit[j][x] = wide_mul(bit[j][x], o->wide.empty() ? cl{o->m[x]} : o->wide[x]);
                } else if (o->kind == kTilePhase && width(o->lmask) == 1) {
                    cl& f = bit[static_cast<uint32_t>(__builtin_ctz(entry_mask(o->lmask)))][1];
                    f = wide_mul(f, phase(*o));
                }
            }
            cl table[1u << (kRegBits + kRegTableThreadBits)];
            std::fill_n(table, size, one);
            for (uint32_t j = 0; j < k; ++j)
                for (uint32_t x = 0; x < (1u << j); ++x) {
                    table[x | (1u << j)] = bit[j][1] == one ? table[x] : wide_mul(table[x], bit[j][1]);
                    if (bit[j][0] != one) table[x] = wide_mul(table[x], bit[j][0]);
                }
            for (const LocalOp* o : members) {
                if (o->kind == kTilePhase) {
                    if (width(o->lmask) == 1) continue;
                    const uint32_t em = entry_mask(o->lmask);
                    for (uint32_t x = 0; x < size; ++x)
                        if ((x & em) == em) table[x] = wide_mul(table[x], phase(*o));
                } else if (o->lt.size() != 1) {
                    for (uint32_t x = 0; x < size; ++x) {
                        uint32_t src = 0;
                        for (size_t j = 0; j < o->lt.size(); ++j)
                            if (x & entry_bit[o->lt[j]]) src |= 1u << j;
                        table[x] = wide_mul(table[x], o->m[src]);
                    }
                }
            }
            e.close();
            r.kind = kRegStage;
            r.table = gated.empty() && narrow_enough ? kRegTableExpanded : kRegTableStrided;
            r.nterm = static_cast<uint8_t>(gated.size());
            r.mat_off = static_cast<uint32_t>(e.mats.size());
            const uint32_t flip = entry_mask(u & e.flipped);
            cd entry[1u << (kRegBits + kRegTableThreadBits)];
            for (uint32_t x = 0; x < size; ++x) entry[x] = narrow(table[x ^ flip]);
            if (r.table == kRegTableExpanded) {
                const uint32_t threads = 1u << width(u & ~S), row = (1u << kRegBits) + 1;
                uint32_t offset[1u << kRegBits] = {};
                for (uint32_t v = 1; v < (1u << kRegBits); ++v)
                    offset[v] = offset[v & (v - 1)] + *reg_offset[__builtin_ctz(v)];
                e.mats.resize(e.mats.size() + threads * row);   // the row's last entry is not read
                cd* out = e.mats.data() + r.mat_off;
                for (uint32_t t = 0; t < threads; ++t, out += row)
                    for (uint32_t v = 0; v < (1u << kRegBits); ++v) out[v] = entry[t + offset[v]];
            } else {
                e.mats.insert(e.mats.end(), entry, entry + size);
            }
            for (const LocalOp* o : gated) {
                const uint32_t em = entry_mask(o->lmask);
                append_term(o->m[0], o->gcmask, em, em & ~flip, e.mats);
            }
            e.push(r);
            e.flops += 6.0;
        }
        for (const LocalOp* o : alone) {
            e.failed |= (o->lmask & e.flipped) != 0;
            e.add(*o, ly, S, m, false);
        }
    }
    static cl phase(const LocalOp& o) { return o.wide.empty() ? cl{o.m[0]} : o.wide[0]; }
};

// Signs of a pass in rotation form that cost nothing until something cannot take them: a CZ
// between tile bit b and a qubit outside is a Z on b in the tiles where that qubit is 1, and a
// CZ between two qubits outside negates whole tiles.
class PendingSigns {
  public:
    explicit PendingSigns(uint32_t m) : m_(m) {}
    bool take(const LocalOp& o, uint32_t flipped) {
        if (o.kind != kTilePhase || !o.gcmask || o.m[0] != cd{-1, 0}) return false;
        if (o.lmask == 0) {
            if (whole_.size() >= 31u - m_) return false;
            whole_.push_back(o.gcmask);
            used_ = true;
            return true;
        }
        if (__builtin_popcount(o.lmask) != 1 || __builtin_popcountll(o.gcmask) != 1) return false;
        z_[__builtin_ctz(o.lmask)] ^= o.gcmask;
        if (o.lmask & flipped) odd_ ^= o.gcmask;   // Z X = - X Z
        used_ = true;
        return true;
    }
    // The outside qubits whose parity puts a Z on an odd number of the tile bits `bits`.
    uint64_t on(uint32_t bits) const {
        uint64_t f = 0;
        for (uint32_t b = bits; b; b &= b - 1) f ^= z_[__builtin_ctz(b)];
        return f;
    }
    bool any(uint32_t bits) const {
        for (uint32_t b = bits; b; b &= b - 1)
            if (z_[__builtin_ctz(b)]) return true;
        return false;
    }
    // Applies the signs on the tile bits `bits`; at the end of the pass all that is left.
    void apply(uint32_t bits, bool last, Emitted& e, const RegLayout& ly) {
        if (last ? !used_ : !any(bits)) return;
        e.close();
        RegOp r{};
        r.kind = kRegSign;
        r.mat_off = static_cast<uint32_t>(e.mats.size());
        auto put = [&](uint64_t f) { e.mats.emplace_back(std::bit_cast<double>(f), 0.0); };
        auto mask = [&](uint32_t b) {
            uint64_t f = 0;
            if ((bits >> b) & 1) std::swap(f, z_[b]);
            put(f);
        };
        for (uint32_t i = 0; i < m_ - kRegBits; ++i) mask(ly.tpos[i]);
        for (uint32_t i = 0; i < kRegBits; ++i) mask(ly.rpos[i]);
        put(last ? odd_ : 0);
        if (last)
            for (uint64_t f : whole_) put(f);
        r.nterm = static_cast<uint8_t>(m_ + 1 + (last ? whole_.size() : 0));
        e.push(r);
    }

  private:
    uint32_t m_;
    uint64_t z_[32] = {};
    uint64_t odd_ = 0;               // outside qubits whose parity negates the tile
    std::vector<uint64_t> whole_;    // outside qubits that negate it where they are all 1
    bool used_ = false;
};

// How the records of a pass in rotation form are written: with bits stored negated, with
// compact tables.
struct RotVariant {
    bool flips = true, compact = false;
};

// Records and matrices of the schedule `seq` for the operations of one state.  In rotation
// form the operations of one layout go out in the order that leaves diagonals waiting longest:
// whatever mixes a bit that nothing waits on goes first, and a table is emitted only when
// every operation that is left needs one.  What waits on the bits that the next layout mixes
// goes out before the remap, while those bits are thread bits: a thread then loads one entry
// per register bit of the table that is left.
void emit_schedule(const std::vector<LocalOp>& ops, const std::vector<Use>& use,
                   const std::vector<uint8_t>& mma,
                   const std::vector<std::pair<int, uint32_t>>& seq,
                   const std::vector<RegLayout>& lays, const std::vector<Lay>& keys, uint32_t m,
                   const std::vector<uint32_t>& store_q, bool rot, RotVariant variant, Emitted& e) {
    DiagonalPool pool(variant.compact);
    std::deque<LocalOp> scales;   // diagonals of mirrored rotations (the pool keeps pointers)
    uint32_t cur = 0;
    if (rot) e.mats.emplace_back(0.0, 0.0);   // what the store undoes
    // bits that controls of records look at are never stored negated
    uint32_t keep = variant.flips ? 0u : ~0u;
    for (const LocalOp& o : ops) {
        e.per_state |= o.variant;
        if (!DiagonalPool::takes(o) && o.kind != kTilePauli) {
            keep |= o.lmask;
            if (o.kind == kTileDiag) keep |= target_mask(o);
        }
    }
    auto exchange = [&](uint32_t bit) {   // the halves of tile bit `bit` trade places
        if (!((keep >> bit) & 1)) {
            e.flipped ^= 1u << bit;
            return;
        }
        LocalOp x;
        x.lt = {bit};
        x.m = {cd{0, 0}, cd{1, 0}, cd{1, 0}, cd{0, 0}};
        e.add(x, lays[cur], keys[cur].S, m, false);
    };
    PendingSigns signs(m);
    std::vector<uint32_t> todo, rest;   // of the current layout
    auto apply = [&](const LocalOp& o) {
        const RegLayout& ly = lays[cur];
        const uint32_t t = target_mask(o);
        const bool x_op = o.kind == kTileDense && !o.variant && !o.lmask && !o.gcmask &&
                          o.sel.empty() && is_x_matrix(o.m);
        if (o.kind == kTileRot) {
            const uint32_t b = o.lt[0];
            if (o.exchange && ((keep >> b) & 1)) {
                if (o.variant) e.failed = true;   // records may not differ between states
                signs.apply(t, false, e, ly);
            }
            if (o.exchange) exchange(b);
            const bool mirrored = (e.flipped & t) != 0;
            // On a negated bit the rotation is [[1 + x y, y], [x, 1]] = diag(e0, e1) [[1, p],
            // [q, 1 + p q]]: the same two steps with other factors, and a diagonal that joins
            // the one waiting behind it (there in every state of a batch).
            cd xy = o.m[0];
            cl e0{1, 0}, e1{1, 0};
            if (mirrored) {
                const long double x = xy.real(), y = xy.imag(), s = 1.0L + x * y, P = y / s,
                                  Q = x / (1.0L - P * x);
                xy = cd{static_cast<double>(P), static_cast<double>(Q)};
                const long double p = xy.real(), q = xy.imag(), r = 1.0L + p * q;
                e0 = std::sqrt((s * s + y * y) / (1.0L + p * p));
                e1 = std::sqrt((x * x + 1.0L) / (q * q + r * r));
            }
            e.rotate(o, ly, xy, signs.on(t));
            if (mirrored || e.per_state) {
                LocalOp& d = scales.emplace_back();
                d.kind = kTileDiag;
                d.lt = o.lt;
                d.variant = e.per_state;
                d.wide = {e1, e0};   // of the true bit, the stored one negated
                d.m = {narrow(e1), narrow(e0)};
                pool.put(d);
            }
        } else if (x_op && !(keep & t)) {
            e.flipped ^= t;
        } else if (o.kind == kTilePauli) {
            LocalOp p = o;   // a Z flips the sign of a string with X or Y on its bit, an X of
            p.pz_out ^= signs.on(t);   // one with Z or Y
            if (__builtin_popcount(e.flipped & o.lmask) & 1) p.m[1] = -p.m[1];
            e.add(p, ly, keys[cur].S, m, false);
        } else {
            if (off_diagonal(o)) signs.apply(t, false, e, ly);
            if (o.kind == kTileDense && (e.flipped & t)) {
                LocalOp d = o;
                uint32_t f = 0;
                for (size_t j = 0; j < o.lt.size(); ++j) f |= ((e.flipped >> o.lt[j]) & 1u) << j;
                const uint32_t D = 1u << o.lt.size();
                for (size_t blk = 0; blk < o.m.size(); blk += D * D)
                    for (uint32_t r = 0; r < D; ++r)
                        for (uint32_t c = 0; c < D; ++c)
                            d.m[blk + (r ^ f) * D + (c ^ f)] = o.m[blk + r * D + c];
                e.add(d, ly, keys[cur].S, m, false);
                return;
            }
            e.add(o, ly, keys[cur].S, m, false);
        }
    };
    auto drain = [&] {
        while (!todo.empty()) {
            bool moved = false;
            uint32_t busy_nd = 0, busy_dg = 0, waits = 0;
            rest.clear();
            for (uint32_t i : todo) {
                const Use& u = use[i];
                const bool blocked = (u.nd & (busy_nd | busy_dg)) != 0 || (u.dg & busy_nd) != 0;
                if (!blocked && !off_diagonal(ops[i]) && DiagonalPool::takes(ops[i])) {
                    if (!signs.take(ops[i], e.flipped)) pool.put(ops[i]);
                    moved = true;
                } else if (!blocked && !pool.touches(u.nd)) {
                    apply(ops[i]);
                    moved = true;
                } else {
                    if (!blocked) waits |= u.nd;
                    busy_nd |= u.nd;
                    busy_dg |= u.dg;
                    rest.push_back(i);
                }
            }
            todo.swap(rest);
            if (!moved && !todo.empty()) pool.flush(waits, e, lays[cur], keys[cur].S, m);
        }
    };
    for (size_t k = 0; k < seq.size(); ++k) {
        const auto [i, l] = seq[k];
        if (i < 0) {
            drain();
            uint32_t next = 0;
            for (size_t j = k + 1; j < seq.size() && seq[j].first >= 0; ++j) next |= use[seq[j].first].nd;
            while (rot && pool.touches(next)) pool.flush(next, e, lays[cur], keys[cur].S, m);
            e.remap(l, i == -1);   // warp-local
        } else if (rot) {
            todo.push_back(static_cast<uint32_t>(i));
        } else {
            e.add(ops[i], lays[l], keys[l].S, m, mma[i] != 0);
        }
        cur = l;
    }
    drain();
    pool.flush_all(e, lays[cur], keys[cur].S, m);
    signs.apply((1u << m) - 1u, true, e, lays[cur]);
    e.close();
    if (rot) {
        uint64_t undo = 0;
        for (uint32_t b = e.flipped; b; b &= b - 1) undo ^= uint64_t{1} << store_q[__builtin_ctz(b)];
        e.mats[0] = cd{std::bit_cast<double>(undo), 0.0};
        e.sign_off = static_cast<uint32_t>(e.mats.size());
        for (uint64_t f : e.signs) e.mats.emplace_back(std::bit_cast<double>(f), 0.0);
    }
}

// selects: set if some block takes one of several matrices, so that fewer selector qubits would
// leave fewer matrices.
bool lower_pass_reg_sel(const PlanItem& item, const std::vector<GateDesc>& gates,
                        const TileConfig& cfg, uint32_t max_select, bool rot, RegPass& pass,
                        std::vector<RegOp>& ops_out, std::vector<RegLayout>& layouts_out,
                        std::vector<cd>& mats_out, double* flops_per_amp,
                        const std::vector<std::vector<std::array<cd, 4>>>* state_slots, bool& selects) {
    const uint32_t m = cfg.L + static_cast<uint32_t>(item.hbits.size());
    const std::vector<std::array<cd, 4>>* slots0 =
        state_slots && !state_slots->empty() ? &(*state_slots)[0] : nullptr;
    std::vector<uint32_t> store_q;
    const std::vector<LocalOp> ops =
        pass_local_ops(item, gates, cfg, max_select, slots0, kRegMaxDiag, true, &store_q, true, rot);
    selects = false;
    for (const LocalOp& o : ops) selects |= !o.sel.empty();
    for (const LocalOp& o : ops)
        if (o.kind != kTilePhase && o.kind != kTilePauli && o.kind != kTileRot &&
            o.lt.size() > (o.kind == kTileDense ? kRegMaxK : kRegMaxDiag))
            return false;
    std::vector<Use> use;
    for (const LocalOp& o : ops) use.push_back(op_use(o));
    // One- and two-target dense blocks run on the FP64 tensor path (lane pair) when cfg.mma
    // is set — all but X operations, which stay register swaps; their tile controls must fit
    // on the register bits, which at most kRegBits can.
    std::vector<uint8_t> mma(ops.size(), 0);
    for (size_t i = 0; i < ops.size(); ++i) {
        const LocalOp& o = ops[i];
        const size_t k = o.lt.size();
        const bool swapx = k == 1 && !o.variant && o.sel.empty() && is_x_matrix(o.m);
        mma[i] = cfg.mma && o.kind == kTileDense && (k == 2 || (k == 1 && !swapx)) &&
                 __builtin_popcount(o.lmask) <= static_cast<int>(kRegBits);
    }

    std::vector<RegLayout> lays;
    std::vector<Lay> lay_keys;
    auto layout_index = [&](uint32_t S, uint32_t W, uint32_t P) {
        if ((P != 0 && __builtin_popcount(P) != 2) || (P & (S | W)) != 0 || (S & W) != 0)
            logic("register tile lowering: inconsistent layout");
        for (size_t i = 0; i < lay_keys.size(); ++i)
            if (lay_keys[i].S == S && lay_keys[i].W == W && lay_keys[i].P == P)
                return static_cast<uint32_t>(i);
        lay_keys.push_back(Lay{S, W, P});
        lays.push_back(make_layout(S, W, m, P));
        return static_cast<uint32_t>(lay_keys.size() - 1);
    };
    // schedule: (op, layout) in application order, remaps as (-1 warp-local / -2 CTA-wide,
    // new layout)
    std::vector<std::pair<int, uint32_t>> seq;
    const uint32_t all = (1u << m) - 1u;
    const uint32_t lanes = (1u << kLaneBits) - 1u;
    const uint32_t high = all & ~lanes;
    const uint32_t nwarp = m - kRegBits - kLaneBits;
    std::vector<uint32_t> pending(ops.size());
    for (uint32_t i = 0; i < ops.size(); ++i) pending[i] = i;
    // Lane pair for tensor-path op i out of the tile bits `pool` (0: none there): its two
    // targets; for one target, the targets of a pending two-target block that contains it,
    // else the target and the lowest free bit of pool (one of `prefer` if there is one).
    auto pair_for = [&](uint32_t i, uint32_t pool, uint32_t prefer) -> uint32_t {
        const uint32_t t = target_mask(ops[i]);
        if ((t & ~pool) != 0) return 0u;
        if (ops[i].lt.size() == 2) return t;
        for (uint32_t j : pending) {
            const uint32_t tj = target_mask(ops[j]);
            if (mma[j] && ops[j].lt.size() == 2 && (tj & t) && !(tj & ~pool) && !(tj & ops[i].lmask))
                return tj;
        }
        const uint32_t free = pool & ~t & ~ops[i].lmask;
        if (free == 0) return 0u;
        const uint32_t pick = (free & prefer) ? (free & prefer) : free;
        return t | (1u << __builtin_ctz(pick));
    };
    // lane pair for a layout whose lanes are `pool`: that of the first pending tensor-path
    // block that has one there
    auto next_pair = [&](uint32_t pool) -> uint32_t {
        for (uint32_t i : pending)
            if (mma[i])
                if (const uint32_t pr = pair_for(i, pool, pool)) return pr;
        return 0u;
    };
    // the first layout loads the tile: lanes on tile bits 0..4 keep the loads coalesced
    uint32_t P = next_pair(lanes);
    uint32_t S = choose_set(ops, use, mma, pending, 0, high, m, rot, 0, P, 0);
    uint32_t W = pick_warp_bits(ops, pending, high & ~S, nwarp, P);
    uint32_t cur = layout_index(S, W, P);
    bool sync_tiles = false;
    while (true) {
        std::vector<uint32_t> applied;
        scan(ops, use, mma, pending, Lay{S, W, P}, applied);
        for (uint32_t i : applied) seq.emplace_back(static_cast<int>(i), cur);
        if (pending.empty()) break;
        const LocalOp& f = ops[pending.front()];
        if (mma[pending.front()]) {   // a tensor-path block: its targets become the lane pair
            P = pair_for(pending.front(), all, all & ~W);
            if ((P & W) == 0) {       // warp-local: the warp bits stay
                S = choose_set(ops, use, mma, pending, f.lmask & ~W, all & ~W & ~P, m, rot, all & ~W,
                               P, W);
                cur = layout_index(S, W, P);
                seq.emplace_back(-1, cur);
            } else {                  // a target is a warp bit: new warp bits, CTA-wide remap
                S = choose_set(ops, use, mma, pending, f.lmask, all & ~P, m, rot, 0, P, 0);
                W = pick_warp_bits(ops, pending, all & ~S & ~P, nwarp, P);
                cur = layout_index(S, W, P);
                seq.emplace_back(-2, cur);
                sync_tiles = true;
            }
            continue;
        }
        if (f.kind == kTilePauli) {   // its flips on warp bits: new warp bits outside them
            W = pick_warp_bits(ops, pending, all & ~target_mask(f), nwarp);
            S = choose_set(ops, use, mma, pending, 0, all & ~W, m, rot, all & ~W, 0, W);
            P = next_pair(all & ~W & ~S);
            cur = layout_index(S, W, P);
            seq.emplace_back(-2, cur);
            sync_tiles = true;
            continue;
        }
        const uint32_t must = target_mask(f);
        if ((must & W) == 0) {   // warp-local: the warp bits stay
            S = choose_set(ops, use, mma, pending, must, all & ~W, m, rot, all & ~W, 0, W);
            P = next_pair(all & ~W & ~S);
            cur = layout_index(S, W, P);
            seq.emplace_back(-1, cur);
        } else {                 // a target is a warp bit: new warp bits, CTA-wide remap
            S = choose_set(ops, use, mma, pending, must, all, m, rot);
            P = next_pair(all & ~S);
            W = pick_warp_bits(ops, pending, all & ~S & ~P, nwarp, P);
            cur = layout_index(S, W, P);
            seq.emplace_back(-2, cur);
            sync_tiles = true;
        }
    }
    // The store wants the lanes on the tile bits that hold qubits of tile bits 0..4 at the
    // load (the same bits unless a relabelling moved those qubits).
    uint32_t slanes = 0;
    for (uint32_t l = 0; l < kLaneBits; ++l) {
        const uint32_t q = l < cfg.L ? l : item.hbits[l - cfg.L];
        for (uint32_t b = 0; b < m; ++b)
            if (store_q[b] == q) slanes |= 1u << b;
    }
    const uint32_t shigh = all & ~slanes;
    if (((S | W) & slanes) != 0) {
        if ((W & slanes) == 0) {
            seq.emplace_back(-1, layout_index(shigh & ~W, W, 0));
        } else {
            uint32_t Sf = 0;   // the four highest tile bits outside the store lanes
            for (int b = static_cast<int>(m) - 1; b >= 0 && __builtin_popcount(Sf) < static_cast<int>(kRegBits); --b)
                if ((shigh >> b) & 1) Sf |= 1u << b;
            W = pick_warp_bits(ops, pending, shigh & ~Sf, nwarp);
            seq.emplace_back(-2, layout_index(Sf, W, 0));
            sync_tiles = true;
        }
    }

    // records and every state's matrices; the states share the records
    struct State {
        std::vector<LocalOp> ops;
        size_t same;   // the state with the same matrices in all of the pass's slots: most often
                       // there is no error at all, and such states share the work
    };
    std::vector<State> states;   // 1 and up
    if (state_slots) {
        std::map<std::string, size_t> known;   // slot matrices -> the state lowered for them
        auto key_of = [&](size_t b) {
            std::string k;
            for (uint32_t gi : item.gates)
                if (gates[gi].slot)
                    k.append(reinterpret_cast<const char*>((*state_slots)[b][gates[gi].slot_id].data()),
                             sizeof(std::array<cd, 4>));
            return k;
        };
        known.emplace(key_of(0), 0);
        for (size_t b = 1; b < state_slots->size(); ++b) {
            const auto [same, fresh] = known.emplace(key_of(b), b);
            states.push_back({{}, same->second});
            if (!fresh) continue;
            std::vector<uint32_t> store_b;
            states.back().ops = pass_local_ops(item, gates, cfg, max_select, &(*state_slots)[b],
                                               kRegMaxDiag, true, &store_b, true, rot);
            const std::vector<LocalOp>& ob = states.back().ops;
            if (ob.size() != ops.size() || store_b != store_q) return false;
            for (size_t i = 0; i < ops.size(); ++i)
                if (!same_shape(ops[i], ob[i])) return false;
        }
    }
    Emitted first;
    bool flipped = false;
    size_t n_mat = 0;
    enum Fit { kFits, kMatrices, kLimits, kForm };   // too many matrices, records, ...; a state whose
                                                     // operations these records cannot express
    auto emit = [&](RotVariant v) {
        first = Emitted{};
        emit_schedule(ops, use, mma, seq, lays, lay_keys, m, store_q, rot, v, first);
        if (first.failed) return kForm;
        if (first.rec.size() > kRegMaxRecords || lays.size() > kRegMaxLayouts ||
            first.dyn_rec.size() > kRegMaxDyn || first.dyn_entries > kRegMaxDynEntries)
            return kLimits;
        if (first.mats.size() > kRegMaxMatrix) return kMatrices;
        flipped = first.flipped != 0;
        n_mat = first.mats.size();
        std::vector<cd>& mats = first.mats;
        for (size_t b = 1; b <= states.size(); ++b) {
            const State& st = states[b - 1];
            if (st.same != b) {
                mats.resize(mats.size() + n_mat);
                std::copy_n(mats.begin() + static_cast<long>(st.same * n_mat), n_mat,
                            mats.end() - static_cast<long>(n_mat));
                continue;
            }
            Emitted eb;
            emit_schedule(st.ops, use, mma, seq, lays, lay_keys, m, store_q, rot, v, eb);
            flipped |= eb.flipped != 0;
            if (eb.failed || eb.mats.size() != n_mat || eb.rec.size() != first.rec.size()) return kForm;
            mats.insert(mats.end(), eb.mats.begin(), eb.mats.end());
        }
        return kFits;
    };
    Fit fit = emit({});
    if (rot && fit == kMatrices) fit = emit({true, true});
    if (rot && fit == kForm) {   // without negated bits
        fit = emit({false, false});
        if (fit == kMatrices) fit = emit({false, true});
    }
    if (fit != kFits) return false;
    const std::vector<RegOp>& rec = first.rec;
    const std::vector<cd>& mats = first.mats;
    const std::vector<uint32_t>& dyn_rec = first.dyn_rec;
    const uint32_t dyn_entries = first.dyn_entries;
    pass = RegPass{};
    pass.L = cfg.L;
    pass.h = static_cast<uint32_t>(item.hbits.size());
    pass.m = m;
    for (uint32_t i = 0; i < pass.h; ++i) pass.hbits[i] = item.hbits[i];
    pass.n_ops = static_cast<uint32_t>(rec.size());
    pass.n_layouts = static_cast<uint32_t>(lays.size());
    pass.n_mat = static_cast<uint32_t>(n_mat);
    pass.mat_stride = state_slots ? static_cast<uint32_t>(n_mat) : 0u;
    // A barrier between a CTA's tiles only where the last layout's warp bits differ from the
    // first's: then a warp's shared-memory slots at the end of one tile are not its slots at
    // the start of the next.  The slots a warp touches in a layout depend only on the warp
    // bits and the warp's index (tile_swizzle is a linear bijection, and a layout only permutes
    // the other bits among lanes and registers), so where they agree each warp meets only its
    // own slots across the tile boundary — up to the next tile's first CTA-wide remap, whose
    // barrier every warp reaches only after finishing this tile.  The host emulation
    // (reg_emulate.cpp) checks this against the barrier model.
    uint32_t last_layout = 0;
    for (const auto& [i, l] : seq)
        if (i < 0) last_layout = l;
    pass.cta_remaps = sync_tiles ? 1u : 0u;
    pass.sync_tiles = sync_tiles && lay_keys[last_layout].W != lay_keys[0].W ? 1u : 0u;
    for (uint32_t b = 0; b < m; ++b) {
        pass.store_qubit[b] = static_cast<uint8_t>(store_q[b]);
        const uint32_t home = b < cfg.L ? b : item.hbits[b - cfg.L];
        if (store_q[b] != home) pass.relabel = 1;
    }
    pass.n_dyn = static_cast<uint32_t>(dyn_rec.size());
    pass.dyn_entries = dyn_entries;
    // A relabelling pass stores amplitudes, in place, to places that other threads (of other
    // warps) load: every load of the tile must come before any store.  A CTA-wide remap or
    // the per-tile table barrier, both after the loads, order them; otherwise the kernel
    // adds a barrier after the loads.
    // So does a negated bit.
    pass.load_barrier = (pass.relabel || flipped) && !sync_tiles && dyn_rec.empty() ? 1u : 0u;
    pass.fma_dense = pass.mma_ops = pass.pauli_ops = 0;
    pass.last_layout = last_layout;
    pass.rot = rot ? 1u : 0u;
    pass.sign_off = first.sign_off;
    pass.n_signs = static_cast<uint32_t>(first.signs.size());
    for (const RegOp& r : rec) {
        if (r.kind == kRegDense || (rot && (r.kind == kRegDiag || r.kind == kRegDiagDyn)))
            pass.fma_dense = 1;
        if (r.kind == kRegMma) pass.mma_ops = 1;
        if (r.kind == kRegPauli) pass.pauli_ops = 1;
    }
    for (size_t d = 0; d < dyn_rec.size(); ++d) pass.dyn_rec[d] = static_cast<uint8_t>(dyn_rec[d]);
    ops_out.insert(ops_out.end(), rec.begin(), rec.end());
    layouts_out.insert(layouts_out.end(), lays.begin(), lays.end());
    mats_out.insert(mats_out.end(), mats.begin(), mats.end());
    if (flops_per_amp) *flops_per_amp = first.flops;
    return true;
}

}  // namespace

bool lower_pass_reg(const PlanItem& item, const std::vector<GateDesc>& gates,
                    const TileConfig& cfg, RegPass& pass, std::vector<RegOp>& ops_out,
                    std::vector<RegLayout>& layouts_out, std::vector<cd>& mats_out,
                    double* flops_per_amp,
                    const std::vector<std::vector<std::array<cd, 4>>>* state_slots) {
    const uint32_t m = cfg.L + static_cast<uint32_t>(item.hbits.size());
    if (m < kRegMinBits || m > kRegMaxBits || item.hbits.size() > kTileMaxHigh) return false;
    // fewer selector qubits when the matrices of a pass outgrow their shared-memory stage (where
    // it has any); where they still do, or where the states of a batch differ in form (a noise
    // matrix that has no rotation form in some state), dense operations with merged diagonals
    for (int rot = uses_rotation_form(cfg) ? 1 : 0; rot >= 0; --rot)
        for (int sel = static_cast<int>(kRegMaxSelect); sel >= 0; --sel) {
            bool selects = false;
            if (lower_pass_reg_sel(item, gates, cfg, static_cast<uint32_t>(sel), rot != 0, pass, ops_out,
                                   layouts_out, mats_out, flops_per_amp, state_slots, selects))
                return true;
            if (!selects) break;
        }
    return false;
}

}  // namespace lqcs_b200
