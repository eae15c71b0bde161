// adj_plan.cpp — planning of the adjoint's register passes of Pauli rotations (adj_pass.cuh).
#include <algorithm>
#include <stdexcept>

#include "adj_pass.cuh"
#include "tile.cuh"

namespace lqcs_b200 {

namespace {

uint32_t parity(uint64_t v) { return static_cast<uint32_t>(__builtin_popcountll(v) & 1); }

// A subspace of the index bits, as reduced vectors with distinct lowest set bits.
struct Span {
    std::vector<uint64_t> v;
    uint64_t reduce(uint64_t x) const {
        for (uint64_t b : v)
            if (x & (b & (~b + 1))) x ^= b;
        return x;
    }
    bool contains(uint64_t x) const { return reduce(x) == 0; }
    bool add(uint64_t x) {   // false: already inside
        x = reduce(x);
        if (!x) return false;
        const uint64_t low = x & (~x + 1);
        for (uint64_t& b : v)
            if (b & low) b ^= x;
        v.push_back(x);
        return true;
    }
};

bool commute(const AdjRotation& a, const AdjRotation& b) {
    return ((__builtin_popcountll(a.x & b.zy) + __builtin_popcountll(a.zy & b.x)) & 1) == 0;
}

// The thread vectors whose slots come first are on the lowest lanes: three with independent
// low slot bits let the eight lanes of a quarter warp hit eight 16-byte bank groups.
void spread_lanes(std::vector<uint64_t>& t, const std::vector<uint16_t>& slot) {
    for (size_t a = 0; a < t.size(); ++a)
        for (size_t b = a + 1; b < t.size(); ++b)
            for (size_t c = b + 1; c < t.size(); ++c) {
                const uint32_t x = slot[a] & 7u, y = slot[b] & 7u, z = slot[c] & 7u;
                if (!x || !y || !z || x == y || (x ^ y) == z || x == z || y == z) continue;
                std::vector<uint64_t> out{t[a], t[b], t[c]};
                for (size_t i = 0; i < t.size(); ++i)
                    if (i != a && i != b && i != c) out.push_back(t[i]);
                t = std::move(out);
                return;
            }
}

AdjPass make_pass(const std::vector<AdjRotation>& rots, Span space, uint32_t n, uint32_t m,
                  uint32_t regs) {
    for (uint32_t q = 0; q < n && space.v.size() < m; ++q) space.add(uint64_t{1} << q);
    std::sort(space.v.begin(), space.v.end(), [](uint64_t a, uint64_t b) {
        return (a & (~a + 1)) < (b & (~b + 1));
    });
    AdjPass p{};
    p.m = m;
    p.regs = regs;
    for (uint32_t i = 0; i < m; ++i) p.pivots[i] = static_cast<uint32_t>(__builtin_ctzll(space.v[i]));
    // coordinates over the reduced basis: the pivot bits
    auto slot = [&](uint64_t w) {
        uint32_t c = 0;
        for (uint32_t i = 0; i < m; ++i) c |= static_cast<uint32_t>((w >> p.pivots[i]) & 1) << i;
        return static_cast<uint16_t>(tile_swizzle(c));
    };
    // groups of rotations whose x masks are one layout's register vectors
    std::vector<std::vector<uint64_t>> reg;
    std::vector<uint32_t> group(rots.size());
    Span in_group;
    for (size_t k = 0; k < rots.size(); ++k) {
        const uint64_t x = rots[k].x;
        const bool have = !reg.empty() && std::find(reg.back().begin(), reg.back().end(), x) != reg.back().end();
        if (reg.empty() || (x && !have && (reg.back().size() >= regs || in_group.contains(x)))) {
            reg.emplace_back();
            in_group = Span{};
        }
        if (x && std::find(reg.back().begin(), reg.back().end(), x) == reg.back().end()) {
            reg.back().push_back(x);
            in_group.add(x);
        }
        group[k] = static_cast<uint32_t>(reg.size() - 1);
    }
    if (reg.empty()) reg.emplace_back();
    p.n_layouts = static_cast<uint32_t>(reg.size());
    std::vector<std::vector<uint64_t>> thr(reg.size());
    for (size_t l = 0; l < reg.size(); ++l) {
        Span s;
        for (uint64_t w : reg[l]) s.add(w);
        // fill the register vectors with vectors that leave qubits 0..2 to the lanes
        Span with_low = s;
        for (uint32_t q = 0; q < 3; ++q) with_low.add(uint64_t{1} << q);
        for (int round = 0; round < 2; ++round)
            for (size_t i = space.v.size(); i-- > 0 && reg[l].size() < regs;) {
                if (round == 0 ? !with_low.add(space.v[i]) : s.contains(space.v[i])) continue;
                s.add(space.v[i]);
                reg[l].push_back(space.v[i]);
            }
        std::vector<uint16_t> slots;
        for (uint32_t i = 0; i < m && thr[l].size() < m - regs; ++i)   // qubits 0..2 first
            if (s.add(space.v[i])) {
                thr[l].push_back(space.v[i]);
                slots.push_back(slot(space.v[i]));
            }
        if (l != 0 && l + 1 != reg.size()) spread_lanes(thr[l], slots);
        for (uint32_t i = 0; i < m - regs; ++i) p.lay[l].t[i] = slot(thr[l][i]);
        for (uint32_t i = 0; i < regs; ++i) p.lay[l].r[i] = slot(reg[l][i]);
    }
    for (int e = 0; e < 2; ++e) {
        const size_t l = e ? reg.size() - 1 : 0;
        std::copy(thr[l].begin(), thr[l].end(), p.tvec[e]);
        std::copy(reg[l].begin(), reg[l].end(), p.rvec[e]);
    }
    p.n_rots = static_cast<uint32_t>(rots.size());
    for (size_t k = 0; k < rots.size(); ++k) {
        AdjRot& r = p.rot[k];
        const uint32_t l = group[k];
        r.zy = rots[k].zy;
        r.param = rots[k].param;
        r.n_y = static_cast<uint8_t>(rots[k].n_y & 3u);
        r.layout = static_cast<uint8_t>(l);
        r.rbit = kAdjDiag;
        for (uint32_t i = 0; i < regs; ++i) {
            if (rots[k].x && reg[l][i] == rots[k].x) r.rbit = static_cast<uint8_t>(i);
            r.rz = static_cast<uint8_t>(r.rz | parity(reg[l][i] & r.zy) << i);
        }
        for (uint32_t i = 0; i < m - regs; ++i)
            r.tz = static_cast<uint16_t>(r.tz | parity(thr[l][i] & r.zy) << i);
    }
    return p;
}

}  // namespace

std::vector<AdjPass> plan_adjoint_passes(const std::vector<AdjRotation>& rots, uint32_t n,
                                         uint32_t bits, uint32_t regs, bool any_order,
                                         uint32_t most) {
    const uint32_t m = std::min(n, std::min(bits, kAdjMaxBits));
    if (m < kAdjMinBits) throw std::logic_error("adjoint pass: too few qubits");
    std::vector<AdjPass> out;
    std::vector<AdjRotation> pend = rots;
    while (!pend.empty()) {
        Span space;
        for (uint32_t q = 0; q < 3; ++q) space.add(uint64_t{1} << q);
        std::vector<AdjRotation> cur, rest;
        uint32_t layouts = 1, in_layout = 0;   // an upper bound on the layouts taken so far
        for (size_t i = 0; i < pend.size(); ++i) {
            const AdjRotation& r = pend[i];
            if (cur.size() == most) {   // full
                rest.insert(rest.end(), pend.begin() + static_cast<std::ptrdiff_t>(i), pend.end());
                break;
            }
            bool ok = layouts < kAdjMaxLayouts && (space.v.size() < m || space.contains(r.x));
            for (size_t k = 0; !any_order && ok && k < rest.size(); ++k) ok = commute(r, rest[k]);
            if (!ok) {
                rest.push_back(r);
                continue;
            }
            space.add(r.x);
            cur.push_back(r);
            if (r.x && ++in_layout > 1) ++layouts;   // (at worst a layout per rotation)
        }
        out.push_back(make_pass(cur, space, n, m, regs));
        pend = std::move(rest);
    }
    return out;
}

}  // namespace lqcs_b200
