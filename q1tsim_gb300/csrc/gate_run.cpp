// Grouping of plain gates into tile passes (gate_run.h).
#include "gate_run.h"

#include <algorithm>
#include <cmath>
#include <cstring>

#include "df64.cuh"
#include "unit_code.h"

namespace q1g {

uint64_t run_need(const GateOp& op) { return op.kind == GateOp::Pair ? (op.o0 ^ op.o1) : 0; }

bool run_takes(const GateOp& op)
{
    // NaN entries compare false and stay out
    auto small = [](const double* m, int n) {
        double s = 0.0;
        for (int e = 0; e < n; ++e) s += std::fabs(m[e]);
        return s <= 2.01;
    };
    if (op.kind == GateOp::Phase) return small(op.ph, 2);
    if (op.kind != GateOp::Pair) return false;
    return small(op.m2, 4) && small(op.m2 + 4, 4);
}

bool is_unit(const GateOp& op)
{
    int swap, u0, u1;
    if (op.kind == GateOp::Phase) return unit_code(op.ph[0], op.ph[1]) >= 0;
    return op.kind == GateOp::Pair && mono_pair(op.m2, swap, u0, u1);
}

bool rounds_all(const GateOp& op) { return op.kind == GateOp::Pair && op.map.nz == 1 && !is_unit(op); }

namespace {

uint64_t positions_mask(const GateOp& op)
{
    uint64_t m = 0;
    for (int q = 0; q < op.map.nz; ++q) m |= uint64_t(1) << op.map.zpos[q];
    return m;
}

// What an op costs (measured on one GB300): microseconds of a CTA that has
// an SM to itself (fixed, and per unit of its tile), and per unit of an SM
// that several tiles fill.  Double-float U3s: 0.5 us on a tile of 2^8
// amplitudes, 1.6 us on one of 2^11, 1.95 cycles per pair when full; the FP64
// pipe does 2 FMAs per cycle.
struct OpCost {
    double fixed, unit, full;
};
OpCost op_cost(const GateOp& op, int prec, bool fp64_exact)
{
    const double w = op.kind == GateOp::Pair ? 1.0 : 0.5;
    if (is_unit(op)) return {0.3, 0.3e-3 * w, 0.2e-3 * w};
    if (prec == kC64) return {0.35, 0.45e-3 * w, 0.3e-3 * w};
    if (fp64_exact) return {0.4, 4.5e-3 * w, 4.0e-3 * w};
    return {0.35, 1.2e-3 * w, 1.0e-3 * w};
}

struct Item {
    uint64_t full, need;
    double units_per_amp;    // of its tile
    OpCost cost;
};

// Takes, in order, every remaining item that can move to the front and
// whose needed positions lie in S (in_order: up to the first whose do not).
double absorb(const std::vector<Item>& items, const int* left, const int* end, uint64_t S, uint64_t all, bool in_order,
              std::vector<int>* taken)
{
    uint64_t blocked = 0;
    double got = 0.0;
    for (; left < end; ++left) {
        const int i = *left;
        const Item& it = items[i];
        if (!(it.full & blocked) && !(it.need & ~S)) {
            got += 0.05e-3 + it.units_per_amp * it.cost.full;
            if (taken) taken->push_back(i);
        } else {
            blocked |= it.full;
            if (in_order || (blocked & all) == all) break;
        }
    }
    return got;
}

RunTile make_tile(uint64_t S, int bits)
{
    RunTile t{};
    t.bits = bits;
    t.map.nz = bits;
    t.map.setmask = 0;
    int k = 0;
    for (int p = 0; p < 64 && k < bits; ++p)
        if ((S >> p) & 1) {
            t.map.zpos[k] = p;
            t.off[k] = uint64_t(1) << p;
            ++k;
        }
    return t;
}

}  // namespace

std::vector<RunPass> group_runs(const std::vector<const GateOp*>& ops, int nbits, uint64_t total, int prec,
                                bool fp64_exact, double* cost_us, int sms)
{
    const int m = (int)ops.size();
    std::vector<Item> items(m);
    for (int i = 0; i < m; ++i) {
        const GateOp& op = *ops[i];
        items[i].full = positions_mask(op);
        items[i].need = run_need(op);
        items[i].units_per_amp = 1.0 / (double)(uint64_t(1) << op.map.nz);
        items[i].cost = op_cost(op, prec, fp64_exact);
    }
    const uint64_t all = nbits >= 64 ? ~uint64_t(0) : ((uint64_t(1) << nbits) - 1);
    // A pass is chosen from the next kAhead ops (it takes kRunMaxOps at most): a
    // qubit that is idle for long would let every look at a window run to the end
    // of the sequence (16 qubits, one idle, 40,000 gates: 1072 ms to the end, 35 so).
    constexpr size_t kAhead = 8 * kRunMaxOps;
    const double bytes = (double)total * (double)amp_bytes(prec);
    // tile sizes to try: the largest fits the SM's shared memory three times;
    // smaller ones give a small state more tiles than one SM takes
    std::vector<int> sizes;
    for (int T = std::min(nbits, kRunMaxTileBits); T >= std::min(nbits, 8); --T) sizes.push_back(T);
    if (total >= (uint64_t(1) << 21)) sizes.assign(1, std::min(nbits, kRunMaxTileBits));
    std::vector<RunPass> best;
    double best_cost = INFINITY;
    for (int T : sizes) {
        // positions every tile holds: runs of 128 bytes in HBM, of a sector
        // pair in a state that stays in L2
        int low = prec == kC128 ? 3 : 4;
        if (bytes <= 32e6) low = prec == kC128 ? 1 : 2;
        low = std::min(low, T);
        const uint64_t low_mask = (uint64_t(1) << low) - 1;
        const double tiles = (double)(total >> T), per_sm = std::ceil(tiles / sms);
        std::vector<RunPass> passes;
        std::vector<int> left(m);
        for (int i = 0; i < m; ++i) left[i] = i;
        double cost = 0.0;
        for (size_t head = 0; head < left.size();) {
            const int* const first = left.data() + head;
            const int* const end = first + std::min(kAhead, left.size() - head);
            uint64_t best_set = 0;
            double best_got = -1.0;
            auto consider = [&](uint64_t S) {
                const double got = absorb(items, first, end, S, all, fp64_exact, nullptr);
                if (got > best_got) {
                    best_got = got;
                    best_set = S;
                }
            };
            // first fit: the set grown along the sequence
            {
                uint64_t S = low_mask, blocked = 0;
                for (const int* i = first; i < end; ++i) {
                    const Item& it = items[*i];
                    if (!(it.full & blocked) && __builtin_popcountll(S | it.need) <= T) {
                        S |= it.need;
                    } else {
                        blocked |= it.full;
                        if (fp64_exact || (blocked & all) == all) break;
                    }
                }
                consider(S);
            }
            // every window of consecutive positions
            const int w = T - low;
            for (int a = low; a + w <= nbits; ++a) consider(low_mask | (((uint64_t(1) << w) - 1) << a));
            RunPass p;
            std::vector<int> taken;
            absorb(items, first, end, best_set, all, fp64_exact, &taken);
            if (taken.empty()) {     // an op that needs more positions than the low ones leave room for
                best_set = items[*first].need;
                taken.push_back(*first);
            }
            if ((int)taken.size() > kRunMaxOps) taken.resize(kRunMaxOps);
            // positions no op needs leave the set; the lowest others fill it up
            uint64_t S = 0;
            for (int i : taken) S |= items[i].need;
            for (int q = 0; q < low && __builtin_popcountll(S) < T; ++q) S |= uint64_t(1) << q;
            for (int q = 0; q < nbits && __builtin_popcountll(S) < T; ++q) S |= uint64_t(1) << q;
            p.tile = make_tile(S, T);
            p.ops = taken;
            // the window's others move up behind the taken ones
            size_t k = taken.size(), to = (size_t)(end - left.data());
            for (size_t from = to; from-- > head;) {
                if (k > 0 && taken[k - 1] == left[from]) --k;
                else left[--to] = left[from];
            }
            head += taken.size();
            // launch and tile traffic, then the ops: alone on an SM or
            // sharing it
            cost += 5.0 + 2.0 * bytes / (bytes <= 64e6 ? 12e6 : 6.4e6);
            for (int i : taken) {
                const double units = items[i].units_per_amp * (double)(uint64_t(1) << T);
                const OpCost& c = items[i].cost;
                cost += std::max((c.fixed + c.unit * units) * std::ceil(per_sm / 4.0), per_sm * units * c.full);
            }
            passes.push_back(std::move(p));
        }
        if (cost < best_cost) {
            best_cost = cost;
            best.swap(passes);
        }
    }
    if (cost_us) *cost_us = best_cost;
    return best;
}

RunOp make_run_op(const GateOp& op, const RunTile& tile)
{
    RunOp r;
    std::memset(&r, 0, sizeof r);
    uint64_t tmask = 0;
    for (int k = 0; k < tile.bits; ++k) tmask |= tile.off[k];
    auto local = [&](uint64_t x) {
        uint32_t l = 0;
        for (int k = 0; k < tile.bits; ++k)
            if (x & tile.off[k]) l |= 1u << k;
        return l;
    };
    auto set = [&](int e, const double* v) {
        const DF re = host_split(v[0]), im = host_split(v[1]);
        r.m[2 * e] = v[0];
        r.m[2 * e + 1] = v[1];
        r.df[e] = make_float4(re.h, re.l, im.h, im.l);
        r.rest[2 * e] = (float)(v[0] - (double)re.h - (double)re.l);
        r.rest[2 * e + 1] = (float)(v[1] - (double)im.h - (double)im.l);
    };
    const uint64_t full = positions_mask(op);
    const uint64_t fixed = op.map.setmask | (op.kind == GateOp::Pair ? (op.o0 & op.o1) : 0);
    const uint64_t differ = run_need(op);
    r.extmask = full & ~tmask;
    r.extset = fixed & ~tmask;
    const uint32_t zl = local(full & tmask);
    for (int k = 0; k < tile.bits; ++k)
        if ((zl >> k) & 1) r.hi[r.nz++] = (uint16_t)~((1u << k) - 1u);
    r.set = local(fixed & tmask);
    if (op.kind == GateOp::Phase) {
        const int code = unit_code(op.ph[0], op.ph[1]);
        r.kind = code >= 0 ? kRunPhaseMono : kRunPhase;
        r.code = code >= 0 ? (uint32_t)code << 1 : 0;
        set(0, op.ph);
        return r;
    }
    r.o0 = local(op.o0 & differ);
    r.o1 = local(op.o1 & differ);
    int swap = 0, u0 = 0, u1 = 0;
    if (mono_pair(op.m2, swap, u0, u1)) {
        r.kind = kRunPairMono;
        r.code = (uint32_t)swap | ((uint32_t)u0 << 1) | ((uint32_t)u1 << 3);
    } else {
        r.kind = kRunPair;
        const double* m = op.m2;
        if (m[1] == 0.0 && m[3] == 0.0 && m[5] == 0.0 && m[7] == 0.0) r.shape = kRunReal;
        else if (m[1] == 0.0 && m[2] == 0.0 && m[4] == 0.0 && m[7] == 0.0) r.shape = kRunCross;
        else if (m[1] == 0.0) r.shape = kRunReal00;
        else r.shape = kRunFull;
    }
    for (int e = 0; e < 4; ++e) set(e, op.m2 + 2 * e);
    return r;
}

}  // namespace q1g
