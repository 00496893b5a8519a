// CPU check of the gate-run grouping and its tile-local ops (group_runs,
// make_run_op in libq1gpu.so): random sequences of pair and phase updates
// with controls (on 1 and on 0), swaps and diagonal pairs on states of 1 to
// 15 qubits, with one or two columns, are replayed pass by pass on the tiles
// as the kernel does, and must equal the ops applied one by one.  Every op
// runs once.  Prints "bad <count> ..."; exit status 1 on any failure.
#include <complex>
#include <cstdio>
#include <random>
#include <vector>

#include "../../q1tsim_gb300/csrc/gate_run.h"

using namespace q1g;

static void apply_direct(std::vector<cd>& a, const GateOp& op)
{
    const uint64_t units = a.size() >> op.map.nz;
    for (uint64_t u = 0; u < units; ++u) {
        const uint64_t i = expand_index(u, op.map);
        if (op.kind == GateOp::Phase) {
            a[i] *= cd(op.ph[0], op.ph[1]);
        } else {
            const cd x0 = a[i | op.o0], x1 = a[i | op.o1];
            const cd* m = reinterpret_cast<const cd*>(op.m2);
            a[i | op.o0] = m[0] * x0 + m[1] * x1;
            a[i | op.o1] = m[2] * x0 + m[3] * x1;
        }
    }
}

static cd unit(uint32_t u) { return u == 0 ? cd(1, 0) : u == 1 ? cd(0, 1) : u == 2 ? cd(-1, 0) : cd(0, -1); }

int main()
{
    std::mt19937 rng(7);
    auto real = [&] { return std::uniform_real_distribution<double>(-1.0, 1.0)(rng); };
    long bad = 0, passes = 0, nops_all = 0;
    for (int trial = 0; trial < 300; ++trial) {
        const int n = 1 + (int)(rng() % 15);
        const uint64_t total = uint64_t(1 + (trial % 4 == 0)) << n;   // two columns: one bit above
        const int prec = trial % 2, exact = trial % 3 == 0;
        std::vector<GateOp> ops;
        const int count = 1 + (int)(rng() % 120);
        for (int g = 0; g < count; ++g) {
            const int k = 1 + (int)(rng() % (n < 4 ? n : 4));
            std::vector<int> pos;
            while ((int)pos.size() < k) {
                const int p = (int)(rng() % n);
                bool has = false;
                for (int q : pos) has |= q == p;
                if (!has) pos.push_back(p);
            }
            GateOp op;
            op.map.nz = k;
            for (int j = 0; j < k; ++j) op.map.zpos[j] = pos[j];
            for (int i = 0; i < k; ++i)
                for (int j = i + 1; j < k; ++j)
                    if (op.map.zpos[j] < op.map.zpos[i]) std::swap(op.map.zpos[i], op.map.zpos[j]);
            const int kind = (int)(rng() % 4);
            // which positions are targets (differ), the others fixed to 0 or 1
            const int targets = kind == 3 ? 0 : (k >= 2 && rng() % 4 == 0 ? 2 : 1);
            for (int j = targets; j < k; ++j)
                if (rng() % 3) op.map.setmask |= uint64_t(1) << pos[j];
            const double t = 3.0 * real(), c = std::cos(t), s = std::sin(t);
            if (kind == 3) {
                op.kind = GateOp::Phase;
                op.ph[0] = rng() % 3 ? c : -1.0;
                op.ph[1] = op.ph[0] == -1.0 ? 0.0 : s;
            } else {
                op.kind = GateOp::Pair;
                if (targets == 1) {
                    op.o1 = uint64_t(1) << pos[0];
                } else {          // a swap's pair, or one of |00>, |11>
                    op.o0 = rng() % 2 ? uint64_t(1) << pos[1] : 0;
                    op.o1 = (uint64_t(1) << pos[0]) | (op.o0 ? 0 : uint64_t(1) << pos[1]);
                }
                const double full[8] = {c, 0, -s * 0.6, s * 0.8, s * 0.6, s * 0.8, c, 0};
                const double x[8] = {0, 0, 1, 0, 0, 1, 0, 0};
                for (int e = 0; e < 8; ++e) op.m2[e] = kind == 2 ? x[e] : full[e];
            }
            if (!run_takes(op)) ++bad;
            ops.push_back(op);
        }
        std::vector<cd> a(total), b;
        for (auto& v : a) v = cd(real(), real());
        b = a;
        for (const auto& op : ops) apply_direct(a, op);
        std::vector<const GateOp*> list;
        for (const auto& op : ops) list.push_back(&op);
        std::vector<int> seen(ops.size(), 0);
        for (const RunPass& p : group_runs(list, n, total, prec, exact)) {
            ++passes;
            if (p.ops.empty() || (int)p.ops.size() > kRunMaxOps || p.tile.bits > kRunMaxTileBits || p.tile.bits > n) ++bad;
            for (uint64_t tile = 0; tile < total >> p.tile.bits; ++tile) {
                const uint64_t base = expand_index(tile, p.tile.map);
                auto at = [&](uint32_t l) -> cd& {
                    uint64_t i = base;
                    for (int k = 0; k < p.tile.bits; ++k)
                        if ((l >> k) & 1) i |= p.tile.off[k];
                    return b[i];
                };
                for (int oi : p.ops) {
                    const RunOp r = make_run_op(ops[oi], p.tile);
                    if (tile == 0) ++seen[oi];
                    if ((base & r.extmask) != r.extset) continue;
                    for (uint32_t u0 = 0; u0 < (1u << (p.tile.bits - (int)r.nz)); ++u0) {
                        uint32_t i = u0;
                        for (uint32_t q = 0; q < r.nz; ++q) i += i & r.hi[q];
                        i |= r.set;
                        const cd* m = reinterpret_cast<const cd*>(r.m);
                        if (r.kind == kRunPhase) {
                            at(i) *= m[0];
                        } else if (r.kind == kRunPhaseMono) {
                            at(i) *= unit((r.code >> 1) & 3);
                        } else {
                            const cd x0 = at(i | r.o0), x1 = at(i | r.o1);
                            if (r.kind == kRunPair) {
                                at(i | r.o0) = m[0] * x0 + m[1] * x1;
                                at(i | r.o1) = m[2] * x0 + m[3] * x1;
                            } else {
                                at(i | r.o0) = unit((r.code >> 1) & 3) * ((r.code & 1) ? x1 : x0);
                                at(i | r.o1) = unit((r.code >> 3) & 3) * ((r.code & 1) ? x0 : x1);
                            }
                        }
                    }
                }
            }
        }
        for (int s : seen) bad += s != 1;
        nops_all += (long)ops.size();
        for (uint64_t i = 0; i < total; ++i)
            if (!(std::abs(a[i] - b[i]) <= 1e-12)) {
                ++bad;
                break;
            }
    }
    std::printf("bad %ld passes %ld ops %ld\n", bad, passes, nops_all);
    return bad ? 1 : 0;
}
