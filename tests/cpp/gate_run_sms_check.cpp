// CPU check of the tile-pass model (group_runs in libq1gpu.so) on devices of
// other sizes: with fewer SMs the same gates cost more, in proportion once the
// tiles outnumber the SMs, and small tiles, which spread a small state over idle
// SMs, are no longer taken.  Prints "bad <count>"; exit status 1 on any failure.
#include <cmath>
#include <cstdio>
#include <vector>

#include "../../q1tsim_gb300/csrc/gate_run.h"

using namespace q1g;

int main()
{
    long bad = 0;
    for (int n : {14, 16, 24}) {
        std::vector<GateOp> ops;
        for (int layer = 0; layer < 4; ++layer)
            for (int q = 0; q < n; ++q) {
                GateOp op;
                op.kind = GateOp::Pair;
                op.map.nz = 1;
                op.map.zpos[0] = q;
                op.o1 = uint64_t(1) << q;
                const double m[8] = {0.8, 0, 0, 0.6, 0.36, 0.48, 0.64, -0.48};
                for (int e = 0; e < 8; ++e) op.m2[e] = m[e];
                ops.push_back(op);
            }
        std::vector<const GateOp*> list;
        for (const auto& op : ops) list.push_back(&op);
        double all = 0.0, few = 0.0, one = 0.0;
        const auto pa = group_runs(list, n, uint64_t(1) << n, kC128, false, &all, 152);
        const auto pf = group_runs(list, n, uint64_t(1) << n, kC128, false, &few, 16);
        const auto po = group_runs(list, n, uint64_t(1) << n, kC128, false, &one, 1);
        bad += !(all < few && few < one);
        bad += !(pa[0].tile.bits <= pf[0].tile.bits && pf[0].tile.bits <= po[0].tile.bits);
        bad += po[0].tile.bits != kRunMaxTileBits;
        // 2048 tiles and more: the arithmetic is 9.5 times as long on 16 SMs
        if (n == 24) bad += !(few > 7.0 * all && few < 9.6 * all);
    }
    std::printf("bad %ld\n", bad);
    return bad ? 1 : 0;
}
