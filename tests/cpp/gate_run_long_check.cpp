// CPU check that grouping a plan's plain gates (group_runs in libq1gpu.so) takes
// time in proportion to their number: 80,000 gates with one idle qubit, and with
// the halves of the circuit on different qubits, against 10,000 of them.  8
// times as long is proportional, 64 times quadratic; more than 25 fails.  Prints
// "bad <count> ..."; exit status 1 on any failure.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <random>
#include <vector>

#include "../../q1tsim_gb300/csrc/gate_run.h"

using namespace q1g;

static std::vector<GateOp> sequence(int m, int n, bool halves)
{
    std::mt19937 rng(1);
    std::vector<GateOp> ops(m);
    for (int i = 0; i < m; ++i) {
        const int lo = !halves ? 1 : i < m / 2 ? n / 2 : 0, hi = halves && i >= m / 2 ? n / 2 : n;
        const int a = lo + (int)(rng() % (hi - lo));
        int b = a;
        while (b == a) b = lo + (int)(rng() % (hi - lo));
        GateOp& op = ops[i];
        op.kind = GateOp::Pair;
        op.o1 = uint64_t(1) << a;
        const bool cx = rng() % 3 == 0;
        op.map.nz = cx ? 2 : 1;
        op.map.zpos[0] = cx ? std::min(a, b) : a;
        if (cx) {
            op.map.zpos[1] = std::max(a, b);
            op.map.setmask = uint64_t(1) << b;
        }
        const double u[8] = {0.8, 0, 0, 0.6, 0.36, 0.48, 0.64, -0.48}, x[8] = {0, 0, 1, 0, 1, 0, 0, 0};
        for (int e = 0; e < 8; ++e) op.m2[e] = cx ? x[e] : u[e];
    }
    return ops;
}

static double group_ms(int m, int n, bool halves, size_t* taken)
{
    const auto ops = sequence(m, n, halves);
    std::vector<const GateOp*> list;
    for (const auto& op : ops) list.push_back(&op);
    double best = 1e30;
    for (int rep = 0; rep < (m < 20000 ? 5 : 2); ++rep) {
        const auto t = std::chrono::steady_clock::now();
        const auto passes = group_runs(list, n, uint64_t(1) << n, kC128, false);
        best = std::min(best, std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t).count());
        *taken = 0;
        for (const auto& p : passes) *taken += p.ops.size();
    }
    return best;
}

int main()
{
    long bad = 0;
    for (int n : {10, 16, 24})
        for (bool halves : {false, true}) {
            size_t few_taken = 0, many_taken = 0;
            const double few = group_ms(10000, n, halves, &few_taken), many = group_ms(80000, n, halves, &many_taken);
            if (few_taken != 10000 || many_taken != 80000 || many > 25.0 * few) {
                ++bad;
                std::printf("n %d halves %d: %.2f ms and %.2f ms\n", n, (int)halves, few, many);
            }
        }
    std::printf("bad %ld\n", bad);
    return bad ? 1 : 0;
}
