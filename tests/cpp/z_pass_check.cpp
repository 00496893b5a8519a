// CPU check of the complex128 tensor-core pass's layout (z_pass_layout in
// libq1gpu.so): in each warp's part of a tile elements and (row, state) pairs
// take every slot once and agree on the offsets, the 8 lanes of a phase hit
// distinct bank groups in both, elements come in runs of 8 or more (2 where
// they are the lanes' own), and the parts of all tiles cover the state.
// Prints "bad <count>"; exit status 1 on any failure.
#include <algorithm>
#include <cstdio>
#include <random>
#include <vector>

#include "../../q1tsim_gb300/csrc/kernels.h"

using namespace q1g;

int main()
{
    std::mt19937 rng(3);
    long bad = 0;
    for (int trial = 0; trial < 400; ++trial) {
        const int n = 12 + (int)(rng() % 6);
        std::vector<int> pos(n);
        for (int p = 0; p < n; ++p) pos[p] = p;
        if (trial > 20) std::shuffle(pos.begin(), pos.end(), rng);
        std::vector<int> g(pos.begin(), pos.begin() + 5), T = g;
        for (int p = 0; p < n && (int)T.size() < 12; ++p)
            if (std::find(T.begin(), T.end(), p) == T.end()) T.push_back(p);
        std::sort(T.begin(), T.end());
        std::sort(g.begin(), g.end());
        int gate_of[5];
        for (int k = 0; k < 5; ++k) gate_of[k] = (int)(std::find(T.begin(), T.end(), g[k]) - T.begin());
        std::vector<int> rows;
        for (int j = 0; j < 12; ++j)
            if (std::find(gate_of, gate_of + 5, j) == gate_of + 5) rows.push_back(j);
        ZPass p;
        z_pass_layout(p, T.data(), gate_of);
        std::vector<uint64_t> at(256, ~0ull);        // offset held by a slot
        for (uint32_t e = 0; e < 256; ++e) {
            uint32_t s = 0;
            uint64_t o = 0;
            for (int i = 0; i < 8; ++i)
                if ((e >> i) & 1) s ^= p.slot[i], o |= p.off[i];
            if (s >= 256 || at[s] != ~0ull) ++bad;
            else at[s] = o;
            bad += (o ^ e) & (p.direct ? 1 : 7);
            if (p.direct) {      // lane e % 32's own row, state e / 32
                uint64_t own = 0;
                for (int b = 0; b < 5; ++b)
                    if ((e >> b) & 1) own |= uint64_t(1) << T[rows[b]];
                for (int k = 0; k < 3; ++k)
                    if ((e >> (5 + k)) & 1) own |= uint64_t(1) << g[k];
                bad += o != own;
            }
            if ((e & 7) == 0) {
                uint32_t banks = 0;
                for (uint32_t l = 0; l < 8; ++l) {
                    uint32_t b = 0;
                    for (int i = 0; i < 8; ++i)
                        if (((e + l) >> i) & 1) b ^= p.slot[i];
                    banks |= 1u << (b & 7);
                }
                bad += banks != 255;
            }
        }
        for (uint32_t lane = 0; lane < 32; ++lane)
            for (uint32_t j = 0; j < 8; ++j) {
                uint32_t s = 0, banks = 0;
                uint64_t o = 0;
                for (int b = 0; b < 5; ++b)
                    if ((lane >> b) & 1) s ^= p.slot[p.row_of[b]], o |= uint64_t(1) << T[rows[b]];
                for (int k = 0; k < 3; ++k)
                    if ((j >> k) & 1) s ^= p.slot[p.gate_of[k]], o |= uint64_t(1) << g[k];
                bad += s >= 256 || at[s] != o;
                for (uint32_t l = 0; l < 8; ++l) {
                    uint32_t b = 0;
                    for (int i = 0; i < 5; ++i)
                        if ((((lane & 24) + l) >> i) & 1) b ^= p.slot[p.row_of[i]];
                    banks |= 1u << (b & 7);
                }
                bad += banks != 255;
            }
        std::vector<int> amp(size_t(1) << n, 0);
        for (uint64_t tile = 0; tile < (uint64_t(1) << n) / 4096; ++tile)
            for (uint32_t w = 0; w < 16; ++w)
                for (uint32_t e = 0; e < 256; ++e) {
                    uint64_t i = expand_index(tile, p.tilemap);
                    for (int b = 0; b < 4; ++b)
                        if ((w >> b) & 1) i |= p.warp[b];
                    for (int b = 0; b < 8; ++b)
                        if ((e >> b) & 1) i |= p.off[b];
                    if (i >= amp.size()) ++bad;
                    else ++amp[i];
                }
        for (int v : amp) bad += v != 1;
        for (int b = 0; b < 2; ++b)
            bad += p.warp[b] != uint64_t(1) << T[rows[5 + b]] || p.warp[2 + b] != uint64_t(1) << g[3 + b];
    }
    std::printf("bad %ld\n", bad);
    return bad ? 1 : 0;
}
