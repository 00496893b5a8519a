// CPU check of the complex128 tensor-core pass's layout and operand image
// (z_pass_layout, z_pass_image in libq1gpu.so): the slots of a tile are a
// permutation of 0..4095, the rows' and gates' slots address every tile
// coordinate once and agree with the copies', the 8 lanes of a phase hit
// distinct bank groups in row reads and in copies, the copies of all tiles
// cover the state, and the digits of the image add up to the real embedding.
// Prints "bad <count>"; exit status 1 on any failure.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

#include "../../q1tsim_gb300/csrc/kernels.h"

using namespace q1g;

static double f16(uint16_t h)
{
    const int e = (h >> 10) & 31, m = h & 1023;
    const double v = e ? std::ldexp(1024 + m, e - 25) : std::ldexp(m, -24);
    return h & 0x8000 ? -v : v;
}

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
        uint32_t gate_bits = 0;
        int gate_of[5];
        for (int k = 0; k < 5; ++k) {
            gate_of[k] = (int)(std::find(T.begin(), T.end(), g[k]) - T.begin());
            gate_bits |= 1u << gate_of[k];
        }
        ZPass p;
        z_pass_layout(p, T.data(), gate_bits, gate_of);
        auto slot_of = [&](uint32_t x) {
            uint32_t s = 0;
            for (int b = 0; b < 12; ++b)
                if ((x >> b) & 1) s ^= p.slot[b];
            return s;
        };
        std::vector<int> seen(4096, 0), rowseen(4096, 0);
        for (uint32_t x = 0; x < 4096; ++x) {
            if (slot_of(x) >= 4096) ++bad;
            else ++seen[slot_of(x)];
        }
        std::vector<int> rows;
        for (int j = 0; j < 12; ++j)
            if (!((gate_bits >> j) & 1)) rows.push_back(j);
        for (uint32_t t = 0; t < 128; ++t)
            for (uint32_t s = 0; s < 32; ++s) {
                uint32_t x = 0, sl = p.gate[s];
                for (int i = 0; i < 7; ++i)
                    if ((t >> i) & 1) {
                        x |= 1u << rows[i];
                        sl ^= p.row[i];
                    }
                for (int k = 0; k < 5; ++k)
                    if ((s >> k) & 1) x |= 1u << gate_of[k];
                bad += sl != slot_of(x);
                ++rowseen[x];
                if ((t & 7) == 0) {      // the phase of lanes t .. t+7
                    uint32_t banks = 0;
                    for (uint32_t l = 0; l < 8; ++l) {
                        uint32_t a = p.gate[s];
                        for (int i = 0; i < 7; ++i)
                            if (((t + l) >> i) & 1) a ^= p.row[i];
                        banks |= 1u << (a & 7);
                    }
                    bad += banks != 255;
                }
            }
        for (uint32_t x = 0; x < 4096; x += 8) {
            uint32_t banks = 0;
            for (uint32_t l = 0; l < 8; ++l) banks |= 1u << (slot_of(x + l) & 7);
            bad += banks != 255;
        }
        for (int x = 0; x < 4096; ++x) bad += seen[x] != 1 || rowseen[x] != 1;
        std::vector<int> amp(size_t(1) << n, 0);
        for (uint64_t tile = 0; tile < (uint64_t(1) << n) / 4096; ++tile)
            for (uint32_t x = 0; x < 4096; ++x) {
                uint64_t i = expand_index(tile, p.tilemap);
                for (int b = 0; b < 12; ++b)
                    if ((x >> b) & 1) i |= p.off[b];
                if (i >= amp.size()) ++bad;
                else ++amp[i];
            }
        for (int v : amp) bad += v != 1;
    }
    std::vector<double> m(2048);
    for (int trial = 0; trial < 20; ++trial) {
        std::uniform_real_distribution<double> u(-1.0, 1.0);
        for (auto& v : m) v = trial == 0 ? (rng() % 3) - 1.0 : u(rng) * std::ldexp(1.0, -(int)(rng() % 60));
        std::vector<unsigned char> out(kZImageBytes);
        z_pass_image(m.data(), out.data());
        const uint16_t* img = reinterpret_cast<const uint16_t*>(out.data());
        for (int gp = 0; gp < 32; ++gp)
            for (int g = 0; g < 32; ++g)
                for (int cp = 0; cp < 2; ++cp)
                    for (int c = 0; c < 2; ++c) {
                        const double re = m[2 * (32 * gp + g)], im = m[2 * (32 * gp + g) + 1];
                        const double want = cp == c ? re : cp ? im : -im;
                        double got = 0.0;
                        for (int t = 5; t >= 0; --t) {
                            const double d =
                                f16(img[(t * 8192 + tc_sw128_offset(2 * gp + cp, 2 * g + c)) / 2]);
                            if (d != std::floor(d) || std::fabs(d) > 257.0) ++bad;
                            got += std::ldexp(d, -8 - 9 * t);
                        }
                        bad += !(std::fabs(got - want) <= std::ldexp(1.0, -53));
                    }
        for (int e = 0; e < 2048; ++e) bad += reinterpret_cast<const double*>(out.data() + 6 * 8192)[e] != m[e];
    }
    std::printf("bad %ld\n", bad);
    return bad ? 1 : 0;
}
