// Runs of diagonal gates as one pass (gate_plan.h, fuse_runs).  Every
// amplitude i is multiplied by e^{i phi(x)}, x = i mod 2^n its basis bits and
//   phi(x) = c + L0(x) + x_p L1(x),   L0, L1 linear in the bits,
// from per-byte tables of complex factors (computed in double on the host):
//   T0[b][v] = e^{i L0(v << 8b)}  (T0[0] also carries e^{ic}),
//   T1[b][v] = e^{i L1(v << 8b)}.
// With a trailing 1-qubit gate on position q, its 2x2 matrix is then applied
// to each pair (i, i | 2^q) in the same pass.  complex64, states of up to 32
// qubits; a persistent grid, so that each CTA loads the 16 KB of tables into
// shared memory once.
#include <algorithm>
#include <cmath>
#include <complex>
#include <vector>

#include "kernels.h"

namespace q1g {

namespace {

constexpr int kPhaseThreads = 256;
constexpr int kPhaseTable = 2048;   // T0 then T1, 4 bytes x 256 values each

__device__ __forceinline__ float2 cmulf(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

__device__ __forceinline__ float2 phase_of(uint64_t i, uint64_t nmask, int pivot, const float2* T)
{
    const uint32_t x = (uint32_t)(i & nmask);
    float2 f = cmulf(cmulf(T[x & 255u], T[256 + ((x >> 8) & 255u)]),
                     cmulf(T[512 + ((x >> 16) & 255u)], T[768 + (x >> 24)]));
    if (pivot >= 0 && ((x >> pivot) & 1u)) {
        const float2* T1 = T + 1024;
        f = cmulf(f, cmulf(cmulf(T1[x & 255u], T1[256 + ((x >> 8) & 255u)]),
                           cmulf(T1[512 + ((x >> 16) & 255u)], T1[768 + (x >> 24)])));
    }
    return f;
}

__device__ __forceinline__ void load_tables(float2* T, const float2* __restrict__ gtab)
{
    for (int e = threadIdx.x; e < kPhaseTable; e += blockDim.x) T[e] = gtab[e];
    __syncthreads();
}

// Phases only: two amplitudes per 16-byte access (total is even).
__global__ void __launch_bounds__(kPhaseThreads)
k_phase_run(float2* a, uint64_t total, uint64_t nmask, int pivot, const float2* __restrict__ gtab)
{
    __shared__ float2 T[kPhaseTable];
    load_tables(T, gtab);
    float4* a4 = reinterpret_cast<float4*>(a);
    const uint64_t n2 = total / 2;
    for (uint64_t v = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; v < n2; v += (uint64_t)gridDim.x * blockDim.x) {
        const float4 q = a4[v];
        const float2 y0 = cmulf(phase_of(2 * v, nmask, pivot, T), make_float2(q.x, q.y));
        const float2 y1 = cmulf(phase_of(2 * v + 1, nmask, pivot, T), make_float2(q.z, q.w));
        a4[v] = make_float4(y0.x, y0.y, y1.x, y1.y);
    }
}

struct Mat2f {
    float2 m00, m01, m10, m11;
};

// Phases, then the 2x2 matrix on the pairs (i, i | bit); map zeroes position q.
__global__ void __launch_bounds__(kPhaseThreads)
k_phase_pair(float2* a, uint64_t pairs, IndexMap map, uint64_t bit, uint64_t nmask, int pivot,
             const float2* __restrict__ gtab, Mat2f m)
{
    __shared__ float2 T[kPhaseTable];
    load_tables(T, gtab);
    for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < pairs;
         u += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t i0 = expand_nz<1>(u, map), i1 = i0 | bit;
        const float2 y0 = cmulf(phase_of(i0, nmask, pivot, T), a[i0]);
        const float2 y1 = cmulf(phase_of(i1, nmask, pivot, T), a[i1]);
        const float2 p0 = cmulf(m.m00, y0), q0 = cmulf(m.m01, y1);
        const float2 p1 = cmulf(m.m10, y0), q1 = cmulf(m.m11, y1);
        a[i0] = make_float2(p0.x + q0.x, p0.y + q0.y);
        a[i1] = make_float2(p1.x + q1.x, p1.y + q1.y);
    }
}

// ------------------------------------------------ groups of phase runs
//
// A ladder of a Fourier transform is a phase run with the next Hadamard; one
// pass each was HBM-bound (0.71 ms at 28 qubits, 0.90 of its rate).  Here a
// thread holds the 2^S amplitudes of S steps' positions and applies the steps
// one after the other in registers, so S of them cost one pass.  A step's
// phase is split into the part of the other index bits, the same for all of
// a thread's amplitudes, and that of the S positions, from a small table.  The
// common part is summed exactly as a fraction of a turn (32 bits, from
// per-byte tables) and turned into a factor once per thread and step
// (sincospif on at most an eighth of a turn): more accurate than the product
// of eight FP32 factors, and 2^S amplitudes share it.  28-qubit QFT, 26 steps
// in 7 passes of 0.78 ms (0.64 for the memory alone; 24 warps per SM, more or
// fewer registers and a prefetch of the next amplitudes measured slower), the
// transform 8.3 ms instead of 21.4.

constexpr int kGroupThreads = 256;

// e^{2 pi i a / 2^32}
__device__ __forceinline__ float2 turn_factor(uint32_t a)
{
    const uint32_t q = (a + 0x20000000u) >> 30;             // nearest quarter turn
    const int r = (int)(a - (q << 30));                     // within an eighth of it
    float s, c;
    sincospif((float)r * (1.0f / 2147483648.0f), &s, &c);
    if (q & 1u) {
        const float x = c;
        c = -s;
        s = x;
    }
    if (q & 2u) c = -c, s = -s;
    return make_float2(c, s);
}

__device__ __forceinline__ uint32_t byte_sum(const uint32_t (&a)[4][256], uint32_t x)
{
    return a[0][x & 255u] + a[1][(x >> 8) & 255u] + a[2][(x >> 16) & 255u] + a[3][x >> 24];
}

// y[m] times f g[m] for the m with index bit BIT set (BIT < 0: every m; the
// set is known at compile time, so no amplitude is tested for it) or clear.
template <int S, int BIT, bool SET>
__device__ __forceinline__ void group_phase(float2 (&y)[1 << S], float2 f, const float2* g)
{
#pragma unroll
    for (int m = 0; m < (1 << S); ++m)
        if (BIT < 0 || ((m >> (BIT < 0 ? 0 : BIT)) & 1) == (SET ? 1 : 0)) y[m] = cmulf(cmulf(f, g[m]), y[m]);
}

template <int S, bool SET>
__device__ __forceinline__ void group_phase_at(float2 (&y)[1 << S], int bit, float2 f, const float2* g)
{
    switch (bit) {
        case 0: group_phase<S, 0, SET>(y, f, g); break;
        case 1: group_phase<S, 1, SET>(y, f, g); break;
        case 2:
            if constexpr (S > 2) group_phase<S, 2, SET>(y, f, g);
            break;
        case 3:
            if constexpr (S > 3) group_phase<S, 3, SET>(y, f, g);
            break;
        default: group_phase<S, -1, SET>(y, f, g); break;
    }
}

// One step on the 2^S amplitudes y; step K's position is index bit K.
template <int S, int K>
__device__ __forceinline__ void group_step(float2 (&y)[1 << S], const PhaseGroup& g, const PhaseStepTables& T,
                                           uint32_t x)
{
    // pivot in the group: half of the amplitudes each way; outside it (or
    // none): all of them one way
    const int in = g.inner[K], v = g.pivot[K];
    const bool on = in >= 0 || (v >= 0 && ((x >> v) & 1u));
    if (!g.trivial0[K] && (in >= 0 || !on))
        group_phase_at<S, false>(y, in, turn_factor(byte_sum(T.a0, x)), T.g0);
    if (on) group_phase_at<S, true>(y, in, turn_factor(byte_sum(T.a1, x)), T.g1);
    const float* m2 = g.m2[K];
    if (g.real[K]) {
#pragma unroll
        for (int m = 0; m < (1 << S); ++m)
            if (!((m >> K) & 1)) {
                const float2 p = y[m], q = y[m | (1 << K)];
                y[m] = make_float2(m2[0] * p.x + m2[2] * q.x, m2[0] * p.y + m2[2] * q.y);
                y[m | (1 << K)] = make_float2(m2[4] * p.x + m2[6] * q.x, m2[4] * p.y + m2[6] * q.y);
            }
    } else {
        const float2 m00 = make_float2(m2[0], m2[1]), m01 = make_float2(m2[2], m2[3]);
        const float2 m10 = make_float2(m2[4], m2[5]), m11 = make_float2(m2[6], m2[7]);
#pragma unroll
        for (int m = 0; m < (1 << S); ++m)
            if (!((m >> K) & 1)) {
                const float2 p = y[m], q = y[m | (1 << K)];
                y[m] = cmuladd2(m00, p, m01, q);
                y[m | (1 << K)] = cmuladd2(m10, p, m11, q);
            }
    }
}

template <int S, int K>
__device__ __forceinline__ void group_steps(float2 (&y)[1 << S], const PhaseGroup& g, const PhaseStepTables* T,
                                            uint32_t x)
{
    if constexpr (K < S) {
        group_step<S, K>(y, g, T[K], x);
        group_steps<S, K + 1>(y, g, T, x);
    }
}

template <int S>
__global__ void __launch_bounds__(kGroupThreads, 3)
k_phase_group(float2* a, uint64_t units, const __grid_constant__ PhaseGroup g, const __grid_constant__ IndexMap map,
              uint64_t nmask, const PhaseStepTables* __restrict__ gtab)
{
    extern __shared__ uint4 group_smem[];
    PhaseStepTables* T = reinterpret_cast<PhaseStepTables*>(group_smem);
    {
        const uint4* src = reinterpret_cast<const uint4*>(gtab);
        for (int e = threadIdx.x; e < S * (int)(sizeof(PhaseStepTables) / 16); e += kGroupThreads) group_smem[e] = src[e];
    }
    __syncthreads();
    for (uint64_t u = (uint64_t)blockIdx.x * kGroupThreads + threadIdx.x; u < units;
         u += (uint64_t)gridDim.x * kGroupThreads) {
        const uint64_t base = expand_nz<S>(u, map);
        float2 y[1 << S];
#pragma unroll
        for (int m = 0; m < (1 << S); ++m) {
            uint64_t i = base;
#pragma unroll
            for (int b = 0; b < S; ++b)
                if ((m >> b) & 1) i |= uint64_t(1) << g.t[b];
            y[m] = a[i];
        }
        group_steps<S, 0>(y, g, T, (uint32_t)(base & nmask));
#pragma unroll
        for (int m = 0; m < (1 << S); ++m) {
            uint64_t i = base;
#pragma unroll
            for (int b = 0; b < S; ++b)
                if ((m >> b) & 1) i |= uint64_t(1) << g.t[b];
            a[i] = y[m];
        }
    }
}

template <int S>
cudaError_t launch_group(float2* amps, uint64_t units, const PhaseGroup& g, const IndexMap& map, uint64_t nmask,
                         const PhaseStepTables* tab, int sm_count, cudaStream_t st)
{
    const uint64_t want = (units + kGroupThreads - 1) / kGroupThreads;
    const unsigned grid = (unsigned)std::min<uint64_t>(std::max<uint64_t>(want, 1), (uint64_t)sm_count * 3);
    // up to 33 KB: within the default limit of dynamic shared memory
    static_assert(kPhaseGroupMax * sizeof(PhaseStepTables) <= 48 * 1024, "the tables fit without an opt-in");
    k_phase_group<S><<<grid, kGroupThreads, S * sizeof(PhaseStepTables), st>>>(amps, units, g, map, nmask, tab);
    return cudaGetLastError();
}

}  // namespace

void phase_group_tables(const PhaseGroup& g, int nbits, double c, const double* lin0, const double* lin1,
                        PhaseStepTables& out)
{
    // coefficients in turns, the group's own positions apart
    std::vector<double> l0(32, 0.0), l1(32, 0.0);
    constexpr double kTurn = 0.15915494309189533577;   // 1 / 2 pi
    for (int p = 0; p < nbits; ++p) {
        l0[p] = lin0[p] * kTurn;
        l1[p] = (lin0[p] + lin1[p]) * kTurn;
    }
    double own0[kPhaseGroupMax] = {}, own1[kPhaseGroupMax] = {};
    for (int b = 0; b < g.nsteps; ++b) {
        std::swap(own0[b], l0[g.t[b]]);
        std::swap(own1[b], l1[g.t[b]]);
    }
    auto fraction = [](double turns) {
        return (uint32_t)(uint64_t)std::llrint((turns - std::floor(turns)) * 4294967296.0);
    };
    for (int b = 0; b < 4; ++b)
        for (int v = 0; v < 256; ++v) {
            double t0 = b == 0 ? c * kTurn : 0.0, t1 = t0;
            for (int k = 0; k < 8; ++k)
                if ((v >> k) & 1) {
                    t0 += l0[8 * b + k];
                    t1 += l1[8 * b + k];
                }
            out.a0[b][v] = fraction(t0);
            out.a1[b][v] = fraction(t1);
        }
    for (int m = 0; m < (1 << kPhaseGroupMax); ++m) {
        double t0 = 0.0, t1 = 0.0;
        for (int b = 0; b < g.nsteps; ++b)
            if ((m >> b) & 1) {
                t0 += own0[b];
                t1 += own1[b];
            }
        out.g0[m] = make_float2((float)std::cos(t0 / kTurn), (float)std::sin(t0 / kTurn));
        out.g1[m] = make_float2((float)std::cos(t1 / kTurn), (float)std::sin(t1 / kTurn));
    }
}

cudaError_t launch_phase_group(float2* amps, uint64_t total, int nbits, const PhaseGroup& g,
                               const PhaseStepTables* d_tables, int sm_count, cudaStream_t st)
{
    if (nbits < 1 || nbits > 32 || g.nsteps < 2 || g.nsteps > kPhaseGroupMax) return cudaErrorInvalidValue;
    const uint64_t nmask = nbits == 32 ? 0xFFFFFFFFull : ((uint64_t(1) << nbits) - 1);
    IndexMap map{};
    map.nz = g.nsteps;
    for (int b = 0; b < g.nsteps; ++b) map.zpos[b] = g.t[b];
    std::sort(map.zpos, map.zpos + map.nz);
    const uint64_t units = total >> g.nsteps;
    switch (g.nsteps) {
        case 2: return launch_group<2>(amps, units, g, map, nmask, d_tables, sm_count, st);
        case 3: return launch_group<3>(amps, units, g, map, nmask, d_tables, sm_count, st);
        default: return launch_group<4>(amps, units, g, map, nmask, d_tables, sm_count, st);
    }
}

void phase_run_tables(int nbits, double c, const double* lin0, const double* lin1, float2* out)
{
    for (int t = 0; t < 2; ++t) {
        const double* coef = t == 0 ? lin0 : lin1;
        for (int b = 0; b < 4; ++b)
            for (int v = 0; v < 256; ++v) {
                double ph = (t == 0 && b == 0) ? c : 0.0;
                for (int k = 0; k < 8; ++k) {
                    const int pos = 8 * b + k;
                    if (pos < nbits && ((v >> k) & 1)) ph += coef[pos];
                }
                out[t * 1024 + b * 256 + v] = make_float2((float)std::cos(ph), (float)std::sin(ph));
            }
    }
}

cudaError_t launch_phase_run(float2* amps, uint64_t total, int nbits, int pivot_pos, const void* dtab, int q_pos,
                             const double* m2, int sm_count, cudaStream_t st)
{
    if (nbits < 1 || nbits > 32) return cudaErrorInvalidValue;
    const uint64_t nmask = nbits == 32 ? 0xFFFFFFFFull : ((uint64_t(1) << nbits) - 1);
    const uint64_t units = total / 2;   // amplitude pairs, or pairs of adjacent amplitudes
    const unsigned want = (unsigned)std::max<uint64_t>(1, (units + kPhaseThreads - 1) / kPhaseThreads);
    const unsigned grid = std::min<unsigned>(want, (unsigned)std::max(1, sm_count) * 8u);
    const float2* tab = static_cast<const float2*>(dtab);
    if (q_pos < 0) {
        k_phase_run<<<grid, kPhaseThreads, 0, st>>>(amps, total, nmask, pivot_pos, tab);
    } else {
        IndexMap map{};
        map.nz = 1;
        map.zpos[0] = q_pos;
        map.setmask = 0;
        Mat2f m{make_float2((float)m2[0], (float)m2[1]), make_float2((float)m2[2], (float)m2[3]),
                make_float2((float)m2[4], (float)m2[5]), make_float2((float)m2[6], (float)m2[7])};
        k_phase_pair<<<grid, kPhaseThreads, 0, st>>>(amps, total / 2, map, uint64_t(1) << q_pos, nmask, pivot_pos,
                                                     tab, m);
    }
    return cudaGetLastError();
}

}  // namespace q1g
