// Batched execution of many independent circuits in one persistent launch.
//
// Each circuit is a short program over its own complex64 state of up to
// kBatchMaxCols run columns (src/vectorstate.rs:24-35): fused gate blocks,
// up to four mid-circuit measurements, each splitting every column by its
// outcome (src/vectorstate.rs:237-329), gates conditioned on a classical bit
// (src/vectorstate.rs:193-227; every run of a column holds the same bits)
// and a final measure_all (src/vectorstate.rs:106-161).  The kernel keeps one CTA
// per SM; a CTA takes the next circuit from an atomic queue (largest circuits
// first) and runs its whole program: the gate passes stream the circuit's
// columns through registers, the measurement reduces and splits the column, and
// the shots are sampled from the final columns with the same search as the
// single-state sampler.  The host replays the launch from a CUDA graph.
//
// A batch's largest circuits can outlast all the others (160 circuits of 8 to 17
// qubits: 5.5 ms, of which the SMs worked a fifth).  Where the host's estimate
// says so (plan_teams) the launch has clusters of 2 to 8 CTAs: a cluster first
// takes circuits from a queue of the largest and runs each as a team, its tiles,
// amplitudes and shots dealt over the CTAs with a cluster barrier where the lone
// CTA has a block barrier, then its CTAs go on alone.  Sums keep the order of
// the lone CTA (the weights' 16 warps are dealt out as such, the scans are done
// by one CTA), so a circuit's words do not depend on how it ran.  The same
// batch: 1.9 ms.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>

#include <cooperative_groups.h>

#include "engine.h"
#include "sampling.cuh"
#include "warp_tile.cuh"

namespace q1g {

namespace {

constexpr int kBatchThreads = 512;
constexpr int kBatchWarps = kBatchThreads / 32;

// The CTAs that run a circuit together: one, or a cluster.  Rank and size are
// in shared memory, read where they are used.  kTeams false: always one CTA.
template <bool kTeams>
struct Team {
    const uint32_t* s;      // rank, size

    __device__ uint32_t rank() const { return kTeams ? lds_u32(s) : 0u; }
    __device__ uint32_t size() const { return kTeams ? lds_u32(s + 1) : 1u; }
    // Every thread of every CTA: what was written to global memory or to a
    // peer's shared memory before is seen by all after.  (The fences put the
    // plain loads that follow past the L1, whose lines a peer may have
    // rewritten.)
    __device__ void sync() const
    {
        if (size() == 1) {
            __syncthreads();
            return;
        }
        __threadfence();
        cooperative_groups::this_cluster().sync();
        __threadfence();
    }
    template <typename T>
    __device__ void tell(T* shared, T v) const      // the peers' copy of a shared variable
    {
        const uint32_t n = size();
        if (n == 1) *shared = v;
        else
            for (uint32_t r = 0; r < n; ++r) *cooperative_groups::this_cluster().map_shared_rank(shared, r) = v;
    }
    __device__ uint64_t first() const { return (uint64_t)rank() * kBatchThreads + threadIdx.x; }
    __device__ uint64_t step() const { return (uint64_t)size() * kBatchThreads; }
    __device__ uint64_t first_warp() const { return (uint64_t)rank() * kBatchWarps + (threadIdx.x >> 5); }
    __device__ uint64_t warps() const { return (uint64_t)size() * kBatchWarps; }
};

__device__ __forceinline__ double block_reduce(double v, double* red)
{
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    for (int k = 0; k < kBatchWarps; ++k) s += red[k];
    return s;
}

// In-place exclusive FP64 scan of n values by the whole CTA; returns the sum.
__device__ double block_scan_excl(double* data, uint64_t n, double* wsum)
{
    double carry = 0.0;
    const int l = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (uint64_t t0 = 0; t0 < n; t0 += 4 * kBatchThreads) {
        const uint64_t base = t0 + 4 * (uint64_t)threadIdx.x;
        double v[4], local = 0.0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            v[k] = base + k < n ? data[base + k] : 0.0;
            local += v[k];
        }
        double incl = local;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, incl, o);
            if (l >= o) incl += y;
        }
        __syncthreads();
        if (l == 31) wsum[w] = incl;
        __syncthreads();
        double before = carry, tile = 0.0;
        for (int k = 0; k < kBatchWarps; ++k) {
            if (k < w) before += wsum[k];
            tile += wsum[k];
        }
        double run = before + (incl - local);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (base + k < n) data[base + k] = run;
            run += v[k];
        }
        carry += tile;
    }
    __syncthreads();
    return carry;
}

// Smallest k with Binomial(n, p) CDF(k) > u; the host's binomial_inv.  The
// CTA evaluates the probability terms of up to kBinomChunk consecutive k in
// parallel into `terms`; thread 0 then accumulates them in ascending k, the
// same sums in the same order as the one-thread loop, so the same k.  Called
// by every thread of the CTA with the same arguments.  lfact[k]: lgamma(k + 1)
// for k < nlfact, made once per batch (1025 terms of two lgamma each took 100 us
// of an SM's FP64 pipe per measured column).
constexpr int kBinomChunk = 4096;
static_assert(kBinomChunk <= kBatchWarps * (1 << 10), "the terms fit in the tile stage");

__device__ __noinline__ uint64_t binomial_inv_block(uint64_t n, double p, double u, const double* lfact, uint64_t nlfact,
                                       double* terms, uint64_t* s_k)
{
    if (n == 0 || p <= 0.0) return 0;
    if (p >= 1.0) return n;
    const double nn = (double)n;
    const double mean = nn * p;
    const double sd = sqrt(nn * p * (1.0 - p));
    const double lo_d = floor(mean - 40.0 * sd - 40.0);
    const double hi_d = ceil(mean + 40.0 * sd + 40.0);
    const uint64_t lo = lo_d < 0.0 ? 0 : (uint64_t)lo_d;
    const uint64_t hi = hi_d > nn ? n : (uint64_t)hi_d;
    const double lp = log(p), lq = log1p(-p);
    const bool listed = n < nlfact;
    const double lnf = listed ? lfact[n] : lgamma(nn + 1.0);
    double cdf = 0.0;   // thread 0's running sum
    for (uint64_t k0 = lo; k0 <= hi; k0 += kBinomChunk) {
        const uint64_t cnt = hi - k0 + 1 < (uint64_t)kBinomChunk ? hi - k0 + 1 : (uint64_t)kBinomChunk;
        for (uint64_t j = threadIdx.x; j < cnt; j += kBatchThreads) {
            const double kk = (double)(k0 + j);
            const double lk = listed ? lfact[k0 + j] : lgamma(kk + 1.0);
            const double lr = listed ? lfact[n - (k0 + j)] : lgamma(nn - kk + 1.0);
            terms[j] = exp(lnf - lk - lr + kk * lp + (nn - kk) * lq);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            uint64_t found = ~uint64_t(0);
            for (uint64_t j = 0; j < cnt; ++j) {
                cdf += terms[j];
                if (u < cdf) {
                    found = k0 + j;
                    break;
                }
            }
            *s_k = found;
        }
        __syncthreads();
        const uint64_t f = *s_k;
        __syncthreads();
        if (f != ~uint64_t(0)) return f;
    }
    return hi;
}

// This CTA's share of a column's m shots.  us[j + 1] / esum: the j-th ascending
// uniform.  (Not inlined, like the other FP64 parts: the dense passes need the
// registers.)
template <bool kTeams>
__device__ __noinline__ void sample_shots(const float2* a, uint64_t chunk, const double* excl, uint64_t nch,
                                          double total, const double* us, double esum, uint64_t m, int nbits,
                                          const uint64_t* cpos, uint64_t mask, uint64_t* res, Team<kTeams> team)
{
    // up to 32 shots per warp at a time, fewer where that leaves warps without any
    const int lane = threadIdx.x & 31;
    const uint64_t per = min((m + team.warps() - 1) / team.warps(), uint64_t(32));
    for (uint64_t j0 = per * team.first_warp(); j0 < m; j0 += per * team.warps()) {
        const int count = (int)min(m - j0, per);
        const double target = lane < count ? shot_target(us[j0 + lane + 1] / esum, total) : 0.0;
        const uint64_t idx =
            sample_warp<false>(a, chunk, excl, nch, (const float*)nullptr, target, count, lane);
        if (lane < count) {
            uint64_t* r = res + j0 + lane;
            *r = (*r & mask) | outcome_word(idx, nbits, cpos);
        }
    }
}

// States below 10 qubits (smaller than a warp tile): one unit (the 2^TB amplitudes a
// block mixes) per thread.  mat[r * D + s] is the block's entry (r, s).
template <int TB>
__device__ void dense_pass(float2* a, uint64_t n_amps, const BatchOp& op, const float2* mat)
{
    constexpr int D = 1 << TB;
    const uint64_t units = n_amps >> op.map.nz;
    for (uint64_t u = threadIdx.x; u < units; u += kBatchThreads) {
        const uint64_t i = expand_index(u, op.map);
        float2 xa[D], xb[D];
#pragma unroll
        for (int s = 0; s < D; ++s) {
            const float2 v = a[i | op.offs[s]];
            xa[s] = make_float2(v.x, v.x);
            xb[s] = make_float2(v.y, v.y);
        }
#pragma unroll
        for (int r = 0; r < D; ++r) {
            float2 ac = make_float2(0.f, 0.f), bc = make_float2(0.f, 0.f);
#pragma unroll
            for (int s = 0; s < D; ++s) {
                const float2 e = lds_entry(mat + r * D + s);
                ac = __ffma2_rn(xa[s], e, ac);
                bc = __ffma2_rn(xb[s], e, bc);
            }
            a[i | op.offs[r]] = cdot_out(ac, bc);
        }
    }
}

template <int TB, bool kTeams>
__device__ __forceinline__ void apply_dense(float2* a, uint64_t n_amps, const BatchOp& op, const float2* mat,
                                            float2* stage, const Team<kTeams>& team)
{
    // (teams take circuits of whole tiles only)
    if (op.tile.tiled)
        tiled_dense_c64<TB, true>(a, n_amps, op.tile, mat, stage, (uint32_t)team.first_warp(),
                                  [&] { return (uint32_t)kBatchWarps * team.size(); });
    else dense_pass<TB>(a, n_amps, op, mat);
}

// This thread's part of a column's weight of outcome 0 as thread `t` of a lone
// CTA.
__device__ __noinline__ double weight_part(const float2* col, uint64_t n_amps, uint64_t bit, uint64_t t)
{
    double acc = 0.0;
    const float4* c4 = reinterpret_cast<const float4*>(col);   // two amplitudes (N >= 2)
#pragma unroll 4
    for (uint64_t v = t; v < n_amps / 2; v += kBatchThreads) {
        const float4 q = c4[v];
        if (!((2 * v) & bit)) acc += (double)psq(make_float2(q.x, q.y));
        if (!((2 * v + 1) & bit)) acc += (double)psq(make_float2(q.z, q.w));
    }
    return acc;
}

// kTeams: launched in clusters.  (The lone CTAs' kernel is one without teams: its
// passes take 10 % less.)
template <bool kTeams>
__global__ void __launch_bounds__(kBatchThreads, 1)
k_batch(BatchArgs args)
{
    __shared__ float2 smat[256];
    __shared__ BatchOp sop;
    __shared__ uint64_t s_n0;
    extern __shared__ float2 stage_all[];
    float2* stage = stage_all + (threadIdx.x >> 5) * (1 << 10);
    __shared__ double red[kBatchWarps];
    __shared__ int s_circ;
    // per run column: runs, classical bits of its runs, and during a
    // measurement the weight of outcome 0, the draw and the first new slot
    __shared__ int s_ncols, s_nnew;
    __shared__ uint64_t s_counts[kBatchMaxCols], s_colword[kBatchMaxCols], s_n0k[kBatchMaxCols];
    __shared__ double s_w0[kBatchMaxCols];
    __shared__ int s_newidx[kBatchMaxCols];
    // a team's weights in parts (column of the round, warp of the lone CTA), and
    // its scans' totals
    __shared__ double s_part[8][kBatchWarps], s_tot[2];
    __shared__ uint32_t s_team[2];
    const Team<kTeams> team{s_team};
    if (kTeams && threadIdx.x == 0) {
        s_team[0] = cooperative_groups::this_cluster().block_rank();
        s_team[1] = cooperative_groups::this_cluster().num_blocks();
    }
    __syncthreads();
    team.sync();      // the peers have started
    // algorithmic bytes (each pass's reads and writes of amplitudes and
    // classical words), counted by thread 0 in shared memory (no register is
    // held across the passes) and summed over the CTAs
    __shared__ unsigned long long s_moved;
    __shared__ unsigned s_cpass;   // dense column passes of the current circuit
    if (threadIdx.x == 0) s_moved = 0;

    for (;;) {
        if (team.size() > 1) {
            if (team.rank() == 0 && threadIdx.x == 0) team.tell(&s_circ, (int)atomicAdd(args.queue, 1u));
            team.sync();
            const bool alone = s_circ >= args.nteam;
            __syncthreads();
            if (alone) {
                if (threadIdx.x == 0) s_team[0] = 0, s_team[1] = 1;
                __syncthreads();
                continue;
            }
        } else {
            if (threadIdx.x == 0) s_circ = args.nteam + (int)atomicAdd(args.queue + 1, 1u);
            __syncthreads();
        }
        const int c = s_circ;
        __syncthreads();
        if (c >= args.ncircuits) break;
        const BatchCircuit C = args.circuits[c];
        const uint64_t N = uint64_t(1) << C.nbits;
        float2* const col0 = args.arena + C.state_off;
        auto col = [&](int k) { return col0 + (uint64_t)k * N; };
        uint64_t* res = args.results + C.res_off;
        for (uint64_t v = team.first(); v < N / 2; v += team.step())
            reinterpret_cast<float4*>(col0)[v] = make_float4(v == 0 ? 1.f : 0.f, 0.f, 0.f, 0.f);
        if (threadIdx.x == 0) {
            s_ncols = 1;
            s_counts[0] = C.nshots;
            s_colword[0] = 0;
        }
        uint64_t ctr = 0;   // position in the circuit's uniform stream
        if (threadIdx.x == 0) {
            if (team.rank() == 0) s_moved += N * sizeof(float2);
            s_cpass = 0;
        }
        team.sync();
        for (uint32_t oi = C.op_begin; oi < C.op_end; ++oi) {
            {
                static_assert(sizeof(BatchOp) % 4 == 0, "BatchOp copies as 32-bit words");
                const uint32_t* src = reinterpret_cast<const uint32_t*>(args.ops + oi);
                uint32_t* dst = reinterpret_cast<uint32_t*>(&sop);
                for (int w = threadIdx.x; w < (int)(sizeof(BatchOp) / 4); w += kBatchThreads) dst[w] = src[w];
            }
            __syncthreads();
            const int kind = sop.kind;
            if (kind == kBatchDense) {
                const int D = 1 << sop.t;
                for (int e = threadIdx.x; e < D * D; e += kBatchThreads) smat[e] = args.mats[sop.mat + e];
                __syncthreads();
                for (int k = 0; k < s_ncols; ++k) {
                    if (sop.cond >= 0 && (int)((s_colword[k] >> sop.ccbit) & 1u) != sop.cond) continue;
                    if (threadIdx.x == 0) ++s_cpass;
                    switch (sop.t) {
                        case 1: apply_dense<1>(col(k), N, sop, smat, stage, team); break;
                        case 2: apply_dense<2>(col(k), N, sop, smat, stage, team); break;
                        case 3: apply_dense<3>(col(k), N, sop, smat, stage, team); break;
                        default: apply_dense<4>(col(k), N, sop, smat, stage, team); break;
                    }
                }
                team.sync();
            } else if (kind == kBatchMeasure) {
                // per column: P(bit = 0) (src/vectorstate.rs:252-261) and
                // n0 ~ Binomial(runs, P) from the next uniform of the stream
                const uint64_t bit = uint64_t(1) << sop.pos;
                const int nc = s_ncols;
                const uint32_t share = kBatchWarps / team.size();      // of the lone CTA's warps, a CTA's
                for (int k = 0; k < nc; ++k) {
                    double w0;
                    if (team.size() == 1) {
                        w0 = block_reduce(weight_part(col(k), N, bit, threadIdx.x), red);
                    } else {
                        // team.size() columns per round: warp w sums column
                        // k + w / share as the lone CTA's warp rank * share + w % share
                        const int at = k % (int)team.size();
                        if (at == 0) {
                            const uint32_t w = threadIdx.x >> 5, mine = w / share, vw = team.rank() * share + w % share;
                            if (k) team.sync();      // the last round's parts have been read
                            if (k + (int)mine < nc) {
                                const double part =
                                    warp_sum(weight_part(col(k + mine), N, bit, vw * 32 + (threadIdx.x & 31)));
                                if ((threadIdx.x & 31) == 0) team.tell(&s_part[mine][vw], part);
                            }
                            __syncwarp();
                            team.sync();
                        }
                        w0 = 0.0;
                        for (int w = 0; w < kBatchWarps; ++w) w0 += s_part[at][w];
                    }
                    const uint64_t n0 = binomial_inv_block(s_counts[k], fmin(w0, 1.0), stream_uniform(C.seed, ctr + k),
                                                           args.lfact, args.nlfact,
                                                           reinterpret_cast<double*>(stage_all), &s_n0);
                    if (threadIdx.x == 0) {
                        s_w0[k] = w0;
                        s_n0k[k] = n0;
                    }
                    __syncthreads();
                }
                ctr += nc;
                // results: a column's first n0 runs read 0, the rest 1
                // (src/vectorstate.rs:290-297)
                {
                    const uint64_t one = uint64_t(1) << sop.cbit;
                    uint64_t r0 = 0;
                    for (int k = 0; k < nc; ++k) {
                        const uint64_t m = s_counts[k], n0 = s_n0k[k];
                        for (uint64_t r = team.first(); r < m; r += team.step())
                            res[r0 + r] = r < n0 ? (res[r0 + r] & ~one) : (res[r0 + r] | one);
                        r0 += m;
                    }
                }
                // the new columns: outcome 0 then outcome 1 of each old column,
                // the empty ones left out (src/vectorstate.rs:299-322)
                if (threadIdx.x == 0) {
                    int nn = 0;
                    for (int k = 0; k < nc; ++k) {
                        s_newidx[k] = nn;
                        nn += (s_n0k[k] > 0 ? 1 : 0) + (s_n0k[k] < s_counts[k] ? 1 : 0);
                    }
                    s_nnew = nn;
                    if (team.rank() == 0)
                        s_moved += (uint64_t)(2 * nc + nn) * N * sizeof(float2) + 2 * C.nshots * sizeof(uint64_t);
                }
                __syncthreads();
                // collapse (src/vectorstate.rs:91-104), in place from the last
                // column down: column k's new slots lie at or above k and
                // below the slots of the columns after it (a team's thread has
                // the same amplitudes of every column, so its order suffices)
                for (int k = nc - 1; k >= 0; --k) {
                    const uint64_t m = s_counts[k], n0 = s_n0k[k];
                    const bool has0 = n0 > 0, has1 = n0 < m;
                    const double w0 = s_w0[k];
                    const float f0 = has0 ? (float)(1.0 / sqrt(w0)) : 0.f;
                    const float f1 = has1 ? (float)(1.0 / sqrt(1.0 - w0)) : 0.f;
                    const int base = s_newidx[k];
                    const float4* src = reinterpret_cast<const float4*>(col(k));
                    float4* d0 = reinterpret_cast<float4*>(col(base));
                    float4* d1 = reinterpret_cast<float4*>(col(base + (has0 ? 1 : 0)));
#pragma unroll 4
                    for (uint64_t v = team.first(); v < N / 2; v += team.step()) {
                        const float4 q = src[v];
                        const bool b0 = ((2 * v) & bit) != 0, b1 = ((2 * v + 1) & bit) != 0;
                        if (has1)
                            d1[v] = make_float4(b0 ? q.x * f1 : 0.f, b0 ? q.y * f1 : 0.f, b1 ? q.z * f1 : 0.f,
                                                b1 ? q.w * f1 : 0.f);
                        if (has0)
                            d0[v] = make_float4(b0 ? 0.f : q.x * f0, b0 ? 0.f : q.y * f0, b1 ? 0.f : q.z * f0,
                                                b1 ? 0.f : q.w * f0);
                    }
                    __syncthreads();
                }
                // the column list (runs and classical bits) follows the split
                if (threadIdx.x == 0) {
                    const uint64_t one = uint64_t(1) << sop.cbit;
                    for (int k = nc - 1; k >= 0; --k) {
                        const uint64_t m = s_counts[k], n0 = s_n0k[k], w = s_colword[k] & ~one;
                        int slot = s_newidx[k];
                        if (n0 > 0) {
                            s_counts[slot] = n0;
                            s_colword[slot] = w;
                            ++slot;
                        }
                        if (n0 < m) {
                            s_counts[slot] = m - n0;
                            s_colword[slot] = w | one;
                        }
                    }
                    s_ncols = s_nnew;
                }
                team.sync();
            } else if (kind == kBatchSample) {
                const uint64_t* cpos = args.cbit_tables + 64 * (uint64_t)sop.cpos;
                const uint64_t mask = ~sop.cmask;
                const uint64_t chunk = N < 256 ? N : 256;
                const uint64_t nch = N / chunk;
                double* excl = args.scratch + (uint64_t)(blockIdx.x - team.rank()) * args.scratch_per_cta;   // the first CTA's
                double* us = excl + nch;
                uint64_t r0 = 0;
                for (int k = 0; k < s_ncols; ++k) {
                    const uint64_t m = s_counts[k];
                    const int lane = threadIdx.x & 31;
                    for (uint64_t ch = team.first_warp(); ch < nch; ch += team.warps()) {
                        const double sum = chunk_sum(col(k), ch * chunk, chunk, lane);
                        if (lane == 0) excl[ch] = sum;
                    }
                    // ascending uniforms: normalised exponential spacings
                    for (uint64_t j = team.first(); j <= m; j += team.step())
                        us[j] = -log1p(-stream_uniform(C.seed, ctr + j));
                    team.sync();
                    if (team.rank() == 0) {
                        const double t = block_scan_excl(excl, nch, red);
                        if (threadIdx.x == 0) team.tell(&s_tot[0], t);
                    }
                    if (team.rank() == team.size() - 1) {
                        const double t = block_scan_excl(us, m + 1, red);
                        if (threadIdx.x == 0) team.tell(&s_tot[1], t);
                    }
                    team.sync();
                    const double total = s_tot[0], esum = s_tot[1];
                    // us[j] now holds S_{j-1}
                    sample_shots(col(k), chunk, excl, nch, total, us, esum, m, C.nbits, cpos, mask, res + r0, team);
                    ctr += m + 1;
                    r0 += m;
                    if (team.rank() == 0 && threadIdx.x == 0)
                        s_moved += N * sizeof(float2) + m * (chunk * sizeof(float2) + 2 * sizeof(uint64_t));
                    team.sync();
                }
            }
        }
        __syncthreads();
        if (team.rank() == 0 && threadIdx.x == 0) s_moved += (unsigned long long)s_cpass * 2 * N * sizeof(float2);
    }
    if (threadIdx.x == 0) atomicAdd(args.traffic, s_moved);
}

__global__ void k_log_factorials(double* out, uint64_t n)
{
    const uint64_t k = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k < n) out[k] = lgamma((double)k + 1.0);
}

}  // namespace

cudaError_t launch_log_factorials(double* out, uint64_t n, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    k_log_factorials<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(out, n);
    return cudaGetLastError();
}

constexpr size_t kBatchStageBytes = size_t(kBatchWarps) * (size_t(1) << 10) * sizeof(float2);

cudaError_t setup_batch_kernel()
{
    const cudaError_t e =
        cudaFuncSetAttribute(k_batch<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBatchStageBytes);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_batch<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBatchStageBytes);
}

static cudaLaunchConfig_t batch_config(unsigned grid, int cluster, cudaLaunchAttribute* attr, cudaStream_t st)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kBatchThreads);
    cfg.dynamicSmemBytes = kBatchStageBytes;
    cfg.stream = st;
    attr->id = cudaLaunchAttributeClusterDimension;
    attr->val.clusterDim.x = (unsigned)cluster;
    attr->val.clusterDim.y = attr->val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 1 : 0;
    return cfg;
}

cudaError_t batch_clusters(int cluster, int sm_count, int* count)
{
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = batch_config((unsigned)(sm_count / cluster * cluster), cluster, &attr, nullptr);
    return cudaOccupancyMaxActiveClusters(count, k_batch<true>, &cfg);
}

cudaError_t launch_batch(const BatchArgs& a, unsigned grid, int cluster, cudaStream_t st)
{
    if (grid == 0) return cudaSuccess;
    cudaLaunchAttribute attr;
    const cudaLaunchConfig_t cfg = batch_config(grid, cluster, &attr, st);
    return cluster > 1 ? cudaLaunchKernelEx(&cfg, k_batch<true>, a) : cudaLaunchKernelEx(&cfg, k_batch<false>, a);
}

}  // namespace q1g
