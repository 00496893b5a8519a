// Device helpers shared by the shot samplers (measure_kernels.cu and the
// batched executor): the SplitMix64 uniform stream, |a|^2 group sums, and the
// per-shot search.
//
// Outcome probabilities are summed hierarchically, with the same arithmetic
// in the reduction and in the search so the two agree: p_i = |a_i|^2 in the
// state's precision, groups of 8 consecutive p_i summed sequentially in that
// precision, chunks of 32 groups (256 amplitudes) summed in the state's
// precision too (FP64 for complex128), and an FP64 exclusive prefix over
// chunks.  A shot finds its chunk by a search on that prefix, its group by a
// warp scan of the chunk's 32 group sums, and its amplitude by a sequential
// scan of the group.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace q1g {

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// SplitMix64 (Steele, Lea & Flood 2014): draw k of stream `seed` is
// mix(seed + (k+1) * golden_gamma) as a 53-bit uniform in [0, 1).
__device__ __forceinline__ uint64_t splitmix_mix(uint64_t z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

__device__ __forceinline__ double stream_uniform(uint64_t seed, uint64_t counter)
{
    const uint64_t z = seed + (counter + 1) * 0x9E3779B97F4A7C15ULL;
    return (double)(splitmix_mix(z) >> 11) * (1.0 / 9007199254740992.0);
}

template <typename T> struct ProbT;
template <> struct ProbT<float2> { using R = float; };
template <> struct ProbT<double2> { using R = double; };

__device__ __forceinline__ float psq(float2 v) { return __fmaf_rn(v.x, v.x, __fmul_rn(v.y, v.y)); }
__device__ __forceinline__ double psq(double2 v) { return __fma_rn(v.x, v.x, __dmul_rn(v.y, v.y)); }
__device__ __forceinline__ float padd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double padd(double a, double b) { return __dadd_rn(a, b); }

// p of the 8 amplitudes [8*lane, 8*lane+8) of the chunk at i0.
__device__ __forceinline__ void group_probs(const float2* a, uint64_t i0, uint64_t chunk, int lane, float p[8])
{
    const uint64_t g0 = (uint64_t)lane * 8;
    if (chunk >= 256) {
        const float4* v = reinterpret_cast<const float4*>(a + i0 + g0);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 w = v[q];
            p[2 * q] = psq(make_float2(w.x, w.y));
            p[2 * q + 1] = psq(make_float2(w.z, w.w));
        }
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) p[e] = g0 + e < chunk ? psq(a[i0 + g0 + e]) : 0.0f;
    }
}

__device__ __forceinline__ void group_probs(const double2* a, uint64_t i0, uint64_t chunk, int lane, double p[8])
{
    const uint64_t g0 = (uint64_t)lane * 8;
#pragma unroll
    for (int e = 0; e < 8; ++e) p[e] = g0 + e < chunk ? psq(a[i0 + g0 + e]) : 0.0;
}

template <typename R>
__device__ __forceinline__ R group_sum(const R p[8])
{
    R s = p[0];
#pragma unroll
    for (int e = 1; e < 8; ++e) s = padd(s, p[e]);
    return s;
}

// The first amplitude of a group whose inclusive prefix exceeds `local`, or the
// last nonzero one.
template <typename R>
__device__ __forceinline__ int pick_in_group(const R p[8], R local)
{
    int e_pick = -1, e_last = 0;
    R run = R(0);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        run = padd(run, p[e]);
        if (p[e] > R(0)) {
            e_last = e;
            if (e_pick < 0 && run > local) e_pick = e;
        }
    }
    return e_pick < 0 ? e_last : e_pick;
}

// Inclusive prefix of v over the warp's lanes, in v's precision: the order
// in which the sampler adds a chunk's 32 group sums.
template <typename R>
__device__ __forceinline__ R warp_incl_scan(R v, int lane)
{
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const R y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
    }
    return v;
}

// A chunk's total from its lanes' group sums (all lanes get it).
// complex64: in FP32, in the sampler's scan order, so that the total is the
// value the sampler's scan reaches at lane 31 (an FP64 warp reduction costs
// 16 cycles of an SM's FP64 pipe per instruction; a chunk holds about 2^-22
// of the mass at 30 qubits, so FP32 leaves it good to about 1e-14).
// complex128: in FP64.
__device__ __forceinline__ double chunk_total(float gs, int lane)
{
    return (double)__shfl_sync(0xffffffffu, warp_incl_scan(gs, lane), 31);
}
__device__ __forceinline__ double chunk_total(double gs, int) { return warp_sum(gs); }

// Chunk sum of one warp's chunk (all lanes get it).
template <typename T>
__device__ __forceinline__ double chunk_sum(const T* a, uint64_t i0, uint64_t chunk, int lane)
{
    typename ProbT<T>::R p[8];
    group_probs(a, i0, chunk, lane, p);
    return chunk_total(group_sum(p), lane);
}

// The shot's target u * total, kept strictly inside the mass if rounding
// pushed it onto the total (u < 1): the shot then lands on the last nonzero
// amplitude.
__device__ __forceinline__ double shot_target(double u, double total)
{
    const double target = u * total;
    return target < total ? target : nextafter(total, 0.0);
}

// 32 shots of a column by a warp: lane r's has the target `target`; lanes from
// `count` on have none.  Each lane finds its shot's chunk (the largest c with
// excl[c] <= target; excl is non-decreasing, excl[0] = 0) by a binary search:
// shots are sorted, so the lanes' probes share their cache lines.  Then the warp
// finds the shots' groups one after the other by a scan of the chunk's 32 group
// sums (from `groups`, or from the amplitudes), and each lane its shot's
// amplitude in its group.  Returns the lane's basis index: the first whose
// inclusive probability prefix exceeds the target.
template <bool kGroups, typename T>
__device__ __forceinline__ uint64_t sample_warp(const T* a, uint64_t chunk, const double* excl, uint64_t nchunks,
                                                const typename ProbT<T>::R* groups, double target, int count, int lane)
{
    using R = typename ProbT<T>::R;
    constexpr int kAhead = kGroups ? 8 : 2;      // chunks read at once
    uint64_t lo = 0, hi = nchunks;
    while (hi - lo > 1) {
        const uint64_t mid = (lo + hi) >> 1;
        if (excl[mid] <= target) lo = mid;
        else hi = mid;
    }
    // the target's offset into the chunk, in the state's precision (it is at
    // most the chunk's mass)
    const R offset = (R)(target - excl[lo]);
    int group = 0;
    R local = R(0);
    for (int k0 = 0; k0 < count; k0 += kAhead) {
        R gs[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const uint64_t c = __shfl_sync(0xffffffffu, lo, k0 + k);
            if (kGroups) {
                gs[k] = groups[c * 32 + lane];
            } else {
                R p[8];
                group_probs(a, c * chunk, chunk, lane, p);
                gs[k] = group_sum(p);
            }
        }
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            // the group sums scanned in the state's precision (the chunk
            // sums add them in the same order, chunk_total)
            const R t = __shfl_sync(0xffffffffu, offset, k0 + k);
            const R incl = warp_incl_scan(gs[k], lane);
            const unsigned hit = __ballot_sync(0xffffffffu, gs[k] > R(0) && incl > t);
            const unsigned nz = __ballot_sync(0xffffffffu, gs[k] > R(0));
            const int owner = hit ? __ffs(hit) - 1 : nz ? 31 - __clz(nz) : 0;
            const R before = __shfl_sync(0xffffffffu, incl - gs[k], owner);
            if (lane == k0 + k) {
                group = owner;
                // past the end: the group's last nonzero amplitude
                local = hit ? t - before : R(INFINITY);
            }
        }
    }
    R p[8];
    group_probs(a, lo * chunk, chunk, group, p);
    return lo * chunk + (uint64_t)group * 8 + (uint64_t)pick_in_group(p, local);
}

// Classical word of outcome idx: bit position p of idx goes to the mask
// cbit_of_pos[p] (qubit q = position n-1-q lands on cbits[q]).
__device__ __forceinline__ uint64_t outcome_word(uint64_t idx, int nbits, const uint64_t* cbit_of_pos)
{
    uint64_t word = 0;
    for (int q = 0; q < nbits; ++q)
        if ((idx >> q) & 1) word |= cbit_of_pos[q];
    return word;
}

}  // namespace q1g
