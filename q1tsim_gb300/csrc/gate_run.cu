// Tile passes of plain gates (gate_run.h): each CTA loads one tile of up to
// 2048 amplitudes into shared memory, applies the pass's gates to it one
// after the other, and stores it back.
//
// complex128 tiles are held as double-float pairs (re.h, re.l, im.h, im.l):
// the same 16 bytes, split once on load and joined once on store instead of
// once per gate, with the arithmetic of the one-gate kernel (df64.cuh).  A
// tile holding an amplitude of 2^63 or more (or an infinity or NaN) is done
// in FP64 instead; run_takes keeps gates that grow amplitudes out of runs.
// Splitting rounds an amplitude to 49 bits, as the arithmetic of one gate does.
// Amplitudes that no gate of a pass rounds keep their bits all the same: passes
// of permutations alone hold doubles (RunArith::kPlain), passes in which gates
// round only some amplitudes follow those that they do not (tags).
//
// What bounds it: on large states the FP32 pipe (double-float products; the
// memory is read and written once per 40-60 gates), on small ones the
// latency of a gate's chain, about 0.5 us.  Measured on one GB300 against one
// launch and one HBM pass per gate: complex128 brick circuits of 10 qubits,
// depth 8 (116 gates), with shots, 0.63 -> 0.12 ms, 16 qubits, depth 20 (470
// gates) 2.86 -> 0.40 ms, both with the plan's launches kept; 26 qubits, depth 6
// (231 gates) 59.9 -> 35.5 ms (most gates of complex128 states of that size take
// the tensor cores now: 9.4 ms).
#include <algorithm>
#include <mutex>
#include <set>
#include <utility>

#include "df64.cuh"
#include "gate_run.h"

namespace q1g {

namespace {

// Threads of a CTA (2^bits): the double-float pairs of a tile keep 256 busy;
// FP32 and FP64 tiles run better as more, smaller blocks (22 qubits,
// complex64, 198 gates: 0.76 ms with 128 threads, 1.09 ms with 256).
constexpr int kRunBitsDf = 8, kRunBitsPlain = 7;

// Slot of local index i in the staged tile.  Consecutive units of a gate at
// a position inside one 128-byte row skip every other run of that row, so
// the next row's lanes take the complement: conflict-free for one zero bit.
template <class E>
__device__ __forceinline__ uint32_t slot(uint32_t i)
{
    constexpr uint32_t P = 128 / sizeof(E);
    return i ^ ((i & P) ? P - 1 : 0u);
}

// Inserts the op's zero bits into unit u.  Two masks are held in registers
// (absent ones zero); further ones, for gates with several controls inside
// the tile, are read from the table.
struct UnitMap {
    uint32_t h0, h1, set;
    int nz;
    const uint16_t* hi;
    __device__ explicit UnitMap(const RunOp& o)
        : h0(o.nz > 0 ? o.hi[0] : 0u), h1(o.nz > 1 ? o.hi[1] : 0u), set(o.set), nz((int)o.nz), hi(o.hi)
    {
    }
    __device__ __forceinline__ uint32_t operator()(uint32_t u) const
    {
        u += u & h0;
        u += u & h1;
        for (int q = 2; q < nz; ++q) u += u & hi[q];
        return u | set;
    }
};

// ------------------------------------------------ FP32 and FP64 arithmetic

template <class E> struct Coef;
template <> struct Coef<float2> {
    static __device__ __forceinline__ float2 at(const RunOp& o, int e)
    {
        return make_float2((float)o.m[2 * e], (float)o.m[2 * e + 1]);
    }
};
template <> struct Coef<double2> {
    static __device__ __forceinline__ double2 at(const RunOp& o, int e) { return make_double2(o.m[2 * e], o.m[2 * e + 1]); }
};

// A gate of 0, +-1 and +-i on a staged tile: amplitudes move bit for bit.
template <class E, int B>
__device__ __forceinline__ void apply_units(E* t, const RunOp& o, int bits)
{
    const uint32_t units = 1u << (bits - (int)o.nz);
    const UnitMap at(o);
    const int u0 = (o.code >> 1) & 3, u1 = (o.code >> 3) & 3;
    if (o.kind == kRunPairMono) {
        const bool swap = o.code & 1;
        for (uint32_t u = threadIdx.x; u < units; u += (1 << B)) {
            const uint32_t i = at(u), s0 = slot<E>(i | o.o0), s1 = slot<E>(i | o.o1);
            const E x0 = t[s0], x1 = t[s1];
            t[s0] = unit_times(u0, swap ? x1 : x0);
            t[s1] = unit_times(u1, swap ? x0 : x1);
        }
    } else {
        for (uint32_t u = threadIdx.x; u < units; u += (1 << B)) {
            const uint32_t s = slot<E>(at(u));
            t[s] = unit_times(u0, t[s]);
        }
    }
}

// One gate on a staged tile, the arithmetic of gate_kernels.cu's one-gate
// kernels.
template <class E, int B>
__device__ __forceinline__ void apply_plain(E* t, const RunOp& o, int bits)
{
    const uint32_t units = 1u << (bits - (int)o.nz);
    const UnitMap at(o);
    if (o.kind == kRunPair) {
        const E m00 = Coef<E>::at(o, 0), m01 = Coef<E>::at(o, 1), m10 = Coef<E>::at(o, 2), m11 = Coef<E>::at(o, 3);
        for (uint32_t u = threadIdx.x; u < units; u += (1 << B)) {
            const uint32_t i = at(u), s0 = slot<E>(i | o.o0), s1 = slot<E>(i | o.o1);
            const E x0 = t[s0], x1 = t[s1];
            t[s0] = cmuladd2(m00, x0, m01, x1);
            t[s1] = cmuladd2(m10, x0, m11, x1);
        }
    } else if (o.kind == kRunPhase) {
        const E ph = Coef<E>::at(o, 0);
        for (uint32_t u = threadIdx.x; u < units; u += (1 << B)) {
            const uint32_t s = slot<E>(at(u));
            t[s] = cmul(ph, t[s]);
        }
    } else {
        apply_units<E, B>(t, o, bits);
    }
}

// ------------------------------------------------ double-float arithmetic
//
// One pair per thread in scalar FP32 instructions.  The packed FP32x2 forms
// run at the same FMA rate but need their operands in adjacent registers: with
// the amplitudes as they lie the moves cost more issue slots than the packing
// saves (26 qubits, depth 6: 43.6 ms, 35.5 scalar).  With parts in planes of their
// own and two pairs per thread that was 30.4 ms, but 16 qubits took 0.38 ms for
// 0.32: a small tile has only as many pairs as threads, one pair's chain is the
// time, and small states are what this kernel serves in complex128.

// A staged amplitude (re.h, re.l, im.h, im.l), component by component.
__device__ __forceinline__ DF re_of(float4 v) { return DF{v.x, v.y}; }
__device__ __forceinline__ DF im_of(float4 v) { return DF{v.z, v.w}; }
__device__ __forceinline__ DF minus(DF v) { return DF{-v.h, -v.l}; }
__device__ __forceinline__ float4 amp_of(DF re, DF im) { return make_float4(re.h, re.l, im.h, im.l); }

// Row (a, b) of a matrix on (x0, x1), with the terms that TERMS names: bit 0
// Re a, 1 Re b, 2 Im a, 3 Im b (the others are zero).  Rows of two terms
// (phases, H, rotations) take the rest of the coefficients too: a Fourier
// transform applies the same few of them again and again, where their
// rounding would add up.
template <int TERMS>
__device__ __forceinline__ float4 df_row(float4 a, float4 b, const float* rest, float4 x0, float4 x1)
{
    constexpr int N = (TERMS & 1) + ((TERMS >> 1) & 1) + ((TERMS >> 2) & 1) + ((TERMS >> 3) & 1);
    DF m[N], u[N], v[N];
    float m2[N];
    int n = 0;
    if (TERMS & 1) m2[n] = rest[0], m[n] = re_of(a), u[n] = re_of(x0), v[n++] = im_of(x0);
    if (TERMS & 2) m2[n] = rest[2], m[n] = re_of(b), u[n] = re_of(x1), v[n++] = im_of(x1);
    if (TERMS & 4) m2[n] = rest[1], m[n] = im_of(a), u[n] = minus(im_of(x0)), v[n++] = re_of(x0);
    if (TERMS & 8) m2[n] = rest[3], m[n] = im_of(b), u[n] = minus(im_of(x1)), v[n++] = re_of(x1);
    return amp_of(dot<N>(m, u, N == 2 ? m2 : nullptr), dot<N>(m, v, N == 2 ? m2 : nullptr));
}

// Where a pass has no gate that rounds every amplitude (controlled gates and
// phases beside permutations), each slot of the tile has a tag: kTouched once
// arithmetic has written it, else the local index that its amplitude came from
// and the unit (2 bits above) that the gates have multiplied it by.  What is not
// touched is stored as the bits in memory.  26 qubits, 60 gates, ms without tags
// and with them: controlled U3 8.79 and 9.35, controlled phases 3.18 and 3.36
// (doubles in the tile, split and joined per gate: 13.9 and 7.8).  60 CX, held as
// doubles: 2.96 (4.07 in pairs).
constexpr uint16_t kTouched = 0x8000;
static_assert((4 << kRunMaxTileBits) <= kTouched, "an index and a unit fit under the mark");
__device__ __forceinline__ uint16_t tag_times(int u, uint16_t tag)
{
    return (uint16_t)((tag + (u << kRunMaxTileBits)) & (kTouched | ((4 << kRunMaxTileBits) - 1)));
}

template <int TERMS0, int TERMS1, bool TAGS>
__device__ __forceinline__ void df_pair(float4* t, uint16_t* tags, const RunOp& o, int bits)
{
    const uint32_t units = 1u << (bits - (int)o.nz), d0 = o.o0, d1 = o.o1;
    const UnitMap at(o);
    const float4 m00 = o.df[0], m01 = o.df[1], m10 = o.df[2], m11 = o.df[3];
    for (uint32_t u = threadIdx.x; u < units; u += (1 << kRunBitsDf)) {
        const uint32_t i = at(u), s0 = slot<float4>(i | d0), s1 = slot<float4>(i | d1);
        const float4 x0 = t[s0], x1 = t[s1];
        t[s0] = df_row<TERMS0>(m00, m01, o.rest, x0, x1);
        t[s1] = df_row<TERMS1>(m10, m11, o.rest + 4, x0, x1);
        if (TAGS) tags[i | d0] = tags[i | d1] = kTouched;
    }
}

__device__ __forceinline__ float4 df_unit_times(int u, float4 x)
{
    switch (u) {
        case 1: return make_float4(-x.z, -x.w, x.x, x.y);
        case 2: return make_float4(-x.x, -x.y, -x.z, -x.w);
        case 3: return make_float4(x.z, x.w, -x.x, -x.y);
        default: return x;
    }
}

template <bool TAGS>
__device__ __forceinline__ void apply_df(float4* t, uint16_t* tags, const RunOp& o, int bits)
{
    if (o.kind == kRunPair) {
        switch (o.shape) {
            case kRunReal00: df_pair<11, 15, TAGS>(t, tags, o, bits); break;
            case kRunReal: df_pair<3, 3, TAGS>(t, tags, o, bits); break;
            case kRunCross: df_pair<9, 6, TAGS>(t, tags, o, bits); break;
            default: df_pair<15, 15, TAGS>(t, tags, o, bits); break;
        }
        return;
    }
    const uint32_t units = 1u << (bits - (int)o.nz);
    const UnitMap at(o);
    if (o.kind == kRunPhase) {
        const float4 p = o.df[0];
        for (uint32_t u = threadIdx.x; u < units; u += (1 << kRunBitsDf)) {
            const uint32_t i = at(u), s = slot<float4>(i);
            t[s] = df_row<5>(p, p, o.rest, t[s], make_float4(0.f, 0.f, 0.f, 0.f));
            if (TAGS) tags[i] = kTouched;
        }
        return;
    }
    const int u0 = (o.code >> 1) & 3, u1 = (o.code >> 3) & 3;
    if (o.kind == kRunPairMono) {
        const bool swap = o.code & 1;
        const uint32_t d0 = o.o0, d1 = o.o1;
        for (uint32_t u = threadIdx.x; u < units; u += (1 << kRunBitsDf)) {
            const uint32_t i = at(u), s0 = slot<float4>(i | d0), s1 = slot<float4>(i | d1);
            const float4 x0 = t[s0], x1 = t[s1];
            t[s0] = df_unit_times(u0, swap ? x1 : x0);
            t[s1] = df_unit_times(u1, swap ? x0 : x1);
            if (TAGS) {
                const uint16_t g0 = tags[i | d0], g1 = tags[i | d1];
                tags[i | d0] = tag_times(u0, swap ? g1 : g0);
                tags[i | d1] = tag_times(u1, swap ? g0 : g1);
            }
        }
    } else {
        for (uint32_t u = threadIdx.x; u < units; u += (1 << kRunBitsDf)) {
            const uint32_t i = at(u), s = slot<float4>(i);
            t[s] = df_unit_times(u0, t[s]);
            if (TAGS) tags[i] = tag_times(u0, tags[i]);
        }
    }
}

// A double as a pair; *big is set when its exponent is 2^63 or above (or it
// is not finite).  Below 2^-74 the low part is dropped and below 2^-126 the
// value is a signed zero, as split_f64 (df64.cuh).
__device__ __forceinline__ DF split_run(uint64_t bits, bool& big)
{
    const uint32_t hw = (uint32_t)(bits >> 32), aw = hw & 0x7FFFFFFFu;
    big |= aw >= (1086u << 20);
    DF v = split_fast(bits);
    if (aw < (949u << 20)) split_f64(bits, v);
    return v;
}

// ------------------------------------------------------------- the kernels

// Amplitude offsets of a thread's local indices tid + 2^B k: the bits of tid
// once, those of k per element.
template <int B>
struct TileWalk {
    uint64_t base;
    int bits;
    const RunTile* tile;
    __device__ TileWalk(const RunTile& t) : bits(t.bits), tile(&t)
    {
        base = expand_index(blockIdx.x, t.map);
        own = base;
#pragma unroll
        for (int b = 0; b < B; ++b)
            if (b < bits && ((threadIdx.x >> b) & 1)) own |= t.off[b];
    }
    uint64_t own;
    __device__ __forceinline__ uint64_t at(uint32_t k) const
    {
        uint64_t o = own;
#pragma unroll
        for (int b = B; b < kRunMaxTileBits; ++b)
            if ((k >> (b - B)) & 1) o |= tile->off[b];
        return o;
    }
};

template <int B>
__device__ __forceinline__ void load_ops(RunOp* sops, const RunOp* __restrict__ ops, int nops)
{
    const uint4* s = reinterpret_cast<const uint4*>(ops);
    uint4* d = reinterpret_cast<uint4*>(sops);
    for (int i = threadIdx.x; i < nops * (int)(sizeof(RunOp) / 16); i += 1 << B) d[i] = s[i];
}

// The ops that apply to this tile, as a bit mask (nops <= 64).
__device__ __forceinline__ uint64_t active_ops(const RunOp* __restrict__ ops, int nops, uint64_t base, uint32_t* words)
{
    if (threadIdx.x < 64) {
        const int j = threadIdx.x;
        const bool on = j < nops && (base & ops[j].extmask) == ops[j].extset;
        const uint32_t b = __ballot_sync(0xffffffffu, on);
        if ((j & 31) == 0) words[j >> 5] = b;
    }
    __syncthreads();
    return words[0] | ((uint64_t)words[1] << 32);
}

// Plain arithmetic in the state's type.
template <class E, int B>
__device__ __forceinline__ void run_plain(E* a, E* t, const RunOp* sops, uint64_t active, const TileWalk<B>& w)
{
    const uint32_t size = 1u << w.bits;
    for (uint32_t l0 = threadIdx.x; l0 < size; l0 += 4 << B) {
        E v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (l0 + (q << B) < size) v[q] = a[w.at((l0 >> B) + q)];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (l0 + (q << B) < size) t[slot<E>(l0 + (q << B))] = v[q];
    }
    __syncthreads();
    for (; active; active &= active - 1) {
        apply_plain<E, B>(t, sops[__ffsll(active) - 1], w.bits);
        __syncthreads();
    }
    for (uint32_t l = threadIdx.x; l < size; l += 1 << B) a[w.at(l >> B)] = t[slot<E>(l)];
}

template <class E>
__global__ void __launch_bounds__(1 << kRunBitsPlain)
k_gate_run(E* a, const __grid_constant__ RunTile tile, const RunOp* __restrict__ ops, int nops)
{
    extern __shared__ uint4 run_smem[];
    __shared__ uint32_t words[2];
    RunOp* sops = reinterpret_cast<RunOp*>(run_smem);
    E* t = reinterpret_cast<E*>(sops + nops);
    load_ops<kRunBitsPlain>(sops, ops, nops);
    const TileWalk<kRunBitsPlain> w(tile);
    run_plain<E, kRunBitsPlain>(a, t, sops, active_ops(ops, nops, w.base, words), w);
}

// A tile outside the split's range, in FP64 from memory.
__device__ __noinline__ void run_fp64_tile(double2* a, double2* t, const RunOp* sops, uint64_t active,
                                           const RunTile& tile)
{
    run_plain<double2, kRunBitsDf>(a, t, sops, active, TileWalk<kRunBitsDf>(tile));
}

template <bool TAGS>
__global__ void __launch_bounds__(1 << kRunBitsDf, 4)
k_gate_run_c128x(double2* a, const __grid_constant__ RunTile tile, const RunOp* __restrict__ ops, int nops)
{
    constexpr int B = kRunBitsDf;
    extern __shared__ uint4 run_smem[];
    __shared__ uint32_t words[2];
    RunOp* sops = reinterpret_cast<RunOp*>(run_smem);
    float4* t = reinterpret_cast<float4*>(sops + nops);
    uint16_t* tags = reinterpret_cast<uint16_t*>(t + (1u << tile.bits));
    load_ops<B>(sops, ops, nops);
    const TileWalk<B> w(tile);
    const ulonglong2* ab = reinterpret_cast<const ulonglong2*>(a);
    const uint32_t size = 1u << w.bits;
    bool big = false;
    for (uint32_t l0 = threadIdx.x; l0 < size; l0 += 4 << B) {
        ulonglong2 v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (l0 + (q << B) < size) v[q] = ab[w.at((l0 >> B) + q)];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            if (l0 + (q << B) < size)
                t[slot<float4>(l0 + (q << B))] = amp_of(split_run(v[q].x, big), split_run(v[q].y, big));
    }
    if (TAGS)
        for (uint32_t l = threadIdx.x; l < size; l += 1 << B) tags[l] = (uint16_t)l;
    uint64_t active = active_ops(ops, nops, w.base, words);
    if (__syncthreads_or(big)) {
        run_fp64_tile(a, reinterpret_cast<double2*>(t), sops, active, tile);
        return;
    }
    for (; active; active &= active - 1) {
        apply_df<TAGS>(t, tags, sops[__ffsll(active) - 1], w.bits);
        __syncthreads();
    }
    ulonglong2* out = reinterpret_cast<ulonglong2*>(a);
    if (TAGS) {
        // every slot's double into the tile, moved amplitudes from memory
        // before any of it is written; then what is not where it was
        ulonglong2* whole = reinterpret_cast<ulonglong2*>(t);
        for (uint32_t l = threadIdx.x; l < size; l += 1 << B) {
            const uint16_t tag = tags[l];
            if (tag == l) continue;
            const uint32_t s = slot<float4>(l);
            if (tag & kTouched) {
                const float4 v = t[s];
                whole[s] = make_ulonglong2(join_f64(re_of(v)), join_f64(im_of(v)));
            } else {
                uint64_t from = w.base;
                for (int b = 0; b < w.bits; ++b)
                    if ((tag >> b) & 1) from |= tile.off[b];
                const double2 x = unit_times((tag >> kRunMaxTileBits) & 3, a[from]);
                whole[s] = make_ulonglong2(__double_as_longlong(x.x), __double_as_longlong(x.y));
            }
        }
        __syncthreads();
        for (uint32_t l = threadIdx.x; l < size; l += 1 << B)
            if (tags[l] != l) out[w.at(l >> B)] = whole[slot<float4>(l)];
        return;
    }
    for (uint32_t l = threadIdx.x; l < size; l += 1 << B) {
        const float4 v = t[slot<float4>(l)];
        out[w.at(l >> B)] = make_ulonglong2(join_f64(re_of(v)), join_f64(im_of(v)));
    }
}

// Opts a kernel in to `bytes` of dynamic shared memory, once per kernel and
// device.
template <typename K>
cudaError_t run_opt_in(K kernel, int bytes)
{
    static std::mutex mu;
    static std::set<std::pair<const void*, int>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), dev);
    if (done.count(key)) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) done.insert(key);
    return e;
}

}  // namespace

cudaError_t launch_gate_run(void* amps, int prec, uint64_t total, const RunTile& tile, const RunOp* d_ops, int nops,
                            RunArith arith, cudaStream_t st)
{
    if (nops < 1 || nops > kRunMaxOps || tile.bits < 0 || tile.bits > kRunMaxTileBits) return cudaErrorInvalidValue;
    const uint64_t tiles = total >> tile.bits;
    if (tiles == 0 || tiles > 0x7fffffffull) return cudaErrorInvalidValue;
    const bool tags = prec != kC64 && arith == RunArith::kPairsPartly;
    const size_t smem = nops * sizeof(RunOp) + ((amp_bytes(prec) + (tags ? sizeof(uint16_t) : 0)) << tile.bits);
    constexpr int most = kRunMaxOps * (int)sizeof(RunOp) + ((16 + (int)sizeof(uint16_t)) << kRunMaxTileBits);
    cudaError_t e;
    if (prec == kC64) {
        if ((e = run_opt_in(k_gate_run<float2>, most)) != cudaSuccess) return e;
        k_gate_run<float2><<<(unsigned)tiles, 1 << kRunBitsPlain, smem, st>>>((float2*)amps, tile, d_ops, nops);
    } else if (arith == RunArith::kPlain) {
        if ((e = run_opt_in(k_gate_run<double2>, most)) != cudaSuccess) return e;
        k_gate_run<double2><<<(unsigned)tiles, 1 << kRunBitsPlain, smem, st>>>((double2*)amps, tile, d_ops, nops);
    } else {
        const auto kernel = tags ? k_gate_run_c128x<true> : k_gate_run_c128x<false>;
        if ((e = run_opt_in(kernel, most)) != cudaSuccess) return e;
        kernel<<<(unsigned)tiles, 1 << kRunBitsDf, smem, st>>>((double2*)amps, tile, d_ops, nops);
    }
    return cudaGetLastError();
}

}  // namespace q1g
