// Dense blocks of up to 5 qubits on a complex128 state, on the tensor cores.
//
// As in fused_tc.cu a block padded to five gate positions is a real GEMM per
// tile of 2^12 amplitudes, D[128][64] = A[128][64] R^T, row t holding one
// group's 32 amplitudes.  FP64-like accuracy comes from splitting both
// operands into signed 9-bit digits (the error-free scheme of Ozaki, Ogita,
// Oishi & Rump 2012, with integers):
//     x 2^e = sum_s a_s 2^(8 - 9 s),  y = sum_t b_t 2^(-8 - 9 t),  s, t = 0..5,
// e per row so that its largest amplitude fills a_0.  Digits are f16
// integers of at most 2^8, a product a_s b_t summed over the row's 64
// components stays below 2^22, and the products of equal weight d = s + t
// share an FP32 accumulator D_d: exact for d <= 3 (four products, 2^24) and
// good to a unit of 2^-36 and 2^-45 for d = 4 and 5; d >= 6 (2^-54 of the row's
// maximum each) is dropped.  21 of the 36 digit products remain: with the
// digits of B stacked, A_s times [B_0; ..; B_(5-s)] is one product of
// N = 64 (6 - s) into D_s .. D_5 (two instructions where that is above 256).
// Measured against 64 bits the result of a block is about 1e-15 off (relative
// 2-norm), where the ~15 gates it replaces left 2.4e-15 each.
//
// One 16-warp CTA per SM, persistent over tiles.  Thread (row t, part) holds 8
// of the row's amplitudes, so a warp's 256 amplitudes lie in whole runs of at
// least 8 (its rows' and states' low bits include the tile's three lowest): it
// copies them in (cp.async) and, rearranged through shared memory, out by
// itself.  Where the lowest positions are rows (kDirect) a thread copies its own
// amplitudes in, and writes them straight to memory.  TMEM has room for one tile only: 128 columns of A (digit s < 4 in
// columns 32 s ..: one 32-bit column per amplitude; the other two digits are in
// shared memory), 384 of accumulators.  So the next tile's digits wait in
// registers while the MMAs of a tile run; when these are done every thread
// stores those digits and reads its 16 columns of the accumulators, and under
// the next MMAs the threads carry the accumulators into one double-float value
// per component (rounding each accumulator's upper part into the next; all
// exact), write the tile out, and read and split the one after the next.  One
// thread issues the MMAs, a K step at a time between its own work: the issue
// blocks while the tensor cores' queue is full.
// Shared memory: B_0..B_5 (48 KB, made from the matrix by each CTA), A_4 and A_5
// (32 KB), the tile coming in and the tile going out (64 KB each),
// XOR-swizzled so that lanes hit distinct banks.
//
// 27 qubits: 1.30 ms per pass of up to five qubits, 1.49 where the lowest
// positions are gates (11.8 k and 13.4 k cycles per tile; its bytes take 5.9 k of
// the SM's share of HBM), against 1.75 ms per pass of three in double-float warp
// tiles.  What bounds it is the threads' own work,
// half of it integer arithmetic at half rate: digits 2.6 k cycles, carries and
// joins 5 k, copies 3 k; the MMAs (3 k) run under it.  One tile after another
// without the overlap took 1.61 ms.  Tried and slower: the digits' carries
// before the next MMAs (1.60 ms), a warp of its own for the MMAs (five warps
// on a scheduler leave 96 registers) with three that copy (1.85), bulk copies
// of 2 KB runs (1.48 to 1.80).  At 13 qubits a pass takes 15 us between
// events, a warp-tile pass of three qubits 28 us.
//
// Rows with an infinity or NaN are done in FP64 as they come in.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <type_traits>

#include "common.cuh"
#include "df64.cuh"
#include "f16_host.h"
#include "kernels.h"
#include "tc_ptx.cuh"
#include "warp_tile.cuh"

namespace q1g {

namespace {

constexpr int kZThreads = 512;
constexpr uint32_t kZTile = 4096;                       // amplitudes
constexpr uint32_t kZWarp = 256;                        // a warp's amplitudes
constexpr uint32_t kZSlice = 8192;                      // one digit of R: 64 rows x 64 f16
constexpr uint32_t kZSliceA = 16384;                    // one digit of A: 128 rows x 64 f16
// shared memory: barrier, tile offsets and row maxima; B_0..B_5; A_4 and A_5;
// the tile coming in; the tile going out
constexpr uint32_t kZOffBar = 0, kZOffSlot = 8, kZOffAbort = 12, kZOffBase = 64, kZOffMax = 1024;
constexpr uint32_t kZOffB = 4096;
constexpr uint32_t kZOffA = kZOffB + 6 * kZSlice;
constexpr uint32_t kZOffIn = kZOffA + 2 * kZSliceA;
constexpr uint32_t kZOffOut = kZOffIn + kZTile * 16;
constexpr uint32_t kZSmem = kZOffOut + kZTile * 16;
constexpr uint32_t kZSmemAlloc = kZSmem + 1024;         // alignment slack
constexpr uint32_t kZBases = 8;                         // ring of tile offsets
static_assert(kZOffBase + kZBases * 8 <= kZOffMax && kZOffMax + 4 * 128 * 4 <= kZOffB && kZOffB % 1024 == 0 &&
                  kZOffIn % 1024 == 0,
              "layout");
static_assert(kZSmemAlloc <= 227 * 1024, "fits the SM's shared memory");
constexpr uint32_t kZColD = 128;                        // accumulators' first TMEM column

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(v[0]),
                 "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

__device__ __forceinline__ float2 splat(float v) { return make_float2(v, v); }
// 1.5 * 2^23: adding and subtracting it rounds |v| < 2^22 to an integer
constexpr float kRound = 12582912.0f;

// x scaled by 2^shift (exponent bits added), as h + l.  High words of |x| below
// `floor` count as it: 2^-74 after scaling, where a row's last digit is 2^-45.
// The scaled exponent is 949 to 1030: split_fast (df64.cuh) on the scaled bits.
__device__ __forceinline__ DF scaled_split(uint64_t bits, uint32_t shift20, uint32_t floor)
{
    const uint32_t top = (uint32_t)(bits >> 32), lw = (uint32_t)bits, sign = top & 0x80000000u;
    const uint32_t hw = max(top & 0x7FFFFFFFu, floor) + shift20;
    const uint32_t t = __funnelshift_r(lw + (1u << 28), hw + (lw > 0xEFFFFFFFu ? 1u : 0u), 29);
    const float h = __uint_as_float((t - (896u << 23)) | sign);
    const float r = (float)((int32_t)(lw << 3) >> 3);
    const float l = r * __uint_as_float((((hw << 3) & 0xFF800000u) - (948u << 23)) | sign);
    return DF{h, l};
}

// The six digits of an amplitude's components as f16 pairs.
__device__ __forceinline__ void digits(DF re, DF im, uint32_t (&d)[6])
{
    float2 r = make_float2(re.h, im.h), t, q;
    const float2 l = make_float2(re.l, im.l);
    t = __fadd2_rn(r, splat(kRound));
    q = __fadd2_rn(t, splat(-kRound));
    d[0] = pack_f16x2(q.x, q.y);
    r = __fadd2_rn(r, neg2(q));
    t = __ffma2_rn(r, splat(512.0f), splat(kRound));
    q = __fadd2_rn(t, splat(-kRound));
    d[1] = pack_f16x2(q.x, q.y);
    r = __ffma2_rn(r, splat(512.0f), neg2(q));
    // what is left of h (exact) and l, which join in the third digit
    const float2 l18 = __fmul2_rn(l, splat(262144.0f));
    t = __fadd2_rn(__ffma2_rn(r, splat(512.0f), l18), splat(kRound));
    q = __fadd2_rn(t, splat(-kRound));
    d[2] = pack_f16x2(q.x, q.y);
    r = __fadd2_rn(__ffma2_rn(r, splat(512.0f), neg2(q)), l18);
#pragma unroll
    for (int s = 3; s < 6; ++s) {
        t = __ffma2_rn(r, splat(512.0f), splat(kRound));
        q = __fadd2_rn(t, splat(-kRound));
        d[s] = pack_f16x2(q.x, q.y);
        r = __ffma2_rn(r, splat(512.0f), neg2(q));
    }
}

// The accumulators of one amplitude's components, as h + l in units of D_0.
__device__ __forceinline__ void carry(const float2 (&a)[5], float2& h, float2& l)
{
    const float2 down = splat(1.0f / 512.0f);
    float2 v = a[4], f[4];
#pragma unroll
    for (int d = 3; d >= 0; --d) {
        // round v / 512 into the next accumulator, keep the fraction
        const float2 q = __fadd2_rn(__ffma2_rn(v, down, splat(kRound)), splat(-kRound));
        f[d] = __ffma2_rn(v, down, neg2(q));
        v = __fadd2_rn(a[d], q);
    }
    // v + f0 + 2^-9 (f1 + 2^-9 (f2 + 2^-9 f3))
    const float2 g = __fadd2_rn(v, f[0]);
    const float2 r = __fadd2_rn(f[0], neg2(__fadd2_rn(g, neg2(v))));
    const float2 lo = __ffma2_rn(__ffma2_rn(__ffma2_rn(f[3], down, f[2]), down, f[1]), down, r);
    h = __fadd2_rn(g, lo);
    l = __fadd2_rn(lo, neg2(__fadd2_rn(h, neg2(g))));
}

// h + l times 2^(shift / 2^20) as a double: zero below the normal range,
// infinite above it.
__device__ __noinline__ double scaled_join(float h, float l, int32_t shift20)
{
    const uint64_t b = join_f64(DF{h, l});
    const uint32_t hw = (uint32_t)(b >> 32);
    const int32_t e = (int32_t)(hw & 0x7FF00000u) + shift20;
    uint32_t out = hw + (uint32_t)shift20, low = (uint32_t)b;
    if ((hw & 0x7FFFFFFFu) == 0 || e < (1 << 20)) out = hw & 0x80000000u, low = 0;
    else if (e >= (2047 << 20)) out = (hw & 0x80000000u) | 0x7FF00000u, low = 0;
    return __hiloint2double((int)out, (int)low);
}

// The same where no output can leave the normal range, |h| at least 2^-60 or
// zero: join_f64 (df64.cuh) without its branches.  up20: shift20 plus the
// difference of the exponent biases.
__device__ __forceinline__ double scaled_join_mid(float h, float l, uint32_t up20)
{
    const uint32_t hb = __float_as_uint(h), lb = __float_as_uint(l);
    const uint32_t ab = hb & 0x7FFFFFFFu, sign = hb & 0x80000000u;
    // |l| is counted in the halved ulp below a power of two
    const bool opposite = (int32_t)(lb ^ hb) < 0;
    const uint32_t down = (opposite && (hb & 0x7FFFFFu) == 0) ? (1u << 23) : 0u;
    const float scale = __uint_as_float((306u << 23) - (ab & 0x7F800000u) + down);
    // |l| with l's sign relative to h's
    const int lm = __float2int_rn(__uint_as_float(lb ^ sign) * scale);
    const uint64_t mag = ((uint64_t)ab << 29) + (uint64_t)(int64_t)lm;
    const uint32_t hi = ((uint32_t)(mag >> 32) + up20) | sign;
    return ab == 0 ? 0.0 : __hiloint2double((int)hi, (int)(uint32_t)mag);
}

__device__ __forceinline__ ulonglong2 lds_amp(uint32_t addr)
{
    ulonglong2 v;
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void sts_amp(uint32_t addr, double re, double im)
{
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(re), "d"(im) : "memory");
}

__device__ __forceinline__ void sts_u32x4(uint32_t addr, const uint32_t* v)
{
    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3])
                 : "memory");
}
__device__ __forceinline__ void sts_raw(uint32_t addr, float2 h, float2 l)
{
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "f"(h.x), "f"(h.y), "f"(l.x), "f"(l.y)
                 : "memory");
}

// Eight outputs of a row (rows of the matrix at mat) from its inputs, which the
// four warps of its parts hold at xa + 4 (warps) * 4 KB * part.
__device__ __noinline__ void row_fp64(uint32_t xa, uint32_t rslot, const ZPass& p, const double2* mat, double2* y)
{
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
        double re = 0.0, im = 0.0;
#pragma unroll 1
        for (uint32_t s = 0; s < 32; ++s) {
            uint32_t slot = rslot;
            for (int k = 0; k < 3; ++k)
                if ((s >> k) & 1u) slot ^= p.slot[p.gate_of[k]];
            const ulonglong2 b = lds_amp(xa + ((s >> 3) * 4u * kZWarp + slot) * 16u);
            const double vr = __longlong_as_double((long long)b.x), vi = __longlong_as_double((long long)b.y);
            const double2 c = mat[32 * j + s];
            re = fma(c.x, vr, fma(-c.y, vi, re));
            im = fma(c.x, vi, fma(c.y, vr, im));
        }
        y[j] = make_double2(re, im);
    }
}

// v (|v| < 2) in units of 2^-53, rounded
__device__ __forceinline__ int64_t fixed53(double v)
{
    const uint64_t b = (uint64_t)__double_as_longlong(v);
    const int e = (int)((b >> 52) & 2047u) - 1022;          // shift of the 53-bit mantissa
    const uint64_t m = (b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
    const uint64_t u = e >= 0 ? m << min(e, 1) : e < -53 ? 0ull : (m + (1ull << (-e - 1))) >> -e;
    return (int64_t)b < 0 ? -(int64_t)u : (int64_t)u;
}

// The 64x64 real embedding of the matrix in digits B_0..B_5.  Digits in -256..255 (the top one up to 257) from the
// low end.
__device__ __forceinline__ void build_operands(const double2* __restrict__ mat, uint8_t* smem, int tid)
{
    const __half2 bias = __float2half2_rn(1536.0f);
    for (int e = tid; e < 1024; e += kZThreads) {
        const double2 c = mat[e];
        int64_t re = fixed53(c.x), im = fixed53(c.y);
        const uint32_t row = 2u * (uint32_t)(e >> 5), k = 2u * (uint32_t)(e & 31);
        const uint32_t at0 = tc_sw128_offset(row, k), at1 = tc_sw128_offset(row + 1, k);
#pragma unroll
        for (int t = 5; t >= 0; --t) {
            int r, i;
            if (t > 0) {
                r = (int)((uint32_t)(re + 256) & 511u) - 256;
                i = (int)((uint32_t)(im + 256) & 511u) - 256;
                re = (re - r) >> 9;
                im = (im - i) >> 9;
            } else {
                r = (int)re;
                i = (int)im;
            }
            // 1024 + field as f16 bits, minus the bias: row (re, -im), row (im, re)
            const uint32_t w0 = 0x64006400u + (uint32_t)(512 + r) + ((uint32_t)(512 - i) << 16);
            const uint32_t w1 = 0x64006400u + (uint32_t)(512 + i) + ((uint32_t)(512 + r) << 16);
            const __half2 h0 = __hsub2(*reinterpret_cast<const __half2*>(&w0), bias);
            const __half2 h1 = __hsub2(*reinterpret_cast<const __half2*>(&w1), bias);
            *reinterpret_cast<__half2*>(smem + kZOffB + t * kZSlice + at0) = h0;
            *reinterpret_cast<__half2*>(smem + kZOffB + t * kZSlice + at1) = h1;
        }
    }
}

// K step ks of a tile's products, by one thread.
__device__ __forceinline__ void issue_step(uint32_t ks, uint32_t tmem, uint32_t sbase, uint32_t mbar)
{
    const uint32_t D = tmem + kZColD, A = tmem + ks * 8u;
    const uint32_t B = sbase + kZOffB + ks * 32u, As = sbase + kZOffA + ks * 32u;
    const uint32_t acc = ks > 0 ? 1u : 0u;      // A_0 [B_0 .. B_5]: every accumulator's first product
    mma_f16_ts(D, A, desc_sw128(B), idesc_f16(192), acc);
    mma_f16_ts(D + 192u, A, desc_sw128(B + 3 * kZSlice), idesc_f16(192), acc);
    mma_f16_ts(D + 64u, A + 32u, desc_sw128(B), idesc_f16(160), 1u);
    mma_f16_ts(D + 224u, A + 32u, desc_sw128(B + 160u * 128u), idesc_f16(160), 1u);
    mma_f16_ts(D + 128u, A + 64u, desc_sw128(B), idesc_f16(256), 1u);
    mma_f16_ts(D + 192u, A + 96u, desc_sw128(B), idesc_f16(192), 1u);
    mma_f16_ss(D + 256u, desc_sw128(As), desc_sw128(B), idesc_f16(128), 1u);
    mma_f16_ss(D + 320u, desc_sw128(As + kZSliceA), desc_sw128(B), idesc_f16(64), 1u);
    if (ks == 3) mma_commit(mbar);
}

template <bool kDirect>
__global__ void __launch_bounds__(kZThreads, 1)
k_fused_tc_c128(double2* __restrict__ a, uint64_t ntiles, const __grid_constant__ ZPass p,
                const double2* __restrict__ mat, int* __restrict__ err, uint64_t wait_ns)
{
    extern __shared__ uint8_t z_raw[];
    uint8_t* smem = z_raw + ((1024u - (smem_addr(z_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_addr(smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t q = (uint32_t)warp & 3u, part = (uint32_t)warp >> 2;
    const uint32_t t = 32u * q + (uint32_t)lane;           // row = TMEM lane
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kZOffAbort);
    uint32_t* rowmax = reinterpret_cast<uint32_t*>(smem + kZOffMax);
    // offsets of this CTA's tiles, the i-th at i % 8: written by the last warp
    // a barrier before their first use
    uint64_t* bases = reinterpret_cast<uint64_t*>(smem + kZOffBase);
    const uint32_t mbar = sbase + kZOffBar;
    const uint64_t count = (ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x;

    build_operands(mat, smem, tid);
    // (every .aligned instruction below follows a __syncwarp, or a vote or block
    // barrier of CUDA's, after the last branch of single lanes; warp 0 has none
    // before it allocates)
    if (tid == 32) {
        *abort_flag = 0;
        mbar_init(mbar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(sbase + kZOffSlot),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    auto put_base = [&](uint64_t i) {
        bases[i % kZBases] = expand_index(blockIdx.x + i * gridDim.x, p.tilemap);
    };
    if (warp == 15 && lane < 2) put_base((uint64_t)lane);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + kZOffSlot);
    bool failed = false;
    uint64_t it = 0;

    const uint32_t tl = tmem + ((32u * q) << 16);          // this warp's lanes
    const uint32_t in = sbase + kZOffIn + (uint32_t)warp * kZWarp * 16u;
    const uint32_t out = sbase + kZOffOut + (uint32_t)warp * kZWarp * 16u;
    // the warp's amplitudes: element lane + 32 k at offset own + (bits of k)
    // and slot cslot ^ (bits of k)
    uint64_t own = 0;
    uint32_t cslot = 0;
#pragma unroll
    for (int b = 0; b < 4; ++b)
        if ((warp >> b) & 1) own |= p.warp[b];
    const uint64_t wown = own;
#pragma unroll
    for (int b = 0; b < 5; ++b)
        if ((lane >> b) & 1) {
            own |= p.off[b];
            cslot ^= p.slot[b];
        }
    auto element = [&](int k, uint64_t& g, uint32_t& s) {
        g = own;
        s = cslot;
#pragma unroll
        for (int b = 0; b < 3; ++b)
            if ((k >> b) & 1) {
                g |= p.off[5 + b];
                s ^= p.slot[5 + b];
            }
    };
    auto load_tile = [&](uint64_t base) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            uint64_t g;
            uint32_t s;
            element(k, g, s);
            cp_async16(smem + (in - sbase) + s * 16u, a + base + g);
        }
        cp_async_commit();
    };
    // the thread's 8 amplitudes: states 8 part + j of row t at byte
    // rbyte ^ (bits of j)
    uint32_t rslot = 0;
#pragma unroll
    for (int b = 0; b < 5; ++b)
        if ((lane >> b) & 1) rslot ^= p.slot[p.row_of[b]];
    const uint32_t g0 = p.slot[p.gate_of[0]] * 16u, g1 = p.slot[p.gate_of[1]] * 16u,
                   g2 = p.slot[p.gate_of[2]] * 16u;
    auto at = [&](uint32_t region, int j) {
        return region + ((rslot * 16u) ^ ((j & 1) ? g0 : 0u) ^ ((j & 2) ? g1 : 0u) ^ ((j & 4) ? g2 : 0u));
    };
    // and their offsets (rows with infinities or NaN only)
    auto offset_of = [&](int j) {
        uint64_t g = wown;
        for (int b = 0; b < 5; ++b)
            if ((lane >> b) & 1) g |= p.off[p.row_of[b]];
        for (int b = 0; b < 3; ++b)
            if ((j >> b) & 1) g |= p.off[p.gate_of[b]];
        return g;
    };

    // its digits of A_4 and A_5 in shared memory: two 16-byte chunks each
    const uint32_t a_own = sbase + kZOffA + tc_sw128_offset(t, 16u * part);

    uint32_t dg[6][8];
    uint32_t m = 0, m_prev = 0;           // the row's largest exponent
    // Reads tile i, which is on its way, asks for the one after it, and splits.
    auto read_split = [&](uint64_t i) {
        cp_async_wait_group<0>();
        __syncwarp();
        ulonglong2 x[8];
        m = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] = lds_amp(at(in, j));
            m = max(m, (uint32_t)(x[j].x >> 32) & 0x7FFFFFFFu);
            m = max(m, (uint32_t)(x[j].y >> 32) & 0x7FFFFFFFu);
        }
        rowmax[part * 128 + t] = m;
        asm volatile("bar.sync %0, 128;" ::"r"(1u + q) : "memory");      // the four parts of these rows
        m = max(max(rowmax[t], rowmax[128 + t]), max(rowmax[256 + t], rowmax[384 + t])) & 0x7FF00000u;
        if (__any_sync(0xFFFFFFFFu, m == 0x7FF00000u)) {
            // (the same lanes in each of the four warps)
            if (m == 0x7FF00000u) {
                double2 y[8];
                row_fp64(sbase + kZOffIn + q * kZWarp * 16u, rslot, p, mat + 256 * part, y);
                for (int j = 0; j < 8; ++j) a[bases[i % kZBases] + offset_of(j)] = y[j];
            }
            __syncwarp();
            asm volatile("bar.sync %0, 128;" ::"r"(1u + q) : "memory");
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = lds_amp(at(in, j));    // (not kept across the call)
            __syncwarp();
        }
        const bool more = i + 1 < count;
        const double2* src = a + bases[(i + 1) % kZBases];
        // the row's largest exponent becomes that of 2^7 .. 2^8; a row
        // below 2^-940 counts as zero
        const bool tiny = m <= (82u << 20);
        const uint32_t shift20 = tiny ? 0u : (1030u << 20) - m;
        const uint32_t floor = tiny ? 949u << 20 : m - (81u << 20);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            uint64_t g;
            uint32_t s;
            element(j, g, s);
            if (more) cp_async16(smem + (in - sbase) + s * 16u, src + g);
            uint32_t d[6];
            digits(scaled_split(x[j].x, shift20, floor), scaled_split(x[j].y, shift20, floor), d);
#pragma unroll
            for (int s = 0; s < 6; ++s) dg[s][j] = d[s];
        }
        cp_async_commit();
    };

    load_tile(bases[0]);
    read_split(0);
    // Step `it`: tile it's digits go to the tensor cores (if any), tile it - 1
    // out (if any).  False: a wait ran out.
    auto step = [&](auto has_tile, auto has_last) {
        constexpr bool kTile = decltype(has_tile)::value, kLast = decltype(has_last)::value;
        bool ok = true;
        float acc[5][16];
        if (warp == 15 && lane == 0) put_base(it + 2);
        __syncwarp();      // (that lane, or lane 0 of warp 0, which issues, may be behind)
        if (kLast) {
            ok = wait_phase(mbar, (uint32_t)(it - 1) & 1u, abort_flag, wait_ns);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        }
        if (kTile) {
#pragma unroll
            for (int s = 0; s < 4; ++s) tmem_st8(tl + 32u * s + 8u * part, dg[s]);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                sts_u32x4(a_own + s * kZSliceA, dg[4 + s]);
                sts_u32x4((a_own ^ 16u) + s * kZSliceA, dg[4 + s] + 4);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        }
        if (kLast) {
#pragma unroll
            for (int d = 4; d >= 0; --d) {
                if (d == 4) {
                    // D_4 + 2^-9 D_5: what this rounds off is far below the result's last digit
                    float low[16];
                    tmem_ld16(tl + kZColD + 64u * 5u + 16u * part, reinterpret_cast<uint32_t*>(low));
                    tmem_ld16(tl + kZColD + 64u * 4u + 16u * part, reinterpret_cast<uint32_t*>(acc[4]));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 0; i < 16; ++i) acc[4][i] = fmaf(low[i], 1.0f / 512.0f, acc[4][i]);
                } else {
                    tmem_ld16(tl + kZColD + 64u * d + 16u * part, reinterpret_cast<uint32_t*>(acc[d]));
                }
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (__syncthreads_or(!ok)) return false;
        const bool issue = kTile && tid == 0;
        if (issue) asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (!kLast && issue)
            for (uint32_t ks = 0; ks < 4; ++ks) issue_step(ks, tmem, sbase, mbar);
        if (kLast) {
            // D_0 is in units of 2^-8 of the scaled row.  Outputs lie within
            // 2^-60 .. 2^3 of the row's maximum (or are zero)
            const int32_t back20 = (int32_t)m_prev - (1038 << 20);
            const bool mid = m_prev > (100u << 20) && m_prev < (1900u << 20);
            double2* dst = a + bases[(it - 1) % kZBases];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (issue && (j & 3) == 0) issue_step((uint32_t)j >> 2, tmem, sbase, mbar);
                float2 c[5], h, l;
#pragma unroll
                for (int d = 0; d < 5; ++d) c[d] = make_float2(acc[d][2 * j], acc[d][2 * j + 1]);
                carry(c, h, l);
                const uint32_t to = at(out, j);
                if (mid) {
                    const uint32_t up20 = (uint32_t)back20 + (896u << 20);
                    const double re = scaled_join_mid(h.x, l.x, up20), im = scaled_join_mid(h.y, l.y, up20);
                    if (kDirect) {
                        uint64_t g;
                        uint32_t s;
                        element(j, g, s);
                        dst[g] = make_double2(re, im);
                    } else {
                        sts_amp(to, re, im);
                    }
                } else {
                    sts_raw(to, h, l);
                }
            }
            if (!mid) {
#pragma unroll 1
                for (int j = 0; j < 8; ++j) {
                    const uint32_t to = at(out, j);
                    const ulonglong2 v = lds_amp(to);
                    if (m_prev == 0x7FF00000u) {
                        const double2 y = dst[offset_of(j)];      // written by read_split
                        sts_amp(to, y.x, y.y);
                    } else {
                        sts_amp(to, scaled_join(__uint_as_float((uint32_t)v.x), __uint_as_float((uint32_t)v.y), back20),
                                scaled_join(__uint_as_float((uint32_t)(v.x >> 32)),
                                            __uint_as_float((uint32_t)(v.y >> 32)), back20));
                    }
                }
            }
            if (issue) issue_step(2u, tmem, sbase, mbar);
            if (!kDirect || !__all_sync(0xFFFFFFFFu, mid)) {
                __syncwarp();
#pragma unroll
                for (int k = 0; k < 8; ++k) {
                    uint64_t g;
                    uint32_t s;
                    element(k, g, s);
                    const ulonglong2 v = lds_amp(out + s * 16u);
                    if (!kDirect || !mid)
                        dst[g] = make_double2(__longlong_as_double((long long)v.x), __longlong_as_double((long long)v.y));
                }
            }
        }
        if (kLast && issue) issue_step(3u, tmem, sbase, mbar);
        m_prev = m;
        if (kTile && it + 1 < count) read_split(it + 1);
        ++it;
        return true;
    };
    using Yes = std::integral_constant<bool, true>;
    using No = std::integral_constant<bool, false>;
    step(Yes(), No());
    while (!failed && it < count) failed = !step(Yes(), Yes());
    if (!failed) failed = !step(No(), Yes());
    if (failed) {
        // what is in flight lands before the CTA's memory is given up
        cp_async_wait_group<0>();
        if (tid == 0) {
            drain_phase(mbar, (uint32_t)(it - 1) & 1u);
            atomicExch(err, 1);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

}  // namespace

void z_pass_layout(ZPass& p, const int* tile_pos, const int* gate_of)
{
    std::memset(&p, 0, sizeof p);
    p.tilemap.nz = 12;
    uint32_t gate_bits = 0;
    for (int j = 0; j < 12; ++j) p.tilemap.zpos[j] = tile_pos[j];
    for (int k = 0; k < 5; ++k) gate_bits |= 1u << gate_of[k];
    // rows: the non-gate tile bits, ascending.  A warp: the five lowest of
    // them and the three lowest gates
    int rows[7], r = 0, wb[8], w = 0;
    for (int j = 0; j < 12; ++j)
        if (!((gate_bits >> j) & 1u)) rows[r++] = j;
    // Straight to memory where that fills whole 32-byte sectors and at least
    // half-lines: tile bit 0 and one of bits 1 and 2 are rows.  26 qubits, us,
    // straight / staged: lowest gate position 3 or higher 660 / 745, 2 670 / 745, 1
    // 708 / 745; 1 and 2 762 / 745.
    p.direct = rows[0] == 0 && rows[1] <= 2;
    if (p.direct) {
        for (int i = 0; i < 5; ++i) wb[w++] = rows[i];
        for (int i = 0; i < 3; ++i) wb[w++] = gate_of[i];
    } else {
        for (int j = 0; j < 12; ++j)
            if (j == gate_of[0] || j == gate_of[1] || j == gate_of[2] || std::find(rows, rows + 5, j) != rows + 5)
                wb[w++] = j;
    }
    for (int i = 0; i < 8; ++i) {
        p.off[i] = uint64_t(1) << tile_pos[wb[i]];
        p.slot[i] = 1u << i;
    }
    for (int i = 0; i < 5; ++i) p.row_of[i] = (uint8_t)(std::find(wb, wb + 8, rows[i]) - wb);
    for (int i = 0; i < 3; ++i) p.gate_of[i] = (uint8_t)(std::find(wb, wb + 8, gate_of[i]) - wb);
    for (int i = 0; i < 2; ++i) {
        p.warp[i] = uint64_t(1) << tile_pos[rows[5 + i]];
        p.warp[2 + i] = uint64_t(1) << tile_pos[gate_of[3 + i]];
    }
    // the three lowest rows vary within a phase of 8 lanes and take the three
    // column bits, their own or those that gate bits leave
    uint32_t used = 0;
    for (int i = 0; i < 3; ++i)
        if (p.row_of[i] < 3) used |= 1u << p.row_of[i];
    for (int i = 0; i < 3; ++i)
        if (p.row_of[i] >= 3) {
            int c = 0;
            while ((used >> c) & 1u) ++c;
            used |= 1u << c;
            p.slot[p.row_of[i]] ^= 1u << c;
        }
}

cudaError_t launch_fused_tc_c128(double2* amps, uint64_t total, const ZPass& p, const void* d_mat, int* d_err,
                                 int sm_count, cudaStream_t st, uint64_t wait_ns)
{
    static std::mutex mu;
    static bool done[64] = {false};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!done[dev]) {
            e = cudaFuncSetAttribute(k_fused_tc_c128<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kZSmemAlloc);
            if (e != cudaSuccess) return e;
            e = cudaFuncSetAttribute(k_fused_tc_c128<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kZSmemAlloc);
            if (e != cudaSuccess) return e;
            done[dev] = true;
        }
    }
    const uint64_t ntiles = total / kZTile;
    if (ntiles == 0) return cudaErrorInvalidValue;
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)sm_count, ntiles);
    const auto kernel = p.direct ? k_fused_tc_c128<true> : k_fused_tc_c128<false>;
    kernel<<<grid, kZThreads, kZSmemAlloc, st>>>(amps, ntiles, p, static_cast<const double2*>(d_mat), d_err,
                                                 wait_ns ? wait_ns : kTcDefaultWaitNs);
    return cudaGetLastError();
}

}  // namespace q1g
