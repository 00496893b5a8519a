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
// good to a unit of 2^-36 for d = 4.  The products of d = 5 (their B digits
// times 2^-9) go to D_4 too, where their fraction is below what matters; d >= 6
// (2^-54 of the row's maximum each) is dropped.  21 of the 36 digit products
// remain: with the digits of B stacked, A_s times [B_0; ..; B_(4-s)] is one
// product of N = 64 (5 - s) into D_s .. D_4, and A_s times B_(5-s) one of N = 64.
// Measured against 64 bits the result of a block is about 1e-15 off (relative
// 2-norm), where the ~15 gates it replaces left 2.4e-15 each.
//
// One 16-warp CTA per SM, persistent over tiles.  Thread (row t, quarter q)
// holds 8 of the row's amplitudes: it reads them from the stage, agrees on
// the row's exponent through shared memory, and stores the digits to TMEM
// (A_s in columns 32 s ..: one 32-bit column per amplitude); one thread issues
// the 48 MMAs; each thread then reads its 16 columns of the five accumulators,
// carries them into one double-float value per component (rounding each
// accumulator's upper part into the next; all exact), and writes the new
// amplitudes over the old ones in the stage.  The next tile's copies
// (cp.async, 16 bytes per amplitude, whole runs per warp) are under way from
// the split on.  TMEM: 192 columns of A, 320 of accumulators.  Shared memory:
// B_0..B_4 (40 KB), the scaled B_0..B_5 (48 KB), two 64 KB stages, whose slots
// are XOR-swizzled so that the lanes of a row read hit distinct banks.
//
// A tile takes 15.5 k cycles where its bytes take 5.9 k of the SM's share of
// HBM: digits 3.6 k, MMAs 4.3 k, carries 3.7 k, store 2.8 k, one after the
// other.  27 qubits: 1.63 ms per pass of up to five qubits, against 1.75 ms per
// pass of three in double-float warp tiles; a 25-qubit brick circuit (10 layers)
// went from 25.8 to 7.8 ms.  At 13 qubits a pass takes 15 us between events, a
// warp-tile pass of three qubits 28 us.
//
// Rows with an infinity or NaN are done in FP64 from the stage.
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>

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
constexpr uint32_t kZStage = kZTile * 16;               // bytes
constexpr uint32_t kZSlice = 8192;                      // one digit of R: 64 rows x 64 f16
// shared memory: barrier and row maxima; B_0..B_4; scaled B_0..B_5; two stages
constexpr uint32_t kZOffBar = 0, kZOffSlot = 8, kZOffAbort = 12, kZOffMax = 1024;
constexpr uint32_t kZOffB = 4096;
constexpr uint32_t kZOffBs = kZOffB + 5 * kZSlice;
constexpr uint32_t kZOffStage = kZOffBs + 6 * kZSlice;
constexpr uint32_t kZSmem = kZOffStage + 2 * kZStage;
constexpr uint32_t kZSmemAlloc = kZSmem + 1024;         // alignment slack
static_assert(kZOffMax + 4 * 128 * 4 <= kZOffB && kZOffB % 1024 == 0 && kZOffStage % 1024 == 0, "layout");
static_assert(kZSmemAlloc <= 227 * 1024, "fits the SM's shared memory");
constexpr uint32_t kZColD = 192;                        // accumulators' first TMEM column

__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint32_t* v)
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(v[0]), "r"(v[1]),
                 "r"(v[2]), "r"(v[3])
                 : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float* v)
{
    uint32_t r[8];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
        : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ float2 splat(float v) { return make_float2(v, v); }
// 1.5 * 2^23: adding and subtracting it rounds |v| < 2^22 to an integer
constexpr float kRound = 12582912.0f;

// x scaled by 2^shift (exponent bits added), as h + l; zero where the high
// word of |x| is below `least`: 2^-47 after scaling (a row's last digit is
// 2^-45).  The scaled exponent is at most 1030: split_fast (df64.cuh) on the
// scaled bits.
__device__ __forceinline__ DF scaled_split(uint64_t bits, uint32_t shift20, uint32_t least)
{
    const uint32_t hw = (uint32_t)(bits >> 32) + shift20, lw = (uint32_t)bits;
    const uint32_t sign = hw & 0x80000000u;
    const uint32_t t = __funnelshift_r(lw + (1u << 28), hw + (lw > 0xEFFFFFFFu ? 1u : 0u), 29);
    const float h = __uint_as_float((t - (896u << 23)) | sign);
    const float r = (float)((int32_t)(lw << 3) >> 3);
    const float l = r * __uint_as_float((((hw << 3) & 0xFF800000u) - (948u << 23)) | sign);
    const bool zero = ((uint32_t)(bits >> 32) & 0x7FFFFFFFu) < least;
    return zero ? DF{0.0f, 0.0f} : DF{h, l};
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

// Eight outputs of a row (rows of the matrix at mat) from its inputs at xa.
__device__ __noinline__ void row_fp64(uint32_t xa, uint32_t rslot, const ZPass& p, const double2* mat, double2* y)
{
#pragma unroll 1
    for (int j = 0; j < 8; ++j) {
        double re = 0.0, im = 0.0;
#pragma unroll 1
        for (int s = 0; s < 32; ++s) {
            const ulonglong2 b = lds_amp(xa + (rslot ^ p.gate[s]) * 16u);
            const double vr = __longlong_as_double((long long)b.x), vi = __longlong_as_double((long long)b.y);
            const double2 c = mat[32 * j + s];
            re = fma(c.x, vr, fma(-c.y, vi, re));
            im = fma(c.x, vi, fma(c.y, vr, im));
        }
        y[j] = make_double2(re, im);
    }
}

__global__ void __launch_bounds__(kZThreads, 1)
k_fused_tc_c128(double2* __restrict__ a, uint64_t ntiles, const __grid_constant__ ZPass p,
                const uint4* __restrict__ image, const double2* __restrict__ mat, int* __restrict__ err,
                uint64_t wait_ns)
{
    extern __shared__ uint8_t z_raw[];
    uint8_t* smem = z_raw + ((1024u - (smem_addr(z_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_addr(smem);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t q = (uint32_t)warp & 3u, part = (uint32_t)warp >> 2;
    const uint32_t t = 32u * q + (uint32_t)lane;           // row = TMEM lane
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kZOffAbort);
    uint32_t* rowmax = reinterpret_cast<uint32_t*>(smem + kZOffMax);
    const uint32_t mbar = sbase + kZOffBar;

    // B_0..B_4, and B_0..B_5 times 2^-9 (exact)
    {
        uint4* B = reinterpret_cast<uint4*>(smem + kZOffB);
        uint4* Bs = reinterpret_cast<uint4*>(smem + kZOffBs);
        const __half2 down = __float2half2_rn(1.0f / 512.0f);
        for (int e = tid; e < (int)(6 * kZSlice / 16); e += kZThreads) {
            uint4 v = image[e];
            if (e < (int)(5 * kZSlice / 16)) B[e] = v;
            __half2* h = reinterpret_cast<__half2*>(&v);
#pragma unroll
            for (int k = 0; k < 4; ++k) h[k] = __hmul2(h[k], down);
            Bs[e] = v;
        }
    }
    if (tid == 0) {
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
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(smem + kZOffSlot);
    const uint32_t tl = tmem + ((32u * q) << 16);          // this warp's lanes

    // copies: thread's amplitude x = tid + 512 k at slot cslot ^ cstep[k]
    uint64_t cown = 0;
    uint32_t cslot = 0;
#pragma unroll
    for (int b = 0; b < 9; ++b)
        if ((tid >> b) & 1) {
            cown |= p.off[b];
            cslot ^= p.slot[b];
        }
    auto copy_at = [&](int k, uint64_t& g, uint32_t& s) {
        g = cown;
        s = cslot;
#pragma unroll
        for (int b = 0; b < 3; ++b)
            if ((k >> b) & 1) {
                g |= p.off[9 + b];
                s ^= p.slot[9 + b];
            }
    };
    auto load_tile = [&](uint64_t tile, uint32_t stage) {
        const double2* src = a + expand_index(tile, p.tilemap);
        double2* dst = reinterpret_cast<double2*>(smem + kZOffStage + stage * kZStage);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            uint64_t g;
            uint32_t s;
            copy_at(k, g, s);
            cp_async16(dst + s, src + g);
        }
        cp_async_commit();
    };
    // the thread's 8 amplitudes: row t, gate states 8 part + j at byte
    // rbyte ^ (gate bits of j)
    uint32_t rslot = 0;
#pragma unroll
    for (int r = 0; r < 7; ++r)
        if ((t >> r) & 1u) rslot ^= p.row[r];
    const uint32_t rbyte = (rslot ^ p.gate[8 * part]) * 16u;
    const uint32_t g0 = p.gate[1] * 16u, g1 = p.gate[2] * 16u, g2 = p.gate[4] * 16u;
    auto at = [&](uint32_t stage_addr, int j) {
        return stage_addr + (rbyte ^ ((j & 1) ? g0 : 0u) ^ ((j & 2) ? g1 : 0u) ^ ((j & 4) ? g2 : 0u));
    };

    if (blockIdx.x < ntiles) load_tile(blockIdx.x, 0);
    uint32_t it = 0;
    bool failed = false;
    for (uint64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
        const uint32_t stage = it & 1u;
        const double2* X = reinterpret_cast<const double2*>(smem + kZOffStage + stage * kZStage);
        const uint32_t xa = sbase + kZOffStage + stage * kZStage;
        cp_async_wait_group<0>();
        __syncthreads();
        ulonglong2 x[8];
        uint32_t m = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            x[j] = lds_amp(at(xa, j));
            m = max(m, (uint32_t)(x[j].x >> 32) & 0x7FFFFFFFu);
            m = max(m, (uint32_t)(x[j].y >> 32) & 0x7FFFFFFFu);
        }
        rowmax[part * 128 + t] = m;
        const bool special = __syncthreads_or(m >= 0x7FF00000u) != 0;    // an infinity or NaN in the tile
        m = max(max(rowmax[t], rowmax[128 + t]), max(rowmax[256 + t], rowmax[384 + t])) & 0x7FF00000u;
        const bool row_special = m == 0x7FF00000u;
        // the row's largest exponent becomes that of 2^7 .. 2^8; a row below
        // 2^-968 counts as zero
        const uint32_t shift20 = (1030u << 20) - m;
        const uint32_t least = m <= (54u << 20) ? 0xFFFFFFFFu : m - (54u << 20);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint32_t v[6][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t d[6];
                digits(scaled_split(x[4 * half + j].x, shift20, least),
                       scaled_split(x[4 * half + j].y, shift20, least), d);
#pragma unroll
                for (int s = 0; s < 6; ++s) v[s][j] = d[s];
            }
#pragma unroll
            for (int s = 0; s < 6; ++s) tmem_st4(tl + 32u * s + 8u * part + 4u * half, v[s]);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t D = tmem + kZColD;
#pragma unroll
            for (uint32_t ks = 0; ks < 4; ++ks) {
                const uint32_t kb = ks * 32u, ka = ks * 8u;
                const uint32_t B = sbase + kZOffB + kb, Bs = sbase + kZOffBs + kb;
                const uint32_t acc = ks > 0 ? 1u : 0u;
                // A_0 [B_0 .. B_4]: every accumulator's first product
                mma_f16_ts(D, tmem + ka, desc_sw128(B), idesc_f16(160), acc);
                mma_f16_ts(D + 160u, tmem + ka, desc_sw128(B + 160u * 128u), idesc_f16(160), acc);
                mma_f16_ts(D + 64u, tmem + 32u + ka, desc_sw128(B), idesc_f16(256), 1u);
                mma_f16_ts(D + 128u, tmem + 64u + ka, desc_sw128(B), idesc_f16(192), 1u);
                mma_f16_ts(D + 192u, tmem + 96u + ka, desc_sw128(B), idesc_f16(128), 1u);
                mma_f16_ts(D + 256u, tmem + 128u + ka, desc_sw128(B), idesc_f16(64), 1u);
#pragma unroll
                for (uint32_t s = 0; s < 6; ++s)
                    mma_f16_ts(D + 256u, tmem + 32u * s + ka, desc_sw128(Bs + (5u - s) * kZSlice), idesc_f16(64), 1u);
            }
            mma_commit(mbar);
        }
        // the other stage's last tile was read out before this tile's first
        // barrier
        if (tile + gridDim.x < ntiles) load_tile(tile + gridDim.x, stage ^ 1u);
        const bool ok = wait_phase(mbar, it & 1u, abort_flag, wait_ns);
        if (__syncthreads_or(!ok)) {
            failed = true;
            break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (special) {
            // rows with infinities or NaN: in FP64 from the stage, every
            // input read before any output is written
            double2 y[8];
            if (row_special) row_fp64(xa, rslot, p, mat + 256 * part, y);
            __syncthreads();
            if (row_special)
#pragma unroll
                for (int j = 0; j < 8; ++j) sts_amp(at(xa, j), y[j].x, y[j].y);
        }
        // D_0 is in units of 2^-8 of the scaled row.  Outputs lie within
        // 2^-60 .. 2^3 of the row's maximum (or are zero)
        const int32_t back20 = (int32_t)m - (1038 << 20);
        const bool mid = m > (100u << 20) && m < (1900u << 20);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float acc[5][8];
#pragma unroll
            for (int d = 0; d < 5; ++d) tmem_ld8(tl + kZColD + 64u * d + 16u * part + 8u * half, acc[d]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float2 c[5], h, l;
#pragma unroll
                for (int d = 0; d < 5; ++d) c[d] = make_float2(acc[d][2 * j], acc[d][2 * j + 1]);
                carry(c, h, l);
                const uint32_t to = at(xa, 4 * half + j);
                if (mid) {
                    const uint32_t up20 = (uint32_t)back20 + (896u << 20);
                    sts_amp(to, scaled_join_mid(h.x, l.x, up20), scaled_join_mid(h.y, l.y, up20));
                } else if (!row_special) {
                    sts_amp(to, scaled_join(h.x, l.x, back20), scaled_join(h.y, l.y, back20));
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        double2* dst = a + expand_index(tile, p.tilemap);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            uint64_t g;
            uint32_t s;
            copy_at(k, g, s);
            dst[g] = X[s];
        }
    }
    if (failed) {
        // what is in flight lands before the CTA's memory is given up
        cp_async_wait_group<0>();
        if (tid == 0) {
            drain_phase(mbar, it & 1u);
            atomicExch(err, 1);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

}  // namespace

void z_pass_layout(ZPass& p, const int* tile_pos, uint32_t gate_bits, const int* gate_of)
{
    std::memset(&p, 0, sizeof p);
    p.tilemap.nz = 12;
    for (int j = 0; j < 12; ++j) {
        p.tilemap.zpos[j] = tile_pos[j];
        p.off[j] = uint64_t(1) << tile_pos[j];
        p.slot[j] = 1u << j;
    }
    // rows: the non-gate tile bits, ascending; the three lowest vary within
    // a phase of 8 lanes and take the three column bits, their own or those
    // that gate bits leave
    int r = 0;
    uint32_t used = 0;
    int rows[7];
    for (int j = 0; j < 12; ++j)
        if (!((gate_bits >> j) & 1u)) rows[r++] = j;
    for (int i = 0; i < 3; ++i)
        if (rows[i] < 3) used |= 1u << rows[i];
    for (int i = 0; i < 3; ++i)
        if (rows[i] >= 3) {
            int c = 0;
            while ((used >> c) & 1u) ++c;
            used |= 1u << c;
            p.slot[rows[i]] ^= 1u << c;
        }
    for (int i = 0; i < 7; ++i) p.row[i] = p.slot[rows[i]];
    for (int g = 0; g < 32; ++g)
        for (int k = 0; k < 5; ++k)
            if ((g >> k) & 1) p.gate[g] ^= (uint16_t)p.slot[gate_of[k]];
}

void z_pass_image(const double* m, unsigned char* out)
{
    uint16_t* img = reinterpret_cast<uint16_t*>(out);
    auto put = [&](int n, int k, const uint16_t (&d)[6], uint16_t flip) {
        for (int t = 0; t < 6; ++t)
            img[(t * kZSlice + tc_sw128_offset((uint32_t)n, (uint32_t)k)) / 2] = d[t] & 0x7FFFu ? d[t] ^ flip : 0;
    };
    for (int gp = 0; gp < 32; ++gp)
        for (int g = 0; g < 32; ++g) {
            uint16_t d[2][6];
            for (int c = 0; c < 2; ++c) {
                double v = m[2 * (gp * 32 + g) + c] * 256.0;
                for (int t = 0; t < 6; ++t) {
                    const double q = std::nearbyint(v);
                    double rounded;
                    d[c][t] = host_f16_bits(q, &rounded);    // an integer of at most 257: exact
                    v = (v - q) * 512.0;
                }
            }
            put(2 * gp, 2 * g, d[0], 0);
            put(2 * gp, 2 * g + 1, d[1], 0x8000u);
            put(2 * gp + 1, 2 * g, d[1], 0);
            put(2 * gp + 1, 2 * g + 1, d[0], 0);
        }
    std::memcpy(out + 6 * kZSlice, m, 2048 * sizeof(double));
}

cudaError_t launch_fused_tc_c128(double2* amps, uint64_t total, const ZPass& p, const void* d_image, int* d_err,
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
            e = cudaFuncSetAttribute(k_fused_tc_c128, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kZSmemAlloc);
            if (e != cudaSuccess) return e;
            done[dev] = true;
        }
    }
    const uint64_t ntiles = total / kZTile;
    if (ntiles == 0) return cudaErrorInvalidValue;
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)sm_count, ntiles);
    const auto* img = static_cast<const unsigned char*>(d_image);
    k_fused_tc_c128<<<grid, kZThreads, kZSmemAlloc, st>>>(amps, ntiles, p, reinterpret_cast<const uint4*>(img),
                                                         reinterpret_cast<const double2*>(img + 6 * kZSlice), d_err,
                                                         wait_ns ? wait_ns : kTcDefaultWaitNs);
    return cudaGetLastError();
}

}  // namespace q1g
