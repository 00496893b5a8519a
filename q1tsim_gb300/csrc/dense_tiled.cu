// Dense blocks (t <= 4 targets, no controls) on one state vector in warp
// tiles (warp_tile.h): each warp of a persistent grid (one 16-warp CTA per
// SM) copies a tile asynchronously into its 8 KB stage with every copy
// instruction moving whole runs of 32 contiguous amplitudes, applies the
// block to the tile's units from the stage, and stores the tile back.
//   complex64:  1024-amplitude tiles, packed FP32x2 complex products
//               (tiled_dense_c64, shared with the batch executor).
//   complex128: 512-amplitude tiles of 16-byte amplitudes, double-float
//               products as in the complex128 pair kernel (df64.cuh); a unit
//               with an amplitude outside the split's range is done in FP64.
// The matrix is a kernel parameter (3 KB at most): nothing is uploaded and the
// host waits for nothing.  A small state's few tiles go one warp to a block,
// over the SMs: a 3-qubit complex128 block at 13 qubits (16 tiles) took 27.9 us
// between events with 16 warps in one CTA, 18.5 us so.
#include <algorithm>
#include <mutex>
#include <set>
#include <utility>

#include "df64.cuh"
#include "kernels.h"
#include "warp_tile.cuh"

namespace q1g {

namespace {

constexpr int kTiledThreads = 512;
constexpr int kTiledWarps = kTiledThreads / 32;
constexpr size_t kTiledWarpBytes = 8192;                 // a warp's stage
constexpr size_t kTiledStageBytes = kTiledWarps * kTiledWarpBytes;

template <int TB>
struct TiledMatC64 {
    float2 m[1 << (2 * TB)];
};
template <int TB>
struct TiledMatC128 {
    float4 terms[2 << (2 * TB)];
    double2 m[1 << (2 * TB)];
};

__device__ __forceinline__ void copy_tile_words(WarpTile& dst, const WarpTile& src)
{
    static_assert(sizeof(WarpTile) % 4 == 0, "WarpTile copies as 32-bit words");
    const uint32_t* s = reinterpret_cast<const uint32_t*>(&src);
    uint32_t* d = reinterpret_cast<uint32_t*>(&dst);
    for (int i = threadIdx.x; i < (int)(sizeof(WarpTile) / 4); i += blockDim.x) d[i] = s[i];
}

template <int TB>
__global__ void __launch_bounds__(kTiledThreads, 1)
k_dense_tiled_c64(float2* a, uint64_t total, const __grid_constant__ WarpTile tile,
                  const __grid_constant__ TiledMatC64<TB> gmat)
{
    constexpr int D = 1 << TB;
    __shared__ WarpTile w;
    __shared__ float2 mat[D * D];
    extern __shared__ float2 stage_c64[];
    copy_tile_words(w, tile);
    for (int e = threadIdx.x; e < D * D; e += blockDim.x) mat[e] = gmat.m[e];
    __syncthreads();
    const int warp = threadIdx.x >> 5;
    tiled_dense_c64<TB, false>(a, total, w, mat, stage_c64 + warp * 1024,
                               (blockIdx.x * blockDim.x >> 5) + warp, [] { return gridDim.x * blockDim.x >> 5; });
}

// Shared-memory load of one 16-byte term, kept at its use.
__device__ __forceinline__ float4 lds_f4(const float4* p)
{
    float4 v;
    const uint32_t sa = (uint32_t)__cvta_generic_to_shared(p);
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(sa));
    return v;
}

// dot_x2 over N terms whose matrix halves come from shared memory, one term
// at a time: t[k] = (ah.x, ah.y, al.x, al.y).  Lane 0 of the result is the
// real part, lane 1 the imaginary part.
template <int N>
__device__ __forceinline__ void dot_terms(const float4* t, const float2* bh, const float2* bl, float2& h, float2& l)
{
    float2 p[N], lo = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < N; ++k) {
        const float4 q = lds_f4(t + k);
        const float2 ah = make_float2(q.x, q.y), al = make_float2(q.z, q.w);
        p[k] = __fmul2_rn(ah, bh[k]);
        const float2 e = __ffma2_rn(ah, bh[k], neg2(p[k]));
        lo = __fadd2_rn(lo, __ffma2_rn(al, bh[k], __ffma2_rn(ah, bl[k], e)));
    }
    float2 s = p[0];
#pragma unroll
    for (int k = 1; k < N; ++k) {
        const float2 tt = __fadd2_rn(s, p[k]);
        const float2 bv = __fadd2_rn(tt, neg2(s));
        const float2 av = __fadd2_rn(tt, neg2(bv));
        lo = __fadd2_rn(lo, __fadd2_rn(__fadd2_rn(s, neg2(av)), __fadd2_rn(p[k], neg2(bv))));
        s = tt;
    }
    h = __fadd2_rn(s, lo);
    const float2 bv = __fadd2_rn(h, neg2(s));
    const float2 av = __fadd2_rn(h, neg2(bv));
    l = __fadd2_rn(__fadd2_rn(s, neg2(av)), __fadd2_rn(lo, neg2(bv)));
}

// Complex128 tiles: terms[r * 2D + 2s] = (m.re, m.re) and
// terms[r * 2D + 2s + 1] = (-m.im, m.im) as (hi, lo) float pairs against the
// inputs (x.re, x.im) and (x.im, x.re); mat is the FP64 matrix for units the
// split cannot take.
template <int TB>
__global__ void __launch_bounds__(kTiledThreads, 1)
k_dense_tiled_c128(double2* a, uint64_t total, const __grid_constant__ WarpTile tile,
                   const __grid_constant__ TiledMatC128<TB> gmat)
{
    constexpr int D = 1 << TB;
    constexpr int U = 16 >> TB;   // units per lane in a 512-amplitude tile
    __shared__ WarpTile w;
    __shared__ float4 terms[2 * D * D];
    __shared__ double2 mat[D * D];
    extern __shared__ ulonglong2 stage_c128[];
    copy_tile_words(w, tile);
    for (int e = threadIdx.x; e < 2 * D * D; e += blockDim.x) terms[e] = gmat.terms[e];
    for (int e = threadIdx.x; e < D * D; e += blockDim.x) mat[e] = gmat.m[e];
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ulonglong2* stage = stage_c128 + warp * 512;
    ulonglong2* ab = reinterpret_cast<ulonglong2*>(a);
    const uint64_t tiles = total >> 9;
    const uint32_t plane = lane_phys(w, lane);
    uint32_t pl = 0;
#pragma unroll
    for (int b = 0; b < 5; ++b)
        if ((lane >> b) & 1) pl ^= w.wbit[b];
    const uint64_t warps = (uint64_t)gridDim.x * blockDim.x >> 5;
    for (uint64_t t = ((uint64_t)blockIdx.x * blockDim.x >> 5) + warp; t < tiles; t += warps) {
        uint32_t gb[4], sb[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            gb[b] = lds_u32(&w.gbit[b]);
            sb[b] = lds_u32(&w.sbit[b]);
        }
        ulonglong2* amps = ab + expand_index(t, w.tile_map) + lane;
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            uint32_t g = 0, so = plane;
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if ((m >> b) & 1) {
                    g |= gb[b];
                    so ^= sb[b];
                }
            cp_async16(stage + so, amps + g);
        }
        cp_async_commit();
        cp_async_wait_group<0>();
        __syncwarp();
#pragma unroll 1
        for (int k = 0; k < U; ++k) {
            uint32_t o = pl;
#pragma unroll
            for (int b = 0; b < 4 - TB; ++b)
                if ((k >> b) & 1) o ^= w.wbit[5 + b];
            ulonglong2 x[D];
            bool fast = true;
#pragma unroll
            for (int s = 0; s < D; ++s) {
                x[s] = stage[o ^ w.gsoff[s]];
                fast = fast & split_fast_ok(x[s].x) & split_fast_ok(x[s].y);
            }
            float2 bh[2 * D], bl[2 * D];
            bool ok = true;
#pragma unroll
            for (int s = 0; s < D; ++s) {
                DF re, im;
                if (fast) {
                    re = split_fast(x[s].x);
                    im = split_fast(x[s].y);
                } else {
                    ok = ok & split_f64(x[s].x, re) & split_f64(x[s].y, im);
                }
                bh[2 * s] = make_float2(re.h, im.h);
                bl[2 * s] = make_float2(re.l, im.l);
                bh[2 * s + 1] = make_float2(im.h, re.h);
                bl[2 * s + 1] = make_float2(im.l, re.l);
            }
            if (ok) {
#pragma unroll 1
                for (int r = 0; r < D; ++r) {
                    float2 h, l;
                    dot_terms<2 * D>(terms + r * 2 * D, bh, bl, h, l);
                    stage[o ^ w.gsoff[r]] = make_ulonglong2(join_f64(DF{h.x, l.x}), join_f64(DF{h.y, l.y}));
                }
            } else {
                double2 y[D];
#pragma unroll
                for (int s = 0; s < D; ++s) y[s] = *reinterpret_cast<const double2*>(&x[s]);
#pragma unroll 1
                for (int r = 0; r < D; ++r) {
                    double re = 0.0, im = 0.0;
#pragma unroll
                    for (int s = 0; s < D; ++s) {
                        const double2 m = mat[r * D + s];
                        re = fma(m.x, y[s].x, fma(-m.y, y[s].y, re));
                        im = fma(m.x, y[s].y, fma(m.y, y[s].x, im));
                    }
                    const double2 out = make_double2(re, im);
                    stage[o ^ w.gsoff[r]] = *reinterpret_cast<const ulonglong2*>(&out);
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int m = 0; m < 16; ++m) {
            uint32_t g = 0, so = plane;
#pragma unroll
            for (int b = 0; b < 4; ++b)
                if ((m >> b) & 1) {
                    g |= gb[b];
                    so ^= sb[b];
                }
            amps[g] = stage[so];
        }
        __syncwarp();
    }
}

// Opts a kernel in to the 128 KB stage, once per kernel and device.
template <typename K>
cudaError_t opt_in(K kernel)
{
    static std::mutex mu;
    static std::set<std::pair<const void*, int>> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_pair(reinterpret_cast<const void*>(kernel), dev);
    if (done.count(key)) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTiledStageBytes);
    if (e == cudaSuccess) done.insert(key);
    return e;
}

}  // namespace

bool dense_tiled_applies(int prec, int nbits, int t, const IndexMap& map, bool fp64_exact)
{
    if (map.nz != t || map.setmask != 0) return false;   // controls: the per-unit kernel
    if (prec == kC128) return !fp64_exact && t >= 1 && t <= 3 && nbits >= 9;
    // complex64: the per-unit kernel is coalesced, and faster, for 1- and
    // 2-qubit blocks whose gate positions are all >= 2
    return t >= 1 && t <= 4 && nbits >= 10 && (t >= 3 || map.zpos[0] <= 1);
}

template <int TB>
static cudaError_t launch_tiled_c64(void* amps, uint64_t total, const WarpTile& w, const double* m, unsigned grid,
                                    unsigned warps, cudaStream_t st)
{
    const cudaError_t e = opt_in(k_dense_tiled_c64<TB>);
    if (e != cudaSuccess) return e;
    TiledMatC64<TB> g;
    for (int i = 0; i < 1 << (2 * TB); ++i) g.m[i] = make_float2((float)m[2 * i], (float)m[2 * i + 1]);
    k_dense_tiled_c64<TB><<<grid, 32 * warps, warps * kTiledWarpBytes, st>>>((float2*)amps, total, w, g);
    return cudaGetLastError();
}

template <int TB>
static cudaError_t launch_tiled_c128(void* amps, uint64_t total, const WarpTile& w, const double* m, unsigned grid,
                                     unsigned warps, cudaStream_t st)
{
    const cudaError_t e = opt_in(k_dense_tiled_c128<TB>);
    if (e != cudaSuccess) return e;
    TiledMatC128<TB> g;
    for (int i = 0; i < 1 << (2 * TB); ++i) {
        const double re = m[2 * i], im = m[2 * i + 1];
        const DF hr = host_split(re), hi = host_split(im);
        g.terms[2 * i] = make_float4(hr.h, hr.h, hr.l, hr.l);
        g.terms[2 * i + 1] = make_float4(-hi.h, hi.h, -hi.l, hi.l);
        g.m[i] = make_double2(re, im);
    }
    k_dense_tiled_c128<TB><<<grid, 32 * warps, warps * kTiledWarpBytes, st>>>((double2*)amps, total, w, g);
    return cudaGetLastError();
}

cudaError_t launch_dense_tiled(void* amps, int prec, uint64_t total, int nbits, const IndexMap& map,
                               const DenseOffsets& offs, int t, const double* m, int sm_count, cudaStream_t st)
{
    WarpTile w;
    const bool c128 = prec == kC128;
    warp_tile_layout(w, map.zpos, t, offs.off, nbits, c128 ? 9 : 10, c128 ? 3 : 4);
    if (!w.tiled) return cudaErrorInvalidValue;
    const uint64_t tiles = total >> w.tile_bits;
    if (tiles == 0) return cudaSuccess;
    const unsigned warps = (unsigned)std::min<uint64_t>(kTiledWarps, (tiles + sm_count - 1) / sm_count);
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)sm_count, (tiles + warps - 1) / warps);
    switch (t) {
        case 1:
            return c128 ? launch_tiled_c128<1>(amps, total, w, m, grid, warps, st)
                        : launch_tiled_c64<1>(amps, total, w, m, grid, warps, st);
        case 2:
            return c128 ? launch_tiled_c128<2>(amps, total, w, m, grid, warps, st)
                        : launch_tiled_c64<2>(amps, total, w, m, grid, warps, st);
        case 3:
            return c128 ? launch_tiled_c128<3>(amps, total, w, m, grid, warps, st)
                        : launch_tiled_c64<3>(amps, total, w, m, grid, warps, st);
        case 4:
            return c128 ? cudaErrorInvalidValue : launch_tiled_c64<4>(amps, total, w, m, grid, warps, st);
        default:
            return cudaErrorInvalidValue;
    }
}

}  // namespace q1g
