// State construction, precision conversion and measurement collapse kernels.
#include "common.cuh"
#include "df64.cuh"
#include "kernels.h"
#include "sampling.cuh"

namespace q1g {

namespace {

constexpr int kThreads = 256;

inline unsigned blocks_for(uint64_t n, int per_block)
{
    uint64_t g = (n + per_block - 1) / per_block;
    if (g > 0x7fffffffULL) g = 0x7fffffffULL;
    return (unsigned)(g ? g : 1);
}

template <typename T>
__global__ void k_set_basis(T* a, const uint64_t* col_index, uint64_t ncols, uint64_t col_len)
{
    uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c < ncols) a[c * col_len + col_index[c]] = cmake<T>(1.0, 0.0);
}

// amp(i) = c_0[b_0] * c_1[b_1] * ... multiplied left to right, b_q the bit of
// qubit q (position n-1-q) -- the kron chain of src/vectorstate.rs:68-74.
template <typename T>
__global__ void k_product_state(T* a, int nbits, const __grid_constant__ ProductCoefs coefs)
{
    const uint64_t n = uint64_t(1) << nbits;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        double re = 1.0, im = 0.0;
        for (int q = 0; q < nbits; ++q) {
            const int b = (i >> (nbits - 1 - q)) & 1;
            const double* c = coefs.c + 4 * q;
            const double cr = b ? c[2] : c[0], ci = b ? c[3] : c[1];
            const double nr = cr * re - ci * im;
            const double ni = cr * im + ci * re;
            re = nr;
            im = ni;
        }
        a[i] = cmake<T>(re, im);
    }
}

// Larger product states: amplitude hi * 2^kProductLow + lo is high[hi] *
// low[lo], high the product state of the other qubits (k_product_state) and
// low[] a table that each block builds by doubling.  One complex product per
// amplitude instead of one per qubit: the n FP64 products were 26.5 ms at 27
// qubits (complex128), this is 1.0 ms (FP64 pipe, 4 operations per
// amplitude; the write alone takes 0.32 ms).
constexpr int kProductLow = 10;
constexpr int kProductPerThread = (1 << kProductLow) / kThreads;
// From this size on: below it the two launches cost more than the products.
constexpr int kProductTwoLevelBits = 15;

__device__ __forceinline__ void product_store(double2* a, double2 h, double2 l)
{
    *a = make_double2(h.x * l.x - h.y * l.y, h.x * l.y + h.y * l.x);
}

struct DfAmp {
    DF re, im;
};
__device__ __forceinline__ DF df_of(double v)
{
    const float h = (float)v;
    return DF{h, (float)(v - (double)h)};
}
__device__ __forceinline__ DfAmp df_amp(double2 v) { return DfAmp{df_of(v.x), df_of(v.y)}; }
// complex64: the product in double-float arithmetic (2^-48), rounded once to
// FP32 as the FP64 product was; the FP64 pipe would bound it at 0.9 ms at 27
// qubits, against 0.16 ms for the write
__device__ __forceinline__ void product_store(float2* a, const DfAmp& h, const DfAmp& l)
{
    const DF u[2] = {h.re, DF{-h.im.h, -h.im.l}}, v[2] = {l.re, l.im};
    const DF w[2] = {h.re, h.im}, z[2] = {l.im, l.re};
    const DF re = dot<2>(u, v), im = dot<2>(w, z);
    *a = make_float2(re.h, im.h);
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
k_product_rows(T* __restrict__ a, uint64_t rows, const double2* __restrict__ high, int nbits,
               const __grid_constant__ ProductCoefs coefs)
{
    constexpr int N = 1 << kProductLow;
    __shared__ double2 low[N];
    if (threadIdx.x == 0) low[0] = make_double2(1.0, 0.0);
    __syncthreads();
    // the last qubit is the lowest bit: entries of bits 0..b-1 give those of
    // bit b by its qubit's two coefficients
    for (int b = 0; b < kProductLow; ++b) {
        const double* c = coefs.c + 4 * (nbits - 1 - b);
        const double2 c0 = make_double2(c[0], c[1]), c1 = make_double2(c[2], c[3]);
        for (int j = threadIdx.x; j < (1 << b); j += kThreads) {
            const double2 v = low[j];
            low[j] = cmul(c0, v);
            low[j + (1 << b)] = cmul(c1, v);
        }
        __syncthreads();
    }
    if constexpr (sizeof(T) == sizeof(double2)) {
        double2 l[kProductPerThread];
#pragma unroll
        for (int k = 0; k < kProductPerThread; ++k) l[k] = low[threadIdx.x + k * kThreads];
        for (uint64_t r = blockIdx.x; r < rows; r += gridDim.x) {
            const double2 h = high[r];
#pragma unroll
            for (int k = 0; k < kProductPerThread; ++k)
                product_store(a + r * N + threadIdx.x + k * kThreads, h, l[k]);
        }
    } else {
        DfAmp l[kProductPerThread];
#pragma unroll
        for (int k = 0; k < kProductPerThread; ++k) l[k] = df_amp(low[threadIdx.x + k * kThreads]);
        for (uint64_t r = blockIdx.x; r < rows; r += gridDim.x) {
            const DfAmp h = df_amp(high[r]);
#pragma unroll
            for (int k = 0; k < kProductPerThread; ++k)
                product_store(a + r * N + threadIdx.x + k * kThreads, h, l[k]);
        }
    }
}

// Amplitude i gets re, im i.i.d. N(0,1) by the Box-Muller transform of
// uniforms 2i and 2i+1 of the SplitMix64 stream `seed`:
// r = sqrt(-2 ln(1 - u1)), (re, im) = r (cos 2 pi u2, sin 2 pi u2).
// complex128 in FP64, complex64 in FP32 (1 - u1 formed in FP64 first, so it
// is never 0).
__global__ void k_random_normal_c128(double2* a, uint64_t total, uint64_t seed)
{
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
        const double u1 = stream_uniform(seed, 2 * i), u2 = stream_uniform(seed, 2 * i + 1);
        const double r = sqrt(-2.0 * log1p(-u1));
        double sn, cs;
        sincospi(2.0 * u2, &sn, &cs);
        a[i] = make_double2(r * cs, r * sn);
    }
}

__global__ void k_random_normal_c64(float2* a, uint64_t total, uint64_t seed)
{
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += stride) {
        const double u1 = stream_uniform(seed, 2 * i), u2 = stream_uniform(seed, 2 * i + 1);
        const float r = sqrtf(-2.0f * logf((float)(1.0 - u1)));
        float sn, cs;
        sincospif(2.0f * (float)u2, &sn, &cs);
        a[i] = make_float2(r * cs, r * sn);
    }
}

__global__ void k_c128_to_c64(float2* dst, const double2* src, uint64_t n)
{
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        double2 v = src[i];
        dst[i] = make_float2((float)v.x, (float)v.y);
    }
}

__global__ void k_c64_to_c128(double2* dst, const float2* src, uint64_t n)
{
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
        float2 v = src[i];
        dst[i] = make_double2(v.x, v.y);
    }
}

// 16 bytes of amplitudes: one complex128 or two complex64.
template <typename T> struct Quad;
template <> struct Quad<double2> {
    using V = double2;
    static constexpr int kShift = 0;
    static __device__ V keep(V v, uint64_t i, int pos, int keep, double scale)
    {
        return ((i >> pos) & 1) == (uint64_t)keep ? make_double2(v.x * scale, v.y * scale) : make_double2(0.0, 0.0);
    }
};
template <> struct Quad<float2> {
    using V = float4;
    static constexpr int kShift = 1;
    static __device__ V keep(V v, uint64_t i, int pos, int keep, double scale)
    {
        const float f = (float)scale;
        const bool k0 = ((i >> pos) & 1) == (uint64_t)keep, k1 = (((i + 1) >> pos) & 1) == (uint64_t)keep;
        return make_float4(k0 ? v.x * f : 0.0f, k0 ? v.y * f : 0.0f, k1 ? v.z * f : 0.0f, k1 ? v.w * f : 0.0f);
    }
};

// Columns of a collapse, blockIdx.y-th and every gridDim.y-th: the amplitudes
// that go are not read (half of each column).  dst may be src where every
// column stays in its place.  Four measurements of a 23-qubit complex128 state
// (to up to 16 columns): 1.21 ms with every amplitude read and a division for
// each, 0.92 ms so.
template <typename T>
__global__ void __launch_bounds__(256)
k_collapse_copy(T* dst, const T* src, uint64_t col_len, int pos, const __grid_constant__ CollapseList list,
                const CollapseCol* __restrict__ cols, uint64_t ncols)
{
    using Q = Quad<T>;
    using V = typename Q::V;
    const uint64_t len = col_len >> Q::kShift, stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t j = blockIdx.y; j < ncols; j += gridDim.y) {
        const CollapseCol c = cols ? cols[j] : list.col[j];
        const V* s = reinterpret_cast<const V*>(src + c.src_col * col_len);
        V* d = reinterpret_cast<V*>(dst + j * col_len);
#pragma unroll 4
        for (uint64_t q = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < len; q += stride) {
            const uint64_t i = q << Q::kShift;
            V v{};
            if (c.keep < 0) {
                v = s[q];
            } else if ((pos < Q::kShift) || (int)((i >> pos) & 1) == c.keep) {
                v = Q::keep(s[q], i, pos, c.keep, c.scale);
            }
            d[q] = v;
        }
    }
}

// Basis columns in one pass: zeros, and a one per column.
template <typename T>
__global__ void __launch_bounds__(256)
k_fill_basis(T* a, uint64_t total, int col_shift, const __grid_constant__ BasisList list)
{
    using Q = Quad<T>;
    using V = typename Q::V;
    const uint64_t len = total >> Q::kShift, stride = uint64_t(gridDim.x) * blockDim.x;
    const uint64_t low = (uint64_t(1) << col_shift) - 1;
#pragma unroll 4
    for (uint64_t q = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < len; q += stride) {
        const uint64_t i = q << Q::kShift;
        const uint64_t at = list.index[i >> col_shift] - (i & low);      // 0 (or 1, in complex64): here
        V v{};
        if (at == 0) v.x = 1;
        if constexpr (Q::kShift == 1)
            if (at == 1) v.z = 1;
        reinterpret_cast<V*>(a)[q] = v;
    }
}

// full[deposit(c) | fixed] = compact[c]: bit k of c goes to position pos[k]
template <typename T>
__global__ void k_scatter_subspace(T* full, const T* compact, uint64_t count, SubspacePositions sp, uint64_t fixed)
{
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t c = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; c < count; c += stride) {
        uint64_t idx = fixed;
#pragma unroll 8
        for (int k = 0; k < sp.n; ++k)
            if ((c >> k) & 1) idx |= uint64_t(1) << sp.pos[k];
        full[idx] = compact[c];
    }
}

// Every amplitude of the full state in one coalesced pass: full[i] is
// compact[i with the excluded positions removed] where i's excluded bits
// equal `fixed`, zero elsewhere.  ex holds the excluded positions, highest
// first, so that removing one leaves the lower ones in place.
struct Excluded {
    int n;
    int pos[kFillMaxExcluded];
};

template <typename T>
__device__ __forceinline__ T fill_value(const T* compact, uint64_t i, uint64_t exmask, uint64_t fixed,
                                        const Excluded& ex)
{
    T v{};
    if ((i & exmask) == fixed) {
        uint64_t c = i;
#pragma unroll
        for (int k = 0; k < kFillMaxExcluded; ++k)
            if (k < ex.n) {
                const int p = ex.pos[k];
                c = ((c >> (p + 1)) << p) | (c & ((uint64_t(1) << p) - 1));
            }
        v = compact[c];
    }
    return v;
}

// One 16-byte unit per thread and iteration (two complex64 amplitudes or
// one complex128), so that each store instruction of a warp writes 512
// contiguous bytes (n even).
template <typename T>
__global__ void k_fill_subspace(T* full, const T* compact, uint64_t n, uint64_t exmask, uint64_t fixed, Excluded ex)
{
    constexpr int kPer = 16 / (int)sizeof(T);
    const uint64_t units = n / kPer;
    const uint64_t stride = uint64_t(gridDim.x) * blockDim.x;
    for (uint64_t u = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; u < units; u += stride) {
        const uint64_t i = u * kPer;
        if constexpr (kPer == 2) {
            const T a = fill_value(compact, i, exmask, fixed, ex);
            const T b = fill_value(compact, i + 1, exmask, fixed, ex);
            reinterpret_cast<float4*>(full)[u] = make_float4(a.x, a.y, b.x, b.y);
        } else {
            full[i] = fill_value(compact, i, exmask, fixed, ex);
        }
    }
}

}  // namespace

cudaError_t launch_scatter_subspace(void* full, const void* compact, int prec, int nbits_full, int nbits_compact,
                                   const SubspacePositions& sp, uint64_t fixed, cudaStream_t st)
{
    const uint64_t n = uint64_t(1) << nbits_full;
    const int nex = nbits_full - nbits_compact;
    if (nex >= 0 && nex <= kFillMaxExcluded && nbits_full >= 2) {
        Excluded ex{};
        uint64_t in = 0;
        for (int k = 0; k < sp.n; ++k) in |= uint64_t(1) << sp.pos[k];
        for (int p = nbits_full - 1; p >= 0; --p)
            if (!((in >> p) & 1)) ex.pos[ex.n++] = p;
        const uint64_t exmask = (n - 1) & ~in;
        const uint64_t units = prec == kC128 ? n : n / 2;
        const unsigned grid = blocks_for(units, kThreads) > 152 * 32 ? 152 * 32 : blocks_for(units, kThreads);
        if (prec == kC128)
            k_fill_subspace<double2><<<grid, kThreads, 0, st>>>((double2*)full, (const double2*)compact, n, exmask,
                                                               fixed & exmask, ex);
        else
            k_fill_subspace<float2><<<grid, kThreads, 0, st>>>((float2*)full, (const float2*)compact, n, exmask,
                                                              fixed & exmask, ex);
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(full, 0, n * (prec == kC128 ? 16 : 8), st);
    if (e != cudaSuccess) return e;
    const uint64_t count = uint64_t(1) << nbits_compact;
    const unsigned grid = blocks_for(count, kThreads) > 152 * 32 ? 152 * 32 : blocks_for(count, kThreads);
    if (prec == kC128)
        k_scatter_subspace<double2><<<grid, kThreads, 0, st>>>((double2*)full, (const double2*)compact, count, sp,
                                                               fixed);
    else
        k_scatter_subspace<float2><<<grid, kThreads, 0, st>>>((float2*)full, (const float2*)compact, count, sp, fixed);
    return cudaGetLastError();
}

cudaError_t launch_fill_basis(void* amps, int prec, int nbits, const BasisList* list, const uint64_t* d_col_index,
                              uint64_t ncols, cudaStream_t st)
{
    const uint64_t n_amps = ncols << nbits;
    if (list && n_amps >= 2 && ncols <= kMaxListCols && nbits >= 1) {
        const uint64_t quads = prec == kC128 ? n_amps : n_amps / 2;
        const unsigned grid = blocks_for(quads, kThreads) > 152 * 32 ? 152 * 32 : blocks_for(quads, kThreads);
        if (prec == kC128) k_fill_basis<double2><<<grid, kThreads, 0, st>>>((double2*)amps, n_amps, nbits, *list);
        else k_fill_basis<float2><<<grid, kThreads, 0, st>>>((float2*)amps, n_amps, nbits, *list);
        return cudaGetLastError();
    }
    cudaError_t e = cudaMemsetAsync(amps, 0, n_amps * amp_bytes(prec), st);
    if (e != cudaSuccess) return e;
    if (ncols == 0) return cudaSuccess;
    if (prec == kC128)
        k_set_basis<double2><<<blocks_for(ncols, kThreads), kThreads, 0, st>>>(
            (double2*)amps, d_col_index, ncols, uint64_t(1) << nbits);
    else
        k_set_basis<float2><<<blocks_for(ncols, kThreads), kThreads, 0, st>>>(
            (float2*)amps, d_col_index, ncols, uint64_t(1) << nbits);
    return cudaGetLastError();
}

uint64_t product_state_tmp_bytes(int nbits)
{
    return nbits < kProductTwoLevelBits ? 0 : sizeof(double2) << (nbits - kProductLow);
}

template <typename T>
static void product_direct(T* a, int nbits, const ProductCoefs& coefs, cudaStream_t st)
{
    const uint64_t n = uint64_t(1) << nbits;
    const unsigned grid = blocks_for(n, kThreads) > 152 * 64 ? 152 * 64 : blocks_for(n, kThreads);
    k_product_state<T><<<grid, kThreads, 0, st>>>(a, nbits, coefs);
}

cudaError_t launch_product_state(void* amps, int prec, int nbits, const ProductCoefs& coefs, void* tmp,
                                 cudaStream_t st)
{
    if (nbits > 48) return cudaErrorInvalidValue;
    if (nbits < kProductTwoLevelBits) {
        if (prec == kC128) product_direct((double2*)amps, nbits, coefs, st);
        else product_direct((float2*)amps, nbits, coefs, st);
        return cudaGetLastError();
    }
    // qubits 0 .. n-1-kProductLow are the row's bits, in the same order
    product_direct((double2*)tmp, nbits - kProductLow, coefs, st);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const uint64_t rows = uint64_t(1) << (nbits - kProductLow);
    const unsigned grid = (unsigned)(rows < 152 * 6 ? rows : 152 * 6);
    if (prec == kC128)
        k_product_rows<double2><<<grid, kThreads, 0, st>>>((double2*)amps, rows, (const double2*)tmp, nbits, coefs);
    else
        k_product_rows<float2><<<grid, kThreads, 0, st>>>((float2*)amps, rows, (const double2*)tmp, nbits, coefs);
    return cudaGetLastError();
}

cudaError_t launch_random_normal(void* amps, int prec, uint64_t total, uint64_t seed, cudaStream_t st)
{
    const unsigned grid = blocks_for(total, kThreads) > 152 * 64 ? 152 * 64 : blocks_for(total, kThreads);
    if (prec == kC128)
        k_random_normal_c128<<<grid, kThreads, 0, st>>>((double2*)amps, total, seed);
    else
        k_random_normal_c64<<<grid, kThreads, 0, st>>>((float2*)amps, total, seed);
    return cudaGetLastError();
}

cudaError_t launch_convert_c128_to_c64(float2* dst, const double2* src, uint64_t n, cudaStream_t st)
{
    const unsigned grid = blocks_for(n, kThreads) > 152 * 64 ? 152 * 64 : blocks_for(n, kThreads);
    k_c128_to_c64<<<grid, kThreads, 0, st>>>(dst, src, n);
    return cudaGetLastError();
}

cudaError_t launch_convert_c64_to_c128(double2* dst, const float2* src, uint64_t n, cudaStream_t st)
{
    const unsigned grid = blocks_for(n, kThreads) > 152 * 64 ? 152 * 64 : blocks_for(n, kThreads);
    k_c64_to_c128<<<grid, kThreads, 0, st>>>(dst, src, n);
    return cudaGetLastError();
}

cudaError_t launch_collapse_copy(void* dst, const void* src, int prec, uint64_t col_len, int pos,
                                 const CollapseList& list, const CollapseCol* d_cols, uint64_t ncols, cudaStream_t st)
{
    if (col_len * ncols == 0) return cudaSuccess;
    if (col_len < 2) return cudaErrorInvalidValue;      // no qubit to measure
    const uint64_t quads = prec == kC128 ? col_len : col_len / 2;
    const uint64_t gy = ncols < 4096 ? ncols : 4096, most = (152 * 64 + gy - 1) / gy;
    const dim3 grid((unsigned)(blocks_for(quads, kThreads) > most ? most : blocks_for(quads, kThreads)), (unsigned)gy);
    if (prec == kC128)
        k_collapse_copy<double2><<<grid, kThreads, 0, st>>>((double2*)dst, (const double2*)src, col_len, pos, list, d_cols,
                                                            ncols);
    else
        k_collapse_copy<float2><<<grid, kThreads, 0, st>>>((float2*)dst, (const float2*)src, col_len, pos, list, d_cols,
                                                           ncols);
    return cudaGetLastError();
}

}  // namespace q1g
