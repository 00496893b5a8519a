// Device-resident VectorState: the host runtime behind the C ABI.
//
// Semantics follow q1tsim's VectorState (src/vectorstate.rs:24-416) column by
// column; only the representation changes: columns are contiguous in HBM,
// collapsed basis columns are kept as indices, and every amplitude pass is
// one of the kernels in gate_kernels.cu / state_kernels.cu / measure_kernels.cu.
#include "engine.h"
#include "gate_run.h"

#include <algorithm>
#include <array>
#include <memory>
#include <mutex>
#include <numeric>
#include <set>
#include <cmath>
#include <cstdlib>
#include <cstring>

namespace q1g {

void check_cuda(cudaError_t e, const char* what)
{
    if (e == cudaSuccess) return;
    const int code = (e == cudaErrorMemoryAllocation) ? Q1G_ERR_OUT_OF_MEMORY : Q1G_ERR_DEVICE;
    throw Error(code, std::string(what) + ": " + cudaGetErrorString(e));
}

// Released device memory, kept per device for the next buffers: cudaMalloc and
// cudaFree of a 27-qubit complex128 state (2 GiB) take 1.7 ms, its product
// state 1.0.  Bounded (kPoolBytes a device, the oldest blocks make room);
// returned when an allocation fails and by q1g_release_cached_memory.  A block
// enters with an event behind its last use and is taken on the stream that used
// it, which then waits for the event on the device, or once the event has
// happened.  Memory that several streams may use waits for all of them with
// finish_device.
namespace {

constexpr size_t kPoolBytes = size_t(4) << 30;
constexpr size_t kPoolBlocks = 256;
constexpr int kPoolDevices = 64;

bool capturing(cudaStream_t st)
{
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &status) == cudaSuccess) return status != cudaStreamCaptureStatusNone;
    (void)cudaGetLastError();
    return true;
}

// Waits for everything on the device: cudaFree does, of a small block in 2 us
// where nothing is under way, and is no invalid call while another thread's
// stream is captured, as cudaDeviceSynchronize is (it ends the capture).
bool finish_device()
{
    void* q = nullptr;
    if (cudaMalloc(&q, 1) == cudaSuccess && cudaFree(q) == cudaSuccess) return true;
    (void)cudaGetLastError();
    return false;
}

struct DevicePool {
    struct Block {
        size_t size;
        void* p;
        cudaStream_t stream;     // of the event
        cudaEvent_t last;        // null: idle
    };
    std::mutex mu;
    std::deque<Block> blocks;      // oldest first
    size_t bytes = 0;

    static void free(const Block& b)
    {
        if (b.last) {
            cudaEventSynchronize(b.last);
            cudaEventDestroy(b.last);
        }
        cudaFree(b.p);
    }
    // The smallest block of at least `size` bytes and not much more that stream
    // `st` (null: any) may use, or null.
    void* take(size_t size, const cudaStream_t* st, size_t* got)
    {
        if (st && capturing(*st)) return nullptr;
        Block b;
        {
            std::lock_guard<std::mutex> lock(mu);
            const size_t most = std::max(size + size / 8, size_t(1) << 16);
            auto best = blocks.end();
            for (auto it = blocks.begin(); it != blocks.end(); ++it) {
                if (it->size < size || it->size > most || (best != blocks.end() && it->size >= best->size)) continue;
                if (it->last && !(st && it->stream == *st)) {
                    if (cudaEventQuery(it->last) != cudaSuccess) {
                        (void)cudaGetLastError();
                        continue;
                    }
                    cudaEventDestroy(it->last);
                    it->last = nullptr;
                }
                best = it;
            }
            if (best == blocks.end()) return nullptr;
            b = *best;
            bytes -= b.size;
            blocks.erase(best);
        }
        if (b.last) {
            // (the handle may be another stream's by now)
            const cudaError_t e = cudaStreamWaitEvent(*st, b.last, 0);
            if (e != cudaSuccess) {
                (void)cudaGetLastError();
                free(b);
                return nullptr;
            }
            cudaEventDestroy(b.last);
        }
        *got = b.size;
        return b.p;
    }
    // Keeps a block; the oldest ones make room.
    void put(const Block& b)
    {
        std::vector<Block> out;
        {
            std::lock_guard<std::mutex> lock(mu);
            while (!blocks.empty() && (bytes + b.size > kPoolBytes || blocks.size() >= kPoolBlocks)) {
                out.push_back(blocks.front());
                bytes -= blocks.front().size;
                blocks.pop_front();
            }
            blocks.push_back(b);
            bytes += b.size;
        }
        for (const Block& o : out) free(o);
    }
    void trim()
    {
        std::deque<Block> all;
        {
            std::lock_guard<std::mutex> lock(mu);
            all.swap(blocks);
            bytes = 0;
        }
        for (const Block& o : all) free(o);
    }
};

// Never destroyed: the driver may be gone by then.
DevicePool* device_pool(int dev)
{
    static DevicePool* const pools = new DevicePool[kPoolDevices];
    return dev >= 0 && dev < kPoolDevices ? &pools[dev] : nullptr;
}

DevicePool* current_pool(int* dev)
{
    if (cudaGetDevice(dev) != cudaSuccess) {
        (void)cudaGetLastError();
        *dev = -1;
    }
    return device_pool(*dev);
}

}  // namespace

size_t cached_device_bytes()
{
    int dev;
    DevicePool* pool = current_pool(&dev);
    if (!pool) return 0;
    std::lock_guard<std::mutex> lock(pool->mu);
    return pool->bytes;
}

void release_cached_memory()
{
    int dev;
    if (DevicePool* pool = current_pool(&dev)) pool->trim();
}

void DevBuf::ensure(size_t b)
{
    if (b <= bytes) return;
    release();
    if (b == 0) return;
    // 512-byte steps, 2 MB ones (the driver's pages) from there on
    const size_t step = b < (size_t(2) << 20) ? 512 : size_t(2) << 20;
    const size_t size = (b + step - 1) / step * step;
    int device;
    DevicePool* pool = current_pool(&device);
    size_t got = size;
    void* q = pool ? pool->take(size, user, &got) : nullptr;
    if (!q) {
        cudaError_t e = cudaMalloc(&q, size);
        if (e == cudaErrorMemoryAllocation && pool) {
            (void)cudaGetLastError();
            pool->trim();
            e = cudaMalloc(&q, b);
            got = b;
        }
        if (e != cudaSuccess) {
            (void)cudaGetLastError();
            throw Error(Q1G_ERR_OUT_OF_MEMORY,
                        "device allocation of " + std::to_string(b) + " bytes failed: " + cudaGetErrorString(e));
        }
    }
    p = q;
    bytes = got;
    dev = device;
}

void DevBuf::release(bool idle)
{
    if (p) {
        int device;
        DevicePool* pool = bytes <= kPoolBytes ? current_pool(&device) : nullptr;
        cudaEvent_t last = nullptr;
        bool keep = pool && device == dev && (idle || !user || !capturing(*user));
        if (keep && !idle) {
            if (user && !lent) {
                keep = cudaEventCreateWithFlags(&last, cudaEventDisableTiming) == cudaSuccess;
                if (keep && cudaEventRecord(last, *user) != cudaSuccess) {
                    cudaEventDestroy(last);
                    keep = false;
                }
                if (!keep) (void)cudaGetLastError();
            } else {
                keep = finish_device();
            }
        }
        if (keep) pool->put({bytes, p, last ? *user : nullptr, last});
        else cudaFree(p);
    }
    p = nullptr;
    bytes = 0;
    lent = false;
    dev = -1;
}

void HostBuf::ensure(size_t b)
{
    if (b <= bytes) return;
    release();
    if (b == 0) return;
    void* q = nullptr;
    cudaError_t e = cudaMallocHost(&q, b);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        throw Error(Q1G_ERR_OUT_OF_MEMORY, "pinned host allocation failed");
    }
    p = q;
    bytes = b;
}

void HostBuf::release()
{
    if (p) cudaFreeHost(p);
    p = nullptr;
    bytes = 0;
}

namespace {

uint64_t splitmix_mix(uint64_t z)
{
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

}  // namespace

double stream_uniform_host(uint64_t seed, uint64_t counter)
{
    const uint64_t z = seed + (counter + 1) * 0x9E3779B97F4A7C15ULL;
    return (double)(splitmix_mix(z) >> 11) * (1.0 / 9007199254740992.0);
}

// Smallest k with CDF(k) > u, pmf in log space from 40 sigma below the mean.
// Stands in for rand_distr::Binomial (src/vectorstate.rs:271, 379).
uint64_t binomial_inv(uint64_t n, double p, double u)
{
    if (n == 0 || p <= 0.0) return 0;
    if (p >= 1.0) return n;
    const double nn = (double)n;
    const double mean = nn * p;
    const double sd = std::sqrt(nn * p * (1.0 - p));
    const double lo_d = std::floor(mean - 40.0 * sd - 40.0);
    const double hi_d = std::ceil(mean + 40.0 * sd + 40.0);
    const uint64_t lo = lo_d < 0.0 ? 0 : (uint64_t)lo_d;
    const uint64_t hi = hi_d > nn ? n : (uint64_t)hi_d;
    const double lp = std::log(p), lq = std::log1p(-p);
    const double lnf = std::lgamma(nn + 1.0);
    double cdf = 0.0;
    for (uint64_t k = lo; k <= hi; ++k) {
        const double kk = (double)k;
        const double lpmf = lnf - std::lgamma(kk + 1.0) - std::lgamma(nn - kk + 1.0) + kk * lp + (nn - kk) * lq;
        cdf += std::exp(lpmf);
        if (u < cdf) return k;
    }
    return hi;
}

}  // namespace q1g

using namespace q1g;

q1g_state::q1g_state(int nbits_, uint64_t nshots_, int prec_)
    : nbits(nbits_), nshots(nshots_), prec(prec_), N(uint64_t(1) << nbits_), ncols(1),
      counts{nshots_}
{
    check_cuda(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
    own_stream = true;
}

q1g_state::q1g_state(int nbits_, uint64_t nshots_, int prec_, cudaStream_t shared)
    : nbits(nbits_), nshots(nshots_), prec(prec_), N(uint64_t(1) << nbits_), ncols(1), counts{nshots_},
      stream(shared), own_stream(false)
{
}

q1g_state::~q1g_state()
{
    compact.reset();   // it runs on this state's stream: free it while the stream exists
    unary_plan.reset();
    const bool idle = stream && cudaStreamSynchronize(stream) == cudaSuccess &&
                      (!copy_stream || cudaStreamSynchronize(copy_stream) == cudaSuccess);
    for (DevBuf* b : {&amps, &spare, &dscratch, &uscratch, &colbuf, &errbuf}) b->release(idle && !b->lent);
    if (copy_stream) {
        cudaEventDestroy(copy_event);
        cudaStreamDestroy(copy_stream);
    }
    for (auto& p : pending) {
        cudaEventDestroy(p.a);
        cudaEventDestroy(p.b);
    }
    if (own_stream && stream) cudaStreamDestroy(stream);
}

void q1g_state::sync()
{
    check_cuda(cudaStreamSynchronize(stream), "cudaStreamSynchronize");
}

void q1g_state::collect_profile()
{
    if (pending.empty()) return;
    sync();
    for (auto& p : pending) {
        float ms = 0.f;
        check_cuda(cudaEventElapsedTime(&ms, p.a, p.b), "cudaEventElapsedTime");
        auto& t = totals[p.name];
        t.launches += 1;
        t.ms += ms;
        t.bytes += p.bytes;
        cudaEventDestroy(p.a);
        cudaEventDestroy(p.b);
    }
    pending.clear();
}

void q1g_state::ensure_dense()
{
    if (!sparse) return;
    amps.ensure(ncols * N * bsz());
    const uint64_t* d_index = nullptr;
    BasisList list;
    if (ncols <= kMaxListCols && nbits >= 1) {
        std::copy_n(basis.data(), ncols, list.index);
    } else {
        uscratch.ensure(ncols * sizeof(uint64_t));
        h2d(uscratch.p, basis.data(), ncols * sizeof(uint64_t), "upload basis");
        d_index = uscratch.as<uint64_t>();
    }
    launch("fill_basis", double(ncols * N * bsz()), [&] {
        return launch_fill_basis(amps.p, prec, nbits, d_index ? nullptr : &list, d_index, ncols, stream);
    });
    // an uploaded list must stay alive until the copy ran: wait here
    if (d_index) sync();
    sparse = false;
    basis.clear();
}

void q1g_state::clear_error_flag()
{
    errbuf.ensure(sizeof(int));
    check_cuda(cudaMemsetAsync(errbuf.p, 0, sizeof(int), stream), "clear error flag");
}

void q1g_state::product_state(const ProductCoefs& c)
{
    amps.ensure(N * bsz());
    dscratch.ensure(std::max<size_t>(product_state_tmp_bytes(nbits), 256));     // the table of the high qubits
    launch("product_state", double(N * bsz()),
           [&] { return launch_product_state(amps.p, prec, nbits, c, dscratch.p, stream); });
    sparse = false;
    basis.clear();
}

void q1g_state::apply_op(const GateOp& op, char* base, uint64_t total_amps)
{
    const double b2 = 2.0 * bsz();
    switch (op.kind) {
        case GateOp::Noop:
            return;
        case GateOp::Pair:
            launch(prec == kC128 ? (fp64_exact ? "pair_c128_fp64" : "pair_c128") : "pair_c64",
                   b2 * op.touched(total_amps), [&] {
                return launch_pair(base, prec, total_amps, op.map, op.o0, op.o1, op.m2, stream, fp64_exact);
            });
            return;
        case GateOp::Phase:
            launch(prec == kC128 ? (fp64_exact ? "phase_c128_fp64" : "phase_c128") : "phase_c64",
                   b2 * op.touched(total_amps), [&] {
                return launch_phase(base, prec, total_amps, op.map, op.ph[0], op.ph[1], stream, fp64_exact);
            });
            return;
        case GateOp::Dense: {
            const double* m = reinterpret_cast<const double*>(op.dense.data());
            if (dense_tiled_applies(prec, nbits, op.t, op.map, fp64_exact)) {
                launch(prec == kC128 ? "dense_tiled_c128" : "dense_tiled_c64", b2 * op.touched(total_amps), [&] {
                    return launch_dense_tiled(base, prec, total_amps, nbits, op.map, op.offs, op.t, m, sm_count(),
                                              stream);
                });
                return;
            }
            launch(prec == kC128 ? "dense_c128" : "dense_c64", b2 * op.touched(total_amps), [&] {
                return launch_dense(base, prec, total_amps, op.map, op.offs, op.t, m, stream);
            });
            return;
        }
    }
}

static void check_gate_bits(int nbits, size_t k, const size_t* bits, size_t nbits_given)
{
    if (nbits_given != k)
        throw Error(Q1G_ERR_INVALID_NR_BITS,
                    "Expected " + std::to_string(k) + " bits for the gate, got " + std::to_string(nbits_given),
                    nbits_given, k);
    for (size_t m = 0; m < nbits_given; ++m)
        if (bits[m] >= (size_t)nbits)
            throw Error(Q1G_ERR_INVALID_QBIT, "Invalid qubit index " + std::to_string(bits[m]), bits[m]);
    for (size_t m = 0; m < nbits_given; ++m)
        for (size_t j = m + 1; j < nbits_given; ++j)
            if (bits[m] == bits[j])
                throw Error(Q1G_ERR_INVALID_ARGUMENT, "qubit " + std::to_string(bits[m]) + " given twice");
}

static GateOp classify_host(const double* mat, size_t k, const size_t* bits, int nbits)
{
    const size_t dim = size_t(1) << k;
    std::vector<cd> m(dim * dim);
    for (size_t e = 0; e < dim * dim; ++e) m[e] = cd(mat[2 * e], mat[2 * e + 1]);
    std::vector<int> b(k);
    for (size_t j = 0; j < k; ++j) b[j] = (int)bits[j];
    return classify(m.data(), (int)k, b.data(), nbits);
}

void q1g_state::apply_gate(const double* mat, size_t k, const size_t* bits, size_t nbits_given)
{
    check_gate_bits(nbits, k, bits, nbits_given);
    const GateOp op = classify_host(mat, k, bits, nbits);
    if (op.kind == GateOp::Noop) return;
    ensure_dense();
    apply_op(op, amps.as<char>(), total());
}

// src/vectorstate.rs:180-189: the same one-qubit gate on every qubit.  The
// reference makes one pass per qubit.  The gates act on different qubits, so
// they commute and fuse into blocks of up to five qubits (one tensor-core pass
// per block, 6 passes at 30 qubits; three in complex128 below 12 qubits:
// double-float warp tiles).  With FP64 arithmetic requested, the gates run
// one by one, as the reference rounds.
void q1g_state::apply_unary_all(const double* mat)
{
    using namespace q1g;
    if (fp64_exact || nbits < 2) {
        for (size_t b = 0; b < (size_t)nbits; ++b) apply_gate(mat, 1, &b, 1);
        return;
    }
    const int width = prec == kC64 || nbits >= 12 ? 5 : 3;
    if (!unary_plan || unary_plan->nbits != nbits || unary_plan->width != width) {
        auto p = std::make_unique<q1g_plan>();
        p->nbits = nbits;
        p->width = width;
        for (int q = 0; q < nbits; ++q) {
            p->mat_off.push_back(p->mat_doubles);
            p->mat_doubles += 8;
            p->gate_bits.push_back({q});
        }
        p->blocks = fuse(p->gate_bits, nbits, width);
        order_blocks_for_tc_pairs(p->blocks, nbits, p->tc_max_high, p->tc_pairs == 5 ? 3 : 2);
        unary_plan = std::move(p);
    }
    std::vector<double> mats(8 * (size_t)nbits);
    for (int q = 0; q < nbits; ++q) std::copy(mat, mat + 8, mats.begin() + 8 * (size_t)q);
    plan_run(unary_plan.get(), this, mats.data(), mats.size());
}

// Every column becomes a random unit vector: re and im of each amplitude
// i.i.d. N(0,1) (column c takes amplitudes c*N .. c*N+N-1 of the stream),
// then normalised -- the column rescale that settles pending norms.
void q1g_state::fill_random_normal(uint64_t seed)
{
    using namespace q1g;
    const uint64_t t = total();
    amps.ensure(t * bsz());
    launch("random_normal", double(t * bsz()),
           [&] { return launch_random_normal(amps.p, prec, t, seed, stream); });
    sparse = false;
    basis.clear();
    norms.assign(ncols, 1.0);
    norm_pending = true;
    settle_norms();
}

// src/qustate.rs:100-127: (column, length, apply) runs of equal control bits.
struct CondRange {
    uint64_t col, len;
    bool apply;
};

static std::vector<CondRange> conditional_ranges(const std::vector<uint64_t>& counts,
                                                 const uint8_t* control)
{
    std::vector<CondRange> r;
    uint64_t off = 0;
    for (uint64_t c = 0; c < counts.size(); ++c) {
        const uint64_t count = counts[c];
        if (count == 0) continue;
        uint64_t begin = off;
        bool prev = control[off] != 0;
        for (uint64_t ib = off + 1; ib < off + count; ++ib) {
            const bool cur = control[ib] != 0;
            if (cur != prev) {
                r.push_back({c, ib - begin, prev});
                begin = ib;
                prev = cur;
            }
        }
        if (begin < off + count) r.push_back({c, off + count - begin, prev});
        off += count;
    }
    return r;
}

void q1g_state::apply_conditional(const uint8_t* control, size_t ncontrol, const double* mat,
                                  size_t k, const size_t* bits, size_t nbits_given)
{
    settle_norms();
    if (ncontrol != nshots)
        throw Error(Q1G_ERR_INVALID_NR_CONTROL_BITS,
                    "Expected " + std::to_string(nshots) + " control bits, got " + std::to_string(ncontrol), ncontrol,
                    nshots);
    check_gate_bits(nbits, k, bits, nbits_given);
    const GateOp op = classify_host(mat, k, bits, nbits);
    const auto ranges = conditional_ranges(counts, control);
    bool same_layout = ranges.size() == ncols;
    for (size_t j = 0; same_layout && j < ranges.size(); ++j) same_layout = ranges[j].col == j;
    if (same_layout && op.kind == GateOp::Noop) return;
    ensure_dense();
    if (!same_layout) {
        const uint64_t nr = ranges.size();
        std::vector<CollapseCol> cols(nr);
        for (uint64_t j = 0; j < nr; ++j) cols[j] = {ranges[j].col, -1, 1.0};
        spare.ensure(nr * N * bsz());
        copy_columns("column_copy", 2.0 * nr, spare.p, 0, cols);
        amps.swap(spare);
        release_spare();
        ncols = nr;
    }
    if (!same_layout) {
        std::vector<double> nn(ranges.size());
        for (size_t j = 0; j < ranges.size(); ++j) nn[j] = norms[ranges[j].col];
        norms.swap(nn);
    }
    counts.resize(ranges.size());
    for (size_t j = 0; j < ranges.size(); ++j) counts[j] = ranges[j].len;
    for (size_t j = 0; j < ranges.size(); ++j)
        if (ranges[j].apply) apply_op(op, col_ptr(j), N);
}

// The columns before a split go to the kept memory, where the next split finds
// them.  A pointer to them that the caller has ended with their shape
// (q1g_state_device_amplitudes), so the state's stream is the last user.
void q1g_state::release_spare()
{
    spare.lent = false;
    spare.release();
}

// New columns `cols` of amps into dst (launch_collapse_copy); moved: columns'
// worth of bytes.
void q1g_state::copy_columns(const char* name, double moved, void* dst, int pos, const std::vector<CollapseCol>& cols)
{
    const CollapseCol* d_cols = nullptr;
    CollapseList list;
    if (cols.size() <= kMaxListCols) {
        std::copy(cols.begin(), cols.end(), list.col);
    } else {
        colbuf.ensure(cols.size() * sizeof(CollapseCol));
        h2d(colbuf.p, cols.data(), cols.size() * sizeof(CollapseCol), "upload columns");
        d_cols = colbuf.as<CollapseCol>();
    }
    launch(name, moved * N * bsz(), [&] {
        return launch_collapse_copy(dst, amps.p, prec, N, pos, list, d_cols, cols.size(), stream);
    });
    if (d_cols) sync();      // the uploaded table must stay alive until the copy ran
}

std::vector<double> q1g_state::zero_weights(size_t qbit)
{
    const int pos = nbits - 1 - (int)qbit;
    std::vector<double> w0(ncols, 0.0);
    if (sparse) {
        for (uint64_t c = 0; c < ncols; ++c) w0[c] = ((basis[c] >> pos) & 1) ? 0.0 : 1.0;
        return w0;
    }
    IndexMap m{};
    m.nz = 1;
    m.zpos[0] = pos;
    m.setmask = 0;
    const uint64_t half = N / 2;
    const uint64_t chunk = std::min<uint64_t>(half, 4096);
    const uint64_t nchunks = ncols * (half / chunk);
    const uint64_t ntmp = segment_sums_tmp_doubles(ncols, half / chunk);
    dscratch.ensure((nchunks + ncols + ntmp) * sizeof(double));
    double* d = dscratch.as<double>();
    launch("qubit_weights", double(ncols * half * bsz()), [&] {
        return launch_chunk_sums(amps.p, prec, ncols * half, chunk, m, d, stream);
    });
    check_cuda(launch_segment_sums(d, ncols, half / chunk, d + nchunks, d + nchunks + ncols, stream),
               "segment_sums");
    hstage.ensure(ncols * sizeof(double));
    d2h(hstage.p, d + nchunks, ncols * sizeof(double), "download weights");
    sync();
    std::memcpy(w0.data(), hstage.p, ncols * sizeof(double));
    return w0;
}

void q1g_state::measure(size_t qbit, size_t cbit, uint64_t* res, size_t res_len,
                        const double* uniforms, size_t nu, q1g_rng* rng, bool collapse)
{
    if (qbit >= (size_t)nbits) throw Error(Q1G_ERR_INVALID_QBIT, "Invalid qubit index " + std::to_string(qbit), qbit);
    settle_norms();     // P(0) is the half's weight against the column's norm
    if (res_len < nshots)
        throw Error(Q1G_ERR_NOT_ENOUGH_SPACE,
                    "Unable to store " + std::to_string(nshots) + " measurements in array of size " +
                        std::to_string(res_len),
                    res_len, nshots);
    if (cbit >= 64) throw Error(Q1G_ERR_INVALID_CBIT, "Invalid classical bit index " + std::to_string(cbit), cbit);
    if (uniforms ? nu < ncols : rng == nullptr)
        throw Error(Q1G_ERR_INVALID_ARGUMENT, "need one uniform per state column or an rng");
    std::vector<double> us(ncols);
    for (uint64_t c = 0; c < ncols; ++c)
        us[c] = uniforms ? uniforms[c] : stream_uniform_host(rng->seed, rng->counter++);
    const std::vector<double> w0 = zero_weights(qbit);
    std::vector<uint64_t> n0(ncols);
    uint64_t new_nr = 0;
    for (uint64_t c = 0; c < ncols; ++c) {
        n0[c] = binomial_inv(counts[c], std::min(w0[c], 1.0), us[c]);
        new_nr += (n0[c] == 0 || n0[c] == counts[c]) ? 1 : 2;
    }
    // results: first n0 runs of a column read 0, the rest 1 (src/vectorstate.rs:290-297)
    const uint64_t one = uint64_t(1) << cbit;
    uint64_t rs = 0;
    for (uint64_t c = 0; c < ncols; ++c) {
        for (uint64_t r = rs; r < rs + n0[c]; ++r) res[r] &= ~one;
        for (uint64_t r = rs + n0[c]; r < rs + counts[c]; ++r) res[r] |= one;
        rs += counts[c];
    }
    if (!collapse) return;
    // collapse (src/vectorstate.rs:299-322, 91-104)
    std::vector<CollapseCol> cols;
    std::vector<uint64_t> nc;
    std::vector<uint64_t> nbasis;
    cols.reserve(new_nr);
    for (uint64_t c = 0; c < ncols; ++c) {
        const double w = w0[c];
        if (n0[c] == counts[c]) {
            cols.push_back({c, 0, 1.0 / std::sqrt(w)});
            nc.push_back(counts[c]);
        } else if (n0[c] == 0) {
            cols.push_back({c, 1, 1.0 / std::sqrt(1.0 - w)});
            nc.push_back(counts[c]);
        } else {
            cols.push_back({c, 0, 1.0 / std::sqrt(w)});
            nc.push_back(n0[c]);
            cols.push_back({c, 1, 1.0 / std::sqrt(1.0 - w)});
            nc.push_back(counts[c] - n0[c]);
        }
    }
    if (sparse) {
        // basis columns are unchanged by their own (certain) outcome
        counts = nc;
        return;
    }
    norms.assign(new_nr, 1.0);
    const int pos = nbits - 1 - (int)qbit;
    const bool split = new_nr != ncols;
    // each column's kept half is read
    if (!split) {
        copy_columns("collapse", 1.5 * ncols, amps.p, pos, cols);
    } else {
        spare.ensure(new_nr * N * bsz());
        copy_columns("collapse", 1.5 * new_nr, spare.p, pos, cols);
        amps.swap(spare);
        release_spare();
    }
    ncols = new_nr;
    counts = nc;
}

void q1g_state::measure_all(const size_t* cbits, size_t ncbits, uint64_t* res, size_t res_len,
                            const double* uniforms, size_t nu, q1g_rng* rng, bool collapse)
{
    if (res_len < nshots)
        throw Error(Q1G_ERR_NOT_ENOUGH_SPACE,
                    "Unable to store " + std::to_string(nshots) + " measurements in array of size " +
                        std::to_string(res_len),
                    res_len, nshots);
    if (ncbits != (size_t)nbits)
        throw Error(Q1G_ERR_INVALID_NR_MEASUREMENT_BITS,
                    "Expected " + std::to_string(nbits) + " measurement bits, got " + std::to_string(ncbits), ncbits,
                    nbits);
    for (size_t q = 0; q < ncbits; ++q)
        if (cbits[q] >= 64)
            throw Error(Q1G_ERR_INVALID_CBIT, "Invalid classical bit index " + std::to_string(cbits[q]), cbits[q]);
    if (uniforms ? nu < nshots : rng == nullptr)
        throw Error(Q1G_ERR_INVALID_ARGUMENT, "need one uniform per run or an rng");
    uint64_t mask = 0;
    std::vector<uint64_t> cbit_of_pos(64, 0);
    for (size_t q = 0; q < ncbits; ++q) {
        mask |= uint64_t(1) << cbits[q];
        cbit_of_pos[nbits - 1 - q] = uint64_t(1) << cbits[q];
    }
    mask = ~mask;
    auto word_of = [&](uint64_t idx) {
        uint64_t w = 0;
        for (int p = 0; p < nbits; ++p)
            if ((idx >> p) & 1) w |= cbit_of_pos[p];
        return w;
    };

    if (sparse) {
        // basis columns stay as they are
        uint64_t off = 0;
        for (uint64_t c = 0; c < ncols; ++c) {
            const uint64_t w = word_of(basis[c]);
            for (uint64_t r = off; r < off + counts[c]; ++r) res[r] = (res[r] & mask) | w;
            if (!uniforms) rng->counter += counts[c] + 1;
            off += counts[c];
        }
        if (!collapse) return;
        // (columns without runs go)
        std::vector<uint64_t> nb, nc;
        for (uint64_t c = 0; c < ncols; ++c) {
            if (counts[c] == 0) continue;
            nb.push_back(basis[c]);
            nc.push_back(counts[c]);
        }
        basis.swap(nb);
        counts.swap(nc);
        norm_pending = false;
        ncols = basis.size();
        norms.assign(ncols, 1.0);
        return;
    }
    // Results of 32 bits where they fit: half the download.  Many words (from
    // 2^17) join the caller's on the device instead: the copies there and back
    // take 80 + 50 us for 10^6, the first one under the chunk sums, the same loop
    // on the host 300 to 400.
    const bool narrow = nbits <= 32;
    const bool join = nshots >= (uint64_t(1) << 17);
    const bool narrow_word = !join && (~mask >> 32) == 0;
    const size_t osz = narrow ? 4 : 8, wsz = narrow_word ? 4 : 8;
    const std::vector<uint64_t> runs(counts.begin(), counts.end());
    const char* h_word = nullptr;
    const char* h_outc = nullptr;
    if (nshots > 0) {
        const uint64_t chunk = std::min<uint64_t>(N, 256);
        const uint64_t ncc = N / chunk;  // chunks per column
        uint64_t mmax = 0;
        for (auto c : counts) mmax = std::max(mmax, c);
        const uint64_t scan_tmp = scan_tmp_doubles(ncc) + scan_tmp_doubles(mmax + 1) + 1;
        const uint64_t nspc = uniforms ? 0 : nshots + ncols;
        // The group sums (1/16 of a complex64 state, 1/16 of a complex128 one)
        // pay where the shots would read more than that from whole chunks:
        // from one shot per 32 chunks on; up to 1 GiB of scratch, and where the
        // device has that.
        const uint64_t group_doubles = prec == kC64 ? ncols * ncc * 16 : ncols * ncc * 32;
        bool groups = chunk == 256 && nshots * 32 >= ncols * ncc && group_doubles <= (uint64_t(1) << 27);
        const uint64_t nd = ncols * ncc + ncols + scan_tmp + nshots + 2 * nspc + 16;
        if (groups) {
            try {
                dscratch.ensure((nd + group_doubles) * sizeof(double));
            } catch (const Error& e) {
                if (e.code != Q1G_ERR_OUT_OF_MEMORY) throw;
                groups = false;
            }
        }
        dscratch.ensure(nd * sizeof(double));
        double* d_sums = dscratch.as<double>();
        double* d_group = d_sums + ((ncols * ncc + 15) & ~uint64_t(15));     // 128-byte lines
        double* d_tot = d_group + (groups ? group_doubles : 0);
        double* d_stmp = d_tot + ncols;
        double* d_u = d_stmp + scan_tmp;
        double* d_e = d_u + nshots;
        double* d_excl = d_e + nspc;
        const size_t out_off = (nshots * wsz + 255) & ~size_t(255);
        const size_t out_bytes = (nshots * osz + 255) & ~size_t(255);
        uscratch.ensure(out_off + out_bytes + 64 * sizeof(uint64_t));
        char* d_word = uscratch.as<char>();
        char* d_out = d_word + out_off;
        uint64_t* d_cpos = reinterpret_cast<uint64_t*>(d_out + out_bytes);
        h2d(d_cpos, cbit_of_pos.data(), 64 * sizeof(uint64_t), "upload cbits");
        Spacings sp{};
        if (!uniforms) {
            sp = {rng->seed, rng->counter, nspc, d_e, d_excl};
            rng->counter += nspc;
        }
        const bool upload = join && mask != 0;
        if (upload) {
            if (!copy_stream) {
                check_cuda(cudaStreamCreateWithFlags(&copy_stream, cudaStreamNonBlocking), "cudaStreamCreate");
                check_cuda(cudaEventCreateWithFlags(&copy_event, cudaEventDisableTiming), "cudaEventCreate");
            }
            // (the buffer is free once what is on the stream now has run)
            check_cuda(cudaEventRecord(copy_event, stream), "copy event");
            check_cuda(cudaStreamWaitEvent(copy_stream, copy_event, 0), "copy wait");
        }
        launch("chunk_sums", double(ncols * N * bsz()), [&] {
            return launch_chunk_sums_dense(amps.p, prec, ncols * N, chunk, d_sums, groups ? d_group : nullptr, sp,
                                           stream);
        });
        std::vector<double> hu;
        if (uniforms) {
            hu.assign(uniforms, uniforms + nshots);
            uint64_t off = 0;
            for (uint64_t c = 0; c < ncols; ++c) {
                std::sort(hu.begin() + off, hu.begin() + off + counts[c]);
                off += counts[c];
            }
            h2d(d_u, hu.data(), nshots * sizeof(double), "upload uniforms");
        }
        if (upload) {
            check_cuda(cudaMemcpyAsync(d_word, res, nshots * wsz, cudaMemcpyHostToDevice, copy_stream), "upload words");
            h2d_bytes += nshots * wsz;
            check_cuda(cudaEventRecord(copy_event, copy_stream), "copy event");
            check_cuda(cudaStreamWaitEvent(stream, copy_event, 0), "copy wait");
        }
        uint64_t off = 0;
        for (uint64_t c = 0; c < ncols; ++c) {
            // column c's spacings: counts + 1 of them, behind the earlier columns'
            launch("scans", 2.0 * ncc * sizeof(double), [&] {
                return launch_scans(d_sums + c * ncc, ncc, d_tot + c, d_excl + off + c, d_e + off + c,
                                    uniforms ? 0 : counts[c], d_u + off, d_stmp, stream);
            });
            SampleArgs a{};
            a.amps = col_ptr(c);
            a.prec = prec;
            a.chunk = chunk;
            a.excl = d_sums + c * ncc;
            a.nchunks = ncc;
            a.groups = groups ? d_group + c * (group_doubles / ncols) : nullptr;
            a.total = d_tot + c;
            a.u = d_u + off;
            a.nruns = counts[c];
            a.narrow = narrow;
            a.narrow_word = narrow_word;
            a.keep = upload ? mask : 0;
            a.outcome = collapse ? d_out + off * osz : nullptr;
            a.word = d_word + off * wsz;
            a.nbits = nbits;
            a.d_cbit_of_pos = d_cpos;
            launch("sample", double(counts[c] * chunk * bsz()), [&] { return launch_sample(a, stream); });
            off += counts[c];
        }
        if (join) {
            if (collapse) {
                hstage.ensure(out_bytes);
                d2h(hstage.p, d_out, nshots * osz, "download outcomes");
            }
            d2h(res, d_word, nshots * wsz, "download words");
        } else {
            hstage.ensure(out_off + out_bytes);
            d2h(hstage.p, d_word, collapse ? out_off + nshots * osz : nshots * wsz, "download outcomes");
        }
        sync();
        h_word = hstage.as<char>();
        h_outc = join ? h_word : h_word + out_off;
    }
    if (!join) {
        if (narrow_word)
            for (uint64_t r = 0; r < nshots; ++r)
                res[r] = (res[r] & mask) | reinterpret_cast<const uint32_t*>(h_word)[r];
        else
            for (uint64_t r = 0; r < nshots; ++r)
                res[r] = (res[r] & mask) | reinterpret_cast<const uint64_t*>(h_word)[r];
    }
    if (!collapse) return;
    // one basis column per distinct (column, outcome), in order: outcomes are
    // sorted within a column, so a column's distinct outcomes are its runs of
    // equal ones (about 10^6 at 30 qubits and 10^6 shots, two for a GHZ
    // state), appended to basis/counts, whose capacity carries over between
    // runs (no zero fill of a resize).  The reservation is capped (2^20
    // entries, 8 MB each): many shots of few outcomes keep no large buffer,
    // and more distinct outcomes grow the vectors as they come.
    auto columns = [&](auto* outc) {
        uint64_t off = 0;
        for (uint64_t c = 0; c < runs.size(); ++c) {
            const uint64_t end = off + runs[c];
            for (uint64_t r = off; r < end; ++r) {
                if (r == off || outc[r] != outc[r - 1]) {
                    basis.push_back(outc[r]);
                    counts.push_back(1);
                } else {
                    ++counts.back();
                }
            }
            off = end;
        }
    };
    basis.clear();
    counts.clear();
    basis.reserve(std::min<uint64_t>(nshots, uint64_t(1) << 20));
    counts.reserve(std::min<uint64_t>(nshots, uint64_t(1) << 20));
    if (narrow) columns(reinterpret_cast<const uint32_t*>(h_outc));
    else columns(reinterpret_cast<const uint64_t*>(h_outc));
    sparse = true;
    norm_pending = false;
    ncols = basis.size();
    norms.assign(ncols, 1.0);
}

void q1g_state::reset_all()
{
    norm_pending = false;
    sparse = true;
    basis.assign(1, 0);
    counts.assign(1, nshots);
    ncols = 1;
    norms.assign(1, 1.0);
}

void q1g_state::download(double* out, size_t len)
{
    if (len < 2 * ncols * N)
        throw Error(Q1G_ERR_NOT_ENOUGH_SPACE, "download buffer too small");
    settle_norms();
    if (sparse) {
        std::memset(out, 0, 2 * ncols * N * sizeof(double));
        for (uint64_t c = 0; c < ncols; ++c) out[2 * (c * N + basis[c])] = 1.0;
        return;
    }
    const uint64_t n = ncols * N;
    if (prec == kC128) {
        d2h(out, amps.p, n * 16, "download");
        sync();
    } else {
        std::vector<float> tmp(2 * n);
        d2h(tmp.data(), amps.p, n * 8, "download");
        sync();
        for (uint64_t e = 0; e < 2 * n; ++e) out[e] = tmp[e];
    }
}

// ---------------------------------------------------------------- plans

void q1g_plan::regrouped()
{
    prefix_known = false;
    prefix_plan.reset();
    for (auto& l : lowered) l.valid = false;
}

q1g_plan::~q1g_plan()
{
    if (staged) {
        cudaEventSynchronize(staged);
        cudaEventDestroy(staged);
    }
}

namespace q1g {


static std::vector<int> positions_of(const std::vector<int>& qubits, int nbits)
{
    std::vector<int> p;
    for (int q : qubits) p.push_back(nbits - 1 - q);
    std::sort(p.begin(), p.end());
    return p;
}

// The tile of a pass: the blocks' positions plus the lowest other positions,
// 12 in all, ascending.
static std::vector<int> tile_positions(const std::vector<const std::vector<int>*>& bits, int nbits)
{
    std::vector<int> T;
    for (auto* b : bits)
        for (int p : positions_of(*b, nbits))
            if (std::find(T.begin(), T.end(), p) == T.end()) T.push_back(p);
    for (int p = 0; (int)T.size() < 12 && p < nbits; ++p)
        if (std::find(T.begin(), T.end(), p) == T.end()) T.push_back(p);
    std::sort(T.begin(), T.end());
    return T;
}

// Tile bits 0..L-1 are positions 0..L-1: the tile is 2^(12-L) contiguous runs.
static int tile_run_bits(const std::vector<int>& T)
{
    int L = 0;
    while (L < (int)T.size() && T[L] == L) ++L;
    return L;
}

// Shortest contiguous run a pass may copy in pieces (2^7 amplitudes = 1 KB):
// at most 32 runs per tile.  Shorter runs need the tile to be one
// tensor-map box, unpadded.
constexpr int kMinTcRunBits = 7;
// Tile positions at or above this one are 2 MB (a large page) or more apart
// in complex64; a pair's tile may have q1g_plan::tc_max_high of them (8 by
// default: at most 256 large pages per tile; a tile over 512 ran 2.4x
// slower, one over 256 as fast as any).
constexpr int kHighPosition = 18;
// Shortest contiguous run (as a power of two of amplitudes) of a three-block
// pass's tile: 8 amplitudes, 64 bytes.
constexpr int kMinTripleRunBits = 3;

static TcPass lower_tc_pass(const std::vector<const std::vector<int>*>& bits, int nbits, uint64_t ncols, int slack,
                            int pair_mode)
{
    const size_t nblk = bits.size();
    const bool shuffle = pair_mode == 2;
    TcPass t;
    const std::vector<int> T = tile_positions(bits, nbits);
    auto tbit = [&](int pos) { return (int)(std::find(T.begin(), T.end(), pos) - T.begin()); };
    t.tilemap.nz = 12;
    for (int j = 0; j < 12; ++j) t.tilemap.zpos[j] = T[j];
    t.tilemap.setmask = 0;
    const int L = tile_run_bits(T);
    t.box = tc_tile_box(T.data(), nbits, ncols);
    if (L < kMinTcRunBits && !t.box.usable)
        throw Error(Q1G_ERR_INVALID_ARGUMENT, "tensor-core tile with runs shorter than 128 amplitudes");
    t.offs.run_bits = (uint32_t)L;
    t.offs.nruns = 1u << (12 - L);
    for (uint32_t r = 0; r < t.offs.nruns && r < 32; ++r) {
        uint64_t o = 0;
        for (int b = L; b < 12; ++b)
            if ((r >> (b - L)) & 1) o |= uint64_t(1) << T[b];
        t.offs.run_off[r] = o;
    }
    t.offs.nblocks = (uint32_t)nblk;
    for (size_t bi = 0; bi < nblk; ++bi) {
        // gate qubits: the block's own, padded from the tile's highest positions
        std::vector<int> gpos = positions_of(*bits[bi], nbits);
        for (int j = 11; (int)gpos.size() < 5; --j)
            if (std::find(gpos.begin(), gpos.end(), T[j]) == gpos.end()) gpos.push_back(T[j]);
        std::vector<int> q;
        for (int p : gpos) q.push_back(nbits - 1 - p);
        std::sort(q.begin(), q.end());   // ascending qubits: q[0] is the matrix MSB
        t.order[bi] = q;
        TcBlockGeom& G = t.offs.blk[bi];
        int r = 0;
        for (int j = 0; j < 12; ++j)
            if (std::find(gpos.begin(), gpos.end(), T[j]) == gpos.end()) G.jrow_bit[r++] = 1u << j;
        for (int g = 0; g < 32; ++g) {
            uint32_t jc = 0;
            for (int j = 0; j < 5; ++j)
                if ((g >> (4 - j)) & 1) jc |= 1u << tbit(nbits - 1 - q[j]);
            G.jgate[g] = jc;
        }
        G.vec2 = G.jgate[1] == 1u ? 1u : 0u;
    }
    t.offs.shuffle = 0;
    int reg1[5];
    if (nblk == 2 && shuffle && tc_shuffle_layout(t.offs.blk[0], t.offs.blk[1], t.offs.swap_lane, reg1)) {
        // the second block takes the first block's results in registers, in
        // their order: matrix index bit k = tile bit reg1[k]
        t.offs.shuffle = 1;
        for (int k = 0; k < 5; ++k) t.order[1][4 - k] = nbits - 1 - T[reg1[k]];
    }
    // pair modes 4 and 5: the four-group kernel, every A operand in shared
    // memory (5: three blocks per pass where they fit)
    const bool quad = pair_mode >= 4;
    // block bi in the gate order a layout chose: matrix index bit k = tile
    // bit gb[k]
    auto reorder = [&](size_t bi, const int* gb) {
        for (int k = 0; k < 5; ++k) t.order[bi][4 - k] = nbits - 1 - T[gb[k]];
    };
    auto finish = [&] {
        if (!quad) return;
        t.offs.groups = 4;
        t.offs.stage_bytes = (t.offs.stage_bytes + 1023u) & ~1023u;
        // the first block's split is dealt to the threads by a map of its
        // own, in a gate order that map chooses
        int gbit0[5];
        tc_split_map(t.offs, gbit0);
        reorder(0, gbit0);
    };
    int gbits[kTcMaxBlocks][5];
    // store boxes for the last block's write-back (an unpadded one-box tile)
    std::vector<TcStoreBox> stores;
    if (quad && nblk >= 2 && t.box.usable)
        stores = tc_store_boxes(T.data(), nbits, ncols, t.offs.blk[nblk - 1].jgate[31]);
    int store = -1;
    if (quad && nblk >= 2 &&
        tc_chain_layout(t.offs, t.box.usable != 0, slack, gbits, &t.cost, &t.ideal, &stores, &store)) {
        if (t.offs.st_box) t.sbox = stores[(size_t)store].box;
        // the later blocks read the operands the previous block's
        // write-back scattered, in the gate orders the layout chose
        for (size_t bi = 1; bi < nblk; ++bi) reorder(bi, gbits[bi]);
        finish();
        return t;
    }
    if (nblk > 2) throw Error(Q1G_ERR_INVALID_ARGUMENT, "a three-block pass needs the four-group kernel");
    int gbit1[5];
    if (nblk == 2 && (pair_mode == 3 || quad) && tc_direct_layout(t.offs, t.box.usable != 0, slack, gbit1)) {
        // the second block reads the operands the first block's write-back
        // scattered, in the gate order that layout chose
        reorder(1, gbit1);
        finish();
        return t;
    }
    tc_choose_padding(t.offs, t.box.usable != 0, slack);
    finish();
    return t;
}

// The f16 images of a pass's blocks, one after the other.
static std::vector<uint16_t> tc_images(const TcPass& t, const std::vector<cd>* const* mats,
                                       const std::vector<int>* const* bits, int nblk)
{
    std::vector<uint16_t> images((size_t)nblk * kTcImageHalves);
    for (int bi = 0; bi < nblk; ++bi) {
        const auto m32 = embed_matrix(*mats[bi], *bits[bi], t.order[bi]);
        build_tc_image(reinterpret_cast<const double*>(m32.data()), images.data() + bi * kTcImageHalves,
                       bi + 1 == nblk ? kTcLastBScaleLog2 : 0);
    }
    return images;
}

// Whether blocks on these qubit sets could share a tensor-core pass: their
// positions fit one 12-position tile, at most max_high of its positions lie
// at 2 MB strides or more, and the tile has runs of >= 128 amplitudes or is
// one tensor-map box (the rule plan_run applies, before any padding choice).
static bool tc_pairable(const std::vector<const std::vector<int>*>& qs, int nbits, int max_high)
{
    std::vector<int> u;
    for (auto* q : qs)
        for (int x : *q)
            if (std::find(u.begin(), u.end(), x) == u.end()) u.push_back(x);
    if (u.size() > 12 || nbits < 12) return false;
    const auto T = tile_positions(qs, nbits);
    int high = 0;
    for (int p : T) high += p >= kHighPosition;
    return high <= max_high && (tile_run_bits(T) >= kMinTcRunBits || tc_tile_box(T.data(), nbits, 1).usable);
}

void order_blocks_for_tc_pairs(std::vector<FusedBlock>& blocks, int nbits, int max_high, int group)
{
    // Blocks on disjoint qubits commute.  Take the earliest block whose
    // predecessors (the last earlier block on each of its qubits) are all
    // taken, then, while the pass has room (group blocks), the earliest
    // ready block that can share its tensor-core pass, so that plan_run
    // finds them next to each other.
    const int m = (int)blocks.size();
    if (m < 3 || nbits < 12) return;
    auto candidate = [&](int i) {
        return !blocks[i].phase_run && !blocks[i].swap_run && blocks[i].qubits.size() >= 3 &&
               blocks[i].qubits.size() <= 5;
    };
    std::vector<std::vector<int>> succ(m);
    std::vector<int> indeg(m, 0), last(nbits, -1);
    for (int j = 0; j < m; ++j) {
        std::vector<int> preds;
        for (int q : blocks[j].qubits) {
            if (last[q] >= 0 && std::find(preds.begin(), preds.end(), last[q]) == preds.end()) preds.push_back(last[q]);
            last[q] = j;
        }
        for (int i : preds) succ[i].push_back(j);
        indeg[j] = (int)preds.size();
    }
    std::set<int> ready;
    for (int j = 0; j < m; ++j)
        if (indeg[j] == 0) ready.insert(j);
    std::vector<int> order;
    auto take = [&](int j) {
        ready.erase(j);
        order.push_back(j);
        for (int k : succ[j])
            if (--indeg[k] == 0) ready.insert(k);
    };
    while (!ready.empty()) {
        const int a = *ready.begin();
        take(a);
        if (!candidate(a)) continue;
        std::vector<const std::vector<int>*> pass = {&blocks[a].qubits};
        while ((int)pass.size() < group) {
            int next = -1;
            for (int b : ready) {
                if (!candidate(b)) continue;
                pass.push_back(&blocks[b].qubits);
                const bool ok = tc_pairable(pass, nbits, max_high);
                pass.pop_back();
                if (ok) {
                    next = b;
                    break;
                }
            }
            if (next < 0) break;
            pass.push_back(&blocks[next].qubits);
            take(next);
        }
    }
    std::vector<FusedBlock> out;
    out.reserve(m);
    for (int j : order) out.push_back(std::move(blocks[j]));
    blocks.swap(out);
}

// A swap-run block (fuse_runs): every gate must be the swap permutation;
// one permutation pass (swap_run.cu), or the swaps one by one when the
// state has fewer than 10 qubits.
template <typename Stage, typename Emit>
static void lower_swap_block(q1g_state* s, const FusedBlock& b, const std::vector<SeqGate>& gates, Stage&& stage,
                             Emit&& emit)
{
    const int n = s->nbits;
    std::vector<int> pa, pb;
    for (int g : b.gates) {
        const SeqGate& q = gates[g];
        if (q.bits.size() != 2) throw Error(Q1G_ERR_INVALID_ARGUMENT, "a gate marked swap acts on two qubits");
        for (int r = 0; r < 4; ++r)
            for (int c = 0; c < 4; ++c) {
                const bool one = (r == c && (r == 0 || r == 3)) || (r == 1 && c == 2) || (r == 2 && c == 1);
                if (q.mat[4 * r + c] != cd(one ? 1.0 : 0.0, 0.0))
                    throw Error(Q1G_ERR_INVALID_ARGUMENT, "a gate marked swap is not the swap");
            }
        pa.push_back(n - 1 - q.bits[0]);
        pb.push_back(n - 1 - q.bits[1]);
    }
    auto t = std::make_unique<SwapTile>();
    if (!swap_run_layout(*t, pa.data(), pb.data(), (int)pa.size(), n, (int)amp_bytes(s->prec))) {
        for (int g : b.gates) {
            const GateOp op = classify(gates[g].mat.data(), 2, gates[g].bits.data(), n);
            if (op.kind != GateOp::Noop) emit([op](q1g_state* x) { x->apply_op(op, x->amps.as<char>(), x->total()); });
        }
        return;
    }
    const void* dt = stage(t.get(), sizeof(SwapTile));
    emit([dt](q1g_state* x) {
        const uint64_t total = x->total();
        x->launch("swap_run", 2.0 * total * x->bsz(), [&] {
            return launch_swap_run(x->amps.p, (int)amp_bytes(x->prec), total, dt, x->sm_count(), x->stream);
        });
    });
}

// Whether phase-run blocks of this state run as one pass of phase kernels
// (otherwise their gates run as plain gates).
static bool phase_kernels_take(const q1g_state* s) { return s->prec == kC64 && s->nbits <= 32; }

// The phase function of a phase-run block: c + L0 + x_pivot L1, coefficients
// per bit position.  Each gate of the run must be diagonal with unit-modulus
// entries: its log-phases theta_s over its (at most two) qubits contribute, by
// the Moebius transform, a constant, one linear term per qubit and, for two
// qubits, the product term, which contains the run's pivot.
struct PhaseFunction {
    int pivot_pos = -1;
    double c = 0.0;
    std::vector<double> lin0, lin1;
};
static PhaseFunction phase_function(const q1g_plan* p, int n, const FusedBlock& b, const std::vector<SeqGate>& gates)
{
    PhaseFunction f;
    const size_t ndiag = b.gates.size() - (b.trailing_pair ? 1 : 0);
    const int pivot_q = phase_run_pivot(b, p->gate_bits);
    f.pivot_pos = pivot_q >= 0 ? n - 1 - pivot_q : -1;
    f.lin0.assign(n, 0.0);
    f.lin1.assign(n, 0.0);
    for (size_t j = 0; j < ndiag; ++j) {
        const SeqGate& g = gates[b.gates[j]];
        const size_t k = g.bits.size(), dim = size_t(1) << k;
        double th[4];
        for (size_t r = 0; r < dim; ++r)
            for (size_t col = 0; col < dim; ++col) {
                const cd v = g.mat[r * dim + col];
                if (r != col && v != cd(0.0, 0.0))
                    throw Error(Q1G_ERR_INVALID_ARGUMENT, "a gate marked diagonal has an off-diagonal entry");
                if (r == col) {
                    if (std::abs(std::abs(v) - 1.0) > 1e-9)
                        throw Error(Q1G_ERR_INVALID_ARGUMENT, "a gate marked diagonal is not a phase");
                    th[r] = std::arg(v);
                }
            }
        if (k == 1) {
            f.c += th[0];
            f.lin0[n - 1 - g.bits[0]] += th[1] - th[0];
        } else {
            // matrix index bit 1 = g.bits[0], bit 0 = g.bits[1]
            f.c += th[0];
            f.lin0[n - 1 - g.bits[0]] += th[2] - th[0];
            f.lin0[n - 1 - g.bits[1]] += th[1] - th[0];
            const double w = th[3] - th[2] - th[1] + th[0];
            if (g.bits[0] == pivot_q) f.lin1[n - 1 - g.bits[1]] += w;
            else if (g.bits[1] == pivot_q) f.lin1[n - 1 - g.bits[0]] += w;
            else throw Error(Q1G_ERR_INVALID_ARGUMENT, "phase run without a common qubit");
        }
    }
    return f;
}

// A phase-run block of a state phase_kernels_take: one pass with the block's
// phase function (and its trailing 1-qubit gate).
template <typename Stage, typename Emit>
static void lower_phase_block(q1g_plan* p, q1g_state* s, const FusedBlock& b, const std::vector<SeqGate>& gates,
                              Stage&& stage, Emit&& emit)
{
    const int n = s->nbits;
    const PhaseFunction f = phase_function(p, n, b, gates);
    const int pivot_pos = f.pivot_pos;
    std::vector<float2> tab(2048);
    phase_run_tables(n, f.c, f.lin0.data(), f.lin1.data(), tab.data());
    const void* dtab = stage(tab.data(), tab.size() * sizeof(float2));
    int q_pos = -1;
    std::array<double, 8> m2 = {1, 0, 0, 0, 0, 0, 1, 0};
    if (b.trailing_pair) {
        const SeqGate& t = gates[b.gates.back()];
        q_pos = n - 1 - t.bits[0];
        for (int e = 0; e < 4; ++e) {
            m2[2 * e] = t.mat[e].real();
            m2[2 * e + 1] = t.mat[e].imag();
        }
    }
    emit([=](q1g_state* x) {
        const uint64_t total = x->total();
        x->launch(q_pos >= 0 ? "phase_pair_run_c64" : "phase_run_c64", 2.0 * total * x->bsz(), [&] {
            return launch_phase_run(x->amps.as<float2>(), total, n, pivot_pos, dtab, q_pos, m2.data(), x->sm_count(),
                                    x->stream);
        });
    });
}

// The trailing gate's position of a phase-run block that can be a step of a
// group (phase_run.cu), -1 otherwise.  Positions 0 and 1 stay out: a thread's
// amplitudes would lie within one 32-byte sector, and every access of a warp
// would touch each sector several times.
static int group_position(const q1g_plan* p, const FusedBlock& b)
{
    if (!b.phase_run || !b.trailing_pair) return -1;
    const int t = p->nbits - 1 - p->gate_bits[b.gates.back()][0];
    return t >= 2 ? t : -1;
}

// Whether every angle is a number (a NaN has no fraction of a turn: such a run
// goes alone, where its tables carry it to the amplitudes that it turns).
static bool finite_phases(const PhaseFunction& f)
{
    auto all = [](const std::vector<double>& v) {
        return std::all_of(v.begin(), v.end(), [](double x) { return std::isfinite(x); });
    };
    return std::isfinite(f.c) && all(f.lin0) && all(f.lin1);
}

// Blocks i .. as one group as far as they go (two at least), after the plain
// gate `before` when the group starts with one (an uncontrolled 1-qubit
// gate).  Returns the number of blocks taken, 0 for none.
template <typename Stage, typename Emit>
static size_t lower_phase_group(q1g_plan* p, q1g_state* s, size_t i, const GateOp* before,
                                const std::vector<SeqGate>& gates, Stage&& stage, Emit&& emit)
{
    const int n = s->nbits;
    PhaseGroup g{};
    auto taken = [&](int t) { return std::find(g.t, g.t + g.nsteps, t) != g.t + g.nsteps; };
    if (before) g.t[g.nsteps++] = before->map.zpos[0];
    size_t count = 0;
    std::vector<PhaseFunction> phases;
    while (g.nsteps < kPhaseGroupMax && i + count < p->blocks.size()) {
        const FusedBlock& b = p->blocks[i + count];
        const int t = group_position(p, b);
        if (t < 0 || taken(t)) break;
        phases.push_back(phase_function(p, n, b, gates));
        if (!finite_phases(phases.back())) break;
        g.t[g.nsteps++] = t;
        ++count;
    }
    if (g.nsteps < 2) return 0;
    std::vector<PhaseStepTables> tables(g.nsteps);
    const std::vector<double> none(n, 0.0);
    for (int k = 0; k < g.nsteps; ++k) {
        double m2[8];
        PhaseFunction f;
        if (before && k == 0) {
            f.lin0 = f.lin1 = none;
            std::copy(before->m2, before->m2 + 8, m2);
        } else {
            const size_t at = (size_t)k - (before ? 1 : 0);
            f = phases[at];
            const SeqGate& t = gates[p->blocks[i + at].gates.back()];
            for (int e = 0; e < 4; ++e) {
                m2[2 * e] = t.mat[e].real();
                m2[2 * e + 1] = t.mat[e].imag();
            }
        }
        g.pivot[k] = f.pivot_pos;
        g.inner[k] = -1;
        for (int j = 0; j < g.nsteps; ++j)
            if (g.t[j] == f.pivot_pos) g.inner[k] = j;
        g.trivial0[k] = f.c == 0.0 && f.lin0 == none;
        g.real[k] = m2[1] == 0.0 && m2[3] == 0.0 && m2[5] == 0.0 && m2[7] == 0.0;
        for (int e = 0; e < 8; ++e) g.m2[k][e] = (float)m2[e];
        phase_group_tables(g, n, f.c, f.lin0.data(), f.lin1.data(), tables[k]);
    }
    const auto* d = static_cast<const PhaseStepTables*>(stage(tables.data(), tables.size() * sizeof(PhaseStepTables)));
    emit([=](q1g_state* x) {
        const uint64_t total = x->total();
        x->launch("phase_group_c64", 2.0 * total * x->bsz(), [&] {
            return launch_phase_group(x->amps.as<float2>(), total, n, g, d, x->sm_count(), x->stream);
        });
    });
    return count;
}

// Whether a dense block (its classified op, matrix and qubits) on this state
// runs on the tensor cores: complex64 in pairs of f16 halves (fused_tc.cu),
// complex128 in six digits (fused_tc_c128.cu) unless FP64 arithmetic was asked
// for.  Complex128 blocks with controls stay on the kernels that leave the other
// amplitudes alone: the digits would round those to the largest of their row.
static bool tc_takes(const q1g_plan* p, const q1g_state* s, const GateOp& op, const std::vector<cd>& mat,
                     const std::vector<int>& bits)
{
    return p->tensor_cores && s->nbits >= 12 && !(s->prec == kC128 && s->fp64_exact) && op.kind == GateOp::Dense &&
           op.t >= 3 && bits.size() <= 5 && (s->prec == kC64 || op.map.nz == op.t) &&
           tc_block_bounded(mat.data(), 1 << bits.size());
}

// A block as a tensor-core pass of a complex128 state.
template <typename Stage, typename Emit>
static void lower_z_block(q1g_state* s, const std::vector<cd>& mat, const std::vector<int>& bits, Stage&& stage,
                          Emit&& emit)
{
    const int n = s->nbits;
    const std::vector<int> T = tile_positions({&bits}, n);
    // gate positions: the block's own, padded from the tile's highest (rows
    // at the lowest positions make whole runs of the copies)
    std::vector<int> gpos = positions_of(bits, n);
    for (int j = 11; (int)gpos.size() < 5; --j)
        if (std::find(gpos.begin(), gpos.end(), T[j]) == gpos.end()) gpos.push_back(T[j]);
    std::sort(gpos.begin(), gpos.end());
    int gate_of[5];
    std::vector<int> order(5);      // qubits, matrix MSB first
    for (int k = 0; k < 5; ++k) {
        gate_of[k] = (int)(std::find(T.begin(), T.end(), gpos[k]) - T.begin());
        order[4 - k] = n - 1 - gpos[k];
    }
    ZPass pass;
    z_pass_layout(pass, T.data(), gate_of);
    const auto m32 = embed_matrix(mat, bits, order);
    const void* d = stage(m32.data(), m32.size() * sizeof(cd));
    emit([pass, d](q1g_state* x) {
        const uint64_t total = x->total();
        x->launch("fused_tc_c128", 2.0 * total * x->bsz(), [&] {
            return launch_fused_tc_c128(x->amps.as<double2>(), total, pass, d, x->errbuf.as<int>(), x->sm_count(),
                                        x->stream, x->tc_wait_ns);
        });
    });
}

// A plain gate (a pair or phase update that run_takes) with its matrix.
struct PlainGate {
    GateOp op;
    SeqGate gate;
};

// Microseconds of a complex128 tensor-core pass, or of a block's matrix on the
// host where that is longer.  26 qubits, 108 tiles per SM: 657 us straight to
// memory and 752 staged (6.1 and 7.0 per tile); which one a block takes is known
// only once it is laid out.
static double z_pass_us(uint64_t total, int sms)
{
    return std::max(5.0 + 6.4 * std::ceil((double)(total >> 12) / sms), 100.0);
}

// A run of plain gates: as tile passes (gate_run.h), or, on complex128
// states where that is faster by both paths' models, multiplied into blocks of
// up to five qubits (in FP64 on the host) for the tensor cores.  10 brick
// layers in us, tile passes and tensor cores: 20 qubits 965 / 412, 22 qubits
// 3680 / 1101, 24 qubits 15205 / 4758; but with new matrices, which the host
// multiplies first, 1175 / 1900, 3864 / 2486 and 15453 / 6337, so the line lies
// at 21 to 22 qubits.  Blocks without a gate that rounds every amplitude
// (controlled gates, phases, permutations alone) stay tile passes: those leave
// the bits of what no arithmetic touches.  A tile pass of one op, or one whose
// ops together touch less than the state where that is what costs (a state
// beyond the L2: two CX read and write half of it each), goes gate by gate.
template <typename Stage, typename Emit, typename Tc>
static void lower_plain_gates(q1g_plan* p, q1g_state* s, const std::vector<PlainGate>& run, Stage&& stage, Emit&& emit,
                              Tc&& tensor_cores)
{
    const uint64_t total = s->total();
    auto one = [&](const GateOp& op) {
        emit([op](q1g_state* x) { x->apply_op(op, x->amps.as<char>(), x->total()); });
    };
    if (run.size() < 2) {
        for (const PlainGate& g : run) one(g.op);
        return;
    }
    // tile passes of the gates `at` of the run
    auto group = [&](const std::vector<int>& at, double* cost) {
        std::vector<const GateOp*> list;
        for (int i : at) list.push_back(&run[i].op);
        return group_runs(list, s->nbits, total, s->prec, s->fp64_exact, cost, s->sm_count());
    };
    const bool pairs = s->prec == kC128 && !s->fp64_exact;
    std::vector<RunOp> table;
    auto emit_passes = [&](const std::vector<int>& at, const std::vector<RunPass>& passes) {
        for (const RunPass& pass : passes) {
            uint64_t touched = 0;
            bool units = true, rounded = false;
            for (int i : pass.ops) {
                const GateOp& op = run[at[i]].op;
                touched += op.touched(total);
                units = units && is_unit(op);
                rounded = rounded || rounds_all(op);
            }
            if (pass.ops.size() < 2 || (touched <= total && total * s->bsz() > (uint64_t(64) << 20))) {
                for (int i : pass.ops) one(run[at[i]].op);
                continue;
            }
            table.clear();
            for (int i : pass.ops) table.push_back(make_run_op(run[at[i]].op, pass.tile));
            const RunArith arith = !pairs || units ? RunArith::kPlain
                                   : rounded       ? RunArith::kPairs
                                                   : RunArith::kPairsPartly;
            const char* name = s->prec == kC64 ? "gate_run_c64" : s->fp64_exact ? "gate_run_c128_fp64" : "gate_run_c128";
            const RunOp* d = static_cast<const RunOp*>(stage(table.data(), table.size() * sizeof(RunOp)));
            emit([name, arith, tile = pass.tile, d, n = (int)table.size()](q1g_state* x) {
                x->launch(name, 2.0 * x->total() * x->bsz(), [&] {
                    return launch_gate_run(x->amps.p, x->prec, x->total(), tile, d, n, arith, x->stream);
                });
            });
        }
    };
    std::vector<int> all(run.size());
    std::iota(all.begin(), all.end(), 0);
    double cost = 0.0;
    const std::vector<RunPass> passes = group(all, &cost);
    if (pairs && p->tensor_cores && s->nbits >= 12 && cost > 2.0 * z_pass_us(total, s->sm_count())) {
        std::vector<std::vector<int>> bits;
        for (const PlainGate& g : run) bits.push_back(g.gate.bits);
        const std::vector<FusedBlock> blocks = fuse(bits, s->nbits, 5);
        // the blocks in order: one for the tensor cores, or the gates of
        // neighbours that are not, as tile passes
        struct Part {
            int block = -1;
            std::vector<int> gates;
            std::vector<RunPass> passes;
        };
        std::vector<Part> parts;
        double us = 0.0;
        bool faster = true;
        for (size_t i = 0; i < blocks.size(); ++i) {
            const FusedBlock& b = blocks[i];
            faster = faster && b.qubits.size() <= 5;
            if (std::any_of(b.gates.begin(), b.gates.end(), [&](int g) { return rounds_all(run[g].op); })) {
                parts.emplace_back();
                parts.back().block = (int)i;
                us += z_pass_us(total, s->sm_count());
                continue;
            }
            if (parts.empty() || parts.back().block >= 0) parts.emplace_back();
            parts.back().gates.insert(parts.back().gates.end(), b.gates.begin(), b.gates.end());
        }
        for (Part& part : parts) {
            if (part.block >= 0 || !faster) continue;
            double tiles = 0.0;
            part.passes = group(part.gates, &tiles);
            us += tiles;
        }
        faster = faster && us < cost;
        if (faster) {
            std::vector<SeqGate> gates;
            for (const PlainGate& g : run) gates.push_back(g.gate);
            std::vector<std::vector<cd>> mats(blocks.size());
            for (const Part& part : parts) {
                if (part.block < 0) continue;
                const FusedBlock& b = blocks[part.block];
                mats[part.block] = block_matrix(b, gates);
                faster = faster && tc_block_bounded(mats[part.block].data(), 1 << b.qubits.size());
            }
            if (faster) {
                for (const Part& part : parts) {
                    if (part.block < 0) {
                        emit_passes(part.gates, part.passes);
                        continue;
                    }
                    const std::vector<int>& q = blocks[part.block].qubits;
                    const std::vector<cd>& mat = mats[part.block];
                    const GateOp op = classify(mat.data(), (int)q.size(), q.data(), s->nbits);
                    if (op.kind == GateOp::Dense) {
                        tensor_cores();
                        lower_z_block(s, mat, q, stage, emit);
                    } else if (op.kind != GateOp::Noop) {
                        one(op);
                    }
                }
                return;
            }
        }
    }
    emit_passes(all, passes);
}

// Device bytes of a block's staged data at most: a run table entry per gate
// (and its alignment), a swap tile or phase tables, a dense matrix in one of
// its forms, or a tensor-core image.
static size_t staging_bytes(const FusedBlock& b)
{
    size_t n = b.gates.size() * 512;
    if (b.phase_run || b.swap_run || b.qubits.size() >= 3) n += 32768;
    else n += 2048;
    return n;
}

// Positions a plan may leave out of its start-of-run subspace: the compact
// state is at most 1/8 of the full one.  Below kPrefixMinQubits a full pass
// costs microseconds, less than the compact plan's own launches and norm
// check (a 16-qubit brick of 20 layers with 8192 runs took 6.4 ms with the
// prefix against 4.3 ms without).
constexpr int kPrefixSpare = 3;
constexpr int kPrefixMinQubits = 24;

// A basis state stays a basis state on every position no gate has touched.
// So the plan's leading blocks, as long as together they touch at most
// nbits - kPrefixSpare positions, run on a compact state of those positions
// (the same blocks on renumbered qubits); the full state is then zeroed and
// the compact one scattered into it, which replaces the fill of the basis
// state.  Returns the number of blocks done.
static size_t run_subspace_prefix(q1g_plan* p, q1g_state* s, const double* mats, size_t n)
{
    const int nb = s->nbits;
    if (!p->prefix_known) {
        p->prefix_known = true;
        uint64_t mask = 0;
        size_t len = 0;
        for (const auto& b : p->blocks) {
            if (b.phase_run || b.swap_run) break;
            uint64_t m = mask;
            for (int q : b.qubits) m |= uint64_t(1) << (nb - 1 - q);
            if (__builtin_popcountll(m) > nb - kPrefixSpare) break;
            mask = m;
            ++len;
        }
        if (len >= 2 && nb >= kPrefixMinQubits) {
            const int na = __builtin_popcountll(mask);
            auto cq = [&](int q) {
                const int pos = nb - 1 - q;
                return na - 1 - __builtin_popcountll(mask & ((uint64_t(1) << pos) - 1));
            };
            auto tp = std::make_unique<q1g_plan>();
            tp->nbits = na;
            tp->width = p->width;
            tp->tensor_cores = p->tensor_cores;
            tp->tc_pairs = p->tc_pairs;
            tp->tc_max_high = p->tc_max_high;
            tp->tc_slack = p->tc_slack;
            tp->gate_bits = p->gate_bits;
            tp->mat_off = p->mat_off;
            tp->mat_doubles = p->mat_doubles;
            tp->kinds = p->kinds;
            for (size_t i = 0; i < len; ++i) {
                FusedBlock b = p->blocks[i];
                for (auto& q : b.qubits) q = cq(q);
                for (int g : b.gates)
                    for (size_t j = 0; j < p->gate_bits[g].size(); ++j) tp->gate_bits[g][j] = cq(p->gate_bits[g][j]);
                tp->blocks.push_back(b);
            }
            p->prefix_len = len;
            p->prefix_mask = mask;
            p->prefix_plan = std::move(tp);
        }
    }
    if (!p->prefix_plan) return 0;
    const uint64_t mask = p->prefix_mask;
    const int na = __builtin_popcountll(mask);
    if (!s->compact || s->compact->nbits != na || s->compact->prec != s->prec)
        s->compact = std::make_unique<q1g_state>(na, s->nshots, s->prec, s->stream);
    q1g_state* c = s->compact.get();
    c->stream = s->stream;
    c->fp64_exact = s->fp64_exact;
    c->tc_wait_ns = s->tc_wait_ns;
    c->prof = s->prof;
    c->nshots = s->nshots;
    const uint64_t b = s->basis[0];
    uint64_t cb = 0;
    SubspacePositions sp{};
    for (int pos = 0; pos < nb; ++pos)
        if ((mask >> pos) & 1) {
            if ((b >> pos) & 1) cb |= uint64_t(1) << sp.n;
            sp.pos[sp.n++] = pos;
        }
    c->sparse = true;
    c->basis.assign(1, cb);
    c->counts.assign(1, s->counts[0]);
    c->ncols = 1;
    c->norms.assign(1, s->norms[0]);
    plan_run(p->prefix_plan.get(), c, mats, n, false);
    c->ensure_dense();
    s->amps.ensure(s->N * s->bsz());
    s->launch("subspace_fill", double(s->N * s->bsz()), [&] {
        return launch_scatter_subspace(s->amps.p, c->amps.p, s->prec, nb, na, sp, b & ~mask, s->stream);
    });
    s->sparse = false;
    s->basis.clear();
    s->norm_pending = c->norm_pending;    // the compact plan's norm correction, if any, is still to come
    c->norm_pending = false;
    for (auto& pe : c->pending) s->pending.push_back(pe);
    c->pending.clear();
    return p->prefix_len;
}

// Lowers the plan's blocks from `first` on into L and launches each pass as
// it is ready, so the host work of pass i+1 (block product, classification,
// tensor-core image) runs while the device executes pass i.
static void lower_and_run(q1g_plan* p, q1g_state* s, const double* mats, size_t first, q1g_plan::Lowered& L)
{
    const size_t ng = p->gate_bits.size();
    std::vector<SeqGate> gates(ng);
    for (size_t g = 0; g < ng; ++g) {
        const size_t k = p->gate_bits[g].size();
        const size_t dim = size_t(1) << k;
        gates[g].bits = p->gate_bits[g];
        gates[g].mat.resize(dim * dim);
        const double* m = mats + p->mat_off[g];
        for (size_t e = 0; e < dim * dim; ++e) gates[g].mat[e] = cd(m[2 * e], m[2 * e + 1]);
    }
    const size_t nb = p->blocks.size();
    std::vector<GateOp> ops(nb);
    std::vector<std::vector<cd>> bmats(nb);
    std::vector<std::vector<int>> bbits(nb);
    std::vector<char> ready(nb, 0);
    auto prepare = [&](size_t bi) {
        if (ready[bi]) return;
        const auto& b = p->blocks[bi];
        if (b.gates.size() == 1) {
            bmats[bi] = gates[b.gates[0]].mat;
            bbits[bi] = gates[b.gates[0]].bits;
        } else {
            bmats[bi] = block_matrix(b, gates);
            bbits[bi] = b.qubits;
        }
        ops[bi] = classify(bmats[bi].data(), (int)bbits[bi].size(), bbits[bi].data(), s->nbits);
        ready[bi] = 1;
    };
    // The layout of a tensor-core pass of nblk blocks from block i on
    auto layout = [&](size_t i, int nblk) -> std::shared_ptr<const TcPass> {
        std::vector<int> key = {s->nbits, (int)s->ncols, p->tc_slack, p->tc_pairs, nblk};
        std::vector<const std::vector<int>*> bits;
        for (int j = 0; j < nblk; ++j) {
            bits.push_back(&bbits[i + j]);
            key.push_back(-1);
            key.insert(key.end(), bbits[i + j].begin(), bbits[i + j].end());
        }
        auto& e = p->tc_layouts[key];
        if (e) return e;
        auto pass = std::make_shared<TcPass>(lower_tc_pass(bits, s->nbits, s->ncols, p->tc_slack,
                                                           nblk > 1 ? p->tc_pairs : p->tc_pairs >= 4 ? 4 : 1));
        if (nblk == 2 && (pass->offs.shuffle || pass->offs.direct) && pass->offs.pad_shift < 31) {
            // the shuffled or direct row layout needs padding (bank
            // conflicts); the staged one, free to order its rows, may not:
            // one tensor-map copy per tile is kept if it can
            TcPass staged = lower_tc_pass(bits, s->nbits, s->ncols, p->tc_slack, 1);
            if (staged.offs.pad_shift >= 31) *pass = std::move(staged);
        }
        e = std::move(pass);
        return e;
    };
    auto eligible = [&](size_t bi) {
        if (p->blocks[bi].phase_run || p->blocks[bi].swap_run) return false;
        prepare(bi);
        return tc_takes(p, s, ops[bi], bmats[bi], bbits[bi]);
    };
    auto tensor_cores = [&] {
        if (L.tensor_cores) return;
        s->clear_error_flag();
        L.tensor_cores = true;
    };
    // Staging: every pass uploads its matrix or tensor-core image from its own
    // slice of a pinned chunk into its own slice of L's chunk of that number.
    // Nothing may still read those: earlier launches on this stream precede
    // the copies, those on others are waited for.
    if (p->staged) check_cuda(cudaEventSynchronize(p->staged), "plan staging wait");
    else check_cuda(cudaEventCreateWithFlags(&p->staged, cudaEventDisableTiming), "cudaEventCreate");
    if (L.several_streams || (L.stream && L.stream != s->stream)) check_cuda(cudaDeviceSynchronize(), "plan upload wait");
    L.several_streams = false;
    L.stream = s->stream;
    L.launches.clear();
    L.tensor_cores = false;
    size_t staging = 256;
    for (const auto& b : p->blocks) staging += staging_bytes(b);
    size_t chunk = 0, room = 0, staged = 0;      // chunks begun; the last one's size, and its bytes in use
    auto stage = [&](const void* src, size_t sz) -> const void* {
        if (staged + sz > room) {
            // the first chunk takes what the blocks themselves need; further
            // ones are for plain gates that became tensor-core blocks
            const size_t want = std::max(sz, chunk == 0 ? staging : size_t(1) << 18);
            if (p->hmats.size() == chunk) p->hmats.emplace_back();
            if (L.dmats.size() == chunk) L.dmats.emplace_back();
            p->hmats[chunk].ensure(want);
            L.dmats[chunk].ensure(want);
            room = std::min(p->hmats[chunk].bytes, L.dmats[chunk].bytes);
            staged = 0;
            ++chunk;
        }
        char* h = p->hmats[chunk - 1].as<char>() + staged;
        char* d = L.dmats[chunk - 1].as<char>() + staged;
        std::memcpy(h, src, sz);
        s->h2d(d, h, sz, "upload plan matrix");
        staged += (sz + 255) & ~size_t(255);
        return d;
    };
    auto emit = [&](std::function<void(q1g_state*)> f) {
        if (L.launches.empty()) s->ensure_dense();
        f(s);
        L.launches.push_back(std::move(f));
    };
    // plain gates (pairs and phases) gathered until another kind of block
    // comes, then grouped into tile passes
    std::vector<PlainGate> plain;
    auto flush_plain = [&] {
        if (plain.empty()) return;
        lower_plain_gates(p, s, plain, stage, emit, tensor_cores);
        plain.clear();
    };
    // A complex128 block of gates of 0, +-1 and +-i alone: a dense product would
    // round the amplitudes that the gates only move, so they go with the plain
    // gates, as long as the tile passes cost no more than a dense pass (about 30
    // CX at 26 qubits).
    auto take_unit_gates = [&](size_t i) {
        std::vector<PlainGate> units;
        for (int g : p->blocks[i].gates) {
            GateOp o = classify(gates[g].mat.data(), (int)gates[g].bits.size(), gates[g].bits.data(), s->nbits);
            if (o.kind == GateOp::Noop) continue;
            if (!is_unit(o)) return false;
            units.push_back({std::move(o), gates[g]});
        }
        std::vector<const GateOp*> list;
        for (const PlainGate& g : units) list.push_back(&g.op);
        double cost = 0.0;
        group_runs(list, s->nbits, s->total(), s->prec, false, &cost, s->sm_count());
        if (cost > z_pass_us(s->total(), s->sm_count())) return false;
        for (PlainGate& g : units) plain.push_back(std::move(g));
        return true;
    };
    // A complex128 block that is not one for the tensor cores, gate by gate (its
    // product would take the FP64 pipe from four qubits on).
    auto take_apart = [&](size_t i) {
        for (int g : p->blocks[i].gates) {
            const SeqGate& q = gates[g];
            GateOp o = classify(q.mat.data(), (int)q.bits.size(), q.bits.data(), s->nbits);
            if (o.kind == GateOp::Noop) continue;
            if (run_takes(o)) {
                plain.push_back({std::move(o), q});
                continue;
            }
            flush_plain();
            if (tc_takes(p, s, o, q.mat, q.bits)) {
                tensor_cores();
                lower_z_block(s, q.mat, q.bits, stage, emit);
            } else {
                emit([o](q1g_state* x) { x->apply_op(o, x->amps.as<char>(), x->total()); });
            }
        }
    };
    for (size_t i = first; i < nb; ++i) {
        if (p->blocks[i].phase_run && !phase_kernels_take(s)) {
            for (int g : p->blocks[i].gates) {
                GateOp op = classify(gates[g].mat.data(), (int)gates[g].bits.size(), gates[g].bits.data(), s->nbits);
                if (op.kind == GateOp::Noop) continue;
                if (run_takes(op)) {
                    plain.push_back({std::move(op), gates[g]});
                } else {
                    flush_plain();
                    emit([op](q1g_state* x) { x->apply_op(op, x->amps.as<char>(), x->total()); });
                }
            }
            continue;
        }
        if (!p->blocks[i].phase_run && !p->blocks[i].swap_run) {
            prepare(i);
            if (ops[i].kind == GateOp::Noop) continue;
            if (run_takes(ops[i])) {
                plain.push_back({ops[i], {bbits[i], bmats[i]}});
                continue;
            }
            if (s->prec == kC128 && !s->fp64_exact && take_unit_gates(i)) continue;
            if (s->prec == kC128 && !s->fp64_exact && p->tensor_cores && s->nbits >= 12 && ops[i].t >= 3 &&
                p->blocks[i].gates.size() > 1 && ops[i].map.nz != ops[i].t) {
                take_apart(i);
                continue;
            }
        }
        if (p->blocks[i].phase_run) {
            // an uncontrolled gate just before (a Fourier transform's first
            // Hadamard) is the group's first step
            const GateOp* before = plain.size() == 1 && plain[0].op.kind == GateOp::Pair &&
                                           plain[0].op.map.nz == 1 && plain[0].op.map.zpos[0] >= 2
                                       ? &plain[0].op
                                       : nullptr;
            size_t count = before ? lower_phase_group(p, s, i, before, gates, stage, emit) : 0;
            if (count) {
                plain.clear();
            } else {
                flush_plain();
                count = lower_phase_group(p, s, i, nullptr, gates, stage, emit);
            }
            if (count) {
                i += count - 1;
                continue;
            }
        }
        if (s->prec == kC128 && !s->fp64_exact && p->tensor_cores && p->width < 5 &&
            s->total() >= (uint64_t(1) << 22) && !p->blocks[i].phase_run && !p->blocks[i].swap_run &&
            ops[i].kind == GateOp::Dense) {
            // A narrow plan's blocks on a large state: a pass takes the same
            // time for three qubits as for five, so their gates are grouped
            // anew with the plain ones (30 qubits, depth 24, plan of width 3:
            // 1.84 s for its 169 passes, 0.58 s so).
            std::vector<PlainGate> again;
            for (int g : p->blocks[i].gates) {
                GateOp o = classify(gates[g].mat.data(), (int)gates[g].bits.size(), gates[g].bits.data(), s->nbits);
                if (o.kind == GateOp::Noop) continue;
                if (!run_takes(o)) {
                    again.clear();
                    break;
                }
                again.push_back({std::move(o), gates[g]});
            }
            if (!again.empty()) {
                for (PlainGate& g : again) plain.push_back(std::move(g));
                continue;
            }
        }
        flush_plain();
        if (p->blocks[i].phase_run) {
            lower_phase_block(p, s, p->blocks[i], gates, stage, emit);
            continue;
        }
        if (p->blocks[i].swap_run) {
            lower_swap_block(s, p->blocks[i], gates, stage, emit);
            continue;
        }
        const GateOp& op = ops[i];
        if (s->prec == kC128 && eligible(i)) {
            tensor_cores();
            lower_z_block(s, bmats[i], bbits[i], stage, emit);
        } else if (eligible(i)) {
            // consecutive blocks share a pass when their qubits fit one
            // 12-position tile with runs of >= 128 amplitudes or as one
            // tensor-map box: up to three in the four-group kernel's direct
            // chain in pair mode 5, else two
            std::shared_ptr<const TcPass> t;
            int group = 1;
            // -1: blocks i .. i+k-1 do not fit one tile; else its run bits
            auto fits = [&](int k) {
                std::vector<const std::vector<int>*> bs;
                std::vector<int> u;
                for (int j = 0; j < k; ++j) {
                    bs.push_back(&bbits[i + j]);
                    for (int q : positions_of(bbits[i + j], s->nbits))
                        if (std::find(u.begin(), u.end(), q) == u.end()) u.push_back(q);
                }
                if (u.size() > 12) return -1;
                const auto Tk = tile_positions(bs, s->nbits);
                int high = 0;
                for (int q : Tk) high += q >= kHighPosition;
                const int L = tile_run_bits(Tk);
                if (high > p->tc_max_high) return -1;
                if (L < kMinTcRunBits && !tc_tile_box(Tk.data(), s->nbits, s->ncols).usable) return -1;
                return L;
            };
            if (p->tc_pairs == 5 && i + 2 < nb && eligible(i + 1) && eligible(i + 2)) {
                const int L3 = fits(3);
                if (L3 >= 0) {
                    t = layout(i, 3);
                    // short runs only as one unpadded tensor-map copy; a
                    // third block only where the tile's runs are at least
                    // 64 bytes (a copy of 16- or 32-byte runs wastes DRAM
                    // sectors: such passes ran at 19-46 % of DRAM rate) and
                    // the layout keeps the bank wavefronts within twice the
                    // minimum (a conflicted write-back costs more than the
                    // saved pass)
                    if ((L3 >= kMinTcRunBits || t->offs.pad_shift >= 31) && L3 >= kMinTripleRunBits &&
                        t->cost <= 2 * t->ideal)
                        group = 3;
                }
            }
            if (group == 1 && p->tc_pairs && i + 1 < nb && eligible(i + 1)) {
                const int L2 = fits(2);
                if (L2 >= 0) {
                    t = layout(i, 2);
                    if (L2 >= kMinTcRunBits || t->offs.pad_shift >= 31) group = 2;
                }
            }
            if (group == 1) t = layout(i, 1);
            tensor_cores();
            const std::vector<cd>* gm[kTcMaxBlocks];
            const std::vector<int>* gq[kTcMaxBlocks];
            for (int j = 0; j < group; ++j) gm[j] = &bmats[i + j], gq[j] = &bbits[i + j];
            const std::vector<uint16_t> images = tc_images(*t, gm, gq, group);
            const void* img = stage(images.data(), images.size() * sizeof(uint16_t));
            emit([t, img](q1g_state* x) {
                TcOffsets offs = t->offs;
                tc_operand_scales(*std::max_element(x->norms.begin(), x->norms.end()), offs);
                const uint64_t total = x->total();
                x->launch("fused_tc_c64", 2.0 * total * x->bsz(), [&] {
                    return launch_fused_tc(x->amps.as<float2>(), total >> 12, t->tilemap, offs, t->box, img,
                                           x->errbuf.as<int>(), x->sm_count(), x->stream, x->tc_wait_ns,
                                           offs.st_box ? &t->sbox : nullptr);
                });
            });
            i += (size_t)(group - 1);   // the next blocks rode in this pass
        } else {
            emit([op](q1g_state* x) { x->apply_op(op, x->amps.as<char>(), x->total()); });
        }
    }
    flush_plain();
    check_cuda(cudaEventRecord(p->staged, s->stream), "cudaEventRecord");
}

// The leading blocks of a plan that act on one qubit each (a circuit's first
// layer), on a basis state: its qubits' vectors multiplied out on the host, and
// the product state written in one pass.  Complex128 in double-float pairs
// only: the result is FP64's, where the gates would each round at 2^-48 (a
// 24-qubit circuit of 2 layers: 9e-15 off before, 5e-15 now), in the time of the
// tile pass that it saves (16 qubits, 20 layers: 400 us either way; 26 qubits,
// 6 layers, in the compact state: 0.6 ms less than with the gates).  Returns the
// number of blocks done.
static size_t run_product_lead(const q1g_plan* p, q1g_state* s, const double* mats)
{
    if (s->prec != kC128 || s->fp64_exact || s->nbits > 40) return 0;
    const int nb = s->nbits;
    size_t lead = 0;
    for (; lead < p->blocks.size(); ++lead) {
        const FusedBlock& b = p->blocks[lead];
        if (b.phase_run || b.swap_run || b.qubits.size() != 1) break;
        bool bounded = true;
        for (int g : b.gates)
            for (int e = 0; e < 8; ++e) bounded = bounded && std::fabs(mats[p->mat_off[g] + e]) <= 2.0;
        if (!bounded) break;       // (nor NaN)
    }
    if (lead < 2) return 0;
    ProductCoefs c{};
    for (int q = 0; q < nb; ++q) c.c[4 * q + (((s->basis[0] >> (nb - 1 - q)) & 1) ? 2 : 0)] = 1.0;
    for (size_t i = 0; i < lead; ++i) {
        const FusedBlock& b = p->blocks[i];
        double* v = c.c + 4 * b.qubits[0];
        for (int g : b.gates) {
            const double* m = mats + p->mat_off[g];
            const cd x0(v[0], v[1]), x1(v[2], v[3]);
            const cd y0 = cd(m[0], m[1]) * x0 + cd(m[2], m[3]) * x1, y1 = cd(m[4], m[5]) * x0 + cd(m[6], m[7]) * x1;
            v[0] = y0.real(), v[1] = y0.imag(), v[2] = y1.real(), v[3] = y1.imag();
        }
    }
    s->product_state(c);
    return lead;
}

void plan_run(q1g_plan* p, q1g_state* s, const double* mats, size_t n, bool subspace_prefix)
{
    if (n != p->mat_doubles)
        throw Error(Q1G_ERR_INVALID_ARGUMENT, "expected " + std::to_string(p->mat_doubles) + " matrix doubles");
    if (s->nbits != p->nbits)
        throw Error(Q1G_ERR_INVALID_ARGUMENT, "plan and state differ in qubit count");
    size_t first = 0;
    if (s->sparse && s->ncols == 1 && s->basis.size() == 1) {
        if (subspace_prefix) first = run_subspace_prefix(p, s, mats, n);
        if (first == 0) first = run_product_lead(p, s, mats);
    }
    q1g_plan::Lowered& L = p->lowered[first > 0];
    const int tiling[4] = {p->tensor_cores, p->tc_pairs, p->tc_max_high, p->tc_slack};
    const bool same = L.valid && L.prec == s->prec && L.fp64_exact == s->fp64_exact && L.ncols == s->ncols &&
                      L.first == first && std::memcmp(L.tiling, tiling, sizeof tiling) == 0 &&
                      std::memcmp(L.mats.data(), mats, n * sizeof(double)) == 0;
    if (same) {
        if (!L.launches.empty()) s->ensure_dense();
        if (L.tensor_cores) s->clear_error_flag();
        if (L.stream != s->stream) {
            // uploaded on another stream
            check_cuda(cudaStreamWaitEvent(s->stream, p->staged, 0), "plan upload wait");
            L.several_streams = true;
            L.stream = s->stream;
        }
        for (auto& f : L.launches) f(s);
    } else {
        L.valid = false;
        try {
            lower_and_run(p, s, mats, first, L);
        } catch (...) {
            // copies out of the staging buffer may be under way
            cudaStreamSynchronize(s->stream);
            throw;
        }
        L.prec = s->prec;
        L.fp64_exact = s->fp64_exact;
        L.ncols = s->ncols;
        L.first = first;
        std::copy(tiling, tiling + 4, L.tiling);
        L.mats.assign(mats, mats + n);
        L.valid = true;
    }
    if (L.tensor_cores) {
        // the tensor-core passes' bounded waits: report an expiry now
        s->hstage.ensure(sizeof(int));
        int* h_flag = s->hstage.as<int>();
        s->d2h(h_flag, s->errbuf.p, sizeof(int), "read error flag");
        s->sync();
        if (*h_flag) throw Error(Q1G_ERR_TIMEOUT, "a tensor-core block kernel gave up waiting on its MMAs");
        // (complex128 passes round to nearest and keep the norm)
        s->norm_pending = s->norm_pending || s->prec == kC64;
    }
}

}  // namespace q1g

std::vector<double> q1g_state::measure_norms()
{
    using namespace q1g;
    if (sparse) return std::vector<double>(ncols, 1.0);
    q1g_state* s = this;
    const uint64_t total = s->total();
    const uint64_t chunk = std::min<uint64_t>(s->N, 256);
    const uint64_t nch = s->N / chunk;
    const uint64_t ntmp = segment_sums_tmp_doubles(s->ncols, nch);
    s->dscratch.ensure((s->ncols * nch + 2 * s->ncols + ntmp) * sizeof(double));
    double* d_sums = s->dscratch.as<double>();
    double* d_norm = d_sums + s->ncols * nch;
    s->launch("column_norms", double(total * s->bsz()), [&] {
        return launch_chunk_sums_dense(s->amps.p, s->prec, total, chunk, d_sums, nullptr, Spacings{}, s->stream);
    });
    check_cuda(launch_segment_sums(d_sums, s->ncols, nch, d_norm, d_norm + 2 * s->ncols, s->stream),
               "segment_sums");
    s->hstage.ensure(s->ncols * sizeof(double));
    double* h_norm = s->hstage.as<double>();
    s->d2h(h_norm, d_norm, s->ncols * sizeof(double), "read norms");
    s->sync();
    return std::vector<double>(h_norm, h_norm + s->ncols);
}

void q1g_state::settle_norms()
{
    using namespace q1g;
    if (!norm_pending || sparse) {
        norm_pending = false;
        return;
    }
    q1g_state* s = this;
    {
        // per-column squared norms now, then rescale each column to the norm
        // it should have (the plans since the last settle were unitary)
        const std::vector<double> h_norm = s->measure_norms();
        const uint64_t total = s->total();
        std::vector<double> scale(s->ncols, 1.0);
        bool any_scale = false;
        for (uint64_t c = 0; c < s->ncols; ++c) {
            if (h_norm[c] > 0.0) scale[c] = std::sqrt(s->norms[c] / h_norm[c]);
            any_scale |= scale[c] != 1.0;
        }
        if (any_scale) {
            // measure_norms left its sums in dscratch: the scales go after them
            const uint64_t nch = s->N / std::min<uint64_t>(s->N, 256);
            double* d_scale = s->dscratch.as<double>() + s->ncols * nch + s->ncols;
            s->h2d(d_scale, scale.data(), s->ncols * sizeof(double), "upload scales");
            s->launch("renormalise", 2.0 * total * s->bsz(), [&] {
                return launch_scale_columns(s->amps.p, s->prec, s->N, s->ncols, d_scale, s->stream);
            });
            s->sync();
        }
    }
    norm_pending = false;
}
