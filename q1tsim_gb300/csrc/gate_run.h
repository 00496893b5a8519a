// Runs of plain gates applied in one pass: consecutive pair and phase
// updates whose target positions lie in one tile of the state are applied to
// the tile in shared memory one after the other, so that the state crosses
// HBM (and the host launches) once per run instead of once per gate.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "gate_plan.h"

namespace q1g {

// Tile bits a run's pass may have (2^11 amplitudes of 16 bytes: 32 KB, four
// tiles resident per SM; 2^12 ran 5 % slower at 26 qubits) and gates per
// launch (their table sits in shared memory beside the tile).
constexpr int kRunMaxTileBits = 11;
constexpr int kRunMaxOps = 64;

// A gate of a run on tile-local indices (local bit k = the tile's k-th
// position).  Unit u of the op is the local index u with zero bits inserted
// at the op's nz local positions (hi[q] = ~((1 << position) - 1), ascending),
// OR set; a pair's members add o0 and o1.  The op applies to the tiles whose
// base index has (base & extmask) == extset (controls outside the tile).
enum RunKind : uint32_t { kRunPair = 0, kRunPairMono = 1, kRunPhase = 2, kRunPhaseMono = 3 };
// Zero coefficients of a pair's matrix: all four terms of each output; U3
// (im m00 = 0); real (H, RY); real diagonal with imaginary off-diagonal (RX).
enum RunShape : uint32_t { kRunFull = 0, kRunReal00 = 1, kRunReal = 2, kRunCross = 3 };
struct RunOp {
    double m[8];          // matrix (re, im) row-major, or the phase in m[0..1]
    float4 df[4];         // double-float: entry e as (re.h, re.l, im.h, im.l)
    float rest[8];        // what df leaves of m
    uint64_t extmask, extset;
    uint32_t kind, shape;
    uint32_t nz, set, o0, o1;
    uint32_t code;        // mono: swap | u0 << 1 | u1 << 3 (gate_kernels.cu's unit codes)
    uint32_t pad_;
    uint16_t hi[12];
    uint16_t pad2_[4];
};
static_assert(sizeof(RunOp) % 16 == 0, "RunOp copies as 16-byte words");

struct RunTile {
    int bits;                     // tile positions
    int pad_;
    uint64_t off[kRunMaxTileBits];   // amplitude offset of local bit k (1 << position)
    IndexMap map;                 // the positions, zeroed: tile number -> base
};

// A launch: tile and ops (indices into the op list it was grouped from).
struct RunPass {
    RunTile tile;
    std::vector<int> ops;
};

// Positions of `op` that a tile must hold for the op to run in it (those in
// which a pair's two members differ; none for a phase).
uint64_t run_need(const GateOp& op);
// Whether an op can be part of a run: a pair or a phase whose matrix does not
// grow amplitudes (rows of |re| + |im| sums <= 2.01), on at most 12 positions.
bool run_takes(const GateOp& op);
// Whether a gate moves and re-signs amplitudes without arithmetic (entries of
// 0, +-1 and +-i).
bool is_unit(const GateOp& op);
// Whether a gate's arithmetic rounds every amplitude of the state (an
// uncontrolled pair update).  Only beside such a gate may the others' amplitudes
// be held rounded: without one, some amplitudes are touched by no arithmetic
// and keep their bits.
bool rounds_all(const GateOp& op);
// Groups `ops` (in order; every one run_takes and not a Noop) into passes on
// a state of nbits qubits.  Ops on disjoint positions may change places, which
// changes roundings; with fp64_exact, whose purpose is the rounding of the gates
// one by one, they keep their order.
// prec / fp64_exact choose the cost model's arithmetic rates.
// *cost_us: the model's time for them, on a device of `sms` SMs.
std::vector<RunPass> group_runs(const std::vector<const GateOp*>& ops, int nbits, uint64_t total, int prec,
                                bool fp64_exact, double* cost_us = nullptr, int sms = 152);
// The op in the tile's local coordinates.
RunOp make_run_op(const GateOp& op, const RunTile& tile);

// A complex128 pass's arithmetic: in the state's type (FP64, or gates that
// is_unit alone), in double-float pairs beside a gate that rounds_all, or in
// pairs with the amplitudes followed that no gate rounds.
enum class RunArith { kPlain, kPairs, kPairsPartly };
// gate_run.cu: applies d_ops[0..nops) (nops <= kRunMaxOps) to every tile of
// `total` amplitudes (complex64: any arith).
cudaError_t launch_gate_run(void* amps, int prec, uint64_t total, const RunTile& tile, const RunOp* d_ops, int nops,
                            RunArith arith, cudaStream_t st);

}  // namespace q1g
