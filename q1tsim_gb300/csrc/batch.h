// Batched executor: host state of a batch of independent circuits.
#pragma once

#include <vector>

#include "engine.h"

namespace q1g {
// How a batch's largest circuits run: the first `circuits` of the queue on
// `count` teams of `size` CTAs.
struct TeamPlan {
    int circuits = 0, size = 1, count = 0;
};
}  // namespace q1g

struct q1g_batch {
    int width = 4;                      // fusion width (<= 4)
    std::vector<q1g::BatchCircuit> circuits;   // in add order; res_off set at build
    std::vector<q1g::BatchOp> ops;
    std::vector<float2> mats;
    std::vector<uint64_t> cbit_tables;
    bool built = false;
    uint64_t total_runs = 0;
    uint64_t arena_amps = 0;
    uint64_t scratch_per_cta = 0;
    int sms = 0;
    int team_size = 0;                  // CTAs of a team as asked for (0: chosen by the estimate)
    q1g::TeamPlan teams;                // set at build
    q1g::DevBuf arena, results, dcircuits, dops, dmats, dtables, lfact, scratch, queue, traffic;
    q1g::HostBuf hresults, htraffic;
    cudaStream_t stream = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    float last_ms = 0.f;
    uint64_t last_traffic = 0;          // algorithmic device-memory bytes of the last run
    ~q1g_batch();
};

namespace q1g {
void batch_add_circuit(q1g_batch* b, size_t nr_bits, size_t nr_shots, uint64_t seed, size_t nops, const int* kinds,
                       const size_t* nbits_per_op, const size_t* bits_flat, const double* mats_flat,
                       const size_t* args);
void batch_run(q1g_batch* b, uint64_t* results, size_t len);
// Teams of `size` CTAs, of which `count` run at once; us: each circuit's time on
// one, in queue order.
struct TeamChoice {
    int size = 1, count = 0;
    std::vector<double> us;
};
// alone, able: per circuit in queue order, its time on one CTA and whether a
// team may run it.
TeamPlan plan_teams(const std::vector<double>& alone, const std::vector<char>& able, int sms,
                    const std::vector<TeamChoice>& choices);
// warp-tile layout of a dense op on nbits qubits, gate positions pos[0..tb)
void batch_tile_layout(BatchOp& op, const int* pos, int tb, int nbits);
}  // namespace q1g
