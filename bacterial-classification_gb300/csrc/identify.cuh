// Arguments shared by the per-read and the grouped identify descent.
#pragma once

#include "hdc_internal.cuh"

namespace hdc {

constexpr int kIdBeam = 8;
constexpr int kIdLevels = 8;

// The beams that a grouped descent has reached.
struct IdentifyState {
    const int32_t* level;  // 0: it did every level; l + 1: level l and the ones after it are still to be done
    const int32_t* done;   // [nq] reads that have stopped (their outputs are written)
    const int32_t* nbeam;  // [nq]
    const int32_t* paths;  // [nq][kIdBeam][kIdLevels] node and score of each beam row's levels so far
    const float* scores;
};

struct IdentifyArgs {
    const int16_t* q;         // [nq][dim] whole-read hypervectors
    const int64_t* qn;        // [nq]
    const int16_t* rows;      // [n_rows][dim] similarity rows
    const int64_t* rn;        // [n_rows]
    const int64_t* node_rows; // [n_nodes+1] CSR: node -> its rows
    const int64_t* child_ptr;
    const int32_t* child_idx;
    const int32_t* roots;
    int n_roots;
    int dim, levels, beam, mode;
    double threshold;
    int32_t* path;            // [nq][levels]
    float* path_score;        // [nq][levels]
    int32_t* depth;           // [nq]
    int32_t* stop_level;      // [nq] level of an early stop, -1 when all levels ran (may be null)
    int32_t* form;            // how the batch ran (hdc_identify_last_form), written by the per-read kernel
    IdentifyState from;       // of a grouped descent that the per-read kernel finishes
};

// The descent of nq reads grouped by parent; *from is its state (in *workspace, which the caller frees on the stream),
// which says afterwards where the per-read kernel has to go on.  Its level null: it was not started.
int launch_identify_grouped(hdc_context* ctx, const IdentifyArgs& args, int64_t nq, IdentifyState* from, void** workspace,
                            cudaStream_t stream);

}  // namespace hdc
