// Arguments shared by the per-read and the grouped identify descent.
#pragma once

#include "hdc_internal.cuh"

namespace hdc {

constexpr int kIdBeam = 8;
constexpr int kIdLevels = 8;

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
    const int32_t* only_if;   // the per-read kernel runs only where this is null or points at a nonzero word
};

// The descent of nq reads grouped by parent.  *flag (in *workspace, which the caller frees on the stream) is nonzero
// afterwards where the per-read kernel has to do the batch instead; null: it was not started.
int launch_identify_grouped(hdc_context* ctx, const IdentifyArgs& args, int64_t nq, int32_t** flag, void** workspace,
                            cudaStream_t stream);

}  // namespace hdc
