// Shared interface of the single-accumulator tensor-core search (search_mm.cu).
#pragma once

#include "hdc_internal.cuh"

namespace hdc {

// Largest squared norms of a set of rows: of whole rows, and of any 64 dims of a K block.
struct alignas(16) MmNorms {
    unsigned long long row, block;
};

// How a search's operands reach the tensor cores.  F16: queries and references as fp16 integers (|v| <= 2048),
// row-major.  F4: +1/0/-1 queries and references split into balanced base-8 digits (-4 .. 4), both as packed e2m1
// in the tile order of mm_pack_*; the digits' weights are the MMA's power-of-two scales.
struct MmOperands {
    bool f4 = false;
    const void* a = nullptr;    // F16: [nq][lda] fp16; F4: mm_pack_queries' tiles
    const void* b = nullptr;    // F16: [nr][ldb] fp16; F4: mm_pack_refs' tiles
    int64_t lda = 0, ldb = 0;   // F16: elements
    int limbs = 1;              // F4: base-8 digits
    int64_t sum_per_dim = 1;    // no partial sum over n dims exceeds n times this
    // Whether a whole dot stays within 2^24 (one segment): known to the host, or decided on the device from the largest
    // squared norms of the rows as they are (not the caller's, which only the scores use), both pointers set (F16).
    bool one_segment = false;
    const MmNorms* q_norms = nullptr;
    const MmNorms* r_norms = nullptr;
    const int64_t* qn = nullptr;
    const float* rr = nullptr;  // references: 1 / sqrt(norm2) in fp32; sqrt(norm2); its reciprocal
    const double* rs = nullptr;
    const double* ri = nullptr;
};

constexpr int kMmQueryTile = 128;  // queries a tile (TMEM lanes)
constexpr int kMmF4Half = 112;     // references of half an F4 tile
constexpr int kMmF4Dims = 128;     // dims of a K block (64 bytes of packed e2m1)
constexpr int64_t kMmMaxSum = (int64_t)1 << 24;  // fp32 holds every integer up to here

// Base-8 digits that hold |v| <= max_abs (0: more than 5).
int mm_f4_limbs(int64_t max_abs);
// F4's sum_per_dim: a value's digits are added from the lowest, and no partial sum of them exceeds this.
int64_t mm_f4_sum_per_dim(int64_t max_abs);
size_t mm_f4_query_bytes(int64_t nq, int dim);
size_t mm_f4_ref_bytes(int64_t nr, int dim, int limbs);
// Whether the accumulators can be emptied often enough (after every MMA at most; digits: every K block).
bool mm_sums_fit(bool f4, int64_t sum_per_dim);

// (a value other than -1, 0, 1 raises *status)
int mm_pack_queries(const void* d_q, bool is_f16, int64_t nq, int dim, void* out, int* status, cudaStream_t stream);
// references from int16 rows, or (limbs16 != null) from a database's fp16 limbs
int mm_pack_refs(const int16_t* d_r, const __half* limbs16, int L16, int bits, int64_t r_pad, int64_t nr, int dim,
                 int limbs, void* out, cudaStream_t stream);
// int16 rows -> fp16 rows of ld elements, zero past dim; *norms = max(*norms, theirs)
int mm_rows_f16(const int16_t* d_v, int64_t n, int dim, int64_t ld, __half* out, MmNorms* norms,
                cudaStream_t stream);
// norms[0] = max(norms[0], those of fp16 integer rows of dim elements, dim % 8 == 0), and norms[1] = other
int mm_norm_max(const __half* d_v, int64_t n, int dim, MmNorms other, MmNorms* norms, cudaStream_t stream);
// F4: the largest |q|^2 |r|^2 at which one segment is exact
double mm_f4_norm_limit(int limbs, int dim);
// the values of a database's limbs as one fp16 row each
int mm_rows_from_limbs(const __half* limbs16, int L16, int bits, int64_t rows, int dim, __half* out,
                       cudaStream_t stream);
// *d_max (cleared by the caller) = the largest |value| of a database's limbs
int mm_limbs_max(const __half* limbs16, int L16, int bits, int64_t rows, int dim, int32_t* d_max, cudaStream_t stream);
// rr, rs, ri of MmOperands from squared norms
int mm_norm_tables(const int64_t* d_n2, int64_t n, float* rr, double* rs, double* ri, cudaStream_t stream);

// A problem of at most one tile a SM: the K loop of a tile split over CTAs, then a selection per query.  splits 0: not
// one (too large, or products whose K block does not fit an accumulator).
struct MmSplit {
    int splits = 0, n_qtiles = 0, n_rtiles = 0, ldd = 0;
};
MmSplit mm_split_plan(const hdc_context* ctx, int64_t nq, int64_t nr, int dim, int k, bool f4, int64_t sum_per_dim);
size_t mm_split_bytes(const MmSplit& p, int64_t nq);
int mm_split_search(hdc_context* ctx, const MmOperands& op, const MmSplit& p, int64_t nq, int64_t nr, int dim, int k,
                    int mode, void* parts, float* d_score, int32_t* d_idx, double* d_cos,
                    int64_t* d_dot, int32_t shape[5], cudaStream_t stream);
// mm_rows_f16 of both operands without their norms, and mm_norm_tables of the references
int mm_rows2_f16(const int16_t* d_q, int64_t nq, const int16_t* d_r, int64_t nr, int dim, int64_t ld, __half* out_q,
                 __half* out_r, const int64_t* d_rn, float* rr, double* rs, double* ri, cudaStream_t stream);

// Workspace of a search's lists for nq queries against nr references (a launch of nr or fewer); its first
// kMmWorkWords 64-bit words are the caller's.
constexpr int kMmWorkWords = 4;
size_t mm_list_bytes(const hdc_context* ctx, int64_t nq, int64_t nr, int dim, int k, bool f4, int limbs);
// Clears the words and the thresholds of nq queries: before the first launch of a call.
int mm_begin(void* work, int64_t nq, cudaStream_t stream);
// Partial top-k lists of nq queries against references r0 .. r0 + nr - 1 (op's tables start at r0).  A later launch of
// a call (first = false) carries the lists on; plan_nr, the largest nr of the call's launches, fixes their layout.
int mm_search(hdc_context* ctx, const MmOperands& op, int64_t nq, int64_t nr, int64_t r0, int64_t plan_nr, int dim, int k,
              int mode, void* work, bool first, int32_t shape[5], cudaStream_t stream);
// The lists of mm_search merged into the outputs.
int mm_finish(hdc_context* ctx, int64_t nq, int64_t plan_nr, int64_t nr_total, int dim, int k, bool f4, int limbs,
              const int64_t* d_qn, const int64_t* d_rn, void* work, float* d_score, int32_t* d_idx, double* d_cos,
              int64_t* d_dot, cudaStream_t stream);

}  // namespace hdc
