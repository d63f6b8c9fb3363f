// Windowed reference similarity and the identify descent over it.
//
// HVCache::similarity (src/encoder.cpp:198-215) scores a query against a
// reference sequence as the best NORM cosine over the reference's windows
// x = 0, step, 2*step, ... while x + L < len (strict), starting from -1 and
// keeping the first window that beats the running best; a reference no longer
// than one window (len <= L) is scored as one whole-sequence hypervector.
// Every "similarity row" below is one such window (or whole sequence), an
// int16 hypervector of compute semantics (src/encoder.cpp:106-132).
//
// identify (targets/identify.cpp:89-202) scores a taxonomy node for a read as
// max(-1, similarity over every sequence of the node) (:138-159), so with the
// node's rows in CSR (node -> rows of all its sequences) a node's score is
// max(-1, max over its rows).  The level loop is the one of the prototype
// descent in beam.cu: level 0 scores the get_order("p__") nodes, each beam
// entry expands to its children (a node without children to itself, :28-33),
// candidates are ranked by score with ties to the lower node index (the
// reference's std::sort leaves tie order unspecified), the read stops with the
// best path when the best score is below the threshold (:174-189), and
// otherwise keeps the entries scoring >= threshold, at most `beam`
// (:191-199).
//
// One CTA per read here: the read's int16 hypervector is staged in shared memory
// once, and the CTA's warps split each candidate node's rows (coalesced
// 16-byte loads of a row per warp step); dots are exact int64.  Batches of reads
// are grouped by parent on the tensor cores instead (identify_grouped.cu) where
// that is faster (launch_identify), and come back to this kernel at the level
// that does not fit there.
#include <algorithm>

#include "hdc_internal.cuh"
#include "identify.cuh"
#include "topk.cuh"

namespace hdc {
namespace {

constexpr int kMaxBeam = kIdBeam;
constexpr int kMaxLevels = kIdLevels;
constexpr int kIdWarps = 8;
constexpr int kSimWarps = 8;
constexpr int64_t kIdBatch = 65536;  // reads of a grouped pass ...
constexpr int64_t kIdRootPairs = 256 << 20;  // ... and its reads times roots: a pass keeps a word for each (1 GiB)

// exact dot of an int16 row (global) with an int16 vector (shared or global),
// one warp; dim % 8 == 0 and both 16-byte aligned.  NARROW: every partial sum
// fits int32, so the products are accumulated in int32 (two multiply-adds a
// word instead of 64-bit additions).
template <bool NARROW>
__device__ __forceinline__ int64_t warp_dot_i16_t(const int16_t* __restrict__ q, const int16_t* __restrict__ v,
                                                  int dim) {
    const int lane = threadIdx.x & 31;
    const uint4* q4 = reinterpret_cast<const uint4*>(q);
    const uint4* v4 = reinterpret_cast<const uint4*>(v);
    int64_t acc = 0;
    int32_t acc32 = 0;
    for (int i = lane; i < dim / 8; i += 32) {
        const uint4 x = q4[i], y = __ldg(v4 + i);
        const uint32_t xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int32_t xl = (int32_t)(xs[u] << 16) >> 16, xh = (int32_t)xs[u] >> 16;
            const int32_t yl = (int32_t)(ys[u] << 16) >> 16, yh = (int32_t)ys[u] >> 16;
            if (NARROW) {
                acc32 += xl * yl + xh * yh;
            } else {
                acc += (int64_t)(xl * yl) + (int64_t)(xh * yh);  // each product fits int32, their sum may not
            }
        }
    }
    if (NARROW) acc = acc32;
    for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

// Cauchy-Schwarz bounds every partial sum of a dot (any subset of its products) by
// sqrt(|q|^2 |r|^2): below 2^62 for the product of the squared norms, int32 never overflows.
__device__ __forceinline__ bool dot_fits_i32(int64_t nq, int64_t nr) {
    return nq <= 0 || nr <= 0 || nr < ((int64_t)1 << 62) / nq;
}

__device__ __forceinline__ int64_t warp_dot_i16(const int16_t* __restrict__ q, const int16_t* __restrict__ v, int dim,
                                                int64_t nq, int64_t nr) {
    return dot_fits_i32(nq, nr) ? warp_dot_i16_t<true>(q, v, dim) : warp_dot_i16_t<false>(q, v, dim);
}

struct Entry {
    uint64_t key;  // make_key(score, node): larger ranks first
    int32_t node;
    int32_t parent_slot;
};

__global__ void __launch_bounds__(32 * kIdWarps) identify_kernel(const IdentifyArgs a) {
    extern __shared__ __align__(16) int16_t qs[];
    __shared__ int32_t paths[2][kMaxBeam][kMaxLevels];  // level L's beams are read from [L & 1] and the next written to the other
    __shared__ float scores[2][kMaxBeam][kMaxLevels];
    __shared__ Entry top[kMaxBeam];
    __shared__ float wbest[2][kIdWarps];
    __shared__ int n_beam_s, done_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t r = blockIdx.x;
    int first = 0;  // level to start from
    if (a.from.level) {
        first = *a.from.level - 1;
        if (blockIdx.x == 0 && threadIdx.x == 0) *a.form = first + 1;
        if (first < 0 || (first > 0 && a.from.done[r])) return;
    } else if (blockIdx.x == 0 && threadIdx.x == 0) {
        *a.form = HDC_IDENTIFY_PER_READ;
    }
    {
        const uint4* src = reinterpret_cast<const uint4*>(a.q + r * a.dim);
        uint4* dst = reinterpret_cast<uint4*>(qs);
        for (int i = threadIdx.x; i < a.dim / 8; i += blockDim.x) dst[i] = src[i];
    }
    const int64_t qn = a.qn[r];
    // thread 0 owns the ranking state; the others follow the beam through shared memory
    int n_top = 0;
    // the outputs, by thread 0 as soon as the read is done.  Kept in local arrays to the end, as the beams once were, they cost
    // the scoring loop spills: 1,000 reads over 4 x 2,000 nodes, four beam rows, D = 1,024: 70.1 -> 60.8 ms.
    auto write_out = [&](const int32_t* path, const float* score, int depth, int stop_at) {
        a.depth[r] = depth;
        if (a.stop_level) a.stop_level[r] = stop_at;
        for (int l = 0; l < a.levels; ++l) {
            a.path[r * a.levels + l] = l < depth ? path[l] : -1;
            a.path_score[r * a.levels + l] = l < depth ? score[l] : 0.0f;
        }
    };
    if (threadIdx.x == 0) {
        n_beam_s = first > 0 ? a.from.nbeam[r] : 0;
        done_s = 0;
    }
    if (first > 0 && threadIdx.x < kMaxBeam * kMaxLevels) {
        const int b = threadIdx.x / kMaxLevels, l = threadIdx.x % kMaxLevels;
        if (b < a.from.nbeam[r] && l < first) {
            paths[first & 1][b][l] = a.from.paths[(r * kMaxBeam + b) * kMaxLevels + l];
            scores[first & 1][b][l] = a.from.scores[(r * kMaxBeam + b) * kMaxLevels + l];
        }
    }
    __syncthreads();
    int parity = 0;
    for (int L = first; L < a.levels; ++L) {
        n_top = 0;
        const int n_src = L == 0 ? 1 : n_beam_s;
        for (int b = 0; b < n_src; ++b) {
            int64_t c0, c1;
            const int32_t* list;
            int32_t self = -1;
            if (L == 0) {
                list = a.roots;
                c0 = 0;
                c1 = a.n_roots;
            } else {
                const int32_t node = paths[L & 1][b][L - 1];
                c0 = a.child_ptr[node];
                c1 = a.child_ptr[node + 1];
                list = a.child_idx;
                if (c0 == c1) self = node;
            }
            const int64_t cnt = self >= 0 ? 1 : c1 - c0;
            for (int64_t c = 0; c < cnt; ++c) {
                const int32_t node = self >= 0 ? self : list[c0 + c];
                const int64_t r0 = a.node_rows[node], r1 = a.node_rows[node + 1];
                float best = -1.0f;  // identify starts every candidate at -1 (:127)
                for (int64_t j = r0 + warp; j < r1; j += kIdWarps) {
                    const int64_t rn = a.rn[j];
                    const int64_t dot = warp_dot_i16(qs, a.rows + j * a.dim, a.dim, qn, rn);
                    best = fmaxf(best, exact_score(dot, qn, rn, a.mode));
                }
                if (lane == 0) wbest[parity][warp] = best;
                __syncthreads();
                if (threadIdx.x == 0) {
                    float s = -1.0f;
                    for (int w = 0; w < kIdWarps; ++w) s = fmaxf(s, wbest[parity][w]);
                    const uint64_t key = make_key(s, (uint32_t)node);
                    if (n_top < a.beam || key > top[n_top - 1].key) {
                        int pos = n_top < a.beam ? n_top++ : a.beam - 1;
                        while (pos > 0 && top[pos - 1].key < key) {
                            top[pos] = top[pos - 1];
                            --pos;
                        }
                        top[pos] = Entry{key, node, b};
                    }
                }
                parity ^= 1;  // the next candidate writes the other buffer: one barrier per candidate
            }
        }
        if (threadIdx.x == 0) {
            const int old = L & 1, now = old ^ 1;
            for (int t = 0; t < n_top; ++t) {
                for (int l = 0; l < L; ++l) {
                    paths[now][t][l] = paths[old][top[t].parent_slot][l];
                    scores[now][t][l] = scores[old][top[t].parent_slot][l];
                }
                paths[now][t][L] = top[t].node;
                scores[now][t][L] = key_score(top[t].key);
            }
            const int best = n_top ? now : old;
            if (n_top == 0 || (double)key_score(top[0].key) < a.threshold) {
                write_out(paths[best][0], scores[best][0], n_top ? L + 1 : L, L);
                done_s = 1;
            } else {
                int keep = 0;
                while (keep < n_top && keep < a.beam && (double)key_score(top[keep].key) >= a.threshold) ++keep;
                n_beam_s = keep;
                if (L == a.levels - 1) write_out(paths[now][0], scores[now][0], a.levels, -1);
            }
        }
        __syncthreads();
        if (done_s) break;
    }
}

struct SimilarityArgs {
    const int16_t* q;
    const int64_t* qn;
    const int16_t* rows;
    const int64_t* rn;
    const int64_t* ref_rows;  // [n_refs+1] CSR: reference sequence -> its rows, in window order
    const uint8_t* ref_whole; // [n_refs] 1: one whole-sequence row, scored as is (may be null: none)
    const int32_t* pair_q;
    const int32_t* pair_ref;
    int64_t n_pairs;
    int dim, mode;
    float* score;             // [n_pairs]
    int32_t* window;          // [n_pairs] first best row within the reference, -1 if none beat -1
};

// one warp per (query, reference) pair, the reference's windows in order
__global__ void __launch_bounds__(32 * kSimWarps) similarity_kernel(const SimilarityArgs a) {
    const int64_t p = (int64_t)blockIdx.x * kSimWarps + (threadIdx.x >> 5);
    if (p >= a.n_pairs) return;
    const int32_t qi = a.pair_q[p], ri = a.pair_ref[p];
    const int16_t* q = a.q + (int64_t)qi * a.dim;
    const int64_t qn = a.qn[qi];
    const int64_t r0 = a.ref_rows[ri];
    int64_t r1 = a.ref_rows[ri + 1];
    float best = -1.0f;
    int32_t win = -1;
    if (a.ref_whole && a.ref_whole[ri] && r1 > r0) {
        // len <= L: the cosine of the two whole-sequence vectors, unclamped (:200-203)
        best = exact_score(warp_dot_i16(q, a.rows + r0 * a.dim, a.dim, qn, a.rn[r0]), qn, a.rn[r0], a.mode);
        win = 0;
        r1 = r0;
    }
    for (int64_t j = r0; j < r1; ++j) {
        const int64_t rn = a.rn[j];
        const int64_t dot = warp_dot_i16(q, a.rows + j * a.dim, a.dim, qn, rn);
        const float s = exact_score(dot, qn, rn, a.mode);
        if (s > best) {  // strict: the first window reaching the maximum wins (:208-212)
            best = s;
            win = (int32_t)(j - r0);
        }
    }
    if ((threadIdx.x & 31) == 0) {
        a.score[p] = best;
        a.window[p] = win;
    }
}

bool rows_ok(const hdc_context* ctx, const void* q, const void* rows) {
    return ctx->dim % 8 == 0 && !(reinterpret_cast<uintptr_t>(q) & 15) && !(reinterpret_cast<uintptr_t>(rows) & 15);
}

// Microseconds that one CTA a read and the grouped form take, for the choice between them: the one grows with the
// candidates and rows that a read meets, the other is a handful of launches a level however few they are.  The tree's sizes
// give its average branching and rows a node.  As measured on trees of 10 to 1,092 nodes of 1 to 150 rows: a candidate
// takes 1.5 us and 2.5-3.8 for every 8 of its rows (a CTA's warps), D = 1,024-8,192, and beyond a CTA an SM the batch
// some 1 / 700 longer with each read; a grouped level 40 us and 0.55 a K block of 64 dims.  8 reads over 14 nodes of 3 rows,
// beam 1, D = 8,192: 59 us against 267; 152 reads, beam 5, D = 1,024: 66 against 167; 4,096: 388 against 190.
struct IdTimes {
    double per_read, grouped;
};
IdTimes id_times(const hdc_context* ctx, int64_t nq, int64_t n_nodes, int64_t n_rows, int n_roots, int levels, int beam) {
    const double roots = std::max(n_roots, 1), dim = ctx->dim;
    auto nodes_of = [&](double b) {
        double sum = 0, rank = roots;
        for (int l = 0; l < levels; ++l, rank *= b) sum += rank;
        return sum;
    };
    double lo = 1, hi = (double)n_nodes;  // children a node, a childless one counted as its own
    for (int i = 0; i < 50 && levels > 1; ++i) {
        const double b = 0.5 * (lo + hi);
        (nodes_of(b) <= (double)n_nodes ? lo : hi) = b;
    }
    double met = roots, rank = roots;
    for (int l = 1; l < levels; ++l) {
        rank *= lo;
        met += std::min(rank, beam * lo);
    }
    const double eights = std::max<int64_t>(1, (n_rows + 8 * n_nodes - 1) / (8 * n_nodes));
    const double crowd = 1 + (double)std::max<int64_t>(0, nq - ctx->num_sms) / 700;
    return {(15 + met * (1.5 + eights * (2.5 + 1.6e-4 * dim))) * crowd, 20 + levels * (40 + 0.55 / 64 * dim)};
}

}  // namespace

int launch_identify(hdc_context* ctx, const int16_t* d_q, const int64_t* d_qn, int64_t nq, const int16_t* d_rows,
                    const int64_t* d_rn, int64_t n_rows, const int64_t* d_node_rows, int64_t n_nodes,
                    const int64_t* d_child_ptr, const int32_t* d_child_idx, const int32_t* d_roots, int n_roots, int levels, int beam,
                    double threshold, int mode, int32_t* d_path, float* d_path_score, int32_t* d_depth,
                    int32_t* d_stop_level, cudaStream_t stream) {
    if (nq == 0) return HDC_OK;
    if (nq > 0x7fffffffLL) return fail(HDC_ERR_INVALID, "identify: too many reads for one launch");
    if (levels < 1 || levels > kMaxLevels) return fail(HDC_ERR_INVALID, "identify: levels must be in 1..8");
    if (beam < 1 || beam > kMaxBeam) return fail(HDC_ERR_INVALID, "identify: beam width must be in 1..8");
    if (n_roots < 0) return fail(HDC_ERR_INVALID, "identify: negative root count");
    if (!rows_ok(ctx, d_q, d_rows))
        return fail(HDC_ERR_INVALID, "identify: dim must be a multiple of 8 and rows 16-byte aligned");
    const size_t smem = (size_t)ctx->dim * sizeof(int16_t);
    if (smem > 200 * 1024) return fail(HDC_ERR_INVALID, "identify: dim too large for a shared-memory query");
    if (smem > 46 * 1024) {  // with the kernel's own shared memory, more than the 48 KiB that a launch has by default
        cudaError_t e = cudaFuncSetAttribute(identify_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return cuda_fail(e, "identify: shared memory attribute");
    }
    // Batches of reads grouped by parent on the tensor cores, each followed by the per-read kernel, which goes on from the
    // level that does not fit there (and exits at once if all did).  A few reads with one beam row each, a CTA a read, wait
    // as long for their own gathers as for the grouped form's five launches a level: 17 reads, D = 1,024, 233 us against
    // 251; 30, D = 2,048, 291 against 299 (10 reads with three rows each: 865 against 293; without a tree's sizes there is no
    // telling the many that lose from the many that gain: 12 candidates of 150 rows, D = 1,024, 605 against 224, 6 of 3
    // rows 46 against 142).  With them the estimates decide, and in that corner the per-read one may be 2.5 times the
    // other, as it takes every node to have the average's rows and most of them are leaves'.
    bool few = nq <= ctx->num_sms && beam == 1 && ctx->dim <= 2048;
    if (n_nodes > 0) {
        const IdTimes t = id_times(ctx, nq, n_nodes, n_rows, n_roots, levels, beam);
        few = t.per_read <= t.grouped * (few ? 2.5 : 1.0);
    }
    // passes of about as many reads each, in whole items of 128; too many roots even for one item of reads: none
    const int64_t most = std::min(kIdBatch, kIdRootPairs / std::max(n_roots, 1) / 128 * 128);
    const bool grouped = !few && most > 0;
    const int64_t passes = (nq + (grouped ? most : kIdBatch) - 1) / (grouped ? most : kIdBatch);
    const int64_t step = ((nq + passes - 1) / passes + 127) / 128 * 128;
    for (int64_t r0 = 0; r0 < nq; r0 += step) {
        const int64_t n = std::min(step, nq - r0);
        IdentifyArgs a{d_q + r0 * ctx->dim, d_qn + r0, d_rows, d_rn, d_node_rows, d_child_ptr, d_child_idx, d_roots, n_roots,
                       ctx->dim, levels, beam, mode, threshold, d_path + r0 * levels, d_path_score + r0 * levels,
                       d_depth + r0, d_stop_level ? d_stop_level + r0 : nullptr, ctx->d_id_form, {}};
        void* ws = nullptr;
        const int st = grouped ? launch_identify_grouped(ctx, a, n, &a.from, &ws, stream) : HDC_OK;
        if (st != HDC_OK) return st;
        identify_kernel<<<(unsigned)n, 32 * kIdWarps, smem, stream>>>(a);
        cudaError_t e = cudaGetLastError();
        if (ws) cudaFreeAsync(ws, stream);
        if (e != cudaSuccess) return cuda_fail(e, "identify: launch");
    }
    return HDC_OK;
}

int launch_similarity(hdc_context* ctx, const int16_t* d_q, const int64_t* d_qn, const int16_t* d_rows,
                      const int64_t* d_rn, const int64_t* d_ref_rows, const uint8_t* d_ref_whole,
                      const int32_t* d_pair_q,
                      const int32_t* d_pair_ref, int64_t n_pairs, int mode, float* d_score, int32_t* d_window,
                      cudaStream_t stream) {
    if (n_pairs == 0) return HDC_OK;
    if (!rows_ok(ctx, d_q, d_rows))
        return fail(HDC_ERR_INVALID, "similarity: dim must be a multiple of 8 and rows 16-byte aligned");
    const int64_t blocks = (n_pairs + kSimWarps - 1) / kSimWarps;
    if (blocks > 0x7fffffffLL) return fail(HDC_ERR_INVALID, "similarity: too many pairs for one launch");
    SimilarityArgs a{d_q, d_qn, d_rows, d_rn, d_ref_rows, d_ref_whole, d_pair_q, d_pair_ref, n_pairs, ctx->dim, mode, d_score,
                     d_window};
    similarity_kernel<<<(unsigned)blocks, 32 * kSimWarps, 0, stream>>>(a);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? HDC_OK : cuda_fail(e, "similarity: launch");
}

}  // namespace hdc
