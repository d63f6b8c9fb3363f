// identify's descent with the reads of a batch grouped by candidate parent, scored on the tensor cores.
//
// The per-read kernel (identify.cu) reads every row of every candidate node once per read: its bound is those gathers
// from L2 (315 GB for 4,096 reads over a 2,000-leaf tree, 38 ms).  Here a level is scored for the whole batch: the
// entries (read, beam row) that stand at the same parent share one dense product
//     [up to 128 reads] x [up to 192 similarity rows of the parent's children],
// so a row leaves DRAM about once a level and the dots run on tcgen05 (the same batch: 1.98 ms, of which the leaf level's
// 4.4 GB of rows take 1.0).
//
// A level is five kernels: entries are put into a hash table by parent (the call does not know the number of nodes),
// each parent reserves its entries' places and its work items, the entries are scattered, the items scored, and each
// read selects its beam exactly as the per-read kernel does.
//
// Exactness.  Rows and reads are int16; |v| <= 2048 is exact in fp16, and by Cauchy-Schwarz every partial sum of a dot is
// at most |q| |r|, so with |q|^2 |r|^2 <= 2^48 the fp32 accumulator holds exact integers.  Whatever does not fit (a
// larger value or norm, a level with more candidates than the workspace, a wait that ran out) raises a flag on the device
// with the level that it happened in, and the per-read kernel, launched behind, takes the reads on from the beams that the
// level started with; it exits at once otherwise.
#include <cuda_fp16.h>

#include <algorithm>
#include <climits>

#include "hdc_internal.cuh"
#include "identify.cuh"
#include "tc_ptx.cuh"
#include "topk.cuh"

namespace hdc {
namespace {

constexpr int kM = 128;           // entries an item (TMEM lanes)
constexpr int kN = 192;           // rows an item
// Copy warps keep kStagesId K blocks in flight; converter warps, in groups that take every kGroups-th block, turn the
// landed int16 rows into fp16 in place.  They are apart because a converter's fence.proxy.async waits for its thread's
// copies too (with both in one warp a block took 0.5 us whatever the copies' depth).
constexpr int kCopyWarps = 4, kCopyThreads = 32 * kCopyWarps;
constexpr int kGroups = 2, kGroupWarps = 4, kGroupThreads = 32 * kGroupWarps;
constexpr int kConvWarps = kGroups * kGroupWarps;
constexpr int kEpiWarp = kCopyWarps + kConvWarps, kMmaWarp = kEpiWarp + 4;
constexpr int kThreadsId = 32 * (kMmaWarp + 1);
constexpr int kBlockDims = 64, kRowBytes = 2 * kBlockDims, kPieces = kRowBytes / 16;  // K blocks of 128-byte rows
constexpr int kStagesId = 5;
constexpr int kABytes = kM * kRowBytes, kBBytes = kN * kRowBytes, kStageBytesId = kABytes + kBBytes;
constexpr int kRowStep = kGroupThreads / kPieces;            // rows between them
constexpr int kTasksA = kM / kRowStep;                 // the first of them are the entries'
static_assert(kCopyThreads == kGroupThreads && (kM + kN) % kRowStep == 0 && kM % kRowStep == 0, "whole chunks a thread");

constexpr int kMaxChildren = 1 << 25;  // a warp's candidates sum to 2^30 at most

struct Item {
    int32_t slot, e0, n, col0;  // parent's table slot (-1: the roots), first entry and entries, first row
    int32_t kid, skip;          // the child that its rows are counted from, and that child's first row to it
};

struct Level {
    IdentifyArgs a;
    int64_t nq;
    int L;
    double* sq;           // [nq] sqrt of the reads' squared norms, and its reciprocal in fp32
    float* rq;
    int32_t* paths;       // [nq][kIdBeam][kIdLevels]
    float* scores;
    int32_t* nbeam;       // [nq]
    int32_t* done;        // [nq]
    int32_t* depth;       // [nq]
    // entries e = read * beam + row
    int32_t* ent_slot;    // [nq * beam] parent's table slot
    int32_t* ent_rank;    // place among its parent's entries
    int32_t* ent_p0;      // first candidate of the entry in `best`
    int32_t* ent_list;    // entries in parent order
    int32_t* tab_key;     // [table] parent (-1: free)
    int32_t* tab_cnt;
    int32_t* tab_off;
    int64_t table;        // a power of two
    Item* items;
    int64_t max_items;
    uint32_t* best;       // [max_pairs] orderable score of each candidate, 0: nothing yet
    int64_t max_pairs;
    unsigned long long* counters;  // entries, items and pairs of the level (64 bits: what does not fit is still counted)
    int32_t* flag;        // 1: leave this level and the ones after it to the per-read kernel ...
    int32_t* from;        // ... which goes on from level *from - 1 (0: not at all), noted by the level's selection
    int* status;
    long long wait_cycles;
    int withhold;         // test hook: no rows are copied
};
enum { kCntEntries, kCntItems, kCntPairs, kCounters };

__device__ __forceinline__ int64_t at(int64_t r, int b, int l) { return (r * kIdBeam + b) * kIdLevels + l; }

// children of a parent (-1: the roots; a childless node is its own candidate)
__device__ __forceinline__ int n_children(const IdentifyArgs& a, int32_t P) {
    if (P < 0) return a.n_roots;
    const int64_t n = a.child_ptr[P + 1] - a.child_ptr[P];
    return n ? (int)n : 1;
}
__device__ __forceinline__ int32_t child(const IdentifyArgs& a, int32_t P, int j) {
    if (P < 0) return a.roots[j];
    const int64_t c0 = a.child_ptr[P];
    return c0 == a.child_ptr[P + 1] ? P : a.child_idx[c0 + j];
}

__device__ __forceinline__ int64_t child_rows(const IdentifyArgs& a, int32_t P, int j) {
    const int32_t c = child(a, P, j);
    return a.node_rows[c + 1] - a.node_rows[c];
}

// Places for the items of a parent of `rows` rows and m entries: the first, or -1 where they do not fit.
__device__ __forceinline__ int64_t take_items(const Level& v, int64_t rows, int32_t m) {
    const int64_t n = (rows + kN - 1) / kN * ((m + kM - 1) / kM);
    if (n <= v.max_items && rows <= 0x7fffffff) {
        const int64_t x = (int64_t)atomicAdd(v.counters + kCntItems, (unsigned long long)n);
        if (x + n <= v.max_items) return x;
    }
    *v.flag = 1;
    return -1;
}

// The items of the row chunks that start in rows s .. s + m_rows - 1 of a parent, counted from its child j, which begins at
// s; x is the parent's first.  The entry tiles of one chunk stand side by side: they read the same rows at about the same time.
__device__ __forceinline__ void put_items(const Level& v, int64_t x, int32_t slot, int32_t m, int j, int64_t s, int64_t m_rows) {
    const int32_t tiles = (m + kM - 1) / kM;
    for (int64_t c = (s + kN - 1) / kN; c * kN < s + m_rows; ++c)
        for (int32_t t = 0; t < tiles; ++t)
            v.items[x + c * tiles + t] = Item{slot, t * kM, min(kM, m - t * kM), (int32_t)(c * kN), j, (int32_t)(c * kN - s)};
}

// A parent of a few children, by one thread (its items' rows are all counted from the first child) ...
constexpr int kThreadChildren = 32;
__device__ __forceinline__ void add_items(const Level& v, int32_t slot, int32_t P, int32_t m, int nch) {
    int64_t rows = 0;
    for (int j = 0; j < nch; ++j) rows += child_rows(v.a, P, j);
    const int64_t x = take_items(v, rows, m);
    if (x >= 0) put_items(v, x, slot, m, 0, 0, rows);
}

// ... and of many, by a warp, 8 a lane at a time, whose look-ups overlap (a flat tree of 300,000 roots would keep one thread
// for seconds).
constexpr int kLaneChildren = 8;
__device__ __forceinline__ void add_items_wide(const Level& v, int32_t slot, int32_t P, int32_t m, int nch, int lane) {
    int64_t rows = 0;
#pragma unroll 8
    for (int j = lane; j < nch; j += 32) rows += child_rows(v.a, P, j);
    for (int o = 16; o; o >>= 1) rows += __shfl_xor_sync(0xffffffffu, rows, o);
    int64_t x = lane == 0 ? take_items(v, rows, m) : 0;
    x = __shfl_sync(0xffffffffu, x, 0);
    if (x < 0) return;
    int64_t s = 0;
    for (int j0 = 0; j0 < nch; j0 += 32 * kLaneChildren) {
        const int j = j0 + lane * kLaneChildren;
        int64_t r[kLaneChildren], sum = 0;
#pragma unroll
        for (int u = 0; u < kLaneChildren; ++u) r[u] = j + u < nch ? child_rows(v.a, P, j + u) : 0;
#pragma unroll
        for (int u = 0; u < kLaneChildren; ++u) sum += r[u];
        int64_t upto = sum;
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += y;
        }
        int64_t at = s + upto - sum;
#pragma unroll
        for (int u = 0; u < kLaneChildren; ++u) {
            put_items(v, x, slot, m, j + u, at, r[u]);
            at += r[u];
        }
        s += __shfl_sync(0xffffffffu, upto, 31);
    }
}

__global__ void read_norms_kernel(const Level v) {
    const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= v.nq) return;
    v.sq[r] = __dsqrt_rn((double)v.a.qn[r]);
    v.rq[r] = rsqrt_norm(v.a.qn[r]);
}

// entries of the level into the table, their candidates' places
__global__ void entries_kernel(const Level v) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    // once the flag is up the beams are no longer kept; read once a warp, since it may rise meanwhile
    if (__shfl_sync(0xffffffffu, lane == 0 ? *v.flag : 0, 0)) return;
    const int beam = v.a.beam;
    const int64_t r = e / beam;
    const int b = (int)(e % beam);
    const bool on = r < v.nq && !v.done[r] && b < (v.L == 0 ? 1 : v.nbeam[r]);
    if (r < v.nq && !on) v.ent_slot[e] = -2;
    int32_t P = -1;
    int nch = 0;
    if (on) {
        if (v.L > 0) P = v.paths[at(r, b, v.L - 1)];
        nch = n_children(v.a, P);
        if (nch > kMaxChildren) {
            *v.flag = 1;
            nch = 0;
        }
    }
    // the candidates' places: one atomic a warp
    int32_t before = nch;
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, before, o);
        if (lane >= o) before += y;
    }
    const int32_t total = __shfl_sync(0xffffffffu, before, 31);
    before -= nch;
    long long p0 = 0;
    if (lane == 0 && total) p0 = (long long)atomicAdd(v.counters + kCntPairs, (unsigned long long)total);
    p0 = __shfl_sync(0xffffffffu, p0, 0);
    if (p0 + total > v.max_pairs) {
        if (lane == 0) *v.flag = 1;
        return;  // the whole warp
    }
    if (!on) return;
    v.ent_p0[e] = (int32_t)p0 + before;  // (below max_pairs < 2^31)
    for (int j = 0; j < nch; ++j) v.best[p0 + before + j] = 0;
    if (v.L == 0) {
        v.ent_slot[e] = -1;
        return;
    }
    uint32_t h = ((uint32_t)P * 2654435761u) & (uint32_t)(v.table - 1);
    while (true) {  // at most half of the table is taken
        const int32_t k = atomicCAS(v.tab_key + h, -1, P);
        if (k == -1 || k == P) break;
        h = (h + 1) & (uint32_t)(v.table - 1);
    }
    const uint32_t peers = __match_any_sync(__activemask(), (int32_t)h);
    const int leader = __ffs(peers) - 1;
    int32_t rank = 0;
    if (lane == leader) rank = atomicAdd(v.tab_cnt + h, __popc(peers));
    rank = __shfl_sync(peers, rank, leader);
    v.ent_slot[e] = (int32_t)h;
    v.ent_rank[e] = rank + __popc(peers & ((1u << lane) - 1u));
}

// each parent's places in the entry list, and its items; level 0: the roots' (the entries are the reads in order)
__global__ void parents_kernel(const Level v) {
    const int64_t h = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    if (__shfl_sync(0xffffffffu, lane == 0 ? *v.flag : 0, 0)) return;  // (it may rise meanwhile)
    int32_t slot = -1, P = -1, m = 0;
    if (v.L == 0) {
        if (h == 0) m = (int32_t)v.nq;
    } else if (h < v.table) {
        m = v.tab_cnt[h];
        if (m) {
            slot = (int32_t)h;
            P = v.tab_key[h];
            v.tab_off[h] = (int32_t)atomicAdd(v.counters + kCntEntries, (unsigned long long)m);
        }
    }
    const int nch = m ? n_children(v.a, P) : 0;
    const bool wide = nch > kThreadChildren;
    if (m && !wide) add_items(v, slot, P, m, nch);
    __syncwarp();
    for (uint32_t w = __ballot_sync(0xffffffffu, wide); w; w &= w - 1) {
        const int from = __ffs(w) - 1;
        add_items_wide(v, __shfl_sync(0xffffffffu, slot, from), __shfl_sync(0xffffffffu, P, from),
                       __shfl_sync(0xffffffffu, m, from), __shfl_sync(0xffffffffu, nch, from), lane);
    }
}

__global__ void scatter_kernel(const Level v) {
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= v.nq * v.a.beam || *v.flag) return;
    const int32_t s = v.ent_slot[e];
    if (s == -1)
        v.ent_list[e / v.a.beam] = (int32_t)e;
    else if (s >= 0)
        v.ent_list[v.tab_off[s] + v.ent_rank[e]] = (int32_t)e;
}

// ---------------------------------------------------------------- scoring
struct Tables {  // of one item
    const int16_t* row[kM + kN];  // entries' reads, then rows (null: unused)
    double sq[kM];       // sqrt of the reads' squared norms, and its reciprocal in fp32
    float rq[kM];
    int64_t rn[kN];
    float rr[kN + 16];   // 1 / sqrt(norm2), -1 for a zero norm (and room for the last chunk's reads)
    int32_t seg[kN + 1]; // first column of each candidate, then n_cols
    int32_t n_seg;
    int32_t p0[kM];      // entry's first candidate (-1: unused)
    int32_t kid[kN];     // the row's candidate (child) number, -1: unused
    int32_t n_cols, n_ent;
};

struct IdShared {
    uint64_t raw[kStagesId], full[kStagesId], empty[kStagesId], accf[2], acce[2], tabf[2], drain;
    uint32_t tmem;
    int err;
    int n_items;  // read once a CTA: the flag may rise meanwhile, and the roles have to agree
    int64_t norm_max[2][kM / 32];
    Tables tab[2];
};

static_assert(kRowStep % 8 == 0 && kM % 8 == 0 && kABytes == kM * kRowBytes, "rows follow the entries in a stage with the same swizzle phase");

__device__ __forceinline__ void cp_async16(void* dst, const void* src, uint32_t bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(tc::smem_u32(dst)), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 1, %0;" ::"n"(kM) : "memory"); }
__device__ __forceinline__ bool epi_all(bool x) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "bar.red.and.pred q, 1, %2, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}\n"
        : "=r"(r)
        : "r"((uint32_t)x), "n"(kM)
        : "memory");
    return r != 0;
}
// arrive on `bar` when this thread's copies so far have landed
__device__ __forceinline__ void cp_async_arrive(uint64_t* bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// Two int16 values as packed fp16 integers: v + 1536 has the bits 0x6600 + v for -512 <= v < 512, and subtracting 1536
// is exact.  `bad` collects the halves for which that does not hold.
__device__ __forceinline__ uint32_t half2_small(uint32_t x, uint32_t& bad) {
    const uint32_t y = x + 0x66006600u - ((x & 0x8000u) << 1);  // the low half's carry taken back
    bad |= (y ^ 0x64006400u) & 0xfc00fc00u;
    const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&y), __half2half2(__ushort_as_half(0x6600)));
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t half2_any(uint32_t x, bool& out) {
    const int lo = (int)(int16_t)(x & 0xffffu), hi = (int)(int16_t)(x >> 16);
    out |= lo > 2048 || lo < -2048 || hi > 2048 || hi < -2048;
    const __half2 h = __halves2half2(__int2half_rn(lo), __int2half_rn(hi));
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Persistent, one CTA per SM: warps 0-3 copy an item's int16 rows into the swizzled stages (cp.async), warps 4-11 convert
// them in place, warp 16 issues the MMAs (M = 128 entries, N = the rows rounded up to 16), warps 12-15 fill the next
// item's tables and take the accumulators' lanes (entries): per candidate the best estimate over its rows, then one exact
// score.  Two accumulators and two tables: a tile is scored, and the next item's rows are on their way, while another
// runs.
__global__ void __launch_bounds__(kThreadsId, 1) score_tc_kernel(const Level v) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = smem_raw + ((1024 - (tc::smem_u32(smem_raw) & 1023)) & 1023);
    IdShared& sm = *reinterpret_cast<IdShared*>(ring + (size_t)kStagesId * kStageBytesId);
    const IdentifyArgs& a = v.a;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
    volatile int* err = &sm.err;
    if (tid == 0) {
        sm.err = 0;
        sm.n_items = *v.flag ? 0 : (int)v.counters[kCntItems];
        for (int s = 0; s < kStagesId; ++s) {
            tc::mbar_init(&sm.raw[s], kCopyThreads);
            tc::mbar_init(&sm.full[s], kGroupWarps);
            tc::mbar_init(&sm.empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&sm.accf[b], 1);
            tc::mbar_init(&sm.acce[b], 4);
            tc::mbar_init(&sm.tabf[b], kM / 32);
        }
        tc::mbar_init(&sm.drain, 1);
        tc::fence_mbar_init();
    }
    if (warp == kMmaWarp) {
        tc::tmem_alloc(&sm.tmem, 512);
        tc::tmem_relinquish();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = sm.tmem;
    const int n_items = sm.n_items;
    const int n_kb = (a.dim + kBlockDims - 1) / kBlockDims;

    // chunks of a copy or converter thread: 16-byte piece `piece` of rows x0, x0 + kRowStep, ... (an entry's read or a
    // row of the parent), at their place with the 128-byte swizzle (chunk ^= row mod 8; rows kRowStep apart share it)
    const int piece = tid % kPieces, x0 = (tid % kGroupThreads) / kPieces;
    const uint32_t place = (uint32_t)(x0 * kRowBytes + ((piece ^ (x0 & 7)) << 4));

    if (warp < kCopyWarps) {
        int stage = 0;
        uint32_t phase = 0;
        bool ok = !v.withhold;
        int n = 0;  // items so far
        for (int it = blockIdx.x; ok && it < n_items; it += gridDim.x, ++n) {
            const int buf = n & 1;
            if (!tc::mbar_wait(&sm.tabf[buf], (n >> 1) & 1, err, 1, v.wait_cycles)) break;
            const Tables& t = sm.tab[buf];
            const int n_cols = t.n_cols;  // at least 1: an item starts at one of its parent's rows
            const int end_a = (t.n_ent + kRowStep - 1) / kRowStep, end_b = kTasksA + (n_cols + kRowStep - 1) / kRowStep;
            for (int kb = 0; kb < n_kb; ++kb) {
                if (!tc::mbar_wait(&sm.empty[stage], phase ^ 1, err, 2, v.wait_cycles)) {
                    ok = false;
                    break;
                }
                uint8_t* dst = ring + (size_t)stage * kStageBytesId + place;
                const int d0 = kb * kBlockDims + piece * 8;
                const uint32_t bytes = d0 < a.dim ? 16 : 0;  // zeros past dim
                const int off = d0 < a.dim ? d0 : 0;
                // four at a time, their loads before their stores: one after the other each would wait for the last
                auto four = [&](int i0, int end) {
                    const int16_t* p[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) p[u] = i0 + u < end ? t.row[x0 + (i0 + u) * kRowStep] : nullptr;
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (p[u]) cp_async16(dst + (i0 + u) * kRowStep * kRowBytes, p[u] + off, bytes);
                };
                for (int i = 0; i < end_a; i += 4) four(i, end_a);
                for (int i = kTasksA; i < end_b; i += 4) four(i, end_b);
                cp_async_arrive(&sm.raw[stage]);
                if (++stage == kStagesId) {
                    stage = 0;
                    phase ^= 1;
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");  // none left in flight, also when giving up
    } else if (warp < kEpiWarp) {
        const int group = (warp - kCopyWarps) / kGroupWarps;
        uint32_t use = 0;  // K blocks of the items so far: block kb of this one is ring use `use` + kb
        bool ok = true;
        int n = 0;
        for (int it = blockIdx.x; ok && it < n_items; it += gridDim.x, ++n) {
            const int buf = n & 1;
            if (!tc::mbar_wait(&sm.tabf[buf], (n >> 1) & 1, err, 7, v.wait_cycles)) break;
            const int n_cols = sm.tab[buf].n_cols, n_ent = sm.tab[buf].n_ent;
            const int end_a = (n_ent + kRowStep - 1) / kRowStep, end_b = kTasksA + (n_cols + kRowStep - 1) / kRowStep;
            for (int kb = group; kb < n_kb; kb += kGroups) {
                const int stage = (int)((use + kb) % kStagesId);
                if (!tc::mbar_wait(&sm.raw[stage], ((use + kb) / kStagesId) & 1, err, 8, v.wait_cycles)) {
                    ok = false;
                    break;
                }
                uint8_t* dst = ring + (size_t)stage * kStageBytesId + place;
                bool out = false;
                auto four = [&](int i0, int end, int used) {  // rows x0 + i kRowStep >= used are never read by anyone
                    uint4 w[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (i0 + u < end) w[u] = *reinterpret_cast<const uint4*>(dst + (i0 + u) * kRowStep * kRowBytes);
                    uint32_t bad[4];
                    uint4 h[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        bad[u] = 0;
                        h[u] = make_uint4(half2_small(w[u].x, bad[u]), half2_small(w[u].y, bad[u]),
                                          half2_small(w[u].z, bad[u]), half2_small(w[u].w, bad[u]));
                        if (i0 + u >= end || x0 + (i0 + u) * kRowStep >= used) bad[u] = 0;
                    }
                    if (bad[0] | bad[1] | bad[2] | bad[3]) {
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (bad[u])
                                h[u] = make_uint4(half2_any(w[u].x, out), half2_any(w[u].y, out), half2_any(w[u].z, out),
                                                  half2_any(w[u].w, out));
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if (i0 + u < end) *reinterpret_cast<uint4*>(dst + (i0 + u) * kRowStep * kRowBytes) = h[u];
                };
                for (int i = 0; i < end_a; i += 4) four(i, end_a, n_ent);
                for (int i = kTasksA; i < end_b; i += 4) four(i, end_b, kM + n_cols);
                if (out) *v.flag = 1;
                tc::fence_proxy_async();
                __syncwarp();
                if (lane == 0) tc::mbar_arrive(&sm.full[stage]);
            }
            use += (uint32_t)n_kb;
        }
    } else if (warp == kMmaWarp) {
        if (tc::elect_one()) {
            int stage = 0;
            uint32_t phase = 0;
            bool ok = true;
            int n = 0;
            for (int it = blockIdx.x; ok && it < n_items; it += gridDim.x, ++n) {
                const int buf = n & 1;
                if (!tc::mbar_wait(&sm.tabf[buf], (n >> 1) & 1, err, 3, v.wait_cycles)) break;
                const int n_pad = (sm.tab[buf].n_cols + 15) & ~15;
                if (!tc::mbar_wait(&sm.acce[buf], ((n >> 1) & 1) ^ 1, err, 5, v.wait_cycles)) break;
                tc::fence_after();
                const uint32_t idesc = tc::idesc_f16_f32(kM, n_pad), d0 = tmem + (uint32_t)(buf * kN);
                for (int kb = 0; kb < n_kb; ++kb) {
                    if (!tc::mbar_wait(&sm.full[stage], phase, err, 4, v.wait_cycles)) {
                        ok = false;
                        break;
                    }
                    tc::fence_after();
                    const uint32_t sa = tc::smem_u32(ring + (size_t)stage * kStageBytesId);
                    const uint64_t ad = tc::kmajor_desc(sa, 8 * kRowBytes, 2), bd = tc::kmajor_desc(sa + kABytes, 8 * kRowBytes, 2);
#pragma unroll
                    for (int kk = 0; kk < kBlockDims / 16; ++kk)
                        tc::mma_f16(d0, ad + 2 * kk, bd + 2 * kk, idesc, (kb | kk) != 0 ? 1u : 0u);
                    tc::mma_commit(&sm.empty[stage]);
                    if (++stage == kStagesId) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (ok) tc::mma_commit(&sm.accf[buf]);
            }
        }
    } else {
        // These warps also fill an item's tables, one item ahead of the copies: while they wait for an accumulator, and
        // after the tile that used the tables before is scored (so nobody reads them any more).
        const int quarter = warp & 3, row = quarter * 32 + lane;
        auto fill = [&](int it, int buf) {
            epi_sync();
            Tables& t = sm.tab[buf];
            const Item item = v.items[it];
            const int32_t P = item.slot < 0 ? -1 : v.tab_key[item.slot];
            // the item's entries ...
            int32_t first = -1;
            const int16_t* src = nullptr;
            int64_t q_max = 0, r_max = 0;
            double q_sq = 0;
            float q_rq = 0;
            if (row < item.n) {
                const int32_t e = v.ent_list[(item.slot < 0 ? 0 : v.tab_off[item.slot]) + item.e0 + row];
                const int64_t r = e / a.beam;
                first = v.ent_p0[e];
                src = a.q + r * a.dim;
                q_max = a.qn[r];
                q_sq = v.sq[r];
                q_rq = v.rq[r];
            }
            t.p0[row] = first;
            t.row[row] = src;
            t.sq[row] = q_sq;
            t.rq[row] = q_rq;
            // ... and rows: the candidate that holds row item.col0 + c of the parent's
            const int nch = n_children(a, P);
            for (int c = row; c < kN; c += kM) {
                int64_t left = (int64_t)item.skip + c;
                int32_t kid = -1;
                int64_t j = 0;
                for (int i = item.kid; i < nch; ++i) {
                    const int32_t node = child(a, P, i);
                    const int64_t r0 = a.node_rows[node], m = a.node_rows[node + 1] - r0;
                    if (left < m) {
                        kid = i;
                        j = r0 + left;
                        break;
                    }
                    left -= m;
                }
                const int64_t rn = kid >= 0 ? a.rn[j] : 0;
                t.kid[c] = kid;
                t.row[kM + c] = kid >= 0 ? a.rows + j * a.dim : nullptr;
                t.rn[c] = rn;
                t.rr[c] = rn > 0 ? __frsqrt_rn(__ll2float_rn(rn)) : -1.0f;
                r_max = max(r_max, rn);
                if (kid >= 0 && c == kN - 1) t.n_cols = kN;
            }
            for (int o = 16; o; o >>= 1) {
                q_max = max(q_max, __shfl_xor_sync(0xffffffffu, q_max, o));
                r_max = max(r_max, __shfl_xor_sync(0xffffffffu, r_max, o));
            }
            if (lane == 0) {
                sm.norm_max[0][quarter] = q_max;
                sm.norm_max[1][quarter] = r_max;
            }
            epi_sync();
            for (int c = row; c < kN - 1; c += kM)
                if (t.kid[c] >= 0 && t.kid[c + 1] < 0) t.n_cols = c + 1;
            if (quarter == 1) {  // the candidates' first columns, in order
                int n = 0;
                for (int c = lane; c < kN; c += 32) {
                    const bool starts = t.kid[c] >= 0 && (c == 0 || t.kid[c] != t.kid[c - 1]);
                    const uint32_t m = __ballot_sync(0xffffffffu, starts);
                    if (starts) t.seg[n + __popc(m & ((1u << lane) - 1u))] = c;
                    n += __popc(m);
                }
                if (lane == 0) t.n_seg = n;
            }
            if (row == 0) {
                t.n_ent = item.n;
                double m[2] = {0, 0};
                for (int w = 0; w < kM / 32; ++w)
                    for (int i = 0; i < 2; ++i) m[i] = fmax(m[i], (double)sm.norm_max[i][w]);
                if (m[0] * m[1] > 281474976710656.0) *v.flag = 1;  // |q| |r| <= 2^24 for every pair of the item
            }
            epi_sync();
            if (row == 0) t.seg[t.n_seg] = t.n_cols;
            epi_sync();
            if (lane == 0) tc::mbar_arrive(&sm.tabf[buf]);
        };
        if ((int)blockIdx.x < n_items) fill(blockIdx.x, 0);
        int n = 0;
        for (int it = blockIdx.x; it < n_items; it += gridDim.x, ++n) {
            const int buf = n & 1;
            if (it + (int)gridDim.x < n_items) fill(it + gridDim.x, buf ^ 1);
            const Tables& t = sm.tab[buf];
            // given up together: the fill's barriers need all four warps
            if (!epi_all(tc::mbar_wait(&sm.accf[buf], (n >> 1) & 1, err, 6, v.wait_cycles))) break;
            {
                tc::fence_after();
                const uint32_t d0 = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * kN);
                const int32_t p0 = t.p0[row];
                const float rq = t.rq[row];
                const double sq = t.sq[row];
                const bool live = p0 >= 0;
                const bool dots = a.mode == HDC_SCORE_DOT;
                // One candidate's columns at a time.  The estimate is the cosine (NORM is monotone in it), or the dot;
                // a row of zero norm scores -1, which is also where every candidate starts, so it never counts.
                for (int g = 0; g < t.n_seg; ++g) {
                    const int c_end = t.seg[g + 1], kid = t.kid[t.seg[g]];
                    float top = -INFINITY, second = -INFINITY, top_dot = 0;
                    int top_c = 0;
                    for (int c0 = t.seg[g]; c0 < c_end; c0 += 16) {
                        uint32_t w[16];
                        tc::tmem_ld16(d0 + (uint32_t)c0, w);  // past c_end: other columns of the allocation, masked
                        float rr[16];
#pragma unroll
                        for (int u = 0; u < 16; ++u) rr[u] = t.rr[c0 + u];
                        tc::tmem_ld_wait();
#pragma unroll
                        for (int u = 0; u < 16; ++u) {
                            const float dot = __uint_as_float(w[u]);
                            float e = dots ? dot : rr[u] < 0.0f ? -INFINITY : dot * rq * rr[u];
                            e = c0 + u < c_end ? e : -INFINITY;
                            second = fmaxf(second, fminf(top, e));
                            top_dot = e > top ? dot : top_dot;
                            top_c = e > top ? c0 + u : top_c;
                            top = fmaxf(top, e);
                        }
                    }
                    float s = -1.0f;
                    const float floor = top - (dots ? fabsf(top) * 4e-6f + 1.0f : kFilterMargin);
                    const bool some = live && top > -INFINITY;
                    const bool close = some && second >= floor;
                    auto exact = [&](float dot, int c) {
                        if (dots) return __ll2float_rn((int64_t)__float2int_rn(dot));
                        return exact_score_sqrt((int64_t)__float2int_rn(dot), sq, __dsqrt_rn((double)t.rn[c]), a.mode);
                    };
                    if (some) s = fmaxf(s, exact(top_dot, top_c));
                    if (__any_sync(0xffffffffu, close)) {  // another row may score higher: all that could, exactly
                        for (int c = t.seg[g]; c < c_end; ++c) {
                            const float dot = __uint_as_float(tc::tmem_ld1(d0 + (uint32_t)c));
                            tc::tmem_ld_wait();
                            const float e = dots ? dot : t.rr[c] < 0.0f ? -INFINITY : dot * rq * t.rr[c];
                            if (close && e >= floor) s = fmaxf(s, exact(dot, c));
                        }
                    }
                    if (live) atomicMax(v.best + p0 + kid, ord_float(s));
                }
            }
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&sm.acce[buf]);
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == kMmaWarp && *err && tc::elect_one()) tc::mma_drain<false>(&sm.drain);
    if (warp == kMmaWarp) {
        __syncwarp();
        tc::fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
    if (tid == 0 && sm.err) {
        *v.flag = 1;
        atomicCAS(v.status, 0, 100 + sm.err);
    }
}

// ---------------------------------------------------------------- selection
// One warp a read: the rule of the per-read kernel (identify.cu).  Candidates are ranked by key, ties to the earlier one
// (the order that its insertion keeps): `beam` rounds of a warp-wide maximum, each lane following its own candidates.
// The level's counters and table, which it does not read, are cleared here for the next level: as three memsets a level
// they took 70 us of a small call (231 reads, D = 1,024: 346 us).
__global__ void select_kernel(const Level v) {
    const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t r = tid >> 5;
    const int lane = threadIdx.x & 31;
    if (v.L + 1 < v.a.levels) {
        for (int64_t i = tid; i < v.table; i += (int64_t)gridDim.x * blockDim.x) {
            v.tab_cnt[i] = 0;
            v.tab_key[i] = -1;
        }
        if (tid < kCounters) v.counters[tid] = 0;
    }
    if (tid == 0 && *v.flag && *v.from == 0) *v.from = v.L + 1;
    if (r >= v.nq) return;
    if (__shfl_sync(0xffffffffu, lane == 0 ? v.done[r] | *v.flag : 0, 0)) return;
    const IdentifyArgs& a = v.a;
    const int L = v.L;
    const int n_src = L == 0 ? 1 : v.nbeam[r];
    // lane b: beam row b's parent, children and candidates
    int32_t P = -1, p0 = 0, nch = 0;
    if (lane < n_src) {
        if (L > 0) P = v.paths[at(r, lane, L - 1)];
        nch = n_children(a, P);
        p0 = v.ent_p0[r * a.beam + lane];
    }
    uint64_t prev_k = 0, my_k = 0;  // lane t < n_top: entry t of the new beam
    int prev_i = -1, my_slot = 0;
    int32_t my_node = 0;
    int n_top = 0;
    for (int t = 0; t < a.beam; ++t) {
        uint64_t bk = 0;
        int bi = INT_MAX, bslot = 0;
        int32_t bnode = 0;
        int base = 0;
        for (int b = 0; b < n_src; ++b) {
            const int32_t Pb = __shfl_sync(0xffffffffu, P, b), pb = __shfl_sync(0xffffffffu, p0, b);
            const int nb = __shfl_sync(0xffffffffu, nch, b);
            for (int j = lane; j < nb; j += 32) {
                const int32_t c = child(a, Pb, j);
                const uint64_t k = make_key(unord_float(max(v.best[pb + j], ord_float(-1.0f))), (uint32_t)c);
                const int i = base + j;
                const bool after = t == 0 || k < prev_k || (k == prev_k && i > prev_i);  // not taken yet
                if (after && (bi == INT_MAX || k > bk)) {
                    bk = k;
                    bi = i;
                    bslot = b;
                    bnode = c;
                }
            }
            base += nb;
        }
        for (int o = 16; o; o >>= 1) {
            const uint64_t ok = __shfl_xor_sync(0xffffffffu, bk, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o), os = __shfl_xor_sync(0xffffffffu, bslot, o);
            const int32_t on = __shfl_xor_sync(0xffffffffu, bnode, o);
            if (oi != INT_MAX && (bi == INT_MAX || ok > bk || (ok == bk && oi < bi))) {
                bk = ok;
                bi = oi;
                bslot = os;
                bnode = on;
            }
        }
        if (bi == INT_MAX) break;
        if (lane == t) {
            my_k = bk;
            my_slot = bslot;
            my_node = bnode;
        }
        prev_k = bk;
        prev_i = bi;
        ++n_top;
    }
    const float my_s = key_score(my_k);
    const bool stop = n_top == 0 || (double)__shfl_sync(0xffffffffu, my_s, 0) < a.threshold;
    const uint32_t over = __ballot_sync(0xffffffffu, lane < n_top && (double)my_s >= a.threshold);
    const int keep = stop ? (n_top ? 1 : 0) : __ffs(~over) - 1;  // the leading entries that reach the threshold
    // entry t's levels 0 .. L, every old value read before any is written: values lane and lane + 32 of keep x 8
    int32_t np[2];
    float ns[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int t = (lane + 32 * h) / kIdLevels, l = (lane + 32 * h) % kIdLevels;
        const int slot = __shfl_sync(0xffffffffu, my_slot, t);
        np[h] = __shfl_sync(0xffffffffu, my_node, t);
        ns[h] = __shfl_sync(0xffffffffu, my_s, t);
        if (t < keep && l < L) {
            np[h] = v.paths[at(r, slot, l)];
            ns[h] = v.scores[at(r, slot, l)];
        }
    }
    __syncwarp();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int t = (lane + 32 * h) / kIdLevels, l = (lane + 32 * h) % kIdLevels;
        if (t < keep && l <= L) {
            v.paths[at(r, t, l)] = np[h];
            v.scores[at(r, t, l)] = ns[h];
        }
    }
    __syncwarp();
    if (lane == 0) v.nbeam[r] = keep;
    if (stop || L == a.levels - 1) {
        const int depth = stop && !n_top ? L : L + 1;
        if (lane < a.levels) {
            a.path[r * a.levels + lane] = lane < depth ? v.paths[at(r, 0, lane)] : -1;
            a.path_score[r * a.levels + lane] = lane < depth ? v.scores[at(r, 0, lane)] : 0.0f;
        }
        if (lane == 0) {
            v.done[r] = 1;
            a.depth[r] = depth;
            if (a.stop_level) a.stop_level[r] = stop ? L : -1;
        }
    }
}

template <typename T>
T* carve(uint8_t*& cur, int64_t n) {
    T* p = reinterpret_cast<T*>(cur);
    cur += ((size_t)std::max<int64_t>(n, 1) * sizeof(T) + 255) & ~(size_t)255;
    return p;
}

}  // namespace

int launch_identify_grouped(hdc_context* ctx, const IdentifyArgs& args, int64_t nq, IdentifyState* from, void** workspace,
                            cudaStream_t stream) {
    *from = IdentifyState{};
    *workspace = nullptr;
    Level v{};
    v.a = args;
    v.nq = nq;
    v.status = ctx->d_status;
    v.wait_cycles = ctx->wait_cycles > 0 ? ctx->wait_cycles : tc::kWaitCycles;
    v.withhold = ctx->test_withhold_loads == 1;
    const int64_t E = nq * args.beam;
    v.table = 1024;
    while (v.table < 2 * E) v.table *= 2;
    v.max_items = 2 * E + 65536;
    // 32 candidates an entry, and 256 up to 32 MB: beams of a few thousand reads over a genus of hundreds stay grouped
    // (4,096 reads, five beam rows, 4 x 20 x 200 nodes of 20 rows, D = 1,024: 2.1 ms against 128 with the last level per read)
    v.max_pairs = std::max<int64_t>(nq * args.n_roots, std::max<int64_t>(32 * E, std::min<int64_t>(256 * E, 8 << 20))) + 4096;
    if (v.max_pairs > 0x7fffffff - 65536) return HDC_OK;
    auto carve_all = [&](uint8_t* base) {
        uint8_t* cur = base;
        v.flag = carve<int32_t>(cur, 2);
        v.from = v.flag + 1;
        v.counters = carve<unsigned long long>(cur, kCounters);
        v.nbeam = carve<int32_t>(cur, nq);
        v.done = carve<int32_t>(cur, nq);
        v.tab_cnt = carve<int32_t>(cur, v.table);
        v.tab_key = carve<int32_t>(cur, v.table);
        v.tab_off = carve<int32_t>(cur, v.table);
        v.paths = carve<int32_t>(cur, nq * kIdBeam * kIdLevels);
        v.scores = carve<float>(cur, nq * kIdBeam * kIdLevels);
        v.ent_slot = carve<int32_t>(cur, E);
        v.ent_rank = carve<int32_t>(cur, E);
        v.ent_p0 = carve<int32_t>(cur, E);
        v.ent_list = carve<int32_t>(cur, E);
        v.items = carve<Item>(cur, v.max_items);
        v.best = carve<uint32_t>(cur, v.max_pairs);
        v.sq = carve<double>(cur, nq);
        v.rq = carve<float>(cur, nq);
        return (size_t)(cur - base);
    };
    const size_t bytes = carve_all(nullptr);
    uint8_t* ws = nullptr;
    if (scratch_alloc(ctx, reinterpret_cast<void**>(&ws), bytes, stream) != cudaSuccess) {
        cudaGetLastError();
        return HDC_OK;  // no room: the per-read kernel needs none
    }
    carve_all(ws);
    *workspace = ws;
    const size_t smem = 1024 + (size_t)kStagesId * kStageBytesId + sizeof(IdShared);
    cudaError_t e = cudaFuncSetAttribute(score_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)  // flag, counters, nbeam, done
        e = cudaMemsetAsync(ws, 0, (size_t)(reinterpret_cast<uint8_t*>(v.tab_cnt) - ws), stream);
    const unsigned eb = (unsigned)((E + 255) / 256), tb = (unsigned)((v.table + 255) / 256), rb = (unsigned)((nq + 3) / 4);
    if (e == cudaSuccess) read_norms_kernel<<<(unsigned)((nq + 255) / 256), 256, 0, stream>>>(v);
    for (int L = 0; L < args.levels && e == cudaSuccess; ++L) {
        v.L = L;
        entries_kernel<<<eb, 256, 0, stream>>>(v);
        parents_kernel<<<L == 0 ? 1 : tb, 256, 0, stream>>>(v);
        scatter_kernel<<<eb, 256, 0, stream>>>(v);
        score_tc_kernel<<<ctx->num_sms, kThreadsId, smem, stream>>>(v);
        select_kernel<<<rb, 128, 0, stream>>>(v);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        cudaFreeAsync(ws, stream);
        *workspace = nullptr;
        return cuda_fail(e, "identify: grouped launch");
    }
    *from = IdentifyState{v.from, v.done, v.nbeam, v.paths, v.scores};
    return HDC_OK;
}

}  // namespace hdc
