// Exact top-k search with one fp32 accumulator per (query, reference): a dense Q x R^T contraction on the sm_103a
// tensor cores whose partial sums are moved into integers before any of them could round.
//
// Two operand forms (MmOperands):
//   * F16 (kind::f16): integers of magnitude <= 2048 are exact in fp16, whatever their number of digits elsewhere;
//   * F4 (kind::mxf4): +1/0/-1 queries against references split into balanced base-8 digits -4 .. 4, which e2m1
//     holds exactly.  The digits of one value lie one after the other along K and the MMA's block scale (2^(3 l), a
//     power of two in ue8m0) gives each its weight, so all digits of a tile add into the same accumulator.  A digit
//     costs a quarter of an fp16 limb's tensor time and bytes; 4 digits hold |v| <= 2340, 5 hold 18,724.
//
// Exactness.  fp32 adds integers exactly while every partial sum stays within 2^24.  By Cauchy-Schwarz no partial sum of
// a dot exceeds |q| |r|, so one accumulator holds a whole dot wherever the largest norms (of the rows themselves) allow
// it, as encoded reads and references do by far (D = 8,192: 3.8e6 for a 150 bp read and a 1,500 bp sequence).  Otherwise
// the K loop runs in segments, each in a fresh accumulator that the drain warps add to int32 registers while the next one
// fills: of as many K blocks as the same inequality on the largest norms of 64 dims allows, or at least of 2^24 /
// sum_per_dim dims (the largest |q| times the largest |r|), down to one MMA.  Count-valued reads of 250 bp against
// references bundled of eight sequences, 4,000 x 50,000 at D = 10,240: six segments, 2.5 ms (1,626 TFLOP/s); a segment a
// K block as the values alone have it 11.3 ms; three exact limbs of the smaller base they need 10.8 ms.
//
// Kernel (one CTA per SM, persistent, 4 warpgroups with their registers redistributed by setmaxnreg):
//   * warp 0 TMA producer, warp 1 MMA issuer;
//   * warps 4-11 drain: each adds its half of a tile's columns of 32 rows to int32 registers (at most 128 a thread)
//     segment by segment, filters the finished dots by an fp32 estimate of their scores, and passes the few that can
//     enter the row's list to its scorer through a ring in shared memory;
//   * warps 12-15 score: one thread a query computes the exact FP64 scores and keeps the list.
// Drain and scoring are apart because a segment lasts only some thousand cycles, about as long as one exact score with
// its insertion: with both in one warp the MMAs waited for the accumulator (measured 955 TFLOP/s on count-valued
// queries and 1,368 at top-10 on +1/-1 queries).
// Pairs (CL = 2): one cta_group::2 MMA over two query tiles, each CTA staging half of the reference tile's rows.
// Single CTAs (CL = 1) with narrow reference tiles serve batches too small to give every pair a tile.
//
// Problems of at most a tile a SM go to mm_dots_kernel and mm_select_kernel below.
//
// What bounds it: the tensor pipe for large batches (10,000 x 50,000 count-valued reads, D = 8,192: 514 cycles a K block of
// 512); the reference bytes for a few queries.
#include <cuda.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <numeric>

#include "search_mm.cuh"
#include "tc_ptx.cuh"
#include "topk.cuh"

namespace hdc {
namespace {

constexpr int kThreadsMm = 512;  // 4 warpgroups: loads and MMA issue, two of drain warps, scorers
constexpr int kDrainWarps = 8;
// Registers a thread of each warpgroup: the launch's 128 redistributed (64 + 2 x 176 + 96 = 4 x 128).
constexpr int kRegsLoad = 64, kRegsDrain = 176, kRegsScore = 96;
constexpr int kRing = 8;  // candidates a row and half may have waiting for their scorer
constexpr int kSlack = 3;  // columns of a row beyond k that a tile may pass without a closer threshold
constexpr int kMaxKMm = 32;
constexpr int kMaxStages = 12;
constexpr int kMaxF4Limbs = 5;
constexpr size_t kMaxDynSmemMm = 225 * 1024;
constexpr uint32_t kScaleCol = 480;  // F4: 4 x 8 TMEM columns of block scales 8^0 .. 8^3

struct MmArgs {
    int64_t nq, nr, r0;
    int k, mode, limbs;
    int n_kb, kb_per_seg;  // K blocks of a tile, and of a segment
    int mma_per_seg;       // F16: MMAs of a segment where a K block's four sum to too much (1 or 2, else 0)
    const MmNorms* q_norms;  // largest squared norms of the queries and references (null: not used)
    const MmNorms* r_norms;
    int n_qtiles, n_rtiles, G, S, n_groups, t_stride;
    double norm_limit;
    int stages;
    int carry;             // the lists of a previous launch go on
    int withhold;          // test hook: the producer issues no loads
    const int64_t* qn;
    const float* rr;
    const double* rs;
    const double* ri;
    uint64_t* ws_key;      // [S][nq][k]
    int64_t* ws_dot;
    uint32_t* kth;         // [nq] the best k-th score of any full list so far (orderable), cleared by the call
    int* status;
    long long wait_cycles;
};

// The operand forms' tile geometry: N references a tile (N / CL rows staged by each CTA), K blocks of ROWB-byte rows.
template <bool F4, int CL>
struct MmTile {
    static constexpr int N = F4 ? (CL == 1 ? kMmF4Half : 2 * kMmF4Half) : (CL == 1 ? 64 : 256);
    static constexpr int ROWS = N / CL;
    static constexpr int ROWB = F4 ? 64 : 128;
    static constexpr int A_BYTES = kMmQueryTile * ROWB;
    static constexpr int B_BYTES = ROWS * ROWB;  // per limb
    static constexpr uint32_t SBO = 8 * ROWB;
    static constexpr uint32_t LAYOUT = F4 ? 4u : 2u;
    static constexpr int NCH = N / 16;               // 16-column chunks
    static constexpr int NCH2 = (NCH + 1) / 2;        // of one epilogue warp
};

__host__ __device__ constexpr int mm_stage_bytes(int a_bytes, int b_bytes, int limbs) { return a_bytes + limbs * b_bytes; }

// Insert (key, dot) into a descending list of k <= KR keys in registers, dropping the last entry, and return the new
// last key.  The dots live in k slots a row's distance apart; nibble i of `slots` is the slot of entry i, and the entry
// that drops out hands its slot to the new dot.  Every index is a compile-time constant after unrolling.
template <int KR>
__device__ __forceinline__ uint64_t mm_insert(uint64_t (&keys)[KR], uint64_t& slots, int k, uint64_t key, int32_t dot,
                                              int32_t* dots) {
    int pos = 0;
#pragma unroll
    for (int i = 0; i < KR - 1; ++i) pos += (i < k - 1 && keys[i] > key) ? 1 : 0;
#pragma unroll
    for (int i = KR - 1; i >= 0; --i) {
        const uint64_t prev = i > 0 ? keys[i > 0 ? i - 1 : 0] : 0;
        const uint64_t sh = 0ull - (uint64_t)(i > pos && i < k);
        const uint64_t at = 0ull - (uint64_t)(i == pos);
        keys[i] = (keys[i] & ~(sh | at)) | (prev & sh) | (key & at);
    }
    const uint64_t freed = (slots >> (4 * (k - 1))) & 15u;
    const uint64_t below = (1ull << (4 * pos)) - 1;
    const uint64_t thru = pos >= 15 ? ~0ull : (1ull << (4 * pos + 4)) - 1;
    const uint64_t upto = k >= 16 ? ~0ull : (1ull << (4 * k)) - 1;
    slots = (slots & below) | (freed << (4 * pos)) | ((slots << 4) & upto & ~thru) | (slots & ~upto);
    dots[(int)freed * kMmQueryTile] = dot;
    uint64_t last = 0;
#pragma unroll
    for (int i = 0; i < KR; ++i) last |= keys[i] & (0ull - (uint64_t)(i == k - 1));
    return last;
}

// The same for a list in shared memory, entry i a row's distance after entry i - 1.
__device__ __forceinline__ uint64_t mm_insert_shared(uint64_t* keys, int32_t* dots, int k, uint64_t key, int32_t dot) {
    int pos = k - 1;
    while (pos > 0 && keys[(pos - 1) * kMmQueryTile] < key) {
        keys[pos * kMmQueryTile] = keys[(pos - 1) * kMmQueryTile];
        dots[pos * kMmQueryTile] = dots[(pos - 1) * kMmQueryTile];
        --pos;
    }
    keys[pos * kMmQueryTile] = key;
    dots[pos * kMmQueryTile] = dot;
    return keys[(k - 1) * kMmQueryTile];
}

// The estimate that any score able to beat sk reaches (see kFilterMargin; DOT estimates are within a relative 4e-6
// plus one unit).
__device__ __forceinline__ float mm_filter_below(float sk, int mode) {
    return mode == HDC_SCORE_DOT ? sk - (fabsf(sk) * 4e-6f + 1.0f) : sk - kFilterMargin;
}

// A word that one thread of the CTA hands to another, ordered after (before) what it guards.
__device__ __forceinline__ void st_release_shared(uint32_t* p, uint32_t v) {
    asm volatile("st.release.cta.shared.u32 [%0], %1;" ::"r"(tc::smem_u32(p)), "r"(v) : "memory");
}
__device__ __forceinline__ uint32_t ld_acquire_shared(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.cta.shared.u32 %0, [%1];" : "=r"(v) : "r"(tc::smem_u32(p)) : "memory");
    return v;
}

template <int R>
__device__ __forceinline__ void regs_up() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R>
__device__ __forceinline__ void regs_down() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}

// Shared state between a row's drain threads and its scorer.
struct MmShared {
    // candidates (dot, reference) of a row from each half: rings of kRing, head written by the drain thread, tail by
    // the scorer
    int2 ring[2][kRing][kMmQueryTile];
    uint32_t head[2][kMmQueryTile], tail[2][kMmQueryTile];
    // (group << 32 | bits of the threshold) as the scorer last knew it
    volatile unsigned long long thr[kMmQueryTile];
    volatile uint32_t beat;  // tiles drained so far by some warp: a scorer's wait restarts when it moves
};
constexpr uint32_t kFlush = 0xffffffffu;  // in a candidate's reference: the group's columns are all drained

// sum += x + kAddWhole (modulo 2^32), for a whole |x| <= 2^24, in three float adds, one integer multiply-add and one
// integer add: x + 1.5 * 2^34 rounds x to a multiple of 2^11, whose quotient and remainder are then read off the bits
// below an exponent.  A segment's drain is bound by conversions at 16 a cycle and SM; with every other one made so, the
// two pipes share them (4,000 x 20,000 queries and references of magnitude 100 and 2,000, D = 8,192, a segment a K
// block: 4.40 -> 3.72 ms).
constexpr uint32_t kAddWhole = 0x50C00000u * 2048u + 0x4B400000u;
__device__ __forceinline__ void add_whole(int32_t& sum, float x) {
    const float high = __fadd_rn(x, 25769803776.0f);                         // 0x50C00000 = 1.5 * 2^34
    const float low = __fsub_rn(x, __fsub_rn(high, 25769803776.0f + 12582912.0f));  // remainder + 0x4B400000 = 1.5 * 2^23
    sum = (int32_t)((uint32_t)sum + __float_as_uint(high) * 2048u + __float_as_uint(low));
}

// KR: a list's keys in KR registers (k <= KR) with its dots in shared memory; 0: lists in shared memory.
template <bool F4, int CL, int KR>
__global__ void __launch_bounds__(kThreadsMm, 1)
    mm_search_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const MmArgs a) {
    using T = MmTile<F4, CL>;
    constexpr int BN = T::N;
    constexpr bool PAIR = CL == 2;
    constexpr uint32_t IDESC = F4 ? tc::idesc_f4_f32(CL * kMmQueryTile, BN) : tc::idesc_f16_f32(CL * kMmQueryTile, BN);
    static_assert(2 * BN <= (F4 ? (int)kScaleCol : 512), "accumulators exceed TMEM");

    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = smem_raw + ((1024 - (tc::smem_u32(smem_raw) & 1023)) & 1023);
    __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], accf_bar[2], acce_bar[2], drain_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int err_s;
    __shared__ int seg_s[2];  // K blocks of a segment; MMAs of one, where less than a K block
    const int stages = a.stages;
    const uint32_t stage_bytes = (uint32_t)mm_stage_bytes(T::A_BYTES, T::B_BYTES, a.limbs);
    MmShared& sh = *reinterpret_cast<MmShared*>(ring + (size_t)stages * stage_bytes);
    uint8_t* lists_s = reinterpret_cast<uint8_t*>(&sh + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        err_s = 0;
        sh.beat = 0;
        for (int s = 0; s < stages; ++s) {
            tc::mbar_init(&full_bar[s], 1);
            tc::mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&accf_bar[b], 1);
            tc::mbar_init(&acce_bar[b], kDrainWarps * CL);  // each drain warp of the MMA's CTAs
        }
        tc::mbar_init(&drain_bar, 1);
        tc::fence_mbar_init();
        tc::prefetch_tmap(&tmA);
        tc::prefetch_tmap(&tmB);
    }
    if (threadIdx.x == kThreadsMm - 1) {  // (a warp that sets nothing else up)
        // One segment when the norms allow it: no partial sum of a dot, over whatever dims, exceeds |q| |r|
        // (Cauchy-Schwarz).  Otherwise as many K blocks a segment as theirs allow: m of them sum to at most m |q_b| |r_b|.
        int kbs = a.kb_per_seg, mmas = a.mma_per_seg;
        if (a.q_norms) {
            if ((double)a.q_norms->row * (double)a.r_norms->row <= a.norm_limit) {
                kbs = a.n_kb;
                mmas = 0;
            } else if (!F4 && a.q_norms->block && a.r_norms->block) {
                const double b = (double)a.q_norms->block * (double)a.r_norms->block;
                const double room = (double)kMmMaxSum * (double)kMmMaxSum * (1 - 1e-9);  // (products are rounded)
                int m = min(a.n_kb, (int)(kMmMaxSum * rsqrtf((float)b)) + 1);
                while (m > 0 && (double)m * m * b > room) --m;
                if (m > (mmas ? 0 : kbs)) {
                    const int n = (a.n_kb + m - 1) / m;
                    kbs = (a.n_kb + n - 1) / n;  // of even length
                    mmas = 0;
                }
            }
        }
        seg_s[0] = kbs;
        seg_s[1] = mmas;
    }
    if (threadIdx.x < kMmQueryTile) {
        for (int h = 0; h < 2; ++h) sh.head[h][threadIdx.x] = sh.tail[h][threadIdx.x] = 0;
        sh.thr[threadIdx.x] = ~0ull;  // of no group
    }
    if (warp == 1) {
        if constexpr (PAIR) {
            tc::tmem_alloc_pair(&tmem_base_s, 512);
            tc::tmem_relinquish_pair();
        } else {
            tc::tmem_alloc(&tmem_base_s, 512);
            tc::tmem_relinquish();
        }
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_base_s;
    if constexpr (F4) {
        // every byte of 8 columns the same scale 2^(3 i), in all lanes: whatever row or 32-dim block the MMA looks up
        if (warp < 4) {
            uint32_t v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0x01010101u * (uint32_t)(127 + 3 * (i / 8));
            tc::tmem_st32(tmem + ((uint32_t)(warp * 32) << 16) + kScaleCol, v);
            tc::tmem_st_wait();
        }
        tc::fence_before();
        __syncthreads();
        tc::fence_after();
    }
    if constexpr (PAIR) tc::cluster_sync();  // the peer's barriers and scales exist before anything uses them
    const int kb_per_seg = seg_s[0], mma_per_seg = F4 ? 0 : seg_s[1];
    const int n_segs = mma_per_seg ? a.n_kb * (4 / mma_per_seg) : (a.n_kb + kb_per_seg - 1) / kb_per_seg;
    const int crank = PAIR ? (int)tc::cluster_ctarank() : 0;
    const int gslot = (int)(blockIdx.x % a.G), lane_j = (int)(blockIdx.x / a.G);
    const int lead_slot = gslot & ~(CL - 1);  // a pair takes part in a group when its first CTA has a query tile

    if (warp < 4) {
        regs_down<kRegsLoad>();
        if (warp == 0 && tc::elect_one()) {
            // -------------------------------------------- TMA producer
            int stage = 0;
            uint32_t phase = 0;
            int64_t issued = 0;
            bool ok = true;
            for (int grp = 0; ok && !a.withhold && grp < a.n_groups; ++grp) {
                if (grp * a.G + lead_slot >= a.n_qtiles) continue;
                const int qt = min(grp * a.G + gslot, a.n_qtiles - 1);
                for (int t0 = lane_j; ok && t0 < a.n_rtiles; t0 += a.S) {
                    const int t = (int)((int64_t)t0 * a.t_stride % a.n_rtiles);
                    for (int kb = 0; kb < a.n_kb; ++kb) {
                        if (!tc::mbar_wait(&empty_bar[stage], phase ^ 1, &err_s, 1, a.wait_cycles)) {
                            ok = false;
                            break;
                        }
                        uint8_t* st = ring + (size_t)stage * stage_bytes;
                        // the bytes of both CTAs of a pair complete on the even CTA's barrier, where its MMA waits
                        if (!PAIR || crank == 0) tc::mbar_arrive_expect_tx(&full_bar[stage], CL * stage_bytes);
                        const uint32_t fb = PAIR ? tc::cluster_addr(&full_bar[stage], 0) : 0;
                        auto load = [&](void* dst, const CUtensorMap* map, int x, int y) {
                            if constexpr (PAIR)
                                tc::tma_load_2d_pair(dst, map, fb, x, y);
                            else
                                tc::tma_load_2d(dst, map, &full_bar[stage], x, y);
                        };
                        if constexpr (F4) {
                            load(st, &tmA, 0, (qt * a.n_kb + kb) * kMmQueryTile);
                            const int tile = PAIR ? t : t >> 1, half = PAIR ? crank : t & 1;
                            const int y = ((tile * a.n_kb + kb) * 2 + half) * a.limbs * kMmF4Half;
                            for (int l = 0; l < a.limbs; ++l)
                                load(st + T::A_BYTES + l * T::B_BYTES, &tmB, 0, y + l * kMmF4Half);
                        } else {
                            load(st, &tmA, kb * 64, qt * kMmQueryTile);
                            load(st + T::A_BYTES, &tmB, kb * 64, t * BN + crank * T::ROWS);
                        }
                        ++issued;
                        if (++stage == stages) {
                            stage = 0;
                            phase ^= 1;
                        }
                    }
                }
            }
            // before leaving, let the last loads land (bounded): their stages' commits come after them
            int s = stage;
            uint32_t ph = phase;
            for (int64_t i = 0; i < (issued < stages ? issued : (int64_t)stages); ++i) {
                if (--s < 0) {
                    s = stages - 1;
                    ph ^= 1;
                }
                uint64_t* bar = PAIR ? &empty_bar[s] : &full_bar[s];
                const long long c0 = clock64();
                while (!tc::mbar_try_wait(tc::smem_u32(bar), ph) && clock64() - c0 < tc::kWaitCycles) {
                }
            }
        } else if (warp == 1 && crank == 0 && tc::elect_one()) {
            // -------------------------------------------- MMA issuer (the even CTA's, in a pair)
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            int64_t segs = 0;
            auto acc_free = [&]() {  // the next accumulator is drained
                const bool got = PAIR ? tc::mbar_wait_cluster(&acce_bar[acc], acc_phase ^ 1, &err_s, 2, a.wait_cycles)
                                      : tc::mbar_wait(&acce_bar[acc], acc_phase ^ 1, &err_s, 2, a.wait_cycles);
                tc::fence_after();
                return got;
            };
            auto acc_done = [&]() {
                if constexpr (PAIR)
                    tc::mma_commit_pair_mc(&accf_bar[acc], 3);
                else
                    tc::mma_commit(&accf_bar[acc]);
                ++segs;
                if (++acc == 2) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            };
            auto stage_done = [&]() {
                if constexpr (PAIR)
                    tc::mma_commit_pair_mc(&empty_bar[stage], 3);
                else
                    tc::mma_commit(&empty_bar[stage]);
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1;
                }
            };
            auto mma16 = [&](uint32_t d0, uint64_t adesc, uint64_t bdesc, uint32_t on) {  // K = 16 fp16 = 32 bytes
                if constexpr (PAIR)
                    tc::mma_f16_pair(d0, adesc, bdesc, IDESC, on);
                else
                    tc::mma_f16(d0, adesc, bdesc, IDESC, on);
            };
            for (int grp = 0; ok && grp < a.n_groups; ++grp) {
                if (grp * a.G + lead_slot >= a.n_qtiles) continue;
                for (int t0 = lane_j; ok && t0 < a.n_rtiles; t0 += a.S) {
                    for (int kb = 0; mma_per_seg && ok && kb < a.n_kb; ++kb) {
                        if (!(ok = tc::mbar_wait(&full_bar[stage], phase, &err_s, 3, a.wait_cycles))) break;
                        tc::fence_after();
                        const uint32_t sa = tc::smem_u32(ring + (size_t)stage * stage_bytes);
                        const uint64_t adesc = tc::kmajor_desc(sa, T::SBO, T::LAYOUT);
                        const uint64_t bdesc = tc::kmajor_desc(sa + (uint32_t)T::A_BYTES, T::SBO, T::LAYOUT);
                        for (int kk = 0; ok && kk < 4; kk += mma_per_seg) {
                            if (!(ok = acc_free())) break;
                            const uint32_t d0 = tmem + (uint32_t)(acc * BN);
                            for (int j = 0; j < mma_per_seg; ++j)
                                mma16(d0, adesc + 2 * (kk + j), bdesc + 2 * (kk + j), j ? 1u : 0u);
                            acc_done();
                        }
                        if (ok) stage_done();
                    }
                    for (int k0 = 0; !mma_per_seg && ok && k0 < a.n_kb; k0 += kb_per_seg) {
                        if (!(ok = acc_free())) break;
                        const uint32_t d0 = tmem + (uint32_t)(acc * BN);
                        const int k1 = min(k0 + kb_per_seg, a.n_kb);
                        for (int kb = k0; kb < k1; ++kb) {
                            if (!tc::mbar_wait(&full_bar[stage], phase, &err_s, 3, a.wait_cycles)) {
                                ok = false;
                                break;
                            }
                            tc::fence_after();
                            const uint32_t sa = tc::smem_u32(ring + (size_t)stage * stage_bytes);
                            const uint64_t adesc = tc::kmajor_desc(sa, T::SBO, T::LAYOUT);
                            const uint64_t bdesc = tc::kmajor_desc(sa + (uint32_t)T::A_BYTES, T::SBO, T::LAYOUT);
                            if constexpr (F4) {
                                for (int l = 0; l < a.limbs; ++l) {
                                    // weight 8^l as the product of the operands' scales (8^4 = 8 * 8^3)
                                    const uint32_t sfa = tmem + kScaleCol + (l == 4 ? 8u : 0u);
                                    const uint32_t sfb = tmem + kScaleCol + 8u * (uint32_t)(l == 4 ? 3 : l);
                                    const uint64_t bl = bdesc + (uint64_t)(l * (T::B_BYTES >> 4));
#pragma unroll
                                    for (int kk = 0; kk < 2; ++kk) {  // K = 64 e2m1 per MMA = 32 bytes
                                        const uint32_t on = (kb - k0) | l | kk ? 1u : 0u;
                                        if constexpr (PAIR)
                                            tc::mma_f4_pair(d0, adesc + 2 * kk, bl + 2 * kk, IDESC, sfa, sfb, on);
                                        else
                                            tc::mma_f4(d0, adesc + 2 * kk, bl + 2 * kk, IDESC, sfa, sfb, on);
                                    }
                                }
                            } else {
#pragma unroll
                                for (int kk = 0; kk < 4; ++kk)
                                    mma16(d0, adesc + 2 * kk, bdesc + 2 * kk, (kb - k0) | kk ? 1u : 0u);
                            }
                            stage_done();
                        }
                        if (!ok) break;
                        acc_done();
                    }
                }
            }
            if constexpr (PAIR) {
                // the odd CTA's drain warps arrive on this CTA's barriers: let the last
                // arrivals land before the CTA can leave (bounded)
                for (int64_t i = 0; i < (segs < 2 ? segs : (int64_t)2); ++i) {
                    const long long c0 = clock64();
                    while (!tc::mbar_try_wait_cluster(tc::smem_u32(&acce_bar[acc]), acc_phase ^ 1) &&
                           clock64() - c0 < tc::kWaitCycles) {
                    }
                    if (++acc == 2) {
                        acc = 0;
                        acc_phase ^= 1;
                    }
                }
            }
        }
    } else if (warp < 4 + kDrainWarps) {
        // ------------------------------------------------ drain and filter: warps 4..11
        regs_up<kRegsDrain>();
        const int quarter = warp & 3;    // TMEM lane quarter this warp may access
        const int half = (warp - 4) >> 2;  // its half of a tile's columns
        const int row = quarter * 32 + lane;
        const int n_chunks = half ? T::NCH - T::NCH2 : T::NCH2;
        const uint32_t col_addr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * T::NCH2 * 16);
        const bool multi = n_segs > 1;
        const int k = a.k;
        int acc = 0;
        uint32_t acc_phase = 0;
        uint32_t head = 0;
        bool ok = true;
        // hand a candidate to the row's scorer; waits (bounded) while its ring is full
        auto push = [&](int32_t dot, uint32_t ref) {
            if (head - ld_acquire_shared(&sh.tail[half][row]) >= (uint32_t)kRing) {
                const long long c0 = clock64();
                while (head - ld_acquire_shared(&sh.tail[half][row]) >= (uint32_t)kRing) {
                    if (err_s) return;
                    if (clock64() - c0 > a.wait_cycles) {
                        atomicCAS(const_cast<int*>(&err_s), 0, 5);
                        return;
                    }
                }
            }
            sh.ring[half][head % kRing][row] = make_int2(dot, (int)ref);
            st_release_shared(&sh.head[half][row], ++head);
        };
        auto release = [&]() {  // this warp is done with the accumulator
            tc::fence_before();
            __syncwarp();
            if (lane == 0) {
                if (!PAIR || crank == 0)
                    tc::mbar_arrive(&acce_bar[acc]);
                else
                    tc::mbar_arrive_cluster(tc::cluster_addr(&acce_bar[acc], 0));
            }
            if (++acc == 2) {
                acc = 0;
                acc_phase ^= 1;
            }
        };
        for (int grp = 0; ok && grp < a.n_groups; ++grp) {
            if (grp * a.G + lead_slot >= a.n_qtiles) continue;
            const int64_t gq = (int64_t)(grp * a.G + gslot) * kMmQueryTile + row;
            const bool live = gq < a.nq;
            const float my_rq = rsqrt_norm(live ? a.qn[gq] : 0);
            float thr = -INFINITY;
            for (int t0 = lane_j; t0 < a.n_rtiles; t0 += a.S) {
                const int t = (int)((int64_t)t0 * a.t_stride % a.n_rtiles);
                uint32_t d0 = 0;  // this warp's columns of the finished tile
                if (multi) {
                    // segment by segment into registers, then back to TMEM as whole numbers
                    int32_t sum[T::NCH2][16];
#pragma unroll
                    for (int i = 0; i < T::NCH2; ++i)
#pragma unroll
                        for (int c = 0; c < 16; ++c) sum[i][c] = 0;
                    for (int s = 0; s < n_segs; ++s) {
                        if (!tc::mbar_wait(&accf_bar[acc], acc_phase, &err_s, 4, a.wait_cycles)) {
                            ok = false;
                            break;
                        }
                        tc::fence_after();
                        d0 = col_addr + (uint32_t)(acc * BN);
                        uint32_t v[2][16];  // the next chunk is on its way while one is added
                        tc::tmem_ld16(d0, v[0]);
#pragma unroll
                        for (int i = 0; i < T::NCH2; ++i) {
                            tc::tmem_ld_wait();
                            if (i + 1 < T::NCH2) tc::tmem_ld16(d0 + 16u * (i + 1), v[(i + 1) & 1]);
#pragma unroll
                            for (int c = 0; c < 16; ++c) {
                                const float x = __uint_as_float(v[i & 1][c]);
                                if (c & 1)
                                    add_whole(sum[i][c], x);
                                else
                                    sum[i][c] += __float2int_rn(x);
                            }
                        }
                        if (s + 1 < n_segs) release();
                    }
                    if (!ok) break;
#pragma unroll
                    for (int i = 0; i < T::NCH2; ++i) {
                        uint32_t v[16];
#pragma unroll
                        for (int c = 0; c < 16; ++c) v[c] = (uint32_t)sum[i][c] - (c & 1 ? (uint32_t)n_segs * kAddWhole : 0u);
                        if (i < n_chunks) tc::tmem_st16(d0 + 16u * i, v);
                    }
                    tc::tmem_st_wait();
                } else {
                    if (!tc::mbar_wait(&accf_bar[acc], acc_phase, &err_s, 4, a.wait_cycles)) {
                        ok = false;
                        break;
                    }
                    tc::fence_after();
                    d0 = col_addr + (uint32_t)(acc * BN);
                }
                if (lane == 0) sh.beat = sh.beat + 1;
                // the threshold: the best k-th score that any list of this query has reached
                if (live) {
                    const unsigned long long w = sh.thr[row];
                    if ((uint32_t)(w >> 32) == (uint32_t)grp) thr = fmaxf(thr, __uint_as_float((uint32_t)w));
                    const uint32_t best = tc::ld_relaxed_u32(a.kth + gq);
                    if (best) thr = fmaxf(thr, mm_filter_below(unord_float(best), a.mode));
                }
                const int64_t col0 = (int64_t)t * BN + half * T::NCH2 * 16;
                const int64_t left = a.nr - col0;
                const int n_ok = left < 16 * n_chunks ? (int)(left < 0 ? 0 : left) : 16 * n_chunks;  // real references
                // f(column, accumulator, estimate) for the 16 columns of chunk i
                auto chunk = [&](int i, auto&& f) {
                    uint32_t v[16];
                    tc::tmem_ld16(d0 + 16u * i, v);
                    const int mine = 16 * i + (lane & 15);
                    const float rr_lane = mine < n_ok ? __ldg(a.rr + col0 + mine) : 0.0f;
                    tc::tmem_ld_wait();
#pragma unroll
                    for (int c = 0; c < 16; ++c) {
                        const float x = multi ? (float)(int32_t)v[c] : __uint_as_float(v[c]);
                        f(c, v[c], approx_score(x, my_rq, __shfl_sync(0xffffffffu, rr_lane, c), a.mode));
                    }
                };
                int n_pass = 0;
                float low = INFINITY, high = -INFINITY;
#pragma unroll 1
                for (int i = 0; i < n_chunks; ++i)
                    chunk(i, [&](int c, uint32_t, float e) {
                        const bool in = 16 * i + c < n_ok;
                        n_pass += e >= thr && in;
                        low = fminf(low, in ? e : INFINITY);
                        high = fmaxf(high, in ? e : -INFINITY);
                    });
                if (!live) n_pass = 0;
                if (__any_sync(0xffffffffu, n_pass > k + kSlack)) {
                    // Many columns of one row pass (nothing known yet, or the tile holds a whole family of relatives):
                    // bisect the estimates for a threshold that between k and k + kSlack of them reach.  k columns of
                    // this tile reach it, so a lower one cannot enter the list.
                    float lo = fmaxf(thr, low), hi = high;
                    bool open = n_pass > k + kSlack;
                    for (int it = 0; it < 12 && __any_sync(0xffffffffu, open); ++it) {
                        const float mid = 0.5f * (lo + hi);
                        int n = 0;
#pragma unroll 1
                        for (int i = 0; i < n_chunks; ++i)
                            chunk(i, [&](int c, uint32_t, float e) { n += e >= mid && 16 * i + c < n_ok; });
                        if (open) {
                            if (n >= k)
                                lo = mid;
                            else
                                hi = mid;
                            open = n < k || n > k + kSlack;
                        }
                    }
                    // (a zero norm's COS estimate is 0 but its score -1: no k columns are known to reach an estimate below)
                    if (a.mode == HDC_SCORE_COS && lo <= 0.0f) lo = -1.0f;
                    if (n_pass > k + kSlack) thr = fmaxf(thr, mm_filter_below(lo, a.mode));
                }
                if (__any_sync(0xffffffffu, n_pass != 0)) {
#pragma unroll 1
                    for (int i = 0; i < n_chunks; ++i) {
                        uint32_t pm = 0, dots[16];
                        chunk(i, [&](int c, uint32_t v, float e) {
                            pm |= (uint32_t)(e >= thr && live && 16 * i + c < n_ok) << c;
                            dots[c] = v;
                        });
                        // each lane hands over its own next column; the dot is picked by masks (plain selects are
                        // folded back into a dynamic index, which would move the columns to local memory)
                        while (__any_sync(0xffffffffu, pm != 0)) {
                            const int at = __ffs(pm) - 1;
                            uint32_t x = 0;
#pragma unroll
                            for (int c = 0; c < 16; ++c) x |= dots[c] & (0u - (uint32_t)(at == c));
                            if (pm) push(multi ? (int32_t)x : __float2int_rn(__uint_as_float(x)), (uint32_t)(col0 + 16 * i + at));
                            pm &= pm - 1;
                            __syncwarp();
                        }
                    }
                }
                release();
            }
            if (!ok) break;
            push(0, kFlush);
            __syncwarp();
        }
    } else {
        // ------------------------------------------------ scorers: warps 12..15, one thread a query
        regs_down<kRegsScore>();
        const int row = (warp & 3) * 32 + lane;
        const int k = a.k;
        uint64_t rkeys[KR > 0 ? KR : 1];
        int32_t* sdots = reinterpret_cast<int32_t*>(lists_s) + row;
        uint64_t* skeys = reinterpret_cast<uint64_t*>(lists_s + (size_t)k * kMmQueryTile * sizeof(int32_t)) + row;
        uint64_t slots = 0;
        uint32_t tail[2] = {0, 0};
        bool ok = true;
        for (int grp = 0; ok && grp < a.n_groups; ++grp) {
            if (grp * a.G + lead_slot >= a.n_qtiles) continue;
            const int64_t gq = (int64_t)(grp * a.G + gslot) * kMmQueryTile + row;
            const bool live = gq < a.nq;
            const int64_t qn = live ? a.qn[gq] : 0;
            const double my_sq = __dsqrt_rn((double)qn);
            const double my_iq = qn ? __drcp_rn(my_sq) : 0.0;
            uint64_t* out_key = a.ws_key + ((int64_t)lane_j * a.nq + gq) * k;
            int64_t* out_dot = a.ws_dot + ((int64_t)lane_j * a.nq + gq) * k;
            const bool carry = a.carry && live;
            uint64_t kth = 0;
            slots = 0xfedcba9876543210ull;
            if constexpr (KR > 0) {
#pragma unroll
                for (int i = 0; i < KR; ++i) {
                    rkeys[i] = carry && i < k ? out_key[i] : 0;
                    if (i < k) sdots[i * kMmQueryTile] = carry ? (int32_t)out_dot[i] : 0;
                    kth |= rkeys[i] & (0ull - (uint64_t)(i == k - 1));
                }
            } else {
                for (int i = 0; i < k; ++i) {
                    skeys[i * kMmQueryTile] = carry ? out_key[i] : 0;
                    sdots[i * kMmQueryTile] = carry ? (int32_t)out_dot[i] : 0;
                }
                kth = skeys[(k - 1) * kMmQueryTile];
            }
            int ended = 0;  // bit h: half h has flushed; what follows in its ring belongs to the next group
            long long c0 = clock64();
            uint32_t seen = sh.beat;
            while (true) {
                int h = -1;
                if (!(ended & 1) && ld_acquire_shared(&sh.head[0][row]) != tail[0])
                    h = 0;
                else if (!(ended & 2) && ld_acquire_shared(&sh.head[1][row]) != tail[1])
                    h = 1;
                if (__all_sync(0xffffffffu, ended == 3)) break;
                if (!__any_sync(0xffffffffu, h >= 0)) {
                    bool stop = err_s != 0;
                    if (sh.beat != seen) {
                        seen = sh.beat;
                        c0 = clock64();
                    } else if (clock64() - c0 > 2 * a.wait_cycles) {
                        atomicCAS(const_cast<int*>(&err_s), 0, 6);
                        stop = true;
                    }
                    if (__any_sync(0xffffffffu, stop)) {
                        ok = false;
                        break;
                    }
                    __nanosleep(200);
                    continue;
                }
                if (h >= 0) {
                    const uint32_t at = h ? tail[1] : tail[0];
                    const int2 cand = sh.ring[h][at % kRing][row];
                    if (h)
                        ++tail[1];
                    else
                        ++tail[0];
                    st_release_shared(&sh.tail[h][row], at + 1);
                    if ((uint32_t)cand.y == kFlush) {
                        ended |= 1 << h;
                    } else {
                        const double rsc = __ldg(a.rs + (uint32_t)cand.y), ric = __ldg(a.ri + (uint32_t)cand.y);
                        const float s = exact_score_recip(cand.x, my_sq, rsc, my_iq, ric, a.mode);
                        const uint64_t key = make_key(s, (uint32_t)(a.r0 + (uint32_t)cand.y));
                        if (key > kth) {
                            if constexpr (KR > 0)
                                kth = mm_insert<KR>(rkeys, slots, k, key, cand.x, sdots);
                            else
                                kth = mm_insert_shared(skeys, sdots, k, key, cand.x);
                            if (kth != 0) {  // a full list: its last score is a floor for every list of the query
                                sh.thr[row] = (unsigned long long)(uint32_t)grp << 32 |
                                              __float_as_uint(mm_filter_below(key_score(kth), a.mode));
                                if (a.S > 1) atomicMax(a.kth + gq, (uint32_t)(kth >> 32));
                            }
                        }
                    }
                }
                __syncwarp();
            }
            if (!ok) break;
            if (live) {
                if (kth != 0) atomicMax(a.kth + gq, (uint32_t)(kth >> 32));
                if constexpr (KR > 0) {
#pragma unroll
                    for (int i = 0; i < KR; ++i)
                        if (i < k) {
                            out_key[i] = rkeys[i];
                            out_dot[i] = rkeys[i] ? sdots[(int)((slots >> (4 * i)) & 15u) * kMmQueryTile] : 0;
                        }
                } else {
                    for (int i = 0; i < k; ++i) {
                        const uint64_t key = skeys[i * kMmQueryTile];
                        out_key[i] = key;
                        out_dot[i] = key ? sdots[i * kMmQueryTile] : 0;
                    }
                }
            }
        }
    }

    tc::fence_before();
    __syncthreads();
    if (warp == 1 && crank == 0 && err_s && tc::elect_one()) tc::mma_drain<PAIR>(&drain_bar);
    if constexpr (PAIR) tc::cluster_sync();  // both CTAs are done with the pair's TMEM
    if (warp == 1) {
        __syncwarp();
        tc::fence_after();
        if constexpr (PAIR)
            tc::tmem_dealloc_pair(tmem, 512);
        else
            tc::tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && err_s) atomicCAS(a.status, 0, 100 + err_s);
    if constexpr (PAIR) tc::cluster_sync();  // no CTA leaves while its peer may still write into it
}

// ---------------------------------------------------------------- small problems: the K loop split over CTAs
// A problem with fewer tiles than SMs leaves most of them idle, and its time is one tile's K loop (157 K blocks of 330
// cycles at D = 10,000, bound by the issuer's waits and commits) plus lists, thresholds and a merge made for thousands of
// tiles.  Here the CTAs of a tile share its K blocks, each stores the whole dots of its part (at most a tile a CTA: 5 MB
// in all on fp16 rows, 9 MB on digits), and one CTA a query adds the parts up and selects.  48 x 2,000 at D = 10,000:
// 80 -> 40 us with its conversion; 190 x 567 at D = 1,024, top-32: 200 -> 36.
constexpr int kDotThreads = 192;   // producer, MMA issuer, four drain warps
constexpr int kSplitRefs = 12288;  // a query's dots and keys in shared memory
constexpr int kMinSplitBlocks = 4; // K blocks that a CTA is worth starting for

struct DotsArgs {
    int64_t nq;
    int n_kb, kb_per_seg, limbs, stages, n_rtiles, splits, ldd, withhold;
    int32_t* parts;  // [splits][nq][ldd]
    int* status;
    long long wait_cycles;
};

template <bool F4>
__global__ void __launch_bounds__(kDotThreads, 1)
    mm_dots_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const DotsArgs a) {
    using T = MmTile<F4, 1>;
    constexpr int BN = T::N;
    constexpr uint32_t IDESC = F4 ? tc::idesc_f4_f32(kMmQueryTile, BN) : tc::idesc_f16_f32(kMmQueryTile, BN);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* ring = smem_raw + ((1024 - (tc::smem_u32(smem_raw) & 1023)) & 1023);
    __shared__ uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], accf_bar[2], acce_bar[2], drain_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int err_s;
    const int stages = a.stages, stage_bytes = mm_stage_bytes(T::A_BYTES, T::B_BYTES, a.limbs);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        err_s = 0;
        for (int s = 0; s < stages; ++s) {
            tc::mbar_init(&full_bar[s], 1);
            tc::mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            tc::mbar_init(&accf_bar[b], 1);
            tc::mbar_init(&acce_bar[b], 4);
        }
        tc::mbar_init(&drain_bar, 1);
        tc::fence_mbar_init();
        tc::prefetch_tmap(&tmA);
        tc::prefetch_tmap(&tmB);
    }
    if (warp == 1) {
        tc::tmem_alloc(&tmem_base_s, 512);
        tc::tmem_relinquish();
    }
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = tmem_base_s;
    if constexpr (F4) {  // the digits' block scales, as in mm_search_kernel
        if (warp < 4) {
            uint32_t v[32];
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0x01010101u * (uint32_t)(127 + 3 * (i / 8));
            tc::tmem_st32(tmem + ((uint32_t)(warp * 32) << 16) + kScaleCol, v);
            tc::tmem_st_wait();
        }
        tc::fence_before();
        __syncthreads();
        tc::fence_after();
    }
    // this CTA's tile and K blocks
    const int split = (int)(blockIdx.x % a.splits), tile = (int)(blockIdx.x / a.splits);
    const int rt = tile % a.n_rtiles, qt = tile / a.n_rtiles;
    const int kb0 = (int)((int64_t)split * a.n_kb / a.splits), kb1 = (int)((int64_t)(split + 1) * a.n_kb / a.splits);
    if (warp == 0) {
        if (tc::elect_one()) {
            int stage = 0, issued = 0;
            uint32_t phase = 0;
            for (int kb = kb0; !a.withhold && kb < kb1; ++kb) {
                if (!tc::mbar_wait(&empty_bar[stage], phase ^ 1, &err_s, 1, a.wait_cycles)) break;
                uint8_t* st = ring + (size_t)stage * stage_bytes;
                tc::mbar_arrive_expect_tx(&full_bar[stage], stage_bytes);
                if constexpr (F4) {
                    tc::tma_load_2d(st, &tmA, &full_bar[stage], 0, (qt * a.n_kb + kb) * kMmQueryTile);
                    const int y = (((rt >> 1) * a.n_kb + kb) * 2 + (rt & 1)) * a.limbs * kMmF4Half;
                    for (int l = 0; l < a.limbs; ++l)
                        tc::tma_load_2d(st + T::A_BYTES + l * T::B_BYTES, &tmB, &full_bar[stage], 0, y + l * kMmF4Half);
                } else {
                    tc::tma_load_2d(st, &tmA, &full_bar[stage], kb * 64, qt * kMmQueryTile);
                    tc::tma_load_2d(st + T::A_BYTES, &tmB, &full_bar[stage], kb * 64, rt * BN);
                }
                ++issued;
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1;
                }
            }
            // the last loads land before the CTA leaves (bounded)
            for (int i = 0; i < min(issued, stages); ++i) {
                if (--stage < 0) {
                    stage = stages - 1;
                    phase ^= 1;
                }
                const long long c0 = clock64();
                while (!tc::mbar_try_wait(tc::smem_u32(&full_bar[stage]), phase) && clock64() - c0 < tc::kWaitCycles) {
                }
            }
        }
    } else if (warp == 1) {
        if (tc::elect_one()) {
            int stage = 0, acc = 0;
            uint32_t phase = 0, acc_phase = 0;
            bool ok = true;
            for (int k0 = kb0; ok && k0 < kb1; k0 += a.kb_per_seg) {
                if (!(ok = tc::mbar_wait(&acce_bar[acc], acc_phase ^ 1, &err_s, 2, a.wait_cycles))) break;
                tc::fence_after();
                const uint32_t d0 = tmem + (uint32_t)(acc * BN);
                for (int kb = k0; kb < min(k0 + a.kb_per_seg, kb1); ++kb) {
                    if (!(ok = tc::mbar_wait(&full_bar[stage], phase, &err_s, 3, a.wait_cycles))) break;
                    tc::fence_after();
                    const uint32_t sa = tc::smem_u32(ring + (size_t)stage * stage_bytes);
                    const uint64_t adesc = tc::kmajor_desc(sa, T::SBO, T::LAYOUT);
                    const uint64_t bdesc = tc::kmajor_desc(sa + (uint32_t)T::A_BYTES, T::SBO, T::LAYOUT);
                    if constexpr (F4) {
                        for (int l = 0; l < a.limbs; ++l) {
                            const uint32_t sfa = tmem + kScaleCol + (l == 4 ? 8u : 0u);
                            const uint32_t sfb = tmem + kScaleCol + 8u * (uint32_t)(l == 4 ? 3 : l);
                            const uint64_t bl = bdesc + (uint64_t)(l * (T::B_BYTES >> 4));
#pragma unroll
                            for (int kk = 0; kk < 2; ++kk)
                                tc::mma_f4(d0, adesc + 2 * kk, bl + 2 * kk, IDESC, sfa, sfb, (kb - k0) | l | kk ? 1u : 0u);
                        }
                    } else {
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk)
                            tc::mma_f16(d0, adesc + 2 * kk, bdesc + 2 * kk, IDESC, (kb - k0) | kk ? 1u : 0u);
                    }
                    tc::mma_commit(&empty_bar[stage]);
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1;
                    }
                }
                if (!ok) break;
                tc::mma_commit(&accf_bar[acc]);
                if (++acc == 2) {
                    acc = 0;
                    acc_phase ^= 1;
                }
            }
        }
    } else {
        const int quarter = warp & 3, row = quarter * 32 + lane;
        const int64_t gq = (int64_t)qt * kMmQueryTile + row;
        int32_t sum[BN];
#pragma unroll
        for (int c = 0; c < BN; ++c) sum[c] = 0;
        int acc = 0;
        uint32_t acc_phase = 0;
        bool ok = true;
        for (int k0 = kb0; k0 < kb1; k0 += a.kb_per_seg) {
            if (!(ok = tc::mbar_wait(&accf_bar[acc], acc_phase, &err_s, 4, a.wait_cycles))) break;
            tc::fence_after();
            const uint32_t d0 = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(acc * BN);
#pragma unroll
            for (int i = 0; i < BN / 16; ++i) {
                uint32_t v[16];
                tc::tmem_ld16(d0 + 16u * i, v);
                tc::tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 16; ++c) sum[16 * i + c] += __float2int_rn(__uint_as_float(v[c]));
            }
            tc::fence_before();
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(&acce_bar[acc]);
            if (++acc == 2) {
                acc = 0;
                acc_phase ^= 1;
            }
        }
        if (ok && gq < a.nq) {
            int4* out = reinterpret_cast<int4*>(a.parts + ((int64_t)split * a.nq + gq) * a.ldd + (int64_t)rt * BN);
#pragma unroll
            for (int i = 0; i < BN / 4; ++i) out[i] = make_int4(sum[4 * i], sum[4 * i + 1], sum[4 * i + 2], sum[4 * i + 3]);
        }
    }
    tc::fence_before();
    __syncthreads();
    if (warp == 1 && err_s && tc::elect_one()) tc::mma_drain<false>(&drain_bar);
    if (warp == 1) {
        __syncwarp();
        tc::fence_after();
        tc::tmem_dealloc(tmem, 512);
    }
    if (threadIdx.x == 0 && err_s) atomicCAS(a.status, 0, 100 + err_s);
}

// One CTA a query: its dots from the parts, a threshold that at least k of them are known to reach (by bisection of the
// threads' best estimates), exact scores of those that an estimate lets through, and their order by counting.  Bound by
// the latency of that chain for a few queries, and by the FP64 pipe (two lanes a cycle) for thousands.
template <int NT>
__global__ void __launch_bounds__(NT) mm_select_kernel(
    const int32_t* __restrict__ parts, int splits, int64_t nq, int nr, int ldd, const int64_t* __restrict__ qn,
    const float* __restrict__ rr, const double* __restrict__ rs, const double* __restrict__ ri, int k, int mode,
    float* __restrict__ out_s, int32_t* __restrict__ out_i, double* __restrict__ out_c, int64_t* __restrict__ out_d) {
    extern __shared__ uint64_t keys[];  // [nr], then the dots
    int32_t* dots = reinterpret_cast<int32_t*>(keys + nr);
    __shared__ uint64_t warp_best[2][NT / 32];
    __shared__ uint32_t warp_ord[2][NT / 32];
    __shared__ double root_s[2];
    __shared__ int n_s;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t q = blockIdx.x, n2 = qn[q];
    if (tid == NT - 1) {  // (with the fewest references)
        n_s = 0;
        root_s[0] = __dsqrt_rn((double)n2);
        root_s[1] = n2 ? __drcp_rn(root_s[0]) : 0.0;
    }
    const float rq = n2 ? __frsqrt_rn(__ll2float_rn(n2)) : 0.0f;
    // a reference's estimate; under COS a zero norm scores -1, where the product would be 0
    auto estimate = [&](int32_t dot, float f) {
        return mode == HDC_SCORE_COS && (f == 0.0f || rq == 0.0f) ? -1.0f : approx_score((float)dot, rq, f, mode);
    };
    float best = -INFINITY;
    for (int j = 4 * tid; j < nr; j += 4 * NT) {  // (ldd is a multiple of 16, and the parts are written that far)
        const int32_t* from = parts + q * ldd + j;
        const int64_t step = nq * ldd;
        int4 d = make_int4(0, 0, 0, 0);
#pragma unroll 8
        for (int s = 0; s < splits; ++s) {
            const int4 x = __ldcg(reinterpret_cast<const int4*>(from + s * step));
            d.x += x.x;
            d.y += x.y;
            d.z += x.z;
            d.w += x.w;
        }
        const int32_t v[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (j + u < nr) {
                dots[j + u] = v[u];
                best = fmaxf(best, estimate(v[u], __ldg(rr + j + u)));
            }
    }
    const uint32_t mine_ord = ord_float(best), none = ord_float(-INFINITY);
    const uint32_t top_ord = __reduce_max_sync(0xffffffffu, mine_ord);
    const uint32_t low_ord = __reduce_min_sync(0xffffffffu, mine_ord == none ? 0xffffffffu : mine_ord);
    if (lane == 0) {
        warp_ord[0][warp] = low_ord;
        warp_ord[1][warp] = top_ord;
    }
    __syncthreads();
    float thr = -INFINITY;
    if (min(NT, (nr + 3) / 4) >= k) {  // as many threads have a best
        uint32_t a = warp_ord[0][0], b = warp_ord[1][0];
#pragma unroll
        for (int w = 1; w < NT / 32; ++w) {
            a = min(a, warp_ord[0][w]);
            b = max(b, warp_ord[1][w]);
        }
        float lo = unord_float(a), hi = unord_float(b);  // all of them reach lo
        for (int it = 0; it < 12; ++it) {
            const float mid = 0.5f * (lo + hi);
            const int n = __syncthreads_count(best >= mid);
            if (n >= k)
                lo = mid;
            else
                hi = mid;
            if (n >= k && n <= k + kSlack) break;
        }
        thr = mm_filter_below(lo, mode);
    }
    const double sq = root_s[0], iq = root_s[1];
    auto exact_key = [&](int j) {
        return make_key(exact_score_recip(dots[j], sq, __ldg(rs + j), iq, __ldg(ri + j), mode), (uint32_t)j);
    };
    auto put = [&](int at, uint64_t key) {
        const uint32_t j = key_idx(key);
        out_s[q * k + at] = key_score(key);
        out_i[q * k + at] = (int32_t)j;
        if (out_d) out_d[q * k + at] = dots[j];
        if (out_c) {  // exact_cos with the roots at hand
            const double sr = __ldg(rs + j);
            out_c[q * k + at] = sq == 0.0 || sr == 0.0 ? 0.0 : __ddiv_rn((double)dots[j], __dmul_rn(sq, sr));
        }
    };
    for (int j = tid; j < nr; j += NT)
        if (estimate(dots[j], __ldg(rr + j)) >= thr) keys[atomicAdd(&n_s, 1)] = (uint64_t)j;
    __syncthreads();
    const int n = n_s;  // at least k
    if (n <= NT) {
        const uint64_t mine = tid < n ? exact_key((int)keys[tid]) : 0;
        __syncthreads();
        if (tid < n) keys[tid] = mine;
        __syncthreads();
        if (tid < n) {
            int at = 0;
            for (int i = 0; i < n; ++i) at += keys[i] > mine;
            if (at < k) put(at, mine);
        }
        return;
    }
    // more of them (scores tied by the hundred): the largest key below the last one, k times
    for (int i = tid; i < n; i += NT) keys[i] = exact_key((int)keys[i]);
    uint64_t last = ~0ull;
    for (int at = 0; at < k; ++at) {
        uint64_t top = 0;
        for (int i = tid; i < n; i += NT) {  // (the keys that this thread wrote)
            const uint64_t x = keys[i];
            top = x < last && x > top ? x : top;
        }
        for (int o = 16; o; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        if (lane == 0) warp_best[at & 1][warp] = top;
        __syncthreads();
        for (int w = 0; w < NT / 32; ++w) top = max(top, warp_best[at & 1][w]);
        last = top;
        if (tid == 0) put(at, top);
    }
}

// ---------------------------------------------------------------- merge
constexpr int kMergeWarps = 4;
constexpr int kMergeHeads = 5;  // lists a lane follows: 160 lists in all

// One warp per query: lane l follows the heads of lists l, l + 32, ... (each sorted), and every round takes the
// largest head.  Keys are distinct (the reference index is part of them).
__global__ void __launch_bounds__(32 * kMergeWarps) mm_merge_kernel(
    const uint64_t* __restrict__ ws_key, const int64_t* __restrict__ ws_dot, int n_lists, int64_t nq, int k,
    const int64_t* __restrict__ qn, const int64_t* __restrict__ rn, int64_t nr, float* __restrict__ out_s,
    int32_t* __restrict__ out_i, double* __restrict__ out_c, int64_t* __restrict__ out_d) {
    const int64_t q = (int64_t)blockIdx.x * kMergeWarps + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (q >= nq) return;
    uint64_t head[kMergeHeads];
    uint64_t pos = 0;  // 6 bits a list: entries taken from it
#pragma unroll
    for (int h = 0; h < kMergeHeads; ++h) {
        const int l = lane + 32 * h;
        head[h] = l < n_lists ? ws_key[((int64_t)l * nq + q) * k] : 0;
    }
    uint64_t my_key = 0;  // entry `lane` of the result and its dot
    int64_t my_dot = 0;
    for (int i = 0; i < k; ++i) {
        uint64_t best = 0;
        int at = 0;
#pragma unroll
        for (int h = 0; h < kMergeHeads; ++h)
            if (head[h] > best) {
                best = head[h];
                at = h;
            }
        uint64_t top = best;
        for (int o = 16; o; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        if (top == 0) break;
        const int src = __ffs(__ballot_sync(0xffffffffu, best == top)) - 1;
        int64_t dot = 0;
        if (lane == src) {
            const int p = (int)((pos >> (6 * at)) & 63u);
            const int64_t base = ((int64_t)(lane + 32 * at) * nq + q) * k;
            dot = ws_dot[base + p];
            const uint64_t next = p + 1 < k ? ws_key[base + p + 1] : 0;
            pos += 1ull << (6 * at);
#pragma unroll
            for (int h = 0; h < kMergeHeads; ++h)
                if (h == at) head[h] = next < top ? next : 0;  // a list a search left unwritten holds stale keys
        }
        dot = __shfl_sync(0xffffffffu, dot, src);
        if (lane == i) {
            my_key = top;
            my_dot = dot;
        }
    }
    if (lane >= k) return;
    const uint32_t idx = key_idx(my_key);
    const bool ok = my_key != 0 && (int64_t)idx < nr;
    out_s[q * k + lane] = ok ? key_score(my_key) : -INFINITY;
    out_i[q * k + lane] = ok ? (int32_t)idx : -1;
    if (out_c) out_c[q * k + lane] = ok ? exact_cos(my_dot, qn[q], rn[idx]) : 0.0;
    if (out_d) out_d[q * k + lane] = ok ? my_dot : 0;
}

// ---------------------------------------------------------------- operand preparation
constexpr int kRowThreads = 128;
constexpr int kCodeQueryBound = 201;  // status: a query value beyond the +1/0/-1 that the caller declared

// e2m1 code of an integer digit of magnitude <= 4
__device__ __forceinline__ uint32_t e2m1(int d) {
    const int m = d < 0 ? -d : d;
    return (d < 0 ? 8u : 0u) | ((0x65420u >> (4 * m)) & 7u);
}

// Element offset of the 16-byte chunk c (0..3) of row r in a tile of 64-byte rows with the 64-byte swizzle of the
// shared-memory descriptor (chunk bits ^= address bits 7..8): a plain copy of the tile is then a swizzled tile.
__device__ __forceinline__ int64_t f4_chunk(int64_t tile_row0, int r, int c) {
    return (tile_row0 + r) * 64 + ((c ^ ((r >> 1) & 3)) << 4);
}

template <typename Q>
__device__ __forceinline__ int as_int(Q x);
template <>
__device__ __forceinline__ int as_int<int16_t>(int16_t x) { return x; }
template <>
__device__ __forceinline__ int as_int<__half>(__half x) { return __half2int_rn(x); }

// Queries of values -1, 0, 1 as e2m1 tiles [query tile][K block][128 rows][64 bytes]; a thread makes 16 bytes (32
// dims of one row).  Bound by the bytes of the 16-bit rows.  A value that the caller's bound does not allow is reported:
// its code would be another number's.
template <typename Q, bool VEC>
__global__ void pack_queries_kernel(const Q* __restrict__ q, int64_t nq, int dim, int n_kb, int64_t n_chunks,
                                    uint8_t* __restrict__ out, int* __restrict__ status) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_chunks) return;
    const int64_t per_row = (int64_t)n_kb * 4;
    const int64_t row = i / per_row;
    const int rc = (int)(i - row * per_row), kb = rc >> 2, c = rc & 3;
    const int d0 = kb * kMmF4Dims + c * 32;
    uint32_t w[4] = {0, 0, 0, 0};
    if (row < nq) {
        const Q* src = q + row * dim + d0;
        bool beyond = false;
        Q x[32];
        if (VEC && d0 + 32 <= dim) {
#pragma unroll
            for (int u = 0; u < 4; ++u) reinterpret_cast<uint4*>(x)[u] = __ldg(reinterpret_cast<const uint4*>(src) + u);
        } else {
#pragma unroll
            for (int u = 0; u < 32; ++u) x[u] = d0 + u < dim ? src[u] : Q(0);
        }
#pragma unroll
        for (int u = 0; u < 32; ++u) {
            const int v = as_int<Q>(x[u]);
            beyond |= (uint32_t)(v + 1) > 2u;
            w[u >> 3] |= e2m1(v) << (4 * (u & 7));
        }
        if (beyond) atomicCAS(status, 0, kCodeQueryBound);
    }
    const int64_t tile = ((row / kMmQueryTile) * n_kb + kb) * kMmQueryTile;
    *reinterpret_cast<uint4*>(out + f4_chunk(tile, (int)(row % kMmQueryTile), c)) = make_uint4(w[0], w[1], w[2], w[3]);
}

// References as base-8 digit tiles [tile][K block][half][digit][112 rows][64 bytes], from int16 rows or from fp16
// limbs; a thread makes one row's 32 dims, 16 bytes per digit.
template <bool LIMBS, bool VEC>
__global__ void pack_refs_kernel(const int16_t* __restrict__ r16, const __half* __restrict__ limbs16, int L16, int bits,
                                 int64_t r_pad, int64_t nr, int dim, int n_kb, int limbs, int64_t n_chunks,
                                 uint8_t* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_chunks) return;
    const int64_t per_row = (int64_t)n_kb * 4;
    const int64_t row = i / per_row;
    const int rc = (int)(i - row * per_row), kb = rc >> 2, c = rc & 3;
    const int d0 = kb * kMmF4Dims + c * 32;
    int v[32];
#pragma unroll
    for (int u = 0; u < 32; ++u) v[u] = 0;
    if (row < nr) {
        for (int l = 0; l < (LIMBS ? L16 : 1); ++l) {
            const int16_t* src = (LIMBS ? reinterpret_cast<const int16_t*>(limbs16) + (int64_t)l * r_pad * dim : r16) +
                                 row * dim + d0;
            int16_t x[32];
            if (VEC && d0 + 32 <= dim) {
#pragma unroll
                for (int u = 0; u < 4; ++u) reinterpret_cast<uint4*>(x)[u] = __ldg(reinterpret_cast<const uint4*>(src) + u);
            } else {
#pragma unroll
                for (int u = 0; u < 32; ++u) x[u] = d0 + u < dim ? src[u] : (int16_t)0;
            }
#pragma unroll
            for (int u = 0; u < 32; ++u)
                v[u] += LIMBS ? __half2int_rn(__short_as_half(x[u])) * (1 << (bits * l)) : (int)x[u];
        }
    }
    const int64_t tile = row / (2 * kMmF4Half);
    const int rt = (int)(row - tile * (2 * kMmF4Half)), half = rt / kMmF4Half, rh = rt % kMmF4Half;
    const int64_t base = ((tile * n_kb + kb) * 2 + half) * limbs * kMmF4Half;
    for (int l = 0; l < limbs; ++l) {
        uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
        for (int u = 0; u < 32; ++u) {
            // the digit nearest zero that leaves a multiple of 8; 4 and -4 both do, the one toward zero is taken
            int d = v[u] & 7;
            if (d > 4 || (d == 4 && v[u] < 0)) d -= 8;
            w[u >> 3] |= e2m1(d) << (4 * (u & 7));
            v[u] = (v[u] - d) / 8;
        }
        *reinterpret_cast<uint4*>(out + f4_chunk(base + (int64_t)l * kMmF4Half, rh, c)) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

__device__ __forceinline__ void norm_tables_one(int64_t v, int64_t i, float* rr, double* rs, double* ri) {
    const double s = __dsqrt_rn((double)v);
    rr[i] = rsqrt_norm(v);
    rs[i] = s;
    ri[i] = v ? __drcp_rn(s) : 0.0;
}

// Eight threads' sums of squares of 8 dims each, as the K block's (the lanes of `group` take part).
template <typename T>
__device__ __forceinline__ T kblock_norm(T s, uint32_t group) {
    for (int o = 4; o; o >>= 1) s += __shfl_xor_sync(group, s, o);
    return s;
}

__device__ __forceinline__ uint32_t warp_most(uint32_t v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ unsigned long long warp_most(unsigned long long v) {
    for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// A CTA's sum of squares and its threads' largest of a K block, as the largest so far.
template <typename T>
__device__ __forceinline__ void block_norm_max(unsigned long long s, T most, MmNorms* out) {
    __shared__ MmNorms part[kRowThreads / 32];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    unsigned long long b = warp_most(most);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = {s, b};
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kRowThreads / 32; ++w) {
            s += part[w].row;
            b = max(b, part[w].block);
        }
        const ulonglong2 now = __ldcg(reinterpret_cast<const ulonglong2*>(out));  // (both only ever grow)
        if (s > now.x) atomicMax(&out->row, s);
        if (b > now.y) atomicMax(&out->block, b);
    }
}

// int16 rows of dim elements -> fp16 rows of ld elements (exact for |v| <= 2048) and their largest squared norm, a CTA
// a row, 8 elements a thread and step.  Bound by the bytes: 2 read and 2 written a value.
template <bool VEC>
__global__ void __launch_bounds__(kRowThreads) rows_f16_kernel(const int16_t* __restrict__ v, int dim, int64_t ld,
                                                               __half* __restrict__ out, MmNorms* __restrict__ norms) {
    const int64_t row = blockIdx.x;
    const uint32_t group = 0xffu << (threadIdx.x & 24);  // (ld is a multiple of 64: the eight run a step together)
    unsigned long long s = 0;
    uint32_t most = 0;  // (64 values of magnitude <= 2048: 2^28)
    for (int d0 = threadIdx.x * 8; d0 < ld; d0 += kRowThreads * 8) {
        const int16_t* src = v + row * dim + d0;
        int16_t x[8];
        if (VEC && d0 + 8 <= dim) {
            *reinterpret_cast<uint4*>(x) = __ldg(reinterpret_cast<const uint4*>(src));
        } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = d0 + u < dim ? src[u] : (int16_t)0;
        }
        __half h[8];
        uint32_t p = 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            h[u] = __short2half_rn(x[u]);
            p += (uint32_t)((int)x[u] * (int)x[u]);
        }
        *reinterpret_cast<uint4*>(out + row * ld + d0) = *reinterpret_cast<const uint4*>(h);
        s += p;
        most = max(most, kblock_norm(p, group));
    }
    block_norm_max(s, most, norms);
}

// The rows of both operands of a small problem in one launch: queries, then references with their norms' tables.
template <bool VEC>
__global__ void __launch_bounds__(kRowThreads) rows2_f16_kernel(const int16_t* __restrict__ q, int64_t nq,
                                                                const int16_t* __restrict__ r, int dim, int64_t ld,
                                                                __half* __restrict__ out_q, __half* __restrict__ out_r,
                                                                const int64_t* __restrict__ rn, float* __restrict__ rr,
                                                                double* __restrict__ rs, double* __restrict__ ri) {
    const bool ref = (int64_t)blockIdx.x >= nq;
    const int64_t row = ref ? (int64_t)blockIdx.x - nq : (int64_t)blockIdx.x;
    const int16_t* v = (ref ? r : q) + row * dim;
    __half* out = (ref ? out_r : out_q) + row * ld;
    if (ref && threadIdx.x == 0) norm_tables_one(rn[row], row, rr, rs, ri);
    for (int d0 = threadIdx.x * 8; d0 < ld; d0 += kRowThreads * 8) {
        int16_t x[8];
        if (VEC && d0 + 8 <= dim) {
            *reinterpret_cast<uint4*>(x) = __ldg(reinterpret_cast<const uint4*>(v + d0));
        } else {
#pragma unroll
            for (int u = 0; u < 8; ++u) x[u] = d0 + u < dim ? v[d0 + u] : (int16_t)0;
        }
        __half h[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) h[u] = __short2half_rn(x[u]);
        *reinterpret_cast<uint4*>(out + d0) = *reinterpret_cast<const uint4*>(h);
    }
}

// the largest squared norms of fp16 integer rows (dim % 8 == 0, 16-byte aligned)
__global__ void __launch_bounds__(kRowThreads) norm_max_kernel(const __half* __restrict__ v, int dim, MmNorms other,
                                                               MmNorms* __restrict__ norms) {
    const uint32_t group = 0xffu << (threadIdx.x & 24);
    unsigned long long s = 0, most = 0;
    const uint4* src = reinterpret_cast<const uint4*>(v + (int64_t)blockIdx.x * dim);
    for (int i = threadIdx.x; i < (dim / 8 + 7) / 8 * 8; i += kRowThreads) {  // whole K blocks
        const uint4 x = i < dim / 8 ? __ldg(src + i) : make_uint4(0, 0, 0, 0);
        const __half* h = reinterpret_cast<const __half*>(&x);
        unsigned long long p = 0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int e = __half2int_rn(h[u]);
            p += (unsigned long long)((long long)e * e);
        }
        s += p;
        most = max(most, kblock_norm(p, group));
    }
    block_norm_max(s, most, norms);
    if (blockIdx.x == 0 && threadIdx.x == 0) norms[1] = other;
}

// the values of a database's limbs (dim % 8 == 0), 8 elements a thread
__global__ void rows_from_limbs_kernel(const __half* __restrict__ limbs, int L, int bits, int64_t total, int64_t n_chunks,
                                       __half* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_chunks) return;
    int v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int l = 0; l < L; ++l) {
        const uint4 x = __ldg(reinterpret_cast<const uint4*>(limbs + (int64_t)l * total) + i);
        const __half* h = reinterpret_cast<const __half*>(&x);
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] += __half2int_rn(h[u]) * (1 << (bits * l));
    }
    __half h[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) h[u] = __int2half_rn(v[u]);
    reinterpret_cast<uint4*>(out)[i] = *reinterpret_cast<const uint4*>(h);
}

__global__ void limbs_max_kernel(const __half* __restrict__ limbs, int L, int bits, int64_t total, int64_t n_chunks,
                                 int32_t* __restrict__ out) {
    int32_t m = 0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_chunks; i += (int64_t)gridDim.x * blockDim.x) {
        int64_t v[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int l = 0; l < L; ++l) {
            const uint4 x = __ldg(reinterpret_cast<const uint4*>(limbs + (int64_t)l * total) + i);
            const __half* h = reinterpret_cast<const __half*>(&x);
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] += (int64_t)__half2int_rn(h[u]) * ((int64_t)1 << (bits * l));
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) m = max(m, (int32_t)min((int64_t)INT32_MAX, v[u] < 0 ? -v[u] : v[u]));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}

__global__ void norm_tables_kernel(const int64_t* __restrict__ n2, int64_t n, float* __restrict__ rr,
                                   double* __restrict__ rs, double* __restrict__ ri) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    norm_tables_one(n2[i], i, rr, rs, ri);
}

// ---------------------------------------------------------------- plan
int n_kblocks(int dim, bool f4) { return (dim + (f4 ? kMmF4Dims : 64) - 1) / (f4 ? kMmF4Dims : 64); }

struct MmPlan {
    int CL = 1, n_qtiles = 0, n_rtiles = 0, G = 1, S = 1, n_groups = 1;
};

// G query tiles at a time on S = SMs / G reference lanes each.  All G x S CTAs step through the same reference tiles
// together, so DRAM sees the references once a group.  The choice minimises
//     groups x (tiles of a lane x cycles of a tile + the start of the lists)
// with cycles a column and K step as measured.  Pairs run at the tensor pipe's rate: 0.53 (digits) and 0.5 (fp16: 514
// cycles a K block of 4 steps and 256 columns).  Single CTAs load as many operand bytes for half the MMA work or less:
// 0.9 (112 columns, 95 cycles a step) and 1.4 (64 columns: 328 cycles a K block where 32 CTAs run, bound by the MMA
// issuer's waits and commits; 400 on all SMs, bound by L2).  More
// lanes cost a little each (their lists start empty; 38 lanes none to speak of, 76 lanes 13 %), and a group whose
// query tiles fill L2 about 5 % (60,000 references, 38,912 queries: 22.4 ms with 38 tiles a group, 23.6 with 152).
MmPlan mm_plan(int sms, int64_t nq, int64_t nr, int dim, bool f4, int limbs) {
    MmPlan best;
    const int qt = (int)((nq + kMmQueryTile - 1) / kMmQueryTile);  // (32-bit divisions below: a call plans several times)
    const double steps = f4 ? (double)limbs * ((dim + 63) / 64) : (double)((dim + 15) / 16);
    double best_cost = 0;
    auto consider = [&](int CL, int n, double col_cycles) {
        const int rt = (int)((nr + n - 1) / n);
        const double tile = steps * n * col_cycles + 2500, row_bytes = f4 ? 0.5 * dim : 2.0 * dim;
        const int g_max = std::min(sms / CL * CL, (qt + CL - 1) / CL * CL);
        for (int G = CL; G <= g_max; G += CL) {
            const int S = std::min(std::min(sms / G, rt), 32 * kMergeHeads);
            if (S < 1) break;
            const int groups = (qt + G - 1) / G, tiles = (rt + S - 1) / S;
            const double in_l2 = std::min(1.0, (double)G * kMmQueryTile * row_bytes / 1e8);
            const double cost = (double)groups * ((double)tiles * tile + 20000) * (1 + 0.001 * (double)S + 0.05 * in_l2);
            if (best_cost == 0 || cost < best_cost) {
                best_cost = cost;
                best.CL = CL;
                best.n_qtiles = qt;
                best.n_rtiles = rt;
                best.G = G;
                best.S = S;
                best.n_groups = groups;
            }
        }
    };
    if (qt >= 2) consider(2, f4 ? MmTile<true, 2>::N : MmTile<false, 2>::N, f4 ? 0.53 : 0.5);
    consider(1, f4 ? MmTile<true, 1>::N : MmTile<false, 1>::N, f4 ? 0.9 : 1.4);
    return best;
}

size_t round256(size_t x) { return (x + 255) / 256 * 256; }

// the caller's words and the queries' thresholds, before the lists
size_t head_bytes(int64_t nq) {
    return round256(kMmWorkWords * sizeof(unsigned long long) + (size_t)nq * sizeof(uint32_t));
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool ok = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                            cudaSuccess &&
                        q == cudaDriverEntryPointSuccess;
        return ok ? reinterpret_cast<EncodeTiledFn>(p) : nullptr;
    }();
    return fn;
}

// F16: rows of `cols` elements, stride ld, boxes of 64 elements with the 128-byte swizzle.  F4: tiles that are
// swizzled in memory already, boxes of 64-byte rows copied as they are.
bool make_map(CUtensorMap* map, bool f4, const void* base, int64_t rows, int64_t cols, int64_t ld, int box_rows) {
    EncodeTiledFn encode = encode_fn();
    if (!encode) return false;
    cuuint64_t gdim[2] = {(cuuint64_t)(f4 ? 64 : cols), (cuuint64_t)rows};
    cuuint64_t gstride[1] = {(cuuint64_t)(f4 ? 64 : ld * 2)};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    return encode(map, f4 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base),
                  gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  f4 ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// see tile_stride of the limb search: a scattered order of the reference tiles
int scattered_stride(int n) {
    if (n <= 2) return 1;
    int s = std::max(1, (int)(0.6180339887 * n));
    while (std::gcd(s, n) != 1) ++s;
    return s % n ? s : 1;
}

template <bool F4, int CL, int KR>
int launch_mm(const MmOperands& op, MmArgs a, int dim, int grid, cudaStream_t stream) {
    using T = MmTile<F4, CL>;
    CUtensorMap tmA, tmB;
    const int64_t a_rows = F4 ? (int64_t)a.n_qtiles * a.n_kb * kMmQueryTile : a.nq;
    const int64_t b_tiles = (a.nr + 2 * kMmF4Half - 1) / (2 * kMmF4Half);
    const int64_t b_rows = F4 ? b_tiles * a.n_kb * 2 * a.limbs * kMmF4Half : a.nr;
    if (!make_map(&tmA, F4, op.a, a_rows, dim, op.lda, kMmQueryTile) ||
        !make_map(&tmB, F4, op.b, b_rows, dim, op.ldb, T::ROWS))
        return fail(HDC_ERR_CUDA, "mm search: cuTensorMapEncodeTiled failed");
    // after the ring: the rows' candidate rings, then the lists' dots (and keys, when not in registers)
    const size_t lists = sizeof(MmShared) + (size_t)a.k * kMmQueryTile * (sizeof(int32_t) + (KR > 0 ? 0 : sizeof(uint64_t)));
    const int stage = mm_stage_bytes(T::A_BYTES, T::B_BYTES, a.limbs);
    a.stages = (int)std::min<size_t>(kMaxStages, (kMaxDynSmemMm - 1024 - lists) / stage);
    const size_t smem = 1024 + (size_t)a.stages * stage + lists;
    auto kern = mm_search_kernel<F4, CL, KR>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxDynSmemMm);
    if (e != cudaSuccess) return cuda_fail(e, "mm search: cudaFuncSetAttribute");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(kThreadsMm, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CL;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = CL > 1 ? 1 : 0;
    e = cudaLaunchKernelEx(&cfg, kern, tmA, tmB, a);
    return e == cudaSuccess ? HDC_OK : cuda_fail(e, "mm search: launch");
}

template <bool F4, int CL>
int launch_mm_k(const MmOperands& op, const MmArgs& a, int dim, int grid, cudaStream_t stream) {
    if (a.k <= 8) return launch_mm<F4, CL, 8>(op, a, dim, grid, stream);
    if (a.k <= 16) return launch_mm<F4, CL, 16>(op, a, dim, grid, stream);
    return launch_mm<F4, CL, 0>(op, a, dim, grid, stream);
}

template <typename F>
int check_launch(F&& launch, const char* what) {
    launch();
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? HDC_OK : cuda_fail(e, what);
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace

int mm_f4_limbs(int64_t max_abs) {
    int64_t cover = 0;
    for (int l = 1; l <= kMaxF4Limbs; ++l) {
        cover = cover * 8 + 4;
        if (max_abs <= cover) return l;
    }
    return 0;
}

int64_t mm_f4_sum_per_dim(int64_t max_abs) {
    int64_t lower = 0;  // the most that the digits below the top one come to
    for (int l = 1; l < mm_f4_limbs(max_abs); ++l) lower = lower * 8 + 4;
    return std::max<int64_t>(1, std::max(max_abs, lower));
}

// Complete dims sum to at most |q| |r| (Cauchy-Schwarz); the K block in progress adds at most its lower digits' sum more.
double mm_f4_norm_limit(int limbs, int dim) {
    int64_t lower = 0;
    for (int l = 1; l < limbs; ++l) lower = lower * 8 + 4;
    const double room = (double)kMmMaxSum - (double)lower * std::min(dim, kMmF4Dims);
    return room > 0 ? room * room : 0;
}

int mm_begin(void* work, int64_t nq, cudaStream_t stream) {
    const cudaError_t e = cudaMemsetAsync(work, 0, head_bytes(nq), stream);
    return e == cudaSuccess ? HDC_OK : cuda_fail(e, "mm search: clear thresholds");
}

size_t mm_f4_query_bytes(int64_t nq, int dim) {
    return (size_t)((nq + kMmQueryTile - 1) / kMmQueryTile) * kMmQueryTile * n_kblocks(dim, true) * 64;
}

size_t mm_f4_ref_bytes(int64_t nr, int dim, int limbs) {
    return (size_t)((nr + 2 * kMmF4Half - 1) / (2 * kMmF4Half)) * 2 * kMmF4Half * n_kblocks(dim, true) * 64 * limbs;
}

bool mm_sums_fit(bool f4, int64_t sum_per_dim) { return sum_per_dim * (f4 ? kMmF4Dims : 16) <= kMmMaxSum; }

int mm_pack_queries(const void* d_q, bool is_f16, int64_t nq, int dim, void* out, int* status, cudaStream_t stream) {
    const int n_kb = n_kblocks(dim, true);
    const int64_t chunks = (nq + kMmQueryTile - 1) / kMmQueryTile * kMmQueryTile * n_kb * 4;
    const unsigned grid = (unsigned)((chunks + 255) / 256);
    uint8_t* o = static_cast<uint8_t*>(out);
    const bool vec = dim % 8 == 0 && aligned16(d_q);
    return check_launch([&] {
        if (is_f16) {
            const __half* q = static_cast<const __half*>(d_q);
            if (vec)
                pack_queries_kernel<__half, true><<<grid, 256, 0, stream>>>(q, nq, dim, n_kb, chunks, o, status);
            else
                pack_queries_kernel<__half, false><<<grid, 256, 0, stream>>>(q, nq, dim, n_kb, chunks, o, status);
        } else {
            const int16_t* q = static_cast<const int16_t*>(d_q);
            if (vec)
                pack_queries_kernel<int16_t, true><<<grid, 256, 0, stream>>>(q, nq, dim, n_kb, chunks, o, status);
            else
                pack_queries_kernel<int16_t, false><<<grid, 256, 0, stream>>>(q, nq, dim, n_kb, chunks, o, status);
        }
    }, "mm search: pack queries");
}

int mm_pack_refs(const int16_t* d_r, const __half* limbs16, int L16, int bits, int64_t r_pad, int64_t nr, int dim,
                 int limbs, void* out, cudaStream_t stream) {
    const int n_kb = n_kblocks(dim, true);
    const int64_t chunks = (nr + 2 * kMmF4Half - 1) / (2 * kMmF4Half) * (2 * kMmF4Half) * n_kb * 4;
    const unsigned grid = (unsigned)((chunks + 255) / 256);
    uint8_t* o = static_cast<uint8_t*>(out);
    const bool vec = dim % 8 == 0 && aligned16(limbs16 ? (const void*)limbs16 : (const void*)d_r);
    return check_launch([&] {
        if (limbs16) {
            if (vec)
                pack_refs_kernel<true, true><<<grid, 256, 0, stream>>>(nullptr, limbs16, L16, bits, r_pad, nr, dim, n_kb,
                                                                     limbs, chunks, o);
            else
                pack_refs_kernel<true, false><<<grid, 256, 0, stream>>>(nullptr, limbs16, L16, bits, r_pad, nr, dim, n_kb,
                                                                      limbs, chunks, o);
        } else {
            if (vec)
                pack_refs_kernel<false, true><<<grid, 256, 0, stream>>>(d_r, nullptr, 1, 0, 0, nr, dim, n_kb, limbs, chunks, o);
            else
                pack_refs_kernel<false, false><<<grid, 256, 0, stream>>>(d_r, nullptr, 1, 0, 0, nr, dim, n_kb, limbs, chunks, o);
        }
    }, "mm search: pack references");
}

int mm_rows_f16(const int16_t* d_v, int64_t n, int dim, int64_t ld, __half* out, MmNorms* norms,
                cudaStream_t stream) {
    return check_launch([&] {
        if (dim % 8 == 0 && aligned16(d_v))
            rows_f16_kernel<true><<<(unsigned)n, kRowThreads, 0, stream>>>(d_v, dim, ld, out, norms);
        else
            rows_f16_kernel<false><<<(unsigned)n, kRowThreads, 0, stream>>>(d_v, dim, ld, out, norms);
    }, "mm search: fp16 rows");
}

int mm_norm_max(const __half* d_v, int64_t n, int dim, MmNorms other, MmNorms* norms, cudaStream_t stream) {
    return check_launch([&] {
        norm_max_kernel<<<(unsigned)n, kRowThreads, 0, stream>>>(d_v, dim, other, norms);
    }, "mm search: largest norm");
}

int mm_rows_from_limbs(const __half* limbs16, int L16, int bits, int64_t rows, int dim, __half* out,
                       cudaStream_t stream) {
    const int64_t total = rows * dim, chunks = total / 8;
    return check_launch([&] {
        rows_from_limbs_kernel<<<(unsigned)((chunks + 255) / 256), 256, 0, stream>>>(limbs16, L16, bits, total, chunks, out);
    }, "mm search: rows from limbs");
}

int mm_limbs_max(const __half* limbs16, int L16, int bits, int64_t rows, int dim, int32_t* d_max, cudaStream_t stream) {
    const int64_t total = rows * dim, chunks = total / 8;
    const unsigned grid = (unsigned)std::min<int64_t>((chunks + 255) / 256, 8192);
    return check_launch([&] {
        limbs_max_kernel<<<grid, 256, 0, stream>>>(limbs16, L16, bits, total, chunks, d_max);
    }, "mm search: largest value");
}

int mm_norm_tables(const int64_t* d_n2, int64_t n, float* rr, double* rs, double* ri, cudaStream_t stream) {
    return check_launch([&] {
        norm_tables_kernel<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(d_n2, n, rr, rs, ri);
    }, "mm search: norm tables");
}

MmSplit mm_split_plan(const hdc_context* ctx, int64_t nq, int64_t nr, int dim, int k, bool f4, int64_t sum_per_dim) {
    MmSplit p;
    const int n = f4 ? MmTile<true, 1>::N : MmTile<false, 1>::N, n_kb = n_kblocks(dim, f4);
    const int64_t qt = (nq + kMmQueryTile - 1) / kMmQueryTile, rt = (nr + n - 1) / n;
    if (k < 1 || k > kMaxKMm || nr > kSplitRefs || qt * rt > ctx->num_sms) return p;
    if (sum_per_dim * (f4 ? kMmF4Dims : 64) > kMmMaxSum) return p;
    p.n_qtiles = (int)qt;
    p.n_rtiles = (int)rt;
    p.splits = (int)std::max<int64_t>(1, std::min<int64_t>(ctx->num_sms / (qt * rt), n_kb / kMinSplitBlocks));
    p.ldd = (int)rt * n;
    return p;
}

size_t mm_split_bytes(const MmSplit& p, int64_t nq) { return (size_t)p.splits * nq * p.ldd * sizeof(int32_t); }

template <bool F4>
static int launch_dots(hdc_context* ctx, const MmOperands& op, const MmSplit& p, DotsArgs a, int64_t nr, int dim,
                       cudaStream_t stream) {
    using T = MmTile<F4, 1>;
    CUtensorMap tmA, tmB;
    const int64_t a_rows = F4 ? (int64_t)p.n_qtiles * a.n_kb * kMmQueryTile : a.nq;
    const int64_t b_tiles = (nr + 2 * kMmF4Half - 1) / (2 * kMmF4Half);
    const int64_t b_rows = F4 ? b_tiles * a.n_kb * 2 * a.limbs * kMmF4Half : nr;
    if (!make_map(&tmA, F4, op.a, a_rows, dim, op.lda, kMmQueryTile) ||
        !make_map(&tmB, F4, op.b, b_rows, dim, op.ldb, T::ROWS))
        return fail(HDC_ERR_CUDA, "mm search: cuTensorMapEncodeTiled failed");
    const int stage = mm_stage_bytes(T::A_BYTES, T::B_BYTES, a.limbs);
    a.stages = (int)std::min<size_t>(kMaxStages, (kMaxDynSmemMm - 1024) / stage);
    const cudaError_t e = cudaFuncSetAttribute(mm_dots_kernel<F4>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)kMaxDynSmemMm);
    if (e != cudaSuccess) return cuda_fail(e, "mm search: cudaFuncSetAttribute");
    return check_launch([&] {
        mm_dots_kernel<F4><<<(unsigned)(p.n_qtiles * p.n_rtiles * p.splits), kDotThreads, 1024 + (size_t)a.stages * stage,
                             stream>>>(tmA, tmB, a);
    }, "mm search: split launch");
}

int mm_split_search(hdc_context* ctx, const MmOperands& op, const MmSplit& p, int64_t nq, int64_t nr, int dim, int k,
                    int mode, void* parts, float* d_score, int32_t* d_idx, double* d_cos,
                    int64_t* d_dot, int32_t shape[5], cudaStream_t stream) {
    DotsArgs a{};
    a.nq = nq;
    a.n_kb = n_kblocks(dim, op.f4);
    const int64_t most = std::max<int64_t>(1, kMmMaxSum / (op.sum_per_dim * (op.f4 ? kMmF4Dims : 64)));
    a.kb_per_seg = (int)std::min<int64_t>(a.n_kb, most);
    a.limbs = op.f4 ? op.limbs : 1;
    a.n_rtiles = p.n_rtiles;
    a.splits = p.splits;
    a.ldd = p.ldd;
    a.withhold = ctx->test_withhold_loads == 1;
    a.parts = static_cast<int32_t*>(parts);
    a.status = ctx->d_status;
    a.wait_cycles = ctx->wait_cycles > 0 ? ctx->wait_cycles : tc::kWaitCycles;
    const int st = op.f4 ? launch_dots<true>(ctx, op, p, a, nr, dim, stream) : launch_dots<false>(ctx, op, p, a, nr, dim, stream);
    if (st != HDC_OK) return st;
    if (shape) {
        shape[0] = 1;
        shape[1] = p.n_qtiles;
        shape[2] = p.n_rtiles;
        shape[3] = 0;
    }
    const size_t smem = (size_t)nr * (sizeof(uint64_t) + sizeof(int32_t));
    auto kern = nr <= 512 ? mm_select_kernel<128> : mm_select_kernel<256>;  // four references a thread, if there are as many
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kSplitRefs * (int)(sizeof(uint64_t) + sizeof(int32_t)));
    if (e != cudaSuccess) return cuda_fail(e, "mm search: cudaFuncSetAttribute");
    return check_launch([&] {
        kern<<<(unsigned)nq, nr <= 512 ? 128 : 256, smem, stream>>>(a.parts, p.splits, nq, (int)nr, p.ldd, op.qn, op.rr, op.rs,
                                                                   op.ri, k, mode, d_score, d_idx, d_cos, d_dot);
    }, "mm search: select launch");
}

int mm_rows2_f16(const int16_t* d_q, int64_t nq, const int16_t* d_r, int64_t nr, int dim, int64_t ld, __half* out_q,
                 __half* out_r, const int64_t* d_rn, float* rr, double* rs, double* ri, cudaStream_t stream) {
    return check_launch([&] {
        if (dim % 8 == 0 && aligned16(d_q) && aligned16(d_r))
            rows2_f16_kernel<true><<<(unsigned)(nq + nr), kRowThreads, 0, stream>>>(d_q, nq, d_r, dim, ld, out_q, out_r, d_rn,
                                                                                    rr, rs, ri);
        else
            rows2_f16_kernel<false><<<(unsigned)(nq + nr), kRowThreads, 0, stream>>>(d_q, nq, d_r, dim, ld, out_q, out_r,
                                                                                     d_rn, rr, rs, ri);
    }, "mm search: fp16 rows");
}

size_t mm_list_bytes(const hdc_context* ctx, int64_t nq, int64_t nr, int dim, int k, bool f4, int limbs) {
    const MmPlan p = mm_plan(ctx->num_sms, nq, nr, dim, f4, limbs);
    return head_bytes(nq) + (size_t)p.S * nq * k * (sizeof(uint64_t) + sizeof(int64_t));
}

int mm_search(hdc_context* ctx, const MmOperands& op, int64_t nq, int64_t nr, int64_t r0, int64_t plan_nr, int dim, int k,
              int mode, void* work, bool first, int32_t shape[5], cudaStream_t stream) {
    if (k < 1 || k > kMaxKMm) return fail(HDC_ERR_INVALID, "mm search: k must be in 1..32");
    const MmPlan p = mm_plan(ctx->num_sms, nq, plan_nr, dim, op.f4, op.limbs);
    MmArgs a{};
    a.nq = nq;
    a.nr = nr;
    a.r0 = r0;
    a.k = k;
    a.mode = mode;
    a.limbs = op.f4 ? op.limbs : 1;
    a.n_kb = n_kblocks(dim, op.f4);
    const int64_t kb_dims = op.f4 ? kMmF4Dims : 64;
    const int64_t most = std::max<int64_t>(1, kMmMaxSum / (op.sum_per_dim * kb_dims));  // K blocks of a segment
    const int64_t segs = (a.n_kb + most - 1) / most;
    a.kb_per_seg = (int)((a.n_kb + segs - 1) / segs);
    if (!op.f4 && op.sum_per_dim * 64 > kMmMaxSum) a.mma_per_seg = op.sum_per_dim * 32 > kMmMaxSum ? 1 : 2;
    a.n_qtiles = p.n_qtiles;
    const int n = p.CL == 2 ? (op.f4 ? MmTile<true, 2>::N : MmTile<false, 2>::N)
                            : (op.f4 ? MmTile<true, 1>::N : MmTile<false, 1>::N);
    a.n_rtiles = (int)((nr + n - 1) / n);
    a.G = p.G;
    a.S = p.S;
    a.n_groups = p.n_groups;
    a.t_stride = (ctx->tc_scatter >= 0 ? ctx->tc_scatter : tc_default_scatter()) ? scattered_stride(a.n_rtiles) : 1;
    a.carry = first ? 0 : 1;
    a.withhold = ctx->test_withhold_loads == 1;
    a.qn = op.qn;
    a.rr = op.rr;
    a.rs = op.rs;
    a.ri = op.ri;
    a.kth = reinterpret_cast<uint32_t*>(static_cast<unsigned long long*>(work) + kMmWorkWords);
    a.ws_key = reinterpret_cast<uint64_t*>(static_cast<uint8_t*>(work) + head_bytes(nq));
    a.ws_dot = reinterpret_cast<int64_t*>(a.ws_key + (size_t)p.S * nq * k);
    a.status = ctx->d_status;
    a.wait_cycles = ctx->wait_cycles > 0 ? ctx->wait_cycles : tc::kWaitCycles;
    const bool several = segs > 1 || a.mma_per_seg;
    if (several && op.one_segment) a.kb_per_seg = a.n_kb;
    if (several && !op.one_segment && op.q_norms) {
        a.q_norms = op.q_norms;
        a.r_norms = op.r_norms;
        a.norm_limit = op.f4 ? mm_f4_norm_limit(op.limbs, dim) : (double)kMmMaxSum * (double)kMmMaxSum;
    }
    if (shape) {
        shape[0] = p.CL;
        shape[1] = p.G;
        shape[2] = p.S;
        shape[3] = p.CL == 2 ? 1 : 0;
    }
    const int grid = p.G * p.S;
    if (op.f4)
        return p.CL == 2 ? launch_mm_k<true, 2>(op, a, dim, grid, stream) : launch_mm_k<true, 1>(op, a, dim, grid, stream);
    return p.CL == 2 ? launch_mm_k<false, 2>(op, a, dim, grid, stream) : launch_mm_k<false, 1>(op, a, dim, grid, stream);
}

int mm_finish(hdc_context* ctx, int64_t nq, int64_t plan_nr, int64_t nr_total, int dim, int k, bool f4, int limbs,
              const int64_t* d_qn, const int64_t* d_rn, void* work, float* d_score, int32_t* d_idx, double* d_cos,
              int64_t* d_dot, cudaStream_t stream) {
    const MmPlan p = mm_plan(ctx->num_sms, nq, plan_nr, dim, f4, limbs);
    const uint64_t* key = reinterpret_cast<const uint64_t*>(static_cast<const uint8_t*>(work) +
                                                            head_bytes(nq));
    const int64_t* dot = reinterpret_cast<const int64_t*>(key + (size_t)p.S * nq * k);
    return check_launch([&] {
        mm_merge_kernel<<<(unsigned)((nq + kMergeWarps - 1) / kMergeWarps), 32 * kMergeWarps, 0, stream>>>(
            key, dot, p.S, nq, k, d_qn, d_rn, nr_total, d_score, d_idx, d_cos, d_dot);
    }, "mm search: merge");
}

}  // namespace hdc
