// Tensor-core scoring of TurboQuantProd keys (d = 128, 1..4 code bits) on B200.
//
//   score(q, key) = norm * ( (R q) . codebook[codes]  +  alpha * rnorm * ((S q) . signs) )
//
// is a small GEMM per tile of 128 keys: the keys are the M side, the (at most 32) queries the N side
// and the 128 coordinates the K side.  Per tile:
//
//   bulk copy (1 thread)   packed codes, sign words and norms of 128 keys -> smem ring (plain 1-D bulk copies)
//   expanders (16 warps)   two threads per key: turn packed codes into fp16 operands and store
//                          them into tensor memory with tcgen05.st (lane = key).  Two codes at a time
//                          index a lookup table of (hi pair, lo pair) half2 values -- centroid * 2^10
//                          split into fp16 hi + lo -- replicated per lane in smem so the lookups are
//                          free of bank conflicts; two sign bits become one half2 of +-1 with a shift
//                          and a logic op (the sign layout keeps them 16 bits apart for that).
//   MMA (1 thread)         D1 = C_hi Q_hi + C_hi Q_lo + C_lo Q_hi,  D2 = Sg P_hi + Sg P_lo  (kind::f16,
//                          fp32 accumulators in TMEM, one column per query each); Q = R q and P = S q are rotated /
//                          projected, scaled by a power of two and split into fp16 hi + lo once per call by a
//                          small preparation kernel, and live in smem as the B operand.
//   epilogue (8 warps)     one thread per key: tcgen05.ld both accumulators, apply the per-query
//                          descale, alpha * rnorm and norm (fma.rn.f32x2), stage the tile for a bulk tensor store.
//
// Expanders and epilogue warps come in two groups that take tiles in turn (a pass of 64 queries: the epilogue groups
// take halves of the queries instead): what a warp does for a tile is a chain of waits, loads and a round trip to tensor
// memory that is longer than a tile may take.  Before -- every warp at every tile, hi and lo products in columns of their own,
// which the epilogue had to fetch and add and which left room for one accumulator at 32 queries -- a tile of 32 queries took
// 3,600 cycles (106 us per 32 x 1,048,576 scores).
//
// A second kernel selects the per-query top-k from a score matrix with a rising threshold and a
// bitonic prune (the same scheme as the general kernel in tq_score.cu), one block per row segment.
#include "tq_common.cuh"
#include "tq_ptx.cuh"
#include "tq_topk.cuh"
#include "tq_filter.cuh"

#include <cuda.h>
#include <math.h>
#include <math_constants.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>

namespace {

using namespace tqptx;
using namespace tqtopk;

constexpr int D = 128;
constexpr int kTileKeys = 128;
constexpr int kExpWarps = 16, kEpiWarps = 8;      // behind the bulk-copy and the MMA warp; two groups each
constexpr int kFirstExpWarp = 2, kFirstEpiWarp = kFirstExpWarp + kExpWarps;
constexpr int kThreads = (2 + kExpWarps + kEpiWarps) * 32;
constexpr int kPendKeys = 64;                     // survivors a warp stages in candidate mode
constexpr int kMaxStages = 8;
constexpr float kCentScale = 1024.f;
constexpr int kRowBytesB = D * 2;  // one query row of one fp16 operand matrix
constexpr int kPrepSmemBytes = D * D * 4;  // the matrix that a block of the preparation kernel stages
constexpr int kEpiBarrier = 1;     // named barriers of the epilogue groups: this one and the next

// Prepared queries of one group: per half of the coordinates (two halves of 128 for d = 256, one otherwise) the four
// fp16 operand matrices q_hi, q_lo, p_hi, p_lo, then one (1 / scale) pair per query.
__host__ __device__ constexpr int prep_group_bytes(int qpad, int halves = 1) { return halves * 4 * qpad * kRowBytesB + 2 * qpad * 4; }

struct ScoreTcArgs {
    const uint32_t* codes;
    const uint32_t* signs;
    const float* rnorms;
    const float* norms;
    const unsigned char* prep;    // [groups][prep_group_bytes]
    const float* codebook;
    int64_t keys_per_group;       // rows between the first keys of consecutive groups
    int64_t key_off;              // first key of every group handled by this launch
    int64_t key_cnt;              // keys per group handled by this launch
    int64_t tiles_per_group, total_tiles;
    int nq;                       // live queries (<= QPAD)
    int64_t out_group_stride;     // floats between groups in `scores`
    int64_t out_row_stride;       // floats between query rows
    float* scores;                // points at (group 0, first query of this pass, key_off)
    int tile_store;               // 1: score tiles leave through shared memory and a bulk tensor store (tmap_out)
    int norms_bulk;               // 1: norms and residual norms travel with the packed rows through the key ring
    int tile_stride;              // tile kt of a group covers keys [kt * tile_stride * 128, +128): > 1 scores a sample of the tiles
    // Top-k without a score matrix (candidate mode): a score that reaches its query's threshold is appended to that
    // query's candidate list (sortable key: score bits | row) instead of being written anywhere else.
    int fused;                    // 0: score matrix; 1: candidates through a staging list; 2: the sampled pass (every score, fixed slots)
    int qpg_total, q0;            // queries per group over all passes, first query of this pass
    const float* thr;             // [groups][qpg_total] lower bound of the k-th best score so far (-inf: none)
    unsigned int* cnt;            // [groups][qpg_total] entries appended to each list
    unsigned long long* cand;     // [groups][qpg_total][cand_cap]
    int64_t cand_cap;
    const unsigned int* dyn_keys; // keys that are really there (one group; tiles behind them are skipped); null: key_cnt
    const unsigned int* run_if;   // the launch does nothing when this word is zero; null: always runs
    float alpha;
    unsigned long long* status;
    int wait_kcycles;             // limit of one bounded wait, in units of 1024 cycles
};

enum {
    SB_K_FULL = 0,      // [8]
    SB_K_EMPTY = 8,     // [8]
    SB_A_FULL = 16,     // [2]: one operand buffer per group of expanders
    SB_A_EMPTY = 18,    // [2]
    SB_D_FULL = 20,     // [4]
    SB_D_EMPTY = 24,    // [4]
    SB_B_FULL = 28,     // [2]
    SB_B_EMPTY = 30,    // [2]
    SB_COUNT = 32
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// Shared memory -> global, one box of a 3-D tensor map (keys, queries of the pass, groups); parts of the box
// outside the tensor are not written.
__device__ __forceinline__ void tensor_store_3d(const CUtensorMap* map, uint32_t src, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];"
                 ::"l"(map), "r"(src), "r"(c0), "r"(c1), "r"(c2)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// Wait until all but the newest `N` bulk groups of this thread have finished reading shared memory.
template <int N> __device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}

// DR is the dimension of the vectors.  The operand layouts are those of d = 128 in every case: for d = 64 the upper
// half of every key is absent (its expander warps idle, the contractions stop after DR / 16 k-blocks); for d = 256 a
// tile of keys passes through the operand buffers as two halves of 128 coordinates, one after the other, whose
// contractions add up in the same accumulators (the prepared queries of a group then fill 64 KB, so that only one
// group's are resident).
template <int BITS, int QPAD, int DR>
struct ScoreSmem {
    static_assert(QPAD <= 32 || DR <= 128, "a pass of 64 queries exists for d <= 128");
    static constexpr int kHalves = DR == 256 ? 2 : 1;
    static constexpr int kSub = DR / kHalves / 64;        // chunks of 32 coordinates per expander thread and half
    static constexpr int kBBufs = (DR == 256 || QPAD == 64) ? 1 : 2;     // 64 KB of prepared queries: one group resident
    static constexpr int kDBufs = 64 / QPAD;              // accumulators: 2 * QPAD of the 128 columns behind the operand buffers
    static constexpr int kQT = QPAD < 32 ? QPAD : 32;     // queries of an epilogue thread
    static constexpr bool kSplitQ = QPAD == 64;           // the epilogue groups split the queries (else they take tiles in turn)
    static constexpr int kPrepBytes = prep_group_bytes(QPAD, kHalves);
    static constexpr int kLutEntries = 1 << (2 * BITS);
    static constexpr int kLutBytes = kLutEntries * 32 * 8;
    static constexpr int kCodeRowBytes = DR * BITS / 8;
    static constexpr int kSignRowBytes = DR / 8;
    static constexpr int kNormOff = kTileKeys * (kCodeRowBytes + kSignRowBytes);   // norms, then residual norms, of the tile's keys
    static constexpr int kStageBytes = kNormOff + 2 * kTileKeys * 4;
    static constexpr int kBBytes = (kPrepBytes + 127) & ~127;
    static constexpr int kOutBytes = kQT * kTileKeys * 4;           // one staged box of scores [query][key] per epilogue group
    // candidate mode, in place of the boxes: per epilogue warp 16 x 32 parked scores and the staged survivors
    static constexpr int kCandBytes = kEpiWarps * (16 * 32 * 4 + kPendKeys * 12);
    static constexpr int kOutArea = 2 * kOutBytes > kCandBytes ? 2 * kOutBytes : kCandBytes;
    static constexpr int kMisc = 512;
    static constexpr int kFixed = kLutBytes + kBBufs * kBBytes + kOutArea + kMisc;
    static constexpr int kFit = (226 * 1024 - kFixed) / kStageBytes;
    static constexpr int kStages = kFit < kMaxStages ? kFit : kMaxStages;
    static_assert(kStages >= 3, "key ring too short");
    static constexpr int off_lut = 0;
    static constexpr int off_b = off_lut + kLutBytes;
    static constexpr int off_out = off_b + kBBufs * kBBytes;
    static constexpr int off_ring = off_out + kOutArea;
    static constexpr int off_misc = off_ring + kStages * kStageBytes;
    static constexpr int total = off_misc + kMisc;
    static_assert(off_ring % 128 == 0 && off_misc % 16 == 0 && off_out % 128 == 0, "alignment");
};

// two words of a ring stage, read exactly once
__device__ __forceinline__ void lds_once_u2(uint32_t& x, uint32_t& y, const volatile uint32_t* p) {
    asm volatile("ld.volatile.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(smem_u32(const_cast<const uint32_t*>(p))));
}

// CAND: candidate mode (top-k without a score matrix) is a kernel of its own, so that the matrix kernel carries none
// of its registers and code.
template <int BITS, int QPAD, int DR, bool CAND>
__global__ void __launch_bounds__(kThreads, 1)
score_tc_kernel(const __grid_constant__ CUtensorMap tmap_out, const __grid_constant__ ScoreTcArgs a) {
    static_assert(DR == 256 || DR == 128 || DR == 64, "written for d = 256, 128 and 64");
    using L = ScoreSmem<BITS, QPAD, DR>;
    constexpr int kHalves = L::kHalves, kBBufs = L::kBBufs, kDBufs = L::kDBufs, kStages = L::kStages, kQT = L::kQT;
    constexpr int kDH = DR / kHalves;            // coordinates per pass through the operand buffers
    extern __shared__ __align__(128) unsigned char smem[];     // (an address the compiler knows: the table lookups fold it in)
    const uint32_t smem_base = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::off_misc);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + SB_COUNT);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t bar0 = smem_u32(bars);
    auto BAR = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (a.run_if || a.dyn_keys) tq_grid_wait();      // words of kernels before
    if (a.run_if && *a.run_if == 0u) return;
    const uint32_t total_tiles = (uint32_t)(a.dyn_keys ? ((int64_t)*a.dyn_keys + kTileKeys - 1) / kTileKeys : a.total_tiles);
    const uint32_t tiles_per_group = (uint32_t)a.tiles_per_group;

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(BAR(SB_K_FULL + i), 1);
            // one group of expanders (d = 256: both) and the epilogue warps that work on the tile read a stage
            mbar_init(BAR(SB_K_EMPTY + i), (kHalves == 2 ? kExpWarps : kExpWarps / 2) + (a.norms_bulk ? (L::kSplitQ ? kEpiWarps : kEpiWarps / 2) : 0));
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(BAR(SB_A_FULL + i), kExpWarps / 2);
            mbar_init(BAR(SB_A_EMPTY + i), 1);
            mbar_init(BAR(SB_B_FULL + i), 1);
            mbar_init(BAR(SB_B_EMPTY + i), 1 + kEpiWarps);      // last MMA of the group + every epilogue warp
        }
        for (int i = 0; i < kDBufs; ++i) {
            mbar_init(BAR(SB_D_FULL + i), 1);
            mbar_init(BAR(SB_D_EMPTY + i), L::kSplitQ ? kEpiWarps : kEpiWarps / 2);
        }
        abort_flag[0] = 0;
        abort_flag[1] = a.wait_kcycles;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {   // pair lookup table: entry e = (code0 | code1 << BITS) -> (half2 hi(c0), hi(c1)), (half2 lo(c0), lo(c1)), a copy per lane
        uint2* lut = reinterpret_cast<uint2*>(smem + L::off_lut);
        for (int i = threadIdx.x; i < L::kLutEntries * 32; i += kThreads) {
            const int e = i >> 5;
            const float c0 = __ldg(a.codebook + (e & ((1 << BITS) - 1))) * kCentScale;
            const float c1 = __ldg(a.codebook + (e >> BITS)) * kCentScale;
            const __half2 h = __floats2half2_rn(c0, c1);
            const float2 hf = __half22float2(h);
            uint2 v;
            v.x = *reinterpret_cast<const uint32_t*>(&h);
            v.y = pack_half2(c0 - hf.x, c1 - hf.y);
            lut[i] = v;
        }
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    tq_grid_wait();         // the prepared queries; so far only constants of the plan have been read
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    // contiguous tile range of this CTA, so that it rarely changes group
    const uint32_t t0 = (uint32_t)((uint64_t)total_tiles * blockIdx.x / gridDim.x);
    const uint32_t t1 = (uint32_t)((uint64_t)total_tiles * (blockIdx.x + 1) / gridDim.x);
    const uint32_t g_first = t0 / tiles_per_group;
    // TMEM: two operand buffers of 192 columns (C_hi | C_lo | Sg), then the accumulators (D1 | D2), QPAD columns each
    constexpr uint32_t kBufCols = 192, kColHi = 0, kColLo = 64, kColSg = 128;
    constexpr uint32_t kColD = 2 * kBufCols, kDCols = 2 * QPAD;
    static_assert(kColD + kDBufs * kDCols <= 512, "tensor memory plan");

    if (warp == 0) {
        if (lane == 0) {
            uint32_t issued = 0, gcount = 0;
            uint32_t g = g_first, kt = t0 - g * tiles_per_group;
            for (uint32_t t = t0; t < t1; ++t, ++kt) {
                if (kt == tiles_per_group) { kt = 0; ++g; }
                if (g - g_first == gcount) {
                    const int bb = kBBufs == 2 ? (int)(gcount & 1) : 0;
                    if (!mbar_wait(BAR(SB_B_EMPTY + bb), ((kBBufs == 2 ? gcount >> 1 : gcount) & 1) ^ 1u, abort_flag)) break;
                    mbar_arrive_expect_tx(BAR(SB_B_FULL + bb), L::kPrepBytes);
                    bulk_load(smem_base + L::off_b + bb * L::kBBytes, a.prep + (size_t)g * L::kPrepBytes, L::kPrepBytes, BAR(SB_B_FULL + bb));
                    ++gcount;
                }
                const uint32_t i = t - t0;
                const int s = (int)(i % kStages);
                if (!mbar_wait(BAR(SB_K_EMPTY + s), ((i / kStages) & 1) ^ 1u, abort_flag)) break;
                const int64_t k0 = (int64_t)kt * a.tile_stride * kTileKeys;      // first key of the tile within this launch's range
                int64_t valid = a.key_cnt - k0;
                if (valid > kTileKeys) valid = kTileKeys;
                const int64_t row0 = (int64_t)g * a.keys_per_group + a.key_off + k0;
                const uint32_t cb = (uint32_t)valid * L::kCodeRowBytes, sb = (uint32_t)valid * L::kSignRowBytes;
                const unsigned char* csrc = reinterpret_cast<const unsigned char*>(a.codes) + row0 * L::kCodeRowBytes;
                const unsigned char* ssrc = reinterpret_cast<const unsigned char*>(a.signs) + row0 * L::kSignRowBytes;
                unsigned char* stage = smem + L::off_ring + s * L::kStageBytes;
                // a ragged last tile of 8- or 24-byte rows need not end on a 16-byte multiple: the bulk copies take
                // the multiple, plain loads the few bytes behind it
                copy_tail_words(stage, csrc, cb);
                copy_tail_words(stage + kTileKeys * L::kCodeRowBytes, ssrc, sb);
                const uint32_t nb = a.norms_bulk ? (uint32_t)valid * 4u : 0u;
                if (nb) {
                    copy_tail_words(stage + L::kNormOff, reinterpret_cast<const unsigned char*>(a.norms + row0), nb);
                    copy_tail_words(stage + L::kNormOff + kTileKeys * 4, reinterpret_cast<const unsigned char*>(a.rnorms + row0), nb);
                }
                mbar_arrive_expect_tx(BAR(SB_K_FULL + s), (cb & ~15u) + (sb & ~15u) + 2 * (nb & ~15u));
                const uint32_t dst = smem_base + L::off_ring + s * L::kStageBytes;
                if (cb & ~15u) bulk_load(dst, csrc, cb & ~15u, BAR(SB_K_FULL + s));
                if (sb & ~15u) bulk_load(dst + kTileKeys * L::kCodeRowBytes, ssrc, sb & ~15u, BAR(SB_K_FULL + s));
                if (nb & ~15u) {
                    bulk_load(dst + L::kNormOff, a.norms + row0, nb & ~15u, BAR(SB_K_FULL + s));
                    bulk_load(dst + L::kNormOff + kTileKeys * 4, a.rnorms + row0, nb & ~15u, BAR(SB_K_FULL + s));
                }
                issued = i + 1;
            }
            if (*abort_flag) {
                // copies armed above may still be on their way into this block's shared memory
                for (uint32_t ii = issued > kStages ? issued - kStages : 0; ii < issued; ++ii)
                    mbar_drain(BAR(SB_K_FULL + (int)(ii % kStages)), (ii / kStages) & 1);
                for (uint32_t gg = gcount > kBBufs ? gcount - kBBufs : 0; gg < gcount; ++gg)
                    mbar_drain(BAR(SB_B_FULL + (kBBufs == 2 ? (int)(gg & 1) : 0)), (kBBufs == 2 ? gg >> 1 : gg) & 1);
            }
        }
    } else if (warp == 1) {
        // The whole warp walks the tiles and waits; one elected lane issues, with every operand computed from
        // warp-uniform values (a single lane of a diverged warp pays about 64 cycles per instruction).
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(QPAD >> 3) << 17) | ((uint32_t)(kTileKeys >> 4) << 24);
        const uint32_t lbo = 128, sbo = (D / 8) * 128;
        uint32_t g = g_first, kt = t0 - g * tiles_per_group, gcount = 0;
        int bb = 0;
        uint64_t dq = 0;                // descriptor of q_hi; q_lo, p_hi and p_lo follow, QPAD rows each
        constexpr uint64_t kMat = (uint64_t)(QPAD * kRowBytesB >> 4);
        bool go = true;
        for (uint32_t t = t0; t < t1 && go; ++t, ++kt) {
            if (kt == tiles_per_group) { kt = 0; ++g; }
            const uint32_t i = t - t0;
            if (g - g_first == gcount) {
                bb = kBBufs == 2 ? (int)(gcount & 1) : 0;
                if (!warp_wait(BAR(SB_B_FULL + bb), (kBBufs == 2 ? gcount >> 1 : gcount) & 1, abort_flag)) break;
                ++gcount;
                dq = make_smem_desc(smem_base + L::off_b + bb * L::kBBytes, lbo, sbo);
            }
            const int db = (int)(i % kDBufs);
            const uint32_t d1 = tm + kColD + db * kDCols, d2 = d1 + QPAD;
            const bool last_of_group = t + 1 == t1 || kt + 1 == tiles_per_group;
            // operand buffers of the tile: the one of its group of expanders, or both, and which filling of them
            const int b0 = kHalves == 2 ? 0 : (int)(i & 1);
            const uint32_t use = kHalves == 2 ? i : i >> 1;
            go = warp_wait(BAR(SB_A_FULL + b0), use & 1u, abort_flag) &&
                 (kHalves == 1 || warp_wait(BAR(SB_A_FULL + 1), use & 1u, abort_flag)) &&
                 warp_wait(BAR(SB_D_EMPTY + db), ((i / kDBufs) & 1) ^ 1u, abort_flag);
            if (!go) break;
            tc_fence_after();
            if (elect_one()) {
                // The products with a lo part come first: the tensor pipe truncates its sums at every instruction, by a share of
                // what they have grown to, and so the small products cost nothing (all three products of a k-block in turn:
                // 1.3 to 1.5 times the error of sums of their own for the lo parts; so 0.7 to 0.9 times).  Rolled up, the loops
                // issue too slowly (32 x 1,048,576 scores at d = 128: 80 us, unrolled by eight 66).
                // The start-address field of a descriptor counts 16-byte units: one k-block is two core matrices further, the
                // operand matrices of the second half of the coordinates follow those of the first.
                constexpr uint64_t kBlock = 2 * 128 >> 4;
#pragma unroll 8
                for (int kb = 0; kb < DR / 16; ++kb) {
                    const int h = kb / (kDH / 16), k = kb % (kDH / 16);
                    const uint32_t buf = tm + (b0 + h) * kBufCols + k * 8;
                    const uint64_t qh = dq + (uint64_t)h * 4 * kMat + k * kBlock;
                    if (kb == 0) {
                        mma_ts_first(d1, buf + kColHi, qh + kMat, kIdesc);
                        mma_ts_first(d2, buf + kColSg, qh + 3 * kMat, kIdesc);
                    } else {
                        mma_ts_acc(d1, buf + kColHi, qh + kMat, kIdesc);
                        mma_ts_acc(d2, buf + kColSg, qh + 3 * kMat, kIdesc);
                    }
                    mma_ts_acc(d1, buf + kColLo, qh, kIdesc);
                }
#pragma unroll 8
                for (int kb = 0; kb < DR / 16; ++kb) {
                    const int h = kb / (kDH / 16), k = kb % (kDH / 16);
                    const uint32_t buf = tm + (b0 + h) * kBufCols + k * 8;
                    const uint64_t qh = dq + (uint64_t)h * 4 * kMat + k * kBlock;
                    mma_ts_acc(d1, buf + kColHi, qh, kIdesc);
                    mma_ts_acc(d2, buf + kColSg, qh + 2 * kMat, kIdesc);
                    if (kHalves == 2 && k + 1 == kDH / 16) mma_commit(BAR(SB_A_EMPTY + h));
                }
                mma_commit(BAR(SB_D_FULL + db));
                if (kHalves == 1) mma_commit(BAR(SB_A_EMPTY + b0));
                if (last_of_group) mma_commit(BAR(SB_B_EMPTY + bb));
            }
            __syncwarp();
        }
    } else if (warp < kFirstEpiWarp) {
        // ---- expanders: two threads per key, every second tile (d = 256: every tile, a half of its coordinates) --------
        const int ew = warp - kFirstExpWarp, group = ew >> 3, part = (ew >> 2) & 1;
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        constexpr uint32_t kPairMask = ((1u << (2 * BITS)) - 1u) << 8;     // a pair of codes, in place as a table row of 256 bytes
        const uint32_t lane8 = lane * 8;
        constexpr uint32_t t_step = kHalves == 2 ? 1u : 2u;
        for (uint32_t t = t0 + (kHalves == 2 ? 0 : group); t < t1; t += t_step) {
            const uint32_t i = t - t0;
            const int s = (int)(i % kStages);
            bool fail = !mbar_wait(BAR(SB_K_FULL + s), (i / kStages) & 1, abort_flag);
            const unsigned char* stage = smem + L::off_ring + s * L::kStageBytes;
            {
                const int h = kHalves == 2 ? group : 0;
                uint32_t w[L::kSub * BITS + 1], sw[L::kSub];
                {
                    // volatile: executed once, before the stage is released (a plain load may be repeated behind it)
                    const int chunk = (h * 2 + part) * L::kSub;
                    const volatile uint32_t* cw = reinterpret_cast<const volatile uint32_t*>(stage + row * L::kCodeRowBytes) + chunk * BITS;
                    const volatile uint32_t* sg = reinterpret_cast<const volatile uint32_t*>(stage + kTileKeys * L::kCodeRowBytes + row * L::kSignRowBytes) + chunk;
                    if constexpr (L::kSub == 2) {
#pragma unroll
                        for (int k = 0; k < 2 * BITS; k += 2) lds_once_u2(w[k], w[k + 1], cw + k);
                        lds_once_u2(sw[0], sw[1], sg);
                    } else {
#pragma unroll
                        for (int k = 0; k < BITS; ++k) w[k] = cw[k];
                        sw[0] = sg[0];
                    }
                    w[L::kSub * BITS] = 0;
                }
                __threadfence_block();   // every lane's loads from the stage are performed before the stage is released
                __syncwarp();
                if (lane == 0 && !fail) mbar_arrive(BAR(SB_K_EMPTY + s));
                const uint32_t use = kHalves == 2 ? i : i >> 1;
                const uint32_t abase = tmem + lane_addr + group * kBufCols + part * L::kSub * 16;
#pragma unroll
                for (int c = 0; c < L::kSub; ++c) {
                    uint32_t hi[16], lo[16], sg[16];
#pragma unroll
                    for (int p = 0; p < 16; ++p) {
                        const int bit = (c * 16 + p) * 2 * BITS, wi = bit >> 5, sh = bit & 31;
                        uint32_t e;      // the pair's bits moved to bit 8
                        if (sh + 2 * BITS > 32) e = __funnelshift_r(w[wi], w[wi + 1], sh) << 8;
                        else if (sh >= 8) e = w[wi] >> (sh - 8);
                        else e = w[wi] << (8 - sh);
                        const uint2 v = *reinterpret_cast<const uint2*>(smem + L::off_lut + ((e & kPairMask) | lane8));
                        hi[p] = v.x;
                        lo[p] = v.y;
                        // the sign word covers the 32 coordinates of the chunk; pair p: bits p, 16+p
                        sg[p] = ((~sw[c] << (15 - p)) & 0x80008000u) | 0x3c003c00u;
                    }
                    if (c == 0) {        // the first chunk is expanded while the buffer may still be in use
                        if (!mbar_wait(BAR(SB_A_EMPTY + group), (use & 1u) ^ 1u, abort_flag)) fail = true;
                        tc_fence_after();
                    }
                    tmem_st16(abase + kColHi + c * 16, hi);
                    tmem_st16(abase + kColLo + c * 16, lo);
                    tmem_st16(abase + kColSg + c * 16, sg);
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(SB_A_FULL + group));
            }
        }
    } else {
        // ---- epilogue: one thread per key ---------------------------------------------------------------
        const int ew = warp - kFirstEpiWarp, group = ew >> 2;
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        const int q_mine = L::kSplitQ ? group * kQT : 0;       // first query of this thread
        const uint32_t t_step = L::kSplitQ ? 1u : 2u;
        const bool leader = quarter == (kFirstEpiWarp & 3) && lane == 0;     // issues the group's tensor stores
        float* box = reinterpret_cast<float*>(smem + L::off_out + group * L::kOutBytes);
        // norm and residual norm of this thread's key when they do not ride in the key ring: fetched one tile of this
        // warp ahead of their use (a load issued in the tile that needs it would stall the stores for a full trip to memory)
        auto fetch_norms = [&](uint32_t t, float& n_out, float& r_out) {
            const uint32_t gg = t / tiles_per_group;
            const int64_t key_n = (int64_t)(t - gg * tiles_per_group) * a.tile_stride * kTileKeys + row;
            const bool live_n = t < t1 && key_n < a.key_cnt;
            const int64_t grow_n = (int64_t)gg * a.keys_per_group + a.key_off + key_n;
            n_out = live_n ? __ldg(a.norms + grow_n) : 0.f;
            r_out = live_n ? __ldg(a.rnorms + grow_n) : 0.f;
        };
        // candidate mode: 16 x 32 parked scores and the staged survivors (keys, then the numbers of their lists) of this warp
        float* parked = reinterpret_cast<float*>(smem + L::off_out) + ew * 16 * 32 + lane;
        unsigned long long* pend = reinterpret_cast<unsigned long long*>(smem + L::off_out + kEpiWarps * 16 * 32 * 4) + ew * kPendKeys;
        uint32_t* pend_list = reinterpret_cast<uint32_t*>(smem + L::off_out + kEpiWarps * (16 * 32 * 4 + kPendKeys * 8)) + ew * kPendKeys;
        int n_pend = 0;
        auto flush = [&]() {
            __syncwarp();
            for (int e = lane; e < n_pend; e += 32) {
                const int64_t l = pend_list[e];
                const int64_t gp = (int64_t)atomicAdd(a.cnt + l, 1u);
                if (gp < a.cand_cap) a.cand[l * a.cand_cap + gp] = pend[e];
            }
            __syncwarp();
            n_pend = 0;
        };
        const uint32_t t_begin = t0 + (L::kSplitQ ? 0u : (uint32_t)group);
        float nrm_next = 0.f, rn_next = 0.f;
        if (t_begin < t1 && !a.norms_bulk) fetch_norms(t_begin, nrm_next, rn_next);
        // Key groups whose prepared queries this warp is done with: it says so once for each, in order, after it has seen
        // that they were there at all (a warp may have no tile of a short group).
        uint32_t g_done = g_first;
        auto release_groups = [&](uint32_t up_to) {
            for (; g_done < up_to; ++g_done) {
                const uint32_t c = g_done - g_first;
                const int bb = kBBufs == 2 ? (int)(c & 1) : 0;
                mbar_wait(BAR(SB_B_FULL + bb), (kBBufs == 2 ? c >> 1 : c) & 1, abort_flag);
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(SB_B_EMPTY + bb));
            }
        };
        for (uint32_t t = t_begin; t < t1; t += t_step) {
            const uint32_t i = t - t0;
            const uint32_t g = t / tiles_per_group, kt = t - g * tiles_per_group;
            release_groups(g);
            const int bb = kBBufs == 2 ? (int)((g - g_first) & 1) : 0;
            const int64_t key = (int64_t)kt * a.tile_stride * kTileKeys + row;          // within this launch's key range
            const bool live = key < a.key_cnt;
            float nrm, arn;
            if (a.norms_bulk) {
                // norms ride in the key ring (a load from global memory here costs a full trip to HBM per tile,
                // which one tile of lookahead does not hide once a tile takes less than a microsecond)
                const int s = (int)(i % kStages);
                mbar_wait(BAR(SB_K_FULL + s), (i / kStages) & 1, abort_flag);
                // volatile: the values stay in registers through the whole tile, and a plain load may be executed again where
                // the value is used (cheaper than keeping or spilling a register) -- after the arrival below, when the
                // stage may already hold another tile.  That happened: in candidate mode, where warps that lag behind
                // their tile for microseconds exist, about one score in 10^9 came out with the norm of a key eight tiles on.
                const volatile float* nr = reinterpret_cast<const volatile float*>(smem + L::off_ring + s * L::kStageBytes + L::kNormOff);
                nrm = live ? nr[row] : 0.f;
                arn = live ? a.alpha * nr[kTileKeys + row] : 0.f;
                __threadfence_block();   // every lane's loads from the stage are performed before the stage is released
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(SB_K_EMPTY + s));
            } else {
                nrm = nrm_next;
                arn = a.alpha * rn_next;
                if (t + t_step < t1) fetch_norms(t + t_step, nrm_next, rn_next);
            }
            const int db = (int)(i % kDBufs);
            const bool got = mbar_wait(BAR(SB_D_FULL + db), (i / kDBufs) & 1, abort_flag);   // false: some role gave up
            tc_fence_after();
            const uint32_t rowid = (uint32_t)((int64_t)g * a.keys_per_group + a.key_off + key);   // row of the key arrays (candidate mode)
            const uint32_t dbase = tmem + lane_addr + kColD + db * kDCols + q_mine;
            const float4* ds = reinterpret_cast<const float4*>(smem + L::off_b + bb * L::kBBytes + kHalves * 4 * QPAD * kRowBytesB) + q_mine / 2;
            const float2 n2 = make_float2(nrm, nrm), r2 = make_float2(arn, arn);
            // A give-up (`got` false) writes nothing for the tile, but every epilogue warp still walks through the named
            // barriers: the warps learn of it at different tiles, and a barrier that some of them skipped would never complete.
            if (!CAND && a.tile_store) {
                // the store of this group's previous tile must have read the box before this tile overwrites it
                if (leader) bulk_wait_read<0>();
                bar_sync(kEpiBarrier + group, 128);
            }
#pragma unroll
            for (int q16 = 0; q16 < kQT; q16 += 16) {
                float sc[16];
                {
                    uint32_t ua[16], ub[16];
                    tmem_ld16(dbase + q16, ua);               // (C_hi + C_lo) q
                    tmem_ld16(dbase + QPAD + q16, ub);        // Sg p
                    tmem_wait_ld();
                    if (q16 + 16 == kQT) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(BAR(SB_D_EMPTY + db));   // the accumulators are free again
                    }
#pragma unroll
                    for (int k = 0; k < 16; k += 2) {
                        const float4 e = ds[(q16 + k) / 2];           // 1 / scales: two of q, two of p
                        const float2 s1 = __fmul2_rn(make_float2(__uint_as_float(ua[k]), __uint_as_float(ua[k + 1])), make_float2(e.x, e.y));
                        const float2 s2 = __fmul2_rn(make_float2(__uint_as_float(ub[k]), __uint_as_float(ub[k + 1])), make_float2(e.z, e.w));
                        const float2 v = __fmul2_rn(n2, __ffma2_rn(r2, s2, s1));
                        sc[k] = v.x;
                        sc[k + 1] = v.y;
                    }
                }
                const int q0 = q_mine + q16;
                if (CAND) {
                    const int64_t list0 = (int64_t)g * a.qpg_total + a.q0 + q0;
                    if (a.fused == 2) {
                        // The sampled pass (thresholds at -inf, every score is a candidate): the slot of a score is known
                        // without a counter (tile of the sample x 128 + row); the host presets the lists' lengths.
                        // A key beyond the end of the group leaves an empty slot.
#pragma unroll
                        for (int k = 0; k < 16; ++k)
                            if (q0 + k < a.nq)
                                a.cand[(list0 + k) * a.cand_cap + (int64_t)kt * kTileKeys + row] = live && got ? make_key(sc[k], rowid) : 0ull;
                    } else {
                        // This thread's scores against their thresholds: a mask, and -- when any of the warp's 32 keys has
                        // a survivor -- the scores parked in shared memory, so that the loop below, once per query with
                        // a survivor and kept rolled (this kernel lives on its instruction cache), can pick them by
                        // a run-time index.  Survivors are staged per warp: a global counter update per survivor would put a trip
                        // to L2 on this warp's path every time.
                        uint32_t m = 0;
#pragma unroll
                        for (int k = 0; k < 16; ++k)
                            m |= (live && got && q0 + k < a.nq && sc[k] >= __ldg(a.thr + (q0 + k < a.nq ? list0 + k : 0))) ? (1u << k) : 0u;
                        uint32_t wm = __reduce_or_sync(0xffffffffu, m);
                        if (wm != 0u) {
#pragma unroll
                            for (int k = 0; k < 16; ++k) parked[k * 32] = sc[k];
#pragma unroll 1
                            while (wm != 0u) {
                                const int k = __ffs(wm) - 1;
                                wm &= wm - 1u;
                                const bool pass = (m >> k) & 1u;
                                const uint32_t votes = __ballot_sync(0xffffffffu, pass);
                                if (n_pend + __popc(votes) > kPendKeys) flush();
                                if (pass) {
                                    const int pos = n_pend + __popc(votes & ((1u << lane) - 1u));
                                    pend[pos] = make_key(parked[k * 32], rowid);
                                    pend_list[pos] = (uint32_t)(list0 + k);
                                }
                                n_pend += __popc(votes);
                            }
                        }
                    }
                } else if (a.tile_store) {
                    // The tile leaves as one box [queries of the group][128 keys]: staged in shared memory (lanes hold
                    // consecutive keys, so the stores are free of bank conflicts) and written by one bulk tensor store,
                    // which clips the keys and queries beyond the matrix.
#pragma unroll
                    for (int k = 0; k < 16; ++k) box[(q16 + k) * kTileKeys + row] = sc[k];
                } else if (live && got) {
                    float* out = a.scores + (int64_t)g * a.out_group_stride + key + (int64_t)q0 * a.out_row_stride;
#pragma unroll
                    for (int k = 0; k < 16; ++k) {
                        if (q0 + k < a.nq) {
                            __stcs(out, sc[k]);
                            out += a.out_row_stride;
                        }
                    }
                }
            }
            if (!CAND && a.tile_store) {
                fence_async_smem();
                bar_sync(kEpiBarrier + group, 128);
                if (leader && got) {
                    tensor_store_3d(&tmap_out, smem_u32(box), (int)(kt * kTileKeys), q_mine, (int)g);
                    bulk_commit();
                }
            }
        }
        if (t0 < t1) release_groups((t1 - 1) / tiles_per_group + 1);
        if (CAND) flush();
        if (leader) bulk_wait_all();   // the staged tiles must have left before the block's shared memory goes away
    }

    if (*abort_flag) __nanosleep(20000);   // tensor instructions issued before the give-up may still be running
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && *abort_flag) report_status(a.status, 2ull);
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// Rotate (z = 0) / project (z = 1) the queries of one pass and lay them out as fp16 hi/lo B operands.
// grid (QPAD, groups, 2), block 128 (thread = coordinate).  A block per matrix: 32 queries at d = 128 4.4 us, 5.1 with both matrices
// in one block.
__global__ void __launch_bounds__(128)
score_prep_kernel(TqDev p, const float* __restrict__ q, int qpg, int q0, int nq, int qpad, unsigned char* __restrict__ prep) {
    tq_grid_release();      // the scoring kernel sets itself up meanwhile
    __shared__ float qs[D];
    __shared__ float red[4];
    const int slot = blockIdx.x, g = blockIdx.y, which = blockIdx.z, j = threadIdx.x;
    unsigned char* base = prep + (size_t)g * prep_group_bytes(qpad);
    const size_t off = (size_t)(slot / 8) * ((D / 8) * 128) + (size_t)(j / 8) * 128 + (size_t)(slot % 8) * 16 + (size_t)(j % 8) * 2;
    __half* hi = reinterpret_cast<__half*>(base + (2 * which) * (size_t)qpad * kRowBytesB + off);
    __half* lo = reinterpret_cast<__half*>(base + (2 * which + 1) * (size_t)qpad * kRowBytesB + off);
    // pairs of queries: two 1 / scales of q, two of p
    float* ds = reinterpret_cast<float*>(base + 4 * (size_t)qpad * kRowBytesB) + (slot >> 1) * 4 + (slot & 1) + 2 * which;
    if (slot >= nq) {
        *hi = *lo = __float2half_rn(0.f);
        if (j == 0) *ds = 0.f;
        return;
    }
    const int d = p.d;   // 128, or 64 with the upper half of every operand row left unused
    qs[j] = j < d ? q[((size_t)g * qpg + q0 + slot) * d + j] : 0.f;
    __syncthreads();
    // The matrices are usually cold (the keys streamed through L2 since the last call), so the time would
    // go into memory latency if the loads trickled in between the arithmetic: bring the matrix into
    // shared memory with all copies in flight at once, then run the chain in order from there.
    extern __shared__ __align__(16) float mat[];   // [D][D]: R^T or S^T
    {
        const uint32_t dst0 = (uint32_t)__cvta_generic_to_shared(mat);
        const float* src = which ? p.St : p.Rt;
#pragma unroll 8
        for (int c = j; c < d * d / 4; c += 128)        // 16-byte chunks
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst0 + c * 16), "l"(src + (size_t)c * 4) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
    float r = 0.f;
    if (j < d) {
#pragma unroll 16
        for (int k = 0; k < d; ++k) r = fmaf(qs[k], mat[k * d + j], r);
    }
    float m = fabsf(r);
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((j & 31) == 0) red[j >> 5] = m;
    __syncthreads();
    m = fmaxf(fmaxf(red[0], red[1]), fmaxf(red[2], red[3]));
    // a power-of-two scale that brings the largest magnitude into [512, 1024): safe in fp16, exact to undo
    const float e = m > 0.f && m < 3.0e38f ? ldexpf(1.f, 9 - ilogbf(m)) : 1.f;
    const float rs = r * e;
    const __half h = __float2half_rn(rs);
    *hi = h;
    *lo = __float2half_rn(rs - __half2float(h));
    if (j == 0) *ds = 1.f / (which ? e : e * kCentScale);
}

// The same for d = 256: the matrices do not fit shared memory and are read from global memory (usually cold), so the
// kernel lives on the number of loads in flight: block 1024, thread = (coordinate, quarter of the sum), 32 loads
// in flight per thread; a block per matrix (16 queries: 10 us, 17 with both matrices in one block).
// The operands are written as two halves of 128 coordinates, each in the layout of d = 128.
__global__ void __launch_bounds__(1024)
score_prep256_kernel(TqDev p, const float* __restrict__ q, int qpg, int q0, int nq, int qpad, unsigned char* __restrict__ prep) {
    constexpr int kD = 256, kParts = 4, kSteps = kD / kParts;
    __shared__ float qs[kD];
    __shared__ float part[kParts][kD];
    __shared__ float red[8];
    const int slot = blockIdx.x, g = blockIdx.y, which = blockIdx.z, j = threadIdx.x & (kD - 1), kq = threadIdx.x >> 8;
    unsigned char* base = prep + (size_t)g * prep_group_bytes(qpad, 2);
    const int jh = j & 127;
    const size_t off = (size_t)(j >> 7) * (4 * (size_t)qpad * kRowBytesB) + (size_t)(slot / 8) * ((D / 8) * 128) +
                       (size_t)(jh / 8) * 128 + (size_t)(slot % 8) * 16 + (size_t)(jh % 8) * 2;
    __half* hi = reinterpret_cast<__half*>(base + (2 * which) * (size_t)qpad * kRowBytesB + off);
    __half* lo = reinterpret_cast<__half*>(base + (2 * which + 1) * (size_t)qpad * kRowBytesB + off);
    float* ds = reinterpret_cast<float*>(base + 8 * (size_t)qpad * kRowBytesB) + (slot >> 1) * 4 + (slot & 1) + 2 * which;
    tq_grid_release();      // the scoring kernel sets itself up meanwhile
    if (slot >= nq) {
        if (kq == 0) {
            *hi = *lo = __float2half_rn(0.f);
            if (j == 0) *ds = 0.f;
        }
        return;
    }
    // four independent chains; the order of the sums differs from the general kernel's, which the fp32
    // tolerance of the scores covers
    const float* M = (which ? p.St : p.Rt) + (size_t)kq * kSteps * kD + j;
    float r[4] = {0.f, 0.f, 0.f, 0.f};
    if (kq == 0) qs[j] = q[((size_t)g * qpg + q0 + slot) * kD + j];
    __syncthreads();
    const float* qk = qs + kq * kSteps;
#pragma unroll 32
    for (int k = 0; k < kSteps; ++k) r[k & 3] = fmaf(qk[k], __ldg(M + (size_t)k * kD), r[k & 3]);
    part[kq][j] = (r[0] + r[1]) + (r[2] + r[3]);
    __syncthreads();
    if (kq != 0) return;      // threads 0..255 (warps 0..7) finish the coordinate
    const float rr = (part[0][j] + part[1][j]) + (part[2][j] + part[3][j]);
    float m = fabsf(rr);
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((j & 31) == 0) red[j >> 5] = m;
    asm volatile("bar.sync 1, 256;" ::: "memory");      // the 256 threads that are left
    m = 0.f;
    for (int w = 0; w < 8; ++w) m = fmaxf(m, red[w]);
    const float e = m > 0.f && m < 3.0e38f ? ldexpf(1.f, 9 - ilogbf(m)) : 1.f;
    const float rs = rr * e;
    const __half h = __float2half_rn(rs);
    *hi = h;
    *lo = __float2half_rn(rs - __half2float(h));
    if (j == 0) *ds = 1.f / (which ? e : e * kCentScale);
}

// grid (segments, rows): block scans scores[row][seg*seg_len ...) and writes its k best as sortable keys
// to part[((group*lists_per_group + list_base + seg) * qpg + qi) * topk ...].  Candidates above the
// running threshold are collected in shared memory; when the buffer could overflow in the next batch
// it is cut back to the k best, which also raises the threshold.
__global__ void __launch_bounds__(kSelThreads)
topk_rows_kernel(const float* __restrict__ scores, int64_t row_stride, int64_t group_stride, int qpg, int64_t n,
                 int64_t seg_len, int64_t first_row_of_group_stride, int64_t key_off, int topk, int k2,
                 int lists_per_group, int list_base, unsigned long long* __restrict__ part, const unsigned int* run_if) {
    if (run_if && *run_if == 0u) return;
    __shared__ __align__(16) unsigned long long buf[kSelCap];
    __shared__ int hist[256];
    __shared__ int scratch[4];
    __shared__ int cnt;
    __shared__ unsigned long long thr;
    const int seg = blockIdx.x, r = blockIdx.y, g = r / qpg, qi = r - g * qpg;
    const float* src = scores + g * group_stride + qi * row_stride;
    const uint32_t row0 = (uint32_t)(g * first_row_of_group_stride + key_off);
    const int64_t k0 = (int64_t)seg * seg_len;
    int64_t k1 = k0 + seg_len;
    if (k1 > n) k1 = n;
    if (threadIdx.x == 0) { cnt = 0; thr = 0ull; }
    __syncthreads();
    // First threshold without filling the buffer: every thread takes the best of 32 scores from the head of the segment
    // (8,192 in all); the k-th best of those 256 maxima is a score that at least k scores of the segment reach, and on
    // data without order about 3 % of all scores do, so the candidates of the whole segment fit the buffer and the one
    // selection at the end is all there is (without it the first 4,096 scores all pass, each through the shared counter,
    // and a selection is needed as soon as they have).  Data that defeats the estimate only brings the cut-backs back.
    constexpr int kPre = 4 * kSelPerThread;
    if (topk <= kSelThreads && k1 - k0 >= (int64_t)kPre * kSelThreads) {
        uint32_t best = 0u;
#pragma unroll
        for (int j = 0; j < kPre; ++j) {
            const uint32_t o = ordered_bits(__ldg(src + k0 + j * kSelThreads + threadIdx.x));
            best = o > best ? o : best;
        }
        buf[threadIdx.x] = (unsigned long long)best;
        block_sort_desc(buf, kSelThreads);
        const unsigned long long t0 = buf[topk - 1] << 32;   // below every key that carries this score
        __syncthreads();
        if (threadIdx.x == 0) thr = t0;
        __syncthreads();
    }
    // The scores of the next batch are already on their way while this one is filtered, and the common
    // case (nothing to prune) costs one barrier per batch.
    float nxt[kSelPerThread];
#pragma unroll
    for (int j = 0; j < kSelPerThread; ++j) {
        const int64_t key = k0 + j * kSelThreads + threadIdx.x;
        nxt[j] = key < k1 ? __ldcs(src + key) : 0.f;
    }
    for (int64_t kb = k0; kb < k1; kb += kSelBatch) {
        float v[kSelPerThread];
#pragma unroll
        for (int j = 0; j < kSelPerThread; ++j) v[j] = nxt[j];
        if (kb + kSelBatch < k1) {
#pragma unroll
            for (int j = 0; j < kSelPerThread; ++j) {
                const int64_t key = kb + kSelBatch + j * kSelThreads + threadIdx.x;
                nxt[j] = key < k1 ? __ldcs(src + key) : 0.f;
            }
        }
        // The test that nearly every score fails is one 32-bit compare of the score's sortable bits with the upper half
        // of the threshold; the 64-bit key, the bound check and the append are behind it.
        const unsigned long long t = thr;
        const uint32_t t_hi = (uint32_t)(t >> 32);
#pragma unroll
        for (int j = 0; j < kSelPerThread; ++j) {
            const uint32_t o = ordered_bits(v[j]);
            if (o >= t_hi) {
                const int64_t key = kb + j * kSelThreads + threadIdx.x;
                const unsigned long long ck = ((unsigned long long)o << 32) | (unsigned long long)(0xffffffffu - (row0 + (uint32_t)key));
                if (key < k1 && ck > t) buf[atomicAdd(&cnt, 1)] = ck;
            }
        }
        // Each thread tests the count it sees after its own appends; the thread that appended last sees the
        // final count, so the OR over the block is the test on the final count and is the same for everyone.
        if (__syncthreads_or(cnt + kSelBatch > kSelCap)) {
            const int c = cnt;  // stable: every thread is in this branch
            if (c > topk) {
                const unsigned long long kth = block_select_topk(buf, c, topk, hist, scratch);
                if (threadIdx.x == 0) { cnt = topk; thr = kth; }
            }
            __syncthreads();
        }
    }
    __syncthreads();
    int c = cnt;
    if (c > topk) { block_select_topk(buf, c, topk, hist, scratch); c = topk; }
    __syncthreads();
    for (int i = c + threadIdx.x; i < k2; i += kSelThreads) buf[i] = 0ull;
    block_sort_desc(buf, k2);
    unsigned long long* dst = part + (((size_t)g * lists_per_group + list_base + seg) * qpg + qi) * topk;
    for (int i = threadIdx.x; i < topk; i += kSelThreads) dst[i] = buf[i];
}

// Candidate mode, after a scoring pass: one block per (query, group) takes the query's candidate list (and, mode 0,
// its best list so far), keeps the k best as sorted keys in best[group][query][topk], raises the query's threshold
// to the k-th best score (once there are k) and empties the list.  Mode 1 (the sampled pass that only finds a
// first threshold) leaves the best list alone: its keys will be scored again by the full pass.
__global__ void __launch_bounds__(256)
select_candidates_kernel(const unsigned long long* __restrict__ cand, unsigned int* __restrict__ cnt, int64_t cap,
                         unsigned long long* __restrict__ best, float* __restrict__ thr, int qpg, int topk, int k2, int mode,
                         const unsigned int* run_if) {
    if (run_if && *run_if == 0u) return;
    __shared__ __align__(16) unsigned long long a[kSelCap];
    __shared__ int hist[256];
    __shared__ int scratch[4];
    __shared__ int count;
    __shared__ unsigned long long cut;   // keys at or below it cannot be among the k best any more
    const int64_t q = (int64_t)blockIdx.y * qpg + blockIdx.x;
    const unsigned long long* list = cand + q * cap;
    unsigned long long* mine = best + q * topk;
    const int64_t n = min((int64_t)cnt[q], cap);
    if (threadIdx.x == 0) { count = 0; cut = 0ull; }
    __syncthreads();
    if (mode == 0) {
        for (int i = threadIdx.x; i < topk; i += blockDim.x) {
            const unsigned long long v = mine[i];
            if (v != 0ull) a[atomicAdd(&count, 1)] = v;
        }
        __syncthreads();
    }
    constexpr int kBatch = 2048;
    for (int64_t base = 0; base < n; base += kBatch) {
        if (count + kBatch > kSelCap) {  // uniform: count only changes between barriers
            const int c = count;
            __syncthreads();
            if (c > topk) {
                const unsigned long long kth = block_select_topk(a, c, topk, hist, scratch);
                if (threadIdx.x == 0) { count = topk; cut = kth; }
            }
            __syncthreads();
        }
        const unsigned long long t = cut;
        const int64_t end = base + kBatch < n ? base + kBatch : n;
        for (int64_t i = base + threadIdx.x; i < end; i += blockDim.x) {
            const unsigned long long v = __ldcs(list + i);
            if (v > t) a[atomicAdd(&count, 1)] = v;      // also drops the empty slots
        }
        __syncthreads();
    }
    const int c = count;
    const int keep = c < topk ? c : topk;
    if (keep < c) block_select_topk(a, c, keep, hist, scratch);
    __syncthreads();
    for (int i = keep + threadIdx.x; i < k2; i += blockDim.x) a[i] = 0ull;
    block_sort_desc(a, k2);
    if (mode == 0)
        for (int i = threadIdx.x; i < topk; i += blockDim.x) mine[i] = a[i];
    if (threadIdx.x == 0) {
        if (keep == topk) thr[q] = unordered_bits((uint32_t)(a[topk - 1] >> 32));
        cnt[q] = 0u;
    }
}

// thresholds to -inf, best lists to empty, list lengths to `first_count` (what the sampled pass will leave in them; 0 without one)
__global__ void init_candidates_kernel(float* thr, unsigned int* cnt, unsigned long long* best, int64_t lists, int topk,
                                       unsigned int first_count, const unsigned int* run_if) {
    if (run_if && *run_if == 0u) return;
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < lists) { thr[i] = -CUDART_INF_F; cnt[i] = first_count; }
    if (i < lists * topk) best[i] = 0ull;
}

int pow2_at_least(int v) {
    int p = 1;
    while (p < v) p <<= 1;
    return p;
}

template <int BITS, int QPAD, int DR>
int launch_score(const tq_plan* p, const CUtensorMap& map, const ScoreTcArgs& args, int grid, cudaStream_t st) {
    const int sm = ScoreSmem<BITS, QPAD, DR>::total;
    if (args.fused) {
        TQ_GRANT_SMEM((score_tc_kernel<BITS, QPAD, DR, true>), sm, p->device);
        TQ_CUDA_TRY(tq_launch_dependent(score_tc_kernel<BITS, QPAD, DR, true>, dim3(grid), dim3(kThreads), (size_t)sm, st, map, args));
        TQ_CUDA_TRY(cudaGetLastError());
        return TQ_OK;
    }
    TQ_GRANT_SMEM((score_tc_kernel<BITS, QPAD, DR, false>), sm, p->device);
    TQ_CUDA_TRY(tq_launch_dependent(score_tc_kernel<BITS, QPAD, DR, false>, dim3(grid), dim3(kThreads), (size_t)sm, st, map, args));
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}

}  // namespace

#ifndef TQ_SCORE_PASS
#define TQ_SCORE_PASS 64     // queries per scoring launch at d <= 128 (32: the measurement build without passes of 64)
#endif

#define TQ_STEP(expr)                         \
    do {                                      \
        const int rc__ = (expr);              \
        if (rc__ != TQ_OK) return rc__;       \
    } while (0)

// ---- host-side planning ---------------------------------------------------------------------------
constexpr int64_t kChunkKeys = 1 << 22;     // keys per group scored into scratch at a time when only top-k is wanted
                                            // (2^20: 221 us per 1M keys and 32 queries, 2^21: 198, 2^23: 185; scratch 16 B x queries per key)
constexpr int64_t kSegLen = 65536;          // scores per selection block (top-100 call at 1,048,576 keys: 32,768 -> 214 us, 65,536 -> 204, 131,072 -> 213, 262,144 -> 241)

// prepared queries of one group in the scratch block: the largest of the passes (64 queries; 32 queries of d = 256)
constexpr size_t kPrepGroupMax = prep_group_bytes(64, 1) > prep_group_bytes(32, 2) ? prep_group_bytes(64, 1) : prep_group_bytes(32, 2);

struct ScoreTcPlan {
    int64_t chunk, nchunks, segs_per_chunk, lists_per_group;
    size_t prep_bytes, part_bytes, matrix_bytes, total;
    size_t off_prep, off_part, off_matrix;
};

static ScoreTcPlan plan_score(int groups, int qpg, int64_t keys_per_group, int topk, bool need_scratch_matrix) {
    ScoreTcPlan s{};
    s.chunk = keys_per_group < kChunkKeys ? keys_per_group : kChunkKeys;
    if (s.chunk < 1) s.chunk = 1;
    s.nchunks = (keys_per_group + s.chunk - 1) / s.chunk;
    if (s.nchunks < 1) s.nchunks = 1;
    s.segs_per_chunk = (s.chunk + kSegLen - 1) / kSegLen;
    s.lists_per_group = s.nchunks * s.segs_per_chunk;
    s.prep_bytes = ((size_t)groups * kPrepGroupMax + 255) & ~size_t(255);
    s.part_bytes = topk > 0 ? (((size_t)groups * s.lists_per_group * qpg * topk * 8) + 255) & ~size_t(255) : 0;
    s.matrix_bytes = (topk > 0 && need_scratch_matrix) ? (((size_t)groups * qpg * s.chunk * 4) + 255) & ~size_t(255) : 0;
    s.off_prep = 0;
    s.off_part = s.prep_bytes;
    s.off_matrix = s.off_part + s.part_bytes;
    s.total = s.off_matrix + s.matrix_bytes;
    return s;
}

// Candidate mode (top-k without any score matrix) for key sets of several chunks: per query a threshold, a counter,
// a best-k list and a candidate list that can hold every key of one chunk (so no list can overflow, whatever the data).
constexpr int64_t kCandChunk = 1 << 21;     // keys per group per scoring launch
constexpr int64_t kSampleEvery = 64;        // the first threshold comes from every 64th tile of the first chunk

struct CandPlan {
    int64_t chunk, nchunks, cand_cap, lists;
    size_t off_thr, off_cnt, off_best, off_cand, total;
};

static CandPlan plan_candidates(int groups, int qpg, int64_t keys_per_group, int topk) {
    CandPlan s{};
    auto pad = [](size_t b) { return (b + 255) & ~size_t(255); };
    s.chunk = keys_per_group < kCandChunk ? (keys_per_group < 1 ? 1 : keys_per_group) : kCandChunk;
    s.nchunks = (keys_per_group + s.chunk - 1) / s.chunk;
    s.cand_cap = s.chunk;
    s.lists = (int64_t)groups * qpg;
    s.off_thr = pad((size_t)groups * kPrepGroupMax);
    s.off_cnt = s.off_thr + pad((size_t)s.lists * 4);
    s.off_best = s.off_cnt + pad((size_t)s.lists * 4);
    s.off_cand = s.off_best + pad((size_t)s.lists * (topk > 0 ? topk : 1) * 8);
    s.total = s.off_cand + pad((size_t)s.lists * s.cand_cap * 8);
    return s;
}

// Candidate mode pays a sampled pass and two selections up front; it wins once a key set spans several chunks
// (measured: 8,388,608 keys x 32 queries 158 us per 1,048,576 keys against 188 us through a scratch matrix; a single
// chunk of 1,048,576 keys 307 us against 224 us).
static bool use_candidates(const float* scores, int topk, int64_t keys_per_group) {
    return scores == nullptr && topk > 0 && keys_per_group > 2 * kCandChunk;
}

// Filtered search (tq_score_filter.cu): one group of keys, no matrix, and lists short enough that a round's keys can be
// gathered: a round whose threshold comes from 1 / r of its keys lists about r * topk keys per query.
// Its fixed part (a sample, two rounds, the skipped fallback: some 25 launches) costs about 80 us, what it saves grows with keys
// and queries.  Search through an index, before / with it: 1,048,576 keys, 64 queries 300 / 249 us, 32 queries 210 / 198, 8 queries
// 160 / 160; 2,097,152 keys, 8 queries 246 / 214, 1 query 219 / 183; 8,388,608 keys, 64 queries 1502 / 622, 1 query 1004 / 424.
// Long lists want more keys too (they are gathered and sorted by query): 32 queries, top 1,000: 1,048,576 keys 304 / 388 us,
// 1,500,000 keys 410 / 432, 2,097,152 keys 514 / 476.
constexpr int64_t kFilterFrom = 1 << 21, kFilterFromMany = 1 << 20;      // keys from which on it pays; from 32 queries on
constexpr int64_t kFilterSample = 1 << 15;     // keys of the first sample
constexpr int kFilterRoom = 1 << 18;           // gathered keys of a round
static bool use_filter(const tq_plan* p, const float* scores, int groups, int qpg, int topk, int64_t keys_per_group) {
    const int nq = qpg < 64 ? qpg : 64;
    return scores == nullptr && topk > 0 && groups == 1 && p->beta_scale > 0.f && keys_per_group >= (qpg >= 32 ? kFilterFromMany : kFilterFrom) &&
           keys_per_group < (int64_t)1 << 31 && (int64_t)nq * topk * 6 <= kFilterRoom && (int64_t)nq * topk * 48 <= keys_per_group;
}
// The procedure that a filtered search falls back to takes the same passes of queries, one after the other, and works in the
// memory that the pass's lists, scores and gathered keys have left: the whole is no larger than one pass of that procedure (64 queries x
// 1,048,576 keys 0.27 GB, from 4,194,304 keys on 1.07 GB, whatever the number of queries), or about 25 MB for a handful of
// queries.  (What a call asks for is still what the unfiltered path would take, which a plan can be switched to.)
struct FilterPlan {
    int pass;                    // queries of the largest pass
    int64_t stride0, first;      // tiles between the sampled ones; keys of the sample, a multiple of 128
    bool matrix;                 // the fallback scores into a matrix (else candidate mode)
    int64_t segs;
    size_t off_thr, off_cnt, off_best, off_prep, off_words;
    size_t off_sample, off_rows, off_offsets, off_codes, off_signs, off_norms, off_rnorms, off_grows, off_scores;
    size_t off_matrix, off_part, off_cand, total;
};
static FilterPlan plan_filter(const tq_plan* p, int qpg, int64_t keys, int topk) {
    FilterPlan f{};
    auto pad = [](size_t bytes) { return (bytes + 255) & ~size_t(255); };
    const int most = p->dev.d == 256 ? 32 : TQ_SCORE_PASS;
    f.pass = qpg < most ? qpg : most;
    const int64_t tiles = (keys + kTileKeys - 1) / kTileKeys;
    f.stride0 = (tiles + kFilterSample / kTileKeys - 1) / (kFilterSample / kTileKeys);
    f.first = (tiles + f.stride0 - 1) / f.stride0 * kTileKeys;
    f.matrix = keys <= 2 * kCandChunk;
    f.segs = (keys + kSegLen - 1) / kSegLen;
    size_t at = pad(kPrepGroupMax);      // the prepared queries come first in every layout
    auto take = [&](size_t bytes) { const size_t o = at; at += pad(bytes); return o; };
    f.off_thr = take((size_t)qpg * 4);
    f.off_cnt = take((size_t)qpg * 4);
    f.off_best = take((size_t)qpg * topk * 8);
    f.off_prep = take(tq_filter_prep_bytes(p->dev.d, 64));
    f.off_words = take(256);
    const size_t shared = at;
    f.off_sample = take((size_t)f.pass * f.first * 8);
    f.off_offsets = take(64 * 4);
    f.off_rows = take((size_t)f.pass * kFilterRoom * 4);
    f.off_codes = take((size_t)kFilterRoom * p->dev.code_words * 4);
    f.off_signs = take((size_t)kFilterRoom * p->dev.sign_words * 4);
    f.off_norms = take((size_t)kFilterRoom * 4);
    f.off_rnorms = take((size_t)kFilterRoom * 4);
    f.off_grows = take((size_t)kFilterRoom * 4);
    f.off_scores = take((size_t)f.pass * kFilterRoom * 4);
    f.total = at;
    at = shared;                          // the fallback, in the same place
    if (f.matrix) {
        f.off_matrix = take((size_t)f.pass * keys * 4);
        f.off_part = take((size_t)f.segs * f.pass * topk * 8);
    } else {
        f.off_cand = take((size_t)f.pass * kCandChunk * 8);
    }
    if (at > f.total) f.total = at;
    return f;
}

int64_t tq_score_tc_scratch(const tq_plan* p, int groups, int qpg, int64_t keys_per_group, int topk) {
    const size_t a = plan_score(groups, qpg, keys_per_group, topk, true).total;
    const size_t b = use_candidates(nullptr, topk, keys_per_group) ? plan_candidates(groups, qpg, keys_per_group, topk).total : 0;
    const size_t c = use_filter(p, nullptr, groups, qpg, topk, keys_per_group) ? plan_filter(p, qpg, keys_per_group, topk).total : 0;
    return (int64_t)std::max(std::max(a, b), c);
}

int tq_merge_keys_launch(const unsigned long long* part, int lists, int qpg, int groups, int topk, int64_t idx_base,
                         float* top_scores, int64_t* top_idx, cudaStream_t st, const unsigned int* run_if = nullptr);

int tq_launch_score_tc(const tq_plan* p, const float* q, int groups, int qpg, const uint32_t* codes,
                       const uint32_t* signs, const float* rnorms, const float* norms, int64_t keys_per_group,
                       float* scores, int topk, float* top_scores, int64_t* top_idx, int64_t idx_base, void* scratch,
                       size_t scratch_bytes, cudaStream_t st, int64_t group_rows) {
    TqRange range("tq.score.tensor_core");
    if (group_rows <= 0) group_rows = keys_per_group;
    const bool filter = p->path == TQ_PATH_AUTO && use_filter(p, scores, groups, qpg, topk, keys_per_group);
    const bool candidates = !filter && use_candidates(scores, topk, keys_per_group);
    const ScoreTcPlan sp = plan_score(groups, qpg, keys_per_group, topk, scores == nullptr);
    const CandPlan cp = plan_candidates(groups, qpg, keys_per_group, topk);
    const FilterPlan fp = filter ? plan_filter(p, qpg, keys_per_group, topk) : FilterPlan{};
    const size_t need = filter ? fp.total : candidates ? cp.total : sp.total;
    if (!scratch || scratch_bytes < need)
        return tq_fail(TQ_ERR_SCRATCH_TOO_SMALL, "score scratch: need %zu bytes, got %zu", need, scratch_bytes);
    unsigned char* sc = static_cast<unsigned char*>(scratch);
    unsigned char* prep = sc;     // every layout starts with the prepared queries
    const int sms = tq_sm_count(p->device);
    const int bits = p->dev.bits;
    float* thr = reinterpret_cast<float*>(sc + (filter ? fp.off_thr : cp.off_thr));
    unsigned int* cnt = reinterpret_cast<unsigned int*>(sc + (filter ? fp.off_cnt : cp.off_cnt));
    unsigned long long* best = reinterpret_cast<unsigned long long*>(sc + (filter ? fp.off_best : cp.off_best));
    // candidate lists: of every query, or (filtered search) of the queries of the pass at work
    struct Lists { unsigned long long* at; int64_t cap; };
    const Lists all_lists{reinterpret_cast<unsigned long long*>(sc + cp.off_cand), cp.cand_cap};

    // Which keys a launch scores: the caller's, or those gathered by a filtered search.
    struct Keys { const uint32_t *codes, *signs; const float *rnorms, *norms; int64_t group_rows; const unsigned int* dyn_keys; };
    const Keys all_keys{codes, signs, rnorms, norms, group_rows, nullptr};
    const int pass = p->dev.d == 256 ? 32 : TQ_SCORE_PASS;
    auto pad_of = [](int nq) { return nq <= 16 ? 16 : nq <= 32 ? 32 : 64; };
    auto prepare_pass = [&](int q0, int nq) -> int {
        const int qpad = pad_of(nq);
        if (p->dev.d == 256) {
            score_prep256_kernel<<<dim3(qpad, groups, 2), 1024, 0, st>>>(p->dev, q, qpg, q0, nq, qpad, prep); tq_count_launch();
        } else {
            TQ_GRANT_SMEM((score_prep_kernel), kPrepSmemBytes, p->device);
            score_prep_kernel<<<dim3(qpad, groups, 2), 128, kPrepSmemBytes, st>>>(p->dev, q, qpg, q0, nq, qpad, prep); tq_count_launch();
        }
        TQ_CUDA_TRY(cudaGetLastError());
        return TQ_OK;
    };
    // One scoring launch for the prepared queries [q0, q0 + nq) over keys [key_off, key_off + key_cnt) of every group (every
    // tile_stride-th tile of them), into a matrix (mat != null) or into the candidate lists.
    auto score_pass = [&](const Keys& keys, int q0, int nq, int64_t key_off, int64_t key_cnt, int tile_stride, float* mat,
                          int64_t row_stride, const Lists& lists, const unsigned int* run_if) -> int {
        const int qpad = pad_of(nq);
        const int64_t group_stride = (int64_t)qpg * row_stride;
        ScoreTcArgs a{};
        a.codes = keys.codes; a.signs = keys.signs; a.rnorms = keys.rnorms; a.norms = keys.norms;
        a.dyn_keys = keys.dyn_keys; a.run_if = run_if;
        a.prep = prep; a.codebook = p->dev.codebook;
        a.keys_per_group = keys.group_rows; a.key_off = key_off; a.key_cnt = key_cnt;
        a.tile_stride = tile_stride;
        const int64_t tiles = (key_cnt + kTileKeys - 1) / kTileKeys;
        a.tiles_per_group = (tiles + tile_stride - 1) / tile_stride;
        a.total_tiles = a.tiles_per_group * groups;
        a.nq = nq;
        a.out_group_stride = group_stride; a.out_row_stride = row_stride;
        a.scores = mat ? mat + (int64_t)q0 * row_stride : nullptr;
        a.alpha = p->dev.alpha;
        a.norms_bulk = (groups == 1 || keys.group_rows % 4 == 0) && key_off % 4 == 0 ? 1 : 0;   // 16-byte aligned tile starts
        a.fused = mat ? 0 : (tile_stride > 1 ? 2 : 1);    // 2: the sampled pass
        a.qpg_total = qpg; a.q0 = q0;
        a.thr = thr; a.cnt = cnt; a.cand = lists.at; a.cand_cap = lists.cap;
        a.status = p->status_dev;
        a.wait_kcycles = p->wait_kcycles;
        if (a.total_tiles == 0) return TQ_OK;
        const int grid = (int)(a.total_tiles < sms ? a.total_tiles : sms);
        // Score tiles leave through a bulk tensor store when the matrix allows one: 16-byte aligned base and
        // row pitch.  Box = 128 keys x the queries of the pass x one group; extents clip ragged edges.
        CUtensorMap map;
        memset(&map, 0, sizeof(map));
        a.tile_store = 0;
        if (mat && (reinterpret_cast<uintptr_t>(a.scores) & 15u) == 0 && row_stride % 4 == 0 && key_cnt > 0 && tq_encode_tiled_fn()) {
            const cuuint64_t gdim[3] = {(cuuint64_t)key_cnt, (cuuint64_t)nq, (cuuint64_t)groups};
            const cuuint64_t gstride[2] = {(cuuint64_t)row_stride * 4, (cuuint64_t)group_stride * 4};
            const cuuint32_t box[3] = {(cuuint32_t)kTileKeys, (cuuint32_t)(qpad < 32 ? qpad : 32), 1};
            const cuuint32_t estr[3] = {1, 1, 1};
            const CUresult cr = tq_encode_tiled_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, a.scores, gdim, gstride, box, estr,
                                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                                     CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
            if (cr == CUDA_SUCCESS) a.tile_store = 1;
        }
        int r = TQ_ERR_UNSUPPORTED;
        tq_timer_mark(p, 1, 0, st);
#define TQ_SC(B)                                                                                             \
case B:                                                                                                  \
    if (p->dev.d == 64) r = qpad == 16 ? launch_score<B, 16, 64>(p, map, a, grid, st) : qpad == 32 ? launch_score<B, 32, 64>(p, map, a, grid, st)       \
                                                                                               : launch_score<B, 64, 64>(p, map, a, grid, st);      \
    else if (p->dev.d == 256) r = qpad == 16 ? launch_score<B, 16, 256>(p, map, a, grid, st) : launch_score<B, 32, 256>(p, map, a, grid, st);          \
    else r = qpad == 16 ? launch_score<B, 16, 128>(p, map, a, grid, st) : qpad == 32 ? launch_score<B, 32, 128>(p, map, a, grid, st)                   \
                                                                                  : launch_score<B, 64, 128>(p, map, a, grid, st);                  \
    break;
        switch (bits) { TQ_SC(1) TQ_SC(2) TQ_SC(3) TQ_SC(4) }
#undef TQ_SC
        tq_timer_mark(p, 1, 1, st);
        if (r != TQ_OK) return r == TQ_ERR_UNSUPPORTED ? tq_fail(r, "no tensor-core scoring kernel for bits=%d", bits) : r;
        return TQ_OK;
    };
    // The same for every pass of at most 64 queries (32 at d = 256).  A pass of 64 expands the keys once for queries that would
    // otherwise take two passes (64 queries x 1,048,576 keys: 171 us against 219 us in two passes of 32; 33 queries: 168
    // against 205 us in passes of 32 and 16).
    // `prepared`: the scratch block still holds the prepared queries of the only pass (a call of several launches
    // over the same queries prepares them once).
    auto score_passes = [&](int64_t key_off, int64_t key_cnt, int tile_stride, float* mat, int64_t row_stride, bool prepared) -> int {
        for (int q0 = 0; q0 < qpg; q0 += pass) {
            const int nq = qpg - q0 < pass ? qpg - q0 : pass;
            if (!(prepared && qpg <= pass)) {
                const int rc = prepare_pass(q0, nq);
                if (rc != TQ_OK) return rc;
            }
            const int rc = score_pass(all_keys, q0, nq, key_off, key_cnt, tile_stride, mat, row_stride, all_lists, nullptr);
            if (rc != TQ_OK) return rc;
        }
        return TQ_OK;
    };

    if (!candidates && !filter) {
        // A score matrix exists: the caller's (everything scored in one go) or, when only the top-k is wanted, a scratch
        // matrix per chunk of keys; the top-k is selected from it segment by segment and the lists are merged at the end.
        unsigned long long* part = reinterpret_cast<unsigned long long*>(sc + sp.off_part);
        float* tmp = reinterpret_cast<float*>(sc + sp.off_matrix);
        if (topk > 0) TQ_CUDA_TRY(cudaMemsetAsync(part, 0, sp.part_bytes, st));  // zero = empty slot
        const int64_t nchunks = scores ? 1 : sp.nchunks;
        for (int64_t c = 0; c < nchunks; ++c) {
            const int64_t key_off = scores ? 0 : c * sp.chunk;
            int64_t key_cnt = scores ? keys_per_group : keys_per_group - key_off;
            if (!scores && key_cnt > sp.chunk) key_cnt = sp.chunk;
            float* mat = scores ? scores : tmp;
            const int64_t row_stride = scores ? keys_per_group : sp.chunk;
            const int rc = score_passes(key_off, key_cnt, 1, mat, row_stride, c > 0);
            if (rc != TQ_OK) return rc;
            if (topk > 0) {
                const int64_t segs = (key_cnt + kSegLen - 1) / kSegLen;
                // lists of chunk c occupy slots [c*segs_per_chunk, ...); unused slots stay zero (= empty)
                topk_rows_kernel<<<dim3((unsigned)segs, (unsigned)(groups * qpg)), kSelThreads, 0, st>>>(
                    mat, row_stride, (int64_t)qpg * row_stride, qpg, key_cnt, kSegLen, group_rows, key_off, topk, pow2_at_least(topk),
                    (int)sp.lists_per_group, (int)(c * sp.segs_per_chunk), part, nullptr); tq_count_launch();
                TQ_CUDA_TRY(cudaGetLastError());
            }
        }
        if (topk > 0)
            return tq_merge_keys_launch(part, (int)sp.lists_per_group, qpg, groups, topk, idx_base, top_scores, top_idx, st);
        return TQ_OK;
    }

    // Top-k only over several chunks.  Every query keeps a threshold (a lower bound of its k-th best score so far); the
    // scoring kernel appends the scores that reach it to the query's candidate list and nothing else leaves the kernel;
    // after every launch the lists are folded into the running best-k lists, which raises the thresholds for the next
    // chunk.  The first threshold comes from scoring every 64th tile of the first chunk with the threshold at -inf: the
    // k-th best of a subset is a lower bound of the k-th best of the whole, so the full pass that follows loses nothing
    // and appends only about 64 k scores per query.
    const int k2 = pow2_at_least(topk);
    const int64_t tiles0 = (std::min(cp.chunk, keys_per_group) + kTileKeys - 1) / kTileKeys;
    const int64_t sample_tiles = (tiles0 + kSampleEvery - 1) / kSampleEvery;
    // (of the queries from q0 on, `queries` per group)
    auto init = [&](int q0, int64_t queries, int64_t first_count, const unsigned int* run_if) -> int {
        init_candidates_kernel<<<(unsigned)((queries * topk + 255) / 256), 256, 0, st>>>(thr + q0, cnt + q0, best + (int64_t)q0 * topk, queries, topk,
                                                                                         (unsigned int)first_count, run_if);
        tq_count_launch();
        TQ_CUDA_TRY(cudaGetLastError());
        return TQ_OK;
    };
    auto select = [&](const Lists& lists, int q0, int queries, int mode, const unsigned int* run_if) -> int {
        select_candidates_kernel<<<dim3((unsigned)queries, (unsigned)groups), 256, 0, st>>>(lists.at + q0 * lists.cap, cnt + q0, lists.cap, best + (int64_t)q0 * topk,
                                                                                            thr + q0, queries, topk, k2, mode, run_if);
        tq_count_launch();
        TQ_CUDA_TRY(cudaGetLastError());
        return TQ_OK;
    };
    // `score`: one scoring launch or several over keys [key_off, key_off + key_cnt), every tile_stride-th tile of them, into the lists
    auto run_candidates = [&](const Lists& lists, int q0, int queries, const unsigned int* run_if, auto score) -> int {
        TQ_STEP(init(q0, (int64_t)groups * queries, sample_tiles * kTileKeys, run_if));
        for (int64_t c = 0; c < cp.nchunks; ++c) {
            const int64_t key_off = c * cp.chunk;
            int64_t key_cnt = keys_per_group - key_off;
            if (key_cnt > cp.chunk) key_cnt = cp.chunk;
            if (c == 0) {
                TQ_STEP(score(key_off, key_cnt, (int)kSampleEvery));
                TQ_STEP(select(lists, q0, queries, 1, run_if));
            }
            TQ_STEP(score(key_off, key_cnt, 1));
            TQ_STEP(select(lists, q0, queries, 0, run_if));
        }
        return TQ_OK;
    };
    if (!filter) {
        bool prepared = false;
        TQ_STEP(run_candidates(all_lists, 0, qpg, nullptr, [&](int64_t key_off, int64_t key_cnt, int stride) {
            const int rc = score_passes(key_off, key_cnt, stride, nullptr, 0, prepared);
            prepared = true;
            return rc;
        }));
        return tq_merge_keys_launch(best, 1, qpg, groups, topk, idx_base, top_scores, top_idx, st);
    }

    // Filtered search over one group, a pass of queries at a time.  A sample of the keys, spread over all of them, is scored in full
    // and gives every query a first threshold; each round lists the keys of a larger sample (the last round: all keys) whose
    // single-fp16 score plus bound reaches the threshold, gathers them, scores them in full and raises the thresholds; the last
    // round's selection is the result.  With the sizes of the samples a geometric series, every round lists about ratio * topk keys
    // per query.  Data that lists more than a round has room for (long runs of equal scores, say), and queries that the bound
    // does not cover, set a flag on the device, upon which the rest of the rounds does nothing and the unfiltered procedure for
    // this many keys, else skipped, does the pass.
    TqFilterPass f{};
    f.cap = kFilterRoom; f.room = kFilterRoom; f.beta_scale = p->beta_scale;
    f.fprep = sc + fp.off_prep;
    f.bad = reinterpret_cast<unsigned int*>(sc + fp.off_words);
    f.gathered = f.bad + 1;
    f.expected = f.bad + 2;
    f.rows = reinterpret_cast<unsigned int*>(sc + fp.off_rows);
    f.offsets = reinterpret_cast<unsigned int*>(sc + fp.off_offsets);
    f.g_codes = reinterpret_cast<uint32_t*>(sc + fp.off_codes);
    f.g_signs = reinterpret_cast<uint32_t*>(sc + fp.off_signs);
    f.g_norms = reinterpret_cast<float*>(sc + fp.off_norms);
    f.g_rnorms = reinterpret_cast<float*>(sc + fp.off_rnorms);
    f.g_rows = reinterpret_cast<unsigned int*>(sc + fp.off_grows);
    f.scores = reinterpret_cast<float*>(sc + fp.off_scores);
    const Keys gathered{f.g_codes, f.g_signs, f.g_rnorms, f.g_norms, kFilterRoom, f.gathered};
    const int64_t tiles = (keys_per_group + kTileKeys - 1) / kTileKeys;
    const int stride0 = (int)fp.stride0;
    for (int q0 = 0; q0 < qpg; q0 += pass) {
        const int nq = qpg - q0 < pass ? qpg - q0 : pass;
        // (rows of the pass's own arrays, addressed as the scoring kernel does: by the number of the query in the call)
        const Lists sample{reinterpret_cast<unsigned long long*>(sc + fp.off_sample) - q0 * fp.first, fp.first};
        f.nq = nq; f.qpad = pad_of(nq);
        f.thr = thr + q0; f.cnt = cnt + q0; f.best = best + (int64_t)q0 * topk;
        TQ_CUDA_TRY(cudaMemsetAsync(f.bad, 0, (2 + kFilterRounds) * sizeof(unsigned int), st));
        TQ_STEP(init(q0, nq, fp.first, nullptr));
        TQ_STEP(prepare_pass(q0, nq));
        TQ_STEP(score_pass(all_keys, q0, nq, 0, keys_per_group, stride0, nullptr, 0, sample, nullptr));
        TQ_STEP(tq_launch_filter_prep(p, prep, f.qpad, nq, p->c_max, p->beta_scale, f.fprep, f.bad, st));
        // rounds: the fewest whose ratio keeps the lists of all queries within two thirds of the room
        const double span = (double)tiles / (double)(fp.first / kTileKeys), most = 0.66 * kFilterRoom / ((double)nq * topk);
        TqFilterRounds rounds{1, {}};
        while (pow(span, 1.0 / rounds.rounds) > most && rounds.rounds < kFilterRounds) ++rounds.rounds;
        int strides[kFilterRounds];
        for (int r = 0; r < rounds.rounds; ++r) {
            strides[r] = r + 1 == rounds.rounds ? 1 : (int)std::max(1.0, stride0 / pow(span, (double)(r + 1) / rounds.rounds));
            rounds.keys[r] = (float)(((tiles + strides[r] - 1) / strides[r]) / (double)(fp.first / kTileKeys));
        }
        TQ_STEP(tq_launch_sample_threshold(f, rounds, sample.at + q0 * fp.first, fp.first, topk, st));
        for (int r = 0; r < rounds.rounds; ++r) {
            const int stride = strides[r];
            TQ_STEP(tq_launch_filter(p, f, codes, signs, rnorms, norms, keys_per_group, stride, st));
            TQ_STEP(tq_launch_filter_gather(p, f, codes, signs, rnorms, norms, st));
            TQ_STEP(score_pass(gathered, q0, nq, 0, kFilterRoom, 1, f.scores - (int64_t)q0 * kFilterRoom, kFilterRoom, all_lists, nullptr));
            TQ_STEP(tq_launch_filter_select(f, topk, k2, r + 1 == rounds.rounds, fp.matrix, st));
        }
        float* pass_scores = top_scores + (int64_t)q0 * topk;
        int64_t* pass_idx = top_idx + (int64_t)q0 * topk;
        if (!fp.matrix) {
            const Lists chunk{reinterpret_cast<unsigned long long*>(sc + fp.off_cand) - q0 * cp.cand_cap, cp.cand_cap};
            TQ_STEP(run_candidates(chunk, q0, nq, f.bad, [&](int64_t key_off, int64_t key_cnt, int stride) {
                return score_pass(all_keys, q0, nq, key_off, key_cnt, stride, nullptr, 0, chunk, f.bad);
            }));
        }
        TQ_STEP(tq_merge_keys_launch(f.best, 1, nq, 1, topk, idx_base, pass_scores, pass_idx, st));
        if (fp.matrix) {
            float* mat = reinterpret_cast<float*>(sc + fp.off_matrix);
            unsigned long long* part = reinterpret_cast<unsigned long long*>(sc + fp.off_part);
            TQ_STEP(score_pass(all_keys, q0, nq, 0, keys_per_group, 1, mat - (int64_t)q0 * keys_per_group, keys_per_group, all_lists, f.bad));
            topk_rows_kernel<<<dim3((unsigned)fp.segs, (unsigned)nq), kSelThreads, 0, st>>>(
                mat, keys_per_group, (int64_t)nq * keys_per_group, nq, keys_per_group, kSegLen, group_rows, 0, topk, k2, (int)fp.segs, 0, part, f.bad);
            tq_count_launch();
            TQ_CUDA_TRY(cudaGetLastError());
            TQ_STEP(tq_merge_keys_launch(part, (int)fp.segs, nq, 1, topk, idx_base, pass_scores, pass_idx, st, f.bad));
        }
    }
    return TQ_OK;
}
