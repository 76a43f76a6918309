// Top-k search over many keys, first stage: which keys can be among the k best of a query at all?
//
//   score(q, key) = norm * ( (R q) . codebook[codes]  +  alpha * rnorm * ((S q) . signs) )
//
// The scoring kernel of tq_score_tc.cu needs three contractions and two accumulators per key to carry the scores to
// float32 accuracy, although nearly every score only loses against its query's threshold.  This kernel computes the scores
// from single fp16 operands instead -- centroids, and signs scaled by alpha * rnorm in the operand itself, so that both
// terms add up in ONE accumulator -- together with a bound of their error, and lists the keys whose score plus bound
// reaches the threshold.  The listed keys, a few thousand per query, are gathered and scored by the full-accuracy
// kernel, and the selection works on those scores alone: the result is the one of scoring everything.
//
// Error of the single-fp16 score, in units of the sum without the norm: rounding to fp16 changes every operand by at most
// 2^-11 of itself, so the two inner products are off by at most (2^-10 + 2^-22) |c| |Rq| and (2^-10 + 2^-22) alpha rnorm sqrt(d)
// |Sq|, with |c| <= sqrt(d) max |codebook|; kBound = 2.3 * 2^-11 leaves room for the float32 sums of the tensor pipe.  With
// A = kBound sqrt(d) max|c| |Rq| per query and kappa = alpha max|Sq| / (max|c| |Rq|) over the queries, the bound of a key's score is
// |norm| (1 + kappa |rnorm|) A: one multiply-add per score on top of the threshold test.
//
// Per tile of 128 keys: bulk copies of codes, signs, norms (ring of up to 8 tiles) -> expander warps (pair lookup table of half2
// centroids, sign bits xor-ed onto +-beta; tcgen05.st) -> per 16 coordinates one contraction of N = queries for the centroids and
// one for the signs -> epilogue warps (threshold test in fma.rn.f32x2 against a value that holds threshold and bound of the
// warp's 32 keys, one maximum per thread; survivors through a staging list per warp).  16 instructions of N = 64 at d = 128 (530
// cycles) stand against 400 cycles of HBM time.  Expanders and epilogue warps come in two groups that take tiles in turn:
// what a warp does for a tile is a chain of waits (barrier, loads, tensor-memory round trip) twice as long as a tile may take
// (one group with half the work per thread and tile: 2,140 cycles per tile).
#include "tq_common.cuh"
#include "tq_ptx.cuh"
#include "tq_topk.cuh"
#include "tq_filter.cuh"

#include <math.h>
#include <math_constants.h>

namespace {

using namespace tqptx;
using namespace tqtopk;

constexpr int kTileKeys = 128;
constexpr int kW = 128;                       // coordinates per pass through the operand buffers
constexpr int kRowBytes = kW * 2;             // one query row of one operand matrix
constexpr float kCentScale = 1024.f;
constexpr float kBetaMax = 60000.f;           // largest scaled alpha * rnorm that fits fp16; other keys are listed unseen
constexpr int kMaxStages = 8;
constexpr int kPend = 64;                     // entries of a warp's staging list

enum { FB_K_FULL = 0, FB_K_EMPTY = 8, FB_A_FULL = 16, FB_A_EMPTY = 18, FB_D_FULL = 20, FB_D_EMPTY = 24, FB_B_FULL = 28, FB_COUNT = 30 };

struct FilterArgs {
    const unsigned char* codes;
    const unsigned char* signs;
    const float* norms;
    const float* rnorms;
    const unsigned char* prep;     // FilterPrep of the pass
    const float* codebook;
    const float* thr;              // [nq] lower bound of the k-th best score (-inf: none)
    unsigned int* cnt;             // [nq] entries of each list
    unsigned int* rows;            // [nq][cap] listed rows
    unsigned int* bad;             // non-zero: the search falls back to scoring everything
    int64_t key_cnt, tiles;
    int tile_stride, nq, cap;
    float beta_scale;              // 2^m: the sign operand is alpha * rnorm * 2^m
    float alpha;
    unsigned long long* status;
    int wait_kcycles;
};

template <int BITS, int QP, int DR>
struct FL {
    static constexpr int kHalves = DR == 256 ? 2 : 1;
    static constexpr int kDH = DR / kHalves;
    static constexpr int kSub = kDH / 64;                       // chunks of 32 coordinates per expander thread and half (two threads per key)
    static constexpr int kExpWarps = 16, kEpiWarps = 8;         // two groups each
    static constexpr int kFirstExp = 2, kFirstEpi = 2 + kExpWarps;
    static constexpr int kThreads = (2 + kExpWarps + kEpiWarps) * 32;
    static constexpr int kQT = QP < 32 ? QP : 32;               // queries an epilogue thread holds at a time
    static constexpr int kDBufs = 4;
    static constexpr uint32_t kBufCols = 128, kColSg = 64, kColD = 2 * kBufCols;
    static constexpr int kCodeRow = DR * BITS / 8, kSignRow = DR / 8;
    static constexpr int kNormOff = kTileKeys * (kCodeRow + kSignRow);
    static constexpr int kStage = kNormOff + 2 * kTileKeys * 4;
    static constexpr int kLutBytes = (1 << (2 * BITS)) * 32 * 4;
    static constexpr int kBBytes = kHalves * 2 * QP * kRowBytes;
    static constexpr int kConstBytes = QP * 8;                  // per query: bound A, - threshold (accumulator units)
    static constexpr int kZBytes = kEpiWarps * 2 * QP * 4;      // per warp, tiles in turn: bound of the warp's keys - threshold
    static constexpr int kPendBytes = kEpiWarps * kPend * 8;
    static constexpr int kFixed = kLutBytes + kBBytes + kConstBytes + kZBytes + kPendBytes + 512;
    static constexpr int kFit = (226 * 1024 - kFixed) / kStage;
    static constexpr int kStages = kFit < kMaxStages ? kFit : kMaxStages;
    static_assert(kStages >= 3, "key ring too short");
    static constexpr int off_lut = 0;
    static constexpr int off_b = off_lut + kLutBytes;
    static constexpr int off_const = off_b + kBBytes;
    static constexpr int off_z = off_const + kConstBytes;
    static constexpr int off_pend = off_z + kZBytes;
    static constexpr int off_bars = off_pend + kPendBytes;
    static constexpr int off_ring = off_bars + 512;
    static constexpr int total = off_ring + kStages * kStage;
};

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* v) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_st16p(uint32_t taddr, const uint32_t* v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
// two words of a ring stage, read exactly once
__device__ __forceinline__ void lds_once_u2(uint32_t& x, uint32_t& y, const volatile uint32_t* p) {
    asm volatile("ld.volatile.shared.v2.u32 {%0, %1}, [%2];" : "=r"(x), "=r"(y) : "r"(smem_u32(const_cast<const uint32_t*>(p))));
}
__device__ __forceinline__ float max3(float m, float a, float b) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(m), "f"(a), "f"(b));
    return r;
}

template <int BITS, int QP, int DR>
__global__ void __launch_bounds__(FL<BITS, QP, DR>::kThreads, 1)
score_filter_kernel(const FilterArgs a) {
    using L = FL<BITS, QP, DR>;
    constexpr int kHalves = L::kHalves, kStages = L::kStages, kQT = L::kQT;
    if (__syncthreads_or(*a.bad != 0u)) return;      // (another block may be setting it: one answer for the block)
    extern __shared__ __align__(128) unsigned char smem[];     // (an address the compiler knows: the table lookups fold it in)
    const uint32_t smem_base = smem_u32(smem);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::off_bars);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + FB_COUNT);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t bar0 = smem_u32(bars);
    auto BAR = [&](int i) { return bar0 + 8u * (uint32_t)i; };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float* consts = reinterpret_cast<const float*>(a.prep + L::kBBytes);   // [QP] A in accumulator units, [QP] accumulator units per unit of score, kappa

    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(BAR(FB_K_FULL + i), 1);
            mbar_init(BAR(FB_K_EMPTY + i), (kHalves == 2 ? L::kExpWarps : L::kExpWarps / 2) + L::kEpiWarps / 2);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(BAR(FB_A_FULL + i), L::kExpWarps / 2);
            mbar_init(BAR(FB_A_EMPTY + i), 1);
        }
        for (int i = 0; i < L::kDBufs; ++i) {
            mbar_init(BAR(FB_D_FULL + i), 1);
            mbar_init(BAR(FB_D_EMPTY + i), L::kEpiWarps / 2);
        }
        mbar_init(BAR(FB_B_FULL), 1);
        abort_flag[0] = 0;
        abort_flag[1] = a.wait_kcycles;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {   // pair lookup table, one copy per lane: entry e = (code0 | code1 << BITS) -> half2 of the two centroids * 2^10
        uint32_t* lut = reinterpret_cast<uint32_t*>(smem + L::off_lut);
        for (int i = threadIdx.x; i < (1 << (2 * BITS)) * 32; i += L::kThreads) {
            const int e = i >> 5;
            lut[i] = pack_half2(__ldg(a.codebook + (e & ((1 << BITS) - 1))) * kCentScale, __ldg(a.codebook + (e >> BITS)) * kCentScale);
        }
        // per query: A, -threshold in accumulator units (queries beyond the pass: never reached)
        float* c = reinterpret_cast<float*>(smem + L::off_const);
        for (int q = threadIdx.x; q < QP; q += L::kThreads) {
            c[q * 2] = q < a.nq ? __ldg(consts + q) : 0.f;
            c[q * 2 + 1] = q < a.nq ? -__ldg(a.thr + q) * __ldg(consts + QP + q) : -CUDART_INF_F;
        }
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(tmem_slot), 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const int64_t t0 = a.tiles * (int64_t)blockIdx.x / gridDim.x, t1 = a.tiles * (int64_t)(blockIdx.x + 1) / gridDim.x;

    if (warp == 0) {
        // The whole warp walks the tiles and waits, one elected lane issues: a copy costs the lane of a diverged warp some 300 cycles,
        // and there are four a tile (16,777,216 keys x 64 queries: 740 us with one lane walking, now 708).
        if (elect_one()) {
            mbar_arrive_expect_tx(BAR(FB_B_FULL), L::kBBytes);
            bulk_load(smem_base + L::off_b, a.prep, L::kBBytes, BAR(FB_B_FULL));
        }
        __syncwarp();
        int64_t issued = 0;
        for (int64_t t = t0; t < t1; ++t) {
            const int64_t i = t - t0;
            const int s = (int)(i % kStages);
            if (!warp_wait(BAR(FB_K_EMPTY + s), (uint32_t)((i / kStages) & 1) ^ 1u, abort_flag)) break;
            const int64_t row0 = t * a.tile_stride * kTileKeys;
            const uint32_t dst = smem_base + L::off_ring + s * L::kStage;
            const unsigned char* src[4] = {a.codes + row0 * L::kCodeRow, a.signs + row0 * L::kSignRow,
                                           reinterpret_cast<const unsigned char*>(a.norms + row0),
                                           reinterpret_cast<const unsigned char*>(a.rnorms + row0)};
            constexpr uint32_t off[4] = {0u, (uint32_t)(kTileKeys * L::kCodeRow), (uint32_t)L::kNormOff, (uint32_t)(L::kNormOff + kTileKeys * 4)};
            if (a.key_cnt - row0 >= kTileKeys) {
                if (elect_one()) {
                    mbar_arrive_expect_tx(BAR(FB_K_FULL + s), (uint32_t)L::kStage);
#pragma unroll
                    for (int k = 0; k < 4; ++k) bulk_load(dst + off[k], src[k], (k < 3 ? off[k < 3 ? k + 1 : 3] : (uint32_t)L::kStage) - off[k], BAR(FB_K_FULL + s));
                }
            } else {         // the last tile: what is left of a row of bytes behind a multiple of 16 goes by plain loads
                const uint32_t valid = (uint32_t)(a.key_cnt - row0);
                const uint32_t len[4] = {valid * L::kCodeRow, valid * L::kSignRow, valid * 4u, valid * 4u};
                if (lane == 0) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) copy_tail_words(smem + L::off_ring + s * L::kStage + off[k], src[k], len[k]);
                }
                __syncwarp();
                if (elect_one()) {
                    uint32_t tx = 0;
#pragma unroll
                    for (int k = 0; k < 4; ++k) tx += len[k] & ~15u;
                    mbar_arrive_expect_tx(BAR(FB_K_FULL + s), tx);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (len[k] & ~15u) bulk_load(dst + off[k], src[k], len[k] & ~15u, BAR(FB_K_FULL + s));
                }
            }
            __syncwarp();
            issued = i + 1;
        }
        if (lane == 0 && *abort_flag) {
            // copies armed above may still be on their way into this block's shared memory
            mbar_drain(BAR(FB_B_FULL), 0u);
            for (int64_t ii = issued > kStages ? issued - kStages : 0; ii < issued; ++ii)
                mbar_drain(BAR(FB_K_FULL + (int)(ii % kStages)), (uint32_t)((ii / kStages) & 1));
        }
    } else if (warp == 1) {
        // The whole warp walks the tiles and waits; one elected lane issues, every operand from warp-uniform values.
        const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
        constexpr uint32_t kIdesc = (1u << 4) | ((uint32_t)(QP >> 3) << 17) | ((uint32_t)(kTileKeys >> 4) << 24);
        const uint32_t lbo = 128, sbo = (kW / 8) * 128;
        const uint64_t dq = make_smem_desc(smem_base + L::off_b, lbo, sbo);
        const uint64_t dp = make_smem_desc(smem_base + L::off_b + QP * kRowBytes, lbo, sbo);
        bool go = warp_wait(BAR(FB_B_FULL), 0u, abort_flag);
        for (int64_t t = t0; t < t1 && go; ++t) {
            const int64_t i = t - t0;
            const int db = (int)(i % L::kDBufs);
            const uint32_t acc = tm + L::kColD + db * QP;
#pragma unroll 1
            for (int h = 0; h < kHalves; ++h) {
                const int b = kHalves == 2 ? h : (int)(i & 1);               // the buffer of a group of expanders, and which
                const uint32_t use = (uint32_t)(kHalves == 2 ? i : i >> 1);  // filling of it
                go = warp_wait(BAR(FB_A_FULL + b), use & 1u, abort_flag) &&
                     (h > 0 || warp_wait(BAR(FB_D_EMPTY + db), (uint32_t)((i / L::kDBufs) & 1) ^ 1u, abort_flag));
                if (!go) break;
                tc_fence_after();
                if (elect_one()) {
                    const uint32_t base = tm + b * L::kBufCols;
                    const uint64_t half = (uint64_t)((uint32_t)h * 2u * QP * kRowBytes >> 4);
                    if (h == 0) mma_ts_first(acc, base, dq, kIdesc);
                    else mma_ts_acc(acc, base, dq + half, kIdesc);
                    mma_ts_acc(acc, base + L::kColSg, dp + half, kIdesc);
#pragma unroll 1
                    for (int kb = 1; kb < L::kDH / 16; ++kb) {
                        const uint64_t step = half + (uint64_t)(kb * 2 * lbo >> 4);
                        mma_ts_acc(acc, base + kb * 8, dq + step, kIdesc);
                        mma_ts_acc(acc, base + L::kColSg + kb * 8, dp + step, kIdesc);
                    }
                    if (h == kHalves - 1) mma_commit(BAR(FB_D_FULL + db));
                    mma_commit(BAR(FB_A_EMPTY + b));
                }
                __syncwarp();
            }
        }
    } else if (warp < L::kFirstEpi) {
        // ---- expanders: two threads per key, every second tile (d = 256: every tile, a half of its coordinates) --------
        const int ew = warp - L::kFirstExp, group = ew >> 3, part = (ew >> 2) & 1;
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        constexpr uint32_t kPairMask = ((1u << (2 * BITS)) - 1u) << 7;     // a pair of codes, in place as a table row of 128 bytes
        const uint32_t lane4 = lane * 4;
        for (int64_t t = t0 + (kHalves == 2 ? 0 : group); t < t1; t += kHalves == 2 ? 1 : 2) {
            const int64_t i = t - t0;
            const int s = (int)(i % kStages);
            bool fail = !mbar_wait(BAR(FB_K_FULL + s), (uint32_t)((i / kStages) & 1), abort_flag);
            const unsigned char* stage = smem + L::off_ring + s * L::kStage;
            float rn;
            {
                const int h = kHalves == 2 ? group : 0;
                uint32_t w[L::kSub * BITS + 1], sw[L::kSub];
                {
                    // volatile: executed once, before the stage is released (a plain load may be repeated behind it)
                    const int chunk = (h * 2 + part) * L::kSub;
                    const volatile uint32_t* cw = reinterpret_cast<const volatile uint32_t*>(stage + row * L::kCodeRow) + chunk * BITS;
                    const volatile uint32_t* sg = reinterpret_cast<const volatile uint32_t*>(stage + kTileKeys * L::kCodeRow + row * L::kSignRow) + chunk;
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
                    rn = *reinterpret_cast<const volatile float*>(stage + L::kNormOff + (kTileKeys + row) * 4);
                }
                __threadfence_block();   // every lane's loads from the stage are performed before the stage is released
                __syncwarp();
                if (lane == 0 && !fail) mbar_arrive(BAR(FB_K_EMPTY + s));
                // +-beta: the sign bits of a pair are 16 apart; keys whose beta does not fit fp16 (or is NaN) get 0 and are
                // listed by the epilogue without a look at their score
                const float beta = a.alpha * rn * a.beta_scale;
                const uint32_t beta2 = fabsf(beta) < kBetaMax ? pack_half2(beta, beta) : 0u;
                uint32_t hi[L::kSub * 16], sg[L::kSub * 16];
#pragma unroll
                for (int p = 0; p < L::kSub * 16; ++p) {
                    const int bit = p * 2 * BITS, wi = bit >> 5, sh = bit & 31;
                    uint32_t e;      // the pair's bits moved to bit 7
                    if (sh + 2 * BITS > 32) e = __funnelshift_r(w[wi], w[wi + 1], sh) << 7;
                    else if (sh >= 7) e = w[wi] >> (sh - 7);
                    else e = w[wi] << (7 - sh);
                    hi[p] = *reinterpret_cast<const uint32_t*>(smem + L::off_lut + ((e & kPairMask) | lane4));
                    sg[p] = ((~sw[p >> 4] << (15 - (p & 15))) & 0x80008000u) ^ beta2;
                }
                const uint32_t use = (uint32_t)(kHalves == 2 ? i : i >> 1);
                if (!mbar_wait(BAR(FB_A_EMPTY + group), (use & 1u) ^ 1u, abort_flag)) fail = true;
                tc_fence_after();
                const uint32_t abase = tmem + lane_addr + group * L::kBufCols + part * L::kSub * 16;
#pragma unroll
                for (int c = 0; c < L::kSub; ++c) {
                    tmem_st16p(abase + c * 16, hi + c * 16);
                    tmem_st16p(abase + L::kColSg + c * 16, sg + c * 16);
                }
                tmem_wait_st();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(BAR(FB_A_FULL + group));
            }
        }
    } else {
        // ---- epilogue: one thread per key, every second tile ------------------------------------------
        const int ew = warp - L::kFirstEpi, group = ew >> 2;
        const int quarter = warp & 3;
        const int row = quarter * 32 + lane;
        const uint32_t lane_addr = (uint32_t)(quarter * 32) << 16;
        const float2* cst = reinterpret_cast<const float2*>(smem + L::off_const);
        float* zbuf = reinterpret_cast<float*>(smem + L::off_z) + ew * 2 * QP;
        unsigned long long* pend = reinterpret_cast<unsigned long long*>(smem + L::off_pend) + ew * kPend;
        int n_pend = 0;
        const float kappa = __ldg(consts + 2 * QP);
        auto flush = [&]() {
            __syncwarp();
            for (int e = lane; e < n_pend; e += 32) {
                const unsigned long long v = pend[e];
                const unsigned int q = (unsigned int)(v >> 32);
                const unsigned int pos = atomicAdd(a.cnt + q, 1u);
                if (pos < (unsigned int)a.cap) a.rows[(size_t)q * a.cap + pos] = (unsigned int)v;
                else *a.bad = 1u;
            }
            __syncwarp();
            n_pend = 0;
        };
        for (int64_t t = t0 + group; t < t1; t += 2) {
            const int64_t i = t - t0;
            const int s = (int)(i % kStages);
            const int db = (int)(i % L::kDBufs);
            const int64_t key = t * a.tile_stride * kTileKeys + row;
            bool live = mbar_wait(BAR(FB_K_FULL + s), (uint32_t)((i / kStages) & 1), abort_flag) && key < a.key_cnt;
            const volatile float* nr = reinterpret_cast<const volatile float*>(smem + L::off_ring + s * L::kStage + L::kNormOff);
            const float nrm = nr[row], rn = nr[kTileKeys + row];
            __threadfence_block();   // every lane's loads from the stage are performed before the stage is released
            __syncwarp();
            if (lane == 0) mbar_arrive(BAR(FB_K_EMPTY + s));
            // bound of the warp's keys: the largest |norm| (1 + kappa |rnorm|) times A; keys without a finite one, or whose
            // beta does not fit the operand, are listed whatever their score
            float h = fabsf(nrm) * fmaf(kappa, fabsf(rn), 1.f);
            const bool unseen = live && (!(h < 3.0e38f) || !(fabsf(a.alpha * rn * a.beta_scale) < kBetaMax));
            if (!live || unseen) h = 0.f;
            h = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(h)));
            float* z = zbuf + ((i >> 1) & 1) * QP;
#pragma unroll
            for (int q = 0; q < QP; q += 32)
                if (QP >= 32 || lane < QP) {
                    const float2 c = cst[q + lane];
                    z[q + lane] = fmaf(h, c.x, c.y);
                }
            __syncwarp();
            live = mbar_wait(BAR(FB_D_FULL + db), (uint32_t)((i / L::kDBufs) & 1), abort_flag) && live;
            tc_fence_after();
            const float2 n2 = make_float2(nrm, nrm);
#pragma unroll
            for (int q0 = 0; q0 < QP; q0 += L::kQT) {
                uint32_t acc[L::kQT];
#pragma unroll
                for (int c = 0; c < L::kQT; c += 16) tmem_ld16(tmem + lane_addr + L::kColD + db * QP + q0 + c, acc + c);
                tmem_wait_ld();
                if (q0 + L::kQT >= QP) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(BAR(FB_D_EMPTY + db));
                }
                float best = -CUDART_INF_F;
#pragma unroll
                for (int k = 0; k < L::kQT; k += 4) {
                    const float4 c = *reinterpret_cast<const float4*>(z + q0 + k);
                    const float2 x = __ffma2_rn(n2, make_float2(__uint_as_float(acc[k]), __uint_as_float(acc[k + 1])), make_float2(c.x, c.y));
                    const float2 y = __ffma2_rn(n2, make_float2(__uint_as_float(acc[k + 2]), __uint_as_float(acc[k + 3])), make_float2(c.z, c.w));
                    acc[k] = __float_as_uint(x.x); acc[k + 1] = __float_as_uint(x.y);
                    acc[k + 2] = __float_as_uint(y.x); acc[k + 3] = __float_as_uint(y.y);
                    best = max3(best, x.x, x.y);
                    best = max3(best, y.x, y.y);
                }
                if (!__any_sync(0xffffffffu, live && (best >= 0.f || unseen))) continue;
                uint32_t m = 0;
#pragma unroll
                for (int k = 0; k < L::kQT; ++k) m |= __uint_as_float(acc[k]) >= 0.f ? 1u << k : 0u;
                if (unseen) m = 0xffffffffu;
                if (!live) m = 0u;
                m &= a.nq - q0 >= 32 ? 0xffffffffu : a.nq > q0 ? (1u << (a.nq - q0)) - 1u : 0u;
                uint32_t wm = __reduce_or_sync(0xffffffffu, m);
#pragma unroll 1
                while (wm != 0u) {
                    const int k = __ffs(wm) - 1;
                    wm &= wm - 1u;
                    const bool pass = (m >> k) & 1u;
                    const uint32_t votes = __ballot_sync(0xffffffffu, pass);
                    if (n_pend + __popc(votes) > kPend) flush();
                    if (pass) pend[n_pend + __popc(votes & ((1u << lane) - 1u))] = ((unsigned long long)(q0 + k) << 32) | (unsigned int)key;
                    n_pend += __popc(votes);
                }
            }
        }
        flush();
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

// The single-fp16 operands and the constants of the bound from the prepared queries of a pass (tq_score_tc.cu): prep holds, per
// half of the coordinates, q_hi, q_lo, p_hi, p_lo as K-major core matrices, then per pair of queries two 1 / (scale of q * 2^10) and two 1 / scale of p.
// out: per half q_hi and the rescaled p, then A and the accumulator units per query, then kappa.  grid (qpad), block d.
__global__ void __launch_bounds__(256)
filter_prep_kernel(const unsigned char* __restrict__ prep, int qpad, int nq, int d, float beta_scale, float alpha, float c_max,
                   unsigned char* __restrict__ out, unsigned int* bad) {
    const int halves = d == 256 ? 2 : 1, slot = blockIdx.x, j = threadIdx.x;
    const int half = j >> 7, jh = j & 127;
    const size_t mat = (size_t)qpad * kRowBytes;
    const size_t off = (size_t)(slot / 8) * ((kW / 8) * 128) + (size_t)(jh / 8) * 128 + (size_t)(slot % 8) * 16 + (size_t)(jh % 8) * 2;
    const unsigned char* src = prep + (size_t)half * 4 * mat + off;
    unsigned char* dst = out + (size_t)half * 2 * mat + off;
    const float* scales = reinterpret_cast<const float*>(prep + (size_t)halves * 4 * mat) + (slot >> 1) * 4 + (slot & 1);
    const float2 ds = make_float2(scales[0], scales[2]);
    float* consts = reinterpret_cast<float*>(out + (size_t)halves * 2 * mat);
    auto H = [&](int which) { return __half2float(*reinterpret_cast<const __half*>(src + which * mat)); };
    float rq = H(0) + H(1), sq = H(2) + H(3);
    *reinterpret_cast<__half*>(dst) = *reinterpret_cast<const __half*>(src);
    if (slot >= nq) {
        *reinterpret_cast<__half*>(dst + mat) = __float2half_rn(0.f);
        return;
    }
    // accumulator = units * (score / norm), units = 2^10 * scale of q; the sign operand carries beta_scale already
    const float units = 1.f / ds.x;
    const float p = sq * ds.y * (units / beta_scale);
    *reinterpret_cast<__half*>(dst + mat) = __float2half_rn(p);
    __shared__ float red[3][8];
    float r2 = rq * rq, s2 = (sq * ds.y) * (sq * ds.y), big = fabsf(p) < kBetaMax ? 0.f : 1.f;
    for (int o = 16; o > 0; o >>= 1) {
        r2 += __shfl_xor_sync(0xffffffffu, r2, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
    }
    if ((j & 31) == 0) { red[0][j >> 5] = r2; red[1][j >> 5] = s2; red[2][j >> 5] = big; }
    __syncthreads();
    if (j == 0) {
        for (int w = 1; w < (d + 31) / 32; ++w) { r2 += red[0][w]; s2 += red[1][w]; big = fmaxf(big, red[2][w]); }
        const float rq_norm = sqrtf(r2) * ds.x * kCentScale, sq_norm = sqrtf(s2);      // |R q|, |S q|
        const float bound = 2.3f / 2048.f * 1.0001f * sqrtf((float)d) * c_max * rq_norm * units;
        const float ratio = alpha * sq_norm / (c_max * rq_norm) * 1.0001f;
        consts[slot] = bound;
        consts[qpad + slot] = units;
        if (rq_norm > 0.f && ratio < 1.0e6f && bound < 1.0e30f && units < 1.0e30f && big == 0.f)
            atomicMax(reinterpret_cast<int*>(consts + 2 * qpad), __float_as_int(ratio));      // positive floats order as integers
        else
            *bad = 1u;      // zero, NaN or extreme queries: score everything
    }
}

// The packed rows of every listed key, list after list, so that the scoring kernel can take them as keys of their own.
// Too many entries in all, or an overflown list: bad, and nothing is gathered.  grid (blocks, queries)
__global__ void __launch_bounds__(256)
gather_listed_kernel(const unsigned int* __restrict__ cnt, const unsigned int* __restrict__ rows, int cap, int room, int nq,
                     const uint32_t* __restrict__ codes, const uint32_t* __restrict__ signs, const float* __restrict__ norms,
                     const float* __restrict__ rnorms, int code_words, int sign_words, uint32_t* __restrict__ g_codes,
                     uint32_t* __restrict__ g_signs, float* __restrict__ g_norms, float* __restrict__ g_rnorms,
                     unsigned int* __restrict__ g_rows, unsigned int* __restrict__ offsets, unsigned int* bad, unsigned int* gathered) {
    __shared__ unsigned int s_cnt[64], s_off, s_total;
    const int q = blockIdx.y;
    if (threadIdx.x < nq) s_cnt[threadIdx.x] = cnt[threadIdx.x];
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long total = 0, off = 0;
        for (int i = 0; i < nq; ++i) {
            if (i == q) off = total;
            total += s_cnt[i];
        }
        s_off = (unsigned int)off;
        s_total = *bad != 0u || total > (unsigned long long)room ? 0u : (unsigned int)total;
        if (blockIdx.x == 0) {
            offsets[q] = s_off;
            if (q == 0) {
                *gathered = s_total;
                if (total > (unsigned long long)room) *bad = 1u;
            }
        }
    }
    __syncthreads();
    if (s_total == 0u) return;
    const unsigned int* list = rows + (size_t)q * cap;
    const unsigned int n = s_cnt[q], off = s_off;
    // eight lanes per key (a warp has four keys' trips to memory in flight)
    const int words = code_words + sign_words + 2, l8 = threadIdx.x & 7;
    for (unsigned int e = blockIdx.x * 32 + (threadIdx.x >> 3); e < n; e += gridDim.x * 32) {
        const unsigned int r = __ldg(list + e), to = off + e;
#pragma unroll 3
        for (int w = l8; w < words; w += 8) {
            if (w < code_words) g_codes[(size_t)to * code_words + w] = __ldg(codes + (size_t)r * code_words + w);
            else if (w < code_words + sign_words) g_signs[(size_t)to * sign_words + w - code_words] = __ldg(signs + (size_t)r * sign_words + w - code_words);
            else if (w == code_words + sign_words) g_norms[to] = __ldg(norms + r);
            else g_rnorms[to] = __ldg(rnorms + r);
        }
        if (l8 == 0) g_rows[to] = r;
    }
}

// First thresholds: the topk-th best of a query's sampled scores (list of sortable keys, empty slots 0), or a score just below it.
// Bisection over the sortable bits of the scores, which the block keeps in registers; the lowest 8 bits stay open, so the
// threshold is a lower bound; at -inf it stays open altogether.  NaN scores do not count.  One block per query.
constexpr int kSampleMax = 32768;
constexpr uint32_t kOrderedMinusInf = 0x007fffffu;     // sortable bits
//
// The sample also tells when the lists will be too short, so that the first stage need not run into it: a query's round lists the
// keys that reach its threshold, as many per key as in the sample, until the better ones among them are enough to raise the
// threshold.  Without ties that is ratio * topk; with half of 4,194,304 keys equal the overflowing lists alone cost 1.3 ms.
__global__ void __launch_bounds__(1024)
sample_threshold_kernel(const unsigned long long* __restrict__ cand, int64_t cap, unsigned int* __restrict__ cnt, float* __restrict__ thr, int topk,
                        const TqFilterRounds rounds, unsigned int* __restrict__ expected, int room, unsigned int* bad) {
    __shared__ int total[26];
    const int q = blockIdx.x;
    const unsigned long long* list = cand + (size_t)q * cap;
    const int n = min((int)cnt[q], kSampleMax);
    if (threadIdx.x < 26) total[threadIdx.x] = 0;
    uint32_t v[kSampleMax / 1024];
#pragma unroll
    for (int j = 0; j < kSampleMax / 1024; ++j) {
        const int e = j * 1024 + threadIdx.x;
        v[j] = e < n ? (uint32_t)(__ldcs(list + e) >> 32) : 0u;
        if (v[j] > 0xff800000u) v[j] = 0u;
    }
    __syncthreads();
    auto count = [&](uint32_t from, int slot) {       // sampled scores from `from` on
        int c = 0;
#pragma unroll
        for (int j = 0; j < kSampleMax / 1024; ++j) c += v[j] >= from ? 1 : 0;
        c = __reduce_add_sync(0xffffffffu, c);
        if ((threadIdx.x & 31) == 0 && c) atomicAdd(&total[slot], c);
        __syncthreads();
        return total[slot];
    };
    uint32_t prefix = 0u;
    for (int b = 0; b < 24; ++b) {
        const uint32_t trial = prefix | (0x80000000u >> b);
        if (count(trial, b) >= topk) prefix = trial;
    }
    const bool open = prefix <= kOrderedMinusInf;       // (the bits of -inf with some of them cleared are a NaN)
    const int reach = count(open ? 0u : prefix, 24), better = count(open ? 0xffffffffu : prefix + 256u, 25);
    if (threadIdx.x == 0) {
        if (!open) thr[q] = unordered_bits(prefix);
        cnt[q] = 0u;
        float before = 1.f;
        bool tied = true;
        for (int r = 0; r < rounds.rounds; ++r) {
            tied = tied && (float)better * before < (float)topk;
            const float mine = tied ? (float)reach * rounds.keys[r] : (float)topk * rounds.keys[r] / before;
            before = rounds.keys[r];
            const unsigned int add = (unsigned int)fminf(mine, 1.0e9f);
            if (open || atomicAdd(expected + r, add) + add > (unsigned int)room) *bad = 1u;
        }
    }
}

// One block per query: the k best of the gathered keys' scores.  final: they become the query's best list; otherwise only its
// threshold is raised (the keys will be listed again).  The lists are empty afterwards.  keep_nan: NaN scores rank by their
// bits, as in a selection from a score matrix; else they are left out, as candidate mode does.
__global__ void __launch_bounds__(256)
select_gathered_kernel(const float* __restrict__ scores, int64_t row_stride, const unsigned int* __restrict__ g_rows,
                       const unsigned int* __restrict__ offsets, unsigned int* __restrict__ cnt, unsigned long long* __restrict__ best,
                       float* __restrict__ thr, int topk, int k2, int final, int keep_nan, const unsigned int* bad) {
    __shared__ __align__(16) unsigned long long a[kSelCap];
    __shared__ int hist[256];
    __shared__ int scratch[4];
    __shared__ int count;
    __shared__ unsigned long long cut;
    if (*bad != 0u) return;
    const int q = blockIdx.x;
    const unsigned int n = cnt[q], off = offsets[q];
    const float* mine = scores + (size_t)q * row_stride + off;
    const unsigned int* rows = g_rows + off;
    if (threadIdx.x == 0) { count = 0; cut = 0ull; }
    __syncthreads();
    constexpr unsigned int kBatch = 2048;
    for (unsigned int base = 0; base < n; base += kBatch) {
        if (count + (int)kBatch > kSelCap) {  // uniform: count only changes between barriers
            const int c = count;
            __syncthreads();
            if (c > topk) {
                const unsigned long long kth = block_select_topk(a, c, topk, hist, scratch);
                if (threadIdx.x == 0) { count = topk; cut = kth; }
            }
            __syncthreads();
        }
        const unsigned long long t = cut;
        const unsigned int end = base + kBatch < n ? base + kBatch : n;
        float v[kBatch / 256];
        unsigned int r[kBatch / 256];
#pragma unroll
        for (int j = 0; j < (int)kBatch / 256; ++j) {
            const unsigned int e = base + j * 256 + threadIdx.x;
            v[j] = e < end ? __ldcs(mine + e) : CUDART_NAN_F;
            r[j] = e < end ? __ldg(rows + e) : 0u;
        }
#pragma unroll
        for (int j = 0; j < (int)kBatch / 256; ++j) {
            const bool have = base + j * 256 + threadIdx.x < end;
            if (have && (keep_nan || v[j] == v[j])) {
                const unsigned long long ck = make_key(v[j], r[j]);
                if (ck > t) a[atomicAdd(&count, 1)] = ck;
            }
        }
        __syncthreads();
    }
    const int c = count;
    const int keep = c < topk ? c : topk;
    if (keep < c) block_select_topk(a, c, keep, hist, scratch);
    __syncthreads();
    for (int i = keep + threadIdx.x; i < k2; i += blockDim.x) a[i] = 0ull;
    block_sort_desc(a, k2);
    if (final)
        for (int i = threadIdx.x; i < topk; i += blockDim.x) best[(size_t)q * topk + i] = a[i];
    if (threadIdx.x == 0) {
        // (a NaN above the others: only keys that are listed unseen can still come before it)
        const uint32_t last = keep == topk ? (uint32_t)(a[topk - 1] >> 32) : 0u;
        if (last >= kOrderedMinusInf) thr[q] = unordered_bits(last);
        cnt[q] = 0u;
    }
}

template <int BITS, int QP, int DR>
int launch_filter(const FilterArgs& a, int device, cudaStream_t st) {
    using L = FL<BITS, QP, DR>;
    TQ_GRANT_SMEM((score_filter_kernel<BITS, QP, DR>), L::total, device);
    const int sms = tq_sm_count(device);
    score_filter_kernel<BITS, QP, DR><<<(int)(a.tiles < sms ? a.tiles : sms), L::kThreads, L::total, st>>>(a); tq_count_launch();
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}
template <int BITS, int DR>
int launch_filter_q(const FilterArgs& a, int qpad, int device, cudaStream_t st) {
    if (qpad == 16) return launch_filter<BITS, 16, DR>(a, device, st);
    if (qpad == 32) return launch_filter<BITS, 32, DR>(a, device, st);
    if constexpr (DR != 256) return launch_filter<BITS, 64, DR>(a, device, st);
    else return TQ_ERR_UNSUPPORTED;
}

}  // namespace

size_t tq_filter_prep_bytes(int d, int qpad) { return (size_t)(d == 256 ? 2 : 1) * 2 * qpad * kRowBytes + 2 * qpad * 4 + 16; }

int tq_launch_filter_prep(const tq_plan* p, const unsigned char* prep, int qpad, int nq, float c_max, float beta_scale, unsigned char* out,
                          unsigned int* bad, cudaStream_t st) {
    TQ_CUDA_TRY(cudaMemsetAsync(out + tq_filter_prep_bytes(p->dev.d, qpad) - 16, 0, 16, st));     // kappa
    filter_prep_kernel<<<qpad, p->dev.d == 256 ? 256 : 128, 0, st>>>(prep, qpad, nq, p->dev.d == 256 ? 256 : 128, beta_scale, p->dev.alpha, c_max, out, bad);
    tq_count_launch();
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}

int tq_launch_sample_threshold(const TqFilterPass& f, const TqFilterRounds& rounds, const unsigned long long* cand, int64_t cap, int topk, cudaStream_t st) {
    sample_threshold_kernel<<<f.nq, 1024, 0, st>>>(cand, cap, f.cnt, f.thr, topk, rounds, f.expected, f.room, f.bad); tq_count_launch();
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}

int tq_launch_filter(const tq_plan* p, const TqFilterPass& f, const uint32_t* codes, const uint32_t* signs, const float* rnorms,
                     const float* norms, int64_t keys, int tile_stride, cudaStream_t st) {
    FilterArgs a{};
    a.codes = reinterpret_cast<const unsigned char*>(codes);
    a.signs = reinterpret_cast<const unsigned char*>(signs);
    a.norms = norms; a.rnorms = rnorms;
    a.prep = f.fprep; a.codebook = p->dev.codebook;
    a.thr = f.thr; a.cnt = f.cnt; a.rows = f.rows; a.bad = f.bad;
    a.key_cnt = keys;
    const int64_t tiles = (keys + kTileKeys - 1) / kTileKeys;
    a.tiles = (tiles + tile_stride - 1) / tile_stride;
    a.tile_stride = tile_stride; a.nq = f.nq; a.cap = f.cap;
    a.beta_scale = f.beta_scale; a.alpha = p->dev.alpha;
    a.status = p->status_dev; a.wait_kcycles = p->wait_kcycles;
    int r = TQ_ERR_UNSUPPORTED;
#define TQ_FI(B)                                                                                               \
    case B:                                                                                                    \
        r = p->dev.d == 64 ? launch_filter_q<B, 64>(a, f.qpad, p->device, st)                                   \
            : p->dev.d == 256 ? launch_filter_q<B, 256>(a, f.qpad, p->device, st) : launch_filter_q<B, 128>(a, f.qpad, p->device, st); \
        break;
    switch (p->dev.bits) { TQ_FI(1) TQ_FI(2) TQ_FI(3) TQ_FI(4) }
#undef TQ_FI
    return r == TQ_ERR_UNSUPPORTED ? tq_fail(r, "no filter kernel for d=%d bits=%d", p->dev.d, p->dev.bits) : r;
}

int tq_launch_filter_gather(const tq_plan* p, const TqFilterPass& f, const uint32_t* codes, const uint32_t* signs, const float* rnorms,
                            const float* norms, cudaStream_t st) {
    const int blocks = (8 * tq_sm_count(p->device) + f.nq - 1) / f.nq;
    gather_listed_kernel<<<dim3((unsigned)blocks, (unsigned)f.nq), 256, 0, st>>>(
        f.cnt, f.rows, f.cap, f.room, f.nq, codes, signs, norms, rnorms, p->dev.code_words, p->dev.sign_words, f.g_codes, f.g_signs, f.g_norms,
        f.g_rnorms, f.g_rows, f.offsets, f.bad, f.gathered); tq_count_launch();
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}

int tq_launch_filter_select(const TqFilterPass& f, int topk, int k2, bool final, bool keep_nan, cudaStream_t st) {
    select_gathered_kernel<<<f.nq, 256, 0, st>>>(f.scores, f.room, f.g_rows, f.offsets, f.cnt, f.best, f.thr, topk, k2, final ? 1 : 0, keep_nan ? 1 : 0, f.bad);
    tq_count_launch();
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}
