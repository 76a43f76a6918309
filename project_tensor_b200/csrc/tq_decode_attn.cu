// Decode attention over a quantized key/value cache, d = 128 or 64:
//
//   out[g][a] = softmax_i( scale * score(q[g][a], key[g][i]) ) . value[g][i]
//
// with keys held as TurboQuantProd encodings (score = TurboQuantProd.attention_score, _quant.py:334-358) and
// values as TurboQuantMSE encodings (value = TurboQuantMSE.dequantize, _quant.py:238-254).  It is the caller
// side of attention_score -- scale, softmax, weighted sum of values: scaled_dot_product_attention,
// _core.py:1606-1683 -- done without ever writing the scores or the dequantized values to memory: per key
// the kernel reads the packed key (d*b/8 + d/8 + 8 bytes) and the packed value (d*b/8 + 4 bytes) once.
//
// dequantize is linear after the centroid gather: sum_i p_i * norm_i * (c[idx_i] R) = (sum_i p_i norm_i
// c[idx_i]) R, so the kernel accumulates in the rotated domain and the d x d rotation is applied once per query
// in the combine kernel.
//
// Both contractions -- keys times queries, weights times values -- run on the tensor cores with warp-level matrix
// instructions (m16n8k16, fp16 operands, fp32 sums): the packed codes are expanded in the registers of the lane that
// feeds them to the instruction, which tcgen05 does not offer (its operands go through tensor or shared memory, and the
// expansion, not the arithmetic, is what costs).  To keep 32-bit accuracy every factor is split into fp16 hi + lo:
//
//   scores   B = queries; up to 4 queries: columns 0..3 are q_hi, columns 4..7 q_lo of the same queries; up to 8: one
//            instruction for q_hi and one for q_lo.  A = keys x 16 coordinates; the order of the rows and of the coordinates inside
//            a contraction is free, so lane t of a quad takes d/4 consecutive coordinates of its key -- whole 32-bit words
//            of the packed row (d = 128) -- and the two halves of the instruction's rows are hi and lo of the same 8 keys:
//            one table row is the operand's registers as they are; signs become +-1 by a shift and a logic operation.
//   values   A = 16 coordinates x 16 keys (transposed: a register holds one coordinate of two keys), B = weights p * norm, hi
//            and lo, which reach their lanes from the scores' layout by one 8 x 8 transposition (movmatrix).
//
// The tables sit in shared memory: two codes (four up to 2 bits) select a row of 256 bytes, replicated so that no two lanes of
// a load meet in a bank; a byte permutation makes the address.  The value codes of neighbouring keys are interleaved
// with a shift and a bit-select first.  What bounds it at d = 128, 2-bit keys, 4-bit values: shared-memory lookups (62 % of the
// pipe's cycles; tensor pipe 24 %, integer 38 %) and the latencies of a chain that 12 warps an SM, which is what the registers
// allow, do not fill (47 % of the issue slots).
//
// Every warp walks its own tiles of 16 keys with its own running softmax; there is no barrier inside the loop, and the
// words of the next tile are fetched while a tile is computed.  A score that exceeds the warp's reference by more than
// 2^8 moves the reference (exact softmax: the reference cancels); weights are scaled by a power of two that follows the
// largest weight x norm seen, so that their fp16 hi parts neither overflow nor lose their lo parts.  Key ranges are split
// over blocks; every block leaves (max, sum, accumulator) per query in scratch and decode_combine_kernel merges.
//
// The kernel this replaced scored from per-query lookup tables and accumulated values with one multiply-add per key,
// coordinate and query: 64 groups x 4 queries x 32,768 keys (d = 128, 2 + 1 bit keys, 4-bit values) took 273 us, now 165.
#include "tq_common.cuh"
#include "tq_mma.cuh"

#include <math_constants.h>
#include <stdint.h>

#include <type_traits>

namespace {

using namespace tqmma;

constexpr int kThreads = 384;
constexpr int kWarps = kThreads / 32;
constexpr int kTile = 16;           // keys a warp takes at a time
constexpr int kMaxSplits = 64;
constexpr float kSlack = 8.f;          // a score may exceed the reference of its softmax by 2^kSlack
constexpr float kWeightMax = 32768.f;  // largest scaled weight (fp16 reaches 65,504)

struct DecodeArgs {
    const float* q;              // [groups][qpg][d]
    const uint32_t* kcodes;
    const uint32_t* ksigns;
    const float* krnorms;
    const float* knorms;
    const uint32_t* vcodes;
    const float* vnorms;
    const uint32_t* vparts;      // centroids of the value quantizer, in parts of vunit
    float vunit;
    int qpg;
    int64_t keys_per_group, group_rows;
    const int64_t* length;       // optional device-side number of keys per group (capped by keys_per_group)
    float scale_log2e;           // scale * log2(e): the softmax runs in base 2
    int splits;
    float* part;                 // [groups][qpg][splits][d + 2]: accumulator, running max, running sum
};

template <int KB, int VB, int DR, int NQ>
struct Plan {
    static constexpr int kSteps = DR / 16;            // contraction steps of the scores
    static constexpr int kMTiles = DR / 16;           // 16-coordinate tiles of the output
    static constexpr int kChunkCodes = VB >= 3 ? 8 : DR / 8;   // value codes that are interleaved as one word ...
    static constexpr int kChunks = DR / 8 / kChunkCodes;       // ... and such words per lane and key
    static constexpr int kKeyBits = DR / 4 * KB, kValBits = DR / 8 * VB;      // bits of a packed row that a lane uses
    static constexpr int kKeyRowWords = DR * KB / 32, kValRowWords = DR * VB / 32, kSignRowWords = DR / 32;
    // words a lane loads per row: its bits may start in the middle of a word
    static constexpr int kKW = kKeyBits % 32 == 0 ? kKeyBits / 32 : kKeyBits / 32 + 1;
    static constexpr int kVW = kValBits % 32 == 0 ? kValBits / 32 : (32 % kValBits == 0 ? 1 : 2);
    static constexpr int off_val = table_rows(KB) * kRowBytes;           // value table behind the key table
    static constexpr int kTables = off_val + (1 << (2 * VB)) * kRowBytes;
    static constexpr int kFragBytes = kSteps * 32 * 16;      // one query operand (NQ = 8): hi and lo registers per lane
    static constexpr int kMerge = kWarps * kMTiles * 4 * 32 * 4;      // accumulators of the warps, over the tables at the end
    // The queries are rotated and projected by all threads at once: four consecutive outputs of one matrix and a slice
    // of the sum per thread, so that both matrices are on their way from the L2 cache in one go.
    static constexpr int kSlices = kThreads / (DR / 2), kSliceLen = (DR + kSlices - 1) / kSlices;
    static constexpr int kLuts = kTables > kMerge ? kTables : kMerge;
    static constexpr int off_frag = kLuts;                               // two query operands
    static constexpr int off_slice = off_frag + (NQ == 8 ? 2 * kFragBytes : 0);   // [kSlices][2][NQ][DR] partial sums
    static constexpr int off_ops = off_slice + kSlices * 2 * NQ * DR * 4;         // four queries: [2][NQ][hi, lo][operand_row(DR)] fp16
    static constexpr int off_qin = off_ops + (NQ == 4 ? (2 * NQ * 2 * operand_row(DR) * 2 + 15) / 16 * 16 : 0);   // [DR][NQ]
    static constexpr int off_small = off_qin + NQ * DR * 4;              // [2][NQ] scales, [kWarps][NQ] max, sum, factor
    static constexpr int total = off_small + (2 * NQ + 3 * kWarps * NQ) * 4;
};

// Packed words of one tile of 16 keys, as the lanes of a warp hold them.
template <class P>
struct TileWords {
    uint32_t kc[2][P::kKW], sg[2][1], vc[4][P::kVW];
    float kn[2], rn[2], vn[2];
};

// grid (splits, passes over the queries of a group, groups)
template <int KB, int VB, int DR, int NQ>
__global__ void __launch_bounds__(kThreads, 1)
decode_partial_kernel(TqDev kp, DecodeArgs a) {
    using P = Plan<KB, VB, DR, NQ>;
    extern __shared__ __align__(128) unsigned char smem[];
    __half* ops = reinterpret_cast<__half*>(smem + P::off_ops);
    (void)ops;
    float* qin = reinterpret_cast<float*>(smem + P::off_qin);
    int* scl = reinterpret_cast<int*>(smem + P::off_small);                   // exponents of the queries' scales
    float* wm = reinterpret_cast<float*>(smem + P::off_small) + 2 * NQ;                                                    // [kWarps][NQ]
    float* wl = wm + kWarps * NQ;
    float* wf = wl + kWarps * NQ;

    const int g = blockIdx.z, q0 = blockIdx.y * NQ, split = blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = lane & 3, r = lane >> 2;      // position in the quad, row of the fragments
    int64_t n = a.keys_per_group;
    if (a.length) {
        const int64_t len = tq_cache_length(a.length);      // (an append on another stream may be at work on the word)
        n = len < n ? len : n;
    }
    const uint32_t keys = (uint32_t)n;           // rows of all groups together stay below 2^32
    const uint32_t tiles_total = (uint32_t)((n + kTile - 1) / kTile), tps = (tiles_total + a.splits - 1) / a.splits;
    const uint32_t tile1 = min((uint32_t)(split + 1) * tps, tiles_total);
    uint32_t tile = (uint32_t)split * tps + warp;

    // ---- packed words of a tile -----------------------------------------------------------------
    // Row r of the score fragments is key (r >> 1) + 4 (r & 1) (+ 8) of the tile, so that the keys 2t, 2t + 1, 2t + 8,
    // 2t + 9 of the value fragments are t, t + 4, t + 8, t + 12: every load of a warp covers consecutive rows.
    const int64_t row_base = (int64_t)g * a.group_rows;
    const int kbit = P::kKeyBits * t, kword = kbit >> 5, kshift = kbit & 31;
    const int vbit = P::kValBits * r, vword = vbit >> 5, vshift = vbit & 31;
    const uint32_t key_r = (uint32_t)((r >> 1) + 4 * (r & 1));
    const uint32_t* kc_base = a.kcodes + row_base * P::kKeyRowWords + kword;
    const uint32_t* sg_base = a.ksigns + row_base * P::kSignRowWords + (DR == 128 ? t : t >> 1);
    const uint32_t* vc_base = a.vcodes + row_base * P::kValRowWords + vword;
    const int vnext = vword + 1 < P::kValRowWords ? 1 : 0;
    const float* kn_base = a.knorms + row_base;
    const float* rn_base = a.krnorms + row_base;
    const float* vn_base = a.vnorms + row_base;
    auto fetch = [&](uint32_t tl, TileWords<P>& w) {
        const uint32_t k0 = tl * kTile, last = keys - 1;       // rows behind the last one: read that one, its weight will be zero
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t key = min(k0 + key_r + 8 * h, last);
            const uint32_t* src = kc_base + (size_t)key * P::kKeyRowWords;
            if constexpr (P::kKW == 4) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(src));
                w.kc[h][0] = v.x; w.kc[h][1] = v.y; w.kc[h][2] = v.z; w.kc[h][3] = v.w;
            } else if constexpr (P::kKeyBits == 64) {
                const uint2 v = __ldg(reinterpret_cast<const uint2*>(src));
                w.kc[h][0] = v.x; w.kc[h][1] = v.y;
            } else {
#pragma unroll
                for (int i = 0; i < P::kKW; ++i) w.kc[h][i] = __ldg(src + i);
            }
            w.sg[h][0] = __ldg(sg_base + (size_t)key * P::kSignRowWords);
            w.kn[h] = __ldg(kn_base + key);
            w.rn[h] = __ldg(rn_base + key);
            w.vn[h] = __ldg(vn_base + key);
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const uint32_t* src = vc_base + (size_t)min(k0 + t + 4 * h, last) * P::kValRowWords;
            if constexpr (P::kValBits == 64) {
                const uint2 v = __ldg(reinterpret_cast<const uint2*>(src));
                w.vc[h][0] = v.x; w.vc[h][1] = v.y;
            } else {
                w.vc[h][0] = __ldg(src);
                if constexpr (P::kVW == 2) w.vc[h][1] = __ldg(src + vnext);
            }
        }
    };
    TileWords<P> cur;
    if (tile < tile1) fetch(tile, cur);        // on its way while the block prepares

    // ---- tables and queries -----------------------------------------------------------------------
    for (int i = tid; i < NQ * DR; i += kThreads) {
        const int qq = i / DR, k = i - qq * DR;
        qin[k * NQ + qq] = q0 + qq < a.qpg ? __ldg(a.q + ((size_t)g * a.qpg + q0 + qq) * DR + k) : 0.f;
    }
    const int xm = tid / (DR / 4) & 1, xj = tid % (DR / 4) * 4, xs = tid / (DR / 2), xk = xs * P::kSliceLen;    // matrix, first output, slice
    float4 mat[P::kSliceLen];
    {
        const float* src = (xm ? kp.St : kp.Rt) + xj;
#pragma unroll
        for (int u = 0; u < P::kSliceLen; ++u)
            mat[u] = xk + u < DR ? __ldg(reinterpret_cast<const float4*>(src + (size_t)(xk + u) * DR)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    // Key table, row e: 128 bytes of copies of (hi, lo) of a pair of codes, or (hi, lo, hi, lo) of four codes: the registers
    // of an A operand.  Value table: 32 copies of hi, 32 copies of lo of the same coordinate of two keys.  A thread fills whole
    // rows, starting at a copy of its own (stores to rows 256 bytes apart would all hit the same banks).
    build_key_table<KB>(smem, kp.cent_parts, tid, kThreads);
    for (int e = kThreads - 1 - tid; e < 1 << (2 * VB); e += kThreads) {
        uint32_t hi, lo;
        pair_parts(__ldg(a.vparts + (e & ((1 << VB) - 1))), __ldg(a.vparts + (e >> VB)), hi, lo);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            *reinterpret_cast<uint4*>(smem + P::off_val + e * kRowBytes + ((i + tid) & 7) * 16) = make_uint4(hi, hi, hi, hi);
            *reinterpret_cast<uint4*>(smem + P::off_val + e * kRowBytes + 128 + ((i + tid) & 7) * 16) = make_uint4(lo, lo, lo, lo);
        }
    }
    __syncthreads();
    // rotated[j] = sum_k q[k] R[j][k], projected[j] = sum_k q[k] S[j][k] in 32-bit arithmetic
    float* slice = reinterpret_cast<float*>(smem + P::off_slice);
    {
#pragma unroll
        for (int qq = 0; qq < NQ; ++qq) {
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
            if (q0 + qq < a.qpg) {
#pragma unroll
                for (int u = 0; u < P::kSliceLen; ++u) {
                    const float v = qin[min(xk + u, DR - 1) * NQ + qq];       // (meets a matrix element of zero behind the end)
                    sum.x = fmaf(v, mat[u].x, sum.x);
                    sum.y = fmaf(v, mat[u].y, sum.y);
                    sum.z = fmaf(v, mat[u].z, sum.z);
                    sum.w = fmaf(v, mat[u].w, sum.w);
                }
            }
            *reinterpret_cast<float4*>(slice + ((xs * 2 + xm) * NQ + qq) * DR + xj) = sum;
        }
    }
    __syncthreads();
    // A warp per vector: slices added up, scale, fp16 hi and lo parts where the operands are read.  Up to 4 queries: rows of parts, from
    // which lane t of a quad takes the coordinates [t DR / 4, + DR / 4), four a step.  Up to 8: (hi b0, hi b1, lo b0, lo b1) of query r
    // per lane and step.
    for (int v = warp; v < 2 * NQ; v += kWarps) {
        float x[DR / 32], m = 0.f;
#pragma unroll
        for (int i = 0; i < DR / 32; ++i) {
            const int k = lane + 32 * i;
            x[i] = slice[v * DR + k];
#pragma unroll
            for (int u = 1; u < P::kSlices; ++u) x[i] += slice[(u * 2 * NQ + v) * DR + k];
            m = fmaxf(m, fabsf(x[i]));
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        const int e = scale_exp(m);
        const float sc = pow2i(e);
        if (lane == 0) scl[v] = e;
#pragma unroll
        for (int i = 0; i < DR / 32; ++i) {
            const int k = lane + 32 * i;
            const float y = x[i] * sc;
            const __half hi = __float2half_rn(y), lo = __float2half_rn(y - __half2float(hi));
            if constexpr (NQ == 4) {
                ops[(v * 2) * operand_row(DR) + k] = hi;
                ops[(v * 2 + 1) * operand_row(DR) + k] = lo;
            } else {
                const int step = k % (DR / 4) / 4, to = v % NQ * 4 + k / (DR / 4);
                __half* at = reinterpret_cast<__half*>(smem + P::off_frag + v / NQ * P::kFragBytes + (step * 32 + to) * 16) + k % 4;
                at[0] = hi;
                at[4] = lo;
            }
        }
    }
    __syncthreads();
    // Query operands of up to 4 queries: column r is hi (r < 4) or lo (r >= 4) of query r & 3.
    constexpr int kRegSteps = NQ == 4 ? P::kSteps : 1;
    uint32_t qf[2][kRegSteps][2];
    if constexpr (NQ == 4) {
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const uint2* x = reinterpret_cast<const uint2*>(ops + ((m * NQ + (r & 3)) * 2 + (r >> 2)) * operand_row(DR) + t * (DR / 4));
#pragma unroll
            for (int s = 0; s < P::kSteps; ++s) {
                const uint2 w = x[s];
                qf[m][s][0] = w.x;
                qf[m][s][1] = w.y;
            }
        }
    }
    // The two queries of this lane's score columns: descaling factors, softmax state.
    float ds1[2], ds2[2], mref[2], lsum[2];
    float wsc[2];                     // power of two that scales the weights
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int qq = (2 * t + c) & (NQ - 1);
        ds1[c] = pow2i(-scl[qq]) * kp.cent_unit;
        ds2[c] = pow2i(-scl[NQ + qq]) * kp.alpha;
        mref[c] = -CUDART_INF_F;
        lsum[c] = 0.f;
        wsc[c] = pow2i(126);
    }
    float acc[P::kMTiles][4];
#pragma unroll
    for (int i = 0; i < P::kMTiles; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;

    // Table lookups.  A byte of a word selects a row with one byte permutation: (lane's copy, byte, 0, 0) is its address.
    const uint32_t lane4 = (uint32_t)lane * 4u, lane8 = (uint32_t)(lane & 15) * 8u, lane16 = (uint32_t)(lane & 7) * 16u;
    auto pick = [&](uint32_t word, int byte, uint32_t copy) { return __byte_perm(word, copy, 0x5504u | (uint32_t)byte << 4); };

    // ---- tiles ----------------------------------------------------------------------------------------
    tq_grid_release();      // (the blocks that merge may take an SM when its last block here has ended)
    for (; tile < tile1; tile += kWarps) {
        TileWords<P> nxt;
        if (tile + kWarps < tile1) fetch(tile + kWarps, nxt);
        const uint32_t left = keys - tile * kTile;      // keys of this tile and behind it
        // -- scores
        KeyWords<KB, DR> key;
        key.unpack(cur.kc, cur.sg, kshift, t);
        float s[2][2] = {{0.f, 0.f}, {0.f, 0.f}};                 // [key r + 8 h][query column c]
        auto half = [&](auto first) {       // (a chain of half the coordinates: the tensor pipe truncates its sums at every instruction)
            float c1[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, c2[4] = {0.f, 0.f, 0.f, 0.f};
            for_steps<P::kSteps / 2>([&](auto sc) {
                constexpr int s = decltype(first)::value + decltype(sc)::value;
                uint32_t ak[2][4], as[4];
                key.template operands<s>(smem, lane8, lane16, ak, as);
                if constexpr (NQ == 4) {
                    mma16816(c1[0], ak[0], qf[0][s][0], qf[0][s][1]);
                    mma16816(c1[1], ak[1], qf[0][s][0], qf[0][s][1]);
                    mma16816(c2, as, qf[1][s][0], qf[1][s][1]);
                } else {
                    const uint4 b = *reinterpret_cast<const uint4*>(smem + P::off_frag + (s * 32 + lane) * 16);
                    const uint4 p = *reinterpret_cast<const uint4*>(smem + P::off_frag + P::kFragBytes + (s * 32 + lane) * 16);
                    mma16816(c1[0], ak[0], b.z, b.w);
                    mma16816(c1[1], ak[1], b.z, b.w);
                    mma16816(c2, as, p.z, p.w);
                    mma16816(c1[0], ak[0], b.x, b.y);
                    mma16816(c1[1], ak[1], b.x, b.y);
                    mma16816(c2, as, p.x, p.y);
                }
            });
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int c = 0; c < 2; ++c) s[h][c] += fmaf(c2[2 * h + c] * ds2[c], cur.rn[h], (c1[h][c] + c1[h][2 + c]) * ds1[c]);
        };
        half(std::integral_constant<int, 0>{});
        half(std::integral_constant<int, P::kSteps / 2>{});
        // the exponent of key r + 8 h is s * f[h]; keys behind the last: -inf
        float f[2];
        bool above = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const bool have = key_r + 8 * h < left;
            f[h] = have ? cur.kn[h] * a.scale_log2e : 1.f;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                if constexpr (NQ == 4) s[h][c] += __shfl_xor_sync(0xffffffffu, s[h][c], 2);     // hi and lo columns
                if (!have) s[h][c] = -CUDART_INF_F;
                above = above || s[h][c] * f[h] > mref[c] + kSlack;
            }
        }
        // -- softmax reference and weights
        if (__any_sync(0xffffffffu, above)) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float m = fmaxf(s[0][c] * f[0], s[1][c] * f[1]);
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                m = fmaxf(m, mref[c]);
                if (m > mref[c]) {
                    const float step = m - mref[c];      // +inf the first time: nothing to carry over
                    const int e0 = (int)(__float_as_uint(wsc[c]) >> 23) - 127, up = step < 252.f ? (int)step : 252;
                    const int e = min(126, e0 + up);          // older weights shrink by 2^-step: their scale may grow
                    const float fl = exp2f(-step), fw = exp2f((float)(e - e0) - step);
                    lsum[c] *= fl;
                    wsc[c] = pow2i(e);
                    mref[c] = m;
#pragma unroll
                    for (int i = 0; i < P::kMTiles; ++i) { acc[i][c] *= fw; acc[i][2 + c] *= fw; }
                }
            }
        }
        float u[2][2];
        bool big = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float vn = key_r + 8 * h < left ? cur.vn[h] : 0.f;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                // (one rounding, of the difference: the exponents near the reference are the ones that count)
                const float p = exp2f(fmaf(s[h][c], f[h], mref[c] == -CUDART_INF_F ? 0.f : -mref[c]));
                lsum[c] += p;
                u[h][c] = p * vn;
                big = big || u[h][c] * wsc[c] > kWeightMax;
            }
        }
        if (__any_sync(0xffffffffu, big)) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float m = fmaxf(u[0][c], u[1][c]);
#pragma unroll
                for (int o = 4; o < 32; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                if (m * wsc[c] > kWeightMax) {
                    const int e0 = (int)(__float_as_uint(wsc[c]) >> 23) - 127;
                    const int e = max(13 - (int)((__float_as_uint(m) >> 23) - 127), -126);     // the largest becomes 2^13 .. 2^14
                    const float fw = pow2i(e - e0) * (e - e0 < -126 ? 0.f : 1.f);
                    wsc[c] = pow2i(e);
#pragma unroll
                    for (int i = 0; i < P::kMTiles; ++i) { acc[i][c] *= fw; acc[i][2 + c] *= fw; }
                }
            }
        }
        uint32_t bh[2], bl[2];          // weights as the B operand: keys 2t, 2t + 1 (+ 8 h) of column r
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            uint32_t hi, lo;
            split_pair(u[h][0] * wsc[0], u[h][1] * wsc[1], hi, lo);
            if constexpr (NQ == 4) {
                bh[h] = transpose8x8(t < 2 ? hi : lo);
            } else {
                bh[h] = transpose8x8(hi);
                bl[h] = transpose8x8(lo);
            }
        }
        // -- values
        uint32_t ve[2][P::kChunks], vo[2][P::kChunks], ve1[2], vo1[2];     // per pair of keys: even and odd coordinates, codes of both keys side by side
        (void)ve1; (void)vo1;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int ch = 0; ch < P::kChunks; ++ch) {
                uint32_t x[2];
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    const uint32_t w0 = cur.vc[2 * h + y][0], w1 = cur.vc[2 * h + y][P::kVW - 1];
                    constexpr int kAt = P::kChunkCodes * VB;            // bits of a chunk
                    if constexpr (P::kValBits == 64) x[y] = ch == 0 ? w0 : w1;
                    else if constexpr (P::kVW == 2) x[y] = ch == 0 ? __funnelshift_r(w0, w1, vshift) : (uint32_t)((((uint64_t)w1 << 32) | w0) >> (vshift + kAt));
                    else x[y] = P::kValBits % 32 == 0 ? w0 : w0 >> vshift;
                }
                constexpr uint32_t kEven = VB == 4 ? 0x0f0f0f0fu : VB == 3 ? 0x001c71c7u : VB == 2 ? 0x33333333u : 0x55555555u;
                ve[h][ch] = (x[0] & kEven) | ((x[1] << VB) & (kEven << VB));
                vo[h][ch] = ((x[0] >> VB) & kEven) | (x[1] & (kEven << VB));
            }
        }
        if constexpr (VB == 2) {            // a field is a nibble: even ones and odd ones in words of their own
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                ve1[h] = (ve[h][0] >> 4) & 0x0f0f0f0fu; ve[h][0] &= 0x0f0f0f0fu;
                vo1[h] = (vo[h][0] >> 4) & 0x0f0f0f0fu; vo[h][0] &= 0x0f0f0f0fu;
            }
        }
        auto value_tile = [&](auto mc) {
            constexpr int mt = decltype(mc)::value;
            uint32_t ah[4], al[4];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                auto row = [&](const uint32_t (&w)[P::kChunks], uint32_t w1) {
                    if constexpr (VB == 4) return pick(w[mt >> 2], mt & 3, lane4);
                    else if constexpr (VB == 3) return (shl<8 - 6 * (mt & 3)>(w[mt >> 2]) & 0x3f00u) | lane4;
                    else if constexpr (VB == 2) return pick(mt & 1 ? w1 : w[0], mt >> 1, lane4);
                    else return (shl<8 - 2 * mt>(w[0]) & 0x300u) | lane4;
                };
                const uint32_t e = row(ve[h], ve1[h]), o = row(vo[h], vo1[h]);
                ah[2 * h] = *reinterpret_cast<const uint32_t*>(smem + P::off_val + e);
                al[2 * h] = *reinterpret_cast<const uint32_t*>(smem + P::off_val + 128 + e);
                ah[2 * h + 1] = *reinterpret_cast<const uint32_t*>(smem + P::off_val + o);
                al[2 * h + 1] = *reinterpret_cast<const uint32_t*>(smem + P::off_val + 128 + o);
            }
            // A tile's products, small ones first, in sums of their own that are rounded onto the accumulator: the tensor pipe
            // truncates, which over a long context (32,768 keys: seven times the error) is a bias.
            float c[4] = {0.f, 0.f, 0.f, 0.f};
            mma16816(c, al, bh[0], bh[1]);
            if constexpr (NQ == 8) mma16816(c, ah, bl[0], bl[1]);
            mma16816(c, ah, bh[0], bh[1]);
#pragma unroll
            for (int i = 0; i < 4; i += 2) {
                const float2 v = __fadd2_rn(make_float2(acc[mt][i], acc[mt][i + 1]), make_float2(c[i], c[i + 1]));
                acc[mt][i] = v.x;
                acc[mt][i + 1] = v.y;
            }
        };
        for_steps<P::kMTiles>(value_tile);
        cur = nxt;
    }

    // ---- merge the warps -----------------------------------------------------------------------------------
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        float v = lsum[c];
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (r == 0 && 2 * t < NQ) {
            wm[warp * NQ + 2 * t + c] = mref[c];
            wl[warp * NQ + 2 * t + c] = v;
        }
    }
    __syncthreads();          // maxima in place; the tables are no longer needed
    for (int qq = tid; qq < NQ; qq += kThreads) {
        float m = -CUDART_INF_F, l = 0.f;
        for (int w = 0; w < kWarps; ++w) m = fmaxf(m, wm[w * NQ + qq]);
        for (int w = 0; w < kWarps; ++w) {
            const float f = wm[w * NQ + qq] == -CUDART_INF_F ? 0.f : exp2f(wm[w * NQ + qq] - m);
            wf[w * NQ + qq] = f;
            l = fmaf(f, wl[w * NQ + qq], l);
        }
        if (q0 + qq < a.qpg) {
            float* dst = a.part + (((size_t)g * a.qpg + q0 + qq) * a.splits + split) * (DR + 2);
            dst[DR] = m;
            dst[DR + 1] = l;
        }
    }
    // accumulators as the lanes hold them, [warp][tile][register][lane]
    float* wacc = reinterpret_cast<float*>(smem);
    constexpr int kAcc = P::kMTiles * 4 * 32;
#pragma unroll
    for (int i = 0; i < P::kMTiles; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) wacc[warp * kAcc + (i * 4 + c) * 32 + lane] = acc[i][c] * (1.f / wsc[c & 1]) * a.vunit;
    __syncthreads();
    for (int i = tid; i < NQ * DR; i += kThreads) {
        const int qq = i / DR, j = i - qq * DR;
        if (q0 + qq >= a.qpg) continue;
        // coordinate j is 2 i + (c >> 1) of row j / (DR / 8), query qq in register c & 1 of lane qq / 2 (lo columns: two lanes further)
        const int jr = j / (DR / 8), jc = j % (DR / 8);
        const float* src = wacc + ((jc >> 1) * 4 + (jc & 1) * 2 + (qq & 1)) * 32 + jr * 4 + (qq >> 1);
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
            const float f = wf[w * NQ + qq];
            const float x = NQ == 4 ? src[w * kAcc] + src[w * kAcc + 2] : src[w * kAcc];
            v = fmaf(f, f == 0.f ? 0.f : x, v);
        }
        a.part[(((size_t)g * a.qpg + q0 + qq) * a.splits + split) * (DR + 2) + j] = v;
    }
}

// One block per (group, query): merge the splits (weights 2^(m_s - M)), divide by the sum, and apply the value
// quantizer's rotation: out[j] = sum_k a[k] R[k][j] (the `@ self.rotation` of _quant.py:241).  Latency is all there is to
// it (it took 7.6 us with one thread per coordinate walking the splits): the matrix is fetched before the wait for the splits,
// the splits and the sum over k are shared out among the threads.
constexpr int kCombineThreads = 256;

template <int DR>
__global__ void __launch_bounds__(kCombineThreads)
decode_combine_kernel(const float* __restrict__ part, int splits, const float* __restrict__ Rv, float* __restrict__ out) {
    constexpr int kParts = kCombineThreads / DR, kSlices = kCombineThreads / (DR / 4), kLen = DR / kSlices;
    __shared__ float weight[kMaxSplits], vec[kParts][DR], total[kSlices][DR];
    __shared__ float inverse;
    const int t = threadIdx.x, lane = t & 31;
    const int j4 = t % (DR / 4) * 4, k0 = t / (DR / 4) * kLen;
    float4 m[kLen];
#pragma unroll
    for (int u = 0; u < kLen; ++u) m[u] = __ldg(reinterpret_cast<const float4*>(Rv + (size_t)(k0 + u) * DR + j4));
    tq_grid_wait();
    const float* pr = part + (size_t)blockIdx.x * splits * (DR + 2);
    const int c = t % DR, slice = t / DR;
    constexpr int kAhead = 8;       // accumulators in flight, fetched before the weights are known
    float x[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) x[u] = slice + u * kParts < splits ? pr[(size_t)(slice + u * kParts) * (DR + 2) + c] : 0.f;
    if (t < 32) {
        float ms[kMaxSplits / 32], ls[kMaxSplits / 32], top = -CUDART_INF_F, sum = 0.f;
#pragma unroll
        for (int u = 0; u < kMaxSplits / 32; ++u) {
            const int s = lane + 32 * u;
            ms[u] = s < splits ? pr[(size_t)s * (DR + 2) + DR] : -CUDART_INF_F;
            ls[u] = s < splits ? pr[(size_t)s * (DR + 2) + DR + 1] : 0.f;
            top = fmaxf(top, ms[u]);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
#pragma unroll
        for (int u = 0; u < kMaxSplits / 32; ++u) {
            const float w = ms[u] == -CUDART_INF_F ? 0.f : exp2f(ms[u] - top);
            weight[lane + 32 * u] = w;
            sum = fmaf(w, ls[u], sum);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) inverse = sum > 0.f ? 1.f / sum : 0.f;     // no keys at all: zeros
    }
    __syncthreads();
    float v = 0.f;
    for (int s0 = slice; s0 < splits; s0 += kAhead * kParts) {
        float next[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int s = s0 + (u + kAhead) * kParts;
            next[u] = s < splits ? pr[(size_t)s * (DR + 2) + c] : 0.f;
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int s = s0 + u * kParts;
            if (s < splits && weight[s] != 0.f) v = fmaf(weight[s], x[u], v);
            x[u] = next[u];
        }
    }
    vec[slice][c] = v;
    __syncthreads();
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < kLen; ++u) {
        float a = vec[0][k0 + u];
#pragma unroll
        for (int i = 1; i < kParts; ++i) a += vec[i][k0 + u];
        a *= inverse;
        o.x = fmaf(a, m[u].x, o.x); o.y = fmaf(a, m[u].y, o.y); o.z = fmaf(a, m[u].z, o.z); o.w = fmaf(a, m[u].w, o.w);
    }
    *reinterpret_cast<float4*>(&total[t / (DR / 4)][j4]) = o;
    __syncthreads();
    if (t < DR) {
        float r = 0.f;
#pragma unroll
        for (int i = 0; i < kSlices; ++i) r += total[i][t];
        out[(size_t)blockIdx.x * DR + t] = r;
    }
}

// Up to four queries share a pass with their hi and lo parts as the eight columns of the operand; more take eight per pass.
int queries_per_pass(int qpg) { return qpg <= 4 ? 4 : 8; }

// One block is resident per SM (its registers), so blocks run in waves of `sms`.  Among the split counts that fill 1..4 waves,
// take the one with the fewest rounds of its warps per SM (a block's set-up counted as four rounds).
int splits_for(int sms, int groups, int passes, int64_t keys_per_group) {
    const int64_t tiles = (keys_per_group + kTile - 1) / kTile;
    const int64_t gq = (int64_t)groups * passes;
    if (tiles <= kWarps || gq <= 0) return 1;
    int64_t best = 1, best_cost = -1;
    for (int w = 1; w <= 4; ++w) {
        int64_t s = (int64_t)sms * w / gq;
        if (s < 1) s = 1;
        if (s > (tiles + kWarps - 1) / kWarps) s = (tiles + kWarps - 1) / kWarps;
        if (s > kMaxSplits) s = kMaxSplits;
        const int64_t waves = (gq * s + sms - 1) / sms;
        const int64_t cost = waves * (((tiles + s - 1) / s + kWarps - 1) / kWarps + 4);
        if (best_cost < 0 || cost < best_cost) { best_cost = cost; best = s; }
    }
    return (int)best;
}

template <int KB, int VB, int DR, int NQ>
int launch_partial(const tq_plan* kp, const DecodeArgs& a, int groups, int passes, cudaStream_t st) {
    using P = Plan<KB, VB, DR, NQ>;
    TQ_GRANT_SMEM((decode_partial_kernel<KB, VB, DR, NQ>), P::total, kp->device);
    decode_partial_kernel<KB, VB, DR, NQ><<<dim3((unsigned)a.splits, (unsigned)passes, (unsigned)groups), kThreads, P::total, st>>>(kp->dev, a);
    tq_count_launch();
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}

template <int KB, int VB>
int launch_partial_dq(const tq_plan* kp, const DecodeArgs& a, int groups, int passes, int qp, cudaStream_t st) {
    if (kp->dev.d == 64) return qp == 4 ? launch_partial<KB, VB, 64, 4>(kp, a, groups, passes, st) : launch_partial<KB, VB, 64, 8>(kp, a, groups, passes, st);
    return qp == 4 ? launch_partial<KB, VB, 128, 4>(kp, a, groups, passes, st) : launch_partial<KB, VB, 128, 8>(kp, a, groups, passes, st);
}

template <int KB>
int launch_partial_v(const tq_plan* kp, int vbits, const DecodeArgs& a, int groups, int passes, int qp, cudaStream_t st) {
    switch (vbits) {
        case 1: return launch_partial_dq<KB, 1>(kp, a, groups, passes, qp, st);
        case 2: return launch_partial_dq<KB, 2>(kp, a, groups, passes, qp, st);
        case 3: return launch_partial_dq<KB, 3>(kp, a, groups, passes, qp, st);
        default: return launch_partial_dq<KB, 4>(kp, a, groups, passes, qp, st);
    }
}

}  // namespace

bool tq_decode_attention_supported(const tq_plan* kp, const tq_plan* vp) {
    const int d = kp->dev.d;
    return kp->has_projection && vp->dev.d == d && (d == 128 || d == 64) && kp->dev.bits >= 1 && kp->dev.bits <= 4 &&
           vp->dev.bits >= 1 && vp->dev.bits <= 4;
}

int64_t tq_decode_attention_scratch(const tq_plan* kp, int groups, int qpg, int64_t keys_per_group) {
    const int qp = queries_per_pass(qpg);
    const int passes = (qpg + qp - 1) / qp;
    const int splits = splits_for(tq_sm_count(kp->device), groups, passes, keys_per_group);
    return (int64_t)groups * qpg * splits * (kp->dev.d + 2) * (int64_t)sizeof(float);
}

int tq_launch_decode_attention(const tq_plan* kp, const tq_plan* vp, const float* q, int groups, int qpg,
                               const uint32_t* kcodes, const uint32_t* ksigns, const float* krnorms, const float* knorms,
                               const uint32_t* vcodes, const float* vnorms, int64_t keys_per_group, int64_t group_rows,
                               const int64_t* length, float scale, float* out, void* scratch, size_t scratch_bytes,
                               cudaStream_t st) {
    TqRange range("tq.decode_attention");
    const int d = kp->dev.d, kb = kp->dev.bits;
    const int qp = queries_per_pass(qpg);
    const int passes = (qpg + qp - 1) / qp;
    DecodeArgs a{};
    a.q = q; a.kcodes = kcodes; a.ksigns = ksigns; a.krnorms = krnorms; a.knorms = knorms;
    a.vcodes = vcodes; a.vnorms = vnorms; a.vparts = vp->dev.cent_parts; a.vunit = vp->dev.cent_unit;
    a.qpg = qpg; a.keys_per_group = keys_per_group; a.group_rows = group_rows; a.length = length;
    a.scale_log2e = scale * 1.4426950408889634f;
    a.splits = splits_for(tq_sm_count(kp->device), groups, passes, keys_per_group);
    a.part = static_cast<float*>(scratch);
    const size_t need = (size_t)groups * qpg * a.splits * (d + 2) * sizeof(float);
    if (!scratch || scratch_bytes < need)
        return tq_fail(TQ_ERR_SCRATCH_TOO_SMALL, "decode attention scratch: need %zu bytes, got %zu", need, scratch_bytes);
    int r = TQ_ERR_UNSUPPORTED;
    switch (kb) {
        case 1: r = launch_partial_v<1>(kp, vp->dev.bits, a, groups, passes, qp, st); break;
        case 2: r = launch_partial_v<2>(kp, vp->dev.bits, a, groups, passes, qp, st); break;
        case 3: r = launch_partial_v<3>(kp, vp->dev.bits, a, groups, passes, qp, st); break;
        case 4: r = launch_partial_v<4>(kp, vp->dev.bits, a, groups, passes, qp, st); break;
    }
    if (r != TQ_OK) return r;
    if (d == 64)
        TQ_CUDA_TRY(tq_launch_dependent(decode_combine_kernel<64>, dim3((unsigned)(groups * qpg)), dim3(kCombineThreads), 0, st,
                                        (const float*)a.part, a.splits, vp->dev.R, out));
    else
        TQ_CUDA_TRY(tq_launch_dependent(decode_combine_kernel<128>, dim3((unsigned)(groups * qpg)), dim3(kCombineThreads), 0, st,
                                        (const float*)a.part, a.splits, vp->dev.R, out));
    return TQ_OK;
}
