// Scores of at most four queries per group of keys (one query against every key is the reference's own call pattern,
// _quant.py:334-358; four are a grouped-query decode step), d = 128, 64 or 256, 1..4 code bits.
//
//   score(q, key) = norm * ( (R q) . codebook[codes]  +  alpha * rnorm * ((S q) . signs) )
//
// The tcgen05 kernel costs the same below 16 queries; here the expansion of the packed keys in the registers of the lane that
// feeds them to a warp-level matrix instruction is all there is to pay, once for up to four queries (their hi and lo parts side
// by side are the eight columns).  A warp takes 16 keys at a time, the words of the next tile in
// flight, no barriers; the tables (tq_mma.cuh) do not depend on the queries, so they are built while the matrices are on
// their way, and the matrices while the queries are (page-locked host memory in a NumPy call).
//
// 1-bit codes need no table: a centroid is (c0 + c1) / 2 +- (c1 - c0) / 2, so their bits become +-1 as the signs do.  (c0 + bit (c1 - c0),
// the bits used where they stand, saved an instruction a register and gave ten times the error: the two terms cancel.)
//
// The tensor pipe truncates a sum at every instruction, so a score is added up from two chains of half the coordinates each (one
// chain: 3 to 12 % more error than the multiply-adds of the table kernel, two: 10 to 40 % less).
//
// Bound: shared-memory lookups, 64 8-byte loads a key at d = 128 and 3-bit codes (2 cycles a warp and load, four lanes a key), and for
// few keys the prologue.  Kernel alone, 3-bit codes, one query, 256 / 262,147 keys: d = 64 2.7 / 8.1 us, d = 128 3.5 / 12.4,
// d = 256 8.1 / 26.1 (4.1 / 9.5, 8.1 / 16.7, 16.5 / 35.2 with every lane splitting the queries for itself).
// Where tables are the faster way (very many keys, very many groups): tq_score_table.cu.
#include "tq_common.cuh"
#include "tq_mma.cuh"

#include <stdint.h>

namespace {

using namespace tqmma;

constexpr int kFewThreads = 512;
constexpr int kFewWarps = kFewThreads / 32;
constexpr int kTile = 16;           // keys a warp takes at a time
constexpr int kMaxQ = 4;            // queries of a pass

struct FewArgs {
    const float* q;              // [groups][qpg][d]
    const uint32_t* codes;
    const uint32_t* signs;
    const float* rnorms;
    const float* norms;
    int qpg;
    int64_t keys_per_group, group_rows;
    float* scores;               // [groups][qpg][keys_per_group]
};

// NQ: queries whose vectors the prologue computes, one or four.
template <int KB, int DR, int NQ>
struct FewPlan {
    static constexpr int kSteps = DR / 16;
    static constexpr int kSlices = kFewThreads / (DR / 2), kSliceLen = DR / kSlices;   // four outputs of one matrix and a slice of the sum per thread
    static constexpr int off_slice = table_rows(KB) * kRowBytes;                     // [kSlices][2][NQ][DR] partial sums
    static constexpr int off_ops = off_slice + kSlices * 2 * NQ * DR * 4;            // [2][NQ][hi, lo][operand_row(DR)] fp16: rotated, projected queries
    static constexpr int off_qin = off_ops + (2 * NQ * 2 * operand_row(DR) * 2 + 15) / 16 * 16;     // [DR][NQ]
    static constexpr int off_small = off_qin + NQ * DR * 4;                          // [2][NQ] scales, [2][NQ] sums of the vectors
    static constexpr int total = off_small + 4 * NQ * 4;
    static_assert(total <= 227 * 1024, "shared memory plan");
};

// Where coordinate k of a query lies among the operands: lane t of a quad takes the coordinates [t DR / 4, + DR / 4), four a step; 1-bit
// codes: coordinates that lie half a word apart make a pair.
template <int DR, bool HALF_APART>
__device__ __forceinline__ int operand_place(int k) {
    if (!HALF_APART) return k;
    constexpr int kHalf = DR == 64 ? 8 : 16;
    const int lane_first = k / (DR / 4) * (DR / 4), rel = k % (DR / 4), i = rel % kHalf;
    return lane_first + 4 * (rel / (2 * kHalf) * (kHalf / 2) + i / 2) + (i & 1) * 2 + (rel % (2 * kHalf) >= kHalf ? 1 : 0);
}

// grid (blocks over the keys, passes over the queries of a group, groups)
template <int KB, int DR, int NQ>
__global__ void __launch_bounds__(kFewThreads, 1)
score_few_kernel(const TqDev p, const FewArgs a) {
    using P = FewPlan<KB, DR, NQ>;
    using W = KeyWords<KB, DR>;
    extern __shared__ __align__(128) unsigned char smem[];
    __half* ops = reinterpret_cast<__half*>(smem + P::off_ops);
    float* qin = reinterpret_cast<float*>(smem + P::off_qin);
    float* slice = reinterpret_cast<float*>(smem + P::off_slice);
    int* scl = reinterpret_cast<int*>(smem + P::off_small);                   // exponents of the queries' scales
    float* psum = reinterpret_cast<float*>(smem + P::off_small) + 2 * NQ;

    const int g = blockIdx.z, q0 = blockIdx.y * kMaxQ;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = lane & 3, r = lane >> 2;      // position in the quad, row of the fragments
    const uint32_t keys = (uint32_t)a.keys_per_group;            // rows of all groups together stay below 2^32
    const uint32_t tiles = (uint32_t)((a.keys_per_group + kTile - 1) / kTile), stride = gridDim.x * kFewWarps;
    // neighbouring tiles go to different blocks: with fewer tiles than warps every SM has some
    uint32_t tile = (uint32_t)warp * gridDim.x + blockIdx.x;

    // the matrices: in flight before anything else is waited for
    const int xm = tid / (DR / 4) & 1, xj = tid % (DR / 4) * 4, xk = tid / (DR / 2) * P::kSliceLen;    // matrix, first output, slice
    constexpr int kBatch = P::kSliceLen < 16 ? P::kSliceLen : 16;
    static_assert(P::kSliceLen % kBatch == 0, "slices");
    const float* msrc = (xm ? p.St : p.Rt) + (size_t)xk * DR + xj;
    float4 mat[kBatch];
#pragma unroll
    for (int u = 0; u < kBatch; ++u) mat[u] = __ldg(reinterpret_cast<const float4*>(msrc + (size_t)u * DR));

    const int64_t row_base = (int64_t)g * a.group_rows;
    const int kbit = W::kBits * t, kshift = kbit & 31;
    const uint32_t* kc_base = a.codes + row_base * (DR * KB / 32) + (kbit >> 5);
    const uint32_t* sg_base = a.signs + row_base * (DR / 32) + (DR == 256 ? 2 * t : DR == 128 ? t : t >> 1);
    const float* kn_base = a.norms + row_base;
    const float* rn_base = a.rnorms + row_base;
    struct Words { uint32_t kc[2][W::kWords], sg[2][W::kSigns]; float kn[2], rn[2]; };
    auto fetch = [&](uint32_t tl, Words& w) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t key = min(tl * kTile + r + 8 * h, keys - 1);       // rows behind the last one: read that one
            const uint32_t* src = kc_base + (size_t)key * (DR * KB / 32);
            if constexpr (W::kBits % 128 == 0) {
#pragma unroll
                for (int i = 0; i < W::kWords; i += 4) {
                    const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + i));
                    w.kc[h][i] = v.x; w.kc[h][i + 1] = v.y; w.kc[h][i + 2] = v.z; w.kc[h][i + 3] = v.w;
                }
            } else if constexpr (W::kBits % 64 == 0) {
#pragma unroll
                for (int i = 0; i < W::kWords; i += 2) {
                    const uint2 v = __ldg(reinterpret_cast<const uint2*>(src + i));
                    w.kc[h][i] = v.x; w.kc[h][i + 1] = v.y;
                }
            } else {
#pragma unroll
                for (int i = 0; i < W::kWords; ++i) w.kc[h][i] = __ldg(src + i);
            }
#pragma unroll
            for (int i = 0; i < W::kSigns; ++i) w.sg[h][i] = __ldg(sg_base + (size_t)key * (DR / 32) + i);
            w.kn[h] = __ldg(kn_base + key);
            w.rn[h] = __ldg(rn_base + key);
        }
    };
    if (KB > 1) build_key_table<KB>(smem, p.cent_parts, tid, kFewThreads);
    tq_grid_release();
    tq_grid_wait();         // (only constants of the plan have been read so far)
    Words cur;
    if (tile < tiles) fetch(tile, cur);
    for (int i = tid; i < NQ * DR; i += kFewThreads) {
        const int qq = i / DR, k = i - qq * DR;
        qin[k * NQ + qq] = q0 + qq < a.qpg ? __ldg(a.q + ((size_t)g * a.qpg + q0 + qq) * DR + k) : 0.f;
    }
    __syncthreads();
    {   // rotated[j] = sum_k q[k] R[j][k], projected[j] = sum_k q[k] S[j][k] in 32-bit arithmetic
        float4 sum[NQ];
#pragma unroll
        for (int qq = 0; qq < NQ; ++qq) sum[qq] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int b = 0; b < P::kSliceLen; b += kBatch) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const float* qk = qin + (xk + b + u) * NQ;
#pragma unroll
                for (int qq = 0; qq < NQ; ++qq) {
                    const float v = qk[qq];
                    sum[qq].x = fmaf(v, mat[u].x, sum[qq].x);
                    sum[qq].y = fmaf(v, mat[u].y, sum[qq].y);
                    sum[qq].z = fmaf(v, mat[u].z, sum[qq].z);
                    sum[qq].w = fmaf(v, mat[u].w, sum[qq].w);
                }
            }
            if (b + kBatch < P::kSliceLen) {
#pragma unroll
                for (int u = 0; u < kBatch; ++u) mat[u] = __ldg(reinterpret_cast<const float4*>(msrc + (size_t)(b + kBatch + u) * DR));
            }
        }
#pragma unroll
        for (int qq = 0; qq < NQ; ++qq) *reinterpret_cast<float4*>(slice + ((tid / (DR / 2) * 2 + xm) * NQ + qq) * DR + xj) = sum[qq];
    }
    __syncthreads();
    for (int v = warp; v < 2 * NQ; v += kFewWarps) {      // a warp per vector: slices added up, largest value, sum, fp16 parts
        float m = 0.f, sum = 0.f, x[DR / 32];
#pragma unroll
        for (int i = 0; i < DR / 32; ++i) {
            const int k = lane + 32 * i;
            x[i] = slice[v * DR + k];
#pragma unroll
            for (int u = 1; u < P::kSlices; ++u) x[i] += slice[(u * 2 * NQ + v) * DR + k];
            m = fmaxf(m, fabsf(x[i]));
            sum += x[i];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            sum += __shfl_xor_sync(0xffffffffu, sum, o);
        }
        const int e = scale_exp(m);
        const float sc = pow2i(e);
#pragma unroll
        for (int i = 0; i < DR / 32; ++i) {
            const int k = lane + 32 * i, at = KB == 1 && v < NQ ? operand_place<DR, true>(k) : operand_place<DR, false>(k);
            const float y = x[i] * sc;
            const __half h = __float2half_rn(y);
            ops[(v * 2) * operand_row(DR) + at] = h;
            ops[(v * 2 + 1) * operand_row(DR) + at] = __float2half_rn(y - __half2float(h));
        }
        if (lane == 0) {
            scl[v] = e;
            psum[v] = sum;
        }
    }
    __syncthreads();
    // Query operands: column r is hi (r < 4) or lo (r >= 4) of query r & 3.  (Split once, by the warp that has the vector: every lane
    // splitting what it needs, from rows whose words all lay in the same banks, took more than half of the prologue.)
    uint32_t qf[2][P::kSteps][2];
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const uint2* x = reinterpret_cast<const uint2*>(ops + ((m * NQ + (r & (NQ - 1))) * 2 + (r >> 2)) * operand_row(DR) + t * (DR / 4));
#pragma unroll
        for (int s = 0; s < P::kSteps; ++s) {
            const uint2 w = (r & 3) < NQ ? x[s] : make_uint2(0u, 0u);
            qf[m][s][0] = w.x;
            qf[m][s][1] = w.y;
        }
    }
    // the two queries of this lane's score columns
    float ds1[2], ds2[2], dbase[2] = {0.f, 0.f};
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const int qq = (2 * t + c) & (NQ - 1);         // (columns without a query: any)
        ds1[c] = pow2i(-scl[qq]) * p.cent_unit;
        if constexpr (KB == 1) {
            const float c0 = __ldg(p.codebook), c1 = __ldg(p.codebook + 1);
            ds1[c] = pow2i(-scl[qq]) * (0.5f * (c1 - c0));
            dbase[c] = 2 * t < kMaxQ ? 0.5f * (c0 + c1) * psum[qq] : 0.f;
        }
        ds2[c] = pow2i(-scl[NQ + qq]) * p.alpha;
    }
    const uint32_t lane8 = (uint32_t)(lane & 15) * 8u, lane16 = (uint32_t)(lane & 7) * 16u;
    // The lane's scores: queries 2 (t & 1) + c of key r + 8 (t >> 1) -- adding hi and lo columns leaves both lanes with the sum.
    const int qs0 = q0 + 2 * (t & 1);
    float* out = a.scores + ((int64_t)g * a.qpg + qs0) * a.keys_per_group;

    for (; tile < tiles; tile += stride) {
        Words nxt;
        if (tile + stride < tiles) fetch(tile + stride, nxt);
        W key;
        key.unpack(cur.kc, cur.sg, kshift, t);
        uint32_t cbits[2][W::kWords];
        if constexpr (KB == 1) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int i = 0; i < W::kWords; ++i) {
                    uint32_t w = cur.kc[h][i];
                    if (DR == 64) { w >>= kshift; w = (w & 0xffu) | ((w & 0xff00u) << 8); }
                    cbits[h][i] = w;
                }
        }
        float v[2][2];                 // [key r + 8 h][query column c]
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < 2; ++c) v[h][c] = dbase[c];
        auto half = [&](auto first) {
            float c1[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, c2[4] = {0.f, 0.f, 0.f, 0.f};
            for_steps<P::kSteps / 2>([&](auto sc) {
                constexpr int s = decltype(first)::value + decltype(sc)::value;
                uint32_t ak[2][4], as[4];
                if constexpr (KB == 1) {
                    plus_minus<s>(cbits, ak[0]);
                    key.template signs<s>(as);
                    mma16816(c1[0], ak[0], qf[0][s][0], qf[0][s][1]);
                } else {
                    key.template operands<s>(smem, lane8, lane16, ak, as);
                    mma16816(c1[0], ak[0], qf[0][s][0], qf[0][s][1]);
                    mma16816(c1[1], ak[1], qf[0][s][0], qf[0][s][1]);
                }
                mma16816(c2, as, qf[1][s][0], qf[1][s][1]);
            });
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    v[h][c] += fmaf(c2[2 * h + c] * ds2[c], cur.rn[h], (KB == 1 ? c1[0][2 * h + c] : c1[h][c] + c1[h][2 + c]) * ds1[c]);
        };
        half(std::integral_constant<int, 0>{});
        half(std::integral_constant<int, P::kSteps / 2>{});
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                v[h][c] += __shfl_xor_sync(0xffffffffu, v[h][c], 2);     // hi and lo columns
                v[h][c] *= cur.kn[h];
            }
        const uint32_t k0 = tile * kTile + r + 8 * (t >> 1);
#pragma unroll
        for (int c = 0; c < 2; ++c)
            if (qs0 + c < a.qpg && k0 < keys) out[c * a.keys_per_group + k0] = t < 2 ? v[0][c] : v[1][c];
        cur = nxt;
    }
}

template <int KB, int DR, int NQ>
int launch_few_queries(const tq_plan* p, const FewArgs& a, int groups, cudaStream_t st) {
    using P = FewPlan<KB, DR, NQ>;
    TQ_GRANT_SMEM((score_few_kernel<KB, DR, NQ>), P::total, p->device);
    const int passes = (a.qpg + kMaxQ - 1) / kMaxQ;
    // at most a block per SM over all groups, as many as run at once (the prologue costs 3 to 14 us: 64 groups in three blocks each
    // took two rounds of it, 28 us for 64 x 4,096 keys of d = 128), and every block of a group gets at least a tile per warp
    const int64_t tiles = (a.keys_per_group + kTile - 1) / kTile, most = (tiles + 3) / 4;
    int64_t blocks = tq_sm_count(p->device) / ((int64_t)passes * groups);
    if (blocks > most) blocks = most;
    if (blocks < 1) blocks = 1;
    TQ_CUDA_TRY(tq_launch_dependent(score_few_kernel<KB, DR, NQ>, dim3((unsigned)blocks, (unsigned)passes, (unsigned)groups), dim3(kFewThreads),
                                    (size_t)P::total, st, p->dev, a));
    return TQ_OK;
}
// One query: a quarter of the prologue's products.
template <int KB, int DR>
int launch_few(const tq_plan* p, const FewArgs& a, int groups, cudaStream_t st) {
    return a.qpg == 1 ? launch_few_queries<KB, DR, 1>(p, a, groups, st) : launch_few_queries<KB, DR, 4>(p, a, groups, st);
}
}  // namespace

// Beyond these counts (d = 128 with up to 3 code bits: four queries; d = 64 and 4 bits: two; d = 256: one) a matrix has the very
// bits of the top-k search, whose kernel is the tcgen05 one, and keeps them.
bool tq_score_few_supported(const tq_plan* p, int qpg) {
    const int d = p->dev.d, bits = p->dev.bits;
    if (!p->has_projection || bits < 1 || bits > 4 || qpg < 1) return false;
    return d == 128 ? qpg <= (bits <= 3 ? 4 : 2) : d == 64 ? qpg <= 2 : d == 256 && qpg == 1;
}

// scores: [groups][qpg][keys_per_group]
int tq_launch_score_few(const tq_plan* p, const float* q, int groups, int qpg, const uint32_t* codes, const uint32_t* signs,
                        const float* rnorms, const float* norms, int64_t keys_per_group, float* scores, cudaStream_t st,
                        int64_t group_rows) {
    TqRange range("tq.score.few_queries");
    if (group_rows <= 0) group_rows = keys_per_group;
    if (tq_score_table_better(p, groups, qpg, keys_per_group))
        return tq_launch_score_table(p, q, groups, qpg, codes, signs, rnorms, norms, keys_per_group, scores, st, group_rows);
    const FewArgs a{q, codes, signs, rnorms, norms, qpg, keys_per_group, group_rows, scores};
    const int d = p->dev.d;
    switch (p->dev.bits) {
#define TQ_FEW(B)                                                                                                    \
    case B:                                                                                                         \
        return d == 64 ? launch_few<B, 64>(p, a, groups, st) : d == 256 ? launch_few<B, 256>(p, a, groups, st) \
                                                                                : launch_few<B, 128>(p, a, groups, st);
        TQ_FEW(1) TQ_FEW(2) TQ_FEW(3) TQ_FEW(4)
#undef TQ_FEW
    }
    return tq_fail(TQ_ERR_UNSUPPORTED, "no few-query scoring kernel for d=%d bits=%d", d, p->dev.bits);
}
