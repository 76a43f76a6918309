// attention_score for one query (_quant.py:334-358) against very many keys, or in very many groups of few keys.
//
//   score(q, key) = norm * ( (R q) . codebook[codes]  +  alpha * rnorm * ((S q) . signs) )
//
// Per (group, query) the rotated and projected query are turned into two lookup tables in shared memory,
//
//   pair table   [d/2 positions][4^bits entries]   c[code0] * (R q)[2p] + c[code1] * (R q)[2p+1]
//   byte table   [d/8 positions][256 entries]      sum over the 8 sign bits of the byte of +-(S q)[coordinate]
//
// and every thread walks the packed codes and sign words of one key: d/2 + d/8 lookups and additions, no unpacking.
// score_few_kernel expands the keys for up to four queries at once; for one it pays that expansion alone (half a million to four million
// keys), and it keeps an SM to itself for a prologue of 2 / 2 / 6 us at d = 64 / 128 / 256, where a block here takes 5 / 9 / 15 us but four to
// eight run beside each other (a thousand groups with a few keys each).  Anything between is its own.
#include "tq_common.cuh"

#include <stdint.h>

namespace {

constexpr int kTableThreads = 256;

// grid (blocks over keys, queries per group, groups)
template <int BITS, int DR>
__global__ void __launch_bounds__(kTableThreads)
score_table_kernel(TqDev p, const float* __restrict__ q, const uint32_t* __restrict__ codes,
                 const uint32_t* __restrict__ signs, const float* __restrict__ rnorms, const float* __restrict__ norms,
                 int64_t keys_per_group, int64_t group_rows, int qpg, float* __restrict__ scores) {
    constexpr int kPairs = DR / 2, kEntries = 1 << (2 * BITS), kBytes = DR / 8;
    constexpr int kCodeWords = DR * BITS / 32, kSignWords = DR / 32;
    constexpr uint32_t kMask = kEntries - 1;
    extern __shared__ float tables[];
    float* pair_t = tables;                       // [kPairs][kEntries]
    float* byte_t = tables + kPairs * kEntries;   // [kBytes][256]
    const int g = blockIdx.z, qi = blockIdx.y;
    // Every block rotates and projects its query itself (2 d^2 FMAs, the matrices come from L2): rotated[j] =
    // sum_k q[k] R[j][k], projected[j] = sum_k q[k] S[j][k], one FMA per k, k ascending as in the reference's
    // matrix products.  That costs a few microseconds per block and saves a launch and a scratch buffer.
    __shared__ float qs[DR], qr[DR], ps[DR];
    if (threadIdx.x < DR) qs[threadIdx.x] = __ldg(q + ((size_t)g * qpg + qi) * DR + threadIdx.x);
    __syncthreads();
    if (threadIdx.x < DR) {
        const int j = threadIdx.x;
        float r = 0.f, sacc = 0.f;
        for (int k0 = 0; k0 < DR; k0 += 16) {
            float mr[16], ms[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                mr[u] = __ldg(p.Rt + (size_t)(k0 + u) * DR + j);
                ms[u] = __ldg(p.St + (size_t)(k0 + u) * DR + j);
            }
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                r = fmaf(qs[k0 + u], mr[u], r);
                sacc = fmaf(qs[k0 + u], ms[u], sacc);
            }
        }
        qr[j] = r;
        ps[j] = sacc;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kPairs * kEntries; i += kTableThreads) {
        const int pp = i / kEntries, e = i - pp * kEntries;
        const float c0 = __ldg(p.codebook + (e & ((1 << BITS) - 1))), c1 = __ldg(p.codebook + (e >> BITS));
        pair_t[i] = fmaf(c1, qr[2 * pp + 1], c0 * qr[2 * pp]);
    }
    for (int i = threadIdx.x; i < kBytes * 256; i += kTableThreads) {
        const int pos = i >> 8, v = i & 255, w = pos >> 2, b = pos & 3;
        float acc = 0.f;
#pragma unroll
        for (int bit = 0; bit < 8; ++bit) {
            // stored order of the sign words: even coordinates in bits 0..15, odd ones in bits 16..31
            const int bp = 8 * b + bit;
            const int coord = 32 * w + (bp < 16 ? 2 * bp : 2 * (bp - 16) + 1);
            const float x = ps[coord];
            acc += (v >> bit) & 1 ? x : -x;
        }
        byte_t[i] = acc;
    }
    __syncthreads();

    const float alpha = p.alpha;
    float* out = scores + ((size_t)g * qpg + qi) * keys_per_group;
    for (int64_t key = (int64_t)blockIdx.x * kTableThreads + threadIdx.x; key < keys_per_group;
         key += (int64_t)gridDim.x * kTableThreads) {
        const int64_t row = (int64_t)g * group_rows + key;
        uint32_t cw[kCodeWords + 1], sw[kSignWords];
        const uint32_t* crow = codes + row * kCodeWords;
        const uint32_t* srow = signs + row * kSignWords;
        if (kCodeWords % 4 == 0) {
#pragma unroll
            for (int k = 0; k < kCodeWords; k += 4) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(crow + k));
                cw[k] = v.x; cw[k + 1] = v.y; cw[k + 2] = v.z; cw[k + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < kCodeWords; k += 2) {
                const uint2 v = __ldg(reinterpret_cast<const uint2*>(crow + k));
                cw[k] = v.x; cw[k + 1] = v.y;
            }
        }
        cw[kCodeWords] = 0u;
#pragma unroll
        for (int k = 0; k < kSignWords; k += 2) {
            const uint2 v = __ldg(reinterpret_cast<const uint2*>(srow + k));
            sw[k] = v.x; sw[k + 1] = v.y;
        }
        const float nrm = __ldg(norms + row), rn = __ldg(rnorms + row);
        float s1[4] = {0.f, 0.f, 0.f, 0.f}, s2[2] = {0.f, 0.f};
#pragma unroll
        for (int pp = 0; pp < kPairs; ++pp) {
            const int bit = pp * 2 * BITS, wi = bit >> 5, sh = bit & 31;
            uint32_t e;
            if (sh + 2 * BITS <= 32) e = (cw[wi] >> sh) & kMask;
            else e = __funnelshift_r(cw[wi], cw[wi + 1], sh) & kMask;
            s1[pp & 3] += pair_t[pp * kEntries + e];
        }
#pragma unroll
        for (int pos = 0; pos < kBytes; ++pos) s2[pos & 1] += byte_t[pos * 256 + ((sw[pos >> 2] >> (8 * (pos & 3))) & 255u)];
        const float a1 = (s1[0] + s1[1]) + (s1[2] + s1[3]);
        out[key] = nrm * fmaf(alpha * rn, s2[0] + s2[1], a1);
    }
}

template <int BITS, int DR>
int launch_table(const tq_plan* p, const float* q, const uint32_t* codes, const uint32_t* signs, const float* rnorms,
               const float* norms, int64_t keys_per_group, int64_t group_rows, int groups, int qpg, float* scores,
               cudaStream_t st) {
    const int sm = ((DR / 2) * (1 << (2 * BITS)) + (DR / 8) * 256) * 4;
    TQ_GRANT_SMEM((score_table_kernel<BITS, DR>), sm, p->device);
    const int sms = tq_sm_count(p->device);
    int64_t blocks = (keys_per_group + kTableThreads - 1) / kTableThreads;
    const int64_t cap = (int64_t)sms * 4;   // the tables cost a few microseconds per block: a few blocks per SM, grid-stride
    if (blocks > cap) blocks = cap;
    score_table_kernel<BITS, DR><<<dim3((unsigned)blocks, (unsigned)qpg, (unsigned)groups), kTableThreads, sm, st>>>(
        p->dev, q, codes, signs, rnorms, norms, keys_per_group, group_rows, qpg, scores); tq_count_launch();
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}

}  // namespace

// The lines lie where the two kernels meet (us, warp-level kernel / this one; 1, 2, 3 code bits):
//   one group   d = 64     524,288 keys  14.6:13.0 / 14.3:14.7 / 14.9:14.9      1,048,576 keys  23:18 / 23:19 / 25:21      (4 bits 23:27)
//               d = 128    524,288 keys  21:23 / 21:23 / 21:27                  800,000 keys  29:27 / 27:27 / 29:33
//                          4,000,000 keys  119:90 / 111:95 / 122:117  (2,097,152 keys, 3 bits 68:74; 4 bits 118:189)
//               d = 256    800,000 keys  51:50 / 54:62 / 69:82                  2,097,152 keys  117:107 / 124:120 / 157:171
//   groups      d = 64     512 x 512  14.2:14.8 / 13.4:14.7 / 14.7:14.8         2,048 x 32  25:20 / 25:21 / 25:21     4,096 x 512  78:76 / 78:78 / 91:85
//               d = 128    512 x 512  21:25 / 21:25 / 23:29                     2,048 x 32  39:39 / 35:40 / 35:46     2,048 x 256  50:45 / 52:45 / 55:50
//                          4,096 x 512  136:157 / 142:164 / 150:170
//               d = 256    512 x 512  44:50 / 45:52 / 51:68                     2,048 x 32  103:76 / 88:79 / 93:105   2,048 x 256  122:89 / 124:95 / 141:123
//               4 bits, any d: 2,048 x 256  d = 64 33:31, d = 128 54:86
bool tq_score_table_better(const tq_plan* p, int groups, int qpg, int64_t keys_per_group) {
    const int d = p->dev.d, bits = p->dev.bits;
    if (!p->has_projection || bits < 1 || bits > 3) return false;
    // many more groups than the other kernel runs at once, and a block for each (d = 64: or two)
    const int64_t blocks = qpg * ((keys_per_group + kTableThreads - 1) / kTableThreads);
    if (groups > 6 * tq_sm_count(p->device)) {
        if (d == 64 ? blocks <= 2 : blocks == 1 && ((d == 256 && bits <= 2) || keys_per_group > kTableThreads / 2)) return true;
    }
    if (qpg != 1) return false;
    if (d == 64) return keys_per_group >= 1 << 19;
    if (bits == 1 || (bits == 2 && d == 128)) return keys_per_group >= 3 << 18;
    return keys_per_group >= (bits == 2 ? 1 << 21 : d == 128 ? 7 << 19 : 1 << 22);
}

// scores: [groups][qpg][keys_per_group]
int tq_launch_score_table(const tq_plan* p, const float* q, int groups, int qpg, const uint32_t* codes, const uint32_t* signs, const float* rnorms,
                          const float* norms, int64_t keys_per_group, float* scores, cudaStream_t st, int64_t group_rows) {
    TqRange range("tq.score.one_query");
    if (group_rows <= 0) group_rows = keys_per_group;
    const int d = p->dev.d;
    switch (p->dev.bits) {
#define TQ_TABLE(B, D) launch_table<B, D>(p, q, codes, signs, rnorms, norms, keys_per_group, group_rows, groups, qpg, scores, st)
        case 1: return d == 256 ? TQ_TABLE(1, 256) : d == 128 ? TQ_TABLE(1, 128) : TQ_TABLE(1, 64);
        case 2: return d == 256 ? TQ_TABLE(2, 256) : d == 128 ? TQ_TABLE(2, 128) : TQ_TABLE(2, 64);
        case 3: return d == 256 ? TQ_TABLE(3, 256) : d == 128 ? TQ_TABLE(3, 128) : TQ_TABLE(3, 64);
#undef TQ_TABLE
    }
    return tq_fail(TQ_ERR_UNSUPPORTED, "no table kernel for d=%d bits=%d", d, p->dev.bits);
}
