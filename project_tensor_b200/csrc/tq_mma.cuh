// Packed TurboQuantProd keys as operands of warp-level matrix instructions (m16n8k16, fp16 hi + lo parts, 32-bit sums): what the
// decode-attention kernel and the scoring kernel for few queries share.
#pragma once

#include "tq_common.cuh"

#include <type_traits>

namespace tqmma {

constexpr int kRowBytes = 256;         // a table row (keys use the first half)

__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t transpose8x8(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
__device__ __forceinline__ uint32_t half2_bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
// (a, b) -> fp16 pairs hi and lo with hi + lo = value to about 22 bits
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    hi = half2_bits(h);
    lo = half2_bits(__floats2half2_rn(a - f.x, b - f.y));
}
// Parts (hi, lo) of two centroids -> hi pair, lo pair.
__device__ __forceinline__ void pair_parts(uint32_t a, uint32_t b, uint32_t& hi, uint32_t& lo) {
    hi = __byte_perm(a, b, 0x5410);
    lo = __byte_perm(a, b, 0x7632);
}
// Shift left by s (negative: right) with s known at compile time.
template <int S> __device__ __forceinline__ uint32_t shl(uint32_t v) {
    if constexpr (S >= 0) return v << S;
    else return v >> -S;
}
// 2^e as a float, e clamped to the normal range
__device__ __forceinline__ float pow2i(int e) { return __int_as_float((min(max(e, -126), 127) + 127) << 23); }
// power of two that brings a magnitude into [2^13, 2^14)
__device__ __forceinline__ int scale_exp(float m) {
    if (!(m > 0.f) || !(m < 3.0e38f)) return 0;
    return min(max(13 - (int)((__float_as_uint(m) >> 23) - 127), -115), 100);      // (the largest float needs -114)
}

// Halves from one row of fp16 query operands to the next: eight rows (hi and lo of four queries) times four lanes of a quad, which
// start d / 4 halves apart, read 8 bytes each from different banks.
constexpr __host__ __device__ int operand_row(int d) { return d + 4; }

// f(0), f(1), ... f(N - 1) with compile-time arguments
template <int N, class F, int I = 0>
__device__ __forceinline__ void for_steps(F&& f) {
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        for_steps<N, F, I + 1>(static_cast<F&&>(f));
    }
}

// Rows of the key table: four codes at a time up to 2 bits, two at a time above (3 bits: whatever the upper two bits of the
// byte are that selects the row).
__host__ __device__ constexpr int codes_per_row(int bits) { return bits <= 2 ? 4 : 2; }
__host__ __device__ constexpr int table_rows(int bits) { return bits == 1 ? 16 : 256; }

// Key table, row e: 128 bytes of copies of (hi, lo) of a pair of codes, or (hi, lo, hi, lo) of four codes: the registers of an A
// operand.  A thread fills whole rows, starting at a copy of its own (stores to rows 256 bytes apart would all hit the same
// banks).
template <int KB>
__device__ __forceinline__ void build_key_table(unsigned char* table, const uint32_t* __restrict__ parts, int tid, int threads) {
    auto pair = [&](int c0, int c1, uint32_t& hi, uint32_t& lo) { pair_parts(__ldg(parts + c0), __ldg(parts + c1), hi, lo); };
    for (int e = tid; e < table_rows(KB); e += threads) {
        constexpr int m = (1 << KB) - 1;
        uint4 v;
        pair(e & m, (e >> KB) & m, v.x, v.y);
        if constexpr (codes_per_row(KB) == 4) pair((e >> 2 * KB) & m, e >> 3 * KB, v.z, v.w);
        else { v.z = v.x; v.w = v.y; }
#pragma unroll
        for (int i = 0; i < 8; ++i) *reinterpret_cast<uint4*>(table + e * kRowBytes + ((i + tid) & 7) * 16) = v;
    }
}

// A byte of a word selects a table row with one byte permutation: (lane's copy, byte, 0, 0) is its address.
__device__ __forceinline__ uint32_t pick(uint32_t word, int byte, uint32_t copy) {
    return __byte_perm(word, copy, 0x5504u | (uint32_t)byte << 4);
}

// Bits of two keys as +-1 (set: +1): step S takes bits 2S and 2S + 1 of the halves of the keys' words.  (Bits used where they stand, as
// subnormal numbers, save an instruction each, but their sums are several times the signed ones, and the rounding of the
// accumulators with them.)
template <int S, int WORDS>
__device__ __forceinline__ void plus_minus(const uint32_t (&w)[2][WORDS], uint32_t (&a)[4]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        a[h] = ((w[h][S >> 3] << (15 - (2 * S & 15))) & 0x80008000u) ^ 0xbc00bc00u;
        a[2 + h] = ((w[h][S >> 3] << (14 - (2 * S & 15))) & 0x80008000u) ^ 0xbc00bc00u;
    }
}

// The words of two keys that lane t of a quad turns into operands: DR / 4 consecutive coordinates of each.
template <int KB, int DR>
struct KeyWords {
    static constexpr int kBits = DR / 4 * KB;                                    // bits of a packed row that a lane uses
    static constexpr int kWords = kBits % 32 == 0 ? kBits / 32 : kBits / 32 + 1; // words it loads: they may start inside a word
    static constexpr int kSigns = DR == 256 ? 2 : 1;                             // sign words it loads
    uint32_t kw[2][kWords], kw1[2][kWords], sw[2][kSigns];
    __device__ __forceinline__ void unpack(const uint32_t (&kc)[2][kWords], const uint32_t (&sg)[2][kSigns], int shift, int t) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if constexpr (kBits % 32 == 0) {
#pragma unroll
                for (int i = 0; i < kWords; ++i) kw[h][i] = kc[h][i];
            } else {
                // half words (d = 64, odd bits): shift them to the front
                if constexpr (kWords == 2) {
                    kw[h][0] = __funnelshift_r(kc[h][0], kc[h][1], shift);
                    kw[h][1] = kc[h][1] >> shift;
                } else {
                    kw[h][0] = kc[h][0] >> shift;
                }
            }
#pragma unroll
            for (int i = 0; i < kSigns; ++i) {
                sw[h][i] = DR >= 128 ? sg[h][i] : sg[h][i] >> (8 * (t & 1));
            }
            if constexpr (KB == 1) {         // four codes: a nibble; even ones and odd ones in words of their own
#pragma unroll
                for (int i = 0; i < kWords; ++i) {
                    kw1[h][i] = (kw[h][i] >> 4) & 0x0f0f0f0fu;
                    kw[h][i] &= 0x0f0f0f0fu;
                }
            }
        }
    }
    // Coordinates 4s .. 4s + 3 of the lane: ak[h] the centroids of key h (rows: hi, then lo), as the signs of both keys.
    template <int S>
    __device__ __forceinline__ void operands(const unsigned char* table, uint32_t lane8, uint32_t lane16, uint32_t (&ak)[2][4], uint32_t (&as)[4]) const {
        auto row8 = [&](uint32_t at) { return *reinterpret_cast<const uint2*>(table + at); };
        auto row16 = [&](uint32_t at) { return *reinterpret_cast<const uint4*>(table + at); };
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if constexpr (KB >= 3) {
                uint2 v0, v1;
                if constexpr (KB == 4) {
                    v0 = row8(pick(kw[h][S >> 1], 2 * (S & 1), lane8));
                    v1 = row8(pick(kw[h][S >> 1], 2 * (S & 1) + 1, lane8));
                } else {
                    // 48 bits hold eight pairs; a word that starts at pair k has pair k in its first byte and pair k + 4 in its last,
                    // so four shifts serve eight pairs (a shift and a mask for each of them before)
                    auto pair = [&](auto pc) {
                        constexpr int p = decltype(pc)::value, bit = p / 8 * 48 + p % 4 * 6, w0 = bit >> 5, sh = bit & 31;
                        const uint32_t x = sh == 0 ? kw[h][w0] : __funnelshift_r(kw[h][w0], kw[h][w0 + 1 < kWords ? w0 + 1 : w0], sh);
                        return row8(pick(x, p % 8 < 4 ? 0 : 3, lane8));
                    };
                    v0 = pair(std::integral_constant<int, 2 * S>{});
                    v1 = pair(std::integral_constant<int, 2 * S + 1>{});
                }
                ak[h][0] = v0.x; ak[h][1] = v0.y; ak[h][2] = v1.x; ak[h][3] = v1.y;
            } else {
                const uint4 v = row16(KB == 2 ? pick(kw[h][S >> 2], S & 3, lane16) : pick(S & 1 ? kw1[h][S >> 3] : kw[h][S >> 3], (S >> 1) & 3, lane16));
                ak[h][0] = v.x; ak[h][1] = v.y; ak[h][2] = v.z; ak[h][3] = v.w;
            }
        }
        signs<S>(as);
    }
    template <int S>
    __device__ __forceinline__ void signs(uint32_t (&as)[4]) const { plus_minus<S>(sw, as); }
};

}  // namespace tqmma
