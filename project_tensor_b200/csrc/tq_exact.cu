// Exact kernels: float32 arithmetic carried out in the same order as the reference's NumPy path
// (tensor_gpu_v2/_quant.py), so that decisions taken on a knife edge -- a rotated coordinate that
// sits on a codebook boundary, a QJL projection that is almost zero -- come out the same way.
//
// Order of operations that is reproduced here:
//   * row reductions (np.linalg.norm, np.sum(axis=1)) use NumPy's pairwise scheme: blocks of at
//     most 128 elements are summed with 8 interleaved accumulators combined as
//     ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)); longer rows are split recursively at n/2 rounded
//     down to a multiple of 8;
//   * matrix products (`@`, BLAS sgemm) accumulate each output element with one fused
//     multiply-add per k, k ascending, starting from zero;
//   * every other elementwise step is a separately rounded float32 operation (no contraction).
//
// These kernels serve arbitrary (d <= 1024, bits <= 8), single tokens appended to a cache and small batches; they are
// also the second stage of the tensor-core quantizers, which hand over lists of coordinates and rows to re-decide.
#include "tq_common.cuh"
#include "tq_ptx.cuh"

namespace {

constexpr int kWarps = 4;

__device__ float np_pairwise_sum(const float* s, int n, int lane) {
    if (n < 8) {
        float r = 0.f;
        for (int i = 0; i < n; ++i) r = __fadd_rn(r, s[i]);
        return r;
    }
    if (n <= 128) {
        const int nb = n - (n & 7);
        float r = 0.f;
        if (lane < 8) {
            r = s[lane];
            for (int i = 8 + lane; i < nb; i += 8) r = __fadd_rn(r, s[i]);
        }
        r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 1));
        r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 2));
        r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 4));
        r = __shfl_sync(0xffffffffu, r, 0);
        for (int i = nb; i < n; ++i) r = __fadd_rn(r, s[i]);
        return r;
    }
    int h = n >> 1;
    h -= h & 7;
    const float a = np_pairwise_sum(s, h, lane);
    const float b = np_pairwise_sum(s + h, n - h, lane);
    return __fadd_rn(a, b);
}

// np.searchsorted(boundaries, v, side="left"): boundaries strictly below v; NaN sorts last.
__device__ __forceinline__ int count_below(const float* b, int nb, float v) {
    if (v != v) return nb;
    int lo = 0, hi = nb;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (b[mid] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// out[j] = sum_k vec[k] * M[k*d + j] for the four columns j0+lane+{0,32,64,96}; FMA chain, k ascending.
__device__ __forceinline__ void chain4(const float* vec, const float* __restrict__ M, int d, int j0, int lane,
                                       float acc[4]) {
    int j[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        j[c] = j0 + lane + 32 * c;
        if (j[c] >= d) j[c] = d - 1;  // keep the load in bounds; the caller ignores the value
        acc[c] = 0.f;
    }
#pragma unroll 4
    for (int k = 0; k < d; ++k) {
        const float v = vec[k];
        const float* m = M + (size_t)k * d;
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = __fmaf_rn(v, __ldg(m + j[c]), acc[c]);
    }
}

// Word w of a packed code row from the row's codes (bytes; zero behind d, eight readable bytes behind the last).  Codes are
// fetched eight at a time, so that a word costs a few loads in flight together and not one after the other.
__device__ __forceinline__ uint32_t packed_code_word(const uint8_t* cs, int bits, uint32_t inv_bits, int w) {
    const int lo_bit = w * 32;
    int j = (int)((uint32_t)lo_bit * inv_bits >> 16);        // lo_bit / bits
    int at = j * bits - lo_bit;                              // bit position of code j in the word, <= 0 for the first
    uint32_t v = 0;
    while (at < 32) {
        uint32_t c[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) c[i] = cs[j + i];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (at < 0) v |= c[i] >> -at;
            else if (at < 32) v |= c[i] << at;
            at += bits;
        }
        j += 8;
    }
    return v;
}
// floor(x / bits) = x * inverse >> 16 for x <= 8192 and bits <= 8
__device__ __forceinline__ uint32_t inverse_of_bits(int bits) { return (65536u + (uint32_t)bits - 1u) / (uint32_t)bits; }

// Boundaries strictly below v among levels - 1 sorted ones (a power of two less one): np.searchsorted(..., side="left");
// NaN sorts last.  N values at a time: every step of the bisection is a dependent load.
template <int N>
__device__ __forceinline__ void codes_of(const float* bnd, int levels, const float (&v)[N], int (&code)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) code[i] = 0;
    for (int step = levels >> 1; step > 0; step >>= 1) {
#pragma unroll
        for (int i = 0; i < N; ++i) code[i] += bnd[code[i] + step - 1] < v[i] ? step : 0;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) code[i] = v[i] != v[i] ? levels - 1 : code[i];
}

// Sum of squares of n values of one row (v[k * stride], k ascending) in NumPy's pairwise scheme, by eight lanes.
template <int STRIDE>
__device__ float np_sumsq8(const float* v, int n, int l8) {
    auto sq = [&](int i) { const float a = v[i * STRIDE]; return __fmul_rn(a, a); };
    if (n < 8) {
        float r = 0.f;
        for (int i = 0; i < n; ++i) r = __fadd_rn(r, sq(i));
        return r;
    }
    if (n <= 128) {
        const int nb = n - (n & 7);
        float r = sq(l8);
        if (nb == 128) {
            float a[15];
#pragma unroll
            for (int i = 0; i < 15; ++i) a[i] = sq(8 + 8 * i + l8);
#pragma unroll
            for (int i = 0; i < 15; ++i) r = __fadd_rn(r, a[i]);
        } else {
#pragma unroll 4
            for (int i = 8; i < nb; i += 8) r = __fadd_rn(r, sq(i + l8));
        }
        r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 1));
        r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 2));
        r = __fadd_rn(r, __shfl_xor_sync(0xffffffffu, r, 4));
        for (int i = nb; i < n; ++i) r = __fadd_rn(r, sq(i));
        return r;
    }
    int h = n >> 1;
    h -= h & 7;
    const float a = np_sumsq8<STRIDE>(v, h, l8);
    const float b = np_sumsq8<STRIDE>(v + h * STRIDE, n - h, l8);
    return __fadd_rn(a, b);
}

// Values l8, l8 + 8, ... of a row (row < 0: zeros) into v[k * stride], by eight lanes; bf16 and fp16 widened to float32.
// Sixteen loads are in flight at a time; the element type is looked at once.
template <class Load>
__device__ __forceinline__ void fill_row(float* v, int stride, int d, int l8, bool have, Load load) {
    for (int k0 = l8; k0 < d; k0 += 128) {
        float q[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) q[i] = have && k0 + 8 * i < d ? load(k0 + 8 * i) : 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (k0 + 8 * i < d) v[(k0 + 8 * i) * stride] = q[i];
    }
}
__device__ __forceinline__ float widen(uint16_t u, int xtype) {
    return xtype == TQ_INPUT_BF16 ? __uint_as_float((uint32_t)u << 16) : __half2float(__ushort_as_half(u));
}
__device__ __forceinline__ void load_row(float* v, int stride, int d, int l8, const void* x, int xtype, int64_t row) {
    const bool have = row >= 0;
    const int64_t at = (have ? row : 0) * d;
    if (xtype == TQ_INPUT_F32) {
        const float* src = static_cast<const float*>(x) + at;
        fill_row(v, stride, d, l8, have, [&](int k) { return __ldg(src + k); });
    } else {
        const uint16_t* src = static_cast<const uint16_t*>(x) + at;
        fill_row(v, stride, d, l8, have, [&](int k) { return widen(__ldg(src + k), xtype); });
    }
}
// Division of a row by its norm (zero rows stay zero); the same lanes own the same values.
__device__ __forceinline__ void divide_row(float* v, int stride, int d, int l8, float nr) {
    const bool ok = nr > 0.f;
#pragma unroll 4
    for (int k = l8; k < d; k += 8) {
        const float q = v[k * stride];
        v[k * stride] = ok ? __fdiv_rn(q, nr) : 0.f;
    }
}

// ------------------------------------------------------------------------------------------------
// Rows against whole matrices
// ------------------------------------------------------------------------------------------------
// One set of rows to quantize; a launch takes up to two (the keys and the values of a cache step).
struct RowsJob {
    TqDev p;
    const void* x;          // [n][d], element type `xtype`
    int xtype;              // TqInput
    int prod;               // TurboQuantProd: residual norm and signs behind the codes
    int64_t n;
    uint32_t* codes;
    uint32_t* signs;
    float* rnorms;
    float* norms;
    TqRecheck lists;        // hdr != null: only the listed rows
    unsigned long long* redo_counter;
    TqRowMap map;           // tokens > 0: rows of a cache
};

// Where rows come from and go to.  Every thread of a block holds the same values.
struct RowSource {
    int64_t limit, len0;
    bool listed, mapped;
    __device__ __forceinline__ void open(const RowsJob& job, bool first_block) {
        mapped = job.map.tokens > 0;
        len0 = !mapped ? 0 : !job.map.length ? job.map.base : tq_cache_length(job.map.length);
        const TqRecheckHeader* hdr = job.lists.hdr;
        // all rows, or the rows of the list (every row again if a list overflowed)
        listed = hdr != nullptr && hdr->overflow == 0;
        limit = listed ? (int64_t)min(hdr->n_rows, job.lists.row_cap) : job.n;
        if (job.redo_counter && first_block && threadIdx.x == 0) *job.redo_counter = (unsigned long long)limit;
    }
    __device__ __forceinline__ int64_t src(const RowsJob& job, int64_t idx) const {
        int64_t row = idx < limit ? (listed ? (int64_t)job.lists.row_entries[idx] : idx) : -1;
        return row < job.n ? row : -1;
    }
    __device__ __forceinline__ int64_t dst(const RowsJob& job, int64_t row) const {
        if (!mapped || row < 0) return row;
        const int64_t grow = row / job.map.tokens, pos = len0 + (row - grow * job.map.tokens);
        return pos < job.map.capacity ? grow * job.map.capacity + pos : -1;   // a full cache takes no more rows
    }
};

// The last block of a launch to get here raises the cache length.  Blocks count themselves in the upper bits of that very
// word, which are zero again when the kernel ends, so a step needs neither a second launch nor a counter of its own; readers
// on other streams mask them off (tq_cache_length) and see the old length or the new one.
// (Every block has read the length before it counts itself.)  advance == 2: nothing in the launch reads it; one block adds.
__device__ __forceinline__ void advance_length(const RowsJob& job, int64_t len0, int advance) {
    if (advance == 2) {
        if (blockIdx.x == 0) *job.map.counter += job.map.tokens;
        return;
    }
    unsigned long long* len = reinterpret_cast<unsigned long long*>(const_cast<int64_t*>(job.map.length));
    const unsigned long long before = atomicAdd(len, 1ull << kLengthBits);
    if ((before >> kLengthBits) == gridDim.x - 1) {
        const int64_t v = len0 + job.map.tokens;
        atomicExch(len, (unsigned long long)(v < job.map.capacity ? v : job.map.capacity));
    }
}

// Few rows, d <= 128 (a decode step's tokens, a handful of vectors): RB rows per block, the three matrices copied whole into
// shared memory (64 bytes a cycle and SM from L2: 1.6 us for the 192 KB of d = 128) while the rows are normalised; one thread
// per output, so that a product is a 128-long FMA chain with its loads running ahead.  64 keys and 64 values of d = 128 with the
// length: 9.8 us in one launch, 120 and 120 with two rows a block 9.6.
template <int RB>
__global__ void __launch_bounds__(128 * RB)
exact_quantize_few_kernel(const __grid_constant__ RowsJob first, const __grid_constant__ RowsJob second, int blocks0, int advance) {
    extern __shared__ __align__(16) float smem[];
    __shared__ __align__(16) float vt[RB][128], ct[RB][128];   // unit vector, later residual; centroids
    __shared__ uint8_t cs[RB][128 + 8];
    __shared__ float bnd[256], cbk[256], row_norm[RB];
    const bool one = (int)blockIdx.x < blocks0;
    const RowsJob& job = one ? first : second;
    const int block = one ? blockIdx.x : blockIdx.x - blocks0, nblocks = one ? blocks0 : gridDim.x - blocks0;
    const TqDev& p = job.p;
    const int d = p.d, levels = p.levels, dd4 = (d * d + 3) / 4;      // 16-byte pieces of a matrix (the slab is padded)
    const bool prod = job.prod != 0;
    constexpr int kThreads = 128 * RB;
    const int t = threadIdx.x, r = t >> 7, j = t & 127, lane = t & 31;
    auto copy = [&](int which, const float* M) {
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(smem + which * dd4 * 4);
#pragma unroll 8
        for (int i = t; i < dd4; i += kThreads)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 16), "l"(M + i * 4) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto product = [&](int which, const float* vec) {
        const float* m = smem + which * dd4 * 4 + (j < d ? j : 0);
        float acc = 0.f, b[16];
        int k = 0;
        constexpr bool kAhead = RB <= 2;      // the next piece on its way while one runs (four rows: other warps fill the time)
        auto fetch = [&](float (&to)[16], int from) {
#pragma unroll
            for (int i = 0; i < 16; ++i) to[i] = m[(from + i) * d];
        };
        if (kAhead && d >= 16) fetch(b, 0);
        for (; k + 16 <= d; k += 16) {
            float next[16];
            if constexpr (kAhead) fetch(next, k + 32 <= d ? k + 16 : k);      // (behind the end: the last piece again)
            else fetch(b, k);
#pragma unroll
            for (int i = 0; i < 16; i += 4) {
                const float4 v = *reinterpret_cast<const float4*>(vec + k + i);
                acc = __fmaf_rn(v.x, b[i], acc);
                acc = __fmaf_rn(v.y, b[i + 1], acc);
                acc = __fmaf_rn(v.z, b[i + 2], acc);
                acc = __fmaf_rn(v.w, b[i + 3], acc);
            }
            if constexpr (kAhead) {
#pragma unroll
                for (int i = 0; i < 16; ++i) b[i] = next[i];
            }
        }
        for (; k < d; ++k) acc = __fmaf_rn(vec[k], m[k * d], acc);
        return acc;
    };
    for (int i = t; i < levels; i += kThreads) {
        cbk[i] = __ldg(p.codebook + i);
        if (i + 1 < levels) bnd[i] = __ldg(p.boundaries + i);
    }
    copy(0, p.Rt);
    // One or two rows: the other two matrices are asked for behind them, or they would have to wait for all 192 KB.  (With that, a thread per
    // value and the products' loads a piece ahead, 100 TurboQuantProd rows of d = 128 take 8.4 us instead of 9.9, 64 keys and 64 values
    // 9.8 instead of 10.8.  Four rows a block are slower that way, 500 rows 14.7 against 13.0; also with two columns of all four rows a
    // thread, which halves the shared-memory traffic and leaves too few warps: 14.7 with the old loading, 15.6 with the new.)
    bool later = prod && RB <= 2;
    if (prod && !later) { copy(1, p.R); copy(2, p.St); }
    if (j < 8) cs[r][128 + j] = 0;
    const uint32_t inv_bits = inverse_of_bits(p.bits);
    tq_grid_release();
    tq_grid_wait();         // (only constants of the plan have been read so far)
    RowSource rows;
    rows.open(job, block == 0);
    for (int64_t g0 = (int64_t)block * RB; g0 < rows.limit; g0 += (int64_t)nblocks * RB) {
        const int64_t row = rows.src(job, g0 + r), to = rows.dst(job, row);
        __syncthreads();
        if constexpr (RB <= 2) {         // a thread per value; a row's sum of squares by eight lanes
            float value = 0.f;
            if (row >= 0 && j < d)
                value = job.xtype == TQ_INPUT_F32 ? __ldg(static_cast<const float*>(job.x) + row * d + j) : widen(__ldg(static_cast<const uint16_t*>(job.x) + row * d + j), job.xtype);
            if (later) {
                copy(1, p.R);
                copy(2, p.St);
                later = false;
            }
            vt[r][j] = value;
            __syncthreads();
            if (j < 32) {
                const float nr = __fsqrt_rn(np_sumsq8<1>(vt[r], d, lane & 7));
                if (j == 0) {
                    row_norm[r] = nr;
                    if (to >= 0) job.norms[to] = nr;
                }
            }
            __syncthreads();
            vt[r][j] = row_norm[r] > 0.f ? __fdiv_rn(value, row_norm[r]) : 0.f;
        } else {
            if (j < 8) {     // eight lanes per row: load, sum of squares, divide
                // (the other lanes of the warp wait here; with 16 values per lane the row is in flight at once)
                load_row(vt[r], 1, d, j, job.x, job.xtype, row);
            }
            if (j < 32) {
                __syncwarp();
                const float nr = __fsqrt_rn(np_sumsq8<1>(vt[r], d, lane & 7));
                __syncwarp();
                if (j < 8) divide_row(vt[r], 1, d, j, nr);
                if (j == 0 && to >= 0) job.norms[to] = nr;
            }
        }
        if (prod) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        {
            const float rotated[1] = {product(0, vt[r])};
            int code[1];
            codes_of<1>(bnd, levels, rotated, code);
            cs[r][j] = j < d ? (uint8_t)code[0] : 0;
            ct[r][j] = cbk[code[0]];
        }
        if (prod) asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (to >= 0 && j >= 128 - 32 && (int)(j - 96) < 32)     // the last warp of the row packs
            for (int w = j - 96; w < p.code_words; w += 32) job.codes[to * p.code_words + w] = packed_code_word(cs[r], p.bits, inv_bits, w);
        if (!prod) continue;
        const float res = __fsub_rn(vt[r][j], product(1, ct[r]));
        vt[r][j] = res;
        __syncthreads();
        if (j < 32) {
            const float rn = __fsqrt_rn(np_sumsq8<1>(vt[r], d, lane & 7));
            if (j == 0 && to >= 0) job.rnorms[to] = rn;
        }
        const float v = product(2, vt[r]);
        const uint32_t word = __ballot_sync(0xffffffffu, j < d && v >= 0.f);
        if (lane == 0 && j < d && to >= 0) job.signs[to * p.sign_words + (j >> 5)] = tq_sign_word_from_natural(word);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (advance) {
        __syncthreads();
        if (t == 0) advance_length(job, rows.len0, advance);
    }
}

// Any d, any number of rows: a block takes RB = RT * TR rows through every step of a call, the matrices stream through shared
// memory.  The vectors lie transposed ([k][row], padded to RB + 4); a thread owns TR rows x TC columns (column c of thread tx:
// tx + CT * c), loads TR + TC values per k and multiplies TR * TC.  The shared-memory pipe delivers one 32-lane register a
// cycle where the FMA pipes take four, so many rows want 8 x 8 sums per thread.  The matrices come in chunks of consecutive
// k -- all d columns, so a chunk is one contiguous piece of memory -- through a ring filled by cp.async, which runs ahead
// over the boundaries between the products and between groups of rows.
// TurboQuantProd, 65,536 rows (one thread per column with 8 rows before): d = 96 171 us, d = 128 251 us (0.37 ms before), bound by
// the FMA and shared-memory pipes (47 % of the FMA rate) and the phases between the products; the listed rows of 1,048,576 keys 18 us
// (29 us before).
template <int RT, int TR, int CT, int TC>
struct Tile {
    static constexpr int kRB = RT * TR, kRS = kRB + 4, kThreads = RT * CT, kCols = CT * TC;
    static_assert(TR % 4 == 0 && kThreads % 32 == 0, "tile");
};
struct TileShape {
    int kc;              // k per chunk (a multiple of 4, so that every chunk starts on a 16-byte boundary)
    int stages;
    int chunk_floats;    // ring stage, a multiple of 4
    size_t bytes;
};
// vectors: transposed arrays of d x kRS floats; the columns behind d of a panel are read (and their sums ignored)
template <class T>
TileShape tile_shape(int d, int vectors, size_t extra_bytes, size_t room) {
    TileShape s{};
    const size_t fixed = (size_t)vectors * d * T::kRS * 4 + extra_bytes + 64 + T::kCols * 4;
    for (int floats = 8192; floats >= 1024; floats >>= 1) {
        s.kc = floats / d / 4 * 4;
        if (s.kc < 4) s.kc = 4;
        s.chunk_floats = (s.kc * d + 3) / 4 * 4;
        for (s.stages = 4; s.stages >= (floats > 1024 ? 3 : 2); --s.stages) {
            s.bytes = fixed + (size_t)s.stages * s.chunk_floats * 4;
            if (s.bytes <= room) return s;
        }
    }
    s.stages = 0;
    return s;
}

template <int THREADS>
struct MatrixRing {
    float* stage;
    const float *m0, *m1, *m2;
    int nmat, d, kc, stages, chunk_floats;
    int m, k0;                  // next chunk to ask for
    int head, tail;             // stages: next to fill, next to use
    __device__ __forceinline__ void start(float* stage_, const float* a, const float* b, const float* c, int nmat_, int d_, const TileShape& t) {
        stage = stage_; m0 = a; m1 = b; m2 = c; nmat = nmat_; d = d_;
        kc = t.kc; stages = t.stages; chunk_floats = t.chunk_floats;
        m = k0 = head = tail = 0;
        for (int i = 0; i + 1 < stages; ++i) fetch();
    }
    __device__ __forceinline__ void fetch() {
        const float* src = (m == 0 ? m0 : m == 1 ? m1 : m2) + (size_t)k0 * d;
        const int n = min(kc, d - k0);
        const int pieces = (n * d + 3) >> 2;      // the last piece may read a few bytes past the matrix, into the slab's padding
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(stage + head * chunk_floats);
#pragma unroll 4
        for (int i = threadIdx.x; i < pieces; i += THREADS)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * 16), "l"(src + i * 4) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
        head = head + 1 == stages ? 0 : head + 1;
        k0 += kc;
        if (k0 >= d) { k0 = 0; m = m + 1 == nmat ? 0 : m + 1; }
    }
    __device__ __forceinline__ void wait() const {
        if (stages == 4) asm volatile("cp.async.wait_group 2;" ::: "memory");
        else if (stages == 3) asm volatile("cp.async.wait_group 1;" ::: "memory");
        else asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
};

// acc[r][c] = sum_k vt[k][row r] * M[k][column c]: one FMA per k, k ascending.
template <int RT, int TR, int CT, int TC>
__device__ __forceinline__ void tile_product(MatrixRing<RT * CT>& ring, const float* vt, int tx, int ty, float (&acc)[TR][TC]) {
    constexpr int kRS = Tile<RT, TR, CT, TC>::kRS;
    float2 two[TR / 2][TC];          // pairs of rows: fma.rn.f32x2 rounds each half as fma.rn.f32 does, in half the instructions
#pragma unroll
    for (int r = 0; r < TR / 2; ++r)
#pragma unroll
        for (int c = 0; c < TC; ++c) two[r][c] = make_float2(0.f, 0.f);
    const int d = ring.d;
    for (int k0 = 0; k0 < d; k0 += ring.kc) {
        ring.wait();
        __syncthreads();             // this chunk has landed for every thread, and everyone is done with the one before
        ring.fetch();
        const float* mt = ring.stage + ring.tail * ring.chunk_floats + tx;
        const float* v = vt + (size_t)k0 * kRS + ty * TR;
        ring.tail = ring.tail + 1 == ring.stages ? 0 : ring.tail + 1;
        const int n = min(ring.kc, d - k0);
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
            float a[TR], b[TC];
#pragma unroll
            for (int r = 0; r < TR; r += 4) *reinterpret_cast<float4*>(a + r) = *reinterpret_cast<const float4*>(v + k * kRS + r);
#pragma unroll
            for (int c = 0; c < TC; ++c) b[c] = mt[k * d + CT * c];
#pragma unroll
            for (int c = 0; c < TC; ++c)
#pragma unroll
                for (int r = 0; r < TR / 2; ++r)
                    two[r][c] = __ffma2_rn(make_float2(a[2 * r], a[2 * r + 1]), make_float2(b[c], b[c]), two[r][c]);
        }
    }
#pragma unroll
    for (int r = 0; r < TR / 2; ++r)
#pragma unroll
        for (int c = 0; c < TC; ++c) {
            acc[2 * r][c] = two[r][c].x;
            acc[2 * r + 1][c] = two[r][c].y;
        }
}

template <int RT, int TR, int CT, int TC>
__global__ void __launch_bounds__(RT * CT, 384 / (RT * CT))
exact_quantize_tile_kernel(const __grid_constant__ RowsJob first, const __grid_constant__ RowsJob second, int blocks0, int advance,
                           const TileShape shape) {
    using T = Tile<RT, TR, CT, TC>;
    constexpr int RB = T::kRB, RS = T::kRS, kGroups = T::kThreads / 8, kCodeRow = T::kCols + 8;
    extern __shared__ __align__(16) float smem[];
    const bool one = (int)blockIdx.x < blocks0;
    const RowsJob& job = one ? first : second;
    const int block = one ? blockIdx.x : blockIdx.x - blocks0, nblocks = one ? blocks0 : gridDim.x - blocks0;
    const TqDev& p = job.p;
    const int d = p.d, levels = p.levels;
    const bool prod = job.prod != 0;
    float* vt = smem;                                        // [d][RS] unit vectors, later residuals
    float* ct = vt + (size_t)d * RS;                         // [d][RS] centroid values
    uint8_t* cs = reinterpret_cast<uint8_t*>(ct + (size_t)d * RS);   // [RB][kCodeRow] codes
    float* stage = reinterpret_cast<float*>(cs + RB * kCodeRow);     // the ring, last: columns behind d are read past its end
    __shared__ float bnd[256], cbk[256];
    __shared__ int64_t src_row[RB], dst_row[RB];
    const int t = threadIdx.x, tx = t % CT, ty = t / CT, lane = t & 31, l8 = t & 7, grp = t >> 3;
    RowSource rows;
    tq_grid_release();
    if (job.lists.hdr != nullptr && !prod) {     // the list of a TurboQuantMSE call is empty as a rule
        tq_grid_wait();
        rows.open(job, block == 0);
        if (rows.limit == 0) {
            if (advance && t == 0) advance_length(job, rows.len0, advance);      // (block 0 raises the length, work or not)
            return;
        }
    }
    // The listed rows of a TurboQuantProd call have their codes as a rule, settled by the coordinate check: what is left are the
    // residual and its signs, two products of three.  (d > 128: below, fetching the codes costs what the product does.  524,309
    // rows, d = 256, with the listed rows' pass at 66 us: 15 us less.)
    const bool expected = prod && d > 128 && job.lists.hdr != nullptr;
    MatrixRing<T::kThreads> ring;
    if (expected) ring.start(stage, p.R, p.St, p.St, 2, d, shape);
    else ring.start(stage, p.Rt, p.R, p.St, prod ? 3 : 1, d, shape);
    for (int i = t; i < levels; i += T::kThreads) {
        cbk[i] = __ldg(p.codebook + i);
        if (i + 1 < levels) bnd[i] = __ldg(p.boundaries + i);
    }
    tq_grid_wait();         // (only constants of the plan have been read so far)
    rows.open(job, block == 0);
    const bool known = expected && rows.listed && job.lists.hdr->whole_rows == 0;
    if (expected && !known) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        ring.start(stage, p.Rt, p.R, p.St, 3, d, shape);
    }
    const uint32_t inv_bits = inverse_of_bits(p.bits);
    if (t < RB)
        for (int i = 0; i < 8; ++i) cs[t * kCodeRow + T::kCols + i] = 0;
    for (int64_t g0 = (int64_t)block * RB; g0 < rows.limit; g0 += (int64_t)nblocks * RB) {
        __syncthreads();             // the previous group is written out
        if (t < RB) {
            src_row[t] = rows.src(job, g0 + t);
            dst_row[t] = rows.dst(job, src_row[t]);
        }
        __syncthreads();
        // eight lanes per row: load, sum of squares, divide (lanes without a row keep the warp's shuffles company)
        for (int r0 = 0; r0 < RB; r0 += kGroups) {
            const bool mine = r0 + grp < RB;
            const int r = mine ? r0 + grp : RB - 1;
            const int64_t row = src_row[r];
            float* v = vt + r;
            if (mine) load_row(v, RS, d, l8, job.x, job.xtype, row);
            __syncwarp();
            const float nr = __fsqrt_rn(np_sumsq8<RS>(v, d, l8));
            __syncwarp();
            if (mine) {
                divide_row(v, RS, d, l8, nr);
                if (l8 == 0 && dst_row[r] >= 0) job.norms[dst_row[r]] = nr;
            }
        }
        // (the barrier in front of the first chunk orders the vectors)
        float acc[TR][TC];
        if (known) {
            constexpr int kAhead = 8;
            for (int i0 = t; i0 < RB * d; i0 += kAhead * T::kThreads) {
                uint32_t code[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; ++u) {
                    const int i = i0 + u * T::kThreads, r = i % RB, j = min(i / RB, d - 1);
                    const int64_t to = dst_row[r];
                    code[u] = tq_get_code(job.codes + (to < 0 ? 0 : to) * p.code_words, j, p.bits);
                }
#pragma unroll
                for (int u = 0; u < kAhead; ++u) {
                    const int i = i0 + u * T::kThreads;
                    if (i < RB * d) ct[i / RB * RS + i % RB] = cbk[code[u]];
                }
            }
        } else {
            // rotated[j] = sum_k unit[k] * R[j][k] -> codes, centroids
            tile_product<RT, TR, CT, TC>(ring, vt, tx, ty, acc);
#pragma unroll
            for (int c = 0; c < TC; ++c) {
                const int j = tx + CT * c;
                float v[TR], cent[TR];
                int code[TR];
#pragma unroll
                for (int r = 0; r < TR; ++r) v[r] = acc[r][c];
                codes_of<TR>(bnd, levels, v, code);
#pragma unroll
                for (int r = 0; r < TR; ++r) {
                    cs[(ty * TR + r) * kCodeRow + j] = j < d ? (uint8_t)code[r] : 0;
                    cent[r] = cbk[code[r]];
                }
                if (prod && j < d) {
#pragma unroll
                    for (int r = 0; r < TR; r += 4)
                        *reinterpret_cast<float4*>(ct + j * RS + ty * TR + r) = make_float4(cent[r], cent[r + 1], cent[r + 2], cent[r + 3]);
                }
            }
            __syncthreads();
            for (int i = t; i < RB * p.code_words; i += T::kThreads) {
                const int r = i / p.code_words, w = i - r * p.code_words;
                if (dst_row[r] >= 0) job.codes[dst_row[r] * p.code_words + w] = packed_code_word(cs + r * kCodeRow, p.bits, inv_bits, w);
            }
        }
        if (!prod) continue;
        // recon[j] = sum_k centroid[k] * R[k][j];  residual = unit - recon, in place (only this thread touches its elements)
        tile_product<RT, TR, CT, TC>(ring, ct, tx, ty, acc);
#pragma unroll
        for (int c = 0; c < TC; ++c) {
            const int j = tx + CT * c;
            if (j < d) {
#pragma unroll
                for (int r = 0; r < TR; r += 4) {
                    float4* at = reinterpret_cast<float4*>(vt + j * RS + ty * TR + r);
                    const float4 u = *at;
                    *at = make_float4(__fsub_rn(u.x, acc[r][c]), __fsub_rn(u.y, acc[r + 1][c]), __fsub_rn(u.z, acc[r + 2][c]),
                                      __fsub_rn(u.w, acc[r + 3][c]));
                }
            }
        }
        __syncthreads();
        for (int r0 = 0; r0 < RB; r0 += kGroups) {
            const bool mine = r0 + grp < RB;
            const int r = mine ? r0 + grp : RB - 1;
            const float rn = __fsqrt_rn(np_sumsq8<RS>(vt + r, d, l8));
            if (mine && l8 == 0 && dst_row[r] >= 0) job.rnorms[dst_row[r]] = rn;
        }
        // projected[j] = sum_k residual[k] * S[j][k] -> signs.  A ballot holds kBits consecutive columns of 32 / kBits rows.
        tile_product<RT, TR, CT, TC>(ring, vt, tx, ty, acc);
        constexpr int kBits = CT < 32 ? CT : 32, kPer = 32 / kBits;      // ballots per sign word
        constexpr uint32_t kMask = kBits == 32 ? 0xffffffffu : (1u << kBits) - 1u;
        const int shift = (lane / kBits) * kBits;
#pragma unroll
        for (int r = 0; r < TR; ++r) {
            const int64_t to = dst_row[ty * TR + r];
#pragma unroll
            for (int c0 = 0; c0 < TC; c0 += kPer) {
                uint32_t word = 0;
#pragma unroll
                for (int c = c0; c < c0 + kPer && c < TC; ++c)
                    word |= ((__ballot_sync(0xffffffffu, tx + CT * c < d && acc[r][c] >= 0.f) >> shift) & kMask) << ((c - c0) * kBits);
                const int j0 = tx / kBits * kBits + CT * c0;      // first column of the word
                if (lane == shift && j0 < d && to >= 0) job.signs[to * p.sign_words + (j0 >> 5)] = tq_sign_word_from_natural(word);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (advance && t == 0) advance_length(job, rows.len0, advance);
}

// ------------------------------------------------------------------------------------------------
// Second stage of the tensor-core quantizers, d <= 128: block b takes what block b of the quantizer left on its lists.  No list, counter
// or matrix is shared with another block, so nothing is cleared before, and one launch does what a memset, a kernel for the
// coordinates and a kernel for the rows did.  Work is small -- 70 coordinates and 16 rows a block of 1,048,576 TurboQuantProd keys at
// d = 128 -- so the kernel is as long as its chain of dependent steps: while eight lanes a coordinate re-decide those (of the keys and
// the values of a cache alike), eight warps fetch and normalise the listed rows, and the matrices come into shared memory; then
// the products of all rows side by side, four rows x four columns a thread.  Listed rows keep their codes, which the first half settles.
// 1,048,576 TurboQuantProd keys: 23 us behind the quantizer (37, and 6 in front of it, in three operations); 65,536 TurboQuantMSE
// rows 7.5 (11 and 4).  Of 36 K cycles the coordinates take 11 K (entry, row and matrix row from L2 or HBM, 16 divisions, a chain of
// 128), codes and matrices 7 K, a product 8 to 9 K: each piece of code runs once, and its instructions come from L2.
// ------------------------------------------------------------------------------------------------
struct StageJob {
    RowsJob rows;            // lists, redo_counter and map among it
    int blocks;              // blocks of its quantizer
};
constexpr int kStageThreads = 1024;
constexpr int kStageRows = 32;                                  // rows side by side: 16 +- 4 a block in the case above
constexpr int kProductRows = 4;                                 // rows x four columns of a product's thread (8: 11 to 16 K cycles a
                                                                // product instead of 8, too few warps and registers)
constexpr int kStageLoaders = kStageRows * 8;                   // threads that fetch rows, the last ones of the block
constexpr int kStageCheckers = kStageThreads - kStageLoaders;   // the others: coordinates first
constexpr int kStageExtra = 128;                                // rows whose codes the coordinates changed

template <int D>
struct StageSmem {
    static constexpr int kRS = kStageRows + 4;                 // vectors lie transposed, [k][row]
    static constexpr int kVec = D * kRS, kCodeRow = 128 + 8;
    static constexpr int bytes(int matrices) { return (matrices * D * D + 2 * kVec) * 4 + kStageRows * kCodeRow; }
};
struct StageWait {           // of a plan: limit of a bounded wait, status word
    int kcycles;
    unsigned long long* status;
};

template <int D>
__global__ void __launch_bounds__(kStageThreads, 1)
second_stage_kernel(const __grid_constant__ StageJob first, const __grid_constant__ StageJob second, int njobs, int advance, const StageWait wait) {
    using namespace tqptx;
    using L = StageSmem<D>;
    constexpr int RS = L::kRS, V = D / 8;
    extern __shared__ __align__(16) float smem[];
    float* vt = smem;                                          // [D][RS] unit vectors, later residuals
    float* ct = vt + L::kVec;                                  // [D][RS] centroids
    uint8_t* cs = reinterpret_cast<uint8_t*>(ct + L::kVec);    // [kStageRows][kCodeRow]
    float* mats = reinterpret_cast<float*>(cs + kStageRows * L::kCodeRow);      // R (or Rt), St: [k][column]
    __shared__ __align__(8) uint64_t arrived;                  // matrices
    __shared__ int give_up[2];                                 // flag, limit of a wait
    __shared__ float bnds[2][64], cbks[2][64];
    __shared__ unsigned int extra[kStageExtra], n_extra;
    __shared__ int64_t dst_row[kStageRows], src_row[kStageRows];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, l8 = t & 7, b = blockIdx.x;
    // Matrices come in by bulk copies (cp.async of the whole block would stand before every other load of the SM: entries took 5 K
    // cycles to arrive).  One thread asks, everybody waits.
    uint32_t phase = 0;
    // (in pieces, every block starting at another one: all of them read the same lines)
    auto fetch_matrices = [&](const float* first_matrix, const float* second_matrix) {      // into the first place, and the second
        if (warp != 0) return;
        constexpr int kPieces = 16, kPiece = D * D / kPieces;
        const int n = second_matrix ? 2 * kPieces : kPieces;
        if (lane == 0) {
            fence_async_smem();
            mbar_arrive_expect_tx(smem_u32(&arrived), (uint32_t)(n * kPiece * 4));
        }
        __syncwarp();
        if (lane < n) {
            const int piece = (lane + b) % n;
            const float* src = (piece < kPieces ? first_matrix : second_matrix) + (piece % kPieces) * kPiece;
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                         ::"r"(smem_u32(mats + piece * kPiece)), "l"(src), "r"(kPiece * 4), "r"(smem_u32(&arrived)) : "memory");
        }
    };
    auto matrices_here = [&]() {                                     // (the whole block; false: the wait ran out)
        const bool ok = mbar_wait(smem_u32(&arrived), phase, give_up);
        phase ^= 1u;
        return __syncthreads_and(ok) != 0;
    };
    if (t == 0) {
        mbar_init(smem_u32(&arrived), 1);
        give_up[0] = 0;
        give_up[1] = wait.kcycles;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    bool pending = first.rows.prod != 0;                       // matrices asked for that nobody has waited for
    if (pending) fetch_matrices(first.rows.p.R, first.rows.p.St);   // (a TurboQuantProd call leaves rows as a rule, a TurboQuantMSE call none)
    for (int i = t; i < kStageRows * L::kCodeRow; i += kStageThreads) cs[i] = 0;
    if (t < 128) {
        const TqDev& p = t < 64 ? first.rows.p : second.rows.p;
        const int i = t & 63;
        if (i < p.levels) cbks[t >> 6][i] = __ldg(p.codebook + i);
        if (i + 1 < p.levels) bnds[t >> 6][i] = __ldg(p.boundaries + i);
    }
    if (t == 0) n_extra = 0;
    tq_grid_release();
    tq_grid_wait();         // (only constants of the plans have been read so far)

    // lengths of this block's lists; a list that overflowed says: all rows of the block's tiles
    auto length_of = [&](const StageJob& j, int which) { return b < j.blocks ? j.rows.lists.counts[2 * b + which] : 0u; };
    unsigned int nc[2] = {length_of(first, 0), 0u}, nr[2] = {length_of(first, 1), 0u};
    if (njobs > 1) { nc[1] = length_of(second, 0); nr[1] = length_of(second, 1); }
    bool whole[2];
#pragma unroll
    for (int w = 0; w < 2; ++w) {
        const TqRecheck& l = w == 0 ? first.rows.lists : second.rows.lists;
        whole[w] = nc[w] > l.code_cap || nr[w] > l.row_cap;
        if (whole[w]) nc[w] = nr[w] = 0;
    }
    auto source = [&](const RowsJob& job) {
        RowSource rows;
        rows.mapped = job.map.tokens > 0;
        rows.len0 = rows.mapped ? job.map.base : 0;
        return rows;
    };
    // eight lanes fetch row src_row[r] and divide it by its norm (whole warps; lanes without a row, `mine` false, keep the warp's
    // shuffles company over its first row, which is there, and write nothing)
    auto fetch_row = [&](const RowsJob& job, int r, bool mine) {
        float* v = vt + (mine ? r : r & ~3);
        if (mine) load_row(v, RS, D, l8, job.x, job.xtype, src_row[r]);
        __syncwarp();
        const float n2 = __fsqrt_rn(np_sumsq8<RS>(v, D, l8));
        __syncwarp();
        if (mine) divide_row(v, RS, D, l8, n2);
        if (mine && l8 == 0 && dst_row[r] >= 0) job.norms[dst_row[r]] = n2;
    };
    __syncthreads();

    // -- coordinates: norm, division and the rotated coordinate as one FMA chain that goes from lane to lane (lane l has the values
    // [l V, + V) of the row); the first job's listed rows beside it
    const unsigned int head = nr[0] < kStageRows ? nr[0] : kStageRows;       // rows of the first batch
    if (t >= kStageCheckers) {
        const int r = (t - kStageCheckers) >> 3;
        const bool mine = r < (int)head;
        if (l8 == 0 && mine) {
            const int64_t row = (int64_t)(first.rows.lists.row_entries[(size_t)b * first.rows.lists.row_cap + r] & kRowNumber);
            src_row[r] = row < first.rows.n ? row : -1;
            dst_row[r] = source(first.rows).dst(first.rows, src_row[r]);
        }
        __syncwarp();
        if ((r & ~3) < (int)head) fetch_row(first.rows, r, mine);
    } else {
        for (unsigned int base = 0; base < nc[0] + nc[1]; base += kStageCheckers / 8) {
            const unsigned int at = base + (t >> 3);
            const int w = at >= nc[0];
            const RowsJob& job = w ? second.rows : first.rows;
            const TqDev& p = job.p;
            const bool given = at < nc[0] + nc[1];
            const unsigned long long ent = given ? job.lists.code_entries[(size_t)b * job.lists.code_cap + (at - (w ? nc[0] : 0u))] : 0ull;
            const int64_t row = (int64_t)(ent >> 8);
            const int j = (int)(ent & 255u);
            const bool valid = given && row < job.n && j < D;
            if (!__any_sync(0xffffffffu, valid)) continue;
            const int64_t to = source(job).dst(job, valid ? row : 0);
            uint32_t* crow = job.codes + to * p.code_words;
            const uint32_t old = valid && l8 == 7 ? tq_get_code(crow, j, p.bits) : 0u;
            const int64_t first_value = (valid ? row : 0) * D;
            float a[V], c[V];        // values l, l + 8, ... (NumPy's eight interleaved sums); values [l V, + V)
            if (first.rows.xtype == TQ_INPUT_F32) {              // (the jobs of a call have one element type)
                const float* x = static_cast<const float*>(job.x) + first_value;
#pragma unroll
                for (int i = 0; i < V; ++i) a[i] = __ldg(x + l8 + 8 * i);
#pragma unroll
                for (int i = 0; i < V; i += 4) *reinterpret_cast<float4*>(c + i) = __ldg(reinterpret_cast<const float4*>(x + l8 * V + i));
            } else {
                const uint16_t* x = static_cast<const uint16_t*>(job.x) + first_value;
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    a[i] = widen(__ldg(x + l8 + 8 * i), first.rows.xtype);
                    c[i] = widen(__ldg(x + l8 * V + i), first.rows.xtype);
                }
            }
            float sum = __fmul_rn(a[0], a[0]);
#pragma unroll
            for (int i = 1; i < V; ++i) sum = __fadd_rn(sum, __fmul_rn(a[i], a[i]));
#pragma unroll
            for (int s = 1; s < 8; s <<= 1) sum = __fadd_rn(sum, __shfl_xor_sync(0xffffffffu, sum, s));
            float m[V];
#pragma unroll
            for (int i = 0; i < V; i += 4) *reinterpret_cast<float4*>(m + i) = __ldg(reinterpret_cast<const float4*>(p.R + (size_t)(valid ? j : 0) * D + l8 * V + i));
            const float n2 = __fsqrt_rn(sum);
#pragma unroll
            for (int i = 0; i < V; ++i) c[i] = n2 > 0.f ? __fdiv_rn(c[i], n2) : 0.f;
            float acc = 0.f;
#pragma unroll 1
            for (int s = 0; s < 8; ++s) {
                const float before = __shfl_sync(0xffffffffu, acc, (lane & 24) + (s > 0 ? s - 1 : 0));
                acc = s > 0 ? before : 0.f;
#pragma unroll
                for (int i = 0; i < V; ++i) acc = __fmaf_rn(c[i], m[i], acc);
            }
            const uint32_t code = valid && l8 == 7 ? (uint32_t)count_below(bnds[w], p.levels - 1, acc) : 0u;
            unsigned int slot = ~0u;
            if (old != code) {
                atomicAdd(&job.lists.hdr->changed, 1u);
                const uint32_t delta = old ^ code;
                const int bit = j * p.bits, word = bit >> 5, sh = bit & 31;
                atomicXor(crow + word, delta << sh);
                if (sh + p.bits > 32) atomicXor(crow + word + 1, delta >> (32 - sh));
                if (job.prod) {          // the row's residual is another one: it joins the rows, as it stands here
                    const unsigned int pos = atomicAdd(&n_extra, 1u);
                    if (pos < kStageExtra) extra[pos] = (unsigned int)row;
                    slot = head + pos;
                }
            }
            slot = __shfl_sync(0xffffffffu, slot, lane | 7);
            if (slot < kStageRows) {
#pragma unroll
                for (int i = 0; i < V; ++i) vt[(l8 * V + i) * RS + slot] = c[i];
                if (l8 == 7) job.norms[to] = n2;
            }
        }
    }
    __threadfence_block();
    __syncthreads();
    const unsigned int extras = n_extra;
    if (extras > kStageExtra) whole[0] = true;
    unsigned int placed = kStageRows - head < extras ? kStageRows - head : extras;
    if (t < (int)placed) {
        const int64_t row = extra[t];
        src_row[head + t] = row;
        dst_row[head + t] = source(first.rows).dst(first.rows, row);
    }

    // -- rows in batches: the one that stands in shared memory, the rest of the lists, or all rows of the block's tiles
    for (int which = 0; which < njobs; ++which) {
        const StageJob& stage = which == 0 ? first : second;
        const RowsJob& job = stage.rows;
        const TqDev& p = job.p;
        const bool prod = job.prod != 0;
        const RowSource rows = source(job);
        const float* bnd = bnds[which];
        const float* cbk = cbks[which];
        const uint32_t inv_bits = inverse_of_bits(p.bits);
        const bool all = whole[which];
        int64_t total = which == 0 ? (int64_t)nr[0] + extras : nr[1], next = 0;
        int ready = which == 0 && !all ? (int)(head + placed) : 0;           // rows of this batch that stand in shared memory
        if (all) {
            const int64_t tiles = (job.n + 127) / 128;
            total = b < tiles ? (tiles - b + stage.blocks - 1) / stage.blocks * 128 : 0;
        }
        bool ok = true;
        if (total > 0 && which == 1) {
            if (pending) ok = matrices_here();       // the first job had no rows: another copy may not meet its matrices
            pending = false;
            if (prod && ok) {
                fetch_matrices(p.R, p.St);
                pending = true;
            }
        }
        for (next = 0; next < total && ok;) {
            int count = ready;
            if (ready == 0) {
                count = (int)(total - next < kStageRows ? total - next : kStageRows);
                __syncthreads();                                         // (the batch before is written out)
                if (t < kStageRows) {
                    const int64_t i = next + t;
                    int64_t row = -1;
                    if (t < count) {
                        if (all) row = (b + i / 128 * stage.blocks) * 128 + i % 128;
                        else if (which == 1) row = (int64_t)job.lists.row_entries[(size_t)b * job.lists.row_cap + i];
                        else if (i - placed < nr[0]) row = (int64_t)job.lists.row_entries[(size_t)b * job.lists.row_cap + (i - placed)];
                        else row = (int64_t)extra[i - nr[0]];
                        row &= kRowNumber;
                        if (row >= job.n) row = -1;
                    }
                    src_row[t] = row;
                    dst_row[t] = rows.dst(job, row);
                }
                __syncthreads();
                if (t >= kStageCheckers) fetch_row(job, (t - kStageCheckers) >> 3, true);
            }
            ready = 0;
            next += count;
            // A listed row has its codes, settled above, unless its norm was outside the tensor-core kernel's range (its number says so).
            bool odd = false;
            if (t < count && !all) {
                const int64_t i = next - count + t;
                const int64_t at = i < head ? i : i - placed;
                if (which == 1) odd = true;
                else if (i < head || (i >= head + placed && at < nr[0])) odd = (job.lists.row_entries[(size_t)b * job.lists.row_cap + at] & ~kRowNumber) != 0;
            }
            const bool full = __syncthreads_or(odd || all || !prod) != 0;

            // acc[q][u] = sum_k vec[k][8 warp + q] * M[k][4 lane + u]: one FMA per k, k ascending
            const int product_warps = (count + kProductRows - 1) / kProductRows;
            const bool product_role = warp < product_warps, in_range = 4 * lane < D;
            auto product = [&](int place, const float* vec, float (&acc)[kProductRows][4]) {
                const float* m = mats + place * D * D + (in_range ? 4 * lane : 0);
                const float* v = vec + kProductRows * warp;
                float2 two[kProductRows / 2][4];        // pairs of rows: fma.rn.f32x2 rounds each half as fma.rn.f32 does
#pragma unroll
                for (int q = 0; q < kProductRows / 2; ++q)
#pragma unroll
                    for (int u = 0; u < 4; ++u) two[q][u] = make_float2(0.f, 0.f);
#pragma unroll 2
                for (int k = 0; k < D; ++k) {
                    float a[kProductRows];
#pragma unroll
                    for (int q = 0; q < kProductRows; q += 4) *reinterpret_cast<float4*>(a + q) = *reinterpret_cast<const float4*>(v + k * RS + q);
                    const float4 bb = *reinterpret_cast<const float4*>(m + k * D);
                    const float col[4] = {bb.x, bb.y, bb.z, bb.w};
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int q = 0; q < kProductRows / 2; ++q)
                            two[q][u] = __ffma2_rn(make_float2(a[2 * q], a[2 * q + 1]), make_float2(col[u], col[u]), two[q][u]);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int q = 0; q < kProductRows / 2; ++q) {
                        acc[2 * q][u] = two[q][u].x;
                        acc[2 * q + 1][u] = two[q][u].y;
                    }
            };
            float acc[kProductRows][4];
            if (full) {
                if (pending && !matrices_here()) { ok = pending = false; break; }
                pending = false;
                fetch_matrices(p.Rt, nullptr);       // (for the one product, in the place of R)
                if (!matrices_here()) { ok = false; break; }
                if (product_role) {
                    product(0, vt, acc);
#pragma unroll
                    for (int q = 0; q < kProductRows; ++q) {
                        int code[4];
                        codes_of<4>(bnd, p.levels, acc[q], code);
                        const int r = kProductRows * warp + q;
                        if (in_range) {
                            *reinterpret_cast<uint32_t*>(cs + r * L::kCodeRow + 4 * lane) = (uint32_t)code[0] | (uint32_t)code[1] << 8 | (uint32_t)code[2] << 16 | (uint32_t)code[3] << 24;
#pragma unroll
                            for (int u = 0; u < 4; ++u) ct[(4 * lane + u) * RS + r] = cbk[code[u]];
                        }
                    }
                }
                __syncthreads();
                if (prod) fetch_matrices(p.R, nullptr);
                for (int i = t; i < count * p.code_words; i += kStageThreads) {
                    const int r = i / p.code_words, w = i - r * p.code_words;
                    if (dst_row[r] >= 0) job.codes[dst_row[r] * p.code_words + w] = packed_code_word(cs + r * L::kCodeRow, p.bits, inv_bits, w);
                }
                if (!prod) continue;
                if (!matrices_here()) { ok = false; break; }
            } else {
                // (through L2, where the corrections went)
                for (int i = t; i < count * D; i += kStageThreads) {
                    const int r = i / D, j = i % D, bit = j * p.bits, w = bit >> 5, sh = bit & 31;
                    const uint32_t* row = job.codes + (dst_row[r] < 0 ? 0 : dst_row[r]) * p.code_words + w;
                    uint32_t v = __ldcg(row) >> sh;
                    if (sh + p.bits > 32) v |= __ldcg(row + 1) << (32 - sh);
                    ct[j * RS + r] = cbk[v & ((1u << p.bits) - 1u)];
                }
                if (pending && !matrices_here()) { ok = pending = false; break; }
                pending = false;
                __syncthreads();
            }
            if (product_role) {          // residual = unit - centroids * R, in place (only this thread touches its elements)
                product(0, ct, acc);
                if (in_range) {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
#pragma unroll
                        for (int q = 0; q < kProductRows; q += 4) {
                            float4* at = reinterpret_cast<float4*>(vt + (4 * lane + u) * RS + kProductRows * warp + q);
                            const float4 unit = *at;
                            *at = make_float4(__fsub_rn(unit.x, acc[q][u]), __fsub_rn(unit.y, acc[q + 1][u]), __fsub_rn(unit.z, acc[q + 2][u]), __fsub_rn(unit.w, acc[q + 3][u]));
                        }
                }
            }
            __syncthreads();
            if (t >= kStageCheckers) {
                const int r = (t - kStageCheckers) >> 3;
                const float rn = __fsqrt_rn(np_sumsq8<RS>(vt + r, D, l8));
                if (l8 == 0 && r < count && dst_row[r] >= 0) job.rnorms[dst_row[r]] = rn;
            } else if (product_role) {
                product(1, vt, acc);
#pragma unroll
                for (int q = 0; q < kProductRows; ++q) {
                    uint32_t word = 0;           // the signs of 32 columns from eight lanes
#pragma unroll
                    for (int u = 0; u < 4; ++u) word |= (acc[q][u] >= 0.f ? 1u : 0u) << (4 * l8 + u);
#pragma unroll
                    for (int s = 1; s < 8; s <<= 1) word |= __shfl_xor_sync(0xffffffffu, word, s);
                    const int r = kProductRows * warp + q;
                    if (l8 == 0 && in_range && r < count && dst_row[r] >= 0) job.signs[dst_row[r] * p.sign_words + (lane >> 3)] = tq_sign_word_from_natural(word);
                }
            }
        }
        if (!ok) break;
        if (t == 0 && total > 0) atomicAdd(&job.lists.hdr->n_rows, (unsigned int)total);
    }
    if (pending) matrices_here();        // (nothing may land in shared memory that the block has left)
    if (t == 0) {
        if (give_up[0]) {
            report_status(wait.status, 1ull);
            mbar_drain(smem_u32(&arrived), phase ^ 1u);
        }
        __threadfence();
        if (atomicAdd(&first.rows.lists.hdr->done, 1u) == gridDim.x - 1) {        // the last block has every block's sum
            __threadfence();
            if (first.rows.redo_counter) *first.rows.redo_counter = atomicAdd(&first.rows.lists.hdr->n_rows, 0u);
            if (njobs > 1 && second.rows.redo_counter) *second.rows.redo_counter = atomicAdd(&second.rows.lists.hdr->n_rows, 0u);
        }
        if (advance) advance_length(first.rows, 0, advance);
    }
}

// d = 256, listed coordinates (those inside the guard band of the tensor-core kernel) re-decided in the reference's order, eight lanes
// each: norm, division, and the rotated coordinate as one FMA chain that goes from lane to lane (lane l has the values [32 l, + 32)).
// A wrong code is corrected in place and (TurboQuantProd) puts its row on the row list.  Every dependent access to global memory
// costs about a microsecond, so what counts is how many entries are on their way side by side: 64 an SM, in registers.  524,309
// TurboQuantProd rows (22,000 entries): 23 us behind the quantizer, 41 with sixteen lanes an entry and the rows in shared memory.
struct CheckJob {
    TqDev p;
    const void* x;
    int xtype, prod;
    int64_t n;
    uint32_t* codes;
    TqRecheck lists;
    TqRowMap map;
};
constexpr int kCheckEntries = 32;        // of a block at a time

__global__ void __launch_bounds__(kCheckEntries * 8, 2)
exact_code_check_kernel(const __grid_constant__ CheckJob first, const __grid_constant__ CheckJob second, int blocks0) {
    constexpr int D = 256, V = D / 8;
    __shared__ float bnd[16];
    const bool one = (int)blockIdx.x < blocks0;
    const CheckJob& job = one ? first : second;
    const TqDev& p = job.p;
    const unsigned int block = one ? blockIdx.x : blockIdx.x - blocks0, nblocks = one ? blocks0 : gridDim.x - blocks0;
    const int t = threadIdx.x, lane = t & 31, l = t & 7;
    const TqRecheck& lists = job.lists;
    if (t < p.levels - 1) bnd[t] = __ldg(p.boundaries + t);      // (at most 15: the kernel at d = 256 takes up to 4 bits)
    __syncthreads();
    tq_grid_release();
    tq_grid_wait();
    // asked for before the header is known to allow it (the list's capacity bounds the index)
    unsigned int at = block * kCheckEntries + (t >> 3);
    unsigned long long ent = at < lists.code_cap ? lists.code_entries[at] : 0ull;
    if (lists.hdr->overflow) return;  // the row pass will redo everything
    const unsigned int count = min(lists.hdr->n_codes, lists.code_cap);
    for (; at - (t >> 3) < count; at += nblocks * kCheckEntries) {
        if (at != block * kCheckEntries + (t >> 3)) ent = at < count ? lists.code_entries[at] : 0ull;
        const int64_t row = (int64_t)(ent >> 8);
        const int j = (int)(ent & 255u);
        const bool valid = at < count && row < job.n;
        if (!__any_sync(0xffffffffu, valid)) continue;
        uint32_t* crow = job.codes + (!valid ? 0 : job.map.tokens > 0 ? row / job.map.tokens * job.map.capacity + job.map.base + row % job.map.tokens : row) * p.code_words;
        const uint32_t old = valid && l == 7 ? tq_get_code(crow, j, p.bits) : 0u;
        const int64_t x0 = (valid ? row : 0) * D;
        float c[V], m[V];
        {
            const float4* src = reinterpret_cast<const float4*>(p.R + (size_t)(valid ? j : 0) * D + l * V);
#pragma unroll
            for (int i = 0; i < V / 4; ++i) *reinterpret_cast<float4*>(m + 4 * i) = __ldg(src + i);
        }
        float half[2];       // NumPy's pairwise sum: eight interleaved sums for each 128 values
        {
            float a[V];
            if (job.xtype == TQ_INPUT_F32) {
                const float* x = static_cast<const float*>(job.x) + x0;
#pragma unroll
                for (int i = 0; i < V; ++i) a[i] = __ldg(x + l + 8 * i);
#pragma unroll
                for (int i = 0; i < V; i += 4) *reinterpret_cast<float4*>(c + i) = __ldg(reinterpret_cast<const float4*>(x + l * V + i));
            } else {
                const uint16_t* x = static_cast<const uint16_t*>(job.x) + x0;
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    a[i] = widen(__ldg(x + l + 8 * i), job.xtype);
                    c[i] = widen(__ldg(x + l * V + i), job.xtype);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                half[h] = __fmul_rn(a[h * 16], a[h * 16]);
#pragma unroll
                for (int i = 1; i < 16; ++i) half[h] = __fadd_rn(half[h], __fmul_rn(a[h * 16 + i], a[h * 16 + i]));
            }
        }
#pragma unroll
        for (int s = 1; s < 8; s <<= 1) {
            half[0] = __fadd_rn(half[0], __shfl_xor_sync(0xffffffffu, half[0], s));
            half[1] = __fadd_rn(half[1], __shfl_xor_sync(0xffffffffu, half[1], s));
        }
        const float nr = __fsqrt_rn(__fadd_rn(half[0], half[1]));
#pragma unroll
        for (int i = 0; i < V; ++i) c[i] = nr > 0.f ? __fdiv_rn(c[i], nr) : 0.f;
        float acc = 0.f;
#pragma unroll 1
        for (int s = 0; s < 8; ++s) {
            const float before = __shfl_sync(0xffffffffu, acc, (lane & 24) + (s > 0 ? s - 1 : 0));
            acc = s > 0 ? before : 0.f;
#pragma unroll
            for (int i = 0; i < V; ++i) acc = __fmaf_rn(c[i], m[i], acc);
        }
        if (valid && l == 7) {
            const uint32_t code = (uint32_t)count_below(bnd, p.levels - 1, acc);
            if (old != code) {
                if (job.prod) {        // the row's residual is another one
                    const unsigned int pos = atomicAdd(&lists.hdr->n_rows, 1u);
                    if (pos < lists.row_cap) lists.row_entries[pos] = (unsigned int)row;
                    else lists.hdr->overflow = 1u;
                }
                const uint32_t delta = old ^ code;
                const int bit = j * p.bits, w = bit >> 5, sh = bit & 31;
                atomicXor(crow + w, delta << sh);
                if (sh + p.bits > 32) atomicXor(crow + w + 1, delta >> (32 - sh));
                atomicAdd(&lists.hdr->changed, 1u);
            }
        }
    }
}

// TurboQuantMSE.dequantize / TurboQuantProd.dequantize (_quant.py:238-242,251-254,317-332): the block shape of
// exact_quantize_tile_kernel.
template <bool PROD, int RT, int TR, int CT, int TC>
__global__ void __launch_bounds__(RT * CT, 384 / (RT * CT))
exact_dequantize_tile_kernel(const __grid_constant__ TqDev p, const uint32_t* __restrict__ codes, const uint32_t* __restrict__ signs,
                             const float* __restrict__ rnorms, const float* __restrict__ norms, int64_t n,
                             float* __restrict__ out, const TileShape shape) {
    using T = Tile<RT, TR, CT, TC>;
    constexpr int RB = T::kRB, RS = T::kRS;
    extern __shared__ __align__(16) float smem[];
    const int d = p.d;
    float* ct = smem;                                        // [d][RS] centroid values
    float* sg = ct + (size_t)d * RS;                         // [d][RS] +-1
    float* stage = sg + (PROD ? (size_t)d * RS : 0);
    __shared__ float cbk[256];
    const int t = threadIdx.x, tx = t % CT, ty = t / CT, l8 = t & 7, grp = t >> 3;
    MatrixRing<T::kThreads> ring;
    ring.start(stage, p.R, p.S, p.S, PROD ? 2 : 1, d, shape);
    for (int i = t; i < p.levels; i += T::kThreads) cbk[i] = __ldg(p.codebook + i);
    for (int64_t g0 = (int64_t)blockIdx.x * RB; g0 < n; g0 += (int64_t)gridDim.x * RB) {
        __syncthreads();
        for (int r = grp; r < RB; r += T::kThreads / 8) {
            const int64_t row = g0 + r < n ? g0 + r : 0;
            const uint32_t* crow = codes + row * p.code_words;
            const uint32_t* srow = PROD ? signs + row * p.sign_words : nullptr;
#pragma unroll 4
            for (int k = l8; k < d; k += 8) {
                ct[k * RS + r] = cbk[tq_get_code(crow, k, p.bits)];
                if (PROD) sg[k * RS + r] = ((__ldg(srow + (k >> 5)) >> tq_sign_bitpos(k)) & 1u) ? 1.f : -1.f;
            }
        }
        float acc[TR][TC], acs[PROD ? TR : 4][TC];
        tile_product<RT, TR, CT, TC>(ring, ct, tx, ty, acc);
        if constexpr (PROD) tile_product<RT, TR, CT, TC>(ring, sg, tx, ty, acs);
#pragma unroll
        for (int r = 0; r < TR; ++r) {
            const int64_t row = g0 + ty * TR + r;
            if (row >= n) continue;
            const float nr = __ldg(norms + row), rn = PROD ? __ldg(rnorms + row) : 0.f;
#pragma unroll
            for (int c = 0; c < TC; ++c) {
                const int j = tx + CT * c;
                float u = acc[r][c];
                if (PROD) u = __fadd_rn(u, __fmul_rn(__fmul_rn(acs[r][c], p.alpha), rn));
                if (j < d) out[row * d + j] = __fmul_rn(u, nr);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// TurboQuantProd.attention_score with one query row per key (_quant.py:342-358), in the
// reference's own order: de-rotate the key, multiply by the query, pairwise-sum.
__global__ void __launch_bounds__(kWarps * 32)
exact_pairwise_score_kernel(TqDev p, const float* __restrict__ q, const uint32_t* __restrict__ codes,
                            const uint32_t* __restrict__ signs, const float* __restrict__ rnorms,
                            const float* __restrict__ norms, int64_t n, float* __restrict__ scores) {
    extern __shared__ float smem[];
    const int d = p.d, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int dp = (d + 31) & ~31;
    float* qa = smem + (size_t)warp * 3 * dp;  // query row
    float* ca = qa + dp;                       // centroid values, then products
    float* pa = ca + dp;                       // products of the second stage
    for (int64_t row = (int64_t)blockIdx.x * kWarps + warp; row < n; row += (int64_t)gridDim.x * kWarps) {
        const uint32_t* crow = codes + row * p.code_words;
        const uint32_t* srow = signs + row * p.sign_words;
        for (int k = lane; k < d; k += 32) {
            qa[k] = q[row * d + k];
            ca[k] = __ldg(p.codebook + tq_get_code(crow, k, p.bits));
        }
        __syncwarp();
        float t1[32], t2[32];  // d <= 1024 -> at most 32 columns per lane
        int cnt = 0;
        for (int j0 = 0; j0 < d; j0 += 128) {
            float r[4], s[4];
            chain4(ca, p.R, d, j0, lane, r);
            chain4(qa, p.St, d, j0, lane, s);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int j = j0 + lane + 32 * c;
                float a = 0.f, b = 0.f;
                if (j < d) {
                    a = __fmul_rn(qa[j], r[c]);
                    b = ((srow[j >> 5] >> tq_sign_bitpos(j)) & 1u) ? s[c] : -s[c];
                }
                t1[cnt] = a;
                t2[cnt] = b;
                ++cnt;
            }
        }
        __syncwarp();
        cnt = 0;
        for (int j0 = 0; j0 < d; j0 += 128) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int j = j0 + lane + 32 * c;
                if (j < d) { ca[j] = t1[cnt]; pa[j] = t2[cnt]; }
                ++cnt;
            }
        }
        __syncwarp();
        const float s1 = np_pairwise_sum(ca, d, lane);
        const float s2 = np_pairwise_sum(pa, d, lane);
        if (lane == 0) {
            const float st2 = __fmul_rn(__fmul_rn(p.alpha, rnorms[row]), s2);
            scores[row] = __fmul_rn(norms[row], __fadd_rn(s1, st2));
        }
        __syncwarp();
    }
}

int grid_for(int64_t work_items, int per_block) {
    int64_t g = (work_items + per_block - 1) / per_block;
    const int64_t cap = 148 * 16;
    if (g > cap) g = cap;
    if (g < 1) g = 1;
    return (int)g;
}

}  // namespace

int tq_launch_exact_code_check(const TqSecondStage* a, const TqSecondStage* b, cudaStream_t st) {
    TqRange range("tq.quantize.recheck_coordinates");
    const int d = a->plan->dev.d;
    if (d != 256) return tq_fail(TQ_ERR_UNSUPPORTED, "the coordinate re-check alone is written for d = 256");
    const int64_t per_block = kCheckEntries, most = tq_sm_count(a->plan->device) * (int64_t)(b ? 1 : 2);
    // as many blocks as a list of typical length has entries for (about 1 in 48 rows of 128 coordinates at 4 bits, in
    // proportion to the coordinates); longer lists take more passes
    auto blocks = [&](const TqSecondStage* s) {
        const int64_t w = (s->n * d / 128 / 48 + per_block - 1) / per_block;
        return (int)(w < 4 ? 4 : w > most ? most : w);
    };
    auto job = [](const TqSecondStage* s) {
        CheckJob j{};
        j.p = s->plan->dev; j.x = s->x; j.xtype = s->xtype; j.prod = s->prod ? 1 : 0; j.n = s->n;
        j.codes = s->out.codes; j.lists = s->lists; j.map = s->out.map;
        return j;
    };
    const CheckJob first = job(a), second = b ? job(b) : first;
    const int b0 = blocks(a), grid = b0 + (b ? blocks(b) : 0);
    TQ_CUDA_TRY(tq_launch_dependent(exact_code_check_kernel, dim3(grid), dim3(kCheckEntries * 8), 0, st, first, second, b0));
    return TQ_OK;
}

namespace {
// Blocks for `rows` rows of one job out of `room` that run at once.
int job_blocks(int64_t rows, int per_block, int64_t room) {
    const int64_t g = (rows + per_block - 1) / per_block;
    return (int)(g < 1 ? 1 : g < room ? g : room < 1 ? 1 : room);
}
// Of two jobs that share a launch the first (TurboQuantProd keys, three products per row) gets two thirds of the blocks.
void split_room(const RowsJob* b, int64_t rows, int per_block, int64_t room, int* b0, int* b1) {
    *b0 = job_blocks(rows, per_block, b ? room * 2 / 3 : room);
    *b1 = b ? job_blocks(rows, per_block, room - *b0) : 0;
}

template <int RB>
int launch_few_rows(const RowsJob& a, const RowsJob* b, int64_t rows, int device, int advance, cudaStream_t st) {
    int b0, b1;
    split_room(b, rows, RB, tq_sm_count(device), &b0, &b1);
    const int sm = (a.prod || (b && b->prod) ? 3 : 1) * ((a.p.d * a.p.d + 3) / 4 * 16);
    TQ_GRANT_SMEM((exact_quantize_few_kernel<RB>), sm, device);
    TQ_CUDA_TRY(tq_launch_dependent(exact_quantize_few_kernel<RB>, dim3(b0 + b1), dim3(128 * RB), (size_t)sm, st, a, b ? *b : a, b0, advance));
    return TQ_OK;
}
// Blocks of a kernel that an SM's registers hold (its shared memory is a matter of the shape); asked for once per kernel.
template <class K>
int blocks_by_registers(K kernel, int threads) {
    cudaFuncAttributes attr;
    if (cudaFuncGetAttributes(&attr, kernel) != cudaSuccess || attr.numRegs <= 0) return 1;
    const int blocks = 65536 / ((attr.numRegs + 7) / 8 * 8 * threads);
    return blocks < 1 ? 1 : blocks > 8 ? 8 : blocks;
}
// Blocks per SM that shared memory leaves room for, at most `most`; the ring takes what is left.
template <class T>
TileShape best_shape(int d, int vectors, size_t extra, int most, int64_t groups, int sms, int* per_sm) {
    TileShape s{};
    if (groups < (int64_t)most * sms) most = (int)((groups + sms - 1) / sms);    // fewer blocks, longer rings
    if (most < 1) most = 1;
    for (int k = most; k >= 1; --k) {
        s = tile_shape<T>(d, vectors, extra, (size_t)227 * 1024 / k - 5 * 1024);    // 5 KB: static shared memory and the system's share
        *per_sm = k;
        if (s.stages >= (k > 1 ? 3 : 2)) return s;
    }
    s.stages = 0;
    return s;
}
template <int RT, int TR, int CT, int TC>
int launch_tile_rows(const RowsJob& a, const RowsJob* b, int64_t rows, int device, int advance, cudaStream_t st) {
    using T = Tile<RT, TR, CT, TC>;
    int per_sm, b0, b1;
    static const int most = blocks_by_registers(exact_quantize_tile_kernel<RT, TR, CT, TC>, T::kThreads);
    const TileShape shape = best_shape<T>(a.p.d, 2, (size_t)T::kRB * (T::kCols + 8), most, (rows * (b ? 2 : 1) + T::kRB - 1) / T::kRB,
                                           tq_sm_count(device), &per_sm);
    if (shape.stages == 0) return tq_fail(TQ_ERR_UNSUPPORTED, "no tile shape for d=%d", a.p.d);
    split_room(b, rows, T::kRB, (int64_t)tq_sm_count(device) * per_sm, &b0, &b1);
    TQ_GRANT_SMEM((exact_quantize_tile_kernel<RT, TR, CT, TC>), shape.bytes, device);
    TQ_CUDA_TRY(tq_launch_dependent(exact_quantize_tile_kernel<RT, TR, CT, TC>, dim3(b0 + b1), dim3(T::kThreads), shape.bytes, st, a, b ? *b : a, b0,
                                    advance, shape));
    return TQ_OK;
}
// d > 256: a block has an SM to itself, so the time is that of a block times the rounds in which they run, and a block of 4, 8 or
// 16 rows takes in proportion 68, 81 and 100 (d = 512, TurboQuantProd: 86 / 103 / 127 us; d = 768 191 / 228 / 291) or 55, 65 and 100 (d = 1,024:
// 293 / 340 / 530 us).  The fewest rows win for single rows, the most for many; the shapes' columns fit d to a quarter.  (16 rows for every
// call: one row of d = 1,024 took 573 us, d = 512 134.)
int wide_block_rows(int d, int64_t rows, int64_t sms) {
    static constexpr int kRows[3] = {4, 8, 16}, kCost[2][3] = {{68, 81, 100}, {55, 65, 100}};
    int best = 0;
    int64_t least = 0;
    for (int i = 0; i < 3; ++i) {
        const int64_t cost = ((rows + kRows[i] * sms - 1) / (kRows[i] * sms)) * kCost[d > 768][i];
        if (i == 0 || cost < least) { least = cost; best = kRows[i]; }
    }
    return best;
}

// Rows per block: one while every row can have an SM to itself (d <= 128), two while every two can, then four, 16 (8 at d = 256) while
// larger blocks would leave SMs idle, 64 or 32 from there on.  (Two against four, us: 120 keys and 120 values of d = 64 / 96 / 128
// 7.5:10.4 / 8.7:12.6 / 9.6:15.0; 296 rows of d = 128, TurboQuantProd 8.9:12.5, TurboQuantMSE 5.2:7.3; two blocks an SM of one or two rows
// each, 400 rows of d = 64, Prod, 12.9 and 11.8 against 8.8 with four.)
int launch_rows(const RowsJob& a, const RowsJob* b, int64_t rows, int device, int advance, cudaStream_t st) {
    const int d = a.p.d;
    const int64_t sms = tq_sm_count(device), total = b ? 2 * rows : rows;
    if (d <= 128 && total <= sms) return launch_few_rows<1>(a, b, rows, device, advance, st);
    if (d <= 128 && total <= sms * 2) return launch_few_rows<2>(a, b, rows, device, advance, st);
    if (d <= 128 && total <= sms * 4) return launch_few_rows<4>(a, b, rows, device, advance, st);
    // (64-row blocks on half the SMs are slower than 16-row blocks on all of them: 4,737 rows of d = 96, TurboQuantMSE, 21.5 us against 10)
    const bool many = total > sms * (d <= 96 ? 64 : d <= 128 ? 56 : 32);
    if (d <= 64) return many ? launch_tile_rows<16, 4, 8, 8>(a, b, rows, device, advance, st) : launch_tile_rows<4, 4, 32, 2>(a, b, rows, device, advance, st);
    if (d <= 96) return many ? launch_tile_rows<16, 4, 8, 12>(a, b, rows, device, advance, st) : launch_tile_rows<4, 4, 32, 3>(a, b, rows, device, advance, st);
    if (d <= 128) return many ? launch_tile_rows<8, 8, 16, 8>(a, b, rows, device, advance, st) : launch_tile_rows<4, 4, 32, 4>(a, b, rows, device, advance, st);
    if (d <= 256) {
        if (total <= sms * 8) return launch_tile_rows<2, 4, 64, 4>(a, b, rows, device, advance, st);
        return many ? launch_tile_rows<4, 8, 32, 8>(a, b, rows, device, advance, st) : launch_tile_rows<2, 8, 64, 4>(a, b, rows, device, advance, st);
    }
    const int block = wide_block_rows(d, total, sms);
#define TQ_WIDE(C4, T4, C8, T8, C16, T16)                                                                                              \
    return block == 4   ? launch_tile_rows<1, 4, C4, T4>(a, b, rows, device, advance, st)                                              \
           : block == 8 ? launch_tile_rows<1, 8, C8, T8>(a, b, rows, device, advance, st)                                              \
                        : launch_tile_rows<2, 8, C16, T16>(a, b, rows, device, advance, st)
    if (d <= 384) TQ_WIDE(128, 3, 128, 3, 128, 3);
    if (d <= 512) TQ_WIDE(256, 2, 128, 4, 128, 4);
    if (d <= 768) TQ_WIDE(256, 3, 128, 6, 128, 6);
    TQ_WIDE(256, 4, 256, 4, 128, 8);
#undef TQ_WIDE
}
RowsJob rows_job(const tq_plan* p, bool prod, const void* x, int xtype, int64_t n, uint32_t* codes, uint32_t* signs, float* rnorms,
                 float* norms, const TqRecheck* lists, unsigned long long* redo_counter, const TqRowMap* map) {
    RowsJob j{};
    j.p = p->dev; j.x = x; j.xtype = xtype; j.prod = prod ? 1 : 0; j.n = n;
    j.codes = codes; j.signs = signs; j.rnorms = rnorms; j.norms = norms;
    if (lists) j.lists = *lists;
    j.redo_counter = redo_counter;
    if (map) j.map = *map;
    return j;
}
}  // namespace

int tq_launch_exact_quantize(const tq_plan* p, bool prod, const void* x, int xtype, int64_t n, uint32_t* codes,
                             uint32_t* signs, float* rnorms, float* norms, unsigned long long* redo_counter, cudaStream_t st) {
    TqRange range("tq.quantize.exact_rows");
    if (n == 0) return TQ_OK;
    const RowsJob job = rows_job(p, prod, x, xtype, n, codes, signs, rnorms, norms, nullptr, redo_counter, nullptr);
    return launch_rows(job, nullptr, n, p->device, 0, st);
}

int tq_launch_exact_mapped(const tq_plan* p, bool prod, const void* x, int xtype, int64_t n, const TqQuantOut& out, int advance,
                           cudaStream_t st) {
    TqRange range("tq.quantize.exact_rows");
    const RowsJob job = rows_job(p, prod, x, xtype, n, out.codes, out.signs, out.rnorms, out.norms, nullptr, nullptr, &out.map);
    return launch_rows(job, nullptr, n, p->device, advance, st);
}

int tq_launch_exact_listed(const TqSecondStage* a, const TqSecondStage* b, int advance, cudaStream_t st) {
    TqRange range("tq.quantize.exact_rows");
    auto job = [](const TqSecondStage* s) {
        return rows_job(s->plan, s->prod, s->x, s->xtype, s->n, s->out.codes, s->out.signs, s->out.rnorms, s->out.norms, &s->lists,
                        s->plan->counters, &s->out.map);
    };
    // A listed pass does not know its size on the host.  About one row in 450 of a TurboQuantProd call at d = 128 is listed
    // (the coordinate re-check and the sign guard), hardly any of a TurboQuantMSE call; the blocks stride on where it is more.
    auto rows = [](const TqSecondStage* s) { return s->prod ? s->n * s->plan->dev.d / 128 / 384 + 1 : s->n / 65536 + 1; };
    const RowsJob first = job(a), second = b ? job(b) : first;
    const int64_t ra = rows(a), rb = b ? rows(b) : 0;
    return launch_rows(first, b ? &second : nullptr, ra > rb ? ra : rb, a->plan->device, advance, st);
}

template <int D>
static int launch_stage(const StageJob& a, const StageJob* b, const tq_plan* plan, int advance, cudaStream_t st) {
    const int device = plan->device;
    const int bytes = StageSmem<D>::bytes(a.rows.prod || (b && b->rows.prod) ? 2 : 1), grid = b && b->blocks > a.blocks ? b->blocks : a.blocks;
    TQ_GRANT_SMEM((second_stage_kernel<D>), bytes, device);
    TQ_CUDA_TRY(tq_launch_dependent(second_stage_kernel<D>, dim3(grid), dim3(kStageThreads), (size_t)bytes, st, a, b ? *b : a, b ? 2 : 1, advance,
                                    StageWait{plan->wait_kcycles, plan->status_dev}));
    return TQ_OK;
}

int tq_launch_second_stage(const TqSecondStage* a, const TqSecondStage* b, int advance, cudaStream_t st) {
    TqRange range("tq.quantize.second_stage");
    auto job = [](const TqSecondStage* s) {
        StageJob j;
        j.rows = rows_job(s->plan, s->prod, s->x, s->xtype, s->n, s->out.codes, s->out.signs, s->out.rnorms, s->out.norms, &s->lists,
                          s->plan->counters, &s->out.map);
        j.blocks = tq_tensor_quantize_blocks(s->plan, s->n);
        return j;
    };
    const StageJob first = job(a), second = b ? job(b) : first;
    switch (a->plan->dev.d) {
        case 64: return launch_stage<64>(first, b ? &second : nullptr, a->plan, advance, st);
        case 96: return launch_stage<96>(first, b ? &second : nullptr, a->plan, advance, st);
        case 128: return launch_stage<128>(first, b ? &second : nullptr, a->plan, advance, st);
    }
    return tq_fail(TQ_ERR_UNSUPPORTED, "the second stage in one launch is written for d = 64, 96 and 128");
}

// One step of a cache: the keys of `kp` (TurboQuantProd), the values of `vp` (TurboQuantMSE), or both (either plan may be
// null), in one launch.
int tq_launch_append(const tq_plan* kp, const void* kx, uint32_t* kcodes, uint32_t* ksigns, float* krnorms, float* knorms,
                     const tq_plan* vp, const void* vx, uint32_t* vcodes, float* vnorms, int xtype, int64_t rows,
                     const TqRowMap& map, int advance, cudaStream_t st) {
    TqRange range("tq.append");
    RowsJob k{}, v{};
    if (kp) k = rows_job(kp, true, kx, xtype, rows, kcodes, ksigns, krnorms, knorms, nullptr, nullptr, &map);
    if (vp) v = rows_job(vp, false, vx, xtype, rows, vcodes, nullptr, nullptr, vnorms, nullptr, nullptr, &map);
    return launch_rows(kp ? k : v, kp && vp ? &v : nullptr, rows, (kp ? kp : vp)->device, advance, st);
}

namespace {
template <bool PROD, int RT, int TR, int CT, int TC>
int launch_tile_dequant(const tq_plan* p, const uint32_t* codes, const uint32_t* signs, const float* rnorms, const float* norms,
                        int64_t n, float* out, cudaStream_t st) {
    using T = Tile<RT, TR, CT, TC>;
    int per_sm;
    static const int most = blocks_by_registers(exact_dequantize_tile_kernel<PROD, RT, TR, CT, TC>, T::kThreads);
    const TileShape shape = best_shape<T>(p->dev.d, PROD ? 2 : 1, 0, most, (n + T::kRB - 1) / T::kRB, tq_sm_count(p->device), &per_sm);
    if (shape.stages == 0) return tq_fail(TQ_ERR_UNSUPPORTED, "no tile shape for d=%d", p->dev.d);
    const int grid = job_blocks(n, T::kRB, (int64_t)tq_sm_count(p->device) * per_sm);
    TQ_GRANT_SMEM((exact_dequantize_tile_kernel<PROD, RT, TR, CT, TC>), shape.bytes, p->device);
    exact_dequantize_tile_kernel<PROD, RT, TR, CT, TC><<<grid, T::kThreads, shape.bytes, st>>>(p->dev, codes, signs, rnorms, norms, n, out, shape);
    tq_count_launch();
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}
template <bool PROD>
int launch_dequant_for(const tq_plan* p, const uint32_t* codes, const uint32_t* signs, const float* rnorms, const float* norms,
                       int64_t n, float* out, cudaStream_t st) {
    const int d = p->dev.d;
    const int64_t sms = tq_sm_count(p->device);
    // (64-row blocks on half the SMs are slower than 16-row blocks on all of them; d = 128, 8,000 rows: 20.6 / 24.3 us)
    const bool many = n > sms * (d <= 96 ? 64 : d <= 128 ? 48 : 32);
#define TQ_DQ(...) return launch_tile_dequant<PROD, __VA_ARGS__>(p, codes, signs, rnorms, norms, n, out, st)
    if (d <= 64) { if (many) TQ_DQ(16, 4, 8, 8); TQ_DQ(4, 4, 32, 2); }
    if (d <= 96) { if (many) TQ_DQ(16, 4, 8, 12); TQ_DQ(4, 4, 32, 3); }
    if (d <= 128) { if (many) TQ_DQ(16, 4, 16, 8); TQ_DQ(4, 4, 32, 4); }
    if (d <= 256) {
        // blocks of 8 rows run two to an SM: where that leaves a last round of few blocks, 16 rows are faster (TurboQuantProd, d = 256:
        // 2,000 rows 29 / 25 us, 3,000 rows 43 / 46, 4,736 rows 53 / 46)
        if (many) TQ_DQ(8, 4, 32, 8);
        if (n > 24 * sms || (n > 8 * sms && n <= 16 * sms)) TQ_DQ(4, 4, 64, 4);
        TQ_DQ(2, 4, 64, 4);
    }
    const int block = wide_block_rows(d, n, sms);
#define TQ_WIDE(C4, T4, C8, T8, C16, T16)      \
    if (block == 4) TQ_DQ(1, 4, C4, T4);       \
    if (block == 8) TQ_DQ(1, 8, C8, T8);       \
    TQ_DQ(2, 8, C16, T16)
    if (d <= 384) { TQ_WIDE(128, 3, 128, 3, 128, 3); }
    if (d <= 512) { TQ_WIDE(256, 2, 128, 4, 128, 4); }
    if (d <= 768) { TQ_WIDE(256, 3, 256, 3, 128, 6); }
    TQ_WIDE(256, 4, 256, 4, 128, 8);
#undef TQ_WIDE
#undef TQ_DQ
}
}  // namespace

int tq_launch_exact_dequantize(const tq_plan* p, bool prod, const uint32_t* codes, const uint32_t* signs,
                               const float* rnorms, const float* norms, int64_t n, float* out,
                               cudaStream_t st) {
    TqRange range("tq.dequantize.exact");
    if (n == 0) return TQ_OK;
    return prod ? launch_dequant_for<true>(p, codes, signs, rnorms, norms, n, out, st)
                : launch_dequant_for<false>(p, codes, signs, rnorms, norms, n, out, st);
}

int tq_launch_exact_pairwise(const tq_plan* p, const float* q, const uint32_t* codes, const uint32_t* signs,
                             const float* rnorms, const float* norms, int64_t n, float* scores,
                             cudaStream_t st) {
    TqRange range("tq.score.pairwise.exact");
    if (n == 0) return TQ_OK;
    const int dp = (p->dev.d + 31) & ~31;
    const size_t sm = (size_t)kWarps * 3 * dp * sizeof(float);
    TQ_GRANT_SMEM((exact_pairwise_score_kernel), sm, p->device);
    exact_pairwise_score_kernel<<<grid_for(n, kWarps), kWarps * 32, sm, st>>>(p->dev, q, codes, signs, rnorms, norms, n, scores); tq_count_launch();
    TQ_CUDA_TRY(cudaGetLastError());
    return TQ_OK;
}
