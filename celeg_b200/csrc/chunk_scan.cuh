// What the chunked scans of matrix states share (decayed_scan.cu, recurrent_scan.cu). A span is cut into chunks of 64 tokens,
// counted from its first token in the step; per head, with S [dim, vdim], numbers weight(i, j) and factor(i) of the chunk's
// tokens, and w_j the weight with which token j's k v^T is left in the state after the chunk,
//
//   o_i = sum_(j<=i) weight(i, j) (q_i . k_j) v_j + factor(i) S_0^T q_i          S_n = f S_0 + sum_j w_j k_j v_j^T
//
//   walk      a block a (span, head, tile of S) goes through the span's chunks in order with its tile of S in registers: it
//             leaves S_0 of every chunk in `states`, and the span's last state in its slot. A chunk's tokens are loaded while
//             the chunk before them is multiplied; their weights are made a chunk ahead too.
//   sums, carry   instead of the walk, where few heads and spans leave it too few blocks: a block a (chunk, head, 64 x 64 of S)
//             makes sum_j w_j k_j v_j^T, all chunks side by side, and a thread a few elements of S takes them in order.
//   read-outs a block a (chunk, heads of a group): the products q.k of the chunk stay in the registers of the warp that owns
//             16 of its tokens, and are the A operand of their product with v as they lie.
//
// All products are on mma.sync m16n8k16 with a float32 number as three bfloat16 ones, x = hi + mid + lo, each rounded from
// what is left: the six products above 2^-24 of the largest (hi hi, hi mid, mid hi, mid mid, hi lo, lo hi) are summed on the
// tensor cores from zero, over 16 products at a time, and added in float32 in registers, because a tensor-core sum is cut off
// towards zero at every link of a chain: read-outs and states are nearer to 64 bits than float32 multiplications and
// additions in order (1.1e-7 against 2.4e-7 over 2,000 tokens of 16 heads of 64 x 128). A number is split once a block, on
// its way into shared memory; split at every use by the warps that load it (two tf32 numbers, m16n8k8), a fragment cost more
// instructions than its products.
//
// Numbers that are not finite. An infinite operand gives NaN (its mid is inf - inf). A token's NaN belongs to it and to the
// tokens behind it, but a weight of zero times a NaN is a NaN, and the tokens before it meet it under a weight of zero in the
// products with v. So v's tiles take a zero in its place and note the column's first such token (BadTokens), and the read-outs
// from that token on are NaN; the same for the right sides of the delta rules' systems. It costs the cases of 2,048 tokens
// between nothing and 1 %, the generalised delta rule 2 % (359 to 365 us with the projections). (A decay a channel that is NaN
// reaches the tokens of its block of eight: decayed_scan.cu.)
#pragma once

#include <cfloat>

#include "mma_tiles.cuh"

namespace celeg_b200 {

constexpr int kChunk = 64;

enum ChunkMode : int {
    kChunkScalar = 0,      // a decay a token and head, a step that scales what is written (Mamba-2)
    kChunkChannel = 1,     // a decay a token and key channel, taken into q and k beforehand (gated linear attention)
    kChunkConstant = 2,    // a decay a head (retention)
    kChunkStable = 3,      // exponential gates in range of a running maximum, with a normaliser (mLSTM)
    kChunkPair = 4,        // read-outs alone: as channel, with a second set of values and products, at most 64 columns and
                           // key channels (generalised delta rule)
};

struct ChunkArgs {
    const float* q; int q_stride; const float* k; int k_stride;        // head (or group) h at h * dim
    const float* v; int v_stride;
    const float2* cum; const float* dt;      // scalar: [tokens, heads]: sums of the decays' logarithms, steps (null: ones)
    const float* total;                      // channel: [chunks, heads * dim], the chunk's product of decays
    const float* products;                   // channel: [chunks, heads, 64, 64], zero above the diagonal
    const float* products_b; const float* v_b; int v_b_stride;         // pair: the same for other values beside v
    const float* direct;                     // scalar: [heads], the values' share of the read-out, or null
    const float* decay; float q_scale;       // constant: [heads], and the keys' factor; stable, scalar: the queries' factor
    const float2* gates;                     // stable: [tokens, 3, heads]: forget sum F, i - F, the largest i - F so far
    double* peaks;                           // stable: [chunks, heads], the running maximum before the chunk
    float* norms;                            // stable: [chunks, heads, dim], the normaliser before the chunk
    const int* chunk_begin; int pieces;      // first tokens of runs of `pieces` chunks; a span's runs are span_first[s] ..
    const int* span_first; int spans;
    float* state; long long slot_stride; const int* span_slot;         // the spans' states (stable: S, normalisers, maxima)
    float* states;                           // [chunks, heads, dim, vdim]: the state before the chunk
    float* out;                              // [tokens, heads * vdim]
    int heads, groups, dim, vdim;
};

// what a chunk's tokens are: a run of `pieces` chunks begins at chunk_begin[run]
__device__ __forceinline__ void chunk_tokens_of(const ChunkArgs& p, int chunk, int& begin, int& count) {
    const int run = chunk / p.pieces;
    begin = p.chunk_begin[run] + (chunk - run * p.pieces) * kChunk;
    count = min(kChunk, p.chunk_begin[run + 1] - begin);
}

// A plan by the threads of one block: spans cut into runs of `length` tokens; runs beyond the last (and beyond max_runs) are empty.
__device__ __forceinline__ void plan_runs(const int* span_begin, int spans, int length, int max_runs, int* run_begin, int* span_first) {
    int n = 0;
    for (int s = 0; s < spans; ++s) {
        const int begin = span_begin[s], end = span_begin[s + 1];
        const int runs = min(max(end - begin + length - 1, 0) / length, max_runs - n);
        if (threadIdx.x == 0) span_first[s] = n;
        for (int i = threadIdx.x; i < runs; i += blockDim.x) run_begin[n + i] = begin + i * length;
        n += runs;
    }
    if (threadIdx.x == 0) span_first[spans] = n;
    for (int i = n + threadIdx.x; i <= max_runs; i += blockDim.x) run_begin[i] = span_begin[spans];
}

// exp of the difference of two numbers that are two floats each
__device__ __forceinline__ float exp_between(const float2& later, const float2& earlier) {
    return expf((later.x - earlier.x) + (later.y - earlier.y));
}
__device__ __forceinline__ float2 two_floats(double x) {
    const float high = (float)x;
    return make_float2(high, (float)(x - (double)high));
}
__device__ __forceinline__ double one_double(const float2& x) { return (double)x.x + (double)x.y; }

// ------------------------------------------------------------------------------------------------------- tensor cores
// two neighbouring numbers as three bfloat16 pairs
__device__ __forceinline__ void split_pair(float x, float y, unsigned& hi, unsigned& mid, unsigned& lo) {
    hi = pack_bf16(x, y);
    x -= __uint_as_float(hi << 16);
    y -= __uint_as_float(hi & 0xffff0000u);
    mid = pack_bf16(x, y);
    lo = pack_bf16(x - __uint_as_float(mid << 16), y - __uint_as_float(mid & 0xffff0000u));
}
__device__ __forceinline__ void mma_step(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// acc[n] += a b[n] over 16 products, the smallest first; the N chains of six take turns
template <int N>
__device__ __forceinline__ void mma_split(float (*acc)[4], const unsigned (&a)[3][4], const unsigned (*b)[3][2]) {
    constexpr int kA[6] = {2, 0, 1, 1, 0, 0}, kB[6] = {0, 2, 1, 0, 1, 0};
    float d[N][4] = {};
#pragma unroll
    for (int i = 0; i < 6; ++i)
#pragma unroll
        for (int n = 0; n < N; ++n) mma_step(d[n], a[kA[i]], b[n][kB[i]]);
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[n][r] += d[n][r];
}

// ----------------------------------------------------------------------------------------------- tiles in shared memory
// Three planes (hi, mid, lo) of ROWS x COLUMNS bfloat16 numbers; the 16-byte pieces of a row are permuted so that eight rows'
// pieces of one column lie in eight different bank groups (COLUMNS 32: two rows fill the 128 bytes of all banks; 16: four).
template <int ROWS, int COLUMNS>
struct SplitTile {
    static constexpr int kPlane = ROWS * COLUMNS;
    static constexpr int kElements = 3 * kPlane;
    static __device__ __forceinline__ int at(int row, int piece) {
        return row * COLUMNS + ((piece ^ (COLUMNS == 16 ? (row >> 2) & 1 : COLUMNS == 32 ? (row >> 1) & 3 : row & 7)) << 3);
    }
};

// rows that begin at multiples of four floats (every offset in them is one of `sizes`, a sum of multiples where those are)
__device__ __forceinline__ bool by_fours(const float* p, long long stride, int sizes) {
    return ((((unsigned long long)p >> 2) | (unsigned long long)stride | (unsigned)sizes) & 3) == 0;
}

// Of a chunk's 64 columns of values the first token with a number that is not finite, in shared memory; every use lies between
// barriers that are there for the tile itself.
struct BadTokens {
    int first[64];
    int any;
    __device__ __forceinline__ void clear() {                // (65 threads at least)
        if (threadIdx.x < 64) first[threadIdx.x] = kChunk;
        if (threadIdx.x == 64) any = 0;
    }
    __device__ __forceinline__ void note(int column, int token) {
        atomicMin(&first[column], token);
        any = 1;
    }
    // a warp's results of tokens t, t + 8 and columns c + 8 n, + 1: NaN from `behind` tokens behind the first bad one on
    __device__ __forceinline__ void mark(float (&acc)[8][4], int t, int c, int behind = 0) const {
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (t + 8 * (r >> 1) >= first[c + 8 * n + (r & 1)] + behind) acc[n][r] = NAN;
    }
};

// A thread's share of a ROWS x COLUMNS tile of floats: pieces of eight neighbours, THREADS apart. load(): zeros from row
// `real_rows` and column `real_columns` on; store(): times scale(row), split, into shared memory.
template <int ROWS, int COLUMNS, int THREADS>
struct TileShare {
    static constexpr int kPieces = COLUMNS / 8, kUnits = ROWS * kPieces / THREADS;
    static_assert(ROWS * kPieces % THREADS == 0 && THREADS % kPieces == 0, "");
    float x[kUnits][8];
    __device__ __forceinline__ void load(const float* src, long long stride, int real_rows, int real_columns, bool four) {
        const int c = (threadIdx.x % kPieces) * 8;
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
            const int r = threadIdx.x / kPieces + u * (THREADS / kPieces);
            const float* from = src + r * stride + c;
            if (four) {
                const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                const float4 p = r < real_rows && c < real_columns ? *reinterpret_cast<const float4*>(from) : zero;
                const float4 q = r < real_rows && c + 4 < real_columns ? *reinterpret_cast<const float4*>(from + 4) : zero;
                x[u][0] = p.x; x[u][1] = p.y; x[u][2] = p.z; x[u][3] = p.w;
                x[u][4] = q.x; x[u][5] = q.y; x[u][6] = q.z; x[u][7] = q.w;
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) x[u][j] = r < real_rows && c + j < real_columns ? from[j] : 0.0f;
            }
        }
    }
    // T: the tile it is part of, from the row's piece `piece` on. False where a number is not finite.
    template <typename T, typename Scale>
    __device__ __forceinline__ bool store(__nv_bfloat16* tile, int piece, Scale scale) const {
        unsigned none = 0;                                   // (two zeros, NaN as soon as a number is infinite or NaN)
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
            const int r = threadIdx.x / kPieces + u * (THREADS / kPieces);
            const float f = scale(r);
            unsigned plane[3][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                split_pair(x[u][2 * j] * f, x[u][2 * j + 1] * f, plane[0][j], plane[1][j], plane[2][j]);
                asm("fma.rn.bf16x2 %0, %1, %2, %0;\n" : "+r"(none) : "r"(plane[0][j]), "r"(0));
            }
            __nv_bfloat16* to = tile + T::at(r, piece + threadIdx.x % kPieces);
#pragma unroll
            for (int n = 0; n < 3; ++n)
                *reinterpret_cast<uint4*>(to + n * T::kPlane) = make_uint4(plane[n][0], plane[n][1], plane[n][2], plane[n][3]);
        }
        return (none & 0x7fff7fffu) == 0;
    }
    // Where store() says so: use(row, column, cell of the first plane) of the share's numbers that are not finite
    template <typename T, typename Use>
    static __device__ __forceinline__ void each_bad(__nv_bfloat16* tile, int piece, Use use) {
#pragma unroll 1
        for (int x = 0; x < 8 * kUnits; ++x) {
            const int r = threadIdx.x / kPieces + (x >> 3) * (THREADS / kPieces), at = threadIdx.x % kPieces;
            __nv_bfloat16* cell = tile + T::at(r, piece + at) + (x & 7);
            if (!(fabsf(__bfloat162float(*cell)) <= FLT_MAX)) use(r, at * 8 + (x & 7), cell);
        }
    }
    // the same: they give way to zeros in the tile and are noted. The share is tokens from `token` on, columns from `column`.
    template <typename T>
    static __device__ __forceinline__ void take_out(__nv_bfloat16* tile, int piece, BadTokens& bad, int token, int column) {
        each_bad<T>(tile, piece, [&](int r, int c, __nv_bfloat16* cell) {
            bad.note(column + c, token + r);
            for (int n = 0; n < 3; ++n) cell[n * T::kPlane] = __float2bfloat16_rn(0.0f);
        });
    }
};
// The same share by way of shared memory, where a thread finds its own pieces again: copied asynchronously, read back later.
template <int ROWS, int COLUMNS, int THREADS>
__device__ __forceinline__ void share_copy(float* raw, const float* src, long long stride, int real_rows, int real_columns,
                                           bool four) {
    using Share = TileShare<ROWS, COLUMNS, THREADS>;
    const int c = (threadIdx.x % Share::kPieces) * 8;
#pragma unroll
    for (int u = 0; u < Share::kUnits; ++u) {
        const int r = threadIdx.x / Share::kPieces + u * (THREADS / Share::kPieces);
        const float* from = src + r * stride + c;
        const unsigned to = (unsigned)__cvta_generic_to_shared(raw + (u * THREADS + threadIdx.x) * 8);
        if (four) {
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                const int bytes = r < real_rows && c + j < real_columns ? 16 : 0;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to + 4 * j), "l"(bytes ? from + j : src), "r"(bytes) : "memory");
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int bytes = r < real_rows && c + j < real_columns ? 4 : 0;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(to + 4 * j), "l"(bytes ? from + j : src), "r"(bytes) : "memory");
            }
        }
    }
}
template <int ROWS, int COLUMNS, int THREADS>
__device__ __forceinline__ void share_read(TileShare<ROWS, COLUMNS, THREADS>& share, const float* raw) {
#pragma unroll
    for (int u = 0; u < TileShare<ROWS, COLUMNS, THREADS>::kUnits; ++u)
#pragma unroll
        for (int j = 0; j < 8; j += 4) {
            const float4 p = *reinterpret_cast<const float4*>(raw + (u * THREADS + threadIdx.x) * 8 + j);
            share.x[u][j] = p.x; share.x[u][j + 1] = p.y; share.x[u][j + 2] = p.z; share.x[u][j + 3] = p.w;
        }
}
struct Unscaled { __device__ __forceinline__ float operator()(int) const { return 1.0f; } };

// The 16 x 16 A operand of rows m0.. and depth k0.. of a tile that lies [m][k], or, transposed, [k][m]
template <typename T>
__device__ __forceinline__ void load_a(unsigned (&a)[3][4], const __nv_bfloat16* tile, int m0, int k0) {
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16* from = tile + T::at(m0 + (lane & 15), (k0 >> 3) + (lane >> 4));
#pragma unroll
    for (int n = 0; n < 3; ++n) ldmatrix_x4(a[n], from + n * T::kPlane);
}
template <typename T>
__device__ __forceinline__ void load_a_transposed(unsigned (&a)[3][4], const __nv_bfloat16* tile, int m0, int k0) {
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16* from = tile + T::at(k0 + (lane & 7) + ((lane >> 4) << 3), (m0 >> 3) + ((lane >> 3) & 1));
#pragma unroll
    for (int n = 0; n < 3; ++n) ldmatrix_x4_trans(a[n], from + n * T::kPlane);
}
// The B operands, depth k0 .. k0 + 15, of columns n0 .. n0 + 7 and n0 + 8 .. n0 + 15 of a tile that lies [n][k], or [k][n]
template <typename T>
__device__ __forceinline__ void load_b(unsigned (*b)[3][2], const __nv_bfloat16* tile, int n0, int k0) {
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16* from = tile + T::at(n0 + (lane & 7) + ((lane >> 4) << 3), (k0 >> 3) + ((lane >> 3) & 1));
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        unsigned r[4];
        ldmatrix_x4(r, from + n * T::kPlane);
        b[0][n][0] = r[0]; b[0][n][1] = r[1]; b[1][n][0] = r[2]; b[1][n][1] = r[3];
    }
}
template <typename T>
__device__ __forceinline__ void load_b_transposed(unsigned (*b)[3][2], const __nv_bfloat16* tile, int n0, int k0) {
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16* from = tile + T::at(k0 + (lane & 15), (n0 >> 3) + (lane >> 4));
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        unsigned r[4];
        ldmatrix_x4_trans(r, from + n * T::kPlane);
        b[0][n][0] = r[0]; b[0][n][1] = r[1]; b[1][n][0] = r[2]; b[1][n][1] = r[3];
    }
}

// -------------------------------------------------------------------------------------------------------------- walk
constexpr int kWalkThreads = 256;
constexpr int kWalkRows = 64;                                // key channels of S a block
template <int COLUMNS> constexpr int walk_buffer() {
    return SplitTile<kChunk, kWalkRows>::kElements + SplitTile<kChunk, COLUMNS>::kElements;
}

// COLUMNS of S a block: 32, two blocks an SM, or 64 and one (walk_columns() below says which and why).
template <int MODE, int COLUMNS>
__global__ void __launch_bounds__(kWalkThreads, 64 / COLUMNS) chunk_walk_kernel(const ChunkArgs p) {
    constexpr int kWalkColumns = COLUMNS, kWalkBuffer = walk_buffer<COLUMNS>();
    constexpr int kTiles = COLUMNS / 16;                     // tiles of eight columns a warp: four warps along the key
    using KTile = SplitTile<kChunk, kWalkRows>;              // channels, two along the columns
    using VTile = SplitTile<kChunk, kWalkColumns>;
    extern __shared__ __align__(128) __nv_bfloat16 tiles[];  // two buffers of a chunk's k and v
    __shared__ float w_s[2][kChunk];                         // weights of a chunk's tokens
    __shared__ float f_s[2];
    __shared__ float ladder[kChunk + 1];                     // constant: powers of the decay
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
    const int span = blockIdx.z, head = blockIdx.y;
    const int dim = p.dim, vdim = p.vdim;
    const int v_tiles = (vdim + kWalkColumns - 1) / kWalkColumns;
    const int e0 = (blockIdx.x / v_tiles) * kWalkRows, c0 = (blockIdx.x % v_tiles) * kWalkColumns;
    const int first = p.span_first[span], last = p.span_first[span + 1];
    if (first >= last) return;
    const int t_begin = p.chunk_begin[first], t_end = p.chunk_begin[last];
    const int chunks = (t_end - t_begin + kChunk - 1) / kChunk;
    const int qk_head = MODE == kChunkScalar ? head / (p.heads / p.groups) : head;
    float* slot = p.state + (long long)p.span_slot[span] * p.slot_stride;
    const float* k_src = p.k + (size_t)qk_head * dim + e0;
    const float* v_src = p.v + (size_t)head * vdim + c0;
    const bool k_four = by_fours(p.k, p.k_stride, dim), v_four = by_fours(p.v, p.v_stride, vdim);
    TileShare<kChunk, kWalkRows, kWalkThreads> k_share;
    TileShare<kChunk, kWalkColumns, kWalkThreads> v_share;
    auto load = [&](int i) {
        if (i >= chunks) return;
        const int begin = t_begin + i * kChunk, count = min(kChunk, t_end - begin);
        k_share.load(k_src + (size_t)begin * p.k_stride, p.k_stride, count, dim - e0, k_four);
        v_share.load(v_src + (size_t)begin * p.v_stride, p.v_stride, count, vdim - c0, v_four);
    };
    load(0);

    // the weights of chunk i: what a token's thread reads for them, and what it makes of that
    double peak = 0.0;                                       // stable: the running maximum after the chunks so far
    if (MODE == kChunkStable) peak = slot[(size_t)p.heads * dim * (vdim + 1) + head];
    if (MODE == kChunkConstant) {
        for (int n = tid; n <= kChunk; n += kWalkThreads) ladder[n] = powf(p.decay[head], (float)n);
        __syncthreads();
    }
    float2 own = make_float2(0.0f, 0.0f), end = own, forget = own;
    float step = 0.0f;
    auto ask = [&](int i) {
        if (MODE == kChunkChannel || MODE == kChunkConstant || i >= chunks || tid >= kChunk) return;
        const int begin = t_begin + i * kChunk, count = min(kChunk, t_end - begin);
        const size_t t = begin + min(tid, count - 1), e = begin + count - 1;
        if (MODE == kChunkScalar) {
            own = p.cum[t * p.heads + head];
            end = p.cum[e * p.heads + head];
            step = p.dt[t * p.heads + head];
        } else {
            own = p.gates[(t * 3 + 1) * p.heads + head];
            end = p.gates[(e * 3 + 2) * p.heads + head];
            forget = p.gates[(e * 3) * p.heads + head];
        }
    };
    auto make = [&](int i) {
        if (MODE == kChunkChannel || i >= chunks || tid >= kChunk) return;
        const int count = min(kChunk, t_end - (t_begin + i * kChunk));
        float w, f;
        if (MODE == kChunkScalar) {
            w = step * exp_between(end, own);
            f = expf(end.x);
        } else if (MODE == kChunkConstant) {
            w = p.q_scale * ladder[max(count - 1 - tid, 0)];
            f = ladder[count];
        } else {
            const double high = fmax(peak, one_double(end));
            if (tid == 0 && blockIdx.x == 0) p.peaks[(size_t)(first * p.pieces + i) * p.heads + head] = peak;
            f = expf((float)(peak - high));
            w = exp_between(own, two_floats(high));
            peak = one_double(forget) + high;
        }
        w_s[i & 1][tid] = tid < count ? w : 0.0f;
        if (tid == 0) f_s[i & 1] = f;
    };
    ask(0);
    make(0);
    ask(1);

    // this warp's part of S: rows er + g, er + g + 8; columns cc + 8 n + 2 tig, + 1
    const int along = warp & 3, across = warp >> 2;
    const int er = e0 + 16 * along, cc = c0 + 8 * kTiles * across;
    float* s_head = slot + (size_t)head * dim * vdim;
    const bool pairs = (vdim & 1) == 0 && (p.slot_stride & 1) == 0 && ((uintptr_t)p.state & 7) == 0;
    float s[kTiles][4];
    auto each = [&](auto&& use) {                            // (row, column, the two numbers there)
#pragma unroll
        for (int n = 0; n < kTiles; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) use(er + g + 8 * h, cc + 8 * n + 2 * tig, s[n][2 * h], s[n][2 * h + 1]);
    };
    each([&](int r, int c, float& a, float& b) {
        const float* src = s_head + (size_t)r * vdim + c;
        a = r < dim && c < vdim ? src[0] : 0.0f;
        b = r < dim && c + 1 < vdim ? src[1] : 0.0f;
    });
    auto store = [&](float* dst, bool two) {
        each([&](int r, int c, float& a, float& b) {
            if (r >= dim || c >= vdim) return;
            float* cell = dst + (size_t)r * vdim + c;
            if (two) {
                *reinterpret_cast<float2*>(cell) = make_float2(a, b);
                return;
            }
            cell[0] = a;
            if (c + 1 < vdim) cell[1] = b;
        });
    };
    // stable: the first columns' warps keep the normaliser of their rows too, the sum of the weighted keys: a column of ones
    const bool keeps_norm = MODE == kChunkStable && c0 == 0 && across == 0;
    float* n_cell = slot + (size_t)p.heads * dim * vdim + (size_t)head * dim + er + g;
    float norm[2] = {0.0f, 0.0f}, keep[2] = {1.0f, 1.0f};    // (keep, channel: the two rows' decays over the chunk)
    if (keeps_norm) {
#pragma unroll
        for (int h = 0; h < 2; ++h) norm[h] = er + g + 8 * h < dim ? n_cell[8 * h] : 0.0f;
    }
    __syncthreads();
    for (int i = 0; i < chunks; ++i) {
        const size_t at = ((size_t)(first * p.pieces + i) * p.heads + head) * dim;      // (the head's rows in this chunk)
        __nv_bfloat16* k_t = tiles + (i & 1) * kWalkBuffer;
        __nv_bfloat16* v_t = k_t + KTile::kElements;
        make(i + 1);
        ask(i + 2);
        if (MODE == kChunkChannel) k_share.template store<KTile>(k_t, 0, Unscaled());
        else k_share.template store<KTile>(k_t, 0, [&](int r) { return w_s[i & 1][r]; });
        v_share.template store<VTile>(v_t, 0, Unscaled());
        load(i + 1);
        if (MODE == kChunkChannel) {
#pragma unroll
            for (int h = 0; h < 2; ++h) keep[h] = er + g + 8 * h < dim ? p.total[at + er + g + 8 * h] : 0.0f;
        } else {
            keep[0] = keep[1] = f_s[i & 1];
        }
        store(p.states + at * vdim, (vdim & 1) == 0);
        if (keeps_norm && tig == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
                if (er + g + 8 * h < dim) p.norms[at + er + g + 8 * h] = norm[h];
        }
        __syncthreads();                                     // the chunk's tiles and the next one's weights are there
        float sum[kTiles][4] = {}, ones[4] = {};
#pragma unroll
        for (int t = 0; t < kChunk; t += 32) {               // two depths of 16 at a time: their chains take turns
            unsigned a[2][3][4], b[2][kTiles][3][2];
            float d[2][kTiles][4] = {}, n_d[2][4] = {};
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                load_a_transposed<KTile>(a[u], k_t, 16 * along, t + 16 * u);
#pragma unroll
                for (int n = 0; n < kTiles; n += 2) load_b_transposed<VTile>(b[u] + n, v_t, 8 * (kTiles * across + n), t + 16 * u);
            }
            constexpr int kA[6] = {2, 0, 1, 1, 0, 0}, kB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
            for (int i6 = 0; i6 < 6; ++i6)
#pragma unroll
                for (int u = 0; u < 2; ++u)
#pragma unroll
                    for (int n = 0; n < kTiles; ++n) mma_step(d[u][n], a[u][kA[i6]], b[u][n][kB[i6]]);
            if (keeps_norm) {
                const unsigned one[2] = {0x3f803f80u, 0x3f803f80u};
#pragma unroll
                for (int plane = 2; plane >= 0; --plane)
#pragma unroll
                    for (int u = 0; u < 2; ++u) mma_step(n_d[u], a[u][plane], one);
            }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
#pragma unroll
                for (int n = 0; n < kTiles; ++n)
#pragma unroll
                    for (int r = 0; r < 4; ++r) sum[n][r] += d[u][n][r];
                ones[0] += n_d[u][0];
                ones[2] += n_d[u][2];
            }
        }
#pragma unroll
        for (int n = 0; n < kTiles; ++n)
#pragma unroll
            for (int r = 0; r < 4; ++r) s[n][r] = fmaf(keep[r >> 1], s[n][r], sum[n][r]);
        norm[0] = fmaf(keep[0], norm[0], ones[0]);
        norm[1] = fmaf(keep[1], norm[1], ones[2]);
    }
    store(s_head, pairs);
    if (keeps_norm && tig == 0) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (er + g + 8 * h < dim) n_cell[8 * h] = norm[h];
    }
    // (the running maximum, which every block of the head has read, is written by the read-outs)
}

// --------------------------------------------------------------------------------------------------------- sums, carry
constexpr int kSumThreads = 128;
constexpr int kSumElements = 2 * SplitTile<kChunk, 64>::kElements;

// states[chunk, head] = sum_j w_j k_j v_j^T (stable: in terms of the chunk's own largest i - F, and norms with it)
template <int MODE>
__global__ void __launch_bounds__(kSumThreads, 4) chunk_sum_kernel(const ChunkArgs p) {
    using Tile = SplitTile<kChunk, 64>;
    extern __shared__ __align__(128) __nv_bfloat16 tiles[];
    __shared__ float w_s[kChunk];
    chain_release();
    chain_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
    const int chunk = blockIdx.z, head = blockIdx.y, dim = p.dim, vdim = p.vdim;
    int begin, count;
    chunk_tokens_of(p, chunk, begin, count);
    if (count <= 0) return;
    const int v_tiles = (vdim + 63) / 64, e0 = (blockIdx.x / v_tiles) * 64, c0 = (blockIdx.x % v_tiles) * 64;
    const int qk_head = MODE == kChunkScalar ? head / (p.heads / p.groups) : head;
    TileShare<kChunk, 64, kSumThreads> share;
    share.load(p.v + (size_t)begin * p.v_stride + (size_t)head * vdim + c0, p.v_stride, count, vdim - c0, by_fours(p.v, p.v_stride, vdim));
    if (MODE != kChunkChannel && tid < kChunk) {
        const size_t t = begin + min(tid, count - 1), e = begin + count - 1;
        float w = 0.0f;
        if (MODE == kChunkScalar) w = p.dt[t * p.heads + head] * exp_between(p.cum[e * p.heads + head], p.cum[t * p.heads + head]);
        if (MODE == kChunkConstant) w = p.q_scale * powf(p.decay[head], (float)max(count - 1 - tid, 0));
        if (MODE == kChunkStable) w = exp_between(p.gates[(t * 3 + 1) * p.heads + head], p.gates[(e * 3 + 2) * p.heads + head]);
        w_s[tid] = tid < count ? w : 0.0f;
    }
    share.template store<Tile>(tiles + Tile::kElements, 0, Unscaled());
    share.load(p.k + (size_t)begin * p.k_stride + (size_t)qk_head * dim + e0, p.k_stride, count, dim - e0, by_fours(p.k, p.k_stride, dim));
    __syncthreads();
    if (MODE == kChunkChannel) share.template store<Tile>(tiles, 0, Unscaled());
    else share.template store<Tile>(tiles, 0, [&](int r) { return w_s[r]; });
    __syncthreads();
    float sum[8][4] = {}, ones[4] = {};
    const bool sums_norm = MODE == kChunkStable && c0 == 0;
#pragma unroll
    for (int t = 0; t < kChunk; t += 16) {
        unsigned a[3][4];
        load_a_transposed<Tile>(a, tiles, 16 * warp, t);
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
            unsigned b[4][3][2];
            load_b_transposed<Tile>(b, tiles + Tile::kElements, 16 * n, t);
            load_b_transposed<Tile>(b + 2, tiles + Tile::kElements, 16 * n + 16, t);
            mma_split<4>(sum + 2 * n, a, b);
        }
        if (sums_norm) {                                     // (a column of ones)
            const unsigned one[2] = {0x3f803f80u, 0x3f803f80u};
            float d[4] = {};
#pragma unroll
            for (int n = 2; n >= 0; --n) mma_step(d, a[n], one);
            ones[0] += d[0];
            ones[2] += d[2];
        }
    }
    const size_t at = ((size_t)chunk * p.heads + head) * dim;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int r = e0 + 16 * warp + g + 8 * h;
        if (r >= dim) continue;
        float* dst = p.states + (at + r) * vdim + c0;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            const int c = 8 * n + 2 * tig;
            if ((vdim & 1) == 0) {
                if (c0 + c < vdim) *reinterpret_cast<float2*>(dst + c) = make_float2(sum[n][2 * h], sum[n][2 * h + 1]);
            } else {
                if (c0 + c < vdim) dst[c] = sum[n][2 * h];
                if (c0 + c + 1 < vdim) dst[c + 1] = sum[n][2 * h + 1];
            }
        }
        if (sums_norm && tig == 0) p.norms[at + r] = ones[2 * h];
    }
}

// a thread V neighbouring elements of the state (stable: or of the normaliser): a chunk's own sum is replaced by the state
// before the chunk
template <int MODE, int V>
__global__ void __launch_bounds__(128) chunk_carry_kernel(const ChunkArgs p) {
    chain_release();
    chain_wait();
    const int matrix = p.heads * p.dim * p.vdim, vector = MODE == kChunkStable ? p.heads * p.dim : 0;
    const int x = (blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (x >= matrix + (vector + V - 1) / V * V) return;
    const int span = blockIdx.y;
    const int first = p.span_first[span], last = p.span_first[span + 1];
    if (first >= last) return;
    const int t_begin = p.chunk_begin[first], t_end = p.chunk_begin[last];
    const int chunks = (t_end - t_begin + kChunk - 1) / kChunk;
    float* slot = p.state + (long long)p.span_slot[span] * p.slot_stride;
    const int elements = x < matrix ? matrix : vector, e = x < matrix ? x : x - matrix;
    float* of_chunks = (x < matrix ? p.states : p.norms) + (size_t)first * p.pieces * elements + e;
    float* cell = slot + x;
    int own = V;                                             // (the normaliser's last elements may be fewer than V)
    if (V > 1 && x >= matrix) own = min(V, vector - e);
    const bool four = V == 4 && (x < matrix || (p.dim & 3) == 0);
    float s[V];
#pragma unroll
    for (int i = 0; i < V; ++i) s[i] = i < own ? cell[i] : 0.0f;
    // (V divides vdim and, where it reads four at a time, dim: the elements are of one head, and of one row of S)
    int heads_of[V];
    const int row = x < matrix ? e / p.vdim : e;
#pragma unroll
    for (int i = 0; i < V; ++i) heads_of[i] = (x < matrix ? row : min(e + i, vector - 1)) / p.dim;
    const int head = heads_of[0];
    const bool one_head = heads_of[V - 1] == head;
    double peak[V];
#pragma unroll
    for (int i = 0; i < V; ++i) peak[i] = MODE == kChunkStable ? (double)slot[matrix + vector + heads_of[i]] : 0.0;
    const float decay = MODE == kChunkConstant ? p.decay[head] : 1.0f;
    constexpr int kAhead = 8;
    for (int c0 = 0; c0 < chunks; c0 += kAhead) {
        float sum[kAhead][V], keep[kAhead];
        float2 high[kAhead], forget[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const int c = c0 + i;
            if (c >= chunks) continue;
            const float* src = of_chunks + (size_t)c * elements;
            if (four) {
                const float4 y = *reinterpret_cast<const float4*>(src);
                sum[i][0] = y.x; sum[i][1 % V] = y.y; sum[i][2 % V] = y.z; sum[i][3 % V] = y.w;
            } else {
#pragma unroll
                for (int k = 0; k < V; ++k) sum[i][k] = k < own ? src[k] : 0.0f;
            }
            const int count = min(kChunk, t_end - (t_begin + c * kChunk));
            const size_t end = t_begin + c * kChunk + count - 1;
            if (MODE == kChunkScalar) keep[i] = p.cum[end * p.heads + head].x;
            if (MODE == kChunkChannel) keep[i] = p.total[(size_t)(first * p.pieces + c) * p.heads * p.dim + row];
            if (MODE == kChunkConstant) keep[i] = (float)count;
            if (MODE == kChunkStable) {
                high[i] = p.gates[(end * 3 + 2) * p.heads + head];
                forget[i] = p.gates[(end * 3) * p.heads + head];
            }
        }
#pragma unroll
        for (int i = 0; i < kAhead; ++i) {
            const int c = c0 + i;
            if (c >= chunks) continue;
            float* dst = of_chunks + (size_t)c * elements;
            if (four) {
                *reinterpret_cast<float4*>(dst) = make_float4(s[0], s[1 % V], s[2 % V], s[3 % V]);
            } else {
#pragma unroll
                for (int k = 0; k < V; ++k)
                    if (k < own) dst[k] = s[k];
            }
            if (MODE == kChunkStable) {
                if (x < matrix && e % (p.dim * p.vdim) == 0) p.peaks[(size_t)(first * p.pieces + c) * p.heads + head] = peak[0];
                const int count = min(kChunk, t_end - (t_begin + c * kChunk));
                const size_t end = t_begin + c * kChunk + count - 1;
#pragma unroll
                for (int k = 0; k < V; ++k) {
                    if (k > 0 && one_head) {                 // (as a rule)
                        peak[k] = peak[0];
                        continue;
                    }
                    const double own_high = one_double(k == 0 ? high[i] : p.gates[(end * 3 + 2) * p.heads + heads_of[k]]);
                    const double top = fmax(peak[k], own_high);
                    const float f = expf((float)(peak[k] - top)), w = expf((float)(own_high - top));
                    peak[k] = one_double(k == 0 ? forget[i] : p.gates[(end * 3) * p.heads + heads_of[k]]) + top;
                    if (one_head) {
#pragma unroll
                        for (int m = 0; m < V; ++m) s[m] = fmaf(f, s[m], w * sum[i][m]);
                    } else {
                        s[k] = fmaf(f, s[k], w * sum[i][k]);
                    }
                }
            } else {
                float f = keep[i];
                if (MODE == kChunkScalar) f = expf(f);
                if (MODE == kChunkConstant) f = powf(decay, f);
#pragma unroll
                for (int k = 0; k < V; ++k) s[k] = fmaf(f, s[k], sum[i][k]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < V; ++i)
        if (i < own) cell[i] = s[i];
    // (the running maximum, which every thread of the head has read, is written by the read-outs)
}

// The same for the mLSTM where a block's 512 elements are all of one head's matrix (they divide it): its threads share the chunks'
// factors. The running maximum x -> forget + max(x, high) is composed along the chunks by a warp's shuffles, the exponentials are a
// thread a chunk, and the first block of a head takes its normaliser too. 16 heads of 64 x 128, 2,048 tokens: 10.4 us (34 MB);
// every thread making its own factors of two doubles a chunk, 20.8.
constexpr int kCarryThreads = 128;
static __global__ void __launch_bounds__(kCarryThreads) chunk_carry_stable_kernel(const ChunkArgs p) {
    constexpr int kBatch = kCarryThreads, kAhead = 16;
    __shared__ double high_s[kBatch], peak_s[kBatch];
    __shared__ float2 factors_s[kBatch];
    chain_release();
    chain_wait();
    const int span = blockIdx.y, first = p.span_first[span], last = p.span_first[span + 1];
    if (first >= last) return;
    const int t_begin = p.chunk_begin[first], t_end = p.chunk_begin[last];
    const int chunks = (t_end - t_begin + kChunk - 1) / kChunk;
    const int of_head = p.dim * p.vdim, matrix = p.heads * of_head, vector = p.heads * p.dim;
    const int x = (blockIdx.x * kCarryThreads + threadIdx.x) * 4, head = blockIdx.x * kCarryThreads * 4 / of_head;
    const bool first_block = blockIdx.x * kCarryThreads * 4 % of_head == 0;
    const bool normalises = first_block && (int)threadIdx.x * 4 < p.dim;
    const int mine = threadIdx.x;
    float* slot = p.state + (long long)p.span_slot[span] * p.slot_stride;
    float* cell = slot + x;
    float* n_cell = slot + matrix + head * p.dim + 4 * mine;
    float4 s = make_float4(cell[0], cell[1], cell[2], cell[3]), norm = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (normalises) norm = make_float4(n_cell[0], n_cell[1], n_cell[2], n_cell[3]);
    double running = slot[matrix + vector + head];
    auto carry = [&](float4& state, float* of_chunks, size_t stride, int n) {
        for (int c0 = 0; c0 < n; c0 += kAhead) {
            float4 sums[kAhead];
#pragma unroll
            for (int i = 0; i < kAhead; ++i)
                if (c0 + i < n) sums[i] = *reinterpret_cast<const float4*>(of_chunks + (c0 + i) * stride);
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
                if (c0 + i >= n) continue;
                *reinterpret_cast<float4*>(of_chunks + (c0 + i) * stride) = state;
                const float2 f = factors_s[c0 + i];
                state.x = fmaf(f.x, state.x, f.y * sums[i].x);
                state.y = fmaf(f.x, state.y, f.y * sums[i].y);
                state.z = fmaf(f.x, state.z, f.y * sums[i].z);
                state.w = fmaf(f.x, state.w, f.y * sums[i].w);
            }
        }
    };
    for (int b0 = 0; b0 < chunks; b0 += kBatch) {
        const int n = min(kBatch, chunks - b0);
        const size_t chunk0 = (size_t)first * p.pieces + b0;
        if (mine < n) {
            const size_t last_token = min(t_begin + (b0 + mine + 1) * kChunk, t_end) - 1;
            high_s[mine] = one_double(p.gates[(last_token * 3 + 2) * p.heads + head]);
            peak_s[mine] = one_double(p.gates[(last_token * 3) * p.heads + head]);
        }
        __syncthreads();
        if (mine < 32) {
            for (int c0 = 0; c0 < n; c0 += 32) {
                const bool there = c0 + mine < n;
                double slope = there ? peak_s[c0 + mine] : 0.0, least = there ? slope + high_s[c0 + mine] : -INFINITY;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const double slope_up = __shfl_up_sync(0xffffffffu, slope, o), least_up = __shfl_up_sync(0xffffffffu, least, o);
                    if (mine >= o) {
                        least = fmax(least_up + slope, least);
                        slope += slope_up;
                    }
                }
                const double after = fmax(running + slope, least), before = __shfl_up_sync(0xffffffffu, after, 1);
                if (there) peak_s[c0 + mine] = mine == 0 ? running : before;
                running = __shfl_sync(0xffffffffu, after, 31);
            }
        }
        __syncthreads();
        if (mine < n) {
            const double before = peak_s[mine], own_high = high_s[mine], top = fmax(before, own_high);
            factors_s[mine] = make_float2(expf((float)(before - top)), expf((float)(own_high - top)));
            if (first_block) p.peaks[(chunk0 + mine) * p.heads + head] = before;
        }
        __syncthreads();
        carry(s, p.states + chunk0 * matrix + x, matrix, n);
        if (normalises) carry(norm, p.norms + chunk0 * vector + head * p.dim + 4 * mine, vector, n);
        __syncthreads();                                     // (the next batch's take the factors' place)
    }
    cell[0] = s.x; cell[1] = s.y; cell[2] = s.z; cell[3] = s.w;
    if (normalises) {
        n_cell[0] = norm.x; n_cell[1] = norm.y; n_cell[2] = norm.z; n_cell[3] = norm.w;
    }
    // (the running maximum, which every thread of the head has read, is written by the read-outs)
}

// --------------------------------------------------------------------------------------------------------- read-outs
constexpr int kReadThreads = 128;
constexpr int kReadColumns = 64;                             // columns of v that a warp's accumulators hold
constexpr int kReadRows = 32;                                // key channels of k, rows of the state or tokens of v at a time
// Blocks on their way: one in registers, or three in a ring in shared memory (by cp.async) where the queries' width lets no
// more than two blocks of threads share an SM anyway.
template <int WIDTH> constexpr int kReadAhead = WIDTH == 64 ? 1 : 3;
template <int WIDTH> constexpr int read_bytes() {
    return (SplitTile<kChunk, WIDTH>::kElements + 2 * SplitTile<kReadRows, kReadColumns>::kElements) * (int)sizeof(__nv_bfloat16) +
           (WIDTH == 64 ? 0 : kReadAhead<WIDTH> * kReadRows * kReadColumns * (int)sizeof(float));
}
static_assert(SplitTile<kChunk, kReadRows>::kElements == SplitTile<kReadRows, kReadColumns>::kElements, "");

// What the read-outs need of a head's gates over the chunk, twice: a head's are made while warps may still read the last one's.
template <int MODE> struct ReadGates;
template <> struct ReadGates<kChunkChannel> {};
template <> struct ReadGates<kChunkPair> {};
template <> struct ReadGates<kChunkScalar> { float2 cum[kChunk]; float step[kChunk], from_start[kChunk]; };
template <> struct ReadGates<kChunkConstant> { float power[kChunk + 1]; };
template <> struct ReadGates<kChunkStable> { float2 high[kChunk], own[kChunk]; float from_start[kChunk], low[kChunk], norm[256]; };

// blockIdx: (heads / heads a block, chunk, run of `columns` columns, a multiple of 64). WIDTH: key channels of the queries that
// lie in shared memory at a time, 64 or 128. What is multiplied with them comes in blocks of 32 x 64 numbers through two
// buffers, the next block's loads under way while one is multiplied: four warps a block and two or four blocks an SM are what
// hides the rest.
template <int MODE, int WIDTH>
__global__ void __launch_bounds__(kReadThreads, WIDTH == 64 ? 4 : 2) chunk_read_kernel(const ChunkArgs p, int heads_a_block, int columns) {
    constexpr int passes = MODE == kChunkPair ? 2 : 1;       // sets of values
    constexpr bool kPrepared = MODE == kChunkChannel || MODE == kChunkPair;
    using QTile = SplitTile<kChunk, WIDTH>;
    using KTile = SplitTile<kChunk, kReadRows>;
    using STile = SplitTile<kReadRows, kReadColumns>;
    extern __shared__ __align__(128) __nv_bfloat16 tiles[];
    __shared__ ReadGates<MODE> gates_s[2];
    __shared__ BadTokens bad;
    chain_release();
    chain_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
    const int chunk = blockIdx.y;
    bad.clear();
    int begin, count;
    chunk_tokens_of(p, chunk, begin, count);
    if (count <= 0) return;
    const int dim = p.dim, vdim = p.vdim;
    const bool whole = dim <= WIDTH;                         // the queries stay in shared memory
    const int head0 = blockIdx.x * heads_a_block;
    const int qk_head = MODE == kChunkScalar ? head0 / (p.heads / p.groups) : head0;
    __nv_bfloat16* q_t = tiles;
    __nv_bfloat16* const buffers = q_t + QTile::kElements;
    float* const ring = reinterpret_cast<float*>(buffers + 2 * STile::kElements);
    const float* q_src = p.q + (size_t)begin * p.q_stride + (size_t)qk_head * dim;
    const float* k_src = p.k + (size_t)begin * p.k_stride + (size_t)qk_head * dim;
    const bool q_four = by_fours(p.q, p.q_stride, dim), k_four = by_fours(p.k, p.k_stride, dim);
    const bool v_four = by_fours(p.v, p.v_stride, vdim) && (passes == 1 || by_fours(p.v_b, p.v_b_stride, vdim)), s_four = by_fours(p.states, vdim, dim * vdim);
    const int row0 = 16 * warp + g;                          // this lane's tokens: row0, row0 + 8
    auto take_q = [&](int e0) {                              // (32 columns at a time: 16 registers)
#pragma unroll 1
        for (int e = 0; e < WIDTH; e += 32) {
            using Part = TileShare<kChunk, 32, kReadThreads>;
            Part share;
            share.load(q_src + e0 + e, p.q_stride, count, dim - e0 - e, q_four);
            share.template store<QTile>(q_t, e >> 3, Unscaled());
        }
    };
    int turn = 0;                                            // the buffer that the next block goes to
    const int s_blocks = (dim + kReadRows - 1) / kReadRows, a_tile = s_blocks + 2 * passes;
    const int c_begin = blockIdx.z * columns, c_end = min(vdim, c_begin + columns);
    const int v_tiles = (c_end - c_begin + kReadColumns - 1) / kReadColumns;
    const int all_blocks = heads_a_block * v_tiles * a_tile;
    TileShare<kReadRows, kReadColumns, kReadThreads> next;
    // block j of what the heads are multiplied with: per head and 64 columns the rows of the state, then the tokens of v
    auto ask = [&](int j) {
        if (j < all_blocks) {
            const int tile = j / a_tile, part = j - tile * a_tile, h = tile / v_tiles, c0 = c_begin + (tile - h * v_tiles) * kReadColumns;
            const bool of_state = part < s_blocks, second = passes == 2 && part >= s_blocks + 2;
            const int head = head0 + h, r0 = (of_state ? part : (part - s_blocks) & 1) * kReadRows;
            const float* values = second ? p.v_b : p.v;
            const long long values_stride = second ? p.v_b_stride : p.v_stride;
            const int real = (of_state ? dim : count) - r0;
            const float* from = of_state ? p.states + (((size_t)chunk * p.heads + head) * dim + r0) * vdim + c0
                                         : values + (size_t)(begin + min(r0, count - 1)) * values_stride + (size_t)head * vdim + c0;
            const long long stride = of_state ? vdim : values_stride;
            const bool four = of_state ? s_four : v_four;
            if (WIDTH == 64) next.load(from, stride, real, vdim - c0, four);
            else share_copy<kReadRows, kReadColumns, kReadThreads>(ring + (j % kReadAhead<WIDTH>) * kReadRows * kReadColumns, from,
                                                                   stride, real, vdim - c0, four);
        }
        if (WIDTH != 64) asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    auto take = [&](int j) {                                 // the pieces of block j that this thread has copied
        if (WIDTH == 64) return;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kReadAhead<WIDTH> - 1) : "memory");
        share_read(next, ring + (j % kReadAhead<WIDTH>) * kReadRows * kReadColumns);
    };
    float2 next_cum = make_float2(0.0f, 0.0f), next_high = next_cum, next_forget = next_cum;     // of a head's gates
    float next_step = 0.0f;
    double before = 0.0;
    auto ask_gates = [&](int h) {
        if (h >= heads_a_block || tid >= kChunk) return;
        const size_t t = begin + min(tid, count - 1), head = head0 + h;
        if (MODE == kChunkScalar) {
            next_cum = p.cum[t * p.heads + head];
            next_step = p.q_scale * (p.dt ? p.dt[t * p.heads + head] : 1.0f);
        } else if (MODE == kChunkStable) {
            before = p.peaks[(size_t)chunk * p.heads + head];
            next_forget = p.gates[(t * 3) * p.heads + head];
            next_cum = p.gates[(t * 3 + 1) * p.heads + head];
            next_high = p.gates[(t * 3 + 2) * p.heads + head];
        }
    };
    ask_gates(0);
    if (WIDTH != 64) {
#pragma unroll
        for (int i = 0; i < kReadAhead<WIDTH>; ++i) ask(i);
    }

    // q.k of the warp's tokens: columns 8 n + 2 tig, + 1
    float raw[8][4] = {};
    auto load_raw = [&](const float* products) {             // channel
        const float* m = products + ((size_t)chunk * p.heads + head0) * kChunk * kChunk;
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            if (n > 2 * warp + 1) break;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = row0 + 8 * h;
                const float2 x = r < count ? *reinterpret_cast<const float2*>(m + r * kChunk + 8 * n + 2 * tig) : make_float2(0.0f, 0.0f);
                raw[n][2 * h] = x.x;
                raw[n][2 * h + 1] = x.y;
            }
        }
    };
    if (kPrepared) {
        if (whole) take_q(0);
        load_raw(p.products);
    } else {
        TileShare<kChunk, kReadRows, kReadThreads> share;
        share.load(k_src, p.k_stride, count, dim, k_four);
        for (int e0 = 0; e0 < dim; e0 += kReadRows, turn ^= 1) {
            __nv_bfloat16* k_t = buffers + turn * KTile::kElements;
            if (e0 % WIDTH == 0) {
                if (e0 > 0) __syncthreads();                 // (the queries before are still being read)
                take_q(e0);
            }
            share.template store<KTile>(k_t, 0, Unscaled());
            if (e0 + kReadRows < dim) share.load(k_src + e0 + kReadRows, p.k_stride, count, dim - e0 - kReadRows, k_four);
            __syncthreads();
#pragma unroll
            for (int e = 0; e < kReadRows; e += 16) {
                unsigned a[3][4];
                load_a<QTile>(a, q_t, 16 * warp, e0 % WIDTH + e);
#pragma unroll
                for (int n = 0; n < 4; n += 2) {
                    if (n > warp) break;                     // (later tokens; a warp may take the 16 beyond its own too)
                    unsigned b[4][3][2];
                    load_b<KTile>(b, k_t, 16 * n, e);
                    load_b<KTile>(b + 2, k_t, 16 * n + 16, e);
                    mma_split<4>(raw + 2 * n, a, b);
                }
            }
        }
    }

    if (WIDTH == 64) ask(0);
    int j = 0;
    for (int h = 0; h < heads_a_block; ++h) {
        const int head = head0 + h;
        ReadGates<MODE>& gates = gates_s[h & 1];
        if constexpr (MODE == kChunkScalar) {
            if (tid < kChunk) {
                gates.cum[tid] = next_cum;
                gates.from_start[tid] = p.q_scale * expf(next_cum.x);
                gates.step[tid] = tid < count ? next_step : 0.0f;
            }
            ask_gates(h + 1);
        } else if constexpr (MODE == kChunkStable) {
            if (tid < kChunk) {
                const double high = fmax(before, one_double(next_high));
                gates.high[tid] = two_floats(high);
                gates.own[tid] = next_cum;
                gates.from_start[tid] = p.q_scale * expf((float)(before - high));
                gates.low[tid] = expf(-(float)(one_double(next_forget) + high));
            }
            for (int e = tid; e < ((dim + 15) & ~15); e += kReadThreads)
                gates.norm[e] = e < dim ? p.norms[((size_t)chunk * p.heads + head) * dim + e] : 0.0f;
            // the last chunk of a span leaves the running maximum after its last token in the span's slot
            for (int s = tid; s < p.spans && c_begin == 0; s += kReadThreads) {
                const int first = p.span_first[s], last = p.span_first[s + 1];
                if (first * p.pieces > chunk || last * p.pieces <= chunk || begin + count != p.chunk_begin[last]) continue;
                const size_t t = begin + count - 1;
                const double high = fmax(p.peaks[(size_t)chunk * p.heads + head], one_double(p.gates[(t * 3 + 2) * p.heads + head]));
                p.state[(long long)p.span_slot[s] * p.slot_stride + (size_t)p.heads * dim * (vdim + 1) + head] =
                    (float)(one_double(p.gates[(t * 3) * p.heads + head]) + high);
            }
        } else if constexpr (MODE == kChunkConstant) {
            if (tid <= kChunk) gates.power[tid] = powf(p.decay[head], (float)tid);
        }
        const float direct = MODE == kChunkScalar && p.direct ? p.direct[head] : 0.0f;
        float lower[2] = {1.0f, 1.0f};                       // stable: the read-outs' denominators
        for (int c0 = c_begin; c0 < c_end; c0 += kReadColumns) {
            float acc[8][4] = {}, nq[4] = {};
            for (int part = 0; part < s_blocks; ++part, ++j, turn ^= 1) {          // the old state's share
                __nv_bfloat16* s_t = buffers + turn * STile::kElements;
                if (!whole && (part * kReadRows) % WIDTH == 0) {
                    __syncthreads();
                    take_q(part * kReadRows);
                }
                take(j);
                next.template store<STile>(s_t, 0, Unscaled());
                ask(j + kReadAhead<WIDTH>);
                __syncthreads();
#pragma unroll
                for (int e = 0; e < kReadRows; e += 16) {
                    unsigned a[3][4];
                    load_a<QTile>(a, q_t, 16 * warp, (part * kReadRows) % WIDTH + e);
#pragma unroll
                    for (int n = 0; n < 4; n += 2) {
                        unsigned b[4][3][2];
                        load_b_transposed<STile>(b, s_t, 16 * n, e);
                        load_b_transposed<STile>(b + 2, s_t, 16 * n + 16, e);
                        mma_split<4>(acc + 2 * n, a, b);
                    }
                    if constexpr (MODE == kChunkStable) {
                        if (c0 == c_begin && part * kReadRows + e < dim) { // the normaliser as a ninth tile's first column
                            unsigned b[1][3][2] = {};
                            if (g == 0) {
                                const float* norm = gates.norm + part * kReadRows + e + 2 * tig;
                                split_pair(norm[0], norm[1], b[0][0][0], b[0][1][0], b[0][2][0]);
                                split_pair(norm[8], norm[9], b[0][0][1], b[0][1][1], b[0][2][1]);
                            }
                            mma_split<1>(&nq, a, b);
                        }
                    }
                }
            }
            if constexpr (!kPrepared) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float f;
                    if constexpr (MODE == kChunkConstant) f = gates.power[row0 + 8 * i + 1];
                    else f = gates.from_start[row0 + 8 * i];
#pragma unroll
                    for (int n = 0; n < 8; ++n)
#pragma unroll
                        for (int r = 0; r < 2; ++r) acc[n][2 * i + r] *= f;
                    nq[2 * i] *= f;
                }
            }
            float sums[2] = {0.0f, 0.0f};
            for (int pass = 0; pass < passes; ++pass) {
            if (passes == 2 && pass == 1) load_raw(p.products_b);          // (one tile of columns: vdim is at most 64)
#pragma unroll
            for (int part = 0; part < 2; ++part, ++j, turn ^= 1) {                 // the chunk's own tokens, 32 at a time
                __nv_bfloat16* v_t = buffers + turn * STile::kElements;
                take(j);
                if (!next.template store<STile>(v_t, 0, Unscaled())) next.template take_out<STile>(v_t, 0, bad, part * kReadRows, 0);
                ask(j + kReadAhead<WIDTH>);
                __syncthreads();
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int m = 2 * part + half;
                    if (m > warp) break;
                    unsigned a[3][4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {            // rows row0, row0 + 8 of the first eight, then of the others
                        const int n = 2 * m + (u >> 1), i = row0 + 8 * (u & 1);
                        float x[2];
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const int t = 8 * n + 2 * tig + r;
                            const bool seen = t <= i && i < count;
                            float weight = 1.0f;
                            if constexpr (MODE == kChunkScalar) weight = exp_between(gates.cum[i], gates.cum[t]) * gates.step[t];
                            if constexpr (MODE == kChunkConstant) weight = p.q_scale * gates.power[max(i - t, 0)];
                            if constexpr (MODE == kChunkStable) weight = p.q_scale * exp_between(gates.own[t], gates.high[i]);
                            x[r] = seen ? raw[n][2 * (u & 1) + r] * weight : 0.0f;
                            if (MODE == kChunkScalar && t == i && seen) x[r] += direct;      // (the value's own share)
                            sums[u & 1] += x[r];
                        }
                        split_pair(x[0], x[1], a[0][u], a[1][u], a[2][u]);
                    }
#pragma unroll
                    for (int n = 0; n < 4; n += 2) {
                        unsigned b[4][3][2];
                        load_b_transposed<STile>(b, v_t, 16 * n, 16 * half);
                        load_b_transposed<STile>(b + 2, v_t, 16 * n + 16, 16 * half);
                        mma_split<4>(acc + 2 * n, a, b);
                    }
                }
            }
            }
            if (bad.any) {                                   // (the same for all threads: it is written before the next barrier only)
                bad.mark(acc, row0, 2 * tig);
                __syncthreads();
                bad.clear();
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int r = row0 + 8 * i;
                if constexpr (MODE == kChunkStable) {
                    if (c0 == c_begin) {
                        float sum = sums[i] + (tig == 0 ? nq[2 * i] : 0.0f);
                        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                        lower[i] = fmaxf(fabsf(sum), gates.low[r]) + 1e-6f;
                    }
                }
                if (r >= count) continue;
                float* dst = p.out + (size_t)(begin + r) * p.heads * vdim + (size_t)head * vdim + c0;
#pragma unroll
                for (int n = 0; n < 8; ++n) {
                    const int c = 8 * n + 2 * tig;
                    float o[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        o[k] = acc[n][2 * i + k];
                        if (MODE == kChunkStable) o[k] = o[k] / lower[i];
                    }
                    if ((vdim & 1) == 0) {
                        if (c0 + c < vdim) *reinterpret_cast<float2*>(dst + c) = make_float2(o[0], o[1]);
                    } else {
                        if (c0 + c < vdim) dst[c] = o[0];
                        if (c0 + c + 1 < vdim) dst[c + 1] = o[1];
                    }
                }
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------------------- launches
template <typename Kernel>
inline int allow_shared(Kernel kernel, size_t bytes, const char* what) {
    if (bytes <= 40 * 1024) return 0;
    const cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (status == cudaSuccess) return 0;
    set_error("%s: %s", what, cudaGetErrorString(status));
    return -2;
}

template <int MODE, int COLUMNS>
inline int launch_walk(const ChunkArgs& p, cudaStream_t stream) {
    constexpr size_t bytes = (size_t)2 * walk_buffer<COLUMNS>() * sizeof(__nv_bfloat16);
    const int status = allow_shared(chunk_walk_kernel<MODE, COLUMNS>, bytes, "chunk_walk");
    if (status != 0) return status;
    const int v_tiles = (p.vdim + COLUMNS - 1) / COLUMNS;
    // A plain launch: blocks of a chained launch that walks for long end up on the few SMs that had room for them.
    chunk_walk_kernel<MODE, COLUMNS><<<dim3(v_tiles * ((p.dim + kWalkRows - 1) / kWalkRows), p.heads, p.spans), kWalkThreads, bytes, stream>>>(p);
    return check_launch("chunk_walk");
}

template <int MODE>
inline int launch_sums(const ChunkArgs& p, int chunks, cudaStream_t stream) {
    constexpr size_t bytes = (size_t)kSumElements * sizeof(__nv_bfloat16);
    int status = allow_shared(chunk_sum_kernel<MODE>, bytes, "chunk_sum");
    if (status != 0) return status;
    launch_chained(chunk_sum_kernel<MODE>, dim3(((p.vdim + 63) / 64) * ((p.dim + 63) / 64), p.heads, chunks), kSumThreads, bytes, stream, p);
    if ((status = check_launch("chunk_sum")) != 0) return status;
    const long long elements = (long long)p.heads * p.dim * (p.vdim + (MODE == kChunkStable ? 1 : 0));
    const bool four = p.vdim % 4 == 0 && ((size_t)p.states & 15) == 0 && ((size_t)p.norms & 15) == 0;
    if constexpr (MODE == kChunkStable) {
        if (four && p.dim % 4 == 0 && p.dim <= 4 * kCarryThreads && p.dim * p.vdim % (4 * kCarryThreads) == 0) {
            launch_chained(chunk_carry_stable_kernel, dim3((unsigned)(p.heads * p.dim * p.vdim / (4 * kCarryThreads)), p.spans),
                           kCarryThreads, 0, stream, p);
            return check_launch("chunk_carry");
        }
    }
    if (four) launch_chained(chunk_carry_kernel<MODE, 4>, dim3((unsigned)((elements + 511) / 512), p.spans), 128, 0, stream, p);
    else launch_chained(chunk_carry_kernel<MODE, 1>, dim3((unsigned)((elements + 127) / 128), p.spans), 128, 0, stream, p);
    return check_launch("chunk_carry");
}

template <int MODE, int WIDTH>
inline int launch_read(const ChunkArgs& p, int chunks, int heads_a_block, cudaStream_t stream) {
    constexpr size_t bytes = (size_t)read_bytes<WIDTH>();
    const int status = allow_shared(chunk_read_kernel<MODE, WIDTH>, bytes, "chunk_read");
    if (status != 0) return status;
    // the columns of a head in as many blocks as they have runs of 64, where the GPU has room for them: a short step waits for
    // its longest block
    const bool apart = (long long)p.heads / heads_a_block * chunks <= 148;
    const int columns = apart ? kReadColumns : p.vdim;
    launch_chained(chunk_read_kernel<MODE, WIDTH>, dim3(p.heads / heads_a_block, chunks, (p.vdim + columns - 1) / columns), kReadThreads,
                   bytes, stream, p, heads_a_block, columns);
    return check_launch("chunk_read");
}

// Heads that share queries and keys share a read-out block's products of them: as many as make the launch shortest, in rounds of the
// blocks that the GPU holds (four an SM, two with wide queries) times a block's steps (products of keys, then of the state's rows
// and of the values of every head). 64 heads on 8 of 128 x 64, 2,048 tokens: 96.8 us with eight heads a block (264 blocks, one
// round), 110 with four (528, two); 300 tokens 30.6 and 39.4 with one.
inline int heads_of_a_read(int heads, int groups, int dim, int vdim, int chunks) {
    const int shared = (dim + kReadRows - 1) / kReadRows + 2, slots = dim <= 64 ? 592 : 296;
    const int per_head = shared * ((vdim + kReadColumns - 1) / kReadColumns);
    int heads_a_block = 1;
    long long best = 0;
    for (int n = 1; n <= 8 && (heads / groups) % n == 0; n *= 2) {
        const long long blocks = (long long)chunks * heads / n, cost = (blocks + slots - 1) / slots * (n * per_head + shared);
        if (n == 1 || cost < best) {
            best = cost;
            heads_a_block = n;
        }
    }
    return heads_a_block;
}

template <int MODE>
inline int launch_reads(const ChunkArgs& p, int chunks, cudaStream_t stream) {
    const int heads_a_block = MODE == kChunkScalar ? heads_of_a_read(p.heads, p.groups, p.dim, p.vdim, chunks) : 1;
    return p.dim <= 64 ? launch_read<MODE, 64>(p, chunks, heads_a_block, stream)
                       : launch_read<MODE, 128>(p, chunks, heads_a_block, stream);
}

// How the states are made: by the walk with 32 or 64 columns a block, or (0) by sums and carry. `longest`: chunks of the longest
// span, as many as the others leave where it is not known (0).
//
// The walk moves a third of the bytes, but a span's chunks come one after another: of the longest span, 1.6 us each with a block of
// 32 columns an SM (the mLSTM 2.1), 2.6 with two blocks, more by what is above two; 2.4 (2.8) with 64 columns. So it is 64 columns
// where the blocks of 32, as many as walk at a time on the whole, would share the SMs and those of 64 do not: 64 heads of 128 x 64,
// 4,096 tokens 158 us, with 32 columns 171; 16 heads of 64 x 128 (64 blocks of 32) 153 and 102, two fifths of a block zeros at values
// of 96. Sums and carry are bound by their work and bytes: 4.5 us, 11 ns a chunk and 64 x 64 of S, the states' bytes at 4.8 TB/s and
// those beyond the L2 twice over, and what a span's beginning and end cost, to the mLSTM most. Walk (by its rule) and sums, us: 64
// heads of 128 x 64, 2,048 tokens 81 / 104, 300 tokens 15.1 / 19.4; 16 of 64 x 128 2,048 tokens 52 / 25, six spans of 512 36 / 34,
// sixteen of 150 34 / 41, one of 4,096 beside seven of 64 104 / 52 (mLSTM 140 / 69).
inline int walk_columns(bool stable, int heads, int dim, int vdim, int spans, int chunks, int longest) {
    const double key_tiles = (double)((dim + kWalkRows - 1) / kWalkRows) * heads;
    const double narrow = key_tiles * ((vdim + 31) / 32), wide = key_tiles * ((vdim + 63) / 64);
    const int most = chunks - spans + 1 > 1 ? chunks - spans + 1 : 1;
    const double chain = longest > 0 && longest < most ? longest : most, at_once = chunks / chain;
    const bool is_wide = narrow * at_once > 148.0 && wide * at_once <= 148.0 && wide < narrow;
    double each = stable ? 2.05 : 1.57;
    if (is_wide) each = stable ? 2.75 : 2.4;
    else if (narrow * at_once > 148.0) each = (stable ? 3.2 : 2.63) * (narrow * at_once > 296.0 ? narrow * at_once / 296.0 : 1.0);
    const double elements = (double)heads * dim * vdim, bytes = elements * chunks * 8.0;
    const double sums = 4.5 + 0.011 * wide * chunks + bytes / 4.8e6 + (bytes > 1e8 ? (bytes - 1e8) / 4e6 : 0.0) +
                        elements / 131072.0 * spans * (stable ? 2.0 : 0.3);
    return 2.8 + chain * each < sums ? (is_wide ? 64 : 32) : 0;
}

// `chunks` bounds the chunks of all spans, `longest` those of the longest (0: not known); p.chunk_begin has chunks / p.pieces + 1
// entries
template <int MODE>
inline int launch_chunk_scan(const ChunkArgs& p, int chunks, int longest, cudaStream_t stream) {
    const int columns = walk_columns(MODE == kChunkStable, p.heads, p.dim, p.vdim, p.spans, chunks, longest);
    const int status = columns == 64 ? launch_walk<MODE, 64>(p, stream) : columns == 32 ? launch_walk<MODE, 32>(p, stream)
                                                                                        : launch_sums<MODE>(p, chunks, stream);
    return status != 0 ? status : launch_reads<MODE>(p, chunks, stream);
}

}  // namespace celeg_b200
