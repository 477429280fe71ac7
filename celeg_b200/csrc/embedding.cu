// Embedding gather: residual[t, :] = multiplier * table[token[t], :], written as float32
// (the residual stream is kept in 32-bit on both precision paths). With positions and a table of frequencies a
// sinusoidal vector of the token's position is added: entry 2i gets sin(p f_i), entry 2i + 1 cos(p f_i), the
// angle a float32 product, sine and cosine the precise float32 functions.
// Counterpart in celeg: embedding_batch_kernel (src/backend/cuda/kernels/embedding.cu:26).
#include "common.cuh"

namespace celeg_b200 {

// next_w != null: the first half of a split RMSNorm (gemv_bf16.cu) for the norm that follows:
// xw_out[t, :] = bf16(residual * next_w) and sumsq_out[t] = sum(residual^2). next_w == null with xw_out given: xw_out is a
// plain bfloat16 copy of the row, for a first block that reads the stream itself.
template <typename W>
__global__ void embedding_kernel(const W* __restrict__ table, const int* tokens, const int* positions,
                                 const float* __restrict__ frequencies,
                                 float* out, int hidden, int vocab, float multiplier, const float* next_w,
                                 __nv_bfloat16* xw_out, float* sumsq_out, int sumsq_stride) {
    __shared__ float scratch[33];
    chain_release();
    chain_wait();
    const int row = blockIdx.x;
    const int token = tokens[row];
    float* dst = out + (size_t)row * hidden;
    const bool valid = token >= 0 && token < vocab;          // the host refuses other ids before launch
    const W* src = table + (size_t)(valid ? token : 0) * hidden;
    float squares = 0.0f;
    const float place = frequencies ? (float)positions[row] : 0.0f;
    // A row of the table is a miss in every cache: eight of a thread's numbers are asked for at a time, since one by one the loads of
    // a turn wait for the stores of the one before. 8 rows of 2,048 with their squares: 2.8 us, 6.5 one by one.
    constexpr int kAhead = 8;
    for (int first = threadIdx.x; first < hidden; first += kAhead * blockDim.x) {
        W x[kAhead];
        float w[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int i = first + u * blockDim.x;
            if (i >= hidden) continue;
            x[u] = src[i];
            if (next_w) w[u] = next_w[i];
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int i = first + u * blockDim.x;
            if (i >= hidden) continue;
            float v = valid ? to_float(x[u]) * multiplier : 0.0f;
            if (frequencies) {
                const float angle = place * frequencies[i >> 1];
                v += (i & 1) ? cosf(angle) : sinf(angle);
            }
            dst[i] = v;
            if (xw_out) xw_out[(size_t)row * hidden + i] = __float2bfloat16_rn(next_w ? v * w[u] : v);
            if (next_w) squares += v * v;
        }
    }
    if (next_w) {
        squares = block_sum(squares, scratch);
        if (threadIdx.x == 0) sumsq_out[(size_t)row * sumsq_stride] = squares;
    }
}

// The same, eight neighbours a thread and access, where rows are multiples of that and there are neither positions to add nor
// squares to add up (whose order the kernel above gives).
template <typename W>
__global__ void __launch_bounds__(256) embedding_eights_kernel(const W* __restrict__ table, const int* tokens, float* __restrict__ out,
                                                               int hidden, int vocab, float multiplier,
                                                               __nv_bfloat16* __restrict__ xw_out) {
    chain_release();
    chain_wait();
    const int row = blockIdx.x, token = tokens[row];
    const bool valid = token >= 0 && token < vocab;          // the host refuses other ids before launch
    const W* src = table + (size_t)(valid ? token : 0) * hidden;
    float* dst = out + (size_t)row * hidden;
    for (int i = threadIdx.x * 8; i < hidden; i += blockDim.x * 8) {
        float v[8];
        if (sizeof(W) == 2) {
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(src + i));
            const __nv_bfloat162* pairs = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 x = __bfloat1622float2(pairs[j]);
                v[2 * j] = x.x;
                v[2 * j + 1] = x.y;
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; j += 4) {
                const float4 x = __ldg(reinterpret_cast<const float4*>(src + i + j));
                v[j] = x.x; v[j + 1] = x.y; v[j + 2] = x.z; v[j + 3] = x.w;
            }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = valid ? v[j] * multiplier : 0.0f;
#pragma unroll
        for (int j = 0; j < 8; j += 4) *reinterpret_cast<float4*>(dst + i + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        if (xw_out) {
            uint4 raw;
            __nv_bfloat162* pairs = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
            for (int j = 0; j < 4; ++j) pairs[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
            *reinterpret_cast<uint4*>(xw_out + (size_t)row * hidden + i) = raw;
        }
    }
}

}  // namespace celeg_b200

using namespace celeg_b200;

static int embedding_checked(const void* table, int table_dtype, const int* tokens, const int* positions,
                             const float* frequencies, float* out, int rows, int hidden,
                             int vocab, float multiplier, const float* next_w, void* xw_out, float* sumsq_out,
                             int sumsq_stride, cudaStream_t stream) {
    CELEG_REQUIRE(rows >= 0 && hidden > 0 && vocab > 0, "embedding: invalid sizes rows=%d hidden=%d vocab=%d",
                  rows, hidden, vocab);
    CELEG_REQUIRE(!next_w || (xw_out && sumsq_out && sumsq_stride >= 1),
                  "embedding: preparing the norm that follows needs its two outputs");
    if (rows == 0) return 0;
    // Its loads need 16-byte addresses, which the row's start has when its length is a multiple of eight (bfloat16) and the
    // buffers' starts have them.
    if (hidden % 8 == 0 && !frequencies && !next_w && (table_dtype == kFloat32 || table_dtype == kBFloat16) &&
        (((size_t)table | (size_t)out | (size_t)xw_out) & 15) == 0) {
        const int eights = hidden / 8, block = eights >= 256 ? 256 : (eights + 31) / 32 * 32;
        if (table_dtype == kFloat32)
            launch_chained(embedding_eights_kernel<float>, rows, block, 0, stream, (const float*)table, tokens, out, hidden, vocab,
                           multiplier, (__nv_bfloat16*)xw_out);
        else
            launch_chained(embedding_eights_kernel<__nv_bfloat16>, rows, block, 0, stream, (const __nv_bfloat16*)table, tokens, out,
                           hidden, vocab, multiplier, (__nv_bfloat16*)xw_out);
        return check_launch("embedding");
    }
    const int threads = hidden >= 1024 ? 256 : 128;
    if (table_dtype == kFloat32)
        launch_chained(embedding_kernel<float>, rows, threads, 0, stream, (const float*)table, tokens, positions,
                       frequencies, out, hidden, vocab, multiplier, next_w, (__nv_bfloat16*)xw_out, sumsq_out, sumsq_stride);
    else if (table_dtype == kBFloat16)
        launch_chained(embedding_kernel<__nv_bfloat16>, rows, threads, 0, stream, (const __nv_bfloat16*)table,
                       tokens, positions, frequencies, out, hidden, vocab, multiplier, next_w, (__nv_bfloat16*)xw_out, sumsq_out, sumsq_stride);
    else
        CELEG_REQUIRE(false, "embedding: unknown dtype code %d", table_dtype);
    return check_launch("embedding");
}

CELEG_API int celeg_embedding(const void* table, int table_dtype, const int* tokens, float* out, int rows,
                              int hidden, int vocab, float multiplier, cudaStream_t stream) {
    return embedding_checked(table, table_dtype, tokens, nullptr, nullptr, out, rows, hidden, vocab, multiplier, nullptr,
                             nullptr, nullptr, 0, stream);
}

// The gather and, for the RMSNorm that follows, the first half of a split norm: xw_out [rows, hidden]
// bfloat16 = residual * next_w, sumsq_out[row * sumsq_stride] = sum of the row's squares.
CELEG_API int celeg_embedding_split_norm(const void* table, int table_dtype, const int* tokens, float* out, int rows,
                                         int hidden, int vocab, float multiplier, const float* next_w, void* xw_out,
                                         float* sumsq_out, int sumsq_stride, cudaStream_t stream) {
    return embedding_checked(table, table_dtype, tokens, nullptr, nullptr, out, rows, hidden, vocab, multiplier, next_w,
                             xw_out, sumsq_out, sumsq_stride, stream);
}

// The gather and a bfloat16 copy of the rows.
CELEG_API int celeg_embedding_copy(const void* table, int table_dtype, const int* tokens, float* out, int rows, int hidden,
                                   int vocab, float multiplier, void* copy, cudaStream_t stream) {
    return embedding_checked(table, table_dtype, tokens, nullptr, nullptr, out, rows, hidden, vocab, multiplier, nullptr,
                             copy, nullptr, 0, stream);
}

// The gather plus the sinusoidal vector of each token's position (frequencies: float32 [(hidden + 1) / 2]); next_w
// may be null (no norm prepared).
CELEG_API int celeg_embedding_sinusoid(const void* table, int table_dtype, const int* tokens, const int* positions,
                                       const float* frequencies, float* out, int rows, int hidden, int vocab,
                                       float multiplier, const float* next_w, void* xw_out, float* sumsq_out,
                                       int sumsq_stride, cudaStream_t stream) {
    CELEG_REQUIRE(positions && frequencies, "embedding: a position vector needs positions and frequencies");
    return embedding_checked(table, table_dtype, tokens, positions, frequencies, out, rows, hidden, vocab, multiplier,
                             next_w, xw_out, sumsq_out, sumsq_stride, stream);
}
