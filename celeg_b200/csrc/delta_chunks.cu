// The gated delta rule over prompts in chunks of 64 tokens (recurrent_scan.cu has it token by token, and says what it is):
//
//   S~ = g S;  u = beta (v - S~^T k);  S' = S~ + k u^T;  o = q_scale S'^T q
//
// With G(i, j) = g_(j+1) .. g_i over the chunk's tokens (G(i) from its first) and S_0 the state before it, the u of the chunk
// are the solution of a unit lower triangular system (the compact form of a product of such updates: Bischof and Van Loan,
// "The WY Representation for Products of Householder Matrices", 1987; Yang et al., "Parallelizing Linear Transformers with the
// Delta Rule over Sequence Length", 2024):
//
//   u_i + sum_(j<i) beta_i G(i, j) (k_i . k_j) u_j = beta_i v_i - beta_i G(i) S_0^T k_i
//
// so u = U_0 - W S_0 with U_0, W the solutions for the right sides beta v and beta G k, and then
//
//   o_i = q_scale [ G(i) S_0^T q_i + sum_(j<=i) G(i, j) (q_i . k_j) u_j ]         S_n = G(n) S_0 + sum_j G(n, j) k_j u_j^T
//
//   decays    the running sums of the decays' logarithms (decayed_scan.cu)
//   solve     a block a (chunk, head): k.k, the system's inverse, its products with the right sides; leaves U_0 in float32,
//             and -W and G(n, j) k_j split for the tensor cores, as they will lie in shared memory
//   walk      a block a (span, head, run of columns) goes through the chunks: u = U_0 - W S, then S, two products a chunk, the
//             next chunk's operands under way as one bulk copy each; leaves u and the states before the chunks
//   read-outs those of the other chunked scans (chunk_scan.cuh) with u in the place of v
//
// Products and their precision: chunk_scan.cuh.
#include "chunk_scan.cuh"
#include "general_delta.cuh"
#include "ring_drain.h"
#include "tcgen05.cuh"

namespace celeg_b200 {

struct DeltaChunkArgs {
    const float* k; int k_stride;            // [tokens, kv_heads * dim], unit vectors
    const float* v; int v_stride;            // [tokens, heads * vdim]
    const float* gates;                      // [tokens, 2 * heads]: beta in the first half
    const float2* cum;                       // [tokens, heads]
    const int* chunk_begin; const int* span_first;
    __nv_bfloat16* operands;                 // [chunks, heads, 2]: -W, G(n, .) k, a SplitTile<64, WIDTH> each
    float* u;                                // [tokens, heads * vdim]: U_0, then u
    float* states;                           // [chunks, heads, dim, vdim]
    float* state; long long slot_stride; const int* span_slot;
    int heads, kv_heads, dim, vdim;
    int* error_flag;
    const float* total;                      // general: [chunks, heads * dim], the channels' decays over a chunk (then cum, gates
                                             // are null, and `states` holds what the chunk's own values add)
};

// ------------------------------------------------------------------------------------------------------------- solve
// The system's matrix is inverted, T = (1 + L)^-1: its four diagonal blocks of 16 by substitution, a warp a block and a lane a
// column; then two blocks of 16 and at last two of 32 are joined, T_21 = -T_22 L_21 T_11; and W and U_0 are products of T with
// the scaled k and v. It is bound by the latency of these steps, so blocks an SM count: T in float32 lies where k did and L where
// T's planes will, 50 KB a block, four of them an SM; the right sides are scaled, so that T is split once. 60 us for 32 heads of
// 64 and 2,048 tokens (57 before it left out tokens that are not finite; 69 with three blocks and T split twice; 138 by substitution over whole right sides, one chain of 64 steps
// a block).
constexpr int kSolveThreads = 128;
constexpr int kSolvePitch = kChunk + 4;
template <int WIDTH> constexpr int solve_bytes() {
    return (SplitTile<kChunk, WIDTH>::kElements + SplitTile<kChunk, 64>::kElements) * 2;
}
static_assert(SplitTile<kChunk, 64>::kElements * 2 >= kChunk * kSolvePitch * 4, "L lies where T's planes will, T where k did");

// out = sign a b of N x N blocks of matrices with kSolvePitch floats a row, 128 / (N * N / 4) of them side by side; a thread four
// neighbours of a row. `a`, `b`, `out`: of the thread's block.
template <int N>
__device__ __forceinline__ void join_product(const float* a, const float* b, float* out, float sign, int slot) {
    const int r = slot / (N / 4), c = (slot % (N / 4)) * 4;
    float4 sum = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 8
    for (int k = 0; k < N; ++k) {
        const float x = a[r * kSolvePitch + k];
        const float4 y = *reinterpret_cast<const float4*>(b + k * kSolvePitch + c);
        sum.x = fmaf(x, y.x, sum.x); sum.y = fmaf(x, y.y, sum.y); sum.z = fmaf(x, y.z, sum.z); sum.w = fmaf(x, y.w, sum.w);
    }
    *reinterpret_cast<float4*>(out + r * kSolvePitch + c) = make_float4(sign * sum.x, sign * sum.y, sign * sum.z, sign * sum.w);
}

// inverse = (1 + L)^-1, kSolvePitch floats a row, `lower` strictly lower triangular, `inverse` zero at first; what is left above
// its diagonal is not to be used. All threads of a block come here, 128 of them work.
__device__ __forceinline__ void invert(const float* lower, float* inverse) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool works = tid < 128;
    __syncthreads();
    if (works && lane < 16) {                                // a diagonal block a warp
        const float* l = lower + 16 * warp * kSolvePitch + 16 * warp;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float sum[4] = {i == lane ? 1.0f : 0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int j = 0; j < i; ++j) sum[j & 3] = fmaf(-l[i * kSolvePitch + j], x[j], sum[j & 3]);
            x[i] = (sum[0] + sum[1]) + (sum[2] + sum[3]);
            inverse[(16 * warp + i) * kSolvePitch + 16 * warp + lane] = x[i];
        }
    }
    __syncthreads();
    // two pairs of blocks of 16, 64 threads each; L_10 T_00 goes where the block above the diagonal is, zero again at the end
    const int o = ((tid >> 6) & 1) * 32 * (kSolvePitch + 1), slot = tid & 63;
    float* spare = inverse + o + 16;
    if (works) join_product<16>(lower + o + 16 * kSolvePitch, inverse + o, spare, 1.0f, slot);
    __syncthreads();
    if (works) join_product<16>(inverse + o + 16 * (kSolvePitch + 1), spare, inverse + o + 16 * kSolvePitch, -1.0f, slot);
    __syncthreads();
    if (works) *reinterpret_cast<float4*>(spare + (slot >> 2) * kSolvePitch + (slot & 3) * 4) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    __syncthreads();
    float* corner = inverse + 32;                            // the same with the two blocks of 32
    for (int i = tid; i < 256; i += blockDim.x) join_product<32>(lower + 32 * kSolvePitch, inverse, corner, 1.0f, i);
    __syncthreads();
    for (int i = tid; i < 256; i += blockDim.x)
        join_product<32>(inverse + 32 * (kSolvePitch + 1), corner, inverse + 32 * kSolvePitch, -1.0f, i);
    __syncthreads();
}

// a warp's rows t, t + 8 of W: NaN from `good` on
__device__ __forceinline__ void leave_out(float (&acc)[8][4], int t, int good) {
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (t + 8 * (r >> 1) >= good) acc[n][r] = NAN;
}

template <int WIDTH>
__global__ void __launch_bounds__(kSolveThreads, WIDTH == 64 ? 4 : 2) delta_solve_kernel(const DeltaChunkArgs p) {
    using Tile = SplitTile<kChunk, WIDTH>;
    using TTile = SplitTile<kChunk, 64>;
    using VTile = SplitTile<kChunk, 64>;
    extern __shared__ __align__(128) __nv_bfloat16 tiles[];
    __shared__ float2 cum_s[kChunk];
    __shared__ float beta_s[kChunk], start_s[kChunk], end_s[kChunk];
    __shared__ BadTokens v_bad;
    __shared__ int k_bad;                                    // the first token with a key, rate or decay that is not finite
    chain_release();
    chain_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
    v_bad.clear();
    if (tid == 0) k_bad = kChunk;
    const int chunk = blockIdx.y, head = blockIdx.x, dim = p.dim, vdim = p.vdim;
    const int begin = p.chunk_begin[chunk], count = p.chunk_begin[chunk + 1] - begin;
    if (count <= 0) return;
    __nv_bfloat16* k_t = tiles;                              // k, then T in float32, then the right sides
    __nv_bfloat16* t_t = tiles + Tile::kElements;            // T's planes, at first L
    float* lower = reinterpret_cast<float*>(t_t);
    float* inverse = reinterpret_cast<float*>(k_t);
    const float* k_src = p.k + (size_t)begin * p.k_stride + (size_t)(head / (p.heads / p.kv_heads)) * dim;
    const float* v_src = p.v + (size_t)begin * p.v_stride + (size_t)head * vdim;
    const bool k_four = by_fours(p.k, p.k_stride, dim), v_four = by_fours(p.v, p.v_stride, vdim);
    if (tid < kChunk) {
        const size_t t = begin + min(tid, count - 1);
        const float2 own = p.cum[t * p.heads + head];
        cum_s[tid] = own;
        beta_s[tid] = tid < count ? p.gates[t * 2 * p.heads + head] : 0.0f;
        start_s[tid] = expf(own.x);
        end_s[tid] = exp_between(p.cum[(size_t)(begin + count - 1) * p.heads + head], own);
    }
    __syncthreads();
    if (tid < kChunk && !(fabsf(beta_s[tid]) <= FLT_MAX && fabsf(cum_s[tid].x) <= FLT_MAX)) atomicMin(&k_bad, tid);
    const size_t at = ((size_t)chunk * p.heads + head) * 2;
    __nv_bfloat16* w_out = p.operands + at * Tile::kElements;
    __nv_bfloat16* k_out = w_out + Tile::kElements;
    using Part = TileShare<kChunk, 32, kSolveThreads>;
    Part share;
#pragma unroll 1
    for (int e = 0; e < WIDTH; e += 32) {
        share.load(k_src + e, p.k_stride, count, dim - e, k_four);
        const bool finite = share.template store<Tile>(k_t, e >> 3, Unscaled());
        share.template store<Tile>(k_out, e >> 3, [&](int r) { return end_s[r]; });      // G(n, j) k_j: what S is given of u_j
        if (!finite) Part::each_bad<Tile>(k_t, e >> 3, [&](int r, int, __nv_bfloat16*) { atomicMin(&k_bad, r); });
    }
    __syncthreads();
    // The rows of the system from the first bad token on are left out (the tokens before it meet them under weights of zero:
    // chunk_scan.cuh); their W is NaN in the end, and with it their u.
    const int good = min(count, k_bad);
    {
        float raw[8][4] = {};                                // k.k: the warp's 16 tokens against 8 n + 2 tig, + 1
#pragma unroll 2
        for (int e = 0; e < WIDTH; e += 16) {
            unsigned a[3][4];
            load_a<Tile>(a, k_t, 16 * warp, e);
#pragma unroll
            for (int n = 0; n < 4; n += 2) {
                if (n > warp) break;
                unsigned b[4][3][2];
                load_b<Tile>(b, k_t, 16 * n, e);
                load_b<Tile>(b + 2, k_t, 16 * n + 16, e);
                mma_split<4>(raw + 2 * n, a, b);
            }
        }
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = 16 * warp + g + 8 * (r >> 1), j = 8 * n + 2 * tig + (r & 1);
                lower[i * kSolvePitch + j] = j < i && i < good ? raw[n][r] * beta_s[i] * exp_between(cum_s[i], cum_s[j]) : 0.0f;
            }
    }
    __syncthreads();                                         // k has been used
    for (int i = tid; i < kChunk * kSolvePitch; i += kSolveThreads) inverse[i] = 0.0f;
    invert(lower, inverse);
    for (int i = tid; i < kChunk * kChunk / 2; i += kSolveThreads) {           // T's planes in the place of L
        const int r = i >> 5, c = (i & 31) * 2;
        const float2 x = *reinterpret_cast<const float2*>(inverse + r * kSolvePitch + c);
        unsigned plane[3];
        split_pair(c <= r ? x.x : 0.0f, c + 1 <= r ? x.y : 0.0f, plane[0], plane[1], plane[2]);
#pragma unroll
        for (int n = 0; n < 3; ++n) *reinterpret_cast<unsigned*>(t_t + n * TTile::kPlane + TTile::at(r, c >> 3) + (c & 7)) = plane[n];
    }
    __syncthreads();
#pragma unroll 1
    for (int e = 0; e < WIDTH; e += 32) {                    // the right sides beta G k
        share.load(k_src + e, p.k_stride, good, dim - e, k_four);
        share.template store<Tile>(k_t, e >> 3, [&](int r) { return r < good ? beta_s[r] * start_s[r] : 0.0f; });
    }
    float acc[8][4];
    auto multiply = [&](auto tile, const __nv_bfloat16* from, int n0) {        // T times 64 columns from n0 on
        using B = decltype(tile);
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[n][r] = 0.0f;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            if (t > warp) break;
            unsigned a[3][4];
            load_a<TTile>(a, t_t, 16 * warp, 16 * t);
#pragma unroll
            for (int n = 0; n < 4; n += 2) {
                unsigned b[4][3][2];
                load_b_transposed<B>(b, from, n0 + 16 * n, 16 * t);
                load_b_transposed<B>(b + 2, from, n0 + 16 * n + 16, 16 * t);
                mma_split<4>(acc + 2 * n, a, b);
            }
        }
    };
    __syncthreads();
#pragma unroll 1
    for (int e = 0; e < WIDTH; e += 64) {                    // -W = -T beta G k
        multiply(Tile(), k_t, e);
        if (good < count) leave_out(acc, 16 * warp + g, good);
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                unsigned plane[3];
                split_pair(-acc[n][2 * h], -acc[n][2 * h + 1], plane[0], plane[1], plane[2]);
                __nv_bfloat16* to = w_out + Tile::at(16 * warp + g + 8 * h, (e >> 3) + n) + 2 * tig;
#pragma unroll
                for (int x = 0; x < 3; ++x) *reinterpret_cast<unsigned*>(to + x * Tile::kPlane) = plane[x];
            }
    }
    for (int c0 = 0; c0 < vdim; c0 += 64) {                  // U_0 = T beta v
        __syncthreads();
#pragma unroll 1
        for (int c = 0; c < 64; c += 32) {
            share.load(v_src + c0 + c, p.v_stride, good, vdim - c0 - c, v_four);
            if (!share.template store<VTile>(k_t, c >> 3, [&](int r) { return r < good ? beta_s[r] : 0.0f; }))
                Part::take_out<VTile>(k_t, c >> 3, v_bad, 0, c);
        }
        __syncthreads();
        multiply(VTile(), k_t, 0);
        if (v_bad.any) {                                     // (the same for all threads)
            v_bad.mark(acc, 16 * warp + g, 2 * tig);
            __syncthreads();
            v_bad.clear();
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int t = 16 * warp + g + 8 * h;
            if (t >= count) continue;
            float* dst = p.u + (size_t)(begin + t) * p.heads * vdim + (size_t)head * vdim + c0;
#pragma unroll
            for (int n = 0; n < 8; ++n) {
                const int c = 8 * n + 2 * tig;
                if ((vdim & 1) == 0) {
                    if (c0 + c < vdim) *reinterpret_cast<float2*>(dst + c) = make_float2(acc[n][2 * h], acc[n][2 * h + 1]);
                } else {
                    if (c0 + c < vdim) dst[c] = acc[n][2 * h];
                    if (c0 + c + 1 < vdim) dst[c + 1] = acc[n][2 * h + 1];
                }
            }
        }
    }
}

// -------------------------------------------------------------------------------------------------------------- walk
constexpr int kDeltaWalkThreads = 256;
template <int WIDTH> constexpr int kDeltaStages = WIDTH == 64 ? 2 : 1;
template <int WIDTH, int COLUMNS> constexpr int delta_walk_bytes() {
    return (kDeltaStages<WIDTH> * 2 * SplitTile<kChunk, WIDTH>::kElements + SplitTile<WIDTH, COLUMNS>::kElements +
            SplitTile<kChunk, COLUMNS>::kElements) * (int)sizeof(__nv_bfloat16);
}

// The B operands of columns n0 .. n0 + 7 of a tile that lies [k][n], depths k0 .. k0 + 15 and k0 + 16 .. k0 + 31
template <typename T>
__device__ __forceinline__ void load_b_two_deep(unsigned (*b)[3][2], const __nv_bfloat16* tile, int n0, int k0) {
    const __nv_bfloat16* from = tile + T::at(k0 + (threadIdx.x & 31), n0 >> 3);
#pragma unroll
    for (int n = 0; n < 3; ++n) {
        unsigned r[4];
        ldmatrix_x4_trans(r, from + n * T::kPlane);
        b[0][n][0] = r[0]; b[0][n][1] = r[1]; b[1][n][0] = r[2]; b[1][n][1] = r[3];
    }
}
// acc += a b over four depths of 16, the four chains of six side by side
__device__ __forceinline__ void mma_four_deep(float (&acc)[4], const unsigned (&a)[4][3][4], const unsigned (&b)[4][3][2]) {
    constexpr int kA[6] = {2, 0, 1, 1, 0, 0}, kB[6] = {0, 2, 1, 0, 1, 0};
    float d[4][4] = {};
#pragma unroll
    for (int k6 = 0; k6 < 6; ++k6)
#pragma unroll
        for (int x = 0; x < 4; ++x) mma_step(d[x], a[x][kA[k6]], b[x][kB[k6]]);
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[r] += d[x][r];
}

// COLUMNS of S a block: 16, or 32 where that is blocks enough. GENERAL: a decay a key channel, and the state is given what lies
// in `states` of the chunk too.
template <int WIDTH, int COLUMNS, bool GENERAL>
__global__ void __launch_bounds__(kDeltaWalkThreads) delta_walk_kernel(const DeltaChunkArgs p) {
    using Tile = SplitTile<kChunk, WIDTH>;
    using STile = SplitTile<WIDTH, COLUMNS>;
    using UTile = SplitTile<kChunk, COLUMNS>;
    constexpr int kStages = kDeltaStages<WIDTH>;
    constexpr int kAlong = WIDTH / 16, kTiles = COLUMNS / 8 * kAlong / 8;      // of S: warps along the keys, tiles of columns
    constexpr int kUTiles = COLUMNS / 16;                    // of u: tiles of columns a warp
    extern __shared__ __align__(128) __nv_bfloat16 tiles[];
    __shared__ __align__(8) unsigned long long full[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
    const int span = blockIdx.z, head = blockIdx.y, c0 = blockIdx.x * COLUMNS, dim = p.dim, vdim = p.vdim;
    const int first = p.span_first[span], last = p.span_first[span + 1];
    if (first >= last) return;
    const int t_begin = p.chunk_begin[first], t_end = p.chunk_begin[last], chunks = last - first;
    __nv_bfloat16* s_t = tiles + kStages * 2 * Tile::kElements;
    __nv_bfloat16* u_t = s_t + STile::kElements;
    float* s_head = p.state + (long long)p.span_slot[span] * p.slot_stride + (size_t)head * dim * vdim;
    constexpr unsigned kBytes = 2 * Tile::kElements * (unsigned)sizeof(__nv_bfloat16);
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(smem_u32(&full[s]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    __syncthreads();
    int brought = 0;
    auto bring = [&](int i) {                                // thread 0: a chunk's two operands, one behind the other
        if (i >= chunks) return;
        brought = i + 1;
        const unsigned bar = smem_u32(&full[i % kStages]);
        mbar_expect_tx(bar, kBytes);
        bulk_load(smem_u32(tiles + (i % kStages) * 2 * Tile::kElements),
                  p.operands + ((size_t)(first + i) * p.heads + head) * 2 * Tile::kElements, kBytes, bar);
    };
    if (tid == 0)
        for (int s = 0; s < kStages; ++s) bring(s);
    // the warp's parts. S: rows er + g, er + g + 8, columns sc + 8 n + 2 tig, + 1. u: tokens tr + g, + 8, columns uc + ..
    const int er = 16 * (warp % kAlong), sc = 8 * kTiles * (warp / kAlong);
    const int tr = 16 * (warp & 3), uc = 8 * kUTiles * (warp >> 2);
    const bool two = (vdim & 1) == 0;
    float s[kTiles][4];
    auto put = [&](__nv_bfloat16* tile, int at, int plane, float x, float y) {
        unsigned h, m, l;
        split_pair(x, y, h, m, l);
        *reinterpret_cast<unsigned*>(tile + at) = h;
        *reinterpret_cast<unsigned*>(tile + at + plane) = m;
        *reinterpret_cast<unsigned*>(tile + at + 2 * plane) = l;
    };
    auto put_s = [&] {
#pragma unroll
        for (int n = 0; n < kTiles; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                put(s_t, STile::at(er + g + 8 * h, (sc >> 3) + n) + 2 * tig, STile::kPlane, s[n][2 * h], s[n][2 * h + 1]);
    };
#pragma unroll
    for (int n = 0; n < kTiles; ++n)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int e = er + g + 8 * (r >> 1), c = c0 + sc + 8 * n + 2 * tig + (r & 1);
            s[n][r] = e < dim && c < vdim ? s_head[(size_t)e * vdim + c] : 0.0f;
        }
    put_s();
    float add[kTiles][4] = {}, keeps[2] = {1.0f, 1.0f};      // general: of the chunk to come
    float next[kUTiles][4], next_keep = 0.0f;                      // U_0 of the chunk to come, its decay
    // Where the thread's rows of S and u of a chunk lie: from one chunk to the next by a constant step. (Made anew from the chunk's
    // number for every access they cost the walk a twentieth, the generalised rule's a tenth.)
    const size_t s_step = (size_t)p.heads * dim * vdim, u_step = (size_t)kChunk * p.heads * vdim;
    float* s_rows = p.states + (((size_t)first * p.heads + head) * dim + er + g) * vdim + c0 + sc + 2 * tig;
    float* u_rows = p.u + (size_t)(t_begin + tr + g) * p.heads * vdim + (size_t)head * vdim + c0 + uc + 2 * tig;
    const size_t s_eight = (size_t)8 * vdim, u_eight = (size_t)8 * p.heads * vdim;
    const int s_left = vdim - (c0 + sc + 2 * tig), u_left = vdim - (c0 + uc + 2 * tig);      // columns from the thread's first on
    auto fetch = [&](const float* src, bool row, int left) {
        if (!row || left <= 0) return make_float2(0.0f, 0.0f);
        if (two) return *reinterpret_cast<const float2*>(src);
        return make_float2(src[0], left > 1 ? src[1] : 0.0f);
    };
    auto store = [&](float* dst, bool row, int left, float x, float y) {
        if (!row || left <= 0) return;
        if (two) *reinterpret_cast<float2*>(dst) = make_float2(x, y);
        else {
            dst[0] = x;
            if (left > 1) dst[1] = y;
        }
    };
    auto ask = [&](int i, const float* u_src, const float* s_src) {      // (the rows of chunk i)
        if (i >= chunks) return;
        const int count = min(kChunk, t_end - (t_begin + i * kChunk));
#pragma unroll
        for (int n = 0; n < kUTiles; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 x = fetch(u_src + h * u_eight + 8 * n, tr + g + 8 * h < count, u_left - 8 * n);
                next[n][2 * h] = x.x;
                next[n][2 * h + 1] = x.y;
            }
        if (!GENERAL) {
            next_keep = p.cum[(size_t)(t_begin + i * kChunk + count - 1) * p.heads + head].x;
            return;
        }
        const size_t rows = ((size_t)(first + i) * p.heads + head) * dim;
#pragma unroll
        for (int h = 0; h < 2; ++h) keeps[h] = er + g + 8 * h < dim ? p.total[rows + er + g + 8 * h] : 0.0f;
#pragma unroll
        for (int n = 0; n < kTiles; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float2 x = fetch(s_src + h * s_eight + 8 * n, er + g + 8 * h < dim, s_left - 8 * n);
                add[n][2 * h] = x.x;
                add[n][2 * h + 1] = x.y;
            }
    };
    ask(0, u_rows, s_rows);
    auto odd_first = [](unsigned (*b)[3][2]) {               // the second tile of eight columns in the first's place
#pragma unroll
        for (int n = 0; n < 3; ++n) {
            b[0][n][0] = b[1][n][0];
            b[0][n][1] = b[1][n][1];
        }
    };
    // Key channels up to 64 and 16 columns: the chain of a chunk is two products deep, and what a warp multiplies S and u with
    // does not wait for them. -W of the next chunk and G k of this one are in registers before the barriers that S and u come
    // through, and the four depths of a product are four chains side by side. 32 heads of 64 x 64, 2,048 tokens: 62.4 us before,
    // 54.5 with it and the constant steps (the generalised rule 67.6 and 58.6); of a chunk's 1.7 us the products are 0.5, what is
    // left without products, loads and stores 0.5.
    constexpr bool kHeld = WIDTH == 64 && COLUMNS == 16;
    static_assert(!kHeld || (kTiles == 1 && kUTiles == 1 && kStages == 2), "");
    unsigned held[kHeld ? 4 : 1][3][4];
    bool ok = true;
    auto hold_w = [&](int i) {                               // (chunk i's operands, once they are there)
        if constexpr (kHeld) {
            ok = mbar_wait(smem_u32(&full[i % kStages]), (i / kStages) & 1);
#pragma unroll
            for (int x = 0; x < 4; ++x) load_a<Tile>(held[x], tiles + (i % kStages) * 2 * Tile::kElements, tr, 16 * x);
        }
    };
    hold_w(0);
    ok = __syncthreads_and(ok);
    int i = 0;
    for (; i < chunks && ok; ++i, s_rows += s_step, u_rows += u_step) {
        const int count = min(kChunk, t_end - (t_begin + i * kChunk));
        const __nv_bfloat16* w_t = tiles + (i % kStages) * 2 * Tile::kElements;
        const __nv_bfloat16* k_t = w_t + Tile::kElements;
        float u[kUTiles][4];
#pragma unroll
        for (int n = 0; n < kUTiles; ++n)
#pragma unroll
            for (int r = 0; r < 4; ++r) u[n][r] = next[n][r];
        const float keep = expf(next_keep);
        float given[kTiles][4], kept[2] = {keeps[0], keeps[1]};
#pragma unroll
        for (int n = 0; n < kTiles; ++n)
#pragma unroll
            for (int r = 0; r < 4; ++r) given[n][r] = add[n][r];
        ask(i + 1, u_rows + u_step, s_rows + s_step);
#pragma unroll
        for (int n = 0; n < kTiles; ++n)                     // the state before the chunk
#pragma unroll
            for (int h = 0; h < 2; ++h)
                store(s_rows + h * s_eight + 8 * n, er + g + 8 * h < dim, s_left - 8 * n, s[n][2 * h], s[n][2 * h + 1]);
        if constexpr (kHeld) {
            unsigned b[4][3][2];
            load_b_two_deep<STile>(b, s_t, uc, 0);
            load_b_two_deep<STile>(b + 2, s_t, uc, 32);
            mma_four_deep(u[0], held, b);
#pragma unroll
            for (int x = 0; x < 4; ++x) load_a_transposed<Tile>(held[x], k_t, er, 16 * x);
        } else {
        ok = __syncthreads_and(mbar_wait(smem_u32(&full[i % kStages]), (i / kStages) & 1));
        if (!ok) break;
#pragma unroll
        for (int e = 0; e < WIDTH; e += 32) {                // u = U_0 - W S
            float d[2][kUTiles][4] = {};
            unsigned a[2][3][4], b[2][2][3][2];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                load_a<Tile>(a[x], w_t, tr, e + 16 * x);
                load_b_transposed<STile>(b[x], s_t, uc & ~15, e + 16 * x);
                if (kUTiles == 1 && (uc & 8)) odd_first(b[x]);
            }
            constexpr int kA[6] = {2, 0, 1, 1, 0, 0}, kB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
            for (int k6 = 0; k6 < 6; ++k6)
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int n = 0; n < kUTiles; ++n) mma_step(d[x][n], a[x][kA[k6]], b[x][n][kB[k6]]);
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int n = 0; n < kUTiles; ++n)
#pragma unroll
                    for (int r = 0; r < 4; ++r) u[n][r] += d[x][n][r];
        }
        }
#pragma unroll
        for (int n = 0; n < kUTiles; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int t = tr + g + 8 * h, c = uc + 8 * n + 2 * tig;
                put(u_t, UTile::at(t, c >> 3) + 2 * tig, UTile::kPlane, u[n][2 * h], u[n][2 * h + 1]);
            }
        __syncthreads();
#pragma unroll
        for (int n = 0; n < kUTiles; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                store(u_rows + h * u_eight + 8 * n, tr + g + 8 * h < count, u_left - 8 * n, u[n][2 * h], u[n][2 * h + 1]);
        float sum[kTiles][4] = {};
        if constexpr (kHeld) {
            unsigned b[4][3][2];
            load_b_two_deep<UTile>(b, u_t, sc, 0);
            load_b_two_deep<UTile>(b + 2, u_t, sc, 32);
            mma_four_deep(sum[0], held, b);
            if (i + 1 < chunks) hold_w(i + 1);
        } else {
#pragma unroll
        for (int t = 0; t < kChunk; t += 32) {               // S = G S + sum_j G k_j u_j^T
            float d[2][kTiles][4] = {};
            unsigned a[2][3][4], b[2][(kTiles + 1) & ~1][3][2];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                load_a_transposed<Tile>(a[x], k_t, er, t + 16 * x);
#pragma unroll
                for (int n = 0; n < kTiles; n += 2) load_b_transposed<UTile>(b[x] + n, u_t, (sc & ~15) + 8 * n, t + 16 * x);
                if (kTiles == 1 && (sc & 8)) odd_first(b[x]);
            }
            constexpr int kA[6] = {2, 0, 1, 1, 0, 0}, kB[6] = {0, 2, 1, 0, 1, 0};
#pragma unroll
            for (int k6 = 0; k6 < 6; ++k6)
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int n = 0; n < kTiles; ++n) mma_step(d[x][n], a[x][kA[k6]], b[x][n][kB[k6]]);
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int n = 0; n < kTiles; ++n)
#pragma unroll
                    for (int r = 0; r < 4; ++r) sum[n][r] += d[x][n][r];
        }
        }
#pragma unroll
        for (int n = 0; n < kTiles; ++n)
#pragma unroll
            for (int r = 0; r < 4; ++r) s[n][r] = fmaf(GENERAL ? kept[r >> 1] : keep, s[n][r], GENERAL ? sum[n][r] + given[n][r] : sum[n][r]);
        put_s();
        // the operands have been used; the state is there
        if constexpr (kHeld) ok = __syncthreads_and(ok);
        else __syncthreads();
        if (tid == 0 && ok) bring(i + kStages);
    }
    if (!ok) {                             // a copy did not come: chunk i's and those behind it (nothing of the block's is left behind)
        if (tid == 0) {
            atomicExch(p.error_flag, 71);
            drain_ring(i, brought, kStages,
                       [&](int stage, unsigned parity) { mbar_wait(smem_u32(&full[stage]), parity); });
        }
        return;
    }
#pragma unroll
    for (int n = 0; n < kTiles; ++n)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int e = er + g + 8 * (r >> 1), c = c0 + sc + 8 * n + 2 * tig + (r & 1);
            if (e < dim && c < vdim) s_head[(size_t)e * vdim + c] = s[n][r];
        }
}

// ------------------------------------------------------------------------------------------------- the generalised rule
// S_t = diag(w_t) S_(t-1) - b_t (u_t^T S_(t-1)) + k_t v_t^T, o_t = S_t^T r_t (general_delta_scan.cu has it in chunks of eight
// tokens). With P_i the product of the chunk's decays through token i (a decay is at least 0.545, so 64 of them at least 1e-17:
// quotients of two of them stay within float32, and lose nothing but rounding), u^ = u P_(i-1), r^ = r P_i, k^ = k / P_j, b^ = b /
// P_j, and s_i = u_i^T S_(i-1),
//
//   s_i + sum_(j<i) (u^_i . b^_j) s_j = u^_i^T S_0 + sum_(j<i) (u^_i . k^_j) v_j
//   o_i = r^_i^T S_0 + sum_(j<=i) [ (r^_i . k^_j) v_j - (r^_i . b^_j) s_j ]
//   S_n = diag(P_n) [ S_0 + sum_j k^_j v_j^T - sum_j b^_j s_j^T ]
//
// the same shape: a system's inverse T, W = T u^ and s_0 = T ((u^ . k^) v), the same walk with s = s_0 + W S_0, and read-outs
// with two sets of values. One block a (chunk, head) of 64 channels makes everything that does not wait for the state:
// 146 us at 32 heads of 64 and 2,048 tokens, two blocks an SM (139 before it left out tokens that are not finite, 187 with one
// block an SM); with the walk's 59 and the read-outs' 47 that is 252 us where chunks of eight tokens take 344.
struct GeneralChunkArgs {
    const float* proj; int stride; int r_off, k_off, v_off, a_off;     // columns of a token's row: head h at h * dim
    const float* z; int z_stride;                              // [tokens, heads * dim], before its bias
    const float* w0; const float* a_bias;
    float unit_eps;
    const int* chunk_begin;
    float* r_out;                                              // [tokens, heads * dim]: r^
    float* products; float* products_b;                        // [chunks, heads, 64, 64]: r^.k^, -r^.b^, zero above the diagonal
    __nv_bfloat16* operands;                                   // [chunks, heads, 2]: W, -b^ P_n
    float* written;                                            // [tokens, heads * dim]: s_0
    float* states; float* total;                               // diag(P_n) sum_j k^_j v_j^T; P_n
    int heads, dim;
};

constexpr int kGeneralThreads = 256;
constexpr int kGeneralBytes = 4 * SplitTile<kChunk, 64>::kElements * 2;

__global__ void __launch_bounds__(kGeneralThreads, 2) general_solve_kernel(const GeneralChunkArgs p) {
    using Tile = SplitTile<kChunk, 64>;
    using Share = TileShare<kChunk, 64, kGeneralThreads>;
    constexpr int kUnits = Share::kUnits, kRows = kGeneralThreads / Share::kPieces;
    extern __shared__ __align__(128) __nv_bfloat16 tiles[];
    __shared__ float last_s[4][64];
    __shared__ BadTokens v_bad;
    __shared__ int k_bad;                                    // the first token with a key, removal or decay that is not finite
    chain_release();
    chain_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, tig = lane & 3;
    const int chunk = blockIdx.y, head = blockIdx.x, dim = p.dim;
    v_bad.clear();
    if (tid == 0) k_bad = kChunk;
    const int begin = p.chunk_begin[chunk], count = p.chunk_begin[chunk + 1] - begin;
    if (count <= 0) return;
    __nv_bfloat16* u_t = tiles;                              // at first P, then u^
    __nv_bfloat16* r_t = u_t + Tile::kElements;              // r^, then v, then L, then T's planes
    __nv_bfloat16* k_t = r_t + Tile::kElements;              // k^, then T in float32
    __nv_bfloat16* b_t = k_t + Tile::kElements;              // b^, then (u^ . k^) v
    float* prefix = reinterpret_cast<float*>(u_t);           // [token][channel]
    float* lower = reinterpret_cast<float*>(r_t);
    float* inverse = reinterpret_cast<float*>(k_t);
    const size_t inner = (size_t)p.heads * dim, at_head = (size_t)head * dim;
    const float* rows = p.proj + (size_t)begin * p.stride;
    const int piece = tid % Share::kPieces, c0 = piece * 8;
    auto load = [&](Share& share, int offset) {
        const float* src = rows + offset + at_head;
        share.load(src, p.stride, count, dim, by_fours(src, p.stride, dim));
    };
    Share k, x;
    load(k, p.k_off);
    {
        const float* src = p.z + (size_t)begin * p.z_stride + at_head;
        x.load(src, p.z_stride, count, dim, by_fours(src, p.z_stride, dim));
    }
    float inv[kUnits];
#pragma unroll
    for (int n = 0; n < kUnits; ++n) {
        const int t = tid / Share::kPieces + n * kRows;
        float squares = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            squares = fmaf(k.x[n][j], k.x[n][j], squares);
            const float w0 = c0 + j < dim ? p.w0[at_head + c0 + j] : 0.0f;
            prefix[t * kSolvePitch + c0 + j] = t < count && c0 + j < dim ? channel_decay(x.x[n][j] + w0) : 1.0f;
        }
#pragma unroll
        for (int offset = 1; offset < Share::kPieces; offset <<= 1) squares += __shfl_xor_sync(0xffffffffu, squares, offset);
        inv[n] = 1.0f / sqrtf(squares + p.unit_eps);
    }
    load(x, p.r_off);
    __syncthreads();
    {
        const int e = tid & 63, quarter = tid >> 6;          // products along 16 tokens, then of the quarters before
        float* column = prefix + quarter * 16 * kSolvePitch + e;
        float f = 1.0f;
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            f *= column[t * kSolvePitch];
            column[t * kSolvePitch] = f;
        }
        last_s[quarter][e] = f;
        __syncthreads();
        f = 1.0f;
        for (int q = 0; q < quarter; ++q) f *= last_s[q][e];
#pragma unroll
        for (int t = 0; t < 16; ++t) column[t * kSolvePitch] *= f;
    }
    __syncthreads();
    const size_t at = ((size_t)chunk * p.heads + head);
    __nv_bfloat16* w_out = p.operands + at * 2 * Tile::kElements;
    __nv_bfloat16* b_out = w_out + Tile::kElements;
    Share a;
    load(a, p.a_off);
    float through[kUnits][8], before[kUnits][8], whole[8];
#pragma unroll
    for (int n = 0; n < kUnits; ++n) {
        const int t = tid / Share::kPieces + n * kRows;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            through[n][j] = prefix[t * kSolvePitch + c0 + j];
            before[n][j] = t > 0 ? prefix[(t - 1) * kSolvePitch + c0 + j] : 1.0f;
            whole[j] = prefix[(kChunk - 1) * kSolvePitch + c0 + j];
        }
    }
    if (tid < 64) last_s[0][tid] = prefix[(kChunk - 1) * kSolvePitch + tid];
    __syncthreads();                                         // (u^ takes the place of P)
    auto put = [&](__nv_bfloat16* tile, int t, const float (&y)[8]) {
        unsigned plane[3][4];
#pragma unroll
        for (int j = 0; j < 4; ++j) split_pair(y[2 * j], y[2 * j + 1], plane[0][j], plane[1][j], plane[2][j]);
#pragma unroll
        for (int n = 0; n < 3; ++n)
            *reinterpret_cast<uint4*>(tile + n * Tile::kPlane + Tile::at(t, piece)) = make_uint4(plane[n][0], plane[n][1], plane[n][2], plane[n][3]);
    };
#pragma unroll
    for (int n = 0; n < kUnits; ++n) {
        const int t = tid / Share::kPieces + n * kRows;
        float u[8], r[8], kk[8], b[8], out[8], none = 0.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int c = c0 + j;
            const bool here = t < count && c < dim;
            const float unit = k.x[n][j] * inv[n], back = 1.0f / through[n][j];
            const float bias = c < dim ? p.a_bias[at_head + c] : 0.0f;
            u[j] = unit * before[n][j];
            r[j] = x.x[n][j] * through[n][j];
            kk[j] = k.x[n][j] * back;
            b[j] = here ? sigmoid_of(a.x[n][j] + bias) * unit * back : 0.0f;
            out[j] = -b[j] * whole[j];
            none = fmaf(u[j], 0.0f, fmaf(b[j], 0.0f, none));
            if (here) p.r_out[(size_t)(begin + t) * inner + at_head + c] = r[j];
            if (t == 0 && c < dim) p.total[(size_t)chunk * inner + at_head + c] = whole[j];
        }
        if (none != 0.0f) {                                  // (NaN: the token's key, removal or decay is not finite)
            atomicMin(&k_bad, t);
#pragma unroll
            for (int j = 0; j < 8; ++j) u[j] = 0.0f;
        }
        put(u_t, t, u);
        put(r_t, t, r);
        put(k_t, t, kk);
        put(b_t, t, b);
        put(b_out, t, out);
    }
    __syncthreads();
    const int good = min(count, k_bad);                      // (what is left out, and why: delta_solve_kernel)
    // products: warps 0-3 r^.k^ and u^.k^, warps 4-7 r^.b^ and u^.b^, 16 tokens each
    const int w4 = warp & 3;
    const bool of_b = warp >= 4;
    float acc[8][4];
    auto product = [&](const __nv_bfloat16* left) {
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int r = 0; r < 4; ++r) acc[n][r] = 0.0f;
#pragma unroll 2
        for (int e = 0; e < 64; e += 16) {
            unsigned l[3][4];
            load_a<Tile>(l, left, 16 * w4, e);
#pragma unroll
            for (int n = 0; n < 4; n += 2) {
                if (n > w4) break;
                unsigned b[4][3][2];
                load_b<Tile>(b, of_b ? b_t : k_t, 16 * n, e);
                load_b<Tile>(b + 2, of_b ? b_t : k_t, 16 * n + 16, e);
                mma_split<4>(acc + 2 * n, l, b);
            }
        }
    };
    product(r_t);
    {
        float* dst = (of_b ? p.products_b : p.products) + at * kChunk * kChunk;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int i = 16 * w4 + g + 8 * h, j = 8 * n + 2 * tig;
                const float sign = of_b ? -1.0f : 1.0f;
                *reinterpret_cast<float2*>(dst + i * kChunk + j) =
                    make_float2(j <= i ? sign * acc[n][2 * h] : 0.0f, j + 1 <= i ? sign * acc[n][2 * h + 1] : 0.0f);
            }
    }
    product(u_t);
    __syncthreads();                                         // r^ has been used
    load(x, p.v_off);
    if (!x.template store<Tile>(r_t, 0, Unscaled())) Share::take_out<Tile>(r_t, 0, v_bad, 0, 0);
    __syncthreads();
    if (!of_b) {                                             // (u^ . k^) v
        float y[8][4] = {};
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            if (m > w4) break;
            unsigned l[3][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int n = 2 * m + (q >> 1), i = 16 * w4 + g + 8 * (q & 1), j = 8 * n + 2 * tig;
                split_pair(j < i && i < good ? acc[n][2 * (q & 1)] : 0.0f, j + 1 < i && i < good ? acc[n][2 * (q & 1) + 1] : 0.0f, l[0][q], l[1][q],
                           l[2][q]);
            }
#pragma unroll
            for (int n = 0; n < 4; n += 2) {
                unsigned b[4][3][2];
                load_b_transposed<Tile>(b, r_t, 16 * n, 16 * m);
                load_b_transposed<Tile>(b + 2, r_t, 16 * n + 16, 16 * m);
                mma_split<4>(y + 2 * n, l, b);
            }
        }
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                unsigned plane[3];
                split_pair(y[n][2 * h], y[n][2 * h + 1], plane[0], plane[1], plane[2]);
                __nv_bfloat16* to = b_t + Tile::at(16 * w4 + g + 8 * h, n) + 2 * tig;
#pragma unroll
                for (int q = 0; q < 3; ++q) *reinterpret_cast<unsigned*>(to + q * Tile::kPlane) = plane[q];
            }
    } else {                                                 // diag(P_n) sum_j k^_j v_j^T
        float y[8][4] = {};
#pragma unroll 2
        for (int t = 0; t < kChunk; t += 16) {
            unsigned l[3][4];
            load_a_transposed<Tile>(l, k_t, 16 * w4, t);
#pragma unroll
            for (int n = 0; n < 4; n += 2) {
                unsigned b[4][3][2];
                load_b_transposed<Tile>(b, r_t, 16 * n, t);
                load_b_transposed<Tile>(b + 2, r_t, 16 * n + 16, t);
                mma_split<4>(y + 2 * n, l, b);
            }
        }
        if (v_bad.any) {                                     // (every row of a column with a bad value)
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int r = 0; r < 4; ++r)
                    if (v_bad.first[8 * n + 2 * tig + (r & 1)] < kChunk) y[n][r] = NAN;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int e = 16 * w4 + g + 8 * h;
            if (e >= dim) continue;
            const float f = last_s[0][e];
            float* dst = p.states + (at * dim + e) * dim;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int r = 0; r < 2; ++r)
                    if (8 * n + 2 * tig + r < dim) dst[8 * n + 2 * tig + r] = f * y[n][2 * h + r];
        }
    }
    __syncthreads();                                         // v and k^ have been used
    if (of_b) {
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = 16 * w4 + g + 8 * (r >> 1), j = 8 * n + 2 * tig + (r & 1);
                lower[i * kSolvePitch + j] = j < i && i < good ? acc[n][r] : 0.0f;
            }
    } else {
        for (int i = tid; i < kChunk * kSolvePitch; i += 128) inverse[i] = 0.0f;
    }
    invert(lower, inverse);
    for (int i = tid; i < kChunk * kChunk / 2; i += kGeneralThreads) {         // T's planes (L has been used)
        const int r = i >> 5, c = (i & 31) * 2;
        const float2 y = *reinterpret_cast<const float2*>(inverse + r * kSolvePitch + c);
        unsigned plane[3];
        split_pair(c <= r ? y.x : 0.0f, c + 1 <= r ? y.y : 0.0f, plane[0], plane[1], plane[2]);
#pragma unroll
        for (int n = 0; n < 3; ++n) *reinterpret_cast<unsigned*>(r_t + n * Tile::kPlane + Tile::at(r, c >> 3) + (c & 7)) = plane[n];
    }
    __syncthreads();
    const __nv_bfloat16* right = of_b ? b_t : u_t;           // s_0 = T (u^ . k^) v, W = T u^
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int r = 0; r < 4; ++r) acc[n][r] = 0.0f;
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        if (t > w4) break;
        unsigned l[3][4];
        load_a<Tile>(l, r_t, 16 * w4, 16 * t);
#pragma unroll
        for (int n = 0; n < 4; n += 2) {
            unsigned b[4][3][2];
            load_b_transposed<Tile>(b, right, 16 * n, 16 * t);
            load_b_transposed<Tile>(b + 2, right, 16 * n + 16, 16 * t);
            mma_split<4>(acc + 2 * n, l, b);
        }
    }
    // (s of a token is of the state before it: NaN behind the first bad value)
    if (of_b && v_bad.any) v_bad.mark(acc, 16 * w4 + g, 2 * tig, 1);
    if (!of_b && good < count) leave_out(acc, 16 * w4 + g, good);
#pragma unroll
    for (int n = 0; n < 8; ++n)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int t = 16 * w4 + g + 8 * h, c = 8 * n + 2 * tig;
            if (of_b) {
                if (t >= count) continue;
                float* dst = p.written + (size_t)(begin + t) * inner + at_head + c;
                if (c < dim) dst[0] = acc[n][2 * h];
                if (c + 1 < dim) dst[1] = acc[n][2 * h + 1];
            } else {
                unsigned plane[3];
                split_pair(acc[n][2 * h], acc[n][2 * h + 1], plane[0], plane[1], plane[2]);
                __nv_bfloat16* to = w_out + Tile::at(t, n) + 2 * tig;
#pragma unroll
                for (int q = 0; q < 3; ++q) *reinterpret_cast<unsigned*>(to + q * Tile::kPlane) = plane[q];
            }
        }
}

template <int WIDTH, int COLUMNS, bool GENERAL>
static int launch_delta_walk(const DeltaChunkArgs& p, int spans, cudaStream_t stream) {
    constexpr size_t bytes = (size_t)delta_walk_bytes<WIDTH, COLUMNS>();
    const int status = allow_shared(delta_walk_kernel<WIDTH, COLUMNS, GENERAL>, bytes, "delta_walk");
    if (status != 0) return status;
    // (a plain launch: see the walk of chunk_scan.cuh)
    delta_walk_kernel<WIDTH, COLUMNS, GENERAL><<<dim3((p.vdim + COLUMNS - 1) / COLUMNS, p.heads, spans), kDeltaWalkThreads, bytes, stream>>>(p);
    return check_launch("delta_walk");
}

template <int WIDTH>
static int launch_delta_chunks(const DeltaChunkArgs& p, int chunks, int spans, cudaStream_t stream) {
    constexpr size_t bytes = (size_t)solve_bytes<WIDTH>();
    int status = allow_shared(delta_solve_kernel<WIDTH>, bytes, "delta_solve");
    if (status != 0) return status;
    launch_chained(delta_solve_kernel<WIDTH>, dim3(p.heads, chunks), kSolveThreads, bytes, stream, p);
    if ((status = check_launch("delta_solve")) != 0) return status;
    // A chunk is two products and two barriers deep however few columns a block has: 16 of them while the blocks are no more
    // than the SMs (32 heads of 64 x 64, one span of 2,048 tokens: 128 blocks 54 us, 64 blocks of 32 columns 73 us).
    const long long blocks = (long long)((p.vdim + 15) / 16) * p.heads * spans;
    return blocks <= 148 ? launch_delta_walk<WIDTH, 16, false>(p, spans, stream) : launch_delta_walk<WIDTH, 32, false>(p, spans, stream);
}

}  // namespace celeg_b200

using namespace celeg_b200;

// Bytes of one (chunk, head)'s operands.
CELEG_API int celeg_delta_operand_bytes(int dim) {
    return 2 * 3 * kChunk * (dim <= 64 ? 64 : 128) * (int)sizeof(__nv_bfloat16);
}

// Over the step's spans from rows that celeg_delta_prepare has convolved and normalised; cum: of the scalar decays' kernel
// (celeg_decay_sums). plan: of celeg_chunk_plan with the same max_chunks. Scratch: operands [chunks, heads, celeg_delta_
// operand_bytes], 16-byte aligned; u [tokens, heads * vdim]; states [chunks, heads, dim, vdim]. dim at most 128.
CELEG_API int celeg_delta_chunk_scan(const float* q, int q_stride, const float* k, int k_stride, const float* v, int v_stride,
                                     const float* gates, const float2* cum, void* operands, float* u, float* states, float* out,
                                     float* state, long long slot_stride, const int* span_slot, const int* plan, int max_chunks,
                                     int spans, int chunks, int heads, int kv_heads, int dim, int vdim, float q_scale,
                                     int* error_flag, cudaStream_t stream) {
    CELEG_REQUIRE(spans >= 0 && chunks >= 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dim > 0 && dim <= 128 && vdim > 0,
                  "delta_chunk_scan: invalid sizes spans=%d heads=%d kv_heads=%d dim=%d (at most 128) vdim=%d", spans, heads, kv_heads,
                  dim, vdim);
    CELEG_REQUIRE(chunks <= max_chunks && chunks <= 65535 && spans <= 65535 && heads <= 65535,
                  "delta_chunk_scan: %d chunks of %d, %d spans or %d heads exceed one launch", chunks, max_chunks, spans, heads);
    CELEG_REQUIRE(((size_t)operands & 15) == 0 && error_flag, "delta_chunk_scan: unaligned operands or no error flag");
    if (spans == 0 || chunks == 0) return 0;
    const int* span_first = plan + max_chunks + 1;
    const DeltaChunkArgs d = {k, k_stride, v, v_stride, gates, cum, plan, span_first, (__nv_bfloat16*)operands, u, states, state,
                              slot_stride, span_slot, heads, kv_heads, dim, vdim, error_flag};
    int status = dim <= 64 ? launch_delta_chunks<64>(d, chunks, spans, stream) : launch_delta_chunks<128>(d, chunks, spans, stream);
    if (status != 0) return status;
    ChunkArgs p = {};
    p.q = q; p.q_stride = q_stride; p.k = k; p.k_stride = k_stride; p.v = u; p.v_stride = heads * vdim;
    p.cum = cum; p.q_scale = q_scale;
    p.chunk_begin = plan; p.pieces = 1; p.span_first = span_first; p.spans = spans;
    p.states = states; p.out = out;
    p.heads = heads; p.groups = kv_heads; p.dim = dim; p.vdim = vdim;
    return launch_reads<kChunkScalar>(p, chunks, stream);
}

// The generalised rule over the step's spans. Offsets: columns of r, k, v and the removal rate in a row of proj (float32, rows
// `stride` apart); z: float32 [tokens, heads * dim]. plan: of celeg_chunk_plan with the same max_chunks. Scratch: r_out, written
// [tokens, heads * dim]; products, products_b [chunks, heads, 64, 64]; operands as above; states [chunks, heads, dim, dim];
// total [chunks, heads * dim]. dim at most 64.
CELEG_API int celeg_general_delta_chunk_scan(const float* proj, int stride, int r_off, int k_off, int v_off, int a_off,
                                             const float* z, int z_stride, const float* w0, const float* a_bias, float unit_eps,
                                             float* r_out, float* products, float* products_b, void* operands, float* written,
                                             float* states, float* total, float* out, float* state, long long slot_stride,
                                             const int* span_slot, const int* plan, int max_chunks, int spans, int chunks, int heads,
                                             int dim, int* error_flag, cudaStream_t stream) {
    CELEG_REQUIRE(spans >= 0 && chunks >= 0 && heads > 0 && dim > 0 && dim <= 64 && unit_eps > 0.0f,
                  "general_delta_chunk_scan: invalid sizes spans=%d heads=%d dim=%d (at most 64)", spans, heads, dim);
    CELEG_REQUIRE(chunks <= max_chunks && chunks <= 65535 && spans <= 65535 && heads <= 65535,
                  "general_delta_chunk_scan: %d chunks of %d, %d spans or %d heads exceed one launch", chunks, max_chunks, spans, heads);
    CELEG_REQUIRE(((size_t)operands & 15) == 0 && error_flag, "general_delta_chunk_scan: unaligned operands or no error flag");
    if (spans == 0 || chunks == 0) return 0;
    const int* span_first = plan + max_chunks + 1;
    const GeneralChunkArgs first = {proj, stride, r_off, k_off, v_off, a_off, z, z_stride, w0, a_bias, unit_eps, plan, r_out, products,
                                    products_b, (__nv_bfloat16*)operands, written, states, total, heads, dim};
    int status = allow_shared(general_solve_kernel, kGeneralBytes, "general_solve");
    if (status != 0) return status;
    launch_chained(general_solve_kernel, dim3(heads, chunks), kGeneralThreads, kGeneralBytes, stream, first);
    if ((status = check_launch("general_solve")) != 0) return status;
    const DeltaChunkArgs d = {nullptr, 0, nullptr, 0, nullptr, nullptr, plan, span_first, (__nv_bfloat16*)operands, written, states, state,
                              slot_stride, span_slot, heads, heads, dim, dim, error_flag, total};
    const long long blocks = (long long)((dim + 15) / 16) * heads * spans;       // (see launch_delta_chunks)
    status = blocks <= 148 ? launch_delta_walk<64, 16, true>(d, spans, stream) : launch_delta_walk<64, 32, true>(d, spans, stream);
    if (status != 0) return status;
    ChunkArgs p = {};
    p.q = r_out; p.q_stride = heads * dim; p.v = proj + v_off; p.v_stride = stride; p.products = products;
    p.products_b = products_b; p.v_b = written; p.v_b_stride = heads * dim;
    p.chunk_begin = plan; p.pieces = 1; p.span_first = span_first; p.spans = spans;
    p.states = states; p.out = out;
    p.heads = heads; p.groups = heads; p.dim = dim; p.vdim = dim;
    return launch_read<kChunkPair, 64>(p, chunks, 1, stream);
}
