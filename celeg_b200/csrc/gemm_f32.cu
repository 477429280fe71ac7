// True 32-bit matrix product Y[M,N] = X[M,K] * W[N,K]^T (both operands row-major with K
// contiguous, as checkpoints store projection weights): float32 operands, FFMA accumulation in
// ascending k, no tensor cores and no reduced-precision operand mode. Every output element is
// produced by one thread with the same order of additions whatever M is, so a row's result
// does not depend on what else is in the batch.
//
// celeg has no 32-bit GPU path (its CUDA backend calls cuBLAS with bf16 operands:
// src/backend/cuda/runtime/gemm_dispatcher.cpp:49-64); this kernel is what makes the float32
// model path independent of any library's math mode.
//
// A thread's 4 x 8 patch (4 x 4 in the small tile) takes its floats from shared memory by 16 bytes, multiplies and adds two a packed
// instruction (the same roundings as one by one), and x lies in shared memory twice over (a, a), so that no instruction pairs it up;
// the next 16 of k are on their way into registers meanwhile. 400 rows, 6,176 columns, k = 2,048: 381 us (26.6 TFLOP/s of about 70 that
// the FMA pipe gives), 553 with a patch of 4 x 4, single products and loads behind a barrier; 490 x 64 68 us, before 147.
#include "common.cuh"

namespace celeg_b200 {

constexpr int kTileK = 16;

__device__ __forceinline__ unsigned long long fma_pair(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// A tile of TM x TN by (TM / PM) x (TN / PN) threads; thread (ty, tx) owns rows ty PM .., and of the columns PN / 4 runs of four, a
// run of all tx side by side. VEC: rows begin at multiples of 16 bytes and k is one of four.
template <int TM, int TN, int PM, int PN, bool VEC>
__global__ void __launch_bounds__((TM / PM) * (TN / PN)) gemm_f32_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                                         float* __restrict__ y, int m, int n, int k, int ldx,
                                                                         int ldw, int ldy, int accumulate) {
    constexpr int kThreads = (TM / PM) * (TN / PN), kAcross = TN / PN, kRuns = PN / 4;
    constexpr int kXQuads = TM * kTileK / 4 / kThreads, kWQuads = TN * kTileK / 4 / kThreads;      // loads a thread
    static_assert(kXQuads * kThreads * 4 == TM * kTileK && kWQuads * kThreads * 4 == TN * kTileK && kThreads % 32 == 0, "");
    __shared__ __align__(16) float2 xs[2][kTileK][TM + 2];    // (a, a)
    __shared__ __align__(16) float ws[2][kTileK][TN + 4];
    const int tid = threadIdx.x, tx = tid % kAcross, ty = tid / kAcross;
    const int row0 = blockIdx.y * TM, col0 = blockIdx.x * TN;
    float4 xq[kXQuads], wq[kWQuads];
    auto fetch = [&](const float* base, int ld, int row, int rows, int at) {
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (row >= rows) return v;
        const float* src = base + (size_t)row * ld + at;
        if (VEC) {
            if (at < k) v = *reinterpret_cast<const float4*>(src);
        } else {
            if (at < k) v.x = src[0];
            if (at + 1 < k) v.y = src[1];
            if (at + 2 < k) v.z = src[2];
            if (at + 3 < k) v.w = src[3];
        }
        return v;
    };
    // unit u of a tile: row u / 4, elements 4 (u % 4) .. of the 16: four lanes read a row's 64 bytes
    auto load = [&](int k0) {
#pragma unroll
        for (int i = 0; i < kXQuads; ++i) xq[i] = fetch(x, ldx, row0 + (tid + i * kThreads) / 4, m, k0 + (tid & 3) * 4);
#pragma unroll
        for (int i = 0; i < kWQuads; ++i) wq[i] = fetch(w, ldw, col0 + (tid + i * kThreads) / 4, n, k0 + (tid & 3) * 4);
    };
    auto put = [&](int buffer) {
        const int kk = (tid & 3) * 4;
#pragma unroll
        for (int i = 0; i < kXQuads; ++i) {
            const int r = (tid + i * kThreads) / 4;
            xs[buffer][kk][r] = make_float2(xq[i].x, xq[i].x);
            xs[buffer][kk + 1][r] = make_float2(xq[i].y, xq[i].y);
            xs[buffer][kk + 2][r] = make_float2(xq[i].z, xq[i].z);
            xs[buffer][kk + 3][r] = make_float2(xq[i].w, xq[i].w);
        }
#pragma unroll
        for (int i = 0; i < kWQuads; ++i) {
            const int r = (tid + i * kThreads) / 4;
            ws[buffer][kk][r] = wq[i].x;
            ws[buffer][kk + 1][r] = wq[i].y;
            ws[buffer][kk + 2][r] = wq[i].z;
            ws[buffer][kk + 3][r] = wq[i].w;
        }
    };
    unsigned long long acc[PM][PN / 2];                       // (0.0f, 0.0f) each
#pragma unroll
    for (int i = 0; i < PM; ++i)
#pragma unroll
        for (int j = 0; j < PN / 2; ++j) acc[i][j] = 0ull;
    load(0);
    put(0);
    __syncthreads();
    int buffer = 0;
    for (int k0 = 0; k0 < k; k0 += kTileK, buffer ^= 1) {
        const bool more = k0 + kTileK < k;
        if (more) load(k0 + kTileK);
#pragma unroll
        for (int kk = 0; kk < kTileK; ++kk) {
            ulonglong2 a[PM / 2], b[kRuns];
#pragma unroll
            for (int i = 0; i < PM / 2; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(&xs[buffer][kk][ty * PM + 2 * i]);
#pragma unroll
            for (int j = 0; j < kRuns; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(&ws[buffer][kk][j * 4 * kAcross + tx * 4]);
#pragma unroll
            for (int i = 0; i < PM; ++i)
#pragma unroll
                for (int j = 0; j < kRuns; ++j) {
                    const unsigned long long both = i & 1 ? a[i / 2].y : a[i / 2].x;
                    acc[i][2 * j] = fma_pair(both, b[j].x, acc[i][2 * j]);
                    acc[i][2 * j + 1] = fma_pair(both, b[j].y, acc[i][2 * j + 1]);
                }
        }
        if (more) put(buffer ^ 1);                           // (the other buffer's readers are behind the last barrier)
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < PM; ++i) {
        const int gr = row0 + ty * PM + i;
        if (gr >= m) continue;
#pragma unroll
        for (int j = 0; j < PN / 2; ++j) {
            const int gc = col0 + (j / 2) * 4 * kAcross + tx * 4 + (j & 1) * 2;
            const float two[2] = {__uint_as_float((unsigned)acc[i][j]), __uint_as_float((unsigned)(acc[i][j] >> 32))};
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                if (gc + r >= n) continue;
                float* dst = y + (size_t)gr * ldy + gc + r;
                *dst = accumulate ? *dst + two[r] : two[r];
            }
        }
    }
}

template <int TM, int TN, int PM, int PN>
static void launch_gemm_f32(const float* x, const float* w, float* y, int m, int n, int k, int ldx, int ldw, int ldy, int accumulate,
                            cudaStream_t stream) {
    const bool vec = k % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (((size_t)x | (size_t)w) & 15) == 0;
    auto kernel = vec ? gemm_f32_kernel<TM, TN, PM, PN, true> : gemm_f32_kernel<TM, TN, PM, PN, false>;
    kernel<<<dim3((n + TN - 1) / TN, (m + TM - 1) / TM), (TM / PM) * (TN / PN), 0, stream>>>(x, w, y, m, n, k, ldx, ldw, ldy, accumulate);
}

}  // namespace celeg_b200

using namespace celeg_b200;

CELEG_API int celeg_gemm_f32(const float* x, const float* w, float* y, int m, int n, int k, int ldx, int ldw,
                             int ldy, int accumulate, cudaStream_t stream) {
    CELEG_REQUIRE(m >= 0 && n > 0 && k > 0 && ldx >= k && ldw >= k && ldy >= n,
                  "gemm_f32: invalid sizes m=%d n=%d k=%d ldx=%d ldw=%d ldy=%d", m, n, k, ldx, ldw, ldy);
    if (m == 0) return 0;
    // Tiles of 64 x 64 where they give every SM work; few rows and narrow matrices in tiles of 32 x 32 (k is never cut: an element
    // is one thread's sum in ascending k). In 64 and in 32, us: 500 x 10,304, k 2,048 673 and 1,012; 400 x 2,048, k 2,048 (224 tiles)
    // 163 and 176; 300 x 1,024, k 1,024 (80) 52 and 52; 200 x 768, k 768 (48) 39 and 30; 490 x 64, k 2,048 (8) 99 and 68; 8 x 6,144,
    // k 2,048 (96) 97 and 76. Patches of 8 x 8 in tiles of 64 x 128 are level with the first where they fill the GPU and slower
    // elsewhere.
    const long long tiles = (long long)((m + 63) / 64) * ((n + 63) / 64);
    CELEG_REQUIRE((m + 63) / 64 <= 65535, "gemm_f32: %d rows exceed one launch", m);      // (so many take the larger tiles)
    if (tiles >= 148) launch_gemm_f32<64, 64, 4, 8>(x, w, y, m, n, k, ldx, ldw, ldy, accumulate, stream);
    else launch_gemm_f32<32, 32, 4, 4>(x, w, y, m, n, k, ldx, ldw, ldy, accumulate, stream);
    return check_launch("gemm_f32");
}
