// C[M,N] = A[M,K] * W[N,K]^T in true fp32: FMA on CUDA cores, no tensor cores, no TF32.
//
// RustInfer's fp32 matrix product on CUDA is cublasGemmEx with
// CUBLAS_COMPUTE_32F_FAST_TF32 (crates/infer-backend-cuda/src/kernels/matmul/matmul.cu:1807-1834),
// which rounds the inputs to 10 mantissa bits; its exact path is the CPU back end
// (crates/infer-backend-cpu/src/lib.rs:377-430).  This kernel is the exact path on the
// GPU.  Every output element is one chain of multiply-adds over k in ascending order whatever M and N
// are, so a token's result does not depend on the batch it was computed in.
//
// That order leaves the fp32 pipes (70 TFLOP/s measured) as the bound for many tokens and the chain's latency for few; K cannot be
// split.  The tiles below: both operands lie in shared memory as they come, k contiguous, rows padded so that eight rows' 16-byte pieces fall into
// different banks; a thread reads four k of its rows at once (a piece of A serves eight lanes, one of W four), and cp.async keeps
// three blocks of 16 k on the way.
#include "common.cuh"

namespace {
constexpr int BK = 16, PITCH = BK + 4, STAGES = 4;

template <bool VEC>
__device__ __forceinline__ void copy_async(float* smem, const float* gmem, bool valid) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    if constexpr (VEC) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 16 : 0));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(s), "l"(gmem), "r"(valid ? 4 : 0));
}

// BM x BN outputs a CTA, TM x TN a thread: rows tr + i * (BM / TM), columns tc + j * (BN / TN).  A warp is 4 x 8 threads.
// VEC: rows come in aligned fours and K is a multiple of four.
template <int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(BM / TM * (BN / TN))
gemm_f32_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                float* __restrict__ C, int ldc, int M, int N, int K) {
    constexpr int TR = BM / TM, TCOL = BN / TN, THREADS = TR * TCOL, WC = TCOL / 8;
    static_assert(TR % 4 == 0 && TCOL % 8 == 0, "warps of 4 x 8 threads");
    __shared__ __align__(16) float sm[STAGES][(BM + BN) * PITCH];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tr = warp / WC * 4 + lane / 8, tc = warp % WC * 8 + lane % 8;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    constexpr int P = VEC ? BK / 4 : BK;                     // copies a row
    auto stage = [&](int block) {
        float* to = sm[block % STAGES];
        const int k0 = block * BK;
        for (int e = tid; e < (BM + BN) * P; e += THREADS) {
            const int r = e / P, kk = (e % P) * (BK / P);
            const bool is_a = r < BM;
            const int row = is_a ? m0 + r : n0 + r - BM;
            const bool valid = k0 + kk < K && row < (is_a ? M : N);
            const float* from = is_a ? A + (size_t)row * lda : W + (size_t)row * ldw;
            copy_async<VEC>(to + r * PITCH + kk, valid ? from + k0 + kk : A, valid);
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;\n" ::); };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    const int blocks = (K + BK - 1) / BK;
#pragma unroll
    for (int b = 0; b < STAGES - 1; ++b) {
        if (b < blocks) stage(b);
        commit();
    }
    for (int b = 0; b < blocks; ++b) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        if (b + STAGES - 1 < blocks) stage(b + STAGES - 1);
        commit();
        const float* as = sm[b % STAGES] + tr * PITCH;
        const float* ws = sm[b % STAGES] + (BM + tc) * PITCH;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            float4 a[TM], w[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + i * TR * PITCH + kk);
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(ws + j * TCOL * PITCH + kk);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].x, w[j].x, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].y, w[j].y, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].z, w[j].z, acc[i][j]);
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i].w, w[j].w, acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + tr + i * TR;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tc + j * TCOL;
            if (gn < N) C[(size_t)gm * ldc + gn] = acc[i][j];
        }
    }
}

// Many outputs: 64 x 128 a CTA, 8 x 8 a thread.  Shared memory delivers 128 bytes a cycle to registers, whatever lanes share, so a
// thread's tile decides how many multiply-adds a delivered byte feeds: 8 x 4 would need 192 bytes a cycle at the pipes' rate, 8 x 8
// needs 128.  k-major tiles (the copies transpose, four bytes each), and pairs of neighbouring columns in the packed multiply-add,
// which rounds each half as the scalar one does and leaves issue slots for the loads.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 twice(float x) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
__device__ __forceinline__ void fma2(f32x2& d, f32x2 a, f32x2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b)); }

constexpr int WM = 64, WN = 128, WTHREADS = 128, WSTAGES = 3;
__global__ void __launch_bounds__(WTHREADS)
gemm_f32_wide_kernel(const float* __restrict__ A, int lda, const float* __restrict__ W, int ldw,
                     float* __restrict__ C, int ldc, int M, int N, int K) {
    constexpr int AP = WM + 4, WP = WN + 4;
    __shared__ __align__(16) float sm[WSTAGES][BK * (AP + WP)];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tr = warp / 2 * 4 + lane / 8, tc = warp % 2 * 8 + lane % 8;
    const int m0 = blockIdx.y * WM, n0 = blockIdx.x * WN;
    // a thread copies one k of every block: rows tid / BK, + WTHREADS / BK, ...
    const int ck = tid % BK, cr = tid / BK;
    constexpr int STEP = WTHREADS / BK;
    // weights on their way into L2 a few blocks before they are copied, a line a row (128 rows, 128 threads)
    auto ask = [&](int k) {
        if (n0 + tid < N && k < K) asm volatile("prefetch.global.L2 [%0];" ::"l"(W + (size_t)(n0 + tid) * ldw + k));
    };
    auto stage = [&](int block) {
        float* to = sm[block % WSTAGES] + ck * AP;
        const int k = block * BK + ck;
#pragma unroll
        for (int r = 0; r < WM; r += STEP) {
            const bool valid = k < K && m0 + r + cr < M;
            copy_async<false>(to + r + cr, valid ? A + (size_t)(m0 + r + cr) * lda + k : A, valid);
        }
        to = sm[block % WSTAGES] + BK * AP + ck * WP;
#pragma unroll
        for (int r = 0; r < WN; r += STEP) {
            const bool valid = k < K && n0 + r + cr < N;
            copy_async<false>(to + r + cr, valid ? W + (size_t)(n0 + r + cr) * ldw + k : W, valid);
        }
    };
    auto commit = [] { asm volatile("cp.async.commit_group;\n" ::); };
    constexpr int LINE = 32, AHEAD = 8 * LINE;               // floats of a line, and how far ahead it is asked for
    for (int k = 0; k < AHEAD; k += LINE) ask(k);
    pdl_wait();
    f32x2 acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    const int blocks = (K + BK - 1) / BK;
#pragma unroll
    for (int b = 0; b < WSTAGES - 1; ++b) {
        if (b < blocks) stage(b);
        commit();
    }
    for (int b = 0; b < blocks; ++b) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(WSTAGES - 2) : "memory");
        __syncthreads();
        if (b + WSTAGES - 1 < blocks) stage(b + WSTAGES - 1);
        commit();
        if (b % (LINE / BK) == 0) ask(b * BK + AHEAD);
        const float* as = sm[b % WSTAGES] + tr * 4;
        const float* ws = sm[b % WSTAGES] + BK * AP + tc * 4;
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 a0 = *reinterpret_cast<const float4*>(as + kk * AP), a1 = *reinterpret_cast<const float4*>(as + kk * AP + WM / 2);
            const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(ws + kk * WP), w1 = *reinterpret_cast<const ulonglong2*>(ws + kk * WP + WN / 2);
            const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const f32x2 x = twice(av[i]);
                fma2(acc[i][0], x, w0.x);
                fma2(acc[i][1], x, w0.y);
                fma2(acc[i][2], x, w1.x);
                fma2(acc[i][3], x, w1.y);
            }
        }
    }
    pdl_trigger();                                           // not before: a successor's CTAs would crowd the SMs this grid leaves free
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gm = m0 + tr * 4 + (i & 3) + (i >> 2) * (WM / 2);
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int gn = n0 + tc * 4 + (j & 3) + (j >> 2) * (WN / 2);
            const f32x2 p = acc[i][j >> 1];
            if (gn < N) C[(size_t)gm * ldc + gn] = __uint_as_float((uint32_t)(j & 1 ? p >> 32 : p));
        }
    }
}

template <int BM, int BN, int TM, int TN>
int launch(const float* A, int lda, const float* W, int ldw, float* C, int ldc, int M, int N, int K, cudaStream_t s) {
    const bool vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) % 16 == 0;
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM), block(BM / TM * (BN / TN));
    if (vec) RI_CHECKED(ri_launch(gemm_f32_kernel<BM, BN, TM, TN, true>, grid, block, 0, s, A, lda, W, ldw, C, ldc, M, N, K));
    else RI_CHECKED(ri_launch(gemm_f32_kernel<BM, BN, TM, TN, false>, grid, block, 0, s, A, lda, W, ldw, C, ldc, M, N, K));
    return ri_launch_status();
}
}  // namespace

RI_API int ri_gemm_f32(const float* A, int lda, const float* W, int ldw, float* C, int ldc,
                       int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    auto tiles = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    // Few tokens: one output a thread, so that as many chains as possible run side by side (8 x 3,072 x 2,048: 25 us, 155 with the
    // 64 x 64 tiles of 4 x 4 a thread that every product ran on; 16: 41 against 53 us with the next).  Else the widest tile that
    // still gives half of the SMs work (300 x 3,072 x 2,048: 199 us, 383 before; 300 x 2,048: 149, 309; 300 x 16,384: 507, 999),
    // 32 x 64 while their number fills two thirds of the SMs (100 x 3,072 x 1,024: 58 us against 71 and 88 before), and the rest
    // on 32 x 32 (64 x 2,048 x 2,048: 55 us against 72 and 152).
    if (M <= 16) return launch<8, 16, 1, 1>(A, lda, W, ldw, C, ldc, M, N, K, s);
    if (2 * tiles(WM, WN) >= ri_device_sms()) {
        RI_CHECKED(ri_launch(gemm_f32_wide_kernel, dim3((N + WN - 1) / WN, (M + WM - 1) / WM), dim3(WTHREADS), 0, s, A, lda, W, ldw, C, ldc, M, N, K));
        return ri_launch_status();
    }
    if (3 * tiles(32, 64) >= 2 * ri_device_sms()) return launch<32, 64, 4, 4>(A, lda, W, ldw, C, ldc, M, N, K, s);
    return launch<32, 32, 4, 2>(A, lda, W, ldw, C, ldc, M, N, K, s);
}
