// C[M,N] = X[M,K] * W[N,K]^T in bf16 for up to 32 rows of X and weights of a few megabytes: the products of a decode step.
//
// Such a product is bound by latencies, not by its bytes (8 MB are 1.3 us at the copy bandwidth): set-up of barriers, tensor
// memory and tensor maps, and K slices that meet in a workspace, put the tcgen05 kernel of gemm_tc.cu at 9 to 12 us.  Here a CTA
// owns 8 NT features outright: its warps take slices of K and meet once in shared memory, in order, so nothing crosses a CTA and
// the sums do not depend on arrival.  Weights go from memory straight into the registers of the tensor-core instruction: a
// sum over k may visit k in any order, so a lane takes 16 consecutive bytes of one weight row and the same 16 of its tokens'
// rows, and calls them the k its fragment holds.  The weights of a warp's first blocks are asked for before the kernel waits for
// its predecessor.  The tensor core cuts off what its accumulator has no bits for, so a warp's products are taken in chains of four
// or eight that join its sum by rounded additions (8 x 128 x 8,192: 4.7e-7 from the 64-bit sum in one chain of 32 a warp, 1.4e-7 in chains; the
// tcgen05 kernel's slices 2.5e-7).
#include "common.cuh"

namespace {
enum { EPI_BF16 = 0, EPI_F32 = 1, EPI_SILU = 2, EPI_RESIDUAL = 3, EPI_RELU2 = 5, EPI_GELU = 6 };   // as in gemm_tc.cu

__device__ __forceinline__ uint4 load_once(const bf16* p) {
    uint4 r;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(r.x), "=r"(r.y), "=r"(r.z), "=r"(r.w) : "l"(p));
    return r;
}
__device__ __forceinline__ void mma(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the sums of one token and two neighbouring features into `out`
__device__ __forceinline__ void store_pair(void* out, int ld_out, int epilogue, int N, int tok, int feat, float s0, float s1) {
    const bool two = feat + 1 < N;
    if (epilogue == EPI_SILU || epilogue == EPI_GELU) {
        float act;
        if (epilogue == EPI_SILU) act = __fdividef(s0, 1.f + __expf(-s0));
        else act = __fdividef(s0, 1.f + __expf(-2.f * (0.7978845608028654f * (s0 + 0.044715f * s0 * s0 * s0))));   // 0.5 (1 + tanh y) = 1 / (1 + e^-2y)
        reinterpret_cast<bf16*>(out)[(size_t)tok * ld_out + (feat >> 1)] = __float2bfloat16_rn(act * s1);
    } else if (epilogue == EPI_F32 || epilogue == EPI_RESIDUAL) {
        float* p = reinterpret_cast<float*>(out) + (size_t)tok * ld_out + feat;
        const bool add = epilogue == EPI_RESIDUAL;
        p[0] = add ? p[0] + s0 : s0;
        if (two) p[1] = add ? p[1] + s1 : s1;
    } else {
        if (epilogue == EPI_RELU2) { s0 = fmaxf(s0, 0.f); s1 = fmaxf(s1, 0.f); s0 *= s0; s1 *= s1; }
        bf16* p = reinterpret_cast<bf16*>(out) + (size_t)tok * ld_out + feat;
        p[0] = __float2bfloat16_rn(s0);
        if (two) p[1] = __float2bfloat16_rn(s1);
    }
}

// MT: tiles of 16 tokens; NT: tiles of 8 features a CTA; U: blocks of 32 k a warp has on the way
template <int MT, int NT, int WARPS, int U>
__global__ void __launch_bounds__(WARPS * 32)
gemm_few_kernel(const bf16* __restrict__ X, const bf16* __restrict__ W, int M, int N, int K, void* __restrict__ out, int ld_out, int epilogue) {
    constexpr int FEATS = 8 * NT, TOKENS = 16 * MT;
    __shared__ float red[WARPS][TOKENS * FEATS];
    pdl_trigger();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int f0 = blockIdx.x * FEATS;
    const int blocks = (K + 31) / 32, per = (blocks + WARPS - 1) / WARPS;
    const int b0 = warp * per, b1 = min(blocks, b0 + per);
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    uint4 w[U][NT];
    auto weights = [&](int b) {
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                const int k = (b + u) * 32 + t * 8, f = f0 + n * 8 + g;
                w[u][n] = b + u < b1 && k < K && f < N ? load_once(W + (size_t)f * K + k) : none;
            }
    };
    weights(b0);
    pdl_wait();
    // rounds of a chain: one, but two of four products where the additions of twice the tokens cost more than a round's loads hide (24 x
    // 2,048 x 8,192: 15.0 us joined every round, 13.8 every second); with four warps K is at most 1,024, sixteen products a warp, which
    // stay one chain
    constexpr int FOLD = MT == 2 && U == 2 ? 2 : 1;
    constexpr bool CHAINS = WARPS > 4;
    float acc[MT][NT][4] = {}, part[MT][NT][4];
    auto join = [&] {
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m][n][e] += part[m][n][e];
    };
    int round = 0;                                           // of the chain under way
    for (int b = b0; b < b1; b += U) {
        uint4 x[U][2 * MT];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int m = 0; m < 2 * MT; ++m) {
                const int k = (b + u) * 32 + t * 8, row = m * 8 + g;
                x[u][m] = b + u < b1 && k < K && row < M ? *reinterpret_cast<const uint4*>(X + (size_t)row * K + k) : none;
            }
        uint4 now[U][NT];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int n = 0; n < NT; ++n) now[u][n] = w[u][n];
        if (b + U < b1) weights(b + U);
        if (CHAINS && round == 0) {
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int n = 0; n < NT; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) part[m][n][e] = 0.f;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    const uint4 lo = x[u][2 * m], hi = x[u][2 * m + 1], v = now[u][n];
                    float (&d)[4] = CHAINS ? part[m][n] : acc[m][n];
                    mma(d, lo.x, hi.x, lo.y, hi.y, v.x, v.y);
                    mma(d, lo.z, hi.z, lo.w, hi.w, v.z, v.w);
                }
        if (CHAINS && (FOLD == 1 || ++round == FOLD)) { join(); round = 0; }
    }
    if (FOLD > 1 && round > 0) join();
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < NT; ++n) {
            float* r = red[warp] + (m * 16 + g) * FEATS + n * 8 + 2 * t;
            *reinterpret_cast<float2*>(r) = make_float2(acc[m][n][0], acc[m][n][1]);
            *reinterpret_cast<float2*>(r + 8 * FEATS) = make_float2(acc[m][n][2], acc[m][n][3]);
        }
    __syncthreads();
    for (int e = tid; e < TOKENS * FEATS / 2; e += WARPS * 32) {         // a pair of features
        const int tok = e / (FEATS / 2), f = (e % (FEATS / 2)) * 2, feat = f0 + f;
        if (tok >= M || feat >= N) continue;
        float s0 = 0.f, s1 = 0.f;
#pragma unroll
        for (int i = 0; i < WARPS; ++i) {
            const float2 p = *reinterpret_cast<const float2*>(red[i] + tok * FEATS + f);
            s0 += p.x;
            s1 += p.y;
        }
        store_pair(out, ld_out, epilogue, N, tok, feat, s0, s1);
    }
}

// K of up to 448: a warp owns 8 features and all of K, its products in one chain of 16 k each in the order of k, which is how one
// accumulator of the tcgen05 kernel takes them: the sums have the same bits.  Bound by the trip to memory of a round of eight steps; the
// next round's weights are on the way while one is multiplied, the first round's before the kernel waits for its predecessor.
constexpr int SHORT_WARPS = 2, SHORT_STEPS = 8;              // warps a CTA; steps of 16 k that are on the way together
template <int MT>
__global__ void __launch_bounds__(SHORT_WARPS * 32)
gemm_short_kernel(const bf16* __restrict__ X, const bf16* __restrict__ W, int M, int N, int K, void* __restrict__ out, int ld_out, int epilogue) {
    pdl_trigger();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int f0 = (blockIdx.x * SHORT_WARPS + (threadIdx.x >> 5)) * 8;
    auto two = [&](const bf16* row, bool valid, int k) { return valid && k < K ? *reinterpret_cast<const uint32_t*>(row + k) : 0u; };
    const bf16* wrow = W + (size_t)min(f0 + g, N - 1) * K;
    uint32_t w[SHORT_STEPS][2], wn[SHORT_STEPS][2];
    auto weights = [&](uint32_t (&to)[SHORT_STEPS][2], int k0) {
#pragma unroll
        for (int s = 0; s < SHORT_STEPS; ++s)
#pragma unroll
            for (int h = 0; h < 2; ++h) to[s][h] = two(wrow, f0 + g < N, k0 + s * 16 + h * 8 + 2 * t);
    };
    weights(w, 0);
    pdl_wait();
    float acc[MT][4] = {};
    for (int k0 = 0; k0 < K; k0 += SHORT_STEPS * 16) {
        uint32_t x[SHORT_STEPS][MT][4];
#pragma unroll
        for (int s = 0; s < SHORT_STEPS; ++s)
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = m * 16 + g + (e & 1) * 8;
                    x[s][m][e] = two(X + (size_t)min(row, M - 1) * K, row < M, k0 + s * 16 + (e >> 1) * 8 + 2 * t);
                }
        weights(wn, k0 + SHORT_STEPS * 16);
#pragma unroll
        for (int s = 0; s < SHORT_STEPS; ++s)
#pragma unroll
            for (int m = 0; m < MT; ++m) mma(acc[m], x[s][m][0], x[s][m][1], x[s][m][2], x[s][m][3], w[s][0], w[s][1]);
#pragma unroll
        for (int s = 0; s < SHORT_STEPS; ++s) { w[s][0] = wn[s][0]; w[s][1] = wn[s][1]; }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int tok = m * 16 + g + 8 * h, feat = f0 + 2 * t;
            if (tok < M && feat < N) store_pair(out, ld_out, epilogue, N, tok, feat, acc[m][2 * h], acc[m][2 * h + 1]);
        }
}

template <int MT, int NT, int WARPS, int U>
int launch(const void* X, const void* W, int M, int N, int K, void* out, int ld_out, int epilogue, cudaStream_t s) {
    RI_CHECKED(ri_launch(gemm_few_kernel<MT, NT, WARPS, U>, dim3((N + 8 * NT - 1) / (8 * NT)), dim3(WARPS * 32), 0, s, (const bf16*)X, (const bf16*)W, M, N,
                         K, out, ld_out, epilogue));
    return ri_launch_status();
}
}  // namespace

// Which tile, or -1: the tcgen05 kernel is as fast or faster.  Times for 8 rows in a captured chain of products over weights that
// do not stay in L2, this kernel against that one: 128 x 1,024 1.8 against 6.6 us, 1,024 x 1,024 2.3 / 7.0, 1,024 x 4,096 4.2 / 9.2,
// 2,048 x 2,048 4.0 / 8.1, 3,072 x 2,048 7.0 / 9.1, 8,192 x 1,024 5.7 / 9.3, 4,096 x 4,096 11.7 / 13.1, 6,144 x 4,096 14.0 / 16.1,
// 16,384 x 1,024 9.8 / 10.7; 16,384 x 2,048 15.5 / 16.0, but behind a chain kernel, where the other one asks for more of its weights
// ahead, the whole step was 3 % slower; 28,672 x 4,096 48 against 45 (the stream of weights is the bound, and TMA keeps more of it
// on the way).  24 rows: 1,024 x 1,024 3.0 / 9.8, 2,048 x 2,048 4.8 / 11.9, 8,192 x 1,024 8.0 / 11.4, 16,384 x 1,024 14.2 / 12.9.
// Narrow tiles while they are few, 16 features a CTA up to two CTAs an SM, sixteen warps where K is long.
// Up to seven k-blocks of 64 no plan of the tcgen05 kernel cuts K, and a token's sums have the same bits in a step of single tokens, in one
// of fifty and in a prompt: models of such sizes, with experts a rounding away from one another, answer the same however their tokens are
// cut.  The kernel with one chain a sum keeps those bits, where it is faster: 8 x 1,024 x 128 1.6 against 4.0 us, 16 x 4,096 x 128 3.3 / 4.7,
// 16 x 1,024 x 448 3.8 / 6.1, 32 x 2,048 x 256 5.9 / 7.2; but 32 x 1,024 x 448 9.5 / 8.0, 8 x 8,192 x 448 14.8 / 6.1.
RI_API int ri_gemm_few_shape(int M, int N, int K) {
    if (M < 1 || M > 32 || N < 1 || K < 8 || K % 8) return -1;
    const long long weights = (long long)N * K;
    if (K <= 7 * 64) return weights <= (1 << 19) && (M <= 16 || K <= 256) ? 4 : -1;
    if (N <= 1024 && K <= 8192) return 0;
    if (N <= 2 * 16 * ri_device_sms() && weights <= (17 << 20)) return 1;
    if (M <= 16) return weights <= (26 << 20) && K <= 4096 ? 2 : -1;
    return weights <= (8 << 20) && K <= 1024 ? 3 : -1;
}

// As ri_gemm_tc's arguments; X and W on 16-byte boundaries.
RI_API int ri_gemm_few(const void* X, const void* W, int M, int N, int K, void* out, int ld_out, int epilogue, int shape, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (M > 32 || K <= 0 || K % 8) return (int)cudaErrorInvalidValue;
    cudaStream_t s = (cudaStream_t)stream;
#define RI_FEW(NT, WARPS, U) return M <= 16 ? launch<1, NT, WARPS, U>(X, W, M, N, K, out, ld_out, epilogue, s) : launch<2, NT, WARPS, U>(X, W, M, N, K, out, ld_out, epilogue, s)
    switch (shape) {
        case 0: RI_FEW(1, 16, 4);
        case 1: RI_FEW(2, 16, 2);
        case 2: if (M > 16) break; return launch<1, 4, 8, 2>(X, W, M, N, K, out, ld_out, epilogue, s);
        case 3: if (M <= 16) break; return launch<2, 4, 4, 4>(X, W, M, N, K, out, ld_out, epilogue, s);
        case 4: {
            const dim3 grid((N + 8 * SHORT_WARPS - 1) / (8 * SHORT_WARPS)), block(SHORT_WARPS * 32);
            if (M <= 16) RI_CHECKED(ri_launch(gemm_short_kernel<1>, grid, block, 0, s, (const bf16*)X, (const bf16*)W, M, N, K, out, ld_out, epilogue));
            else RI_CHECKED(ri_launch(gemm_short_kernel<2>, grid, block, 0, s, (const bf16*)X, (const bf16*)W, M, N, K, out, ld_out, epilogue));
            return ri_launch_status();
        }
    }
#undef RI_FEW
    return (int)cudaErrorInvalidValue;
}
