// The recurrences with decays over long portions of a prompt, in chunks of 64 tokens as matrix products (compiled with
// recurrent.cu for one key size; key sizes 64 and 128, value sizes that are multiples of 64):
//
//   head    S_t = a_t S_{t-1} + k_t (g_t v_t)^T         o_t = S_t^T q_t      a, g one number a head
//   gated   S_t = diag(alpha_t) S_{t-1} + k_t v_t^T     o_t = S_t^T q_t
//   delta   further down
//
// The walk of recurrent.cu takes a prompt token by token: one request offers heads x value channels of columns, and every
// column's state waits for the last token's.  With D_ij the product of the decays of the tokens j + 1 .. i, a chunk that starts
// from the state S is
//
//   O = (Q * D_i0) S + (Q K^T * D) V                    (D_ij = 0 for j > i)
//   S' = D_end,0 S + (K * D_end,j)^T V
//
// so the chunks' own contributions (K * D)^T V need no state (`chunk_states`, all chunks at once), the state in front of every
// chunk is a sum over chunks, element by element (`chunk_scan`), and the outputs are products again (`chunk_outputs`).
//
// Everything stays 32-bit: a factor is cut into three bf16 pieces whose sum it is, and the six products of pieces above 2^-24
// are added up in fp32 on the tensor cores, the small ones first.  bf16 inputs are one piece.  The products of decays are formed
// by multiplication, never as quotients or through logarithms, so they stay below one and a decay of zero is a zero.  A value
// that is no number keeps out of the products (zero times infinity in a masked place would reach earlier tokens) and makes its
// column's later outputs NaN by itself.  An infinity in a query, a key, a decay or a state is NaN from its place on too: its pieces are
// infinity and what is left of it, where the walk carries it until two of either sign meet.
#include "common.cuh"

#ifndef RI_KDIM
#error "compile with -DRI_KDIM=<key size>"
#endif

namespace {
constexpr int CK = 64;                          // tokens of a chunk
constexpr bool BUILT = RI_KDIM == 64 || RI_KDIM == 128;
}

#if RI_KDIM == 64 || RI_KDIM == 128
namespace {
constexpr int DK = RI_KDIM;
constexpr int KP = DK + 8;                      // bf16 of a padded row: an odd count of 16-byte pieces, ldmatrix meets no conflict
constexpr int QUARTERS = CK / 16;
// States between the kernels lie in blocks of 16 value x 16 key channels, [value block][key block][lane][8]: what a lane of
// m16n8k16 holds of a block, (v, k) (v, k + 8) (v + 8, k) (v + 8, k + 8) and each one's neighbour in k, v = lane / 4, k = 2 (lane % 4),
// is both a lane's accumulators of one product and its operand of the next.
constexpr int KS = DK / 16;                     // key blocks

// The entry and tokens of chunk `index` among the entries that bring at least `least` tokens.
struct Chunk { int entry, t0, n; };
__device__ __forceinline__ int chunks_of(int tokens, int least) { return tokens >= least ? (tokens + CK - 1) / CK : 0; }

// every lane of a warp calls; entry -1: no such chunk
__device__ __forceinline__ Chunk find_chunk(const int* cu_q, int entries, int least, int index) {
    const int lane = threadIdx.x & 31;
    int base = 0;
    for (int e0 = 0; e0 < entries; e0 += 32) {
        const int e = e0 + lane;
        const int begin = e < entries ? cu_q[e] : 0, len = e < entries ? cu_q[e + 1] - begin : 0;
        const int own = chunks_of(len, least);
        int sum = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += up;
        }
        const int at = index - base - (sum - own);           // the chunk's number in this lane's entry
        const unsigned hit = __ballot_sync(0xffffffffu, at >= 0 && at < own);
        if (hit) {
            const int src = __ffs(hit) - 1, a = __shfl_sync(0xffffffffu, at, src);
            Chunk c;
            c.entry = e0 + src;
            c.t0 = __shfl_sync(0xffffffffu, begin, src) + a * CK;
            c.n = min(CK, __shfl_sync(0xffffffffu, len, src) - a * CK);
            return c;
        }
        base += __shfl_sync(0xffffffffu, sum, 31);
    }
    return Chunk{-1, 0, 0};
}
// number of the first chunk of entry `e` (every lane of a warp calls)
__device__ __forceinline__ int first_chunk(const int* cu_q, int e, int least) {
    int sum = 0;
    for (int i = threadIdx.x & 31; i < e; i += 32) sum += chunks_of(cu_q[i + 1] - cu_q[i], least);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return sum;
}

// ---- pieces
__device__ __forceinline__ uint32_t pair_bf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float low_of(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float high_of(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }
// x, y -> their pieces as bf16 pairs, each the rounded rest of the one before: their sum is the number, and what the products
// left out add up to has either sign
__device__ __forceinline__ void cut(float x, float y, uint32_t (&p)[3]) {
    p[0] = pair_bf16(x, y);
    x -= low_of(p[0]); y -= high_of(p[0]);
    p[1] = pair_bf16(x, y);
    p[2] = pair_bf16(x - low_of(p[1]), y - high_of(p[1]));
}
// four neighbours into a tile of P pieces: `tile` points at the first one's place in piece 0, pieces lie `stride` bf16 apart
template <int P>
__device__ __forceinline__ void put4(bf16* tile, size_t stride, float4 x) {
    if constexpr (P == 1) {
        *reinterpret_cast<uint2*>(tile) = make_uint2(pair_bf16(x.x, x.y), pair_bf16(x.z, x.w));
    } else {
        uint32_t lo[3], hi[3];
        cut(x.x, x.y, lo);
        cut(x.z, x.w, hi);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(tile + p * stride) = make_uint2(lo[p], hi[p]);
    }
}
// one number into three tiles
__device__ __forceinline__ void put1(bf16* tile, int stride, float x) {
    uint32_t p[3];
    cut(x, 0.f, p);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<unsigned short*>(tile + i * stride) = (unsigned short)p[i];
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const bf16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    return make_float4(low_of(raw.x), high_of(raw.x), low_of(raw.y), high_of(raw.y));
}
__device__ __forceinline__ float4 times(float4 v, float s) { return make_float4(v.x * s, v.y * s, v.z * s, v.w * s); }
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }

// ---- fragments of m16n8k16
__device__ __forceinline__ void ldsm(uint32_t (&r)[4], const bf16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void ldsm_t(uint32_t (&r)[4], const bf16* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((uint32_t)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// where a lane's ldmatrix row lies in a 16 x 16 block of rows of `ld` bf16
__device__ __forceinline__ int at_a(int lane, int ld) { return (lane & 15) * ld + (lane >> 4) * 8; }                          // A of [m][k]
__device__ __forceinline__ int at_at(int lane, int ld) { return ((lane & 7) + (lane >> 4) * 8) * ld + ((lane >> 3) & 1) * 8; } // A of [k][m], trans
__device__ __forceinline__ int at_b(int lane, int ld) { return ((lane & 7) + (lane >> 4) * 8) * ld + ((lane >> 3) & 1) * 8; }  // B of [n][k]
__device__ __forceinline__ int at_bt(int lane, int ld) { return ((lane & 7) + ((lane >> 3) & 1) * 8) * ld + (lane >> 4) * 8; } // B of [k][n], trans

// d[m][n] += A B over one step of 16: the products of pieces that matter, the small ones first.  The tensor core cuts off what
// its accumulator has no bits for, half a unit of the last place a product on average and always downwards: a chain of them
// into one accumulator was ten times further from the 64-bit sum than the token-by-token walk.  So a step's products start
// from zero and join the sum by one rounded addition.
template <int MT, int NT, int PA, int PB>
__device__ __forceinline__ void products(float (&d)[MT][2 * NT][4], const uint32_t (&a)[PA][MT][4], const uint32_t (&b)[PB][NT][4]) {
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        float x[2 * NT][4] = {};
#pragma unroll
        for (int s = PA + PB - 2; s >= 0; --s) {
            if (s > 2) continue;                             // below 2^-24 of the product
#pragma unroll
            for (int pa = 0; pa < PA; ++pa) {
                const int pb = s - pa;
                if (pb < 0 || pb >= PB) continue;
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    mma(x[2 * n], a[pa][m], b[pb][n][0], b[pb][n][1]);
                    mma(x[2 * n + 1], a[pa][m], b[pb][n][2], b[pb][n][3]);
                }
            }
        }
#pragma unroll
        for (int n = 0; n < 2 * NT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) d[m][n][e] += x[n][e];
    }
}

// Products of a head's decays inside a chunk, by one warp: pre[i] = a_0 .. a_i, suf[j] = a_{j+1} .. a_last; tokens behind the
// chunk's end have decay 1.  Returns the product of all.  In 64 bits: with one fixed decay the roundings of 32-bit products
// all fall the same way, and the next chunk's again.
__device__ __forceinline__ double chunk_products(const float* a, float* pre, float* suf) {
    const int lane = threadIdx.x & 31;
    const double x = a[2 * lane], y = a[2 * lane + 1], xy = x * y;
    double up = xy, down = xy;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, up, o), d = __shfl_down_sync(0xffffffffu, down, o);
        if (lane >= o) up *= u;
        if (lane + o < 32) down *= d;
    }
    double before = __shfl_up_sync(0xffffffffu, up, 1), after = __shfl_down_sync(0xffffffffu, down, 1);
    if (lane == 0) before = 1.0;
    if (lane == 31) after = 1.0;
    if (pre) { pre[2 * lane] = (float)(before * x); pre[2 * lane + 1] = (float)up; }
    if (suf) { suf[2 * lane] = (float)(y * after); suf[2 * lane + 1] = (float)after; }
    return __shfl_sync(0xffffffffu, down, 0);
}

// ------------------------------------------------------------------------------------------------- the chunks' own contributions
// dS[value channel][key channel] of one chunk and a tile of VT value channels of one key head (several heads' where they share
// their keys).  Eight warps, 2 x 4 over 64 value channels at a time.  GATED: a decay a key channel, on the keys; else one a
// head, on the values.  Totals: the products of a chunk's decays, as two floats whose sum is the 64-bit product (head form),
// one a key channel (gated form).
constexpr int ST_THREADS = 256;
template <typename TA, int VT, bool GATED>
constexpr int states_bytes() {
    return ((sizeof(TA) == 2 && !GATED ? 1 : 3) * CK * KP + (GATED ? 1 : 3) * CK * (VT + 8)) * 2 + (GATED ? QUARTERS * DK : 4 * CK) * 4;
}

template <typename TA, int VT, bool GATED>
__global__ void __launch_bounds__(ST_THREADS, 2)
chunk_states_kernel(const TA* __restrict__ k, int k_stride, const TA* __restrict__ v, int v_stride,
                    const float* __restrict__ decay, int a_stride, const float* __restrict__ gain, int g_stride,
                    float* __restrict__ states, float* __restrict__ totals, const int* __restrict__ cu_q, int entries,
                    int least, int H, int dv, int share) {
    constexpr int PK = sizeof(TA) == 2 && !GATED ? 1 : 3, PV = GATED ? 1 : 3, VP = VT + 8;
    static_assert(!GATED || sizeof(TA) == 2, "the gated form takes bf16 values as they come");
    extern __shared__ __align__(16) unsigned char raw[];
    bf16* ks = reinterpret_cast<bf16*>(raw);                 // [PK][CK][KP]
    bf16* vs = ks + PK * CK * KP;                            // [PV][CK][VP]
    float* fs = reinterpret_cast<float*>(vs + PV * CK * VP); // a[2][CK], suf[2][CK], or the quarters' products [4][DK]
    pdl_trigger();
    pdl_wait();
    const Chunk c = find_chunk(cu_q, entries, least, blockIdx.x);
    if (c.entry < 0) return;
    const int kh = blockIdx.y, c0 = blockIdx.z * VT, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int col0 = kh * share * dv + c0;                   // the tile's first column of v
    constexpr int VN = CK * VT / 4 / ST_THREADS;
    if constexpr (!GATED) {
        constexpr int KN = CK * DK / 4 / ST_THREADS;
        float4 kv[KN], vv[VN];
#pragma unroll
        for (int j = 0; j < KN; ++j) {
            const int e = tid + j * ST_THREADS, t = e / (DK / 4), i = (e % (DK / 4)) * 4;
            kv[j] = t < c.n ? load4(k + (size_t)(c.t0 + t) * k_stride + (size_t)kh * DK + i) : zero4();
        }
#pragma unroll
        for (int j = 0; j < VN; ++j) {
            const int e = tid + j * ST_THREADS, t = e / (VT / 4), i = (e % (VT / 4)) * 4;
            vv[j] = t < c.n ? load4(v + (size_t)(c.t0 + t) * v_stride + col0 + i) : zero4();
        }
        const int first_head = kh * share + c0 / dv, heads = VT > dv ? VT / dv : 1;      // at most two
        float* a = fs + (warp & 1) * CK;
        if (warp < heads) {
            for (int t = lane; t < CK; t += 32) a[t] = t < c.n ? decay[(size_t)(c.t0 + t) * a_stride + first_head + warp] : 1.f;
            __syncwarp();
            float* suf = fs + 2 * CK + warp * CK;
            const double total = chunk_products(a, nullptr, suf);
            if (lane == 0 && c0 % dv == 0) {
                float* to = totals + ((size_t)blockIdx.x * H + first_head + warp) * 2;
                const float hi = (float)total;
                to[0] = hi;
                to[1] = (float)(total - (double)hi);
            }
            __syncwarp();
            if (gain)
                for (int t = lane; t < c.n; t += 32) suf[t] *= gain[(size_t)(c.t0 + t) * g_stride + first_head + warp];
        }
#pragma unroll
        for (int j = 0; j < KN; ++j) {
            const int e = tid + j * ST_THREADS, t = e / (DK / 4), i = (e % (DK / 4)) * 4;
            put4<PK>(ks + t * KP + i, CK * KP, kv[j]);
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < VN; ++j) {
            const int e = tid + j * ST_THREADS, t = e / (VT / 4), i = (e % (VT / 4)) * 4, which = heads > 1 ? i / dv : 0;
            put4<PV>(vs + t * VP + i, CK * VP, times(vv[j], fs[2 * CK + which * CK + t]));
        }
    } else {
        uint2 vv[VN];                                        // bf16 values as they come
#pragma unroll
        for (int j = 0; j < VN; ++j) {
            const int e = tid + j * ST_THREADS, t = e / (VT / 4), i = (e % (VT / 4)) * 4;
            vv[j] = t < c.n ? *reinterpret_cast<const uint2*>(v + (size_t)(c.t0 + t) * v_stride + col0 + i) : make_uint2(0u, 0u);
        }
        // a key channel of a quarter (16 tokens) a thread: the keys times the decays behind them inside the quarter
        constexpr int PASSES = QUARTERS * DK / ST_THREADS;
        float kk[PASSES][16];
#pragma unroll
        for (int p = 0; p < PASSES; ++p) {
            const int unit = tid + p * ST_THREADS, ch = unit % DK, r = unit / DK;
            float a[16];
#pragma unroll
            for (int t = 0; t < 16; ++t) {
                const bool in = r * 16 + t < c.n;
                const size_t at = (size_t)(c.t0 + r * 16 + t);
                a[t] = in ? decay[at * a_stride + (size_t)kh * DK + ch] : 1.f;
                kk[p][t] = in ? to_f32<TA>(k[at * k_stride + (size_t)kh * DK + ch]) : 0.f;
            }
            float f = 1.f;
#pragma unroll
            for (int t = 15; t >= 0; --t) { kk[p][t] *= f; f *= a[t]; }
            fs[r * DK + ch] = f;
        }
        __syncthreads();
#pragma unroll
        for (int p = 0; p < PASSES; ++p) {
            const int unit = tid + p * ST_THREADS, ch = unit % DK, r = unit / DK;
            float f = 1.f;
            for (int m = r + 1; m < QUARTERS; ++m) f *= fs[m * DK + ch];
            if (r == 0 && c0 == 0) totals[((size_t)blockIdx.x * H + kh) * DK + ch] = f * fs[ch];
#pragma unroll
            for (int t = 0; t < 16; ++t) put1(ks + (r * 16 + t) * KP + ch, CK * KP, kk[p][t] * f);
        }
#pragma unroll
        for (int j = 0; j < VN; ++j) {
            const int e = tid + j * ST_THREADS, t = e / (VT / 4), i = (e % (VT / 4)) * 4;
            *reinterpret_cast<uint2*>(vs + t * VP + i) = vv[j];
        }
    }
    __syncthreads();
    constexpr int NT = DK / 64;                              // blocks of 16 key channels a warp
    const int n0 = (warp & 3) * (16 * NT);
    float* to = states + ((size_t)blockIdx.x * H * dv + col0) * DK;
#pragma unroll 1
    for (int half = 0; half < VT / 64; ++half) {
        const int m0 = half * 64 + (warp >> 2) * 32;
        float d[2][2 * NT][4] = {};
#pragma unroll
        for (int t0 = 0; t0 < CK; t0 += 16) {
            uint32_t fa[PV][2][4], fb[PK][NT][4];
#pragma unroll
            for (int p = 0; p < PV; ++p)
#pragma unroll
                for (int m = 0; m < 2; ++m) ldsm_t(fa[p][m], vs + p * CK * VP + t0 * VP + m0 + m * 16 + at_at(lane, VP));
#pragma unroll
            for (int p = 0; p < PK; ++p)
#pragma unroll
                for (int n = 0; n < NT; ++n) ldsm_t(fb[p][n], ks + p * CK * KP + t0 * KP + n0 + n * 16 + at_bt(lane, KP));
            products<2, NT, PV, PK>(d, fa, fb);
        }
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < NT; ++n) {
                float* x = to + ((size_t)(m0 / 16 + m) * KS + n0 / 16 + n) * 256 + lane * 8;
                *reinterpret_cast<float4*>(x) = make_float4(d[m][2 * n][0], d[m][2 * n][1], d[m][2 * n + 1][0], d[m][2 * n + 1][1]);
                *reinterpret_cast<float4*>(x + 4) = make_float4(d[m][2 * n][2], d[m][2 * n][3], d[m][2 * n + 1][2], d[m][2 * n + 1][3]);
            }
    }
}

// ------------------------------------------------------------------------------------------------- the state in front of every chunk
// A lane's eight numbers of one block a thread, the chunks of its entry in order: cuts[chunk] becomes the state the chunk starts
// from, in pieces ([chunk][head][piece][block][lane]), the entry's slot the state behind the last.
constexpr int SCAN_AHEAD = 8;                   // chunks whose loads are in flight together
constexpr int SCAN_THREADS = 128;
template <bool GATED>
__global__ void __launch_bounds__(SCAN_THREADS)
chunk_scan_kernel(const float* __restrict__ states, const float* __restrict__ totals, bf16* __restrict__ cuts,
                  float* __restrict__ state, const int* __restrict__ cu_q, const int* __restrict__ state_slots, int least,
                  int H, int dv) {
    pdl_trigger();
    pdl_wait();
    const int b = blockIdx.y;
    const int count = chunks_of(cu_q[b + 1] - cu_q[b], least);
    if (count == 0) return;
    const int base = first_chunk(cu_q, b, least);
    const size_t one = (size_t)dv * DK, per = H * one, at = ((size_t)blockIdx.x * SCAN_THREADS + threadIdx.x) * 8;
    if (at >= per) return;
    const int h = (int)(at / one), lane = threadIdx.x & 31;
    const int block = (int)(at % one / 256), v0 = block / KS * 16 + (lane >> 2), i = block % KS * 16 + (lane & 3) * 2;
    float* own = state + (size_t)state_slots[b] * per + ((size_t)h * dv + v0) * DK + i;
    float2 S[4];                                             // (v0, i), (v0, i + 8), (v0 + 8, i), (v0 + 8, i + 8)
#pragma unroll
    for (int j = 0; j < 4; ++j) S[j] = *reinterpret_cast<const float2*>(own + (j >> 1) * 8 * DK + (j & 1) * 8);
    for (int c0 = 0; c0 < count; c0 += SCAN_AHEAD) {
        float4 x[SCAN_AHEAD][2];
        float2 a[GATED ? SCAN_AHEAD : 1][2], t[GATED ? 1 : SCAN_AHEAD];
#pragma unroll
        for (int j = 0; j < SCAN_AHEAD; ++j) {
            const size_t chunk = base + min(c0 + j, count - 1);
            x[j][0] = load4(states + chunk * per + at);
            x[j][1] = load4(states + chunk * per + at + 4);
            if constexpr (GATED) {
                const float* p = totals + (chunk * H + h) * DK + i;
                a[j][0] = *reinterpret_cast<const float2*>(p);
                a[j][1] = *reinterpret_cast<const float2*>(p + 8);
            } else {
                t[j] = *reinterpret_cast<const float2*>(totals + (chunk * H + h) * 2);
            }
        }
#pragma unroll
        for (int j = 0; j < SCAN_AHEAD; ++j)
            if (c0 + j < count) {
                uint32_t p[4][3];
#pragma unroll
                for (int n = 0; n < 4; ++n) cut(S[n].x, S[n].y, p[n]);
                bf16* to = cuts + ((size_t)(base + c0 + j) * H + h) * 3 * one + at % one;
#pragma unroll
                for (int n = 0; n < 3; ++n) *reinterpret_cast<uint4*>(to + n * one) = make_uint4(p[0][n], p[1][n], p[2][n], p[3][n]);
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const float4 xx = x[j][n >> 1];
                    const float u = n & 1 ? xx.z : xx.x, w = n & 1 ? xx.w : xx.y;
                    if constexpr (GATED) {
                        S[n] = make_float2(fmaf(a[j][n & 1].x, S[n].x, u), fmaf(a[j][n & 1].y, S[n].y, w));
                    } else {
                        const float hi = t[j].x, lo = t[j].y;
                        S[n] = make_float2(fmaf(hi, S[n].x, fmaf(lo, S[n].x, u)), fmaf(hi, S[n].y, fmaf(lo, S[n].y, w)));
                    }
                }
            }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(own + (j >> 1) * 8 * DK + (j & 1) * 8) = S[j];
}

// ------------------------------------------------------------------------------------------------- outputs
// The outputs of one chunk for `heads` heads of one key head, two CTAs an SM.  A warp owns a block of 16 value channels for MH
// quarters of the tokens and works for itself: queries, scores and values, cut up, come from shared memory, the state's pieces
// straight from memory in the order of the fragments, a step ahead, so that no tile of the state is waited for.
constexpr int OUT_THREADS = 256;
constexpr int AP = CK + 8;
constexpr int OUT_V = 128, VP = OUT_V + 8;      // value channels of a CTA of the gated form
struct OutLayout {                              // offsets in bf16, then floats
    static constexpr int q = 0, a = q + 3 * CK * KP;         // queries; keys, later the scores, and behind them the values
    static constexpr int k = a, v = a + 3 * CK * AP;
    static constexpr int end = 3 * CK * KP > 3 * CK * (AP + 64) ? a + 3 * CK * KP : v + 3 * CK * 64;
    static constexpr int floats = 5 * CK + 4 * 16 * 16 + 64;
    static constexpr int bytes = end * 2 + floats * 4, gated_bytes = (v + CK * VP) * 2;
};

__device__ __forceinline__ void cp16(bf16* smem, const bf16* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}

__device__ __forceinline__ void cp8(bf16* smem, const bf16* gmem, bool there) {      // not there: zeros
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem), "r"(there ? 8 : 0));
}

// The values of a warp's 16 channels as fragments of a quarter of the tokens.  A value that is no number is left out and its
// token noted: `bad` is the first such token of the columns lane / 4 and lane / 4 + 8.
struct StagedValues {                                        // bf16, in shared memory
    const bf16* at;                                          // [CK][VP] at the warp's first channel
    __device__ __forceinline__ void take(int quarter, uint32_t (&b)[1][1][4], int (&bad)[2]) {
        const int lane = threadIdx.x & 31;
        ldsm_t(b[0][0], at + quarter * 16 * VP + at_bt(lane, VP));
#pragma unroll
        for (int r = 3; r >= 0; --r) {
            const int t = quarter * 16 + 2 * (lane & 3) + (r & 1) * 8;
            if ((b[0][0][r] & 0x7f800000u) == 0x7f800000u) { bad[r >> 1] = min(bad[r >> 1], t + 1); b[0][0][r] &= 0xffffu; }
            if ((b[0][0][r] & 0x7f80u) == 0x7f80u) { bad[r >> 1] = min(bad[r >> 1], t); b[0][0][r] &= 0xffff0000u; }
        }
    }
};
struct GainedValues {                                        // three pieces in shared memory, 64 channels a row, 16 bytes at i ^ row % 8
    const bf16* at;
    int col;                                                 // the warp's first channel
    const int* noted;                                        // [64] the first such token of every channel
    __device__ __forceinline__ void take(int quarter, uint32_t (&b)[3][1][4], int (&bad)[2]) {
        const int lane = threadIdx.x & 31, t = quarter * 16 + (lane & 15);
#pragma unroll
        for (int p = 0; p < 3; ++p) ldsm_t(b[p][0], at + p * CK * 64 + t * 64 + (((col >> 3) + (lane >> 4)) ^ (t & 7)) * 8);
        bad[0] = noted[col + (lane >> 2)];
        bad[1] = noted[col + (lane >> 2) + 8];
    }
};

// The outputs of a warp's 16 value channels, tokens 16 first .. 16 (first + MH) - 1: pre: the decays from the chunk's start, null
// where the queries carry them; cuts: the channels' blocks of the state in front of the chunk, pieces dv * DK apart; out: the
// channels of the chunk's first token.
template <int PQ, int PV, int MH, typename Values>
__device__ __forceinline__ void value_columns(const bf16* qs, const bf16* as, const float* pre, int tokens, int first, const bf16* cuts,
                                              size_t one, Values& values, float q_scale, float* out, int out_stride) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
    float o[MH][1][2][4] = {};
    uint4 next[3];
#pragma unroll
    for (int p = 0; p < 3; ++p) next[p] = *reinterpret_cast<const uint4*>(cuts + p * one + lane * 8);
#pragma unroll
    for (int k = 0; k < KS; ++k) {                           // from the state in front of the chunk
        uint32_t fb[3][1][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            fb[p][0][0] = next[p].x; fb[p][0][1] = next[p].y; fb[p][0][2] = next[p].z; fb[p][0][3] = next[p].w;
            if (k + 1 < KS) next[p] = *reinterpret_cast<const uint4*>(cuts + p * one + (k + 1) * 256 + lane * 8);
        }
#pragma unroll
        for (int m = 0; m < MH; ++m) {
            uint32_t fa[PQ][1][4];
#pragma unroll
            for (int p = 0; p < PQ; ++p) ldsm(fa[p][0], qs + p * CK * KP + (first + m) * 16 * KP + k * 16 + at_a(lane, KP));
            products<1, 1, PQ, 3>(o[m], fa, fb);
        }
    }
    if (pre) {
#pragma unroll
        for (int m = 0; m < MH; ++m) {
            const float p0 = pre[(first + m) * 16 + g], p1 = pre[(first + m) * 16 + g + 8];
#pragma unroll
            for (int n = 0; n < 2; ++n) { o[m][0][n][0] *= p0; o[m][0][n][1] *= p0; o[m][0][n][2] *= p1; o[m][0][n][3] *= p1; }
        }
    }
    int bad[2] = {CK, CK};
#pragma unroll
    for (int k = 0; k < QUARTERS; ++k) {                     // from the chunk's own tokens
        if (k >= first + MH) continue;
        uint32_t fb[PV][1][4];
        values.take(k, fb, bad);
#pragma unroll
        for (int m = 0; m < MH; ++m) {
            if (first + m < k) continue;
            uint32_t fa[3][1][4];
#pragma unroll
            for (int p = 0; p < 3; ++p) ldsm(fa[p][0], as + p * CK * AP + (first + m) * 16 * AP + k * 16 + at_a(lane, AP));
            products<1, 1, 3, PV>(o[m], fa, fb);
        }
    }
    const bool any_bad = __any_sync(0xffffffffu, min(bad[0], bad[1]) < CK);
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        int b0 = CK, b1 = CK;
        if (any_bad) {                                       // later outputs of such a column are NaN
            int b = min(bad[n], __shfl_xor_sync(0xffffffffu, bad[n], 1));
            b = min(b, __shfl_xor_sync(0xffffffffu, b, 2));
            b0 = __shfl_sync(0xffffffffu, b, 8 * t4);
            b1 = __shfl_sync(0xffffffffu, b, 8 * t4 + 4);
        }
#pragma unroll
        for (int m = 0; m < MH; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int t = (first + m) * 16 + g + 8 * r;
                if (t < tokens)
                    *reinterpret_cast<float2*>(out + (size_t)t * out_stride + n * 8 + t4 * 2) =
                        make_float2(t >= b0 ? __int_as_float(0x7fc00000) : o[m][0][n][2 * r] * q_scale,
                                    t >= b1 ? __int_as_float(0x7fc00000) : o[m][0][n][2 * r + 1] * q_scale);
            }
    }
}

template <typename TA>
__global__ void __launch_bounds__(OUT_THREADS, 2)
head_chunk_outputs_kernel(const TA* __restrict__ q, int q_stride, const TA* __restrict__ k, int k_stride,
                          const TA* __restrict__ v, int v_stride, const float* __restrict__ decay, int a_stride,
                          const float* __restrict__ gain, int g_stride, float q_scale, const bf16* __restrict__ cuts,
                          float* __restrict__ out, const int* __restrict__ cu_q, int entries, int least, int H, int dv,
                          int share, int heads) {
    constexpr int PQ = sizeof(TA) == 2 ? 1 : 3;              // pieces of queries and keys
    extern __shared__ __align__(16) unsigned char raw[];
    bf16* sm = reinterpret_cast<bf16*>(raw);
    bf16 *qs = sm + OutLayout::q, *ks = sm + OutLayout::k, *as = sm + OutLayout::a;
    float* a = reinterpret_cast<float*>(sm + OutLayout::end);
    float *pre = a + CK, *pre_in = pre + CK, *suf_in = pre_in + CK;      // from the chunk's start; inside a quarter: from its start, to its end
    float* gains = suf_in + CK;
    float* dq = gains + CK;                                  // [4][16][16] decays inside a quarter
    int* noted = reinterpret_cast<int*>(dq + QUARTERS * 256);            // [64]
    bf16* vs = sm + OutLayout::v;
    pdl_trigger();
    pdl_wait();
    const Chunk c = find_chunk(cu_q, entries, least, blockIdx.x);
    if (c.entry < 0) return;
    const int h0 = blockIdx.y * heads, kh = h0 / share;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = warp >> 1, wn = warp & 1;
    const int g = lane >> 2, t4 = lane & 3;
    // a head's decays and gains, a token a thread, one head ahead
    float next_a = 1.f, next_g = 1.f;
    auto ask = [&](int h) {
        if (tid < c.n) {
            next_a = decay[(size_t)(c.t0 + tid) * a_stride + h];
            if (gain) next_g = gain[(size_t)(c.t0 + tid) * g_stride + h];
        }
    };
    {
        constexpr int KN = CK * DK / 4 / OUT_THREADS;
        float4 x[KN], y[KN];
#pragma unroll
        for (int j = 0; j < KN; ++j) {
            const int e = tid + j * OUT_THREADS, t = e / (DK / 4), i = (e % (DK / 4)) * 4;
            x[j] = t < c.n ? load4(q + (size_t)(c.t0 + t) * q_stride + (size_t)kh * DK + i) : zero4();
            y[j] = t < c.n ? load4(k + (size_t)(c.t0 + t) * k_stride + (size_t)kh * DK + i) : zero4();
        }
        ask(h0);
#pragma unroll
        for (int j = 0; j < KN; ++j) {
            const int e = tid + j * OUT_THREADS, t = e / (DK / 4), i = (e % (DK / 4)) * 4;
            put4<PQ>(qs + t * KP + i, CK * KP, x[j]);
            put4<PQ>(ks + t * KP + i, CK * KP, y[j]);
        }
    }
    __syncthreads();
    // scores of this warp's 16 tokens against 32 keys (none where every key is later)
    float s[1][4][4] = {};
    if (2 * wn <= wm) {
#pragma unroll
        for (int k0 = 0; k0 < DK; k0 += 16) {
            uint32_t fa[PQ][1][4], fb[PQ][2][4];
#pragma unroll
            for (int p = 0; p < PQ; ++p) {
                ldsm(fa[p][0], qs + p * CK * KP + wm * 16 * KP + k0 + at_a(lane, KP));
#pragma unroll
                for (int n = 0; n < 2; ++n) ldsm(fb[p][n], ks + p * CK * KP + (wn * 32 + n * 16) * KP + k0 + at_b(lane, KP));
            }
            products<1, 2, PQ, PQ>(s, fa, fb);
        }
    }
    for (int hh = 0; hh < heads; ++hh) {
        const int h = h0 + hh;
        const bf16* from = cuts + ((size_t)blockIdx.x * H + h) * 3 * dv * DK;
        const TA* own = v + (size_t)c.t0 * v_stride + (size_t)h * dv;
        constexpr int VN = CK * 64 / 4 / OUT_THREADS;        // 64 channels' values: fours a thread
        float4 x[VN];
        auto ask_values = [&](int c0) {
#pragma unroll
            for (int j = 0; j < VN; ++j) {
                const int e = tid + j * OUT_THREADS, t = e >> 4;
                x[j] = t < c.n ? load4(own + (size_t)t * v_stride + c0 + (e & 15) * 4) : zero4();
            }
        };
        auto put_values = [&]() {
#pragma unroll
            for (int j = 0; j < VN; ++j) {
                const int e = tid + j * OUT_THREADS, t = e >> 4, i = (e & 15) * 4;
                float4 y = gain ? times(x[j], gains[t]) : x[j];
                const float most = 3.402823466e38f;
                if (!(fabsf(y.x) <= most) || !(fabsf(y.y) <= most) || !(fabsf(y.z) <= most) || !(fabsf(y.w) <= most)) {
                    if (!(fabsf(y.x) <= most)) { atomicMin(noted + i, t); y.x = 0.f; }
                    if (!(fabsf(y.y) <= most)) { atomicMin(noted + i + 1, t); y.y = 0.f; }
                    if (!(fabsf(y.z) <= most)) { atomicMin(noted + i + 2, t); y.z = 0.f; }
                    if (!(fabsf(y.w) <= most)) { atomicMin(noted + i + 3, t); y.w = 0.f; }
                }
                put4<3>(vs + t * 64 + (((i >> 3) ^ (t & 7)) << 3) + (i & 7), CK * 64, y);
            }
        };
        ask_values(0);
        if (tid < CK) a[tid] = tid < c.n ? next_a : 1.f;
        __syncthreads();                                     // the last head's (or the keys') readers are done, the decays are there
        if (tid < CK) { gains[tid] = next_g; noted[tid] = CK; }
        if (hh + 1 < heads) ask(h + 1);
        if (warp == 7) chunk_products(a, pre, nullptr);
        if (warp >= 2 && warp < 4) {                         // 64 threads: the column of key j inside its quarter
            const int j = tid - 64, r = j >> 4, jj = j & 15;
            double f = 1.0;
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                if (i > jj) f *= a[r * 16 + i];
                dq[(r * 16 + i) * 16 + jj] = (float)f;
            }
            suf_in[j] = (float)f;
        }
        if (warp >= 4 && warp < 6) {
            const int i = tid - 128, r = i >> 4;
            double f = 1.0;
            for (int m = r * 16; m <= i; ++m) f *= a[m];
            pre_in[i] = (float)f;
        }
        __syncthreads();
        // scores times decays, cut up: the quarters on the diagonal by the table, those left of it by their factors; a later
        // key's weight is zero by choice, not by product
        if (2 * wn <= wm) {
#pragma unroll
            for (int n = 0; n < 4; ++n) {
                const int cq = wn * 2 + (n >> 1);            // the keys' quarter
                if (cq > wm) continue;
                float between = 1.f;
                for (int m = cq + 1; m < wm; ++m) between *= pre_in[m * 16 + 15];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const int col = wn * 32 + n * 8 + t4 * 2, row = wm * 16 + g + 8 * r;
                    float x, y;
                    if (cq == wm) {
                        const float* d = dq + row * 16 + (col & 15);
                        x = col <= row ? s[0][n][2 * r] * d[0] : 0.f;
                        y = col + 1 <= row ? s[0][n][2 * r + 1] * d[1] : 0.f;
                    } else {
                        const float w = pre_in[row] * between;
                        x = s[0][n][2 * r] * (w * suf_in[col]);
                        y = s[0][n][2 * r + 1] * (w * suf_in[col + 1]);
                    }
                    uint32_t p[3];
                    cut(x, y, p);
#pragma unroll
                    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(as + i * CK * AP + row * AP + col) = p[i];
                }
            }
        }
        for (int c0 = 0; c0 < dv; c0 += 64) {
            if (c0 > 0) {
                __syncthreads();                             // the last channels' values are read
                if (tid < 64) noted[tid] = CK;
                __syncthreads();
            }
            put_values();
            if (c0 + 64 < dv) ask_values(c0 + 64);
            __syncthreads();
            GainedValues values{vs, (warp & 3) * 16, noted};
            value_columns<PQ, 3, 2>(qs, as, pre, c.n, warp / 4 * 2, from + (c0 / 16 + (warp & 3)) * KS * 256, (size_t)dv * DK, values, q_scale,
                                    out + (size_t)c.t0 * H * dv + (size_t)h * dv + c0 + (warp & 3) * 16, H * dv);
        }
    }
}

// Sums of 16 values over a warp's lanes: at every offset a lane hands half of its values to its partner and keeps the other
// half's sums.  The lane gets value `lane >> 1` (both lanes of a pair).
__device__ __forceinline__ float sums16(float (&x)[16]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 16, o = 16; n > 1; n /= 2, o /= 2) {
        const bool upper = lane & o;
#pragma unroll
        for (int i = 0; i < n / 2; ++i) {
            const float send = upper ? x[i] : x[i + n / 2], keep = upper ? x[i + n / 2] : x[i];
            x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    return x[0] + __shfl_xor_sync(0xffffffffu, x[0], 1);
}

// A decay a key channel: the scores cannot be one product.  Inside a quarter (16 tokens) a thread takes a key channel and
// multiplies its way through the pairs of tokens in fp32, and the channels' parts are summed; between quarters r > s the
// decays part at quarter r's start, q_i (a_start .. a_i) on one side and (a_{j+1} .. a_{start-1}) k_j on the other, both below
// one, and the score is a product again, with the keys scaled for each r.
// The scores and the queries from the chunk's start go out in pieces, [chunk][head]{scores [3][CK][CK], queries [3][CK][DK]}, for
// the CTAs that take the chunk's value channels (the scores are most of the work where one CTA makes them for itself).
constexpr int GATED_PARTS = 3 * CK * (CK + DK);
struct ScoreLayout {                            // queries, keys (48 rows) or the scores, floats
    static constexpr int q = 0, k = 3 * CK * KP, end = k + (48 * KP > CK * AP ? 3 * 48 * KP : 3 * CK * AP);
    static constexpr int bytes = end * 2 + QUARTERS * DK * 4;
    static_assert(3 * CK * AP <= end - k && 16 * 144 * 2 <= end - k, "scores and the warps' parts fit where the keys lie");
};
__global__ void __launch_bounds__(OUT_THREADS, 2)
gated_chunk_scores_kernel(const bf16* __restrict__ q, int q_stride, const bf16* __restrict__ k, int k_stride,
                          const float* __restrict__ decay, int a_stride, bf16* __restrict__ parts, const int* __restrict__ cu_q,
                          int entries, int least, int H) {
    constexpr int UNITS = QUARTERS * DK / OUT_THREADS, WQ = DK / 32;     // (channel, quarter) pairs a thread; warps of channels
    extern __shared__ __align__(16) unsigned char raw[];
    bf16* sm = reinterpret_cast<bf16*>(raw);
    bf16 *qs = sm + ScoreLayout::q, *ks = sm + ScoreLayout::k, *as = ks;
    float* qt = reinterpret_cast<float*>(sm + ScoreLayout::end);         // [4][DK] products of a quarter's decays
    float* part = reinterpret_cast<float*>(ks);                          // [4 * WQ][144], before the keys are laid out
    static_assert(QUARTERS * WQ <= 16, "the warps' parts fit");
    pdl_trigger();
    pdl_wait();
    const Chunk c = find_chunk(cu_q, entries, least, blockIdx.x);
    if (c.entry < 0) return;
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float kk[UNITS][16];
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {
        const int unit = tid + u * OUT_THREADS, ch = unit % DK, r = unit / DK;
        float a[16], qq[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            const bool in = r * 16 + t < c.n;
            const size_t at = (size_t)(c.t0 + r * 16 + t);
            a[t] = in ? decay[at * a_stride + (size_t)h * DK + ch] : 1.f;
            qq[t] = in ? to_f32<bf16>(q[at * q_stride + (size_t)h * DK + ch]) : 0.f;
            kk[u][t] = in ? to_f32<bf16>(k[at * k_stride + (size_t)h * DK + ch]) : 0.f;
        }
        // pairs i >= j of the quarter: keys j and 16 - j have 16 queries between them
#pragma unroll
        for (int set = 0; set <= 8; ++set) {
            float x[16];
            float f = kk[u][set];
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                if (i < set) continue;
                if (i > set) f *= a[i];
                x[i - set] = qq[i] * f;
            }
            if (set > 0) {
                const int j = 16 - set;
                float e = set == 8 ? 0.f : kk[u][j];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    if (i < j) continue;
                    if (i > j) e *= a[i];
                    x[i] = qq[i] * e;
                }
            }
            const float sum = sums16(x);
            if ((lane & 1) == 0) part[(unit >> 5) * 144 + set * 16 + (lane >> 1)] = sum;
        }
        float f = 1.f;
#pragma unroll
        for (int t = 0; t < 16; ++t) { f *= a[t]; put1(qs + (r * 16 + t) * KP + ch, CK * KP, qq[t] * f); }   // from the quarter's start
        qt[r * DK + ch] = f;
        f = 1.f;
#pragma unroll
        for (int t = 15; t >= 0; --t) { kk[u][t] *= f; f *= a[t]; }      // to the quarter's end
    }
    __syncthreads();
    // the quarters on the diagonal: the channels' warps in order
    float diag[QUARTERS * 256 / OUT_THREADS];
#pragma unroll
    for (int n = 0; n < QUARTERS * 256 / OUT_THREADS; ++n) {
        const int e = tid + n * OUT_THREADS, b = e >> 8, i = e >> 4 & 15, j = e & 15;
        diag[n] = 0.f;
        if (j <= i) {
            const int at = j <= 8 ? j * 16 + i - j : (16 - j) * 16 + i;
            for (int w = 0; w < WQ; ++w) diag[n] += part[(b * WQ + w) * 144 + at];
        }
    }
    // quarters right of the first: 16 x 8 scores a warp, quarter `to` against the keys of those before it, kept till all are read
    float s[QUARTERS - 1][4];
#pragma unroll
    for (int to = 1; to < QUARTERS; ++to) {
        __syncthreads();                                     // the parts, or the last quarter's keys, are read
#pragma unroll
        for (int u = 0; u < UNITS; ++u) {
            const int unit = tid + u * OUT_THREADS, ch = unit % DK, r = unit / DK;
            if (r < to) {
                float f = 1.f;
                for (int m = r + 1; m < to; ++m) f *= qt[m * DK + ch];
#pragma unroll
                for (int t = 0; t < 16; ++t) put1(ks + (r * 16 + t) * KP + ch, 48 * KP, kk[u][t] * f);
            }
        }
        __syncthreads();
        if (warp < 2 * to) {
            float d[1][2][4] = {};                           // the second half is not used
            const int n0 = warp * 8;
#pragma unroll
            for (int k0 = 0; k0 < DK; k0 += 16) {
                uint32_t fa[3][4], fb[3][2];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    ldsm(fa[p], qs + p * CK * KP + to * 16 * KP + k0 + at_a(lane, KP));
                    const bf16* b = ks + p * 48 * KP + (n0 + (lane >> 2)) * KP + k0 + (lane & 3) * 2;
                    fb[p][0] = *reinterpret_cast<const uint32_t*>(b);
                    fb[p][1] = *reinterpret_cast<const uint32_t*>(b + 8);
                }
                float x[4] = {};
                mma(x, fa[0], fb[2][0], fb[2][1]);
                mma(x, fa[1], fb[1][0], fb[1][1]);
                mma(x, fa[2], fb[0][0], fb[0][1]);
                mma(x, fa[0], fb[1][0], fb[1][1]);
                mma(x, fa[1], fb[0][0], fb[0][1]);
                mma(x, fa[0], fb[0][0], fb[0][1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) d[0][0][e] += x[e];
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) s[to - 1][e] = d[0][0][e];
        }
    }
    __syncthreads();
#pragma unroll
    for (int to = 1; to < QUARTERS; ++to)
        if (warp < 2 * to) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                uint32_t p[3];
                cut(s[to - 1][2 * e], s[to - 1][2 * e + 1], p);
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    *reinterpret_cast<uint32_t*>(as + i * CK * AP + (to * 16 + (lane >> 2) + 8 * e) * AP + warp * 8 + (lane & 3) * 2) = p[i];
            }
        }
#pragma unroll
    for (int n = 0; n < QUARTERS * 256 / OUT_THREADS; ++n) {
        const int e = tid + n * OUT_THREADS, b = e >> 8, i = e >> 4 & 15, j = e & 15;
        put1(as + (b * 16 + i) * AP + b * 16 + j, CK * AP, diag[n]);
    }
#pragma unroll
    for (int u = 0; u < UNITS; ++u) {                        // queries from the chunk's start: the pieces' sum is the number
        const int unit = tid + u * OUT_THREADS, ch = unit % DK, r = unit / DK;
        if (r == 0) continue;
        float f = 1.f;
        for (int m = 0; m < r; ++m) f *= qt[m * DK + ch];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            bf16* x = qs + (r * 16 + t) * KP + ch;
            const float sum = __bfloat162float(x[0]) + (__bfloat162float(x[CK * KP]) + __bfloat162float(x[2 * CK * KP]));
            put1(x, CK * KP, sum * f);
        }
    }
    __syncthreads();
    bf16* to = parts + ((size_t)blockIdx.x * H + h) * GATED_PARTS;
    for (int e = tid; e < 3 * CK * CK / 8; e += OUT_THREADS)             // [piece][row]
        *reinterpret_cast<uint4*>(to + e * 8) = *reinterpret_cast<const uint4*>(as + (e / (CK / 8)) * AP + (e % (CK / 8)) * 8);
    to += 3 * CK * CK;
    for (int e = tid; e < 3 * CK * DK / 8; e += OUT_THREADS)
        *reinterpret_cast<uint4*>(to + e * 8) = *reinterpret_cast<const uint4*>(qs + (e / (DK / 8)) * KP + (e % (DK / 8)) * 8);
}

// OUT_V (MH 4) or all (MH 2) value channels of one chunk and head
template <int MH>
__global__ void __launch_bounds__(OUT_THREADS, 2)
gated_chunk_outputs_kernel(const bf16* __restrict__ parts, const bf16* __restrict__ v, int v_stride, float q_scale,
                           const bf16* __restrict__ cuts, float* __restrict__ out, const int* __restrict__ cu_q, int entries,
                           int least, int H, int dv) {
    extern __shared__ __align__(16) unsigned char raw[];
    bf16* sm = reinterpret_cast<bf16*>(raw);
    constexpr int COLS = 64 * (MH / 2);                      // value channels at a time
    pdl_trigger();
    pdl_wait();
    const Chunk c = find_chunk(cu_q, entries, least, blockIdx.x);
    if (c.entry < 0) return;
    const int h = blockIdx.y, warp = threadIdx.x >> 5, col = warp % (COLS / 16) * 16;
    const bf16* from = cuts + ((size_t)blockIdx.x * H + h) * 3 * dv * DK;
    const bf16* own = parts + ((size_t)blockIdx.x * H + h) * GATED_PARTS;
    for (int e = threadIdx.x; e < 3 * CK * CK / 8; e += OUT_THREADS)
        cp16(sm + OutLayout::a + (e / (CK / 8)) * AP + (e % (CK / 8)) * 8, own + e * 8);
    own += 3 * CK * CK;
    for (int e = threadIdx.x; e < 3 * CK * DK / 8; e += OUT_THREADS)
        cp16(sm + OutLayout::q + (e / (DK / 8)) * KP + (e % (DK / 8)) * 8, own + e * 8);
    bf16* vs = sm + OutLayout::v;
    for (int c0 = blockIdx.z * COLS; c0 < dv; c0 += gridDim.z * COLS) {
        const bf16* src = v + (size_t)c.t0 * v_stride + (size_t)h * dv + c0;
        uint2 x[CK * COLS / 4 / OUT_THREADS];
#pragma unroll
        for (int j = 0; j < CK * COLS / 4 / OUT_THREADS; ++j) {
            const int e = threadIdx.x + j * OUT_THREADS, t = e / (COLS / 4), i = (e % (COLS / 4)) * 4;
            x[j] = t < c.n ? *reinterpret_cast<const uint2*>(src + (size_t)t * v_stride + i) : make_uint2(0u, 0u);
        }
        if (c0 != (int)blockIdx.z * COLS) __syncthreads();   // the last channels' values are read
#pragma unroll
        for (int j = 0; j < CK * COLS / 4 / OUT_THREADS; ++j) {
            const int e = threadIdx.x + j * OUT_THREADS, t = e / (COLS / 4), i = (e % (COLS / 4)) * 4;
            *reinterpret_cast<uint2*>(vs + t * VP + i) = x[j];
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        StagedValues values{vs + col};
        value_columns<3, 1, MH>(sm + OutLayout::q, sm + OutLayout::a, nullptr, c.n, MH == 4 ? 0 : warp / 4 * 2, from + (c0 + col) / 16 * KS * 256,
                                (size_t)dv * DK, values, q_scale, out + (size_t)c.t0 * H * dv + (size_t)h * dv + c0 + col, H * dv);
    }
}

// ------------------------------------------------------------------------------------------------- the delta rule
// delta   S_t = diag(w_t) S_{t-1} - au_t (u_t^T S_{t-1}) + k_t v_t^T      o_t = S_t^T r_t
//
// With d_t = u_t^T S_{t-1} a chunk is the gated form over keys k and values v less keys au and values d, and the d are a
// triangular system: (I + A) d = U S + B V, A_ij = u_i^T D_{i-1,j} au_j and B_ij = u_i^T D_{i-1,j} k_j for j < i.  With T = (I + A)^-1
// and P, Q the scores of r against k and au,
//
//   d = X S + Y V                     X = T U D, Y = T B
//   O = (R D - Q T U D) S + (P - Q Y) V                          as the gated form's outputs: queries R', scores P'
//   S' = D S - (AU D)^T X S + (K D - (AU D)^T Y)^T V
//
// so one kernel makes X, R', P' and each chunk's own contribution for all chunks at once (`delta_chunk_parts`), the scan over the
// chunks takes two products a chunk, d = X S and AU^T d (`delta_chunk_scan`), and the outputs are the gated form's.
//
// The decays part at the chunk's middle: a row carries the product from there to its token, a key the product from its token to
// there, on the other side of the middle the reciprocal.  A term of a score is then a product of two rounded numbers whatever
// their sizes; the host sends only decays here whose products over half a chunk stay far from the ends of fp32 (DELTA_MOST_DECAY).
// (The gated form's decays have no such bound, so its scores part at every quarter and multiply their way inside one.)
//
// 2,444 tokens in four entries, 16 heads of 128 x 128: 296 us with what prepares it (parts some 145, scan 80, outputs 47), where the walk
// takes 395; one entry of 2,048 tokens and 8 heads 163, the walk 678.  The parts are bound by what a CTA's phases wait for (products of a
// few blocks, the inverse: tensor cores a third busy, 10 cycles an instruction and warp), the scan by its products (half of the tensor
// cores' rate, one chunk after the other).  Tried: the parts' next channels asked for ahead (registers; 2 % slower).
constexpr float DELTA_MOST_DECAY = 1.0f;        // of -log w: factors of a middle lie between e^-32 and e^32
constexpr int DP_THREADS = 256;
constexpr int SC = 32, SP = SC + 8;             // channels staged at a time
constexpr int LOWER = 10;                       // 16 x 16 blocks on and under the diagonal of a chunk
struct PartsLayout {                            // bytes
    static constexpr int PF = DK + 4, AF = CK + 4;
    static constexpr int decay = 0, ends = decay + CK * PF * 4, noted = ends + 2 * DK * 4, work = noted + 128;
    static constexpr int stage = work, exch = stage + 4 * 3 * CK * SP * 2, one_end = exch + 16 * SC * 8;
    static constexpr int BLOCKS = LOWER * 3 * 256 * 2;       // three pieces
    static constexpr int a = work, t = a + CK * AF * 4, b = t + BLOCKS, q = b + BLOCKS, p = q + BLOCKS, two_end = p + LOWER * 256 * 4;
    static constexpr int y = a, w = b, v = q;                // later tenants
    static constexpr int bytes = two_end > one_end ? two_end : one_end;
    static_assert(BLOCKS <= CK * AF * 4 && v + CK * VP * 2 <= bytes, "later tenants fit");
};
__device__ __forceinline__ int lower_block(int i, int j) { return i * (i + 1) / 2 + j; }
// A block's row of 16 is two pieces of 16 bytes that change places every fourth row: ldmatrix meets no conflict.
__device__ __forceinline__ const bf16* lane_row(const bf16* block, int lane) {
    const int row = lane & 15;
    return block + row * 16 + (((lane >> 4) ^ (row >> 2 & 1)) << 3);
}
// one block's accumulators into three pieces at `to`
__device__ __forceinline__ void put_block(bf16* to, const float (&d)[2][4], int lane) {
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int row = (lane >> 2) + 8 * r;
            uint32_t x[3];
            cut(d[n][2 * r], d[n][2 * r + 1], x);
#pragma unroll
            for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(to + p * 256 + row * 16 + ((n ^ (row >> 2 & 1)) << 3) + (lane & 3) * 2) = x[p];
        }
}
// d += sum over k = j .. i of left(i, k) right(k, j), blocks on and under the diagonal
__device__ __forceinline__ void block_product(float (&d)[1][2][4], const bf16* left, const bf16* right, int i, int j, int lane) {
    for (int k = j; k <= i; ++k) {
        uint32_t fa[3][1][4], fb[3][1][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            ldsm(fa[p][0], lane_row(left + (lower_block(i, k) * 3 + p) * 256, lane));
            ldsm_t(fb[p][0], lane_row(right + (lower_block(k, j) * 3 + p) * 256, lane));
        }
        products<1, 1, 3, 3>(d, fa, fb);
    }
}
// a warp's blocks, so that the longest sums (i - j + 1 products) are shared out: at most two
__device__ __forceinline__ int warp_blocks(int warp, int which) {        // i * 4 + j, -1: none
    constexpr int first[8] = {12, 8, 13, 4, 9, 14, 15, -1}, second[8] = {-1, -1, -1, 0, 5, 10, -1, -1};
    return which ? second[warp] : first[warp];
}
// 1 / x for x between 2^-60 and 2^60: one step of Newton's method, y + y (1 - x y), from the special-function unit's approximation.  That is off
// by a unit of the last place at the most, so the step leaves its square, 2^-46, and one rounding: half a unit, as the correctly rounded
// __frcp_rn, whose way costs 3 % of a call with keys of 128 and up to 10 % with keys of 64 (16 heads, 2,444 tokens in four entries: 304 us
// against 296, and 180 against 166).
__device__ __forceinline__ float reciprocal(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return fmaf(y, fmaf(-x, y, 1.f), y);
}
__global__ void reciprocal_kernel(const float* x, float* y, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = reciprocal(x[i]);
}
__device__ __forceinline__ bool finite(float x) { return fabsf(x) <= 3.402823466e38f; }

// One chunk and head.  Outputs, all in the order of fragments ([piece][token block][key block][lane][8] for xs and au): xs: X; au: the
// au with their factor to the middle; ends: the decays' products from the middle to the chunk's end and over the whole chunk;
// parts: P' and R' as the gated form's; states: the chunk's own contribution.  From the first token on whose k, u, au or w is no number
// the chunk counts no tokens, and its outputs there and the state behind it are NaN.
__global__ void __launch_bounds__(DP_THREADS, 2)
delta_chunk_parts_kernel(const bf16* __restrict__ r, int r_stride, const bf16* __restrict__ k, int k_stride, const bf16* __restrict__ v, int v_stride,
                         const float* __restrict__ w, const float* __restrict__ u, const float* __restrict__ au, int f_stride,
                         bf16* xs, bf16* aus, float* __restrict__ ends, bf16* __restrict__ parts, float* __restrict__ states,
                         const int* __restrict__ cu_q, int entries, int least, int H, int dv) {
    using L = PartsLayout;
    extern __shared__ __align__(16) unsigned char raw[];
    float* ps = reinterpret_cast<float*>(raw + L::decay);                // [CK][PF]: t < 32: w_{t+1} .. w_31, else w_32 .. w_t
    float* mid = reinterpret_cast<float*>(raw + L::ends);                // [2][DK]: w_0 .. w_31, w_32 .. w_63
    int* noted = reinterpret_cast<int*>(raw + L::noted);
    bf16* stage = reinterpret_cast<bf16*>(raw + L::stage);               // u, r, k, au: [4][3][CK][SP]
    double* exch = reinterpret_cast<double*>(raw + L::exch);             // [16][SC]
    float* as = reinterpret_cast<float*>(raw + L::a);                    // [CK][AF]
    bf16 *ts = reinterpret_cast<bf16*>(raw + L::t), *bs = reinterpret_cast<bf16*>(raw + L::b), *qs = reinterpret_cast<bf16*>(raw + L::q);
    bf16 *ys = reinterpret_cast<bf16*>(raw + L::y), *ws = reinterpret_cast<bf16*>(raw + L::w), *vs = reinterpret_cast<bf16*>(raw + L::v);
    float* pf = reinterpret_cast<float*>(raw + L::p);                    // [LOWER][lane][8]
    pdl_trigger();
    pdl_wait();
    const Chunk c = find_chunk(cu_q, entries, least, blockIdx.x);
    if (c.entry < 0) return;
    const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t4 = lane & 3;
    const size_t unit = (size_t)blockIdx.x * H + h;
    xs += unit * 3 * CK * DK;
    aus += unit * 3 * CK * DK;
    parts += unit * GATED_PARTS;
    // ---- scores: rows u and r against k and au.  A warp takes one of each and two rows of blocks, 3 and 0 or 2 and 1.
    const int rows_of = warp & 1, cols_of = warp >> 1 & 1, long_row = warp < 4 ? 3 : 2, short_row = 3 - long_row;
    float sl[4][1][2][4], ss[2][1][2][4];
    if (tid == 0) *noted = CK;
    __syncthreads();
    int tokens = c.n;
    for (bool again = true; again;) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    sl[j][0][n][e] = 0.f;
                    if (j < 2) ss[j][0][n][e] = 0.f;
                }
#pragma unroll 1
        for (int q0 = 0; q0 < DK; q0 += SC) {
            const int pair = tid & 15, seg = tid >> 4, ch = q0 + 2 * pair;           // two channels, four tokens a thread
            float2 ww[4], uu[4], aa[4];
            uint32_t rr[4], kk[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int t = seg * 4 + i;
                const size_t at = (size_t)(c.t0 + t), col = (size_t)h * DK + ch;
                const bool in = t < tokens;
                ww[i] = in ? *reinterpret_cast<const float2*>(w + at * f_stride + col) : make_float2(1.f, 1.f);
                uu[i] = in ? *reinterpret_cast<const float2*>(u + at * f_stride + col) : make_float2(0.f, 0.f);
                aa[i] = in ? *reinterpret_cast<const float2*>(au + at * f_stride + col) : make_float2(0.f, 0.f);
                rr[i] = in ? *reinterpret_cast<const uint32_t*>(r + at * r_stride + col) : 0u;
                kk[i] = in ? *reinterpret_cast<const uint32_t*>(k + at * k_stride + col) : 0u;
            }
            double px = 1.0, py = 1.0;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                px *= ww[i].x;
                py *= ww[i].y;
            }
            float none = 0.f;                                // stays zero while everything is a number
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                none = fmaf(ww[i].x, 0.f, none); none = fmaf(ww[i].y, 0.f, none); none = fmaf(uu[i].x, 0.f, none); none = fmaf(uu[i].y, 0.f, none);
                none = fmaf(aa[i].x, 0.f, none); none = fmaf(aa[i].y, 0.f, none);
                none = fmaf(low_of(kk[i]), 0.f, none); none = fmaf(high_of(kk[i]), 0.f, none);
            }
            if (!(none == 0.f)) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (!finite(ww[i].x) || !finite(ww[i].y) || !finite(uu[i].x) || !finite(uu[i].y) || !finite(aa[i].x) || !finite(aa[i].y) ||
                        !finite(low_of(kk[i])) || !finite(high_of(kk[i])))
                        atomicMin(noted, seg * 4 + i);
            }
            *reinterpret_cast<double2*>(exch + seg * SC + 2 * pair) = make_double2(px, py);
            __syncthreads();
            // from the middle to this thread's tokens, then token by token away from it (64 bits, rounded once)
            double fx = 1.0, fy = 1.0;
            const bool early = seg < 8;
            for (int m = early ? seg + 1 : 8; m < (early ? 8 : seg); ++m) {
                const double2 e = *reinterpret_cast<const double2*>(exch + m * SC + 2 * pair);
                fx *= e.x;
                fy *= e.y;
            }
            if (seg == 0 || seg == 15) {
                mid[(seg & 1) * DK + ch] = (float)(fx * px);
                mid[(seg & 1) * DK + ch + 1] = (float)(fy * py);
            }
            float2 beyond = make_float2(1.f, 1.f);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = early ? 3 - j : j, t = seg * 4 + i;
                // early: fours from the last to the first
                const float2 wi = early ? ww[3 - j] : ww[j], ui = early ? uu[3 - j] : uu[j], ai = early ? aa[3 - j] : aa[j];
                const uint32_t ri = early ? rr[3 - j] : rr[j], ki = early ? kk[3 - j] : kk[j];
                const double nx = fx * wi.x, ny = fy * wi.y;             // with this token's decay
                const float bx = (float)fx, by = (float)fy, ax = (float)nx, ay = (float)ny;
                // the product between the middle and the state behind token t, and that between the middle and the state in front of it
                const float2 behind = early ? make_float2(bx, by) : make_float2(ax, ay), front = early ? make_float2(ax, ay) : make_float2(bx, by);
                *reinterpret_cast<float2*>(ps + t * L::PF + ch) = behind;
                // (early: what lies in front of a token lies behind the next)
                const float2 inv = early && j > 0 ? beyond : make_float2(reciprocal(behind.x), reciprocal(behind.y));
                if (early) beyond = make_float2(reciprocal(front.x), reciprocal(front.y));
                const float2 row = early ? inv : behind, col = early ? behind : inv;
                const float2 urow = early ? beyond : front;
                uint32_t x[3];
                bf16* to = stage + t * SP + 2 * pair;
                auto put = [&](int which, float p0, float p1) {
                    cut(p0, p1, x);
#pragma unroll
                    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(to + (which * 3 + p) * CK * SP) = x[p];
                };
                put(0, ui.x * urow.x, ui.y * urow.y);
                put(1, low_of(ri) * row.x, high_of(ri) * row.y);
                put(2, low_of(ki) * col.x, high_of(ki) * col.y);
                put(3, ai.x * col.x, ai.y * col.y);
                fx = nx;
                fy = ny;
            }
            __syncthreads();
            // u and au as operands of the later products
#pragma unroll
            for (int j = 0; j < 6; ++j) {
                const int id = warp + 8 * j, p = id % 3, blk = id / 3 % 8, which = id / 24;      // 8 blocks of 16 x 16, 3 pieces, 2 arrays
                uint32_t x[4];
                ldsm_t(x, stage + ((which ? 9 : 0) + p) * CK * SP + (blk >> 1) * 16 * SP + (blk & 1) * 16 + at_bt(lane, SP));
                bf16* to = (which ? aus : xs) + p * CK * DK + (((blk >> 1) * KS + q0 / 16 + (blk & 1)) * 32 + lane) * 8;
                *reinterpret_cast<uint4*>(to) = make_uint4(x[0], x[1], x[2], x[3]);
            }
            const bf16 *rows = stage + rows_of * 3 * CK * SP, *cols = stage + (2 + cols_of) * 3 * CK * SP;
#pragma unroll
            for (int k0 = 0; k0 < SC; k0 += 16) {
                uint32_t fl[3][1][4], fs[3][1][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    ldsm(fl[p][0], rows + p * CK * SP + long_row * 16 * SP + k0 + at_a(lane, SP));
                    ldsm(fs[p][0], rows + p * CK * SP + short_row * 16 * SP + k0 + at_a(lane, SP));
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (j > long_row) continue;
                    uint32_t fb[3][1][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) ldsm(fb[p][0], cols + p * CK * SP + j * 16 * SP + k0 + at_b(lane, SP));
                    products<1, 1, 3, 3>(sl[j], fl, fb);
                    if (j < 2 && j <= short_row) products<1, 1, 3, 3>(ss[j], fs, fb);
                }
            }
            __syncthreads();
        }
        again = *noted < tokens;
        if (again) tokens = *noted;                          // once more without the tokens from there on
    }
    const int bad = tokens < c.n ? tokens : CK;
    const float nan = __int_as_float(0x7fc00000);
    // ---- A in fp32, B and Q in pieces, P in fp32
    auto put_scores = [&](int i, int j, float (&d)[1][2][4]) {
        if (rows_of == 0 && cols_of == 1) {
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e)
                    *reinterpret_cast<float2*>(as + (i * 16 + g + 8 * e) * L::AF + j * 16 + n * 8 + t4 * 2) = make_float2(d[0][n][2 * e], d[0][n][2 * e + 1]);
            return;
        }
        if (i == j) {                                        // rows u: earlier tokens; rows r: and the token itself
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int row = g + 8 * (e >> 1), col = n * 8 + t4 * 2 + (e & 1);
                    if (col > row || (rows_of == 0 && col == row)) d[0][n][e] = 0.f;
                }
        }
        const int at = lower_block(i, j);
        if (rows_of == 1 && cols_of == 0) {
            float* to = pf + (at * 32 + lane) * 8;
            *reinterpret_cast<float4*>(to) = make_float4(d[0][0][0], d[0][0][1], d[0][0][2], d[0][0][3]);
            *reinterpret_cast<float4*>(to + 4) = make_float4(d[0][1][0], d[0][1][1], d[0][1][2], d[0][1][3]);
        } else {
            put_block((rows_of ? qs : bs) + at * 3 * 256, d[0], lane);
        }
    };
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j <= long_row) put_scores(long_row, j, sl[j]);
        if (j < 2 && j <= short_row) put_scores(short_row, j, ss[j]);
    }
    __syncthreads();
    // ---- T = (I + A)^-1: blocks of 16 on the diagonal by substitution, then the ones one, two and three blocks below it,
    // T_ij = -T_ii sum of A_ik T_kj over k = j .. i - 1, a warp a block.  Where keys resemble one another the terms of these sums cancel, and
    // sixteen at a time from the tensor cores they lose less than one after another in 32 bits, in less time (304 us a call for 312).
    // Repeated keys of 64 and 128 that hardly decay: the outputs 2.0e-6 and 1.8e-6 from 64 bits where they were 3.5e-6 and 3.4e-6 (the walk
    // 1.0e-6 and 1.1e-6); that decay by 2 % a token 0.8e-6 and 1.0e-6, were 3.4e-6 and 3.5e-6 (0.35e-6); a twentieth of noise in the keys and
    // hardly any decay 1.6e-6, were 1.7e-6 and 1.8e-6 (1.4e-6 and 1.5e-6).  What is left is the scores' own rounding: sums in 64 bits give no less.
    if (tid < CK) {
        float x[16];
        const float* blk = as + (tid >> 4) * 16 * (L::AF + 1);
        const int col = tid & 15;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float s0 = i == col ? 1.f : 0.f, s1 = 0.f;
#pragma unroll
            for (int m = 0; m < 16; ++m) {
                if (m >= i) continue;
                if (m & 1) s1 = fmaf(-blk[i * L::AF + m], x[m], s1);
                else s0 = fmaf(-blk[i * L::AF + m], x[m], s0);
            }
            x[i] = s0 + s1;
        }
        __syncwarp();
        float* to = as + (tid >> 4) * 16 * (L::AF + 1) + col;
#pragma unroll
        for (int i = 0; i < 16; ++i) to[i * L::AF] = (float)x[i];
    }
    __syncthreads();
    for (int e = tid; e < QUARTERS * 128; e += DP_THREADS) {
        const int i = e >> 7, row = (e & 127) >> 3, col = (e & 7) * 2;
        const float2 x = *reinterpret_cast<const float2*>(as + (i * 16 + row) * L::AF + i * 16 + col);
        uint32_t y[3];
        cut(x.x, x.y, y);
#pragma unroll
        for (int p = 0; p < 3; ++p)
            *reinterpret_cast<uint32_t*>(ts + (lower_block(i, i) * 3 + p) * 256 + row * 16 + (((col >> 3) ^ (row >> 2 & 1)) << 3) + (col & 7)) = y[p];
    }
    __syncthreads();
#pragma unroll 1
    for (int below = 1; below < QUARTERS; ++below) {
        const int j = warp, i = warp + below;
        if (i < QUARTERS) {
            uint32_t fa[3][1][4], fb[3][1][4];
            float d[1][2][4] = {}, z[1][2][4] = {};
#pragma unroll 1
            for (int k = j; k < i; ++k) {
                const float* from = as + (i * 16 + g) * L::AF + k * 16 + t4 * 2;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 x = *reinterpret_cast<const float2*>(from + (e & 1) * 8 * L::AF + (e >> 1) * 8);
                    uint32_t y[3];
                    cut(x.x, x.y, y);
#pragma unroll
                    for (int p = 0; p < 3; ++p) fa[p][0][e] = y[p];
                }
#pragma unroll
                for (int p = 0; p < 3; ++p) ldsm_t(fb[p][0], lane_row(ts + (lower_block(k, j) * 3 + p) * 256, lane));
                products<1, 1, 3, 3>(d, fa, fb);
            }
            bf16* to = ts + lower_block(i, j) * 3 * 256;     // the sum, then the block itself
            put_block(to, d[0], lane);
            __syncwarp();
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                ldsm(fa[p][0], lane_row(ts + (lower_block(i, i) * 3 + p) * 256, lane));
                ldsm_t(fb[p][0], lane_row(to + p * 256, lane));
            }
            products<1, 1, 3, 3>(z, fa, fb);
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) z[0][n][e] = -z[0][n][e];
            __syncwarp();
            put_block(to, z[0], lane);
        }
        __syncthreads();
    }
    // ---- Y = T B;  then W = Q T and P' = P - Q Y
    for (int n = 0; n < 2; ++n) {
        const int at = warp_blocks(warp, n);
        if (at < 0) continue;
        float d[1][2][4] = {};
        block_product(d, ts, bs, at >> 2, at & 3, lane);
        put_block(ys + lower_block(at >> 2, at & 3) * 3 * 256, d[0], lane);
    }
    __syncthreads();
    for (int n = 0; n < 2; ++n) {
        const int at = warp_blocks(warp, n), i = at >> 2, j = at & 3;
        if (at < 0) continue;
        float d[1][2][4] = {};
        block_product(d, qs, ts, i, j, lane);
        put_block(ws + lower_block(i, j) * 3 * 256, d[0], lane);
        float e[1][2][4] = {};
        block_product(e, qs, ys, i, j, lane);
        const float* own = pf + (lower_block(i, j) * 32 + lane) * 8;
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int row = i * 16 + g + 8 * x;
                const float2 was = *reinterpret_cast<const float2*>(own + m * 4 + x * 2);
                uint32_t y[3];
                cut(row >= bad ? nan : was.x - e[0][m][2 * x], row >= bad ? nan : was.y - e[0][m][2 * x + 1], y);
#pragma unroll
                for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(parts + p * CK * CK + row * CK + j * 16 + m * 8 + t4 * 2) = y[p];
            }
    }
    parts += 3 * CK * CK;
    for (int e = tid; e < DK; e += DP_THREADS) {
        float* to = ends + unit * 2 * DK + e;
        to[0] = bad < CK ? nan : mid[DK + e];
        to[DK] = bad < CK ? nan : mid[e] * mid[DK + e];
    }
    auto stage_values = [&](int c0) {
        for (int e = tid; e < CK * OUT_V / 4; e += DP_THREADS) {
            const int t = e / (OUT_V / 4), i = (e % (OUT_V / 4)) * 4;
            if (c0 + i < dv) cp8(vs + t * VP + i, t < tokens ? v + (size_t)(c.t0 + t) * v_stride + (size_t)h * dv + c0 + i : v, t < tokens);
        }
    };
    __syncthreads();
    stage_values(0);
    const int kb = warp;                                     // this warp's 16 channels
    if (kb < KS) {
        // ---- X = T U D and R' = (R D - W U D), from the middle to the chunk's start by the channel's product
        uint32_t fu[QUARTERS][3][1][4];
#pragma unroll
        for (int t = 0; t < QUARTERS; ++t)
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const uint4 x = *reinterpret_cast<const uint4*>(xs + p * CK * DK + ((t * KS + kb) * 32 + lane) * 8);
                fu[t][p][0][0] = x.x; fu[t][p][0][1] = x.y; fu[t][p][0][2] = x.z; fu[t][p][0][3] = x.w;
            }
        uint32_t rc[QUARTERS][4];
#pragma unroll
        for (int i = 0; i < QUARTERS; ++i)
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int t = i * 16 + g + 8 * e;
                    rc[i][n * 2 + e] = t < tokens ? *reinterpret_cast<const uint32_t*>(r + (size_t)(c.t0 + t) * r_stride + (size_t)h * DK + kb * 16 + n * 8 + t4 * 2) : 0u;
                }
#pragma unroll
        for (int i = 0; i < QUARTERS; ++i) {
            float dx[1][2][4] = {}, dr[1][2][4] = {};
#pragma unroll
            for (int t = 0; t <= i; ++t) {
                uint32_t ft[3][1][4], fw[3][1][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    ldsm(ft[p][0], lane_row(ts + (lower_block(i, t) * 3 + p) * 256, lane));
                    ldsm(fw[p][0], lane_row(ws + (lower_block(i, t) * 3 + p) * 256, lane));
                }
                products<1, 1, 3, 3>(dx, ft, fu[t]);
                products<1, 1, 3, 3>(dr, fw, fu[t]);
            }
            uint32_t x[4][3];
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int ch = kb * 16 + n * 8 + t4 * 2;
                const float2 m = *reinterpret_cast<const float2*>(mid + ch);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int t = i * 16 + g + 8 * e;
                    cut(dx[0][n][2 * e] * m.x, dx[0][n][2 * e + 1] * m.y, x[e * 2 + n]);
                    float2 f = *reinterpret_cast<const float2*>(ps + t * L::PF + ch);
                    if (t < 32) f = make_float2(reciprocal(f.x), reciprocal(f.y));
                    const uint32_t r2 = rc[i][n * 2 + e];
                    uint32_t y[3];
                    cut(t >= bad ? nan : (low_of(r2) * f.x - dr[0][n][2 * e]) * m.x, t >= bad ? nan : (high_of(r2) * f.y - dr[0][n][2 * e + 1]) * m.y, y);
#pragma unroll
                    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint32_t*>(parts + p * CK * DK + t * DK + ch) = y[p];
                }
            }
#pragma unroll
            for (int p = 0; p < 3; ++p)
                *reinterpret_cast<uint4*>(xs + p * CK * DK + ((i * KS + kb) * 32 + lane) * 8) = make_uint4(x[0][p], x[1][p], x[2][p], x[3][p]);
        }
    }
    // ---- K D - Y^T AU D, from the middle to the chunk's end by the channel's product
    uint32_t kp[QUARTERS][3][1][4];                          // as the right operand of the last product
    if (kb < KS) {
        uint32_t fa[QUARTERS][3][1][4], kc[QUARTERS][4];
#pragma unroll
        for (int t = 0; t < QUARTERS; ++t) {
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                const uint4 x = *reinterpret_cast<const uint4*>(aus + p * CK * DK + ((t * KS + kb) * 32 + lane) * 8);
                fa[t][p][0][0] = x.x; fa[t][p][0][1] = x.y; fa[t][p][0][2] = x.z; fa[t][p][0][3] = x.w;
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int at = t * 16 + g + 8 * e;
                    kc[t][n * 2 + e] = at < tokens ? *reinterpret_cast<const uint32_t*>(k + (size_t)(c.t0 + at) * k_stride + (size_t)h * DK + kb * 16 + n * 8 + t4 * 2) : 0u;
                }
        }
#pragma unroll
        for (int j = 0; j < QUARTERS; ++j) {
            float d[1][2][4] = {};
#pragma unroll
            for (int t = j; t < QUARTERS; ++t) {
                uint32_t fy[3][1][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) {                // the block's transpose as the left operand
                    const int row = (lane & 7) + (lane >> 4) * 8;
                    ldsm_t(fy[p][0], ys + (lower_block(t, j) * 3 + p) * 256 + row * 16 + (((lane >> 3 & 1) ^ (row >> 2 & 1)) << 3));
                }
                products<1, 1, 3, 3>(d, fy, fa[t]);
            }
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int ch = kb * 16 + n * 8 + t4 * 2;
                const float2 m = *reinterpret_cast<const float2*>(mid + DK + ch);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float2 f = *reinterpret_cast<const float2*>(ps + (j * 16 + g + 8 * e) * L::PF + ch);
                    if (j >= 2) f = make_float2(reciprocal(f.x), reciprocal(f.y));
                    uint32_t x[3];
                    cut((low_of(kc[j][n * 2 + e]) * f.x - d[0][n][2 * e]) * m.x, (high_of(kc[j][n * 2 + e]) * f.y - d[0][n][2 * e + 1]) * m.y, x);
#pragma unroll
                    for (int p = 0; p < 3; ++p)              // 8 tokens by 8 keys, turned: a lane has two tokens of a key
                        asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(kp[j][p][0][n * 2 + e]) : "r"(x[p]));
                }
            }
        }
    }
    // ---- the chunk's own contribution: values by keys
    for (int c0 = 0; c0 < dv; c0 += OUT_V) {
        const int cols = min(OUT_V, dv - c0);
        if (c0 > 0) {
            __syncthreads();
            stage_values(c0);
        }
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        if (kb < KS) {
            for (int m = 0; m < cols / 16; ++m) {
                float d[1][2][4] = {};
#pragma unroll
                for (int t = 0; t < QUARTERS; ++t) {
                    uint32_t fv[1][1][4];
                    ldsm_t(fv[0][0], vs + t * 16 * VP + m * 16 + at_at(lane, VP));
                    products<1, 1, 1, 3>(d, fv, kp[t]);
                }
                float* to = states + (unit * dv + c0 + m * 16) * DK + (kb * 32 + lane) * 8;
                *reinterpret_cast<float4*>(to) = make_float4(d[0][0][0], d[0][0][1], d[0][1][0], d[0][1][1]);
                *reinterpret_cast<float4*>(to + 4) = make_float4(d[0][0][2], d[0][0][3], d[0][1][2], d[0][1][3]);
            }
        }
    }
}

// The state in front of every chunk: 16 MT value channels x MG of one head of one entry, the chunks in order.  Four warps a group of
// 16 MT channels: the d of a quarter of the tokens each, then the state of a quarter of the keys; they meet in shared memory
// twice a chunk.  X and au of the chunks come through a ring of three slots, each asked for a chunk ahead.
template <int MT, int MG>
struct ScanLayout {                             // bytes
    static constexpr int SLOT = 3 * CK * DK * 2;
    static constexpr int ring = 0, s = 3 * SLOT, d = s + MG * 3 * MT * KS * 512, bytes = d + MG * 3 * MT * QUARTERS * 512;
};
template <int MT, int MG>
__global__ void __launch_bounds__(128 * MG, 1)
delta_chunk_scan_kernel(const bf16* __restrict__ xs, const bf16* __restrict__ aus, const float* __restrict__ ends, const float* __restrict__ states,
                        bf16* __restrict__ cuts, float* __restrict__ state, const int* __restrict__ cu_q, const int* __restrict__ state_slots,
                        int least, int H, int dv) {
    using L = ScanLayout<MT, MG>;
    constexpr int KBW = KS / 4;                              // key blocks of a warp
    extern __shared__ __align__(16) unsigned char raw[];
    pdl_trigger();
    pdl_wait();
    const int b = blockIdx.z, h = blockIdx.y;
    const int count = chunks_of(cu_q[b + 1] - cu_q[b], least);
    if (count == 0) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, group = warp >> 2, wn = warp & 3, g = lane >> 2, t4 = lane & 3;
    const size_t base = first_chunk(cu_q, b, least), one = (size_t)dv * DK;
    uint4* sp = reinterpret_cast<uint4*>(raw + L::s) + group * 3 * MT * KS * 32;             // [piece][m][key block][lane]
    uint4* dp = reinterpret_cast<uint4*>(raw + L::d) + group * 3 * MT * QUARTERS * 32;       // [piece][m][token block][lane]
    auto ask = [&](int item) {                               // X of chunk item / 2, or its au
        if (item < 2 * count) {
            const bf16* from = (item & 1 ? aus : xs) + ((base + (item >> 1)) * H + h) * 3 * CK * DK;
            bf16* to = reinterpret_cast<bf16*>(raw + L::ring + item % 3 * L::SLOT);
            for (int e = tid; e < 3 * CK * DK / 8; e += 128 * MG) cp16(to + e * 8, from + e * 8);
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    ask(0);
    ask(1);
    const int vb0 = (blockIdx.x * MG + group) * MT;          // the group's first value block
    float* own = state + ((size_t)state_slots[b] * H + h) * one;
    float S[MT][KBW][2][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < KBW; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {                    // rows (value) g, g + 8; keys 2 t4 of the block's halves
                const float2 x = *reinterpret_cast<const float2*>(own + (size_t)((vb0 + m) * 16 + g + 8 * (e >> 1)) * DK + (wn * KBW + n) * 16 + (e & 1) * 8 + t4 * 2);
                S[m][n][e & 1][(e >> 1) * 2] = x.x;
                S[m][n][e & 1][(e >> 1) * 2 + 1] = x.y;
            }
    for (int c = 0; c < count; ++c) {
        const size_t unit = (base + c) * H + h;
        // the state in front of the chunk: to the outputs' kernel as the right operand, to the other warps as the left one
#pragma unroll
        for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int n = 0; n < KBW; ++n) {
                uint32_t x[4][3];                            // value row half, key half
#pragma unroll
                for (int e = 0; e < 4; ++e) cut(S[m][n][e & 1][(e >> 1) * 2], S[m][n][e & 1][(e >> 1) * 2 + 1], x[e]);
                const int kb = wn * KBW + n;
                bf16* to = cuts + unit * 3 * one + ((size_t)(vb0 + m) * KS + kb) * 256 + lane * 8;
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    *reinterpret_cast<uint4*>(to + p * one) = make_uint4(x[0][p], x[1][p], x[2][p], x[3][p]);
                    sp[((p * MT + m) * KS + kb) * 32 + lane] = make_uint4(x[0][p], x[2][p], x[1][p], x[3][p]);
                }
            }
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();                                     // X is there, so is the state, and the last chunk's au are read
        ask(2 * c + 2);
        // what the chunk itself adds, and its decays, on their way
        float4 x0[MT][KBW], x1[MT][KBW];
        float2 f[KBW][2], all[KBW][2];
#pragma unroll
        for (int n = 0; n < KBW; ++n) {
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const float* from = states + unit * one + ((size_t)(vb0 + m) * KS + wn * KBW + n) * 256 + lane * 8;
                x0[m][n] = load4(from);
                x1[m][n] = load4(from + 4);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float* from = ends + unit * 2 * DK + (wn * KBW + n) * 16 + e * 8 + t4 * 2;
                f[n][e] = *reinterpret_cast<const float2*>(from);
                all[n][e] = *reinterpret_cast<const float2*>(from + DK);
            }
        }
        const uint4* ring = reinterpret_cast<const uint4*>(raw + L::ring + (2 * c) % 3 * L::SLOT);
        {
            float d[MT][1][2][4] = {};
#pragma unroll 2
            for (int k = 0; k < KS; ++k) {
                uint32_t fb[3][1][4];
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const uint4 x = ring[(p * QUARTERS + wn) * KS * 32 + k * 32 + lane];
                    fb[p][0][0] = x.x; fb[p][0][1] = x.y; fb[p][0][2] = x.z; fb[p][0][3] = x.w;
                }
#pragma unroll
                for (int m = 0; m < MT; ++m) {
                    uint32_t fa[3][1][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const uint4 x = sp[((p * MT + m) * KS + k) * 32 + lane];
                        fa[p][0][0] = x.x; fa[p][0][1] = x.y; fa[p][0][2] = x.z; fa[p][0][3] = x.w;
                    }
                    products<1, 1, 3, 3>(d[m], fa, fb);
                }
            }
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                uint32_t x[4][3];
#pragma unroll
                for (int e = 0; e < 4; ++e) cut(d[m][0][e >> 1][(e & 1) * 2], d[m][0][e >> 1][(e & 1) * 2 + 1], x[e]);
#pragma unroll
                for (int p = 0; p < 3; ++p) dp[((p * MT + m) * QUARTERS + wn) * 32 + lane] = make_uint4(x[0][p], x[1][p], x[2][p], x[3][p]);
            }
        }
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();                                     // the au are there, so are all tokens' d, and X is read
        ask(2 * c + 3);
        ring = reinterpret_cast<const uint4*>(raw + L::ring + (2 * c + 1) % 3 * L::SLOT);
        {
            float d[MT][KBW][1][2][4] = {};
#pragma unroll 2
            for (int t = 0; t < QUARTERS; ++t) {
                uint32_t fa[MT][3][1][4];
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const uint4 x = dp[((p * MT + m) * QUARTERS + t) * 32 + lane];
                        fa[m][p][0][0] = x.x; fa[m][p][0][1] = x.y; fa[m][p][0][2] = x.z; fa[m][p][0][3] = x.w;
                    }
#pragma unroll
                for (int n = 0; n < KBW; ++n) {
                    uint32_t fb[3][1][4];
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const uint4 x = ring[(p * QUARTERS + t) * KS * 32 + (wn * KBW + n) * 32 + lane];
                        fb[p][0][0] = x.x; fb[p][0][1] = x.y; fb[p][0][2] = x.z; fb[p][0][3] = x.w;
                    }
#pragma unroll
                    for (int m = 0; m < MT; ++m) products<1, 1, 3, 3>(d[m][n], fa[m], fb);
                }
            }
#pragma unroll
            for (int m = 0; m < MT; ++m)
#pragma unroll
                for (int n = 0; n < KBW; ++n) {
                    const float l[2][4] = {{x0[m][n].x, x0[m][n].y, x1[m][n].x, x1[m][n].y}, {x0[m][n].z, x0[m][n].w, x1[m][n].z, x1[m][n].w}};
#pragma unroll
                    for (int e = 0; e < 2; ++e)
#pragma unroll
                        for (int z = 0; z < 4; ++z) {
                            const float ff = z & 1 ? f[n][e].y : f[n][e].x, aa = z & 1 ? all[n][e].y : all[n][e].x;
                            S[m][n][e][z] = fmaf(aa, S[m][n][e][z], fmaf(-ff, d[m][n][0][e][z], l[e][z]));
                        }
                }
        }
        // (the state's pieces and the d are written again after the others have read them: the next barriers)
    }
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int n = 0; n < KBW; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                *reinterpret_cast<float2*>(own + (size_t)((vb0 + m) * 16 + g + 8 * (e >> 1)) * DK + (wn * KBW + n) * 16 + (e & 1) * 8 + t4 * 2) =
                    make_float2(S[m][n][e & 1][(e >> 1) * 2], S[m][n][e & 1][(e >> 1) * 2 + 1]);
}

inline bool aligned4(const void* p, int esize) { return (reinterpret_cast<uintptr_t>(p) % (4 * (size_t)esize)) == 0; }
template <typename Kernel>
int allow(Kernel kernel, int bytes) { return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); }
inline bool aligned2(const float* p) { return (reinterpret_cast<uintptr_t>(p) % 8) == 0; }      // outputs leave in pairs
}  // namespace

// Whether the head form (`gated` 0) or the gated one takes these arrays; what they do not take walks.  (The outputs' address, and that of
// the delta rule's decays, the callers look at.)
RI_API int ri_chunks_ok(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride, int act_dtype, int dv, int gated) {
    const int esize = act_dtype == RI_BF16 ? 2 : 4;
    return dv > 0 && dv % 64 == 0 && q_stride % 4 == 0 && k_stride % 4 == 0 && v_stride % 4 == 0 && aligned4(q, esize) &&
           aligned4(k, esize) && aligned4(v, esize) && (!gated || act_dtype == RI_BF16);
}

// The entries of at least `least` tokens in chunks; `chunks`: the number the grids are made for, at least that of all those
// entries.  Scratch: states fp32 [chunks][H][dv][DK], totals fp32 [chunks][H][2], cuts bf16 [chunks][H][3][dv][DK].
RI_API int ri_head_chunks(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride,
                          const float* decay, int a_stride, const float* gain, int g_stride, int act_dtype, float q_scale,
                          float* out, float* state, const int* cu_q, const int* state_slots, int entries, int least, int chunks,
                          int H, int dv, int share, float* states, float* totals, void* cuts, void* stream) {
    if (entries <= 0 || chunks <= 0) return 0;
    if (share <= 0 || H % share || !aligned2(out) || !ri_chunks_ok(q, q_stride, k, k_stride, v, v_stride, act_dtype, dv, 0)) return (int)cudaErrorInvalidValue;
    cudaStream_t s = (cudaStream_t)stream;
    // heads a CTA of the outputs serves: the scores of a key head, as much work as a head's 64 channels, are made once a CTA, and
    // CTAs go in waves of two an SM.  The layer over 2,048 tokens, heads a CTA 1, 2, 4, 8: 32 heads of 64 in 4 key heads 245, 236, 234,
    // 277 us (the rule takes 4), 64 in 8 key heads 419, 411, 404, 403 (8).
    int heads = 1;
    double best = 0;
    for (int n = 1; n <= share; ++n) {
        if (share % n) continue;
        const long long waves = ((long long)chunks * (H / n) + 2 * ri_device_sms() - 1) / (2 * ri_device_sms());
        const double cost = (double)waves * (64 + (double)n * dv);
        if (n == 1 || cost < best) { best = cost; heads = n; }
    }
    const int scan_blocks = (int)(((size_t)H * dv * DK / 8 + SCAN_THREADS - 1) / SCAN_THREADS);
#define RI_STATES(TA, VT) do { \
    static bool allowed = false; \
    if (!allowed) { RI_CHECKED(allow(chunk_states_kernel<TA, VT, false>, states_bytes<TA, VT, false>())); allowed = true; } \
    RI_CHECKED(ri_launch(chunk_states_kernel<TA, VT, false>, dim3(chunks, H / share, share * dv / VT), dim3(ST_THREADS), \
        states_bytes<TA, VT, false>(), s, (const TA*)k, k_stride, (const TA*)v, v_stride, decay, a_stride, gain, g_stride, states, totals, \
        cu_q, entries, least, H, dv, share)); } while (0)
#define RI_HC(TA) do { \
    static bool allowed = false; \
    if (!allowed) { RI_CHECKED(allow(head_chunk_outputs_kernel<TA>, OutLayout::bytes)); allowed = true; } \
    if (dv % 128 == 0 || (dv == 64 && share % 2 == 0)) RI_STATES(TA, 128); else RI_STATES(TA, 64); \
    RI_CHECKED(ri_launch(chunk_scan_kernel<false>, dim3(scan_blocks, entries), dim3(SCAN_THREADS), 0, s, states, totals, (bf16*)cuts, state, cu_q, \
        state_slots, least, H, dv)); \
    RI_CHECKED(ri_launch(head_chunk_outputs_kernel<TA>, dim3(chunks, H / heads), dim3(OUT_THREADS), OutLayout::bytes, s, (const TA*)q, q_stride, \
        (const TA*)k, k_stride, (const TA*)v, v_stride, decay, a_stride, gain, g_stride, q_scale, (const bf16*)cuts, out, cu_q, entries, least, \
        H, dv, share, heads)); } while (0)
    if (act_dtype == RI_BF16) RI_HC(bf16);
    else RI_HC(float);
#undef RI_HC
#undef RI_STATES
    return ri_launch_status();
}

// The gated form (bf16 q, k, v; fp32 decays [T][a_stride], a_stride 0: one row for all tokens); totals fp32 [chunks][H][DK],
// parts bf16 [chunks][H][ri_gated_chunk_parts()].
RI_API int ri_gated_chunk_parts() { return GATED_PARTS; }
RI_API int ri_gated_chunks(const void* q, int q_stride, const void* k, int k_stride, const void* v, int v_stride,
                           const float* alpha, int a_stride, int act_dtype, float q_scale, float* out, float* state, const int* cu_q,
                           const int* state_slots, int entries, int least, int chunks, int H, int dv, float* states, float* totals,
                           void* cuts, void* parts, void* stream) {
    if (entries <= 0 || chunks <= 0) return 0;
    if (!aligned2(out) || !ri_chunks_ok(q, q_stride, k, k_stride, v, v_stride, act_dtype, dv, 1)) return (int)cudaErrorInvalidValue;
    cudaStream_t s = (cudaStream_t)stream;
    const int scan_blocks = (int)(((size_t)H * dv * DK / 8 + SCAN_THREADS - 1) / SCAN_THREADS);
    static bool allowed = false;
    if (!allowed) {
        RI_CHECKED(allow(gated_chunk_scores_kernel, ScoreLayout::bytes));
        RI_CHECKED(allow(gated_chunk_outputs_kernel<4>, OutLayout::gated_bytes));
        RI_CHECKED(allow(gated_chunk_outputs_kernel<2>, OutLayout::gated_bytes));
        RI_CHECKED(allow(chunk_states_kernel<bf16, 128, true>, states_bytes<bf16, 128, true>()));
        RI_CHECKED(allow(chunk_states_kernel<bf16, 64, true>, states_bytes<bf16, 64, true>()));
        allowed = true;
    }
#define RI_STATES(VT) RI_CHECKED(ri_launch(chunk_states_kernel<bf16, VT, true>, dim3(chunks, H, dv / VT), dim3(ST_THREADS), \
        states_bytes<bf16, VT, true>(), s, (const bf16*)k, k_stride, (const bf16*)v, v_stride, alpha, a_stride, (const float*)nullptr, 0, states, \
        totals, cu_q, entries, least, H, dv, 1))
    if (dv % 128 == 0) RI_STATES(128);
    else RI_STATES(64);
#undef RI_STATES
    RI_CHECKED(ri_launch(chunk_scan_kernel<true>, dim3(scan_blocks, entries), dim3(SCAN_THREADS), 0, s, states, totals, (bf16*)cuts, state, cu_q, state_slots,
                         least, H, dv));
    RI_CHECKED(ri_launch(gated_chunk_scores_kernel, dim3(chunks, H), dim3(OUT_THREADS), ScoreLayout::bytes, s, (const bf16*)q, q_stride,
                         (const bf16*)k, k_stride, alpha, a_stride, (bf16*)parts, cu_q, entries, least, H));
    RI_CHECKED(ri_launch(dv % OUT_V == 0 ? gated_chunk_outputs_kernel<4> : gated_chunk_outputs_kernel<2>, dim3(chunks, H, dv % OUT_V == 0 ? dv / OUT_V : 1), dim3(OUT_THREADS), OutLayout::gated_bytes, s,
                         (const bf16*)parts, (const bf16*)v, v_stride, q_scale, (const bf16*)cuts, out, cu_q, entries, least, H, dv));
    return ri_launch_status();
}
// The delta rule (bf16 r, k, v; w, u, au fp32 [T][f_stride] as the walk's, -log w at most ri_delta_chunk_decay()): xs and aus bf16
// [chunks][H][3][CK][DK], ends fp32 [chunks][H][2][DK], the rest as the gated form's.
RI_API float ri_delta_chunk_decay() { return DELTA_MOST_DECAY; }
// The reciprocals that the decays' products take (n floats), for their test.
RI_API int ri_delta_chunk_reciprocals(const float* x, float* y, int n, void* stream) {
    if (n <= 0) return 0;
    reciprocal_kernel<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(x, y, n);
    return ri_launch_status();
}
RI_API int ri_delta_chunks(const void* r, int r_stride, const void* k, int k_stride, const void* v, int v_stride, const float* w,
                           const float* u, const float* au, int f_stride, int act_dtype, float* out, float* state, const int* cu_q,
                           const int* state_slots, int entries, int least, int chunks, int H, int dv, float* states, float* ends, void* cuts,
                           void* parts, void* xs, void* aus, void* stream) {
    if (entries <= 0 || chunks <= 0) return 0;
    if (!aligned2(out) || !ri_chunks_ok(r, r_stride, k, k_stride, v, v_stride, act_dtype, dv, 1) || f_stride % 4 || !aligned4(w, 4) || !aligned4(u, 4) || !aligned4(au, 4))
        return (int)cudaErrorInvalidValue;
    cudaStream_t s = (cudaStream_t)stream;
    static bool allowed = false;
    if (!allowed) {
        RI_CHECKED(allow(delta_chunk_parts_kernel, PartsLayout::bytes));
        RI_CHECKED(allow(delta_chunk_scan_kernel<1, 1>, ScanLayout<1, 1>::bytes));
        RI_CHECKED(allow(delta_chunk_scan_kernel<2, 1>, ScanLayout<2, 1>::bytes));
        RI_CHECKED(allow(delta_chunk_scan_kernel<2, 2>, ScanLayout<2, 2>::bytes));
        RI_CHECKED(allow(gated_chunk_outputs_kernel<4>, OutLayout::gated_bytes));
        RI_CHECKED(allow(gated_chunk_outputs_kernel<2>, OutLayout::gated_bytes));
        allowed = true;
    }
    RI_CHECKED(ri_launch(delta_chunk_parts_kernel, dim3(chunks, H), dim3(DP_THREADS), PartsLayout::bytes, s, (const bf16*)r, r_stride,
                         (const bf16*)k, k_stride, (const bf16*)v, v_stride, w, u, au, f_stride, (bf16*)xs, (bf16*)aus, ends, (bf16*)parts,
                         states, cu_q, entries, least, H, dv));
    // value channels a CTA of the scan takes, one CTA an SM: the fewest that leave no CTA waiting for an SM
    const long long blocks = (long long)entries * H * dv / 16;
#define RI_DSCAN(MT, MG) RI_CHECKED(ri_launch(delta_chunk_scan_kernel<MT, MG>, dim3(dv / (16 * MT * MG), H, entries), dim3(128 * MG), \
        ScanLayout<MT, MG>::bytes, s, (const bf16*)xs, (const bf16*)aus, (const float*)ends, (const float*)states, (bf16*)cuts, state, cu_q, \
        state_slots, least, H, dv))
    if (blocks <= ri_device_sms()) RI_DSCAN(1, 1);
    else if (blocks <= 2LL * ri_device_sms()) RI_DSCAN(2, 1);
    else RI_DSCAN(2, 2);
#undef RI_DSCAN
    RI_CHECKED(ri_launch(dv % OUT_V == 0 ? gated_chunk_outputs_kernel<4> : gated_chunk_outputs_kernel<2>, dim3(chunks, H, dv % OUT_V == 0 ? dv / OUT_V : 1),
                         dim3(OUT_THREADS), OutLayout::gated_bytes, s, (const bf16*)parts, (const bf16*)v, v_stride, 1.0f, (const bf16*)cuts, out,
                         cu_q, entries, least, H, dv));
    return ri_launch_status();
}
#else
RI_API int ri_chunks_ok(const void*, int, const void*, int, const void*, int, int, int, int) { return 0; }
RI_API int ri_head_chunks(const void*, int, const void*, int, const void*, int, const float*, int, const float*, int, int, float, float*,
                          float*, const int*, const int*, int, int, int, int, int, int, float*, float*, void*, void*) {
    return (int)cudaErrorInvalidValue;
}
RI_API int ri_gated_chunks(const void*, int, const void*, int, const void*, int, const float*, int, int, float, float*, float*, const int*,
                           const int*, int, int, int, int, int, float*, float*, void*, void*, void*) {
    return (int)cudaErrorInvalidValue;
}
RI_API int ri_gated_chunk_parts() { return 0; }
RI_API float ri_delta_chunk_decay() { return 0.f; }
RI_API int ri_delta_chunk_reciprocals(const float*, float*, int, void*) { return (int)cudaErrorInvalidValue; }
RI_API int ri_delta_chunks(const void*, int, const void*, int, const void*, int, const float*, const float*, const float*, int, int, float*,
                           float*, const int*, const int*, int, int, int, int, int, float*, float*, void*, void*, void*, void*, void*) {
    return (int)cudaErrorInvalidValue;
}
#endif

RI_API int ri_recurrent_chunk_tokens() { return BUILT ? CK : 0; }
