// True 32-bit matrix product C[M,N] = A[M,K] * W[N,K]^T with plain FFMA: no
// tensor core, no TF32, no library. Each output element is summed over k in four
// interleaved chains (of every 64 columns chain g takes the 16 from 16 g on), each in ascending order, that
// are added as (c0 + c1) + (c2 + c3), in every kernel and tile here, so the value of C[m,n] depends on row m of A
// and row n of W only, never on M, on the other rows of the batch, or on where the operands lie in memory.
// W may be stored in float32 or in bfloat16 (widened exactly on load).
//
// What bounds it: the FMA pipe for many rows (128 products a cycle and SM, which take the two-product instruction:
// the plain one runs at half that rate), shared memory nearly as much (an LDS.128 of a warp takes four cycles
// however many lanes read the same words, so an 8 x 8 block of outputs a thread needs as many cycles of loads as of
// products), and for few rows the stream over W. So: large blocks of outputs a thread, four groups of warps a
// tile that divide k (a tile of 64 x 64 then keeps eight warps busy, and 300 rows x 2,048 outputs, 160 tiles,
// the device), the next 64 columns on their way while these are worked on, one barrier a step.
// Weights of 1,024 x 1,024 and more come here only where they are asked for (gemm_f32_tc.cu takes them: 120 us, L2 cold, for the first
// size below); what is always made here are smaller ones, 300 rows x 512 x 512 17.7 us, 2,048 x 256 x 256 11.
// Measured, us (one thread a 4 x 4 block, 16 columns at a time, nothing under way -> this): 300 rows x 16,384
// outputs x 2,048: 1,125 -> 511 (39 TFLOP/s); 300 x 2,048 x 8,192: 1,024 -> 439; 300 x 3,072 x 2,048: 248 -> 116;
// 16 x 32,768 x 2,048: 428 -> 82; 8 x 3,072 x 2,048: 167 -> 18. Against a 64-bit product 4.1e-7 (2-norm) where one chain
// of 2,048 is 8.1e-7 off. Tried: one chain with 64 x 128 tiles, 557 and 581 us at the first two sizes; two
// blocks an SM with 128 registers a thread, 573 and 516.
#include "common.cuh"

#define BM 64
#define BN 64
#define BK 16
#define GK 4             // chains an output is summed in

// NG: chains that are not empty (four, or as many as a K of up to 32 has).
template <typename TW, int NG>
__global__ void __launch_bounds__(256)
gemm_f32_kernel(const float* __restrict__ A, const TW* __restrict__ W, float* __restrict__ C, int M,
                int N, int K) {
    pdl_wait();      // nothing of this kernel touches global memory before this
    pdl_trigger();
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float acc[NG][4][4];                       // chain g: the columns 16 g to 16 g + 15 of every 64
#pragma unroll
    for (int g = 0; g < NG; ++g)
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[g][i][j] = 0.0f;

    for (int kb = 0; kb < K; kb += GK * BK) {
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const int k0 = kb + g * BK;
            if (k0 >= K) break;
            // 64x16 tile of each operand, 4 elements a thread, k fastest in memory.
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int idx = threadIdx.x + i * 256;  // 0..1023
                const int r = idx >> 4, kk = idx & 15;
                const int gm = m0 + r, gn = n0 + r, gk = k0 + kk;
                As[kk][r] = (gm < M && gk < K) ? A[(size_t)gm * K + gk] : 0.0f;
                Ws[kk][r] = (gn < N && gk < K) ? to_f32(W[(size_t)gn * K + gk]) : 0.0f;
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                float a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = Ws[kk][tx * 4 + j];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[g][i][j] = fmaf(a[i], b[j], acc[g][i][j]);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            const float c01 = NG > 1 ? acc[0][i][j] + acc[NG > 1][i][j] : acc[0][i][j];
            if (gn < N) C[(size_t)gm * N + gn] = NG > 2 ? c01 + (acc[NG > 2 ? 2 : 0][i][j] + acc[NG > 2 ? 3 : 0][i][j]) : c01;
        }
    }
}

// Rows of K a multiple of 4 that start on 16 bytes (float32) or 8 bytes (bfloat16).
__device__ __forceinline__ float4 load4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 r = __ldg(reinterpret_cast<const uint2*>(p));       // the low half of a word comes first in memory
    return make_float4(__uint_as_float(r.x << 16), __uint_as_float(r.x & 0xffff0000u), __uint_as_float(r.y << 16),
                       __uint_as_float(r.y & 0xffff0000u));
}

// Two FFMAs in one instruction, each rounded as fmaf rounds: the plain instruction runs at half the pipe's rate here.
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long twice(float x) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
// A block's warps are GK groups that share the tile and divide k among themselves: of every TK = 64 columns group g
// takes the 16 from 16 g on, so every output is the sum of GK chains, (c0 + c1) + (c2 + c3), in all tile sizes.
// Within a group a warp is 4 x 8 lanes, a lane's outputs rows ty + 4 i and columns tx + 8 j of its warp's tile;
// columns j and j + 1 share an instruction, so W's rows lie in pairs (n, n + 8), their values of one k side by side.
// Shared memory: a row of A is 16 16-byte pieces (four k each), a pair of rows of W 32 (two k of both rows);
// piece c of row r lies at c ^ (r & 7), piece c of pair q at c ^ (q & 7): what eight lanes read at one k, and what
// eight lanes write, touches every bank once.
#define TK 64
template <typename TW, int WM, int WN, int TM, int TN, int MINB>
__global__ void __launch_bounds__(GK * WM * WN * 32, MINB)
gemm_f32_tiled_kernel(const float* __restrict__ A, const TW* __restrict__ W, float* __restrict__ C, int M, int N, int K) {
    constexpr int P = TK / 4, NT = GK * WM * WN * 32, TBM = WM * 4 * TM, TBN = WN * 8 * TN;
    constexpr int IA = TBM * TK / 4, IW = TBN * TK / 8;               // fetches: four k of a row, of a pair of rows
    constexpr int LA = (IA + NT - 1) / NT, LW = (IW + NT - 1) / NT;   // fetches a thread
    constexpr int BUF = (TBM + TBN) * TK;                             // floats a buffer: A, then W
    extern __shared__ __align__(128) float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, grp = warp / (WM * WN), wt = warp % (WM * WN);
    const int ty = (wt / WN) * 4 * TM + (lane >> 3), tx = (wt % WN) * 8 * TN + (lane & 7);
    const int m0 = blockIdx.y * TBM, n0 = blockIdx.x * TBN;
    float4 rw[LW][2];
    auto fetch_w = [&](int k0) {
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int idx = threadIdx.x + i * NT, q = idx / P, gk = k0 + 4 * (idx & (P - 1));
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int gn = n0 + (q >> 3) * 16 + (q & 7) + 8 * h;
                rw[i][h] = (idx < IW && gn < N && gk < K) ? load4(W + (size_t)gn * K + gk) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    };
    auto put_w = [&](int buf) {
        float* ws = sm + buf * BUF + TBM * TK;
#pragma unroll
        for (int i = 0; i < LW; ++i) {
            const int idx = threadIdx.x + i * NT, q = idx / P, c = 2 * (idx & (P - 1));
            const float4 x = rw[i][0], y = rw[i][1];
            if (idx < IW) {
                *reinterpret_cast<float4*>(ws + q * 2 * TK + 4 * (c ^ (q & 7))) = make_float4(x.x, y.x, x.y, y.y);
                *reinterpret_cast<float4*>(ws + q * 2 * TK + 4 * ((c + 1) ^ (q & 7))) = make_float4(x.z, y.z, x.w, y.w);
            }
        }
    };
    auto copy_a = [&](int k0, int buf) {        // asynchronous; zeros (a copy of no bytes) outside the matrix
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int idx = threadIdx.x + i * NT, r = idx / P, c = idx & (P - 1), gm = m0 + r, gk = k0 + 4 * c;
            const bool in = gm < M && gk < K;
            if (idx < IA)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                                 (uint32_t)__cvta_generic_to_shared(sm + buf * BUF + r * TK + 4 * (c ^ (r & 7)))),
                             "l"(in ? A + (size_t)gm * K + gk : A), "r"(in ? 16 : 0)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int ao[8], wo[8];       // where piece u (its low three bits) of one of this lane's rows (of A: for i even) or pairs lies
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        ao[u] = 4 * (u ^ (4 * (grp & 1)) ^ (ty & 3));
        wo[u] = 4 * (u ^ (lane & 7));
    }
    unsigned long long acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;

    pdl_wait();      // nothing of this kernel touches global memory before this
    pdl_trigger();
    copy_a(0, 0);
    fetch_w(0);
    put_w(0);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += TK, buf ^= 1) {
        const bool more = k0 + TK < K;
        if (more) { copy_a(k0 + TK, buf ^ 1); fetch_w(k0 + TK); }      // that buffer was last read before the last barrier
        const float* as = sm + buf * BUF + ty * TK + (grp >> 1) * 32;
        const float* ws = sm + buf * BUF + TBM * TK + ((wt % WN) * 4 * TN + (lane & 7)) * 2 * TK + grp * 32;
#pragma unroll
        for (int kq = 0; kq < 4; ++kq) {        // piece 4 grp + kq of A's rows, 8 grp + 2 kq and + 1 of W's pairs
            float4 a[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const int u = kq ^ (4 * (i & 1));
                a[i] = *reinterpret_cast<const float4*>(as + i * 4 * TK + ao[u]);
            }
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                ulonglong2 b[TN / 2];        // (k, k + 1) of a pair of columns
#pragma unroll
                for (int j = 0; j < TN / 2; ++j)
                    b[j] = *reinterpret_cast<const ulonglong2*>(ws + j * 8 * 2 * TK + wo[2 * kq + half]);
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const unsigned long long d = twice(half ? a[i].z : a[i].x);
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], d, b[j].x);
                }
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const unsigned long long d = twice(half ? a[i].w : a[i].y);
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], d, b[j].y);
                }
            }
        }
        if (more) put_w(buf ^ 1);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
    // the groups' sums meet in shared memory: [GK][TBM][TBN + 1]
    constexpr int RP = TBN + 1;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j)
            sm[(grp * TBM + ty + 4 * i) * RP + tx + 8 * j] = __uint_as_float((unsigned)(acc[i][j >> 1] >> (32 * (j & 1))));
    __syncthreads();
    for (int e = threadIdx.x; e < TBM * TBN; e += NT) {
        const int r = e / TBN, c = e % TBN, gm = m0 + r, gn = n0 + c;
        const float* p = sm + r * RP + c;
        if (gm < M && gn < N) C[(size_t)gm * N + gn] = (p[0] + p[TBM * RP]) + (p[2 * TBM * RP] + p[3 * TBM * RP]);
    }
}

template <typename TW, int WM, int WN, int TM, int TN, int MINB>
static int gemm_f32_tiled(const float* A, const TW* W, float* C, int M, int N, int K, cudaStream_t stream) {
    constexpr int TBM = WM * 4 * TM, TBN = WN * 8 * TN;
    constexpr int ring = 2 * (TBM + TBN) * TK, sums = GK * TBM * (TBN + 1);
    constexpr size_t smem = (ring > sums ? ring : sums) * sizeof(float);
    auto k = gemm_f32_tiled_kernel<TW, WM, WN, TM, TN, MINB>;
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
    }
    lumen_launch(k, dim3((N + TBN - 1) / TBN, (M + TBM - 1) / TBM), dim3(GK * WM * WN * 32), smem, stream, A, W, C, M, N, K);
    LUMEN_LAUNCH_CHECK();
    return 0;
}

template <typename TW>
static int gemm_f32_go(const float* A, const TW* W, float* C, int M, int N, int K, cudaStream_t stream) {
    if ((M + BM - 1) / BM > 65535) return LUMEN_ERR_UNSUPPORTED;
    const bool vec = (K & 3) == 0 && ((uintptr_t)A & 15) == 0 && ((uintptr_t)W & (4 * sizeof(TW) - 1)) == 0;
    // More than 32 short rows go to the small-tile kernel: the large tiles' ring, four groups and their sums pay from some steps
    // of 64 columns on (us, small / large tiles: 300 x 4,096 x 16 6.4 / 13.9, 4,000 x 4,096 x 16 32 / 120, 33 x 64 x 32 3.1 / 5.1,
    // 1,000 x 1,000 x 48 8.9 / 10.0, 4,000 x 4,096 x 64 91 / 121, but 300 x 4,096 x 64 16.4 / 14.0). The same sums either way.
    const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
    const bool is_short = M > 32 && (K <= 48 || (K <= 64 && tiles >= 512));
    if (!vec || is_short) {
        const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
        if (K <= BK) lumen_launch(gemm_f32_kernel<TW, 1>, grid, dim3(256), 0, stream, A, W, C, M, N, K);
        else if (K <= 2 * BK) lumen_launch(gemm_f32_kernel<TW, 2>, grid, dim3(256), 0, stream, A, W, C, M, N, K);
        else lumen_launch(gemm_f32_kernel<TW, GK>, grid, dim3(256), 0, stream, A, W, C, M, N, K);
        LUMEN_LAUNCH_CHECK();
        return 0;
    }
    // tiles no higher than the rows there are: 16 x 32, 32 x 32 (24 rows x 16,384 x 2,048: 72 us) and 64 x 64
    if (M <= 16) return gemm_f32_tiled<TW, 1, 1, 4, 4, 3>(A, W, C, M, N, K, stream);
    if (M <= 32) return gemm_f32_tiled<TW, 1, 1, 8, 4, 3>(A, W, C, M, N, K, stream);
    return gemm_f32_tiled<TW, 2, 1, 8, 8, 1>(A, W, C, M, N, K, stream);
}

LUMEN_API int lumen_gemm_f32(const float* A, const void* W, int w_is_bf16, float* C, int M, int N,
                             int K, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return LUMEN_ERR_BAD_ARGUMENT;
    return w_is_bf16 ? gemm_f32_go(A, (const __nv_bfloat16*)W, C, M, N, K, stream)
                     : gemm_f32_go(A, (const float*)W, C, M, N, K, stream);
}
