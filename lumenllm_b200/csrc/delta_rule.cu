// The gated delta rule with a decay of its own for every key channel: a linear recurrence over
// time with a matrix state S [d, dv] per head,
//   S <- diag(g_t) S;  u = beta_t (v_t - S^T k_t);  S <- S + k_t u^T;  o_t = S^T q_t,
// where q_t and k_t are unit vectors (x / sqrt(sum x^2 + 1e-6), q also times d^-1/2), beta_t =
// sigmoid(b_t) and g_t = exp(-exp(A_log_h) softplus(a_t + dt_bias)), a_t one number a (head, key
// channel). Query/key head of value head h: h / (H / G). Everything is float32.
//
// A block takes one (sequence, head, slice of value channels) and walks the sequence's tokens of
// the step strictly in order, so a token's sums do not depend on how the sequence was cut or
// batched. A column j of S is independent of the others:
//   r = sum_i g_i S_ij k_i,  w = sum_i g_i S_ij q_i,  u_j = beta (v_j - r),  o_j = w + u_j (k . q),
//   S_ij <- g_i S_ij + k_i u_j,
// so the DR_ROWS rows a thread keeps in registers are read once a token; the NS threads of a
// column (adjacent lanes) add r by shuffles at once, since u_j waits for it, and w a chunk at a time: the
// shares of eight tokens change lanes so that a lane adds up a token of its own (7 shuffles for 8 tokens
// where one token after the other takes 8 log2(NS)). Four warps of a block share a staged row, and what they read of
// it (48 values a thread and token) is what bounds a token, with the chain of dependent steps: 220 of its 400
// cycles go to shared-memory reads. 2,048 tokens of 16 heads of 128 x 128: 466 us with the kernel that
// prepares them (732 with 16 threads a column, 8 rows each, and w summed token by token), four sequences of 2,048 tokens
// in all: 400 (668), one token of 64 sequences: 36 (44). Two columns a thread over 16 lanes halve the reads and
// lengthen the chain by two shuffles: 497 and 412 us.
// What does not depend on the state is made for
// all tokens at once by a kernel of its own (a warp a (token, head): normed q and k, the decays,
// k . q and beta, one row [q | k | g | k.q, beta] of a scratch matrix), so that the walk itself is
// nothing but the recurrence: rows are staged DR_CHUNK tokens at a time by asynchronous copies, the
// next chunk under way while this one is walked, with no barrier between a chunk's tokens. The
// state is stored [H, dv, d] (a column's rows lie together).
#include "common.cuh"

#define DR_THREADS 128
#define DR_ROWS 16          // rows of S a thread keeps (4 groups of 4 consecutive rows)
#define DR_CHUNK 8
#define DR_PREP_WARPS 4

__device__ __forceinline__ float dr_parts(const float* p, int S, size_t stride) {
    float x = p[0];
    for (int s = 1; s < S; ++s) x += p[(size_t)s * stride];
    return x;
}
// Two float32 operations in one instruction, each rounded as by itself.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f32x2 pair2(float lo, float hi) {
    f32x2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 unpair2(f32x2 a) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(a));
    return v;
}
__device__ __forceinline__ float dr_softplus(float x) { return x > 20.0f ? x : log1pf(expf(x)); }
__device__ __forceinline__ void dr_cp4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void dr_cp16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void dr_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void dr_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// prep [N, H, 3 dp + 4]: row (n, h) = [q normed and scaled (dp) | k normed (dp) | decays (dp) | k . q, beta, 0, 0];
// the dp - d values past a head's own are 0, 0 and 1.
__global__ void __launch_bounds__(32 * DR_PREP_WARPS)
delta_prepare_kernel(const float* __restrict__ x, int C, int q_col, int k_col,
                     const float* __restrict__ u, int uS, size_t u_stride, int uW, int b_col,
                     const float* __restrict__ a, int aS, size_t a_stride, const float* __restrict__ dt_bias,
                     const float* __restrict__ a_log, float* __restrict__ prep, int N, int H, int G, int d, int dp) {
    // No early trigger here: the walk that follows has about one block an SM and must find the SMs
    // empty, so that its blocks are spread one an SM; started under this kernel's blocks they were
    // packed several an SM wherever room was, and the walk took twice as long.
    pdl_wait();
    const int n = blockIdx.x, h = blockIdx.y * DR_PREP_WARPS + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (h >= H) return;
    const int g = h / (H / G);
    const float a_neg = -expf(a_log[h]);
    const float q_scale = rsqrtf((float)d);
    const float* row = x + (size_t)n * C;
    float* out = prep + ((size_t)n * H + h) * (3 * dp + 4);
    float sq = 0.0f, sk = 0.0f;
    for (int e = lane; e < d; e += 32) {
        const float qv = row[q_col + g * d + e], kv = row[k_col + g * d + e];
        sq += qv * qv;
        sk += kv * kv;
    }
    sq = warp_sum(sq);
    sk = warp_sum(sk);
    const float rq = q_scale / sqrtf(sq + 1e-6f), rk = 1.0f / sqrtf(sk + 1e-6f);
    float dot = 0.0f;
    for (int e = lane; e < dp; e += 32) {
        float qv = 0.0f, kv = 0.0f, gv = 1.0f;
        if (e < d) {
            qv = row[q_col + g * d + e] * rq;
            kv = row[k_col + g * d + e] * rk;
            const float av = dr_parts(a + (size_t)n * H * d + h * d + e, aS, a_stride) + dt_bias[h * d + e];
            gv = expf(a_neg * dr_softplus(av));
        }
        out[e] = qv;
        out[dp + e] = kv;
        out[2 * dp + e] = gv;
        dot += qv * kv;
    }
    dot = warp_sum(dot);
    if (lane < 4) {
        float v = 0.0f;
        if (lane == 0) v = dot;
        if (lane == 1) v = 1.0f / (1.0f + expf(-dr_parts(u + (size_t)n * uW + b_col + h, uS, u_stride)));
        out[3 * dp + lane] = v;
    }
}

// NS: threads that share a column of S (a power of two), NS DR_ROWS >= d; every offset of the walk is a constant
// of the instance. AHEAD: a token's rows are read from shared memory while the one before is worked on, which
// takes twice the registers: for steps of several tokens a sequence. THREADS: of a block. Same sums either way.
template <int NS, bool AHEAD, int THREADS>
__global__ void __launch_bounds__(THREADS)
delta_rule_kernel(const float* __restrict__ x, int C, int v_col, const float* __restrict__ prep,
                  float* __restrict__ state, size_t slot_stride, const int* __restrict__ cu_q,
                  const int* __restrict__ seq_slot, float* __restrict__ y, int H, int d, int dv, int vec) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr int ROWS = DR_ROWS;
    constexpr int dp = NS * ROWS;                   // d padded to what the threads of a column hold
    constexpr int GR = ROWS / 4;
    constexpr int PW = 3 * dp + 4;
    constexpr int cols = THREADS / NS;
    float* rows = sm;                               // [2][DR_CHUNK][PW]
    float* vs = sm + 2 * DR_CHUNK * PW;             // [2][DR_CHUNK][cols]
    const int b = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int t_begin = cu_q[b], t_end = cu_q[b + 1];
    if (t_end <= t_begin) return;
    const int s = tid % NS, cj = tid / NS, j = blockIdx.z * cols + cj;
    const bool live = j < dv;
    float* Sj = state + (size_t)seq_slot[b] * slot_stride + ((size_t)h * dv + (live ? j : 0)) * d;
    f32x2 S[2 * GR];                                // rows 4 (i NS + s) .. + 3 in S[2 i], S[2 i + 1]
#pragma unroll
    for (int i = 0; i < GR; ++i) {
        const int row0 = (i * NS + s) * 4;
        if (vec) {                                  // d a multiple of 4 and the state's columns on 16 bytes
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (live && row0 < d) v = *reinterpret_cast<const float4*>(Sj + row0);
            S[2 * i] = pair2(v.x, v.y);
            S[2 * i + 1] = pair2(v.z, v.w);
        } else {
            float v[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = (live && row0 + c < d) ? Sj[row0 + c] : 0.0f;
            S[2 * i] = pair2(v[0], v[1]);
            S[2 * i + 1] = pair2(v[2], v[3]);
        }
    }

    auto issue = [&](int t0, int buf) {
        const int nt = min(DR_CHUNK, t_end - t0);
        constexpr int pieces = PW / 4;
        float* rb = rows + buf * DR_CHUNK * PW;
        for (int i = tid; i < nt * pieces; i += THREADS) {
            const int tt = i / pieces, p = i - tt * pieces;
            dr_cp16(rb + tt * PW + 4 * p, prep + ((size_t)(t0 + tt) * H + h) * PW + 4 * p);
        }
        float* vb = vs + buf * DR_CHUNK * cols;
        for (int i = tid; i < nt * cols; i += THREADS) {
            const int tt = i / cols, c = i - tt * cols, jj = blockIdx.z * cols + c;
            if (jj < dv) dr_cp4(vb + i, x + (size_t)(t0 + tt) * C + v_col + h * dv + jj);
            else vb[i] = 0.0f;
        }
        dr_commit();
    };
    issue(t_begin, 0);

    for (int t0 = t_begin, it = 0; t0 < t_end; t0 += DR_CHUNK, ++it) {
        const int nt = min(DR_CHUNK, t_end - t0), buf = it & 1;
        if (t0 + DR_CHUNK < t_end) {
            issue(t0 + DR_CHUNK, buf ^ 1);          // under way while this chunk is walked
            dr_wait<1>();
        } else {
            dr_wait<0>();
        }
        __syncthreads();
        const float* rb = rows + buf * DR_CHUNK * PW;
        const float* vb = vs + buf * DR_CHUNK * cols;
        float wt[DR_CHUNK];                         // this lane's share of w (lane 0 of a column: and of u_j k.q)
        struct Row { ulonglong2 q[GR], k[GR], g[GR]; float v, kq, beta; };
        auto load = [&](int t) {
            Row x;
            const float* p = rb + t * PW + 4 * s;
#pragma unroll
            for (int i = 0; i < GR; ++i) {
                x.g[i] = *reinterpret_cast<const ulonglong2*>(p + 2 * dp + 4 * i * NS);
                x.k[i] = *reinterpret_cast<const ulonglong2*>(p + dp + 4 * i * NS);
                x.q[i] = *reinterpret_cast<const ulonglong2*>(p + 4 * i * NS);
            }
            const float2 e = *reinterpret_cast<const float2*>(rb + t * PW + 3 * dp);
            x.kq = e.x;
            x.beta = e.y;
            x.v = vb[t * cols + cj];
            return x;
        };
        // The chain from one token's S to the next one's is: S g, the sums of r over four short chains, their
        // lanes, u_j, S. All else (w, the next token's rows) is put where it waits for shuffles.
        auto walk = [&](const Row& x, Row& next, int t_next) {
            f32x2 rp[GR], wp[2];
#pragma unroll
            for (int i = 0; i < GR; ++i) {
                S[2 * i] = mul2(S[2 * i], x.g[i].x);
                S[2 * i + 1] = mul2(S[2 * i + 1], x.g[i].y);
            }
#pragma unroll
            for (int i = 0; i < GR; ++i) rp[i] = fma2(S[2 * i + 1], x.k[i].y, mul2(S[2 * i], x.k[i].x));
            const float2 r2 = unpair2(add2(add2(rp[0], rp[1]), add2(rp[2], rp[3])));
            float r = r2.x + r2.y;
            if (AHEAD && t_next >= 0) next = load(t_next);
#pragma unroll
            for (int o = NS >> 1; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
#pragma unroll
            for (int i = 0; i < GR; ++i) {
                wp[i & 1] = i < 2 ? mul2(S[2 * i], x.q[i].x) : fma2(S[2 * i], x.q[i].x, wp[i & 1]);
                wp[i & 1] = fma2(S[2 * i + 1], x.q[i].y, wp[i & 1]);
            }
            const float2 w2 = unpair2(add2(wp[0], wp[1]));
            const float w = w2.x + w2.y;
            const float uj = x.beta * (x.v - r);
            const f32x2 u2 = pair2(uj, uj);
#pragma unroll
            for (int i = 0; i < GR; ++i) {
                S[2 * i] = fma2(x.k[i].x, u2, S[2 * i]);
                S[2 * i + 1] = fma2(x.k[i].y, u2, S[2 * i + 1]);
            }
            if (!AHEAD && t_next >= 0) next = load(t_next);
            return s == 0 ? fmaf(uj, x.kq, w) : w;
        };
        Row now = load(0), next = now;
        if (AHEAD && nt == DR_CHUNK) {                       // no branch between the tokens
#pragma unroll
            for (int t = 0; t < DR_CHUNK; ++t) {
                wt[t] = walk(now, next, t + 1 < DR_CHUNK ? t + 1 : -1);
                now = next;
            }
        } else {
#pragma unroll
            for (int t = 0; t < DR_CHUNK; ++t) {
                wt[t] = 0.0f;
                if (t >= nt) continue;
                wt[t] = walk(now, next, t + 1 < nt ? t + 1 : -1);
                now = next;
            }
        }
        // Halve the tokens a lane has with every step over the column's lanes; what is left of the steps adds
        // up the one token it has. The tree of lanes is the same for every place in the chunk.
        int n = DR_CHUNK, first = 0;
#pragma unroll
        for (int o = NS >> 1; o > 0; o >>= 1) {
            if (n > 1) {
                n >>= 1;
                const bool up = (s & o) != 0;
#pragma unroll
                for (int i = 0; i < DR_CHUNK / 2; ++i) {
                    if (i >= n) break;
                    const float give = up ? wt[i] : wt[i + n], keep = up ? wt[i + n] : wt[i];
                    wt[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
                first += up ? n : 0;
            } else {
                wt[0] += __shfl_xor_sync(0xffffffffu, wt[0], o);
            }
        }
        constexpr int OWN = NS >= DR_CHUNK ? 1 : DR_CHUNK / NS, TWINS = NS > DR_CHUNK ? NS / DR_CHUNK : 1;
        if (live && (s & (TWINS - 1)) == 0) {
#pragma unroll
            for (int i = 0; i < OWN; ++i)
                if (first + i < nt) y[(size_t)(t0 + first + i) * H * dv + h * dv + j] = wt[i];
        }
        __syncthreads();                            // this chunk has been read by everyone before its buffer is filled again
    }
    if (live) {
#pragma unroll
        for (int i = 0; i < GR; ++i) {
            const int row0 = (i * NS + s) * 4;
            const float2 a = unpair2(S[2 * i]), c = unpair2(S[2 * i + 1]);
            if (vec) {
                if (row0 < d) *reinterpret_cast<float4*>(Sj + row0) = make_float4(a.x, a.y, c.x, c.y);
            } else {
                if (row0 < d) Sj[row0] = a.x;
                if (row0 + 1 < d) Sj[row0 + 1] = a.y;
                if (row0 + 2 < d) Sj[row0 + 2] = c.x;
                if (row0 + 3 < d) Sj[row0 + 3] = c.y;
            }
        }
    }
}

// Threads a column for d key channels.
static inline int delta_rule_threads(int d) {
    int NS = 1;
    while (NS * DR_ROWS < d) NS <<= 1;
    return NS;
}

// Floats of scratch lumen_delta_rule needs for every (token, head) with d key channels.
LUMEN_API int lumen_delta_rule_scratch_row(int d) {
    return 3 * delta_rule_threads(d) * DR_ROWS + 4;
}

// x float32 [N, C]: the convolved and activated q (G heads of d, from column q_col), k (k_col)
// and v (H heads of dv, v_col). u: the projection's partial sums [uS, N, uW] with the H beta
// logits from column b_col. a: partial sums [aS, N, H d] of the decay logits (before dt_bias).
// state float32, row seq_slot[b] of stride slot_stride holds [H, dv, d]. y float32 [N, H dv]. prep:
// N H lumen_delta_rule_scratch_row(d) floats of scratch.
LUMEN_API int lumen_delta_rule(const float* x, int C, int q_col, int k_col, int v_col, const float* u, int uS,
                               long long u_stride, int uW, int b_col, const float* a, int aS, long long a_stride,
                               const float* dt_bias, const float* a_log, float* state, long long slot_stride,
                               const int* cu_q, const int* seq_slot, int n_seqs, float* y, float* prep, int N, int H,
                               int G, int d, int dv, cudaStream_t stream) {
    if (n_seqs <= 0 || N <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || d <= 0 || dv <= 0 || d > 32 * DR_ROWS || uS < 1 || aS < 1 || H > 65535)
        return LUMEN_ERR_UNSUPPORTED;
    if (q_col < 0 || k_col < 0 || v_col < 0 || q_col + G * d > C || k_col + G * d > C || v_col + H * dv > C ||
        b_col < 0 || b_col + H > uW || !prep)
        return LUMEN_ERR_BAD_ARGUMENT;
    const int NS = delta_rule_threads(d), dp = NS * DR_ROWS;
    // Heads wider than 256 leave a block of 128 threads four columns to share a staged row: right while every block has an SM,
    // else twice as many (us, 128 / 256 threads, heads of 500 x 64: one sequence of 2,048 tokens, 64 blocks of 128, 629 / 821;
    // four of 512 255 / 235; one token of 64 sequences 42 / 32, of 200 131 / 90).
    const bool wide = NS == 32 && (long long)n_seqs * H * ((dv + DR_THREADS / NS - 1) / (DR_THREADS / NS)) > 148;
    const int threads = wide ? 2 * DR_THREADS : DR_THREADS, cols = threads / NS;
    const int vec = (d & 3) == 0 && (slot_stride & 3) == 0 && ((uintptr_t)state & 15) == 0;
    dim3 pgrid(N, (H + DR_PREP_WARPS - 1) / DR_PREP_WARPS);
    if (pgrid.y > 65535) return LUMEN_ERR_UNSUPPORTED;
    lumen_launch(delta_prepare_kernel, pgrid, dim3(32 * DR_PREP_WARPS), 0, stream, x, C, q_col, k_col, u, uS,
                 (size_t)u_stride, uW, b_col, a, aS, (size_t)a_stride, dt_bias, a_log, prep, N, H, G, d, dp);
    LUMEN_LAUNCH_CHECK();
    dim3 grid(n_seqs, H, (dv + cols - 1) / cols);
    if (grid.z > 65535) return LUMEN_ERR_UNSUPPORTED;
    const size_t smem = (size_t)2 * DR_CHUNK * (3 * dp + 4 + cols) * sizeof(float);
#define DR_LAUNCH(S, A, T)                                                                                            \
    do {                                                                                                              \
        auto k = delta_rule_kernel<S, A, T>;                                                                           \
        if (smem > 48 * 1024) {                                                                                       \
            cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);          \
            if (e != cudaSuccess) return (int)e;                                                                      \
        }                                                                                                             \
        lumen_launch(k, grid, dim3(T), smem, stream, x, C, v_col, (const float*)prep, state,                 \
                     (size_t)slot_stride, cu_q, seq_slot, y, H, d, dv, vec);                                          \
    } while (0)
    // reading ahead takes twice the registers, and a second such block an SM is worth more (heads of 512 x 128, 8 a sequence, four
    // sequences of 512 tokens: 845 us ahead, 750 not)
    const bool ahead = N > n_seqs && !(wide && (long long)grid.x * grid.y * grid.z > 148);
#define DR_GO(S, T) { if (ahead) DR_LAUNCH(S, true, T); else DR_LAUNCH(S, false, T); }
    switch (NS) {
        case 1: DR_GO(1, DR_THREADS) break;
        case 2: DR_GO(2, DR_THREADS) break;
        case 4: DR_GO(4, DR_THREADS) break;
        case 8: DR_GO(8, DR_THREADS) break;
        case 16: DR_GO(16, DR_THREADS) break;
        default: if (wide) DR_GO(32, 2 * DR_THREADS) else DR_GO(32, DR_THREADS)
    }
#undef DR_GO
#undef DR_LAUNCH
    LUMEN_LAUNCH_CHECK();
    return 0;
}
