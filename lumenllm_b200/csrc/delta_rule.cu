// The gated delta rule with a decay of its own for every key channel: a linear recurrence over
// time with a matrix state S [d, dv] per head,
//   S <- diag(g_t) S;  u = beta_t (v_t - S^T k_t);  S <- S + k_t u^T;  o_t = S^T q_t,
// where q_t and k_t are unit vectors (x / sqrt(sum x^2 + 1e-6), q also times d^-1/2), beta_t =
// sigmoid(b_t) and g_t = exp(-exp(A_log_h) softplus(a_t + dt_bias)), a_t one number a (head, key
// channel). Query/key head of value head h: h / (H / G). Everything is float32.
//
// A block takes one (sequence, head, slice of value channels) and walks the sequence's tokens of
// the step strictly in order, so a token's sums do not depend on how the
// sequence was cut or batched (heads of 65 to 128 go in chunks where a sequence has 48 tokens or more in the step, below: their sums
// depend on where it is cut, never on other sequences). A column j of S is independent of the others:
//   r = sum_i g_i S_ij k_i,  w = sum_i g_i S_ij q_i,  u_j = beta (v_j - r),  o_j = w + u_j (k . q),
//   S_ij <- g_i S_ij + k_i u_j,
// so the DR_ROWS rows a thread keeps in registers are read once a token; the NS threads of a
// column (adjacent lanes) add r by shuffles at once, since u_j waits for it, and w a chunk at a time: the
// shares of eight tokens change lanes so that a lane adds up a token of its own (7 shuffles for 8 tokens
// where one token after the other takes 8 log2(NS)). Four warps of a block share a staged row, and what they read of
// it (48 values a thread and token) is what bounds a token, with the chain of dependent steps: 220 of its 400
// cycles go to shared-memory reads. Of 16 heads of 128 x 128, one token of 64 sequences: 36 us with the kernel that
// prepares them (44 with 16 threads a column, 8 rows each, and w summed token by token), 200 sequences of eight tokens 302. Prompts, before
// they went in chunks: 2,048 tokens 466 (732), four sequences of 2,048 tokens in all 400 (668); two columns a thread over 16 lanes halve the
// reads and lengthen the chain by two shuffles: 497 and 412.
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
// What a (token, head) needs, in one place.
struct DrIn {
    const float* x;           // [N, C]
    const float* u;           // projection partial sums with the beta logits
    const float* a;           // partial sums of the decay logits
    const float* dt_bias;
    const float* a_log;
    size_t u_stride, a_stride;
    int C, q_col, k_col, uS, uW, b_col, aS, H, G, d;
};
// One row, by a warp. out: dp floats each of q, k and decays, then k . q and beta.
__device__ __forceinline__ void dr_prepare_row(const DrIn& in, int n, int h, int dp, float* out) {
    const int lane = threadIdx.x & 31, d = in.d;
    const int g = h / (in.H / in.G);
    const float a_neg = -expf(in.a_log[h]);
    const float q_scale = rsqrtf((float)d);
    const float* row = in.x + (size_t)n * in.C;
    float sq = 0.0f, sk = 0.0f;
    for (int e = lane; e < d; e += 32) {
        const float qv = row[in.q_col + g * d + e], kv = row[in.k_col + g * d + e];
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
            qv = row[in.q_col + g * d + e] * rq;
            kv = row[in.k_col + g * d + e] * rk;
            const float av = dr_parts(in.a + (size_t)n * in.H * d + h * d + e, in.aS, in.a_stride) + in.dt_bias[h * d + e];
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
        if (lane == 1) v = 1.0f / (1.0f + expf(-dr_parts(in.u + (size_t)n * in.uW + in.b_col + h, in.uS, in.u_stride)));
        out[3 * dp + lane] = v;
    }
}

__global__ void __launch_bounds__(32 * DR_PREP_WARPS)
delta_prepare_kernel(const DrIn in, float* __restrict__ prep, int dp) {
    // No early trigger here: the walk that follows has about one block an SM and must find the SMs
    // empty, so that its blocks are spread one an SM; started under this kernel's blocks they were
    // packed several an SM wherever room was, and the walk took twice as long.
    pdl_wait();
    const int n = blockIdx.x, h = blockIdx.y * DR_PREP_WARPS + (threadIdx.x >> 5);
    if (h >= in.H) return;
    dr_prepare_row(in, n, h, dp, prep + ((size_t)n * in.H + h) * (3 * dp + 4));
}

// NS: threads that share a column of S (a power of two), NS DR_ROWS >= d; every offset of the walk is a constant
// of the instance. AHEAD: a token's rows are read from shared memory while the one before is worked on, which
// takes twice the registers: for steps of several tokens a sequence. THREADS: of a block. Same sums either way.
// row0: the row of the sequence's first token, the next ones row_stride floats on; zblock: which columns.
template <int NS, bool AHEAD, int THREADS>
__device__ __forceinline__ void dr_walk(float* sm, const float* __restrict__ x, int C, int v_col, const float* __restrict__ row0,
                                        size_t row_stride, int t_begin, int t_end, int zblock, float* __restrict__ S_head,
                                        float* __restrict__ y, int H, int d, int dv, int vec) {
    constexpr int ROWS = DR_ROWS;
    constexpr int dp = NS * ROWS;                   // d padded to what the threads of a column hold
    constexpr int GR = ROWS / 4;
    constexpr int PW = 3 * dp + 4;
    constexpr int cols = THREADS / NS;
    float* rows = sm;                               // [2][DR_CHUNK][PW]
    float* vs = sm + 2 * DR_CHUNK * PW;             // [2][DR_CHUNK][cols]
    const int h = blockIdx.y, tid = threadIdx.x;
    const int s = tid % NS, cj = tid / NS, j = zblock * cols + cj;
    const bool live = j < dv;
    float* Sj = S_head + (size_t)(live ? j : 0) * d;
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
            dr_cp16(rb + tt * PW + 4 * p, row0 + (size_t)(t0 + tt - t_begin) * row_stride + 4 * p);
        }
        float* vb = vs + buf * DR_CHUNK * cols;
        for (int i = tid; i < nt * cols; i += THREADS) {
            const int tt = i / cols, c = i - tt * cols, jj = zblock * cols + c;
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

template <int NS, bool AHEAD, int THREADS>
__global__ void __launch_bounds__(THREADS)
delta_rule_kernel(const float* __restrict__ x, int C, int v_col, const float* __restrict__ prep,
                  float* __restrict__ state, size_t slot_stride, const int* __restrict__ cu_q,
                  const int* __restrict__ seq_slot, float* __restrict__ y, int H, int d, int dv, int vec) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    constexpr int PW = 3 * NS * DR_ROWS + 4;
    const int b = blockIdx.x, h = blockIdx.y, t_begin = cu_q[b], t_end = cu_q[b + 1];
    if (t_end <= t_begin) return;
    dr_walk<NS, AHEAD, THREADS>(sm, x, C, v_col, prep + ((size_t)t_begin * H + h) * PW, (size_t)H * PW, t_begin, t_end, blockIdx.z,
                                state + (size_t)seq_slot[b] * slot_stride + (size_t)h * dv * d, y, H, d, dv, vec);
}

// ------------------------------------------------------------------- sixteen tokens at a time
// For heads of 65 to 128 key channels a sequence's tokens go in chunks of sixteen (from its first of the step on). With
// P_t = g_1 .. g_t the decays since the chunk's start, channel by channel, and S the state there,
//   u_t = beta_t (v_t - S^T (P_t k_t) - sum_{i<t} A_ti u_i),   A_ti = k_t . (g_{i+1} .. g_t k_i)
//   o_t = S^T (P_t q_t) + sum_{i<=t} B_ti u_i,                 B_ti = q_t . (g_{i+1} .. g_t k_i)
//   S  <- P_16 S + sum_i (g_{i+1} .. g_16 k_i) u_i^T,
// the same numbers as token by token, in another order of sums. A, B, the three sets of scaled vectors and
// T = (1 + beta A)^-1 beta (so that u = T (v - S^T P k)) need no state: a kernel makes them for all chunks at once. Every
// factor is a product of decays, at most 1, never a quotient; T's entries are at most 1 in size, as unit vectors and beta
// below 1 make every step a contraction. What is left to the walk is three products with S a chunk, which have no chain
// from token to token. A thread keeps 4 key channels of 4 columns of S, a warp all channels of four columns; sums over
// channels change lanes a chunk at a time, 64 sums by 62 exchanges. What bounds it is instructions: pairs are of
// neighbouring channels, as they lie in the records, and u is also written twice over, so that no operand of a two-product
// instruction has to be put together. Zeros above the diagonal are not multiplied, so that what is not finite in a token
// reaches no earlier one.
// Sequences of fewer than DC_MIN tokens walk them one by one, with the sums of a decode step: a few chunks are no faster
// (us, 16 heads of 128 x 128, chunks / tokens: 33 tokens 14.5 / 13.6, 64 sequences of 24 218 / 215, 200 tokens 36 / 50). How a sequence
// goes is its own number of tokens in the step alone.
// Their rows lie where their tokens' shares of records would (a record a sequence of any length took 66 MB for 128 sequences of two
// tokens of 16 heads; 11 so), and a step that is known to have no longer sequences goes to the kernels above (us, 128 sequences of two tokens
// 136 here, 128 there; 200 of eight 317 / 302).
// 2,048 tokens of 16 heads of 128 x 128: 303 us with the kernel ahead (465 token by token), four sequences of 512 241 (339), nine
// of 300 286 (396), one of 200 36 (50). The walk issues 1,480 instructions a chunk and warp, one in 2.6 cycles. Tried: two warps for the
// same columns, one for P k and u, one for P q and o: 286 for one sequence, but 255 and 313 for four and nine.
#define DC_T 16
#define DC_MIN 48
#define DC_D 128
#define DC_PITCH 20                                              // floats a row of T and of B
#define DC_KT 0
#define DC_QT (DC_T * DC_D)
#define DC_KB (2 * DC_T * DC_D)
#define DC_P (3 * DC_T * DC_D)
#define DC_TM (DC_P + DC_D)
#define DC_BM (DC_TM + DC_T * DC_PITCH)
#define DC_REC (DC_BM + DC_T * DC_PITCH)                         // floats of a (chunk, head)
#define DC_ROW (3 * DC_D + 4)                                    // a token's row, as above
#define DC_WARPS 16                                              // of the kernel that prepares: one a token
#define DC_TOKEN (DC_REC / DC_T)                                 // floats of scratch a (token, head)
static_assert(DC_REC % DC_T == 0 && DC_ROW <= DC_TOKEN && DC_TOKEN % 4 == 0 && DC_ROW % 4 == 0, "a short sequence's rows lie where its share of a record would");

// The block of the preparing kernel that sequence b's chunks begin at: room for every cut of N tokens.
__device__ __forceinline__ int dc_first(const int* cu_q, int b) { return cu_q[b] / DC_T + b; }
// The last sequence whose blocks begin at or before block x: for a whole warp, 32 sequences a look.
__device__ __forceinline__ int dc_of_block(const int* cu_q, int n_seqs, int x) {
    int lo = 0, n = n_seqs;
    while (n > 1) {
        const int step = (n + 31) / 32, b = lo + (int)(threadIdx.x & 31) * step;
        const unsigned before = __ballot_sync(0xffffffffu, b < lo + n && dc_first(cu_q, min(b, n_seqs)) <= x);
        const int k = max(__popc(before) - 1, 0);           // they are ordered: the first k + 1 lanes
        n = min(step, n - k * step);
        lo += k * step;
    }
    return lo;
}
// Where sequence b's share of the scratch begins, in (token, head) floats: records chunk by chunk, or rows token by token, all heads
// side by side. A sequence in chunks may need one record more than its tokens' shares, the others do not.
__host__ __device__ __forceinline__ size_t dc_place(int tokens, int seqs) {
    return (size_t)tokens * DC_TOKEN + (size_t)DC_REC * (seqs < tokens / DC_MIN ? seqs : tokens / DC_MIN);
}

__global__ void __launch_bounds__(32 * DC_WARPS)
delta_chunk_prepare_kernel(const DrIn in, float* __restrict__ prep, const int* __restrict__ cu_q, int n_seqs) {
    pdl_wait();              // no early trigger, as above
    __shared__ __align__(16) float rows[DC_T * DC_ROW];
    __shared__ float A[DC_T][DC_T + 1];
    const int h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int lo = dc_of_block(cu_q, n_seqs, (int)blockIdx.x);
    const int t_begin = cu_q[lo], t_end = cu_q[lo + 1], t0 = t_begin + ((int)blockIdx.x - dc_first(cu_q, lo)) * DC_T;
    if (t0 < t_begin || t0 >= t_end) return;
    const int nt = min(DC_T, t_end - t0);
    float* place = prep + dc_place(t_begin, lo) * in.H;
    if (t_end - t_begin < DC_MIN) {                // rows only; the warps of the first blocks share out all heads' tokens
        const int i = h * DC_WARPS + warp;
        if (i < nt * in.H)
            dr_prepare_row(in, t0 + i / in.H, i % in.H, DC_D, place + ((size_t)(t0 - t_begin) * in.H + i) * DC_ROW);
        return;
    }
    float* rec = place + ((size_t)((t0 - t_begin) / DC_T) * in.H + h) * DC_REC;
    {
        float* row = rows + warp * DC_ROW;
        if (warp < nt) {
            dr_prepare_row(in, t0 + warp, h, DC_D, row);
        } else {                                   // no token: nothing decays, nothing is written
            for (int e = lane; e < DC_ROW; e += 32) row[e] = (e >= 2 * DC_D && e < 3 * DC_D) ? 1.0f : 0.0f;
        }
    }
    __syncthreads();
    {                                              // columns i = warp of A and B, a lane four channels
        const int i = warp;
        float4 p = *reinterpret_cast<const float4*>(rows + i * DC_ROW + DC_D + 4 * lane);
        f32x2 v[DC_T];                             // this lane's shares of A_ti and B_ti
#pragma unroll
        for (int t = 0; t < DC_T; ++t) {
            v[t] = 0ull;
            if (t < i) continue;
            const float* r = rows + t * DC_ROW + 4 * lane;
            const float4 q = *reinterpret_cast<const float4*>(r), k = *reinterpret_cast<const float4*>(r + DC_D);
            if (t > i) {
                const float4 g = *reinterpret_cast<const float4*>(r + 2 * DC_D);
                p.x *= g.x;
                p.y *= g.y;
                p.z *= g.z;
                p.w *= g.w;
            }
            v[t] = pair2(fmaf(p.y, k.y, p.x * k.x) + fmaf(p.w, k.w, p.z * k.z), fmaf(p.y, q.y, p.x * q.x) + fmaf(p.w, q.w, p.z * q.z));
        }
#pragma unroll
        for (int o = 16; o > 1; o >>= 1) {         // lanes 2 t and 2 t + 1 get the sums of t, but for their own two shares
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int t = 0; t < o / 2; ++t) {
                const f32x2 give = up ? v[t] : v[t + o / 2], keep = up ? v[t + o / 2] : v[t];
                v[t] = add2(keep, __shfl_xor_sync(0xffffffffu, give, o));
            }
        }
        const float2 ab = unpair2(add2(v[0], __shfl_xor_sync(0xffffffffu, v[0], 1)));
        const int t = lane >> 1;
        if (t >= i) {
            if (lane & 1) rec[DC_BM + t * DC_PITCH + i] = ab.y;
            else A[t][i] = ab.x;
        }
    }
    __syncthreads();
    if (warp == 0) {
        if (lane < DC_T) {                         // column `lane` of T, from its diagonal down
            float T[DC_T];
#pragma unroll
            for (int t = 0; t < DC_T; ++t) {
                const float beta = rows[t * DC_ROW + 3 * DC_D + 1];
                float s = 0.0f;
#pragma unroll
                for (int i = 0; i < t; ++i)
                    if (i >= lane) s = fmaf(A[t][i], T[i], s);
                T[t] = t < lane ? 0.0f : t == lane ? beta : -beta * s;
                rec[DC_TM + t * DC_PITCH + lane] = T[t];
            }
        }
    } else if (warp >= 4 && warp < 8) {            // a thread a channel
        const int c = threadIdx.x - 4 * 32;
        float P = 1.0f;
#pragma unroll
        for (int t = 0; t < DC_T; ++t) {
            const float* r = rows + t * DC_ROW + c;
            P *= r[2 * DC_D];
            rec[DC_KT + t * DC_D + c] = P * r[DC_D];
            rec[DC_QT + t * DC_D + c] = P * r[0];
        }
        rec[DC_P + c] = P;
        float R = 1.0f;
#pragma unroll
        for (int t = DC_T - 1; t >= 0; --t) {
            const float* r = rows + t * DC_ROW + c;
            rec[DC_KB + t * DC_D + c] = R * r[DC_D];
            R *= r[2 * DC_D];
        }
    }
}

#define DC_COLS 16                                              // columns of S a block: four a warp
#define DC_BUF (DC_REC + DC_T * DC_COLS)                        // floats of a staged chunk: the record, the values
#define DC_WORK (DC_T * 4 * 4)                                  // floats a warp: v - S^T P k, u, u twice over
#define DC_SMEM ((2 * DC_BUF + 4 * DC_WORK) * (int)sizeof(float))

// 32 pairs of sums over the lanes: lane l gets pair l.
__device__ __forceinline__ f32x2 dc_reduce(f32x2 (&v)[32]) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const f32x2 give = up ? v[i] : v[i + o], keep = up ? v[i + o] : v[i];
            v[i] = add2(keep, __shfl_xor_sync(0xffffffffu, give, o));
        }
    }
    return v[0];
}

__global__ void __launch_bounds__(DR_THREADS)
delta_chunk_kernel(const float* __restrict__ x, int C, int v_col, const float* __restrict__ prep, float* __restrict__ state,
                   size_t slot_stride, const int* __restrict__ cu_q, const int* __restrict__ seq_slot, float* __restrict__ y, int H,
                   int d, int dv, int vec) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    const int b = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int t_begin = cu_q[b], t_end = cu_q[b + 1];
    if (t_end <= t_begin) return;
    const float* rec0 = prep + dc_place(t_begin, b) * H;
    float* S_head = state + (size_t)seq_slot[b] * slot_stride + (size_t)h * dv * d;
    if (t_end - t_begin < DC_MIN) {
        dr_walk<8, true, DR_THREADS>(sm, x, C, v_col, rec0 + (size_t)h * DC_ROW, (size_t)H * DC_ROW, t_begin, t_end, blockIdx.z, S_head, y, H, d, dv, vec);
        return;
    }
    const int j0 = blockIdx.z * DC_COLS + 4 * warp, c0 = 4 * lane;
    float* xs = sm + 2 * DC_BUF + warp * DC_WORK;               // [16][4]
    float* us = xs + 4 * DC_T;                                  // [16][4]
    float* uu = us + 4 * DC_T;                                  // [16][4][2]
    f32x2 S[4][2];                                              // column j0 + j, channels c0 + 2 p and + 1
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float* p = S_head + (size_t)(j0 + j) * d + c0;
        const bool live = j0 + j < dv;
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (vec) {
            if (live && c0 < d) *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(p);
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (live && c0 + c < d) v[c] = p[c];
        }
        S[j][0] = pair2(v[0], v[1]);
        S[j][1] = pair2(v[2], v[3]);
    }
    auto issue = [&](int t0, int chunk, int buf) {
        float* to = sm + buf * DC_BUF;
        const float* from = rec0 + ((size_t)chunk * H + h) * DC_REC;
        for (int i = tid; i < DC_REC / 4; i += DR_THREADS) dr_cp16(to + 4 * i, from + 4 * i);
#pragma unroll
        for (int i = tid; i < DC_T * DC_COLS; i += DR_THREADS) {
            const int t = t0 + i / DC_COLS, j = blockIdx.z * DC_COLS + i % DC_COLS;
            if (t < t_end && j < dv) dr_cp4(to + DC_REC + i, x + (size_t)t * C + v_col + h * dv + j);
            else to[DC_REC + i] = 0.0f;
        }
        dr_commit();
    };
    // rows of scaled vectors against S: lane l gets the sums of token l / 2, columns j0 + 2 (l % 2) and + 1
    auto times_S = [&](const float* vecs) {
        f32x2 v[32];
#pragma unroll
        for (int t = 0; t < DC_T; ++t) {
            const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(vecs + t * DC_D + c0);
            float w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float2 r = unpair2(fma2(k.y, S[j][1], mul2(k.x, S[j][0])));
                w[j] = r.x + r.y;
            }
            v[2 * t] = pair2(w[0], w[1]);
            v[2 * t + 1] = pair2(w[2], w[3]);
        }
        return dc_reduce(v);
    };
    issue(t_begin, 0, 0);
    const int tt = lane >> 1, jp = 2 * (lane & 1);
    for (int t0 = t_begin, it = 0; t0 < t_end; t0 += DC_T, ++it) {
        const int nt = min(DC_T, t_end - t0);
        if (t0 + DC_T < t_end) {
            issue(t0 + DC_T, it + 1, (it + 1) & 1);             // under way while this chunk is worked on
            dr_wait<1>();
        } else {
            dr_wait<0>();
        }
        __syncthreads();
        const float* rec = sm + (it & 1) * DC_BUF;
        // sum_{i <= tt} M[tt][i] z[i], from a start, in two chains
        auto lower = [&](const float* M, const float* z, f32x2 s) {
            float m[DC_T];
#pragma unroll
            for (int i = 0; i < DC_T; i += 4)
                *reinterpret_cast<float4*>(m + i) = *reinterpret_cast<const float4*>(M + tt * DC_PITCH + i);
            f32x2 s2 = 0ull;
#pragma unroll
            for (int i = 0; i < DC_T; i += 2) {
                const f32x2 z0 = *reinterpret_cast<const f32x2*>(z + i * 4 + jp), z1 = *reinterpret_cast<const f32x2*>(z + i * 4 + 4 + jp);
                if (i <= tt) s = fma2(pair2(m[i], m[i]), z0, s);
                if (i + 1 <= tt) s2 = fma2(pair2(m[i + 1], m[i + 1]), z1, s2);
            }
            return add2(s, s2);
        };
        const float2 R = unpair2(times_S(rec + DC_KT));
        const float2 v = *reinterpret_cast<const float2*>(rec + DC_REC + tt * DC_COLS + 4 * warp + jp);
        *reinterpret_cast<float2*>(xs + tt * 4 + jp) = make_float2(v.x - R.x, v.y - R.y);
        const f32x2 Q = times_S(rec + DC_QT);
        __syncwarp();
        const float2 u = unpair2(lower(rec + DC_TM, xs, 0ull));
        *reinterpret_cast<float2*>(us + tt * 4 + jp) = u;
        *reinterpret_cast<float4*>(uu + tt * 8 + 2 * jp) = make_float4(u.x, u.x, u.y, u.y);
        __syncwarp();
        const float2 o = unpair2(lower(rec + DC_BM, us, Q));
        if (tt < nt) {
            float* dst = y + (size_t)(t0 + tt) * H * dv + (size_t)h * dv + j0 + jp;
            if ((dv & 1) == 0) {
                if (j0 + jp < dv) *reinterpret_cast<float2*>(dst) = o;
            } else {
                if (j0 + jp < dv) dst[0] = o.x;
                if (j0 + jp + 1 < dv) dst[1] = o.y;
            }
        }
        const ulonglong2 P = *reinterpret_cast<const ulonglong2*>(rec + DC_P + c0);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            S[j][0] = mul2(P.x, S[j][0]);
            S[j][1] = mul2(P.y, S[j][1]);
        }
        auto add = [&](int t) {
            const ulonglong2 k = *reinterpret_cast<const ulonglong2*>(rec + DC_KB + t * DC_D + c0);
            const ulonglong2 u01 = *reinterpret_cast<const ulonglong2*>(uu + t * 8), u23 = *reinterpret_cast<const ulonglong2*>(uu + t * 8 + 4);
            S[0][0] = fma2(k.x, u01.x, S[0][0]);
            S[0][1] = fma2(k.y, u01.x, S[0][1]);
            S[1][0] = fma2(k.x, u01.y, S[1][0]);
            S[1][1] = fma2(k.y, u01.y, S[1][1]);
            S[2][0] = fma2(k.x, u23.x, S[2][0]);
            S[2][1] = fma2(k.y, u23.x, S[2][1]);
            S[3][0] = fma2(k.x, u23.y, S[3][0]);
            S[3][1] = fma2(k.y, u23.y, S[3][1]);
        };
        if (nt == DC_T) {
#pragma unroll
            for (int t = 0; t < DC_T; ++t) add(t);
        } else {
            for (int t = 0; t < nt; ++t) add(t);
        }
        __syncthreads();                            // this chunk has been read by everyone before its buffer is filled again
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (j0 + j >= dv) continue;
        float* p = S_head + (size_t)(j0 + j) * d + c0;
        const float2 lo = unpair2(S[j][0]), hi = unpair2(S[j][1]);
        const float v[4] = {lo.x, lo.y, hi.x, hi.y};
        if (vec) {
            if (c0 < d) *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (c0 + c < d) p[c] = v[c];
        }
    }
}

// Threads a column for d key channels.
static inline int delta_rule_threads(int d) {
    int NS = 1;
    while (NS * DR_ROWS < d) NS <<= 1;
    return NS;
}

// Steps in which a sequence may go in chunks: heads of 65 to 128, and tokens for one long enough. Whether it does is its own
// number of tokens alone: not how many sequences there are beside it, empty ones among them.
static inline bool delta_rule_chunks(int d, int longest) { return d > DC_D / 2 && d <= DC_D && longest >= DC_MIN; }

// Floats of scratch lumen_delta_rule needs for a step of N tokens in n_seqs sequences, H heads of d key channels.
LUMEN_API long long lumen_delta_rule_scratch(int N, int n_seqs, int longest, int H, int d) {
    if (delta_rule_chunks(d, longest)) return (long long)dc_place(N, n_seqs) * H;
    return (long long)N * H * (3 * delta_rule_threads(d) * DR_ROWS + 4);
}

// x float32 [N, C]: the convolved and activated q (G heads of d, from column q_col), k (k_col)
// and v (H heads of dv, v_col). u: the projection's partial sums [uS, N, uW] with the H beta
// logits from column b_col. a: partial sums [aS, N, H d] of the decay logits (before dt_bias).
// state float32, row seq_slot[b] of stride slot_stride holds [H, dv, d]. y float32 [N, H dv]. prep:
// lumen_delta_rule_scratch(N, n_seqs, longest, H, d) floats of scratch. cu_q covers at most N tokens. longest: no sequence has
// more tokens (N where that is not known); it decides what is launched, not how a sequence is summed.
LUMEN_API int lumen_delta_rule(const float* x, int C, int q_col, int k_col, int v_col, const float* u, int uS,
                               long long u_stride, int uW, int b_col, const float* a, int aS, long long a_stride,
                               const float* dt_bias, const float* a_log, float* state, long long slot_stride,
                               const int* cu_q, const int* seq_slot, int n_seqs, int longest, float* y, float* prep, int N, int H,
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
    const DrIn in = {x, u, a, dt_bias, a_log, (size_t)u_stride, (size_t)a_stride, C, q_col, k_col, uS, uW, b_col, aS, H, G, d};
    if (delta_rule_chunks(d, longest)) {
        if ((dv + DC_COLS - 1) / DC_COLS > 65535) return LUMEN_ERR_UNSUPPORTED;
        cudaError_t e = cudaFuncSetAttribute(delta_chunk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DC_SMEM);
        if (e != cudaSuccess) return (int)e;
        lumen_launch(delta_chunk_prepare_kernel, dim3(N / DC_T + n_seqs, H), dim3(32 * DC_WARPS), 0, stream, in, prep, cu_q, n_seqs);
        LUMEN_LAUNCH_CHECK();
        lumen_launch(delta_chunk_kernel, dim3(n_seqs, H, (dv + DC_COLS - 1) / DC_COLS), dim3(DR_THREADS), DC_SMEM, stream, x, C, v_col,
                     (const float*)prep, state, (size_t)slot_stride, cu_q, seq_slot, y, H, d, dv, vec);
        LUMEN_LAUNCH_CHECK();
        return 0;
    }
    dim3 pgrid(N, (H + DR_PREP_WARPS - 1) / DR_PREP_WARPS);
    if (pgrid.y > 65535) return LUMEN_ERR_UNSUPPORTED;
    lumen_launch(delta_prepare_kernel, pgrid, dim3(32 * DR_PREP_WARPS), 0, stream, in, prep, dp);
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
