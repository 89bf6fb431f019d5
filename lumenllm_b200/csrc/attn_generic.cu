// General causal attention over the paged cache, for any number of new tokens
// per sequence (whole prompts and single decoded tokens alike), any key size and
// any value size up to 512 (the two may differ), any number of heads and groups,
// with an optional window. All arithmetic is float32 with the precise expf. It is the
// attention of the 32-bit path and the plain device reference of the faster
// bfloat16 kernels.
//
// Options, each a parameter: `chunk` > 0 limits a query's sight to the keys of its own run of
// `chunk` positions counted from the sequence's start; `softcap` > 0 replaces a score s by
// softcap * tanh(s / softcap); `sink` adds exp(sink[head]) to the softmax's denominator (a key of
// that score that has no value); `v_in_k` takes a key's value from the first dv numbers of the key's own
// row (a latent cache, where keys and values are one vector); `gate` multiplies the output by
// sigmoid of some columns of a projection that arrives as partial sums, one number a value or one
// a head; `keep_first` first keys of a sequence stay in sight of every later query whatever the window
// and the chunk say; value tiles may be wider (v_width) than the dv numbers that are used. Queries and
// outputs may be float32 over a bfloat16 cache (TQ).
//
// One block per (query token, HB query heads of one group): a key's and a value's numbers are read once
// for all of them, and 16 bytes at a time where the rows allow it. What bounds it is how many lines of the
// first-level cache the keys' reads touch (a thread has a key, so a warp's read lies in 32 rows). 300 tokens of 16
// heads of 128 over 4 key heads, float32: 552 -> 107 us; one token after 1,000 keys: 338 -> 89.
// Keys are walked in chunks of 128
// whose boundaries are multiples of 128 in absolute position, so the order of
// every sum depends only on the query's own position: the result for a token
// is the same bit for bit whether it came in a prompt, alone, or in any batch.
#include "common.cuh"

#define AG_THREADS 128
#define AG_ACC 4
#define AG_MAX_D (AG_ACC * AG_THREADS)   // widest value
#define AG_MAX_Q 1024       // widest key (a latent cache's keys are the latent and the rotated part)

struct AttnOptions {
    int chunk;            // 0: none
    float softcap;        // 0: none
    const float* sink;    // [nq]: the denominator of head h has one more term exp(sink[h]); null: none
    int v_in_k;           // 1: values are the first dv numbers of the key rows
    const float* gate;    // partial sums [gS][N][g_width]; columns g_col0 + head * dv + e
    int gS;
    long long g_split_stride;
    int g_width, g_col0;  // g_head 1: column g_col0 + head for all of a head's values
    int g_head;
    int keep_first;
    int v_width;          // numbers a value row of the cache has (0: dv)
};

// Sums and maxima over the block of NV values a thread, each in block_sum's and block_max's order. red: 32 NV floats.
template <int NV, bool MAX>
__device__ __forceinline__ void ag_block_reduce(float (&v)[NV], float (*red)[32]) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int h = 0; h < NV; ++h) v[h] = MAX ? warp_max(v[h]) : warp_sum(v[h]);
    __syncthreads();
    if (lane == 0) {
#pragma unroll
        for (int h = 0; h < NV; ++h) red[h][warp] = v[h];
    }
    __syncthreads();
#pragma unroll
    for (int h = 0; h < NV; ++h) {
        const float t = (lane < AG_THREADS / 32) ? red[h][lane] : (MAX ? -INFINITY : 0.0f);
        v[h] = MAX ? warp_max(t) : warp_sum(t);
    }
}

// VEC: rows of keys are read 16 bytes at a time (float32 plain tiles with d a multiple of 4, or swizzled tiles).
// The products of a dot are added in the order of the key's numbers either way.
// WIDE: four of a value row's numbers are read at a time instead of one and then the next for the whole page, so that more
// of it is under way: float32 values beyond 384, where few blocks wait for memory (us, as the others / this: one token after
// 1,000 keys, 16 sequences of 4 heads over one key head of 576 with values of 512: 981 / 651, of 4 heads of 512 1,126 / 774;
// 300 tokens of 16 heads 440 / 284; 100 tokens of 8 heads of 384 after 1,000 562 / 672). The same sums. bfloat16 values gain
// nothing by it.
template <typename T, typename TQ, int HB, bool VEC, bool WIDE>
__global__ void __launch_bounds__(AG_THREADS)
attn_generic_kernel(const TQ* __restrict__ q, const T* __restrict__ kcache, const T* __restrict__ vcache,
                    const int* __restrict__ block_table, int bt_stride,
                    const int* __restrict__ tok_seq, const int* __restrict__ tok_pos,
                    TQ* __restrict__ out, int nq, int nkv, int d, int dv, int window, float scale,
                    int layout, int v_layout, AttnOptions opt) {
    pdl_wait();      // nothing of this kernel touches global memory before this
    pdl_trigger();
    __shared__ __align__(16) float qs[HB][AG_MAX_Q];
    __shared__ float ps[HB][AG_THREADS];
    __shared__ float red[HB][32];
    const int head0 = blockIdx.y * HB, n = blockIdx.x, tid = threadIdx.x;
    const int kvh = head0 / (nq / nkv);
    const int p = tok_pos[n];
    const int* bt = block_table + (size_t)tok_seq[n] * bt_stride;
#pragma unroll
    for (int h = 0; h < HB; ++h) {
        const TQ* qrow = q + ((size_t)n * nq + head0 + h) * d;
        for (int e = tid; e < d; e += AG_THREADS) qs[h][e] = to_f32(qrow[e]);
    }
    __syncthreads();

    int lo = 0;
    if (window > 0 && p - window + 1 > 0) lo = p - window + 1;
    if (opt.chunk > 0) lo = max(lo, (p / opt.chunk) * opt.chunk);
    // with a sink the head starts as if a key of that score had been seen
    float m[HB], l[HB];
#pragma unroll
    for (int h = 0; h < HB; ++h) {
        m[h] = opt.sink ? opt.sink[head0 + h] : -INFINITY;
        l[h] = opt.sink ? 1.0f : 0.0f;
    }
    const int v_row = opt.v_in_k ? d : opt.v_width;        // numbers a value row lies apart from the next
    const int keep = min(opt.keep_first, lo);             // kept keys before the window: [0, keep)
    float acc[HB][AG_ACC];               // dims tid, tid + 128, ...
#pragma unroll
    for (int h = 0; h < HB; ++h)
#pragma unroll
        for (int i = 0; i < AG_ACC; ++i) acc[h][i] = 0.0f;

    const int kept_chunks = min((keep + AG_THREADS - 1) / AG_THREADS, lo / AG_THREADS);
    for (int it = 0; it <= kept_chunks + p / AG_THREADS - lo / AG_THREADS; ++it) {
        const int c = it < kept_chunks ? it : lo / AG_THREADS + it - kept_chunks;
        const int j = c * AG_THREADS + tid;
        const bool valid = (j >= lo || j < keep) && (j <= p);
        float s[HB], cm[HB];
#pragma unroll
        for (int h = 0; h < HB; ++h) s[h] = -INFINITY;
        if (valid) {
            const int page = bt[j / LUMEN_PAGE];
            const T* ktile = kcache + ((size_t)page * nkv + kvh) * LUMEN_PAGE * d;
            const int r = j % LUMEN_PAGE;
            float dot[HB];
#pragma unroll
            for (int h = 0; h < HB; ++h) dot[h] = 0.0f;
            if (VEC) {
                constexpr int W = 16 / (int)sizeof(T);
#pragma unroll 4
                for (int e = 0; e < d; e += W) {
                    const uint4 raw = *reinterpret_cast<const uint4*>(ktile + tile_offset(layout, r, e, d));
                    const T* kv = reinterpret_cast<const T*>(&raw);
#pragma unroll
                    for (int h = 0; h < HB; ++h) {
                        float qv[W];
#pragma unroll
                        for (int x = 0; x < W; x += 4) *reinterpret_cast<float4*>(qv + x) = *reinterpret_cast<const float4*>(&qs[h][e + x]);
#pragma unroll
                        for (int x = 0; x < W; ++x) dot[h] = fmaf(qv[x], to_f32(kv[x]), dot[h]);
                    }
                }
            } else {
                for (int e = 0; e < d; ++e) {
                    const float kv = to_f32(ktile[tile_offset(layout, r, e, d)]);
#pragma unroll
                    for (int h = 0; h < HB; ++h) dot[h] = fmaf(qs[h][e], kv, dot[h]);
                }
            }
#pragma unroll
            for (int h = 0; h < HB; ++h) {
                s[h] = dot[h] * scale;
                if (opt.softcap > 0.0f) s[h] = opt.softcap * tanhf(s[h] / opt.softcap);
            }
        }
#pragma unroll
        for (int h = 0; h < HB; ++h) cm[h] = s[h];
        ag_block_reduce<HB, true>(cm, red);
        float pj[HB], corr[HB];
        __syncthreads();
#pragma unroll
        for (int h = 0; h < HB; ++h) {
            const float m_new = fmaxf(m[h], cm[h]);
            pj[h] = valid ? expf(s[h] - m_new) : 0.0f;
            corr[h] = (m[h] == -INFINITY) ? 0.0f : expf(m[h] - m_new);
            ps[h][tid] = pj[h];
#pragma unroll
            for (int i = 0; i < AG_ACC; ++i) acc[h][i] *= corr[h];
            m[h] = m_new;
        }
        ag_block_reduce<HB, false>(pj, red);         // has a __syncthreads before ps is read below
#pragma unroll
        for (int h = 0; h < HB; ++h) l[h] = l[h] * corr[h] + pj[h];
        const int jbeg = c * AG_THREADS, jend = min(c * AG_THREADS + AG_THREADS - 1, p);
        // the kept keys of the chunk, then those of the window
        for (int part = 0; part < 2; ++part) {
            const int last = part == 0 ? min(jend, keep - 1) : jend;
            for (int j0 = part == 0 ? jbeg : max(jbeg, lo); j0 <= last;) {
                const int r0 = j0 % LUMEN_PAGE, nr = min(LUMEN_PAGE - r0, last - j0 + 1);      // a run within a page
                const T* vtile = vcache + ((size_t)bt[j0 / LUMEN_PAGE] * nkv + kvh) * LUMEN_PAGE * v_row;
                const float* w = &ps[0][j0 - jbeg];
                if (WIDE) {
#pragma unroll 4
                    for (int k = 0; k < nr; ++k) {
                        float v[AG_ACC];
#pragma unroll
                        for (int i = 0; i < AG_ACC; ++i) {
                            const int e = tid + i * AG_THREADS;
                            v[i] = e < dv ? to_f32(vtile[tile_offset(v_layout, r0 + k, e, v_row)]) : 0.0f;
                        }
#pragma unroll
                        for (int i = 0; i < AG_ACC; ++i)
#pragma unroll
                            for (int h = 0; h < HB; ++h) acc[h][i] = fmaf(w[h * AG_THREADS + k], v[i], acc[h][i]);
                    }
                } else
#pragma unroll
                for (int i = 0; i < AG_ACC; ++i) {
                    const int e = tid + i * AG_THREADS;
                    if (e >= dv) break;
#pragma unroll 8
                    for (int k = 0; k < nr; ++k) {
                        const float v = to_f32(vtile[tile_offset(v_layout, r0 + k, e, v_row)]);
#pragma unroll
                        for (int h = 0; h < HB; ++h) acc[h][i] = fmaf(w[h * AG_THREADS + k], v, acc[h][i]);
                    }
                }
                j0 += nr;
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int h = 0; h < HB; ++h) {
        const int head = head0 + h;
        TQ* orow = out + ((size_t)n * nq + head) * dv;
        const float inv = 1.0f / l[h];
#pragma unroll
        for (int i = 0; i < AG_ACC; ++i) {
            const int e = tid + i * AG_THREADS;
            if (e >= dv) break;
            float o = acc[h][i] * inv;
            if (opt.gate) {
                const float* g = opt.gate + (size_t)n * opt.g_width + opt.g_col0 + (opt.g_head ? head : head * dv + e);
                float z = g[0];
                for (int sp = 1; sp < opt.gS; ++sp) z += g[(size_t)sp * opt.g_split_stride];
                o *= 1.0f / (1.0f + expf(-z));
            }
            orow[e] = from_f32<TQ>(o);
        }
    }
}

// Float32 prompts without options, heads of up to 128: the kernel above with AP_Q neighbouring tokens a block, so that the keys and
// values are fetched once for all of them (a token each read them again). A chunk's keys are staged in shared memory; products of two
// rows share an instruction, each rounded as by itself, and every sum runs in the order of the kernel above: the same bits. Tokens of
// different sequences in a block are walked one sequence after the other. A key past a row's own token is not multiplied into it.
// What bounds it is shared memory (a 16-byte read of a warp takes four cycles however many lanes share it): a thread makes the dots
// of two keys and adds up two value numbers, for half of the rows, so that a read of queries or of weights serves twice. Then the
// time of the longest block, a chunk after the other: so a page is looked up once a chunk, and values are fetched sixteen keys ahead.
// 300 tokens of 16 heads of 128 over 4 key heads, inside the step: 122 us a layer with a token a block, 46 so (63 with one key and one
// value number a thread, 56 with a predicate a key and long blocks beside long ones).
#define AP_Q 4
typedef unsigned long long ap_f2;
__device__ __forceinline__ ap_f2 ap_pair(float lo, float hi) {
    ap_f2 d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ float2 ap_unpair(ap_f2 a) {
    float2 v;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(a));
    return v;
}
__device__ __forceinline__ void ap_fma(ap_f2& c, ap_f2 a, ap_f2 b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b)); }
__device__ __forceinline__ void ap_mul(ap_f2& c, ap_f2 a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(c) : "l"(a)); }
__host__ __device__ constexpr int ap_smem(int HB, int d) {           // floats: keys, queries, weights
    return AG_THREADS * (d + 4) + (d + AG_THREADS) * (HB * AP_Q + 4);
}

template <int HB>
__global__ void __launch_bounds__(AG_THREADS)
attn_prompt_f32_kernel(const float* __restrict__ q, const float* __restrict__ kcache, const float* __restrict__ vcache,
                       const int* __restrict__ block_table, int bt_stride, const int* __restrict__ tok_seq,
                       const int* __restrict__ tok_pos, float* __restrict__ out, int N, int nq, int nkv, int d, int dv, float scale, int q_vec) {
    pdl_wait();      // nothing of this kernel touches global memory before this
    pdl_trigger();
    constexpr int R = HB * AP_Q, RP = R + 4;         // rows (token t, head h: t HB + h); floats a key's weights lie apart
    extern __shared__ __align__(16) float sm[];
    float* ks = sm;                                  // [128][d + 4]
    float* qs = ks + AG_THREADS * (d + 4);           // [d][RP]
    float* ps = qs + d * RP;                         // [128][RP]
    __shared__ float red[R][32];
    const int tid = threadIdx.x, head0 = blockIdx.y * HB, kvh = head0 / (nq / nkv);
    const int kp = tid & 63, half = tid >> 6;        // of a warp the same
    // the upper half of the heads from the last tokens on, so that blocks that see many keys and few share an SM
    const int n0 = (int)(2 * blockIdx.y < gridDim.y ? blockIdx.x : gridDim.x - 1 - blockIdx.x) * AP_Q, nt = min(AP_Q, N - n0);
    // pairs of rows of this half, side by side
    auto rows2 = [&](const float* p, ap_f2 (&x)[R / 4]) {
        if constexpr (R >= 8) {
#pragma unroll
            for (int r = 0; r < R / 8; ++r) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p + half * (R / 2) + 4 * r);
                x[2 * r] = v.x;
                x[2 * r + 1] = v.y;
            }
        } else {
            x[0] = *reinterpret_cast<const ap_f2*>(p + half * (R / 2));
        }
    };
    const int warp = tid >> 5, e4 = 4 * (tid & 31);  // a warp a row, a lane 16 bytes of it
#pragma unroll
    for (int i = 0; i < R / 4; ++i) {
        const int r = 4 * i + warp, t = r / HB;
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (e4 < d && t < nt) {
            const float* p = q + ((size_t)(n0 + t) * nq + head0 + r % HB) * d + e4;
            if (q_vec) x = *reinterpret_cast<const float4*>(p);
            else x = make_float4(p[0], p[1], p[2], p[3]);
        }
        if (e4 < d) {
            qs[e4 * RP + r] = x.x;
            qs[(e4 + 1) * RP + r] = x.y;
            qs[(e4 + 2) * RP + r] = x.z;
            qs[(e4 + 3) * RP + r] = x.w;
        }
    }
    for (int g0 = 0, g1; g0 < nt; g0 = g1) {
        const int seq = tok_seq[n0 + g0];
        for (g1 = g0 + 1; g1 < nt && tok_seq[n0 + g1] == seq; ++g1) {}
        const int* bt = block_table + (size_t)seq * bt_stride;
        int pos[AP_Q], p_max = -1, p_min = 0x7fffffff;
#pragma unroll
        for (int t = 0; t < AP_Q; ++t) {
            pos[t] = (t >= g0 && t < g1) ? tok_pos[n0 + t] : -1;       // -1: no row of this walk
            if (pos[t] >= 0) {
                p_max = max(p_max, pos[t]);
                p_min = min(p_min, pos[t]);
            }
        }
        float m[R], l[R];
        ap_f2 acc[2][R / 4];                         // value numbers kp and kp + 64, this half's rows
#pragma unroll
        for (int r = 0; r < R; ++r) {
            m[r] = -INFINITY;
            l[r] = 0.0f;
            acc[r & 1][r / 4] = 0ull;
        }
        for (int c = 0; c <= p_max / AG_THREADS; ++c) {
            const int j = c * AG_THREADS + tid, jend = min(c * AG_THREADS + AG_THREADS - 1, p_max);
            __syncthreads();                         // the keys and weights of the chunk before have been read
            const int jc = c * AG_THREADS;           // a chunk is two pages, or less
            const size_t page[2] = {((size_t)bt[jc / LUMEN_PAGE] * nkv + kvh) * LUMEN_PAGE,
                                    jc + LUMEN_PAGE <= jend ? ((size_t)bt[jc / LUMEN_PAGE + 1] * nkv + kvh) * LUMEN_PAGE : 0};
            static_assert(AG_THREADS == 2 * LUMEN_PAGE, "");
            if (e4 < d) {
                for (int r = warp; r <= jend - jc; r += 4)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                     (uint32_t)__cvta_generic_to_shared(ks + r * (d + 4) + e4)),
                                 "l"(kcache + ((r < LUMEN_PAGE ? page[0] : page[1]) + r % LUMEN_PAGE) * d + e4)
                                 : "memory");
            }
            asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            float s[R], cm[R];
            {
                ap_f2 dot[2][R / 4];
#pragma unroll
                for (int r = 0; r < R / 4; ++r) dot[0][r] = dot[1][r] = 0ull;
#pragma unroll 2
                for (int e = 0; e < d; e += 4) {
                    float k[2][4];
                    *reinterpret_cast<float4*>(k[0]) = *reinterpret_cast<const float4*>(ks + kp * (d + 4) + e);
                    *reinterpret_cast<float4*>(k[1]) = *reinterpret_cast<const float4*>(ks + (kp + 64) * (d + 4) + e);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        ap_f2 qq[R / 4];
                        rows2(qs + (e + x) * RP, qq);
                        const ap_f2 k0 = ap_pair(k[0][x], k[0][x]), k1 = ap_pair(k[1][x], k[1][x]);
#pragma unroll
                        for (int r = 0; r < R / 4; ++r) {
                            ap_fma(dot[0][r], qq[r], k0);
                            ap_fma(dot[1][r], qq[r], k1);
                        }
                    }
                }
                // from here on a thread has the key tid, for all rows
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int r = 0; r < R / 4; ++r)
                        *reinterpret_cast<ap_f2*>(ps + (kp + 64 * x) * RP + half * (R / 2) + 2 * r) = dot[x][r];
                __syncthreads();
#pragma unroll
                for (int r = 0; r < R; r += 4) *reinterpret_cast<float4*>(s + r) = *reinterpret_cast<const float4*>(ps + tid * RP + r);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    s[r] = j <= pos[r / HB] ? __fmul_rn(s[r], scale) : -INFINITY;
                    cm[r] = s[r];
                }
            }
            ag_block_reduce<R, true>(cm, red);
            __syncthreads();
            float corr[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float m_new = fmaxf(m[r], cm[r]);
                s[r] = j <= pos[r / HB] ? expf(s[r] - m_new) : 0.0f;
                corr[r] = (m[r] == -INFINITY) ? 0.0f : expf(m[r] - m_new);
                m[r] = m_new;
            }
#pragma unroll
            for (int r = 0; r < R; r += 4) *reinterpret_cast<float4*>(ps + tid * RP + r) = make_float4(s[r], s[r + 1], s[r + 2], s[r + 3]);
#pragma unroll
            for (int r = 0; r < R / 4; ++r) {
                const ap_f2 c2 = half ? ap_pair(corr[R / 2 + 2 * r], corr[R / 2 + 2 * r + 1]) : ap_pair(corr[2 * r], corr[2 * r + 1]);
                ap_mul(acc[0][r], c2);
                ap_mul(acc[1][r], c2);
            }
            ag_block_reduce<R, false>(s, red);       // has a __syncthreads before ps is read below
#pragma unroll
            for (int r = 0; r < R; ++r) l[r] = l[r] * corr[r] + s[r];
            const bool two = kp + 64 < dv;
            if (kp < dv) {
                const int all = min(jend, p_min) - jc + 1;       // keys of the chunk in sight of every row
                constexpr int AHEAD = 16;
                float x0[AHEAD], x1[AHEAD];
                static_assert(LUMEN_PAGE % AHEAD == 0, "");
                auto fetch = [&](int k0) {               // keys k0 to k0 + 15 of the chunk, of one page
                    const float* v = vcache + ((k0 < LUMEN_PAGE ? page[0] : page[1]) + k0 % LUMEN_PAGE) * dv + kp;
#pragma unroll
                    for (int i = 0; i < AHEAD; ++i) {
                        x0[i] = k0 + i < all ? v[(size_t)i * dv] : 0.0f;
                        x1[i] = k0 + i < all && two ? v[(size_t)i * dv + 64] : 0.0f;
                    }
                };
                auto add = [&](int k, float a, float b) {
                    const ap_f2 v0 = ap_pair(a, a), v1 = ap_pair(b, b);
                    ap_f2 ww[R / 4];
                    rows2(ps + k * RP, ww);
#pragma unroll
                    for (int r = 0; r < R / 4; ++r) {
                        ap_fma(acc[0][r], ww[r], v0);
                        ap_fma(acc[1][r], ww[r], v1);
                    }
                };
                fetch(0);
                for (int k0 = 0; k0 < all; k0 += AHEAD) {
                    float y0[AHEAD], y1[AHEAD];
#pragma unroll
                    for (int i = 0; i < AHEAD; ++i) {
                        y0[i] = x0[i];
                        y1[i] = x1[i];
                    }
                    fetch(min(k0 + AHEAD, AG_THREADS - AHEAD));      // of the last batch again, if there is none
                    if (k0 + AHEAD <= all) {
#pragma unroll
                        for (int i = 0; i < AHEAD; ++i) add(k0 + i, y0[i], y1[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < AHEAD; ++i)
                            if (k0 + i < all) add(k0 + i, y0[i], y1[i]);
                    }
                }
                int j0 = jc + max(all, 0);
                for (; j0 <= jend; ++j0) {           // the last few, of some rows only
                    const float* v = vcache + ((j0 - jc < LUMEN_PAGE ? page[0] : page[1]) + j0 % LUMEN_PAGE) * dv + kp;
                    const float x0 = v[0], x1 = two ? v[64] : 0.0f;
                    const float* w = ps + (j0 - c * AG_THREADS) * RP + half * (R / 2);
#pragma unroll
                    for (int r = 0; r < R / 2; ++r) {
                        if (j0 > (half ? pos[(R / 2 + r) / HB] : pos[r / HB])) continue;
                        float2 a = ap_unpair(acc[0][r / 2]), b = ap_unpair(acc[1][r / 2]);
                        float& a0 = (r & 1) ? a.y : a.x;
                        float& b0 = (r & 1) ? b.y : b.x;
                        a0 = fmaf(w[r], x0, a0);
                        b0 = fmaf(w[r], x1, b0);
                        acc[0][r / 2] = ap_pair(a.x, a.y);
                        acc[1][r / 2] = ap_pair(b.x, b.y);
                    }
                }
            }
        }
#pragma unroll
        for (int r = 0; r < R / 2; ++r) {
            const int row = half * (R / 2) + r, t = row / HB;
            if (t < g0 || t >= g1) continue;
            const float2 a = ap_unpair(acc[0][r / 2]), b = ap_unpair(acc[1][r / 2]);
            const float inv = 1.0f / (half ? l[R / 2 + r] : l[r]);
            float* dst = out + ((size_t)(n0 + t) * nq + head0 + row % HB) * dv + kp;
            if (kp < dv) dst[0] = ((r & 1) ? a.y : a.x) * inv;
            if (kp + 64 < dv) dst[64] = ((r & 1) ? b.y : b.x) * inv;
        }
    }
}

// Heads a block of it: more of them share the staged keys, but a block's time grows with its rows, so a step of few tokens takes as few
// as keep the SMs busy (us, 1 / 2 / 4 heads a block, 16 heads of 128 over 4: 8 tokens 6.5 / 7.7 / 10.1, after 3,000 others 156 / 195 / 260;
// 48 tokens, 192 blocks of one head, 8.5 / 9.2 / 11.8; 64 tokens, 256, 11.2 / 9.7 / 12.6; 3 x 48, 576, 17.6 / 11.0 / 12.4; 3 x 64, 768, 19.6 /
// 19.4 / 16.3; 300, 1,200, 59 / 52 / 43. With a token a block 8 tokens take 7.6 and 274, 300 106). The same bits.
static int attn_prompt_heads(int N, int nq, int nkv) {
    const long long blocks = (long long)((N + AP_Q - 1) / AP_Q) * nq;
    const int G = nq / nkv;
    int hb = 1;
    while (hb < 4 && G % (2 * hb) == 0 && blocks / (2 * hb) >= (hb == 1 ? 128 : 148)) hb *= 2;
    return hb;
}
LUMEN_API int lumen_attn_prompt_heads(int N, int nq, int nkv) { return attn_prompt_heads(N, nq, nkv); }

template <int HB>
static int attn_prompt_f32_go(const float* q, const float* kcache, const float* vcache, const int* block_table, int bt_stride,
                              const int* tok_seq, const int* tok_pos, float* out, int N, int nq, int nkv, int d, int dv, float scale,
                              cudaStream_t stream) {
    const int smem = ap_smem(HB, d) * (int)sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(attn_prompt_f32_kernel<HB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    lumen_launch(attn_prompt_f32_kernel<HB>, dim3((N + AP_Q - 1) / AP_Q, nq / HB), dim3(AG_THREADS), smem, stream, q, kcache, vcache,
                 block_table, bt_stride, tok_seq, tok_pos, out, N, nq, nkv, d, dv, scale, ((uintptr_t)q & 15) == 0);
    LUMEN_LAUNCH_CHECK();
    return 0;
}

static int attn_generic_launch(const void* q, int q_is_f32, const void* kcache, const void* vcache,
                               const int* block_table, int bt_stride, const int* tok_seq, const int* tok_pos,
                               void* out, int is_bf16, int N, int nq, int nkv, int d, int dv, int window,
                               float scale, int layout, int v_layout, AttnOptions opt, cudaStream_t stream) {
    if (N <= 0) return 0;
    if (d <= 0 || dv <= 0 || dv > AG_MAX_D || nq <= 0 || nkv <= 0 || nq % nkv != 0 || window < 0 || opt.chunk < 0)
        return LUMEN_ERR_UNSUPPORTED;
    if (d > AG_MAX_Q) return LUMEN_ERR_UNSUPPORTED;
    if (opt.v_in_k && (dv > d || v_layout != layout)) return LUMEN_ERR_BAD_ARGUMENT;
    if (opt.v_width == 0) opt.v_width = dv;
    if (opt.v_width < dv || opt.keep_first < 0) return LUMEN_ERR_BAD_ARGUMENT;
    if (nq > 65535) return LUMEN_ERR_UNSUPPORTED;
    if (layout == LUMEN_LAYOUT_SW128 && (!is_bf16 || d % 64 != 0)) return LUMEN_ERR_UNSUPPORTED;
    if (v_layout == LUMEN_LAYOUT_SW128 && (!is_bf16 || (opt.v_in_k ? d : opt.v_width) % 64 != 0)) return LUMEN_ERR_UNSUPPORTED;
    const int esz = is_bf16 ? 2 : 4;
    const bool vec = ((uintptr_t)kcache & 15) == 0 && (d * esz) % 16 == 0;
    // as many heads a block as the group divides into, while two blocks an SM are left
    const int G = nq / nkv;
    int hb = 1;
    while (vec && hb < 4 && G % (2 * hb) == 0 && (long long)N * nq / (2 * hb) >= 2 * 148) hb *= 2;
#define AG_GO(T, TQ, HB, VEC, WIDE)                                                                                    \
    lumen_launch(attn_generic_kernel<T, TQ, HB, VEC, WIDE>, dim3(N, nq / HB), dim3(AG_THREADS), 0, stream, (const TQ*)q, \
                 (const T*)kcache, (const T*)vcache, block_table, bt_stride, tok_seq, tok_pos, (TQ*)out, nq, nkv, d, dv, \
                 window, scale, layout, v_layout, opt)
#define AG_PICK(T, TQ, WIDE)                                                                                           \
    do {                                                                                                               \
        if (!vec) AG_GO(T, TQ, 1, false, false);                                                                       \
        else if (hb == 1) AG_GO(T, TQ, 1, true, WIDE);                                                                 \
        else if (hb == 2) AG_GO(T, TQ, 2, true, WIDE);                                                                 \
        else AG_GO(T, TQ, 4, true, WIDE);                                                                              \
    } while (0)
    if (is_bf16 && !q_is_f32) AG_PICK(__nv_bfloat16, __nv_bfloat16, false);
    else if (is_bf16) AG_PICK(__nv_bfloat16, float, false);
    else if (dv > 3 * AG_THREADS) AG_PICK(float, float, true);
    else AG_PICK(float, float, false);
#undef AG_PICK
#undef AG_GO
    LUMEN_LAUNCH_CHECK();
    return 0;
}

// n_seqs: how many sequences the tokens come from (a sequence's lie together); it decides between kernels of the same bits.
LUMEN_API int lumen_attn_generic(const void* q, const void* kcache, const void* vcache,
                                 const int* block_table, int bt_stride, const int* tok_seq,
                                 const int* tok_pos, void* out, int is_bf16, int N, int n_seqs, int nq, int nkv,
                                 int d, int dv, int window, float scale, int layout, int v_layout,
                                 cudaStream_t stream) {
    AttnOptions opt = {};
    // several tokens a block where most blocks' tokens are of one sequence
    const bool rows = !is_bf16 && window == 0 && layout == LUMEN_LAYOUT_LINEAR && v_layout == LUMEN_LAYOUT_LINEAR && d % 4 == 0 &&
                      d > 0 && d <= AG_THREADS && dv > 0 && dv <= AG_THREADS && ((uintptr_t)kcache & 15) == 0 && nkv > 0 && nq > 0 &&
                      nq % nkv == 0 && nq <= 65535 && n_seqs > 0 && N / n_seqs >= 2 * AP_Q;
    if (rows) {
#define AP_GO(HB)                                                                                                              \
    return attn_prompt_f32_go<HB>((const float*)q, (const float*)kcache, (const float*)vcache, block_table, bt_stride, tok_seq, \
                                  tok_pos, (float*)out, N, nq, nkv, d, dv, scale, stream)
        const int hb = attn_prompt_heads(N, nq, nkv);
        if (hb == 4) AP_GO(4);
        if (hb == 2) AP_GO(2);
        AP_GO(1);
#undef AP_GO
    }
    return attn_generic_launch(q, 0, kcache, vcache, block_table, bt_stride, tok_seq, tok_pos, out, is_bf16, N, nq,
                               nkv, d, dv, window, scale, layout, v_layout, opt, stream);
}

// The same with the options of AttnOptions; q_is_f32: queries and outputs are float32 whatever
// the cache's type.
LUMEN_API int lumen_attn_generic_opt(const void* q, int q_is_f32, const void* kcache, const void* vcache,
                                     const int* block_table, int bt_stride, const int* tok_seq,
                                     const int* tok_pos, void* out, int is_bf16, int N, int nq, int nkv,
                                     int d, int dv, int window, float scale, int layout, int v_layout,
                                     int chunk, float softcap, const float* sink, int v_in_k, const float* gate, int gS,
                                     long long g_split_stride, int g_width, int g_col0, int g_head, int keep_first,
                                     int v_width, cudaStream_t stream) {
    AttnOptions opt = {chunk, softcap, sink, v_in_k, gate, gS, g_split_stride, g_width, g_col0, g_head, keep_first, v_width};
    if (gate && (gS < 1 || g_col0 < 0 || g_col0 + (g_head ? nq : nq * dv) > g_width)) return LUMEN_ERR_BAD_ARGUMENT;
    return attn_generic_launch(q, q_is_f32, kcache, vcache, block_table, bt_stride, tok_seq, tok_pos, out, is_bf16, N,
                               nq, nkv, d, dv, window, scale, layout, v_layout, opt, stream);
}
