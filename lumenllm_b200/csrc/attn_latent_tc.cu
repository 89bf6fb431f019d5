// Causal flash attention over a latent cache for prompts, on the 5th-generation tensor cores. As in attn_latent.cu
// one row a token, W values wide, is the key of every query head and its first dv values are the value of every head;
// queries come already carried into that space ([N, H, W], bfloat16).
//
// A block takes 128 consecutive rows of the query matrix [N H, W] that belong to one sequence, and a slice of up
// to 256 value columns (the accumulator of 128 x 512 would fill tensor memory and leave no room for scores, so two
// blocks of a 512-wide value both make the scores: 1.5 times the products of one block that could hold them all).
// It walks the keys 32 at a time (tiles start at multiples of 32 in absolute position, so what a row computes depends
// only on its own position):
//   S = Q K^T   tcgen05.mma 128 x 32 x W from shared memory (K-major, 128-byte swizzle), two S buffers in tensor
//               memory, so the next tile's scores are made while this tile's softmax runs;
//   softmax     four warps, a thread a row: scale, mask, running maximum and sum in float32, P over the columns its
//               scores came from as two bfloat16 numbers, the rounded weight and the rest. (The kernel this one stands
//               beside moves its reference with every new maximum, so its largest weight is exactly 1; a reference that
//               lags by up to 2^8 rounds that weight too, and alone gave up to 1.7 times its error on peaked rows.)
//   O += P V    tcgen05.mma 128 x slice x 32, P from tensor memory, V the slice's 64-column blocks of the SAME key tile
//               (N-major). O is rescaled only when a row's maximum has grown by more than 2^8 (P and the row sum use the
//               same reference, so the result is exact).
// Q (144 KB at W = 576) and two key tiles (36 KB each) fill an SM's shared memory, so a tile's blocks are freed as
// early as they can be: those outside the slice once the scores are made, the slice's once O has been added to; each
// part has barriers of its own, and the scores of the tile after next start on the first part. Everything arrives by
// TMA (the cache's plain rows get the swizzle on the way). What bounds it is the tensor pipe's operand traffic: every
// 128 x 32 x 16 product reads 5 KB of shared memory for 16 cycles of arithmetic.
// 2,048 tokens, 16 heads, W = 576, dv = 512, window 1,024: 209 us (mma.sync 446; 201 with one bfloat16 number a weight);
// without the window 259 (625). Against 64 bits 2.7e-6 where mma.sync's rounded weights are 1.4e-3 off.
// Every wait is bounded; when one runs out the block raises the error flag, the other roles give up on theirs, and the
// block leaves once its own copies have landed and the products it has issued are done (waits with a bound of their own).
#include <cuda.h>

#include "common.cuh"
#include "mma_utils.cuh"

#define LT_THREADS 192
#define LT_ROWS 128
#define LT_KEYS 32
#define LT_SLICE 256
#define LT_O_COL 256
#define LT_QBLOCK (LT_ROWS * 128)      // bytes of a 64-column block of Q, of a key tile
#define LT_KBLOCK (LT_KEYS * 128)
#define LT_RESCALE 8.0f
#define LT_MAX_W 576

__device__ __forceinline__ void lt_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void lt_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void lt_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void lt_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void lt_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The A operand in tensor memory: lane = row, two bfloat16 a column.
__device__ __forceinline__ void lt_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void lt_tma_2d(void* dst, const CUtensorMap* map, int c0, int c1, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void lt_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void lt_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ float lt_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// As mbar_wait, but given up as soon as another role of the block has.
__device__ __forceinline__ bool lt_wait(uint64_t* bar, uint32_t parity, const volatile int* abort_flag) {
    for (uint32_t it = 0; it < LUMEN_SPIN_LIMIT; ++it) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if ((it & 63u) == 63u && *abort_flag) return false;
    }
    return false;
}
// A 128-byte-swizzled operand: rows of 128 bytes, groups of 8 rows 1024 bytes apart; lbo: distance between the
// 64-value blocks of an N-major operand.
__device__ __forceinline__ uint64_t lt_desc(uint32_t smem_addr, uint32_t lbo_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// D float32, A and B bfloat16, M = 128; b_mn: B is N-major.
__host__ __device__ constexpr uint32_t lt_idesc(int n, int b_mn) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)b_mn << 16) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(LT_ROWS >> 4) << 24);
}

__global__ void __launch_bounds__(LT_THREADS, 1)
attn_latent_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                      const int* __restrict__ block_table, int bt_stride, const int* __restrict__ cu_q,
                      const int* __restrict__ seq_start, int B, float* __restrict__ out, int H, int W, int dv, int window,
                      float scale_log2, int give_up_at, int* __restrict__ err) {
    pdl_wait();      // nothing of this kernel touches global memory before this
    pdl_trigger();
    // operand tiles must start on 1024-byte boundaries; there is no static shared memory ahead of the dynamic part
    extern __shared__ __align__(1024) unsigned char smem[];
    if (smem_u32(smem) & 1023u) {
        if (threadIdx.x == 0) atomicExch(err, 1);
        return;
    }
    const int wb = W >> 6;                                   // 64-column blocks of a row
    const int v0 = (int)blockIdx.y * (LT_SLICE / 64);        // the slice's blocks
    const int nv = min(LT_SLICE / 64, (dv >> 6) - v0), na = wb - nv;
    unsigned char* sQ = smem;
    unsigned char* sK = sQ + wb * LT_QBLOCK;                 // [2][wb][32][128 bytes]
    uint64_t* bars = reinterpret_cast<uint64_t*>(sK + 2 * wb * LT_KBLOCK);
    uint64_t* q_full = bars;
    uint64_t* a_full = bars + 1;        // [2] the blocks outside the slice have landed
    uint64_t* a_empty = bars + 3;       // [2] the scores that read them are made
    uint64_t* v_full = bars + 5;        // [2] the slice's blocks have landed
    uint64_t* v_empty = bars + 7;       // [2] O has been added to
    uint64_t* s_full = bars + 9;        // [2] S is in tensor memory
    uint64_t* p_ready = bars + 11;      // [2] P is in tensor memory, O corrected
    uint64_t* pv_done = bars + 13;      // [2] that tile's product is in O
    uint64_t* mma_done = bars + 15;     // all products of the block are done
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 16);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

    // which sequence, which tile of its rows; the last tiles of a sequence see the most keys and come first
    int tile = blockIdx.x, b = 0, rows_seq = 0;
    for (; b < B; ++b) {
        rows_seq = (cu_q[b + 1] - cu_q[b]) * H;
        const int nt = (rows_seq + LT_ROWS - 1) / LT_ROWS;
        if (tile < nt) break;
        tile -= nt;
    }
    if (b >= B) return;
    const int row0 = ((rows_seq + LT_ROWS - 1) / LT_ROWS - 1 - tile) * LT_ROWS;      // within the sequence
    const int nrows = min(LT_ROWS, rows_seq - row0);
    const size_t grow0 = (size_t)cu_q[b] * H + row0;
    const int start = seq_start[b];
    const int pos_first = start + row0 / H, pos_last = start + (row0 + nrows - 1) / H;
    const int j_lo = window > 0 ? max(0, pos_first - window + 1) : 0;
    const int kt_lo = j_lo / LT_KEYS, nkt = pos_last / LT_KEYS - kt_lo + 1;
    const int* bt = block_table + (size_t)b * bt_stride;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 16; ++i) mbar_init(&bars[i], (i == 11 || i == 12) ? 4 : 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmQ)) : "memory");
        asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmK)) : "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    lt_fence_before();
    __syncthreads();
    lt_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    int a_issued[2] = {0, 0}, v_issued[2] = {0, 0};          // the producer's copies into each stage

    if (warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(q_full, (uint32_t)(wb * LT_QBLOCK));
            // rows beyond the sequence are another sequence's (or, past the matrix, zeros): computed, never written
            for (int c = 0; c < wb; ++c) lt_tma_2d(sQ + c * LT_QBLOCK, &tmQ, c * 64, (int)grow0, q_full);
            for (int i = 0; i < nkt && !*abort_flag; ++i) {
                const int st = i & 1, ph = ((i >> 1) & 1) ^ 1, kt = kt_lo + i;
                const int row = bt[kt / (LUMEN_PAGE / LT_KEYS)] * LUMEN_PAGE + (kt % (LUMEN_PAGE / LT_KEYS)) * LT_KEYS;
                unsigned char* dst = sK + st * wb * LT_KBLOCK;
                if (na > 0) {
                    if (!lt_wait(&a_empty[st], ph, abort_flag)) { *abort_flag = 1; atomicExch(err, 1); break; }
                    mbar_expect_tx(&a_full[st], (uint32_t)(na * LT_KBLOCK));
                    ++a_issued[st];
                    for (int c = 0; c < wb; ++c)
                        if (c < v0 || c >= v0 + nv) lt_tma_2d(dst + c * LT_KBLOCK, &tmK, c * 64, row, &a_full[st]);
                }
                if (!lt_wait(&v_empty[st], ph, abort_flag)) { *abort_flag = 1; atomicExch(err, 1); break; }
                mbar_expect_tx(&v_full[st], (uint32_t)(nv * LT_KBLOCK));
                ++v_issued[st];
                for (int c = v0; c < v0 + nv; ++c) lt_tma_2d(dst + c * LT_KBLOCK, &tmK, c * 64, row, &v_full[st]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            constexpr uint32_t idesc_s = lt_idesc(LT_KEYS, 0);
            const uint32_t idesc_pv = lt_idesc(nv * 64, 1);
            const uint32_t q0 = smem_u32(sQ);
            bool issued = false;
            auto scores = [&](int i) -> bool {          // S[i & 1] = Q K(i)^T
                const int st = i & 1, ph = (i >> 1) & 1;
                const uint32_t k0 = smem_u32(sK + st * wb * LT_KBLOCK), d = tmem_base + st * LT_KEYS;
                uint32_t acc = 0;
                auto block = [&](int c) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        lt_mma(d, lt_desc(q0 + c * LT_QBLOCK + k * 32, 16), lt_desc(k0 + c * LT_KBLOCK + k * 32, 16), idesc_s, acc);
                        acc = 1;
                    }
                };
                if (na > 0) {
                    if (!lt_wait(&a_full[st], ph, abort_flag)) return false;
                    lt_fence_after();
                    for (int c = 0; c < wb; ++c)
                        if (c < v0 || c >= v0 + nv) block(c);
                    issued = true;
                    lt_commit(&a_empty[st]);
                }
                if (!lt_wait(&v_full[st], ph, abort_flag)) return false;
                lt_fence_after();
                for (int c = v0; c < v0 + nv; ++c) block(c);
                issued = true;
                lt_commit(&s_full[st]);
                return true;
            };
            bool ok = lt_wait(q_full, 0, abort_flag);
            if (ok) {
                lt_fence_after();
                ok = scores(0);
            }
            for (int it = 0; ok && it < nkt && !*abort_flag; ++it) {
                if (it + 1 < nkt && !scores(it + 1)) { ok = false; break; }
                const int st = it & 1;
                if (!lt_wait(&p_ready[st], (it >> 1) & 1, abort_flag)) { ok = false; break; }
                lt_fence_after();
                const uint32_t vt = smem_u32(sK + (st * wb + v0) * LT_KBLOCK);
#pragma unroll
                for (int kk = 0; kk < 2 * (LT_KEYS / 16); ++kk)        // 16 keys a step: 8 columns of P, then the same of its rest
                    lt_mma_ts(tmem_base + LT_O_COL, tmem_base + st * LT_KEYS + kk * 8,
                              lt_desc(vt + (kk & 1) * (16 * 128), LT_KBLOCK), idesc_pv, (it > 0 || kk > 0) ? 1u : 0u);
                lt_commit(&v_empty[st]);
                lt_commit(&pv_done[st]);
            }
            if (!ok) { *abort_flag = 1; atomicExch(err, 1); }
            // The block keeps its shared and tensor memory until the products that use them are done: a commit covers all
            // that this lane has issued, those of a step that was broken off too.
            if (issued) {
                lt_commit(mma_done);
                if (!mbar_wait(mma_done, 0)) atomicExch(err, 1);
            }
        }
    } else {
        const int qd = warp & 3;                           // lanes of tensor memory this warp may read
        const int r = qd * 32 + lane;
        const bool row_ok = r < nrows;
        const int prow = row_ok ? start + (row0 + r) / H : -1;                  // -1: nothing is seen
        const int lorow = window > 0 ? prow - window + 1 : 0;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16);
        const int vcols = nv * 64;
        float m_ref = -INFINITY, l = 0.0f;
        bool ok = true;
        for (int it = 0; it < nkt; ++it) {
            const int st = it & 1;
            if (__any_sync(0xffffffffu, *abort_flag != 0)) { ok = false; break; }
            bool w = it != give_up_at && lt_wait(&s_full[st], (it >> 1) & 1, abort_flag);
            if (!__all_sync(0xffffffffu, w)) { ok = false; break; }
            lt_fence_after();
            float s[32];
            lt_ld32(lane_addr + st * LT_KEYS, s);
            const int jb = (kt_lo + it) * LT_KEYS;
            if (!__all_sync(0xffffffffu, jb + LT_KEYS - 1 <= prow && jb >= lorow)) {      // the diagonal or the window's edge
#pragma unroll
                for (int j = 0; j < 32; ++j) s[j] = (jb + j <= prow && jb + j >= lorow) ? s[j] : -INFINITY;
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};      // the scale is positive
#pragma unroll
            for (int j = 0; j < 32; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], s[j]);
            const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
            float corr = 1.0f;
            if (mx > m_ref + LT_RESCALE || m_ref == -INFINITY) {
                const float nref = fmaxf(mx, m_ref);
                if (nref != -INFINITY) {
                    corr = (m_ref == -INFINITY) ? 0.0f : lt_ex2(m_ref - nref);
                    m_ref = nref;
                }
            }
            const float nbase = (m_ref == -INFINITY) ? 0.0f : -m_ref;
            uint32_t hi[16], lo[16];
            float rs4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const float p0 = lt_ex2(fmaf(s[2 * c], scale_log2, nbase)), p1 = lt_ex2(fmaf(s[2 * c + 1], scale_log2, nbase));
                rs4[(2 * c) & 3] += p0;
                rs4[(2 * c + 1) & 3] += p1;
                hi[c] = pack_bf16(p0, p1);
                lo[c] = pack_bf16(p0 - __uint_as_float(hi[c] << 16), p1 - __uint_as_float(hi[c] & 0xffff0000u));
            }
            l = l * corr + ((rs4[0] + rs4[1]) + (rs4[2] + rs4[3]));
            // only a rescale needs the product of the tile before to be done (it adds into O)
            if (it > 0 && __any_sync(0xffffffffu, corr != 1.0f)) {
                w = lt_wait(&pv_done[(it - 1) & 1], ((it - 1) >> 1) & 1, abort_flag);
                if (!__all_sync(0xffffffffu, w)) { ok = false; break; }
                lt_fence_after();
#pragma unroll 1
                for (int c0 = 0; c0 < vcols; c0 += 32) {
                    float ov[32];
                    lt_ld32(lane_addr + LT_O_COL + c0, ov);
                    uint32_t h[16];
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) h[j] = __float_as_uint(ov[16 * half + j] * corr);
                        lt_st16(lane_addr + LT_O_COL + c0 + 16 * half, h);
                    }
                }
            }
            lt_st16(lane_addr + st * LT_KEYS, hi);
            lt_st16(lane_addr + st * LT_KEYS + 16, lo);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            lt_fence_before();
            __syncwarp();
            if (lane == 0) lt_arrive(&p_ready[st]);
        }
        if (ok) {
            const bool w = lt_wait(&pv_done[(nkt - 1) & 1], ((nkt - 1) >> 1) & 1, abort_flag);
            ok = __all_sync(0xffffffffu, w);
        }
        if (!ok) {
            *abort_flag = 1;
            if (lane == 0) atomicExch(err, 1);
        } else {
            lt_fence_after();
            const float inv = (l > 0.0f) ? 1.0f / l : 0.0f;
            float* dst = out + (grow0 + r) * dv + v0 * 64;
#pragma unroll 1
            for (int c0 = 0; c0 < vcols; c0 += 32) {
                float ov[32];
                lt_ld32(lane_addr + LT_O_COL + c0, ov);
                if (row_ok) {
#pragma unroll
                    for (int j = 0; j < 32; j += 4)
                        *reinterpret_cast<float4*>(dst + c0 + j) =
                            make_float4(ov[j] * inv, ov[j + 1] * inv, ov[j + 2] * inv, ov[j + 3] * inv);
                }
            }
        }
    }

    if (threadIdx.x == 0) {
        // the block's own copies have landed before it leaves; they have by now, unless a wait ran out
        mbar_wait(q_full, 0);
        for (int st = 0; st < 2; ++st) {
            if (a_issued[st] > 0) mbar_wait(&a_full[st], (uint32_t)(a_issued[st] - 1) & 1u);
            if (v_issued[st] > 0) mbar_wait(&v_full[st], (uint32_t)(v_issued[st] - 1) & 1u);
        }
    }
    lt_fence_before();
    __syncthreads();
    if (warp == 1) {
        lt_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// ------------------------------------------------------------------------------------ host
typedef CUresult (*LtEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// A row-major bfloat16 matrix [rows, W] in boxes of box_rows x 64 values, 128-byte swizzle, zeros outside.
static int lt_map(CUtensorMap* map, const void* base, long long rows, int W, int box_rows) {
    static LtEncodeFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult res;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &res) == cudaSuccess &&
            res == cudaDriverEntryPointSuccess)
            fn = (LtEncodeFn)ptr;
    }
    if (!fn) return LUMEN_ERR_UNSUPPORTED;
    cuuint64_t dims[2] = {(cuuint64_t)W, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)W * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : LUMEN_ERR_BAD_ARGUMENT;
}

// 1 if lumen_attn_latent_tc takes rows of W values with dv of them the value: whole 64-column blocks, and Q with two key
// tiles within a block's shared memory.
LUMEN_API int lumen_attn_latent_tc_takes(int W, int dv) {
    return (W > 0 && W % 64 == 0 && W <= LT_MAX_W && dv > 0 && dv % 64 == 0 && dv <= W) ? 1 : 0;
}

// q bfloat16 [N, H, W]; cache bfloat16 [n_pages, 1, PAGE, W] (plain tiles), both 16-byte aligned; out float32 [N, H, dv];
// cu_q, seq_start, window as in lumen_attn_latent; n_tiles >= the sum over sequences of ceil(q_len H / 128).
// give_up_at: the key tile of a block at which its softmax takes the wait for its scores as run out (-1: none; for tests of
// what a block does then).
LUMEN_API int lumen_attn_latent_tc(const void* q, const void* cache, int n_pages, const int* block_table, int bt_stride,
                                   const int* cu_q, const int* seq_start, int B, int n_tiles, float* out, int N, int H,
                                   int W, int dv, int window, float scale, int give_up_at, int* err, cudaStream_t stream) {
    if (B <= 0 || n_tiles <= 0 || N <= 0) return 0;
    if (H <= 0 || window < 0 || !(scale > 0.0f) || !lumen_attn_latent_tc_takes(W, dv)) return LUMEN_ERR_UNSUPPORTED;
    if ((long long)N * H > 2147483647LL || (long long)n_pages * LUMEN_PAGE > 2147483647LL) return LUMEN_ERR_UNSUPPORTED;
    if (((uintptr_t)q & 15) || ((uintptr_t)cache & 15) || ((uintptr_t)out & 15)) return LUMEN_ERR_BAD_ARGUMENT;
    CUtensorMap mq, mk;
    int rc;
    if ((rc = lt_map(&mq, q, (long long)N * H, W, LT_ROWS))) return rc;
    if ((rc = lt_map(&mk, cache, (long long)n_pages * LUMEN_PAGE, W, LT_KEYS))) return rc;
    int smem = (W / 64) * (LT_QBLOCK + 2 * LT_KBLOCK) + 256;
    if (smem < 116 * 1024) smem = 116 * 1024;              // a block has the SM's tensor memory to itself
    cudaError_t e = cudaFuncSetAttribute(attn_latent_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    lumen_launch(attn_latent_tc_kernel, dim3(n_tiles, (dv + LT_SLICE - 1) / LT_SLICE), dim3(LT_THREADS), smem, stream, mq, mk,
                 block_table, bt_stride, cu_q, seq_start, B, out, H, W, dv, window, scale * 1.4426950408889634f, give_up_at, err);
    LUMEN_LAUNCH_CHECK();
    return 0;
}
