// Float32 matrix product C[M,N] = A[M,K] * W[N,K]^T on the 5th-generation tensor cores, with the error of a 32-bit
// product: every float32 operand is cut into three bfloat16 numbers, x = x1 + 2^-8 x2 + 2^-16 x3 exactly, from the smallest
// number to where one rounds to infinity (x1 is the number rounded to eight significant bits, x2 2^8 times what is left,
// rounded likewise, x3 2^8 times what is left then: scaled, so that the parts of a small number are still bfloat16 numbers).
// Of the nine products of parts the six largest are made, x3 y1 + x1 y3 + x2 y2, 2^-8 of that + x2 y1 + x1 y2, 2^-8 of that
// + x1 y1 (the accumulator is scaled by the instruction that goes on with it), each exactly, as a product of two eight-bit numbers is. The three
// left out reach 2^-24 of a product (2^-27.4 rms). A subnormal operand has fewer bits in front, and counts as if it were off by up to
// the spacing of the numbers there, 2^-149. W may be bfloat16 (one part, three products, nothing left out).
//
// The tensor core's own sums are short: 64 values of k and their parts, small ones first, into a fresh accumulator, which loses up to
// an ulp an instruction and is then added to a running sum in registers, rounded to nearest. So an output is a chain of K / 64 float32 adds (in
// up to four shares of k, added in rising order) where the FFMA kernel's is K / 4. Against a 64-bit product, 2-norm,
// this / FFMA: K = 1,000 9.7e-8 / 2.8e-7, 2,048 1.0e-7 / 4.1e-7, 8,192 1.4e-7 / 8.1e-7; of numbers that are all positive
// 9.4e-8 / 1.3e-7, 8.8e-8 / 1.6e-7, 9.4e-8 / 3.1e-7. Rows of zeros but for a few numbers gain nothing by short chains: one number of 2,048
// 4.5e-8 / 2.5e-8, 16 7.2e-8 / 5.8e-8, 64 8.1e-8 / 8.4e-8.
//
// A block takes 128 rows of W (the 128-row side of the MMA) times up to 160 rows of A, for a share of k; the blocks of
// one tile, one for each share, are a cluster and add up their sums through distributed shared memory. The number of
// shares depends on N and K alone, so C[m,n] depends on row m of A and row n of W only, never on M or where they lie.
//   warps 0..7   fetch 64 columns of W into registers, cut them and store the parts as 128-byte-swizzled tiles, two buffers.
//                Up to 32 rows of A go the same way; more are cut once, by a kernel
//                ahead of this one, into the image their tiles have in shared memory (a block that cut 160 rows of A for its
//                128 of W spent half of its time on them), and are copied by
//   a warp       that does nothing else;
//   two warps    issue the products in turns (a lane that issues is held up until the tensor pipe takes its product, so a
//                single one would leave the pipe idle while it goes through its barriers); one allocates tensor memory;
//   the others   add the finished accumulator (two of them, in tensor memory) to the sums in their registers.
// An infinity or a NaN leaves NaN in its parts, and so in its outputs: a block's sums that are not finite, for this or any other
// reason, are made again with plain FMAs.
//
// What bounds it: for many rows the chain of a buffer, parts stored (1,270 cycles a block of 64 columns), products (1,900, the tensor
// pipe's time for 24 of 128 x 160 x 16) and the barriers between, of which two are under way; for few rows the stream over W, of which
// 64 KB an SM are under way; and some 9 us a block for its start, first fetch and sums.
// us, L2 cold, FFMA -> this (with the kernel ahead): 300 rows x 16,384 outputs x 2,048 518 -> 120 (1.0 PFLOP/s of bfloat16 products); 300 x 2,048 x
// 8,192 447 -> 69; 300 x 2,048 x 2,048 121 -> 30; 300 x 3,072 x 2,048 121 -> 48; 100 x 2,048 x 8,192 226 -> 60; 64 x 16,384 x 2,048 123 -> 54; 16 x
// 32,768 x 2,048 107 -> 84; 8 x 16,384 x 2,048 72 -> 57; 8 x 2,048 x 8,192 117 -> 55; 8 x 1,024 x 1,024 21 -> 14. Parts that were not
// scaled, with marks of the rows that hold something that is not finite: 126 for the first, 6 % over all sizes. Tried, 300 x 16,384 x 2,048, L2 warm (118
// then): A cut by every block 169; one warp issuing, loads asked for before the fence 136; two groups of cutting warps in turns 147; parts
// waiting in registers for a buffer 172. Eight shares: 300 x 2,048 x 8,192 101 (67), 300 x 2,048 x 2,048 43 (23), but 8 x 2,048 x 8,192 32 (39):
// few rows over a long k pay for many.
// Every wait is bounded; when one runs out the block raises the error flag, its other roles give up on theirs, and the
// block leaves, through the same cluster barriers as ever, once the products it has issued are done.
#include "common.cuh"
#include "mma_utils.cuh"

#define FT_ROWS 128                      // rows of W a block
#define FT_BK 64
#define FT_MAX_BN 160                    // rows of A a block
#define FT_CONV 8                        // warps that fetch and cut
#define FT_W_TILE (FT_ROWS * 128)        // bytes of one part of a tile of W
#define FT_MAX_SHARES 4                  // 16 clusters of eight blocks that fill an SM each take two rounds, 32 of four one
#define FT_MIN_N 1024                    // see lumen_gemm_f32_tc_takes
#define FT_MIN_K 1024
#define FT_IMAGE_MAX (256ll << 20)       // bytes of cut activations at a time (or one tile): products of a millisecond and more

__device__ __forceinline__ void ft_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void ft_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ft_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void ft_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void ft_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// The same onto 2^-8 times the accumulator.
__device__ __forceinline__ void ft_mma_2m8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
    asm volatile(
        "{\n .reg .pred p;\n setp.eq.b32 p, 0, 0;\n"
        " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p, 8;\n}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc)
        : "memory");
}
__device__ __forceinline__ void ft_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// As mbar_wait, but given up as soon as another role of the block has.
__device__ __forceinline__ bool ft_wait(uint64_t* bar, uint32_t parity, const volatile int* abort_flag) {
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
// A K-major operand tile of 128-byte rows in the 128-byte swizzle, groups of 8 rows 1024 bytes apart.
__device__ __forceinline__ uint64_t ft_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// D float32, A and B bfloat16, both K-major, M = 128.
__device__ __forceinline__ uint32_t ft_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(FT_ROWS >> 4) << 24);
}
__device__ __forceinline__ void ft_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 ft_peer(uint32_t addr, uint32_t rank) {         // 16 bytes of another block's shared memory
    uint32_t a;
    float4 v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
    return v;
}

// Four values of a row as they lie in memory (zeros where there are none).
template <typename T> struct FtRaw;
template <> struct FtRaw<float> { float4 v; };
template <> struct FtRaw<__nv_bfloat16> { uint2 v; };
__device__ __forceinline__ void ft_fetch(FtRaw<float>& x, const float* p, int left, bool vec) {
    x.v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (vec) {
        if (left > 0) x.v = __ldg(reinterpret_cast<const float4*>(p));
    } else {
        if (left > 0) x.v.x = __ldg(p);
        if (left > 1) x.v.y = __ldg(p + 1);
        if (left > 2) x.v.z = __ldg(p + 2);
        if (left > 3) x.v.w = __ldg(p + 3);
    }
}
__device__ __forceinline__ void ft_fetch(FtRaw<__nv_bfloat16>& x, const __nv_bfloat16* p, int left, bool vec) {
    x.v = make_uint2(0u, 0u);
    if (vec) {
        if (left > 0) x.v = __ldg(reinterpret_cast<const uint2*>(p));
    } else {
        const unsigned short* q = reinterpret_cast<const unsigned short*>(p);
        if (left > 0) x.v.x = __ldg(q);
        if (left > 1) x.v.x |= (uint32_t)__ldg(q + 1) << 16;
        if (left > 2) x.v.y = __ldg(q + 2);
        if (left > 3) x.v.y |= (uint32_t)__ldg(q + 3) << 16;
    }
}
// Two numbers rounded to bfloat16, side by side; x becomes what is left of each, times 2^8 (exactly).
__device__ __forceinline__ uint32_t ft_cut(unsigned long long& x) {
    uint32_t a, b;
    unsigned long long r;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(a), "=r"(b) : "l"(x));
    const uint32_t h = pack_bf16(__uint_as_float(a), __uint_as_float(b));
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(h << 16), "r"(h & 0xffff0000u));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(x) : "l"(r), "l"(0xbf800000bf800000ull));       // x - r
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(x) : "l"(0x4380000043800000ull));
    return h;
}
// Cuts four values and stores their parts `part` bytes apart. What is not finite (or rounds to infinity) leaves NaN in its second part.
__device__ __forceinline__ void ft_store(const FtRaw<float>& x, unsigned char* dst, int part) {
    unsigned long long a, b;
    asm("mov.b64 %0, {%1, %2};" : "=l"(a) : "f"(x.v.x), "f"(x.v.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(x.v.z), "f"(x.v.w));
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        uint2 h;
        h.x = ft_cut(a);
        h.y = ft_cut(b);
        *reinterpret_cast<uint2*>(dst + i * part) = h;
    }
}
__device__ __forceinline__ void ft_store(const FtRaw<__nv_bfloat16>& x, unsigned char* dst, int) { *reinterpret_cast<uint2*>(dst) = x.v; }

// DEEP: a block has an SM to itself and two blocks of W under way (up to 16 rows, where two blocks share an SM if there are that many).
template <typename TW, int BN, bool DEEP>
struct FtShape {
    static constexpr int NW = sizeof(TW) == 4 ? 3 : 1;                   // parts of a weight
    static constexpr int HALVES = BN > 64 ? 2 : 1;                       // groups of four adding warps, by columns
    static constexpr bool IMAGE = BN > 32;                               // A arrives cut
    static constexpr int EPI = 4 * HALVES, MMA = FT_CONV + EPI, COPY = MMA + 2, WARPS = IMAGE ? COPY + 1 : COPY;
    static constexpr int A_TILE = BN * 128;
    static constexpr int BUF = NW * FT_W_TILE + 3 * A_TILE;
    static constexpr int TMEM = 2 * BN <= 32 ? 32 : 2 * BN <= 64 ? 64 : 2 * BN <= 128 ? 128 : 2 * BN <= 256 ? 256 : 512;
    static constexpr int CTL = 1024;                                     // barriers, flags
    static constexpr int SMEM = 2 * BUF + CTL;
    static constexpr int MINB = DEEP ? 1 : 2;
    static_assert(DEEP || 2 * SMEM <= 220 * 1024, "two blocks fit an SM");
    static constexpr int SETS = MINB == 1 ? 2 : 1;                       // blocks of W under way in registers
    static_assert(BN * FT_ROWS * 4 <= 2 * BUF, "the sums are staged where the tiles were");
};

template <typename TW, int BN, bool DEEP>
__global__ void __launch_bounds__(32 * FtShape<TW, BN, DEEP>::WARPS, FtShape<TW, BN, DEEP>::MINB)
gemm_f32_tc_kernel(const float* __restrict__ A, const unsigned char* __restrict__ image, const TW* __restrict__ W, float* __restrict__ C, int M, int N, int K, int bn, int vec, int early, int give_up_at,
                   int* __restrict__ err) {
    using F = FtShape<TW, BN, DEEP>;
    constexpr int NW = F::NW, EPI = F::EPI, ACOL = F::TMEM / 2;
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* tiles = smem;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + 2 * F::BUF);
    uint64_t* full = bars;              // [2] the parts of a block of k are in shared memory
    uint64_t* done = bars + 2;          // [2] its products are in the accumulator: the buffer is free, the sums can be taken
    uint64_t* taken = bars + 4;         // [2] the accumulator has been read
    uint64_t* landed = bars + 6;        // [2] the parts of A have been copied
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 8);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* any_odd = reinterpret_cast<volatile int*>(tmem_slot + 2);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = gridDim.x, share = blockIdx.x;                             // the cluster is one tile's shares of k
    const int m0 = blockIdx.y * bn, n0 = blockIdx.z * FT_ROWS;
    const int num_kb = (K + FT_BK - 1) / FT_BK, per = (num_kb + S - 1) / S;
    const int kb0 = min(share * per, num_kb), nk = min(kb0 + per, num_kb) - kb0;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&full[i], FT_CONV);
            mbar_init(&done[i], 1);
            mbar_init(&taken[i], EPI);
            mbar_init(&landed[i], 1);
        }
        *abort_flag = 0;
        *any_odd = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == F::MMA) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(F::TMEM)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const int rows = min(bn, M - m0), cols = min(FT_ROWS, N - n0);
    // fetches of a cutting warp's thread: 16 threads a row
    constexpr int LW = FT_ROWS / 16, LA = BN / 16;
    const int c = threadIdx.x & 15, r = threadIdx.x >> 4;
    FtRaw<TW> rw[F::SETS][LW];
    auto fetch_w = [&](int kb, FtRaw<TW> (&x)[LW]) {
        const int k = (kb0 + kb) * FT_BK + 4 * c;
        const TW* p = W + (size_t)(n0 + r) * K + k;
#pragma unroll
        for (int i = 0; i < LW; ++i) ft_fetch(x[i], p + (size_t)(16 * i) * K, kb < nk && r + 16 * i < cols ? K - k : 0, vec);
    };
    // A model's weights never change: its first ones are asked for before the kernel ahead has ended. Nothing else of this
    // kernel touches global memory before the wait.
    if (early && warp < FT_CONV) {
#pragma unroll
        for (int i = 0; i < F::SETS; ++i) fetch_w(i, rw[i]);
    }
    pdl_wait();
    pdl_trigger();
    if (!early && warp < FT_CONV) {
#pragma unroll
        for (int i = 0; i < F::SETS; ++i) fetch_w(i, rw[i]);
    }
    ft_fence_before();
    __syncthreads();
    ft_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    float* sums = reinterpret_cast<float*>(tiles);             // [BN][128], over the tiles once they have been read

    if (warp < FT_CONV) {
        FtRaw<float> ra[F::IMAGE ? 1 : LA];
        auto fetch_a = [&](int kb) {
            const int k = (kb0 + kb) * FT_BK + 4 * c;
            const float* p = A + (size_t)(m0 + r) * K + k;
            if constexpr (!F::IMAGE) {
#pragma unroll
                for (int i = 0; i < LA; ++i) ft_fetch(ra[i], p + (size_t)(16 * i) * K, kb < nk && r + 16 * i < rows ? K - k : 0, vec);
            }
        };
        // this thread's four values of row r: 8 bytes in the 16-byte piece c / 2, which lies at (c / 2) ^ (row & 7)
        const uint32_t at = r * 128 + (((c >> 1) ^ (r & 7)) << 4) + (c & 1) * 8;
        auto room = [&](int kb) -> bool {        // the buffer of block kb is free
            if (kb < 2 || __all_sync(0xffffffffu, ft_wait(&done[kb & 1], ((kb >> 1) & 1) ^ 1, abort_flag))) return true;
            *abort_flag = 1;
            if (lane == 0) atomicExch(err, 1);
            return false;
        };
        auto step = [&](int kb, FtRaw<TW> (&x)[LW]) -> bool {
            if (!room(kb)) return false;
            unsigned char* tw = tiles + (kb & 1) * F::BUF + at;
            unsigned char* ta = tw + NW * FT_W_TILE;
#pragma unroll
            for (int i = 0; i < LW; ++i) ft_store(x[i], tw + i * 16 * 128, FT_W_TILE);
            if constexpr (!F::IMAGE) {
#pragma unroll
                for (int i = 0; i < LA; ++i) ft_store(ra[i], ta + i * 16 * 128, F::A_TILE);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // before the next loads, which it would wait for
            __syncwarp();
            if (lane == 0) ft_arrive(&full[kb & 1]);
            fetch_w(kb + F::SETS, x);
            fetch_a(kb + 1);
            return true;
        };
        fetch_a(0);
        for (int kb = 0; kb < nk; kb += F::SETS) {
            if (!step(kb, rw[0])) break;
            if (F::SETS == 2 && kb + 1 < nk && !step(kb + 1, rw[F::SETS - 1])) break;
        }
    } else if (warp == F::MMA || warp == F::MMA + 1) {
        if (lane == 0) {
            const uint32_t idesc = ft_idesc(bn);
            int issued = 0;
            bool ok = true;
            for (int kb = warp - F::MMA; kb < nk; kb += 2) {
                const int b = kb & 1;
                ok = (kb < 2 || ft_wait(&taken[b], ((kb >> 1) & 1) ^ 1, abort_flag)) &&
                     (!F::IMAGE || ft_wait(&landed[b], (kb >> 1) & 1, abort_flag)) && ft_wait(&full[b], (kb >> 1) & 1, abort_flag);
                if (!ok) break;
                ft_fence_after();
                const uint32_t tw = smem_u32(tiles + b * F::BUF), ta = tw + NW * FT_W_TILE, d = tmem_base + b * ACOL;
                // first: what the accumulator does at this product's start, 0 it begins anew, 1 goes on, 2 goes on 2^-8 times
                auto product = [&](int pw, int pa, int first) {
                    const uint64_t wd = ft_desc(tw + pw * FT_W_TILE), ad = ft_desc(ta + pa * F::A_TILE);
                    if (first == 2) ft_mma_2m8(d, wd, ad, idesc);
                    else ft_mma(d, wd, ad, idesc, first);
#pragma unroll
                    for (int k = 1; k < FT_BK / 16; ++k) ft_mma(d, wd + 2 * k, ad + 2 * k, idesc, 1);
                };
                if (NW == 3) {
                    product(2, 0, 0);
                    product(0, 2, 1);
                    product(1, 1, 1);
                    product(1, 0, 2);
                    product(0, 1, 1);
                } else {
                    product(0, 2, 0);
                    product(0, 1, 2);
                }
                product(0, 0, 2);
                ft_commit(&done[b]);
                issued = kb + 1;
            }
            if (!ok) { *abort_flag = 1; atomicExch(err, 1); }
            // the block keeps its shared and tensor memory until the products that use them are done
            if (issued > 0 && !mbar_wait(&done[(issued - 1) & 1], ((issued - 1) >> 1) & 1)) atomicExch(err, 1);
        }
        __syncwarp();
    } else if (F::IMAGE && warp == F::COPY) {
        if (lane == 0) {
            const unsigned char* from = image + ((size_t)blockIdx.y * num_kb + kb0) * 3 * bn * 128;
            int asked = 0;
            for (int kb = 0; kb < nk; ++kb) {
                const int b = kb & 1;
                if (kb >= 2 && !ft_wait(&done[b], ((kb >> 1) & 1) ^ 1, abort_flag)) {
                    *abort_flag = 1;
                    atomicExch(err, 1);
                    break;
                }
                mbar_expect_tx(&landed[b], 3 * bn * 128);
                for (int i = 0; i < 3; ++i)
                    bulk_load(tiles + b * F::BUF + NW * FT_W_TILE + i * F::A_TILE, from + ((size_t)kb * 3 + i) * bn * 128, bn * 128, &landed[b]);
                asked = kb + 1;
            }
            // the block stays until its copies have landed
            for (int kb = max(0, asked - 2); kb < asked; ++kb)
                if (!mbar_wait(&landed[kb & 1], (kb >> 1) & 1)) atomicExch(err, 1);
        }
        __syncwarp();
    } else {
        constexpr int COLS = BN / F::HALVES;                    // rows of A an adding warp keeps
        const int qd = warp & 3, first = ((warp - FT_CONV) >> 2) * COLS, n = qd * 32 + lane;
        const uint32_t lane_addr = tmem_base + ((uint32_t)(qd * 32) << 16) + first;
        float acc[COLS];
#pragma unroll
        for (int j = 0; j < COLS; ++j) acc[j] = 0.0f;
        for (int kb = 0; kb < nk; ++kb) {
            const int b = kb & 1;
            const bool w = kb != give_up_at && ft_wait(&done[b], (kb >> 1) & 1, abort_flag);
            if (!__all_sync(0xffffffffu, w)) {
                *abort_flag = 1;
                if (lane == 0) atomicExch(err, 1);
                break;
            }
            ft_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < COLS; c0 += 16) {
                float v[16];
                ft_ld16(lane_addr + b * ACOL + c0, v);
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c0 + j] += v[j];
            }
            ft_fence_before();
            __syncwarp();
            if (lane == 0) ft_arrive(&taken[b]);
        }
        // the last block's products are done, so no tile is read or written any more (unless a wait ran out)
        bool odd = false;
#pragma unroll
        for (int j = 0; j < COLS; ++j) odd |= first + j < rows && !isfinite(acc[j]);
        if (odd) *any_odd = 1;
        asm volatile("bar.sync 1, %0;" ::"n"(32 * EPI) : "memory");
        if (S == 1 && !*any_odd) {
            if (n < cols) {
                float* dst = C + (size_t)(m0 + first) * N + n0 + n;
#pragma unroll
                for (int j = 0; j < COLS; ++j)
                    if (first + j < rows) dst[(size_t)j * N] = acc[j];
            }
        } else {
#pragma unroll
            for (int j = 0; j < COLS; ++j) sums[(first + j) * FT_ROWS + n] = acc[j];
        }
    }

    ft_fence_before();
    __syncthreads();
    ft_fence_after();
    if (warp == F::MMA)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(F::TMEM) : "memory");
    const bool odd = *any_odd != 0;
    if (S == 1 && !odd) return;
    if (odd) {
        for (int e = threadIdx.x; e < rows * FT_ROWS; e += blockDim.x) {
            const int m = e / FT_ROWS, n = e % FT_ROWS;
            if (n >= cols || isfinite(sums[e])) continue;
            float s = 0.0f;
            const int k1 = min(K, (kb0 + nk) * FT_BK);
            for (int k = kb0 * FT_BK; k < k1; ++k) s = fmaf(A[(size_t)(m0 + m) * K + k], to_f32(W[(size_t)(n0 + n) * K + k]), s);
            sums[e] = s;
        }
    }
    if (S > 1) ft_cluster_sync();
    else __syncthreads();
    for (int e = 4 * (share * blockDim.x + threadIdx.x); e < rows * FT_ROWS; e += 4 * S * blockDim.x) {
        const int m = e / FT_ROWS, n = e % FT_ROWS;
        if (n >= cols) continue;
        float4 s = *reinterpret_cast<const float4*>(sums + e);
        if (S > 1) {
            float4 part[FT_MAX_SHARES];                        // all on their way before the first is added
            const uint32_t a = smem_u32(sums + e);
#pragma unroll
            for (int p = 0; p < FT_MAX_SHARES; ++p)
                if (p < S) part[p] = ft_peer(a, p);
            s = part[0];
#pragma unroll
            for (int p = 1; p < FT_MAX_SHARES; ++p)
                if (p < S) {
                    s.x += part[p].x;
                    s.y += part[p].y;
                    s.z += part[p].z;
                    s.w += part[p].w;
                }
        }
        float* dst = C + (size_t)(m0 + m) * N + n0 + n;
        if ((N & 3) == 0 && ((uintptr_t)C & 15) == 0) {
            *reinterpret_cast<float4*>(dst) = s;
        } else {
            dst[0] = s.x;
            if (n + 1 < cols) dst[1] = s.y;
            if (n + 2 < cols) dst[2] = s.z;
            if (n + 3 < cols) dst[3] = s.w;
        }
    }
    if (S > 1) ft_cluster_sync();          // a block's sums stay until the others have read them
}

// A cut into parts, in the image the blocks copy: tile of bn rows after tile, block of 64 columns after block, part after part, a
// part bn rows of 128 bytes in the 128-byte swizzle. A block of threads a row (of the last tile's absent rows too, zeros).
__global__ void __launch_bounds__(256)
gemm_f32_image_kernel(const float* __restrict__ A, unsigned char* __restrict__ image, int M, int K, int bn, int vec) {
    pdl_wait();
    pdl_trigger();
    const int row = blockIdx.x, r = row % bn, num_kb = (K + FT_BK - 1) / FT_BK;
    unsigned char* tile = image + (size_t)(row / bn) * num_kb * 3 * bn * 128 + r * 128;
    for (int i = threadIdx.x; i < num_kb * 16; i += 256) {
        const int c = i & 15;
        FtRaw<float> x;
        ft_fetch(x, A + (size_t)row * K + 4 * i, row < M ? K - 4 * i : 0, vec);
        ft_store(x, tile + (size_t)(i >> 4) * 3 * bn * 128 + (((c >> 1) ^ (r & 7)) << 4) + (c & 1) * 8, bn * 128);
    }
}

// Rows of A a block: as few tiles as there can be, of even height.
static int gemm_f32_tc_tile(int M) {
    const int tiles = (M + FT_MAX_BN - 1) / FT_MAX_BN;
    return ((M + tiles - 1) / tiles + 15) / 16 * 16;
}
// Tiles of bn rows that are cut at a time; more go through the same scratch one lot after the other (six bytes a number of A
// would be 1.26 GB for 8,192 rows of 25,600).
static int gemm_f32_tc_lot(int M, int K, int bn) {
    const long long tile = (long long)bn * ((K + FT_BK - 1) / FT_BK) * 3 * 128, tiles = (M + bn - 1) / bn;
    return (int)(tiles * tile <= FT_IMAGE_MAX ? tiles : FT_IMAGE_MAX / tile > 0 ? FT_IMAGE_MAX / tile : 1);
}
static size_t gemm_f32_tc_image(int M, int K) {               // bytes of the image
    const int bn = gemm_f32_tc_tile(M);
    return bn <= 32 ? 0 : (size_t)gemm_f32_tc_lot(M, K, bn) * bn * ((K + FT_BK - 1) / FT_BK) * 3 * 128;
}

template <typename TW, int BN, bool DEEP>
static int gemm_f32_tc_go(const float* A, const TW* W, float* C, unsigned char* work, int M, int N, int K, int bn, int S,
                          int early, int give_up_at, int* err, cudaStream_t stream) {
    using F = FtShape<TW, BN, DEEP>;
    auto k = gemm_f32_tc_kernel<TW, BN, DEEP>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, F::SMEM);
    if (e != cudaSuccess) return (int)e;
    const int vec_a = (K & 3) == 0 && ((uintptr_t)A & 15) == 0, vec_w = (K & 3) == 0 && ((uintptr_t)W & (4 * sizeof(TW) - 1)) == 0;
    int lot = M;
    if (F::IMAGE) {
        // of the lots that fit, the one whose blocks take the fewest rounds on the SMs (ms, all at once / in lots: 8,192 x 2,048 x 25,600
        // 5.33 / 5.46, 1.28 GB / 0.25; 6,000 x 3,000 x 16,384 4.38 / 4.44; 3,000 x 2,048 x 16,384 1.74 / 1.62)
        const long long most = gemm_f32_tc_lot(M, K, bn), tiles = (M + bn - 1) / bn, tile_blocks = (long long)S * ((N + FT_ROWS - 1) / FT_ROWS);
        const int at_once = S == 1 ? 148 : 144;
        auto rounds = [&](long long t) { return (t * tile_blocks + at_once - 1) / at_once; };
        long long fewest = 0;
        for (long long t = most; most < tiles && t > most / 2; --t) {
            const long long all = tiles / t * rounds(t) + rounds(tiles % t);
            if (fewest == 0 || all < fewest) {
                fewest = all;
                lot = (int)t * bn;
            }
        }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(32 * F::WARPS);
    cfg.dynamicSmemBytes = F::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = lumen_pdl_enabled() ? 2 : 1;
    for (int m = 0; m < M; m += lot) {           // the kernel that cuts the next lot waits for the product of the one before
        const int rows = lot < M - m ? lot : M - m, tiles = (rows + bn - 1) / bn;
        if (F::IMAGE) {
            lumen_launch(gemm_f32_image_kernel, dim3(tiles * bn), dim3(256), 0, stream, A + (size_t)m * K, work, rows, K, bn, vec_a);
            LUMEN_LAUNCH_CHECK();
        }
        cfg.gridDim = dim3(S, tiles, (N + FT_ROWS - 1) / FT_ROWS);
        e = cudaLaunchKernelEx(&cfg, k, A + (size_t)m * K, (const unsigned char*)work, W, C + (size_t)m * N, rows, N, K, bn,
                               F::IMAGE ? vec_w : vec_a && vec_w, early, give_up_at, err);
        if (e != cudaSuccess) return (int)e;
        LUMEN_LAUNCH_CHECK();
    }
    return 0;
}

// Shares of k: as many as keep the blocks of one row of tiles within the SMs, with four blocks of k each, taken over all.
static int gemm_f32_tc_shares(int N, int K) {
    const int tiles = (N + FT_ROWS - 1) / FT_ROWS, num_kb = (K + FT_BK - 1) / FT_BK;
    int S = 1;
    while (S < FT_MAX_SHARES && 2 * S * tiles <= 148 && num_kb >= 8 * S) S *= 2;
    return S;
}

template <typename TW>
static int gemm_f32_tc_rows(const float* A, const TW* W, float* C, unsigned char* work, int M, int N, int K, int early, int give_up_at,
                            int* err, cudaStream_t stream) {
    const int S = gemm_f32_tc_shares(N, K), bn = gemm_f32_tc_tile(M);
#define FT_GO(BN, DEEP) \
    if (bn <= BN) return gemm_f32_tc_go<TW, BN, DEEP>(A, W, C, work, M, N, K, bn, S, early, give_up_at, err, stream)
    // two blocks an SM where there are more blocks than SMs (8 x 16,384 x 2,048, 128 blocks: 48 us, 52 with one
    // block of weights under way)
    if ((long long)S * ((N + FT_ROWS - 1) / FT_ROWS) > 148) FT_GO(16, false);
    FT_GO(16, true);
    FT_GO(32, true);
    FT_GO(64, true);
    FT_GO(96, true);
    FT_GO(128, true);
    FT_GO(160, true);
#undef FT_GO
    return LUMEN_ERR_UNSUPPORTED;
}

// 1 if weights [N, K] go through this kernel, whatever M: by N and K alone, so that a row's value is the same in any batch.
// Smaller weights leave most SMs idle and are FFMA's: 300 rows x 512 x 512 17.7 us there, 21.7 here; 300 x 1,024 x 300 13 / 21;
// 2,048 x 256 x 256 11 / 18. Weights that are long one way only (16,384 x 896) have not been measured and stay there too.
LUMEN_API int lumen_gemm_f32_tc_takes(int N, int K) { return N >= FT_MIN_N && K >= FT_MIN_K ? 1 : 0; }

// Bytes of scratch lumen_gemm_f32_tc needs.
LUMEN_API long long lumen_gemm_f32_tc_scratch(int M, int K) {
    return M > 0 && K > 0 ? (long long)gemm_f32_tc_image(M, K) : 0;
}

// A float32 [M, K], W float32 or bfloat16 [N, K], C float32 [M, N], rows dense, of any alignment their types
// have. work: lumen_gemm_f32_tc_scratch(M, K) bytes, 16-byte aligned. early: W was written before the kernels that are still on
// their way in the stream (a model's weights), and may be read before they end. give_up_at: the block of k at which the adding warps
// take their wait as run out (-1: none; for tests of what a block does then).
LUMEN_API int lumen_gemm_f32_tc(const float* A, const void* W, int w_is_bf16, float* C, void* work, int M, int N, int K,
                                int early, int give_up_at, int* err, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || ((uintptr_t)work & 15) || (!work && gemm_f32_tc_image(M, K))) return LUMEN_ERR_BAD_ARGUMENT;
    if ((M + 63) / 64 > 65535 || (N + FT_ROWS - 1) / FT_ROWS > 65535) return LUMEN_ERR_UNSUPPORTED;
    unsigned char* w = (unsigned char*)work;
    return w_is_bf16 ? gemm_f32_tc_rows(A, (const __nv_bfloat16*)W, C, w, M, N, K, early, give_up_at, err, stream)
                     : gemm_f32_tc_rows(A, (const float*)W, C, w, M, N, K, early, give_up_at, err, stream);
}
