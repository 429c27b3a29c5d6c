// Matrix product of the true 32-bit path for more rows than a decode step has:
//   y[m][n] = sum_k a[m][k] * W[n][k] (+ bias[n]),  float in, float out, dense sums no further from exact than by float FMAs,
// on the fifth-generation tensor cores.
//
// How a float product gets onto bfloat16 tensor cores (the split of Henry, Tang and Heinecke, "Leveraging the bfloat16 artificial intelligence
// datatype for higher-precision computations", 2019).  A float has 24 significant bits, a bfloat16 eight, so
// x = x1 + x2 + x3 exactly with x1 = bf16(x), x2 = bf16(x - x1), x3 = x - x1 - x2 (the differences are exact, and the last
// one has at most seven bits left).  Products of two bfloat16 are exact in float.  Of the nine partial products
// the six of weight 2^-16 and above are computed (1.1, 1.2, 2.1, 2.2, 1.3, 3.1); the three that are left out come to at most
// 2^-24 of |x||y| together, as much as a float rounding.  The tensor core adds up 64 k at a time, the
// smallest products first, and cuts off what does not fit; every such piece is then added to a float accumulator in registers, rounded to
// nearest: a sum over K is K / 64 float additions long instead of K.  For a sum of one term, or a few, that is more than a float FMA
// loses (which rounds once); for dense ones it is less, and against float64 the result is closer than that of the
// library's FMA product, which this replaces: 1.3e-7 against 8.1e-7 of its 2-norm at K = 2,048, 2.2e-7 against 1.6e-6 at
// K = 8,192.  Six tensor-core products in place of one still leave it far ahead: 1,024 tokens x 16,384 x 2,048 in 336 us against
// 1,225 us (204 TFLOP/s, 1,227 on the tensor cores), 1,024 x 2,048 x 8,192 in 182 against 616 us, 64 x 2,048 x 2,048 in 28
// against 51 us (in a captured chain of products).
// Elements below 2^-109 in magnitude lose what lies below 2^-134.  A row with an element of 2^127 or more, an
// infinity or a NaN cannot be split, and where a product overflows the partial ones do so in different directions (x1 y1 to infinity, x1 y2 to
// minus infinity); such results are computed by plain FMAs, so they are what they always were.
//
// Orientation.  The weight rows are the 128-row operand, the tokens the columns (NT = 64 or 128 a tile): an epilogue
// thread owns a weight row, and the 32 threads of a warp store 32 neighbouring features of a token, a whole line.
// The tokens are split once by a kernel of their own into three bfloat16 planes (few bytes beside the product's
// arithmetic) and come by TMA; the weights, which are many and used by few tiles, come as floats by TMA, are split by four
// warps, a weight row a thread, and go to tensor memory as the product's A operand, so nothing but the float weights is
// ever kept.  Six products of one pair of tiles read their operands over and over, and shared memory is what that strains: with
// both operands there a stage of 64 k reads 192 KB and is written 96 KB (2,250 cycles at 128 bytes each, for 1,536 cycles of
// MMA); with A in tensor memory it is 96 KB of B, 48 KB of planes and 64 KB of floats in and out (1,625 cycles).  (A in shared
// memory, split from registers: 467 and 285 us for the first two products above, tensor pipe active 38 %.)
//
// Roles.  Warps 0..3: epilogue (tensor memory quarter = warp), the accumulators of the tile in registers.  Warps 4..7:
// split of the weights (tensor memory quarter = warp - 4).  Warp 8: TMA of the tokens' planes.  Warp 9: tensor memory and MMA
// issue.  Warp 10: TMA of the weights.  Two stages of 64 k (three of float weights), two accumulators.
//
// Few tiles.  Where the tiles would leave most multiprocessors idle, a cluster of S blocks shares a tile: each takes a part of
// K, and the partial sums are added in the order of the ranks through distributed shared memory.
//
// Every wait on an mbarrier is bounded: after the limit a role gives up and the others follow; the block records status 16, waits
// (with a limit) for the copies and products that are under way, and leaves its tile unwritten, as do the blocks that share it.  The
// cluster barriers are reached by every thread on every path.
#include "tcgen05.cuh"

using namespace vapi;

constexpr int LF_BM = 128;                // weight rows a tile
constexpr int LF_BK = 64;                 // k a stage: 128 bytes of bfloat16, one swizzle row
constexpr int LF_STAGES = 2;
constexpr int LF_W_STAGES = 3;
constexpr int LF_THREADS = 352;
constexpr int LF_W_BYTES = LF_BM * LF_BK * 4;             // two boxes of 32 k (128 bytes) x 128 rows
constexpr int LF_A_COLS = LF_BK / 2;                      // tensor-memory columns of one plane: two bfloat16 each
constexpr int LF_A_COL0 = 256;                            // the accumulators lie before it
constexpr int LF_TMEM_COLS = 512;
constexpr float LF_LIMIT = 1.7014118346046923e38f;        // 2^127: from here on a row is not split
constexpr int LF_BAD_TILES = 8;           // the warps that split are at most 5 tiles ahead of the epilogue

template <int NT> struct LfCfg {
    static constexpr int B_PLANE = NT * LF_BK * 2;
    static constexpr int STAGE_BYTES = 3 * B_PLANE;
    static constexpr size_t SMEM = (size_t)LF_W_STAGES * LF_W_BYTES + (size_t)LF_STAGES * STAGE_BYTES + 1024 /*alignment*/ + 256 /*barriers*/ + LF_BAD_TILES * LF_BM;
};

struct LfParams {
    const float* W; const float* act; const float* bias; const int* tok_bad; float* out; int* status;
    int N, K, M, num_kb, num_m, num_tiles, split;
    unsigned polls;                       // of an mbarrier before a role gives up, where that is not the usual limit
    long long out_stride;
};

// the same MMA as umma_f16 with A (two bfloat16 a column, a row a lane) in tensor memory
__device__ __forceinline__ void lf_umma_ts(unsigned tmem_d, unsigned tmem_a, unsigned long long db, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void lf_tmem_st16(unsigned taddr, const unsigned (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
                   "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ unsigned lf_map_rank(unsigned addr, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void lf_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The tokens as three bfloat16 planes [3][M][Kp] (Kp: K rounded up to 8, zeros behind K), and per token whether it
// holds something that cannot be split.  One block a token.
__global__ void __launch_bounds__(256) split_rows_kernel(const float* x, __nv_bfloat16* planes, int* bad, int M, int K, int Kp) {
    const int m = blockIdx.x;
    pdl_trigger();
    pdl_wait();
    const size_t plane = (size_t)M * Kp;
    __nv_bfloat16* row = planes + (size_t)m * Kp;
    float top = 0.f;
    for (int k = threadIdx.x * 4; k < Kp; k += blockDim.x * 4) {
        const float4 v = k < K ? *reinterpret_cast<const float4*>(x + (size_t)m * K + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        top = absmax_nan(absmax_nan(absmax_nan(absmax_nan(top, v.x), v.y), v.z), v.w);
        uint2 p1, p2, p3;
        split_f32x2(v.x, v.y, p1.x, p2.x, p3.x);
        split_f32x2(v.z, v.w, p1.y, p2.y, p3.y);
        *reinterpret_cast<uint2*>(row + k) = p1;
        *reinterpret_cast<uint2*>(row + plane + k) = p2;
        *reinterpret_cast<uint2*>(row + 2 * plane + k) = p3;
    }
    const int any = __syncthreads_or(!(top < LF_LIMIT));
    if (threadIdx.x == 0) bad[m] = any;
}

// a result whose row or token cannot be split, or that came out as no finite number
__device__ __forceinline__ float lf_plain(const float* __restrict__ a, const float* __restrict__ w, int K) {
    float s = 0.f;
#pragma unroll 1
    for (int k = 0; k < K; k += 4) {
        const float4 x = *reinterpret_cast<const float4*>(a + k), y = *reinterpret_cast<const float4*>(w + k);
        s = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, s))));
    }
    return s;
}
__device__ __forceinline__ bool lf_finite(float x) { return fabsf(x) <= 3.402823466e38f; }

// TRIAL: the number of polls before a role gives up comes with the call (a limit that is not a constant costs the thread that issues
// the products 3 %, a second barrier to wait for before a stage's products 4 %)
template <int NT, bool TRIAL>
__global__ void __launch_bounds__(LF_THREADS, 1)
linear_f32_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_tok, const LfParams p) {
    using Cfg = LfCfg<NT>;
    const unsigned polls = TRIAL ? p.polls : TC5_WAIT_LIMIT;
    extern __shared__ unsigned char lf_smem_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(lf_smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char* tok_mem = base + (size_t)LF_W_STAGES * LF_W_BYTES;
    unsigned long long* bars = reinterpret_cast<unsigned long long*>(tok_mem + (size_t)LF_STAGES * Cfg::STAGE_BYTES);
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(bars + 2 * LF_STAGES + 4 + 2 * LF_W_STAGES + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    unsigned char* w_bad = reinterpret_cast<unsigned char*>(bars) + 256;            // [LF_BAD_TILES][128]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int split = p.split, rank = (int)blockIdx.x % split;
    const int first = (int)blockIdx.x / split, step = (int)gridDim.x / split;
    // this block's part of K, in stages
    const int per = (p.num_kb + split - 1) / split;
    const int kb0 = min(rank * per, p.num_kb), kb1 = min(kb0 + per, p.num_kb);
    const unsigned full0 = smem_u32(bars), empty0 = smem_u32(bars + LF_STAGES);
    const unsigned accfull0 = smem_u32(bars + 2 * LF_STAGES), accempty0 = smem_u32(bars + 2 * LF_STAGES + 2);
    const unsigned wfull0 = smem_u32(bars + 2 * LF_STAGES + 4), wempty0 = smem_u32(bars + 2 * LF_STAGES + 4 + LF_W_STAGES);
    const unsigned drained = smem_u32(bars + 2 * LF_STAGES + 4 + 2 * LF_W_STAGES);

    if (threadIdx.x == 0) {
        for (int i = 0; i < LF_STAGES; ++i) { mbar_init(full0 + 8 * i, 1 + 4); mbar_init(empty0 + 8 * i, 1); }
        for (int i = 0; i < 2; ++i) { mbar_init(accfull0 + 8 * i, 1); mbar_init(accempty0 + 8 * i, 4); }
        for (int i = 0; i < LF_W_STAGES; ++i) { mbar_init(wfull0 + 8 * i, 1); mbar_init(wempty0 + 8 * i, 4); }
        mbar_init(drained, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"((unsigned)LF_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc5_fence_before();
    __syncthreads();
    tc5_fence_after();
    const unsigned tmem_base = *tmem_slot;
    pdl_trigger();

    float* part = reinterpret_cast<float*>(base);        // [NT][128]: a shared tile's partial sums, over the weights' stages
    int it = 0;                                          // stages that this thread's role has finished

    if (warp >= 4 && warp < 8) {
        // ---- split of the weights: a row a thread ----
        const int row = (int)threadIdx.x - 128;
        const unsigned a0 = tmem_base + ((unsigned)((warp - 4) * 32) << 16) + LF_A_COL0;
        int tl = 0;
        bool ok = true;
        for (int t = first; t < p.num_tiles && ok; t += step, ++tl) {
            float top = 0.f;
            for (int kb = kb0; kb < kb1; ++kb, ++it) {
                const int s = it % LF_STAGES, ws = it % LF_W_STAGES;
                if (!mbar_wait_role(wfull0 + 8 * ws, (it / LF_W_STAGES) & 1, abort_flag, polls)) ok = false;
                if (!mbar_wait_role(empty0 + 8 * s, ((it / LF_STAGES) & 1) ^ 1, abort_flag, polls)) ok = false;
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                tc5_fence_after();
                const unsigned char* w = base + (size_t)ws * LF_W_BYTES + row * 128;
#pragma unroll
                for (int h = 0; h < 2; ++h) {            // 32 k a time: 16 columns of each plane
                    unsigned p1[16], p2[16], p3[16];
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        const float4 v = *reinterpret_cast<const float4*>(w + h * (LF_W_BYTES / 2) + ((c ^ (row & 7)) << 4));
                        top = absmax_nan(absmax_nan(absmax_nan(absmax_nan(top, v.x), v.y), v.z), v.w);
                        split_f32x2(v.x, v.y, p1[2 * c], p2[2 * c], p3[2 * c]);
                        split_f32x2(v.z, v.w, p1[2 * c + 1], p2[2 * c + 1], p3[2 * c + 1]);
                    }
                    const unsigned a = a0 + (unsigned)(s * 3 * LF_A_COLS + h * 16);
                    lf_tmem_st16(a, p1);
                    lf_tmem_st16(a + LF_A_COLS, p2);
                    lf_tmem_st16(a + 2 * LF_A_COLS, p3);
                }
                if (kb + 1 == kb1) w_bad[(tl % LF_BAD_TILES) * LF_BM + row] = !(top < LF_LIMIT);
                tmem_st_wait();
                tc5_fence_before();
                __syncwarp();
                if (lane == 0) { mbar_arrive(wempty0 + 8 * ws); mbar_arrive(full0 + 8 * s); }
            }
        }
    } else if (warp == 10) {
        if (lane == 0) {
            // ---- TMA of the weights (they do not depend on the kernel before this one) ----
            bool ok = true;
            for (int t = first; t < p.num_tiles && ok; t += step) {
                const int n0 = (t / p.num_m) * LF_BM;
                for (int kb = kb0; kb < kb1; ++kb, ++it) {
                    const int ws = it % LF_W_STAGES;
                    if (!mbar_wait_role(wempty0 + 8 * ws, ((it / LF_W_STAGES) & 1) ^ 1, abort_flag, polls)) { ok = false; break; }
                    const unsigned w = smem_u32(base + (size_t)ws * LF_W_BYTES);
                    mbar_expect_tx(wfull0 + 8 * ws, LF_W_BYTES);
                    tma_load_2d(w, &tm_w, wfull0 + 8 * ws, kb * LF_BK, n0);
                    tma_load_2d(w + LF_W_BYTES / 2, &tm_w, wfull0 + 8 * ws, kb * LF_BK + LF_BK / 2, n0);
                }
            }
        }
    } else if (warp == 8) {
        if (lane == 0) {
            // ---- TMA of the tokens' planes ----
            pdl_wait();
            bool ok = true;
            for (int t = first; t < p.num_tiles && ok; t += step) {
                const int m0 = (t % p.num_m) * NT;
                for (int kb = kb0; kb < kb1; ++kb, ++it) {
                    const int s = it % LF_STAGES;
                    if (!mbar_wait_role(empty0 + 8 * s, ((it / LF_STAGES) & 1) ^ 1, abort_flag, polls)) { ok = false; break; }
                    const unsigned b = smem_u32(tok_mem + (size_t)s * Cfg::STAGE_BYTES);
                    mbar_expect_tx(full0 + 8 * s, 3 * Cfg::B_PLANE);
#pragma unroll
                    for (int i = 0; i < 3; ++i)          // (rows behind the last token are the next plane's, or zeros: never stored)
                        tma_load_2d(b + i * Cfg::B_PLANE, &tm_tok, full0 + 8 * s, kb * LF_BK, i * p.M + m0);
                }
            }
        }
    } else if (warp == 9) {
        if (lane == 0) {
            // ---- MMA issue ----
            const unsigned idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(NT >> 3) << 17) | ((unsigned)(LF_BM >> 4) << 24);
            bool ok = true;
            for (int t = first; t < p.num_tiles && ok; t += step) {
                for (int kb = kb0; kb < kb1; ++kb, ++it) {
                    const int s = it % LF_STAGES, buf = it & 1;
                    if (!mbar_wait_role(accempty0 + 8 * buf, ((it >> 1) & 1) ^ 1, abort_flag, polls) ||
                        !mbar_wait_role(full0 + 8 * s, (it / LF_STAGES) & 1, abort_flag, polls)) { ok = false; break; }
                    tc5_fence_after();
                    const unsigned a = tmem_base + LF_A_COL0 + (unsigned)(s * 3 * LF_A_COLS), b = smem_u32(tok_mem + (size_t)s * Cfg::STAGE_BYTES);
                    const unsigned d = tmem_base + (unsigned)(buf * NT);
                    // smallest products first
                    constexpr int PA[6] = {0, 1, 2, 0, 1, 0}, PB[6] = {2, 1, 0, 1, 0, 0};
#pragma unroll
                    for (int q = 0; q < 6; ++q)
#pragma unroll
                        for (int k = 0; k < LF_BK / 16; ++k)
                            lf_umma_ts(d, a + (unsigned)(PA[q] * LF_A_COLS + k * 8), umma_desc(b + PB[q] * Cfg::B_PLANE + k * 32), idesc, (q > 0 || k > 0) ? 1u : 0u);
                    umma_commit(empty0 + 8 * s);
                    umma_commit(accfull0 + 8 * buf);
                }
            }
        }
    } else {
        // ---- epilogue: this thread's weight row, NT tokens ----
        pdl_wait();                                      // the tokens' flags; the output may still be read by what ran before
        const unsigned lanes = tmem_base + ((unsigned)(warp * 32) << 16);
        float acc[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) acc[j] = 0.f;
        int tl = 0;
        bool ok = true;
        for (int t = first; t < p.num_tiles && ok; t += step, ++tl) {
            for (int kb = kb0; kb < kb1; ++kb, ++it) {
                const int buf = it & 1;
                if (!mbar_wait_role(accfull0 + 8 * buf, (it >> 1) & 1, abort_flag, polls)) ok = false;
                if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
                tc5_fence_after();
#pragma unroll
                for (int c = 0; c < NT; c += 16) {       // (sixteen at a time: more would not fit beside the accumulators)
                    float r[16];
                    tmem_ld16(lanes + (unsigned)(buf * NT + c), r);
#pragma unroll
                    for (int j = 0; j < 16; ++j) acc[c + j] += r[j];
                }
                tc5_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(accempty0 + 8 * buf);
            }
            if (!ok) break;
            if (split > 1) {                             // (one tile a cluster, finished below; the stages have been read: the last accumulator is here)
#pragma unroll
                for (int j = 0; j < NT; ++j) part[j * LF_BM + threadIdx.x] = acc[j];
                break;
            }
            const int m0 = (t % p.num_m) * NT;
            const long long n = (long long)(t / p.num_m) * LF_BM + warp * 32 + lane;
            const bool wb = w_bad[(tl % LF_BAD_TILES) * LF_BM + warp * 32 + lane] != 0;
            const float b = (p.bias && n < p.N) ? p.bias[n] : 0.f;
            unsigned odd[NT / 32];
#pragma unroll
            for (int c = 0; c < NT / 32; ++c) odd[c] = 0u;
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                if (n < p.N && m0 + j < p.M) p.out[(size_t)(m0 + j) * p.out_stride + n] = acc[j] + b;
                if (!lf_finite(acc[j])) odd[j / 32] |= 1u << (j % 32);
                acc[j] = 0.f;
            }
#pragma unroll
            for (int c = 0; c < NT; c += 32) {           // (rare) what could not be split, over what was just written
                const unsigned tb = __ballot_sync(0xffffffffu, m0 + c + lane < p.M && p.tok_bad[m0 + c + lane] != 0);
                const unsigned again = wb ? 0xffffffffu : (tb | odd[c / 32]);
                if (n >= p.N || again == 0u) continue;
#pragma unroll 1
                for (int j = 0; j < 32 && m0 + c + j < p.M; ++j)
                    if (again >> j & 1)
                        p.out[(size_t)(m0 + c + j) * p.out_stride + n] = lf_plain(p.act + (size_t)(m0 + c + j) * p.K, p.W + (size_t)n * p.K, p.K) + b;
            }
        }
    }

    if (split > 1) {
        // ---- a tile shared by the cluster: partial sums through shared memory, each block finishes NT / split tokens ----
        __syncthreads();
        __syncwarp();
        lf_cluster_sync();
        bool whole = true;                               // (a block that gave up has left no partial sums)
        for (int r = 0; r < split; ++r) {
            unsigned gone;
            asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(gone) : "r"(lf_map_rank(smem_u32(const_cast<int*>(abort_flag)), (unsigned)r)));
            whole &= gone == 0u;
        }
        if (warp < 4 && first < p.num_tiles && whole) {
            const int m0 = (first % p.num_m) * NT;
            const long long n = (long long)(first / p.num_m) * LF_BM + threadIdx.x;
            bool wb = false;
            for (int r = 0; r < split && r * per < p.num_kb; ++r) {     // (a block without a part of K leaves no mark)
                unsigned f;
                asm volatile("ld.shared::cluster.u8 %0, [%1];" : "=r"(f) : "r"(lf_map_rank(smem_u32(w_bad + threadIdx.x), (unsigned)r)));
                wb |= f != 0;
            }
            const float b = (p.bias && n < p.N) ? p.bias[n] : 0.f;
            // (a load from another block's memory takes about as long as one from L2: eight tokens' at a time, of two ranks before they are
            // added.  One by one, with the sum between them, they were 13 to 26 us of a call: 65 x 2,048 x 512 34 us, so 19, 300 x 1,536 x 1,536
            // 53 and 39, 129 x 1,024 x 1,024 24 and 17)
            const int cols = NT / split;                 // (at least eight)
            for (int j = rank * cols; j < (rank + 1) * cols && m0 + j < p.M; j += 8) {
                float y[8];
                int tb[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) { y[i] = 0.f; tb[i] = m0 + j + i < p.M ? p.tok_bad[m0 + j + i] : 0; }
#pragma unroll 2
                for (int r = 0; r < split; ++r) {
                    const unsigned src = lf_map_rank(smem_u32(part + j * LF_BM + threadIdx.x), (unsigned)r);
                    float f[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(f[i]) : "r"(src + i * LF_BM * 4));
#pragma unroll
                    for (int i = 0; i < 8; ++i) y[i] += f[i];
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int m = m0 + j + i;
                    if (n < p.N && m < p.M) {
                        if (wb || tb[i] != 0 || !lf_finite(y[i])) y[i] = lf_plain(p.act + (size_t)m * p.K, p.W + (size_t)n * p.K, p.K);
                        p.out[(size_t)m * p.out_stride + n] = y[i] + b;
                    }
                }
            }
        }
        __syncwarp();
        lf_cluster_sync();                               // nobody reads this block's shared memory any more
    }
    tc5_fence_before();
    __syncthreads();
    if (*abort_flag) {                                   // (the same for all: every role is through)
        if (threadIdx.x == 0 && p.status) atomicExch(p.status, 16);
        if (threadIdx.x == 8 * 32) abort_flag[1] = it;
        __syncthreads();
        if (lane == 0) {                                 // what is under way ends before its memory is given back
            if (warp >= 4 && warp < 8)                   // (a tokens' stage is full when these warps have arrived too)
                for (int i = it; i < abort_flag[1]; ++i) mbar_arrive(full0 + 8 * (i % LF_STAGES));
            if (warp == 8)
                for (int i = max(it - LF_STAGES, 0); i < it; ++i) mbar_wait(full0 + 8 * (i % LF_STAGES), (i / LF_STAGES) & 1);
            if (warp == 10)
                for (int i = max(it - LF_W_STAGES, 0); i < it; ++i) mbar_wait(wfull0 + 8 * (i % LF_W_STAGES), (i / LF_W_STAGES) & 1);
            if (warp == 9 && it > 0) {
                umma_commit(drained);
                mbar_wait(drained, 0);
            }
        }
        __syncthreads();
    }
    if (warp == 9) {
        __syncwarp();
        tc5_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"((unsigned)LF_TMEM_COLS) : "memory");
    }
}

// ---- host side -------------------------------------------------------------------------------
// a [rows][cols] matrix with contiguous rows, boxes of 128 bytes x box_rows rows, 128-byte swizzle
static int lf_encode(CUtensorMap* map, CUtensorMapDataType type, int size, const void* ptr, long long rows, long long cols, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(-102, "linear_f32: cuTensorMapEncodeTiled is not available from the driver");
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * size};
    cuuint32_t box[2] = {(cuuint32_t)(128 / size), (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, type, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : fail(-103, "linear_f32: cuTensorMapEncodeTiled failed with %d", (int)r);
}

template <int NT, bool TRIAL>
static int launch_lf(const CUtensorMap& tw, const CUtensorMap& tm, const LfParams& p, cudaStream_t stream) {
    using Cfg = LfCfg<NT>;
    auto kern = linear_f32_kernel<NT, TRIAL>;
    static bool attr_done = false;
    if (!attr_done) {
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::SMEM);
        if (e != cudaSuccess) return fail(-101, "linear_f32: cannot reserve %zu bytes of shared memory: %s", Cfg::SMEM, cudaGetErrorString(e));
        attr_done = true;
    }
    int groups = sm_count() / p.split;
    if (p.split > 1 || groups > p.num_tiles) groups = p.num_tiles;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(groups * p.split);
    cfg.blockDim = dim3(LF_THREADS);
    cfg.dynamicSmemBytes = Cfg::SMEM;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    int na = 0;
    if (pdl_enabled()) {
        attr[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[na].val.programmaticStreamSerializationAllowed = 1;
        ++na;
    }
    if (p.split > 1) {
        attr[na].id = cudaLaunchAttributeClusterDimension;
        attr[na].val.clusterDim.x = p.split;
        attr[na].val.clusterDim.y = 1;
        attr[na].val.clusterDim.z = 1;
        ++na;
    }
    cfg.attrs = attr;
    cfg.numAttrs = na;
    return check_launch("linear_f32", cudaLaunchKernelEx(&cfg, kern, tw, tm, p));
}

// How a call is cut: tokens a tile and blocks that share a tile's K.
VAPI_EXPORT int vapi_linear_f32_plan(int N, int K, int M, int* nt, int* split) {
    *nt = M <= 64 ? 64 : 128;
    const int tiles = ((M + *nt - 1) / *nt) * ((N + LF_BM - 1) / LF_BM), num_kb = (K + LF_BK - 1) / LF_BK;
    int s = 1;
    while (s < 8 && tiles * s * 2 <= sm_count() && num_kb >= s * 2 * 4) s *= 2;
    *split = s;
    return 0;
}

// y = act W^T (+ bias).  ``planes``: scratch of 3 * M * (K rounded up to 8) bfloat16; ``bad``: scratch of M ints.
// ``polls``: of an mbarrier before a role gives up, below zero for the usual limit (about a second).
VAPI_EXPORT int vapi_linear_f32(const float* W, int N, int K, int M, const float* act, void* planes, int* bad, const float* bias,
                                float* out, long long out_stride, int polls, int* status, cudaStream_t stream) {
    if (M <= 0) return 0;
    if (N <= 0 || K <= 0 || K % 4 != 0) return fail(-1, "linear_f32: K=%d must be a positive multiple of 4 (N=%d)", K, N);
    if (!W || !act || !planes || !bad || !out) return fail(-1, "linear_f32: missing array");
    if ((((uintptr_t)W | (uintptr_t)act | (uintptr_t)planes) & 15) != 0) return fail(-1, "linear_f32: operands must be 16-byte aligned");
    const int Kp = (K + 7) & ~7;
    int rc = check_launch("linear_f32: split", launch(split_rows_kernel, dim3(M), dim3(256), 0, stream, act, (__nv_bfloat16*)planes, bad, M, K, Kp));
    if (rc) return rc;
    LfParams p;
    int nt;
    vapi_linear_f32_plan(N, K, M, &nt, &p.split);
    p.W = W; p.act = act; p.bias = bias; p.tok_bad = bad; p.out = out; p.status = status;
    p.N = N; p.K = K; p.M = M; p.out_stride = out_stride; p.polls = polls < 0 ? 0u : (unsigned)polls;
    p.num_kb = (K + LF_BK - 1) / LF_BK;
    p.num_m = (M + nt - 1) / nt;
    p.num_tiles = p.num_m * ((N + LF_BM - 1) / LF_BM);
    CUtensorMap tw, tm;
    rc = lf_encode(&tw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, W, N, K, LF_BM);
    if (rc == 0) rc = lf_encode(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, planes, 3LL * M, Kp, nt);
    if (rc) return rc;
    if (polls >= 0) return nt == 64 ? launch_lf<64, true>(tw, tm, p, stream) : launch_lf<128, true>(tw, tm, p, stream);
    return nt == 64 ? launch_lf<64, false>(tw, tm, p, stream) : launch_lf<128, false>(tw, tm, p, stream);
}

VAPI_EXPORT const char* vapi_last_error() { return error_buffer(); }
