// The gated delta rule and the state-space recurrence of recurrent.cu, 64 tokens at a time on the tensor cores, for
// sequences that bring many tokens (bfloat16 inputs, states of 128 rows).  Same equations, same states, and what is float
// there is float here: whatever is not bfloat16 to begin with (the state, decayed scores, decayed inputs, the solved
// writes) enters a product as the sum of three bfloat16 numbers, which is all 24 bits of it (x1 = bf16(x), x2 = bf16(x - x1),
// x3 = the rest), against an operand that is bfloat16 exactly; where both sides are float, the six products of weight 2^-16
// and above are taken.  Accumulators are float, and short: a tensor core cuts what it adds to an accumulator off where a
// float FMA rounds, so the planes below the first have accumulators of their own, the first plane's sums over 128
// rows are halves in two accumulators, and what a chunk adds to the state is summed apart and added to it by an FMA.  Sums of decay logarithms inside a chunk are formed in double and kept as
// two floats, so that their differences have a float's relative accuracy however long the chunk's decay is.
//
// Why chunks.  Token by token, a sequence is a chain of dependent steps of ~0.31 us on a fraction of the chip (2,000 tokens: 0.63
// and 0.70 ms a layer, issue slots a quarter used, no bandwidth).  With t, s counted inside a chunk, l_t the sum of the decay
// logarithms up to and with t, and S the state before the chunk:
//
//   state space   y_t = e^{l_t} C_t.S + sum_{s<=t} e^{l_t-l_s} step_s (C_t.B_s) x_s + D x_t
//                 S'  = e^{l_L} S + sum_s B_s (e^{l_L-l_s} step_s x_s)^T
//   delta rule    (I + A) U = R,  A_ts = beta_t e^{l_t-l_s} (k_t.k_s) for s < t,  R_t = beta_t (v_t - e^{l_t} k_t.S)
//                 o_t = e^{l_t} q_t.S + sum_{s<=t} e^{l_t-l_s} (q_t.k_s) u_s
//                 S'  = e^{l_L} S + sum_s k_s (e^{l_L-l_s} u_s)^T
//
// so that the chain has an entry per chunk instead of per token, and what lies between is matrix products.  Columns of S are
// independent of each other: a block owns a head and 32 (state space) or 16 (delta rule) of them, which gives 128 blocks for
// one sequence of either recurrence at the widths this is for.  T = (I + A)^-1 and the scores do not depend on the state: a
// kernel before the walk works them out for all chunks at once (its own substitution, in float) and leaves them as
// bfloat16 planes in scratch memory.  One sequence of 2,000 tokens: state space (64 heads of 64) 701 -> 167 us, delta rule (16
// heads of 128) 624 -> 152 us with the kernel before it; of 300 tokens 110 -> 30 and 97 -> 33 us.  Against float64 neither is
// further off than the walk (1.0e-7 to 1.7e-7 of the outputs' 2-norm against 1.1e-7 to 1.9e-7).  What bounds it now is the chain
// of a chunk's matrix products and barriers, ~5 us a chunk.
//
// Every sequence of a step takes the walk of recurrent.cu or the chunks by its own number of tokens alone.
#include "common.cuh"
#include "attention_mma.cuh"       // ldmatrix_x4, ldmatrix_x4_trans, mma_bf16_16816, cp_async_16

using namespace vapi;

constexpr int RC_T = 64;           // tokens of a chunk
constexpr int RC_ROWS = 128;       // rows of a state
// Sequences with fewer tokens in the step are walked.  One chunk takes 8.8 us (state space, 64 heads) and 18 us (delta rule, 16 heads,
// both kernels), the walk 8.7 us at 16 tokens and 14.6 at 32 of the one, 12.4 at 32, 17.4 at 48 and 22.6 at 64 of the other.
constexpr int RC_SS_MIN = 20, RC_GD_MIN = 48;
constexpr int RC_THREADS = 256;
// shared rows end 16 bytes further than their data: ldmatrix without bank conflicts
constexpr int RC_LD = RC_ROWS + 8;
constexpr int RC_SS_COLS = 32, RC_SS_XLD = RC_SS_COLS + 8;
constexpr int RC_GD_COLS = 16, RC_GD_CLD = RC_GD_COLS + 8, RC_TLD = RC_T + 8;

__device__ __forceinline__ float rc_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }
// what is left of x beside its bfloat16 part; nothing where that part is not finite
__device__ __forceinline__ float rc_rest(float x, unsigned bits) {
    const float p = __uint_as_float(bits);
    return (bits & 0x7f800000u) == 0x7f800000u ? 0.f : x - p;
}
// two floats as three pairs of bfloat16 that add up to them
__device__ __forceinline__ void rc_split(float a, float b, unsigned& p1, unsigned& p2, unsigned& p3) {
    p1 = pack_bf16(a, b);
    a = rc_rest(a, p1 << 16);
    b = rc_rest(b, p1 & 0xffff0000u);
    p2 = pack_bf16(a, b);
    a = rc_rest(a, p2 << 16);
    b = rc_rest(b, p2 & 0xffff0000u);
    p3 = pack_bf16(a, b);
}
template <int N> __device__ __forceinline__ void rc_zero(float (&t)[N][4]) {
#pragma unroll
    for (int i = 0; i < N; ++i) t[i][0] = t[i][1] = t[i][2] = t[i][3] = 0.f;
}
// fragments from a row-major matrix in shared memory (ld elements a row), 16 x 16 at (row, col):
// operand A (m16 x k16) with k along the row
__device__ __forceinline__ void rc_a(unsigned (&a)[4], const __nv_bfloat16* m, int ld, int row, int col) {
    const int lane = threadIdx.x & 31;
    ldmatrix_x4(a[0], a[1], a[2], a[3], m + (row + (lane & 15)) * ld + col + (lane >> 4) * 8);
}
// operand A with m along the row and k down the column
__device__ __forceinline__ void rc_a_trans(unsigned (&a)[4], const __nv_bfloat16* m, int ld, int k, int mcol) {
    const int lane = threadIdx.x & 31, mat = lane >> 3, r = lane & 7;
    ldmatrix_x4_trans(a[0], a[1], a[2], a[3], m + (k + (mat >> 1) * 8 + r) * ld + mcol + (mat & 1) * 8);
}
// operand B (k16 x n16: b[0..1] the first eight n, b[2..3] the next) with k along the row
__device__ __forceinline__ void rc_b(unsigned (&b)[4], const __nv_bfloat16* m, int ld, int n, int k) {
    const int lane = threadIdx.x & 31, mat = lane >> 3, r = lane & 7;
    ldmatrix_x4(b[0], b[1], b[2], b[3], m + (n + (mat >> 1) * 8 + r) * ld + k + (mat & 1) * 8);
}
// operand B with n along the row and k down the column
__device__ __forceinline__ void rc_b_trans(unsigned (&b)[4], const __nv_bfloat16* m, int ld, int k, int n) {
    const int lane = threadIdx.x & 31, mat = lane >> 3, r = lane & 7;
    ldmatrix_x4_trans(b[0], b[1], b[2], b[3], m + (k + (mat & 1) * 8 + r) * ld + n + (mat >> 1) * 8);
}
// 64 rows of `pieces` 16-byte pieces from global memory (rows of `stride` elements), zeros behind `count` rows
__device__ __forceinline__ void rc_rows(__nv_bfloat16* dst, int ld, const __nv_bfloat16* src, long long stride, int count, int pieces, int tid, int threads) {
    for (int i = tid; i < RC_T * pieces; i += threads) {
        const int r = i / pieces, c = i - r * pieces;
        cp_async_16(dst + r * ld + c * 8, src + (size_t)(r < count ? r : 0) * stride + c * 8, r < count ? 16 : 0);
    }
}
// One warp: sums of the decay logarithms of a chunk's tokens 2 lane and 2 lane + 1, and of the whole chunk
__device__ __forceinline__ void rc_scan(float a0, float a1, double& l0, double& l1, double& all) {
    const int lane = threadIdx.x & 31;
    // (a decay of e^-10000 is zero as much as any beyond it, and differences of sums stay finite)
    a0 = a0 < -1e4f ? -1e4f : a0;
    a1 = a1 < -1e4f ? -1e4f : a1;
    double run = (double)a0 + (double)a1;
    const double own = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
    }
    all = __shfl_sync(0xffffffffu, run, 31);
    l1 = run;
    l0 = run - own + (double)a0;
}

// ---- state space ----------------------------------------------------------------------------------------
struct RcSsSmem {
    __nv_bfloat16 B[2][RC_T][RC_LD], C[2][RC_T][RC_LD];
    __nv_bfloat16 X[2][RC_T][RC_SS_XLD];
    __nv_bfloat16 S[2][3][RC_SS_COLS][RC_LD];              // the state's planes, a column a row
    float hi[2][RC_T], lo[2][RC_T], step[2][RC_T];         // l_t as two floats, the step size
    float w[2][RC_T], e[2][RC_T], last[2];                 // e^{l_L - l_t} step_t, e^{l_t}, e^{l_L}
};

// Warps 0..3 compute the outputs of 16 tokens each, warps 4..7 move 32 rows of the state on each; the two halves need
// nothing of one another inside a chunk (the state's planes are double-buffered), so a chunk has one barrier.
__global__ void __launch_bounds__(RC_THREADS, 1)
state_space_chunks_kernel(const __nv_bfloat16* __restrict__ xbc, long long xbc_stride, const __nv_bfloat16* __restrict__ dt, long long dt_stride,
                          const float* __restrict__ A_log, const float* __restrict__ dt_bias, const float* __restrict__ D,
                          float* __restrict__ state, long long slot_stride, const int* __restrict__ state_slots,
                          const int* __restrict__ cu_q, const int* __restrict__ positions, float* __restrict__ out, int nh,
                          int groups, int cols, int num_slots, int least, int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char rc_smem[];
    RcSsSmem& sm = *reinterpret_cast<RcSsSmem*>(rc_smem);
    const int s = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * RC_SS_COLS;
    const int t0 = cu_q[s], qlen = cu_q[s + 1] - t0;
    if (qlen < least) return;
    const int slot = state_slots[s];
    if (slot < 0 || slot >= num_slots) {
        if (threadIdx.x == 0 && status) atomicExch(status, 3);
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g4 = lane >> 2, p4 = (lane & 3) * 2;
    const int g = h / (nh / groups);
    const float rate = expf(A_log[h]), bias = dt_bias[h], skip = D[h];
    const __nv_bfloat16* xs = xbc + (size_t)t0 * xbc_stride + (size_t)h * cols + col0;
    const __nv_bfloat16* Bs = xbc + (size_t)t0 * xbc_stride + (size_t)nh * cols + (size_t)g * RC_ROWS;
    const __nv_bfloat16* Cs = Bs + (size_t)groups * RC_ROWS;
    float* S_glob = state + (size_t)slot * slot_stride + (size_t)h * RC_ROWS * cols + col0;
    const bool fresh = positions[t0] == 0;
    const int chunks = (qlen + RC_T - 1) / RC_T;
    pdl_wait();

    auto load = [&](int c) {
        const int buf = c & 1, count = min(RC_T, qlen - c * RC_T);
        const size_t off = (size_t)c * RC_T * xbc_stride;
        rc_rows(&sm.B[buf][0][0], RC_LD, Bs + off, xbc_stride, count, RC_ROWS / 8, tid, RC_THREADS);
        rc_rows(&sm.C[buf][0][0], RC_LD, Cs + off, xbc_stride, count, RC_ROWS / 8, tid, RC_THREADS);
        rc_rows(&sm.X[buf][0][0], RC_SS_XLD, xs + off, xbc_stride, count, RC_SS_COLS / 8, tid, RC_THREADS);
        cp_async_commit();
        if (warp == 4) {
            float st[2], a[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = c * RC_T + 2 * lane + i;
                st[i] = t < qlen ? rc_softplus(to_f32(dt[(size_t)(t0 + t) * dt_stride + h]) + bias) : 0.f;
                a[i] = t < qlen ? -rate * st[i] : 0.f;
            }
            double l[2], all;
            rc_scan(a[0], a[1], l[0], l[1], all);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int t = 2 * lane + i;
                const float hi = (float)l[i];
                sm.hi[buf][t] = hi;
                sm.lo[buf][t] = (float)(l[i] - (double)hi);
                sm.step[buf][t] = st[i];
                sm.w[buf][t] = expf((float)(all - l[i])) * st[i];
                sm.e[buf][t] = expf(hi);
            }
            if (lane == 0) sm.last[buf] = expf((float)all);
        }
    };

    // state warps: S^T, rows = columns of the state (two tiles of 16), 32 rows of it (four tiles of 8)
    const int r0 = (warp & 3) * 32;
    float acc[2][4][4];
    auto publish = [&](int buf) {                          // the state's planes for the outputs of the next chunk
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    unsigned p1, p2, p3;
                    rc_split(acc[m][n][2 * q], acc[m][n][2 * q + 1], p1, p2, p3);
                    const int c = m * 16 + q * 8 + g4, r = r0 + n * 8 + p4;
                    *reinterpret_cast<unsigned*>(&sm.S[buf][0][c][r]) = p1;
                    *reinterpret_cast<unsigned*>(&sm.S[buf][1][c][r]) = p2;
                    *reinterpret_cast<unsigned*>(&sm.S[buf][2][c][r]) = p3;
                }
    };
    load(0);
    if (warp >= 4) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int c = m * 16 + (i >> 1) * 8 + g4, r = r0 + n * 8 + p4 + (i & 1);
                    acc[m][n][i] = fresh ? 0.f : S_glob[(size_t)r * cols + c];
                }
        publish(0);
    }

    for (int c = 0; c < chunks; ++c) {
        const int buf = c & 1;
        cp_async_wait<0>();
        __syncthreads();                                   // this chunk's rows, scalars and state planes are in place; the other buffers are free
        if (c + 1 < chunks) load(c + 1);
        if (warp < 4) {
            // ---- outputs of tokens 16 warp .. 16 warp + 15 ----
            const int m0 = warp * 16;
            float cb[2][8][4], y[2][4][4], low[4][4];       // [k even | odd], first plane; the other planes
            rc_zero(cb[0]); rc_zero(cb[1]); rc_zero(y[0]); rc_zero(y[1]); rc_zero(low);
#pragma unroll
            for (int k = 0; k < RC_ROWS / 16; ++k) {
                unsigned a[4], b[4];
                rc_a(a, &sm.C[buf][0][0], RC_LD, m0, k * 16);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j <= warp) {
                        rc_b(b, &sm.B[buf][0][0], RC_LD, j * 16, k * 16);
                        mma_bf16_16816(cb[k & 1][2 * j], a, b[0], b[1]);
                        mma_bf16_16816(cb[k & 1][2 * j + 1], a, b[2], b[3]);
                    }
#pragma unroll
                for (int pl = 2; pl >= 0; --pl)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        rc_b(b, &sm.S[buf][pl][0][0], RC_LD, q * 16, k * 16);
                        mma_bf16_16816(pl ? low[2 * q] : y[k & 1][2 * q], a, b[0], b[1]);
                        mma_bf16_16816(pl ? low[2 * q + 1] : y[k & 1][2 * q + 1], a, b[2], b[3]);
                    }
            }
            const int ta = m0 + g4, tb = ta + 8;           // this lane's two tokens
            const float ea = sm.e[buf][ta], eb = sm.e[buf][tb];
            const float ha = sm.hi[buf][ta], hb = sm.hi[buf][tb], la = sm.lo[buf][ta], lb = sm.lo[buf][tb];
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    y[1][n][i] = ((y[0][n][i] + y[1][n][i]) + low[n][i]) * (i < 2 ? ea : eb);       // what the state gives
                    y[0][n][i] = low[n][i] = 0.f;                                                   // what this chunk's tokens give
                }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (j <= warp) {
                    unsigned a[3][4];
#pragma unroll
                    for (int i = 0; i < 2; ++i) {          // decayed scores of eight tokens s
                        const int sx = j * 16 + i * 8 + p4;
                        const float2 hs = *reinterpret_cast<const float2*>(&sm.hi[buf][sx]), ls = *reinterpret_cast<const float2*>(&sm.lo[buf][sx]);
                        const float2 st = *reinterpret_cast<const float2*>(&sm.step[buf][sx]);
                        const float v[4] = {cb[0][2 * j + i][0] + cb[1][2 * j + i][0], cb[0][2 * j + i][1] + cb[1][2 * j + i][1],
                                            cb[0][2 * j + i][2] + cb[1][2 * j + i][2], cb[0][2 * j + i][3] + cb[1][2 * j + i][3]};
                        const float w0 = sx <= ta ? v[0] * (st.x * expf((ha - hs.x) + (la - ls.x))) : 0.f;
                        const float w1 = sx + 1 <= ta ? v[1] * (st.y * expf((ha - hs.y) + (la - ls.y))) : 0.f;
                        const float w2 = sx <= tb ? v[2] * (st.x * expf((hb - hs.x) + (lb - ls.x))) : 0.f;
                        const float w3 = sx + 1 <= tb ? v[3] * (st.y * expf((hb - hs.y) + (lb - ls.y))) : 0.f;
                        rc_split(w0, w1, a[0][2 * i], a[1][2 * i], a[2][2 * i]);
                        rc_split(w2, w3, a[0][2 * i + 1], a[1][2 * i + 1], a[2][2 * i + 1]);
                    }
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        unsigned b[4];
                        rc_b_trans(b, &sm.X[buf][0][0], RC_SS_XLD, j * 16, q * 16);
#pragma unroll
                        for (int pl = 2; pl >= 0; --pl) {
                            mma_bf16_16816(pl ? low[2 * q] : y[0][2 * q], a[pl], b[0], b[1]);
                            mma_bf16_16816(pl ? low[2 * q + 1] : y[0][2 * q + 1], a[pl], b[2], b[3]);
                        }
                    }
                }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int t = q ? tb : ta, at = c * RC_T + t;
                    if (at < qlen) {
                        const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&sm.X[buf][t][n * 8 + p4]));
                        *reinterpret_cast<float2*>(out + ((size_t)(t0 + at) * nh + h) * cols + col0 + n * 8 + p4) =
                            make_float2(fmaf(skip, x.x, (y[0][n][2 * q] + low[n][2 * q]) + y[1][n][2 * q]),
                                        fmaf(skip, x.y, (y[0][n][2 * q + 1] + low[n][2 * q + 1]) + y[1][n][2 * q + 1]));
                    }
                }
        } else {
            // ---- the state: rows r0 .. r0 + 31 ----
            const float last = sm.last[buf];
            float add[2][4][4], low[2][4][4];
            rc_zero(add[0]); rc_zero(add[1]); rc_zero(low[0]); rc_zero(low[1]);
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) {
                unsigned b[2][4];
#pragma unroll
                for (int q = 0; q < 2; ++q) rc_b_trans(b[q], &sm.B[buf][0][0], RC_LD, kt * 16, r0 + q * 16);
                const float2 wl = *reinterpret_cast<const float2*>(&sm.w[buf][kt * 16 + p4]), wh = *reinterpret_cast<const float2*>(&sm.w[buf][kt * 16 + 8 + p4]);
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    unsigned x[4], a[3][4];
                    rc_a_trans(x, &sm.X[buf][0][0], RC_SS_XLD, kt * 16, m * 16);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {          // x_s times its weight; words 0, 1: the first eight tokens
                        const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&x[i]));
                        const float2 w = i < 2 ? wl : wh;
                        rc_split(f.x * w.x, f.y * w.y, a[0][i], a[1][i], a[2][i]);
                    }
#pragma unroll
                    for (int pl = 2; pl >= 0; --pl)
#pragma unroll
                        for (int q = 0; q < 2; ++q) {
                            mma_bf16_16816(pl ? low[m][2 * q] : add[m][2 * q], a[pl], b[q][0], b[q][1]);
                            mma_bf16_16816(pl ? low[m][2 * q + 1] : add[m][2 * q + 1], a[pl], b[q][2], b[q][3]);
                        }
                }
            }
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[m][n][i] = fmaf(last, acc[m][n][i], add[m][n][i] + low[m][n][i]);
            publish(buf ^ 1);
        }
    }
    pdl_trigger();
    if (warp >= 4) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    S_glob[(size_t)(r0 + n * 8 + p4 + (i & 1)) * cols + m * 16 + (i >> 1) * 8 + g4] = acc[m][n][i];
    }
}

// ---- delta rule -----------------------------------------------------------------------------------------
// what the first kernel leaves of a (chunk, head): T and the decayed scores P as planes [3][64][64], and per token
// beta, beta e^{l_t} / |k|, e^{l_t} / |q|, e^{l_L - l_t} / |k|, and e^{l_L} (64 times)
struct RcPrepared {
    __nv_bfloat16 T[3][RC_T][RC_T], P[3][RC_T][RC_T];
    float scal[5][RC_T];
};

// chunks of the sequences before s
__device__ __forceinline__ int rc_chunks_before(const int* cu_q, int s, int least) {
    int n = 0;
    for (int i = threadIdx.x & 31; i < s; i += 32) {
        const int q = cu_q[i + 1] - cu_q[i];
        n += q >= least ? (q + RC_T - 1) / RC_T : 0;
    }
    return __reduce_add_sync(0xffffffffu, n);
}

__global__ void __launch_bounds__(128)
delta_prepare_kernel(const __nv_bfloat16* __restrict__ qkv, long long qkv_stride, int q_off, int k_off, const __nv_bfloat16* __restrict__ ab,
                     long long ab_stride, const float* __restrict__ A_log, const float* __restrict__ dt_bias,
                     const int* __restrict__ cu_q, RcPrepared* __restrict__ prep, int num_seqs, int nh, int nkv, float norm_eps, int least) {
    __shared__ __align__(16) __nv_bfloat16 sK[RC_T][RC_LD], sQ[RC_T][RC_LD];
    static_assert(sizeof(sQ) >= sizeof(float) * RC_T * (RC_T + 4), "A takes the queries' place, T the keys'");
    float (*sA)[RC_T + 4] = reinterpret_cast<float (*)[RC_T + 4]>(&sQ[0][0]), (*sT)[RC_T + 4] = reinterpret_cast<float (*)[RC_T + 4]>(&sK[0][0]);
    __shared__ float hi[RC_T], lo[RC_T], beta[RC_T], kinv[RC_T], qinv[RC_T];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g4 = lane >> 2, p4 = (lane & 3) * 2;
    const int h = blockIdx.y, g = h / (nh / nkv);
    // which sequence's chunk this is
    int s = 0, c = (int)blockIdx.x;
    for (; s < num_seqs; ++s) {
        const int q = cu_q[s + 1] - cu_q[s], n = q >= least ? (q + RC_T - 1) / RC_T : 0;
        if (c < n) break;
        c -= n;
    }
    if (s >= num_seqs) return;
    const int t0 = cu_q[s] + c * RC_T, count = min(RC_T, cu_q[s + 1] - t0);
    RcPrepared* P = prep + (size_t)blockIdx.x * nh + h;
    pdl_wait();
    rc_rows(&sK[0][0], RC_LD, qkv + (size_t)t0 * qkv_stride + k_off + g * RC_ROWS, qkv_stride, count, RC_ROWS / 8, tid, 128);
    rc_rows(&sQ[0][0], RC_LD, qkv + (size_t)t0 * qkv_stride + q_off + g * RC_ROWS, qkv_stride, count, RC_ROWS / 8, tid, 128);
    cp_async_commit();
    double l[2] = {0., 0.}, all = 0.;
    if (warp == 0) {
        const float rate = expf(A_log[h]), bias = dt_bias[h];
        float a[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = 2 * lane + i;
            const __nv_bfloat16* row = ab + (size_t)(t0 + (t < count ? t : 0)) * ab_stride;
            a[i] = t < count ? -rate * rc_softplus(to_f32(row[h]) + bias) : 0.f;
            beta[t] = t < count ? 1.f / (1.f + expf(-to_f32(row[nh + h]))) : 0.f;
        }
        rc_scan(a[0], a[1], l[0], l[1], all);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            hi[2 * lane + i] = (float)l[i];
            lo[2 * lane + i] = (float)(l[i] - (double)(float)l[i]);
        }
    }
    cp_async_wait<0>();
    __syncthreads();
    {
        const int t = tid >> 1, half = (tid & 1) * 64;
        float kk = 0.f, qq = 0.f;
#pragma unroll 8
        for (int r = 0; r < 64; r += 2) {
            const float2 k = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&sK[t][half + r]));
            const float2 q = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&sQ[t][half + r]));
            kk = fmaf(k.x, k.x, kk); kk = fmaf(k.y, k.y, kk);
            qq = fmaf(q.x, q.x, qq); qq = fmaf(q.y, q.y, qq);
        }
        kk += __shfl_xor_sync(0xffffffffu, kk, 1);
        qq += __shfl_xor_sync(0xffffffffu, qq, 1);
        if ((tid & 1) == 0) {
            kinv[t] = t < count ? rsqrtf(kk + norm_eps) : 0.f;       // (tokens behind the end write nothing)
            qinv[t] = t < count ? rsqrtf(qq + norm_eps) * rsqrtf((float)RC_ROWS) : 0.f;
        }
    }
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int t = 2 * lane + i;
            const float e = expf(hi[t]);
            P->scal[0][t] = beta[t];
            P->scal[1][t] = beta[t] * e * kinv[t];
            P->scal[2][t] = e * qinv[t];
            P->scal[3][t] = expf((float)(all - l[i])) * kinv[t];
            P->scal[4][t] = expf((float)all);
        }
    }
    // scores of 16 tokens a warp against the tokens up to them
    float kk[2][8][4], qk[2][8][4];                        // [k even | odd]
    rc_zero(kk[0]); rc_zero(kk[1]); rc_zero(qk[0]); rc_zero(qk[1]);
#pragma unroll
    for (int k = 0; k < RC_ROWS / 16; ++k) {
        unsigned ak[4], aq[4], b[4];
        rc_a(ak, &sK[0][0], RC_LD, warp * 16, k * 16);
        rc_a(aq, &sQ[0][0], RC_LD, warp * 16, k * 16);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (j <= warp) {
                rc_b(b, &sK[0][0], RC_LD, j * 16, k * 16);
                mma_bf16_16816(kk[k & 1][2 * j], ak, b[0], b[1]);
                mma_bf16_16816(kk[k & 1][2 * j + 1], ak, b[2], b[3]);
                mma_bf16_16816(qk[k & 1][2 * j], aq, b[0], b[1]);
                mma_bf16_16816(qk[k & 1][2 * j + 1], aq, b[2], b[3]);
            }
    }
    __syncthreads();                                       // keys and queries have been read
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int t = warp * 16 + q * 8 + g4, sx = i * 8 + p4;
            float av[2] = {0.f, 0.f}, pv[2] = {0.f, 0.f};
            if (i / 2 <= warp) {
#pragma unroll
                for (int x = 0; x < 2; ++x)
                    if (sx + x <= t) {
                        const float d = expf((hi[t] - hi[sx + x]) + (lo[t] - lo[sx + x])) * kinv[sx + x];
                        pv[x] = (qk[0][i][2 * q + x] + qk[1][i][2 * q + x]) * (d * qinv[t]);
                        if (sx + x < t) av[x] = (kk[0][i][2 * q + x] + kk[1][i][2 * q + x]) * (d * kinv[t] * beta[t]);
                    }
                unsigned p1, p2, p3;
                rc_split(pv[0], pv[1], p1, p2, p3);
                *reinterpret_cast<unsigned*>(&P->P[0][t][sx]) = p1;
                *reinterpret_cast<unsigned*>(&P->P[1][t][sx]) = p2;
                *reinterpret_cast<unsigned*>(&P->P[2][t][sx]) = p3;
            }
            *reinterpret_cast<float2*>(&sA[t][sx]) = make_float2(av[0], av[1]);
        }
    }
    __syncthreads();
    // T = (I + A)^-1 in float: the four blocks of 16 on the diagonal by substitution, a column a thread, then twice
    // T21 = -T22 (A21 T11), with A21 T11 in the place of T12.  (One substitution over 64, a column a thread, is a chain four times
    // as long: 25 us for this kernel and one chunk against the rest of it in 9.)
    if (tid < RC_T) {
        const int d0 = tid & ~15, j = tid & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float sum[4] = {i == j ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int m = 0; m < i; m += 4) {
                const float4 a = *reinterpret_cast<const float4*>(&sA[d0 + i][d0 + m]);
                sum[0] = fmaf(-a.x, x[m], sum[0]);
                if (m + 1 < i) sum[1] = fmaf(-a.y, x[m + 1], sum[1]);
                if (m + 2 < i) sum[2] = fmaf(-a.z, x[m + 2], sum[2]);
                if (m + 3 < i) sum[3] = fmaf(-a.w, x[m + 3], sum[3]);
            }
            x[i] = (sum[0] + sum[1]) + (sum[2] + sum[3]);
            sT[d0 + i][d0 + j] = x[i];
        }
    }
    __syncthreads();
    // out (rows i, four columns from j on) = sign * L (rows) R (columns), `size` long
    auto product = [&](float* out, const float* L, const float* R, int size, float sign) {
        constexpr int LD = RC_T + 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int m = 0; m < size; ++m) {
            const float l = L[m];
            const float4 r = *reinterpret_cast<const float4*>(R + m * LD);
            acc.x = fmaf(l, r.x, acc.x); acc.y = fmaf(l, r.y, acc.y); acc.z = fmaf(l, r.z, acc.z); acc.w = fmaf(l, r.w, acc.w);
        }
        *reinterpret_cast<float4*>(out) = make_float4(sign * acc.x, sign * acc.y, sign * acc.z, sign * acc.w);
    };
    {
        const int d0 = (tid >> 6) * 32, i = (tid & 63) >> 2, j = (tid & 3) * 4;
        product(&sT[d0 + i][d0 + 16 + j], &sA[d0 + 16 + i][d0], &sT[d0][d0 + j], 16, 1.f);
        __syncthreads();
        product(&sT[d0 + 16 + i][d0 + j], &sT[d0 + 16 + i][d0 + 16], &sT[d0][d0 + 16 + j], 16, -1.f);
        __syncthreads();
        *reinterpret_cast<float4*>(&sT[d0 + i][d0 + 16 + j]) = make_float4(0.f, 0.f, 0.f, 0.f);
        __syncthreads();
    }
    {
        const int i = tid >> 2, j = (tid & 3) * 8;
        product(&sT[i][32 + j], &sA[32 + i][0], &sT[0][j], 32, 1.f);
        product(&sT[i][36 + j], &sA[32 + i][0], &sT[0][j + 4], 32, 1.f);
        __syncthreads();
        product(&sT[32 + i][j], &sT[32 + i][32], &sT[0][32 + j], 32, -1.f);
        product(&sT[32 + i][j + 4], &sT[32 + i][32], &sT[0][36 + j], 32, -1.f);
        __syncthreads();
    }
    for (int i = tid; i < RC_T * RC_T / 2; i += 128) {     // (the walk reads tiles up to the diagonal's only)
        const int r = i >> 5, cc = (i & 31) * 2;
        if (cc > (r | 15)) continue;
        unsigned p1, p2, p3;
        rc_split(sT[r][cc], sT[r][cc + 1], p1, p2, p3);
        *reinterpret_cast<unsigned*>(&P->T[0][r][cc]) = p1;
        *reinterpret_cast<unsigned*>(&P->T[1][r][cc]) = p2;
        *reinterpret_cast<unsigned*>(&P->T[2][r][cc]) = p3;
    }
}

struct RcGdSmem {
    __nv_bfloat16 K[2][RC_T][RC_LD], Q[2][RC_T][RC_LD], V[2][RC_T][RC_GD_CLD];
    __nv_bfloat16 T[3][RC_T][RC_TLD], P[3][RC_T][RC_TLD];
    __nv_bfloat16 S[3][RC_GD_COLS][RC_LD];                 // the state's planes, a column a row
    __nv_bfloat16 R[3][RC_T][RC_GD_CLD], U[3][RC_T][RC_GD_CLD], W[3][RC_T][RC_GD_CLD];     // W: the writes e^{l_L - l_s} u_s / |k_s|
    float scal[2][5][RC_T];
};

// The six products of weight 2^-16 and above of two operands in planes: the first planes' into acc, the others into low
__device__ __forceinline__ void rc_mma6(float (&acc)[4], float (&low)[4], const unsigned (&a)[3][4], const unsigned (&b)[3][4], int half) {
    mma_bf16_16816(low, a[2], b[0][2 * half], b[0][2 * half + 1]);
    mma_bf16_16816(low, a[0], b[2][2 * half], b[2][2 * half + 1]);
    mma_bf16_16816(low, a[1], b[1][2 * half], b[1][2 * half + 1]);
    mma_bf16_16816(low, a[1], b[0][2 * half], b[0][2 * half + 1]);
    mma_bf16_16816(low, a[0], b[1][2 * half], b[1][2 * half + 1]);
    mma_bf16_16816(acc, a[0], b[0][2 * half], b[0][2 * half + 1]);
}

// A chunk has three parts with a barrier behind each: k.S (warps 0..3, 16 tokens each: R) and q.S (warps 4..7, kept in
// registers); U = T R (all warps, 16 tokens x 8 columns each); the outputs (warps 4..7) and the new state (warps 0..3, 32 rows each).
__global__ void __launch_bounds__(RC_THREADS, 1)
delta_chunks_kernel(const __nv_bfloat16* __restrict__ qkv, long long qkv_stride, int q_off, int k_off, int v_off,
                    const RcPrepared* __restrict__ prep, float* __restrict__ state, long long slot_stride,
                    const int* __restrict__ state_slots, const int* __restrict__ cu_q, const int* __restrict__ positions,
                    float* __restrict__ out, int nh, int nkv, int cols, int num_slots, int least, int* __restrict__ status) {
    extern __shared__ __align__(16) unsigned char rc_smem[];
    RcGdSmem& sm = *reinterpret_cast<RcGdSmem*>(rc_smem);
    const int s = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * RC_GD_COLS;
    const int t0 = cu_q[s], qlen = cu_q[s + 1] - t0;
    if (qlen < least) return;
    const int slot = state_slots[s];
    if (slot < 0 || slot >= num_slots) {
        if (threadIdx.x == 0 && status) atomicExch(status, 3);
        return;
    }
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g4 = lane >> 2, p4 = (lane & 3) * 2, quad = warp & 3;
    const int g = h / (nh / nkv);
    const __nv_bfloat16* Ks = qkv + (size_t)t0 * qkv_stride + k_off + (size_t)g * RC_ROWS;
    const __nv_bfloat16* Qs = qkv + (size_t)t0 * qkv_stride + q_off + (size_t)g * RC_ROWS;
    const __nv_bfloat16* Vs = qkv + (size_t)t0 * qkv_stride + v_off + (size_t)h * cols + col0;
    float* S_glob = state + (size_t)slot * slot_stride + (size_t)h * RC_ROWS * cols + col0;
    const bool fresh = positions[t0] == 0;
    const int chunks = (qlen + RC_T - 1) / RC_T;
    const RcPrepared* mine = prep + (size_t)rc_chunks_before(cu_q, s, least) * nh + h;
    pdl_wait();

    auto load_rows = [&](int c) {                          // keys, queries, values and scalars of a chunk
        const int buf = c & 1, count = min(RC_T, qlen - c * RC_T);
        const size_t off = (size_t)c * RC_T * qkv_stride;
        rc_rows(&sm.K[buf][0][0], RC_LD, Ks + off, qkv_stride, count, RC_ROWS / 8, tid, RC_THREADS);
        rc_rows(&sm.Q[buf][0][0], RC_LD, Qs + off, qkv_stride, count, RC_ROWS / 8, tid, RC_THREADS);
        rc_rows(&sm.V[buf][0][0], RC_GD_CLD, Vs + off, qkv_stride, count, RC_GD_COLS / 8, tid, RC_THREADS);
        if (tid < 5 * RC_T / 4) cp_async_16(&sm.scal[buf][0][0] + tid * 4, &mine[(size_t)c * nh].scal[0][0] + tid * 4, 16);
        cp_async_commit();
    };
    auto load_planes = [&](__nv_bfloat16 (&dst)[3][RC_T][RC_TLD], const __nv_bfloat16 (&src)[3][RC_T][RC_T]) {
        for (int i = tid; i < 3 * RC_T * 8; i += RC_THREADS)
            cp_async_16(&dst[0][0][0] + (i >> 3) * RC_TLD + (i & 7) * 8, &src[0][0][0] + (i >> 3) * RC_T + (i & 7) * 8, 16);
        cp_async_commit();
    };
    const int r0 = quad * 32;
    float acc[4][4];                                       // warps 0..3: S^T, 16 columns of the state x 32 of its rows
    auto publish = [&]() {
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                unsigned p1, p2, p3;
                rc_split(acc[n][2 * q], acc[n][2 * q + 1], p1, p2, p3);
                const int c = q * 8 + g4, r = r0 + n * 8 + p4;
                *reinterpret_cast<unsigned*>(&sm.S[0][c][r]) = p1;
                *reinterpret_cast<unsigned*>(&sm.S[1][c][r]) = p2;
                *reinterpret_cast<unsigned*>(&sm.S[2][c][r]) = p3;
            }
    };
    load_rows(0);
    load_planes(sm.T, mine->T);
    if (warp < 4) {
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                acc[n][i] = fresh ? 0.f : S_glob[(size_t)(r0 + n * 8 + p4 + (i & 1)) * cols + (i >> 1) * 8 + g4];
        publish();
    }

    for (int c = 0; c < chunks; ++c) {
        const int buf = c & 1;
        cp_async_wait<0>();
        __syncthreads();                                   // rows and T of this chunk, the state's planes; the last chunk's P and W have been read
        load_planes(sm.P, mine[(size_t)c * nh].P);
        if (c + 1 < chunks) load_rows(c + 1);
        else cp_async_commit();
        const int ta = quad * 16 + g4, tb = ta + 8;
        // ---- k.S and q.S ----
        float ks[2][4], low[2][4];
        {
            float odd[2][4];
            rc_zero(ks); rc_zero(odd); rc_zero(low);
            const __nv_bfloat16* rows = warp < 4 ? &sm.K[buf][0][0] : &sm.Q[buf][0][0];
#pragma unroll
            for (int k = 0; k < RC_ROWS / 16; ++k) {
                unsigned a[4], b[4];
                rc_a(a, rows, RC_LD, quad * 16, k * 16);
#pragma unroll
                for (int pl = 2; pl >= 0; --pl) {
                    rc_b(b, &sm.S[pl][0][0], RC_LD, 0, k * 16);
                    mma_bf16_16816(pl ? low[0] : (k & 1 ? odd[0] : ks[0]), a, b[0], b[1]);
                    mma_bf16_16816(pl ? low[1] : (k & 1 ? odd[1] : ks[1]), a, b[2], b[3]);
                }
            }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) ks[n][i] = (ks[n][i] + odd[n][i]) + low[n][i];
        }
        if (warp < 4) {
            const float ba = sm.scal[buf][0][ta], bb = sm.scal[buf][0][tb], ra = sm.scal[buf][1][ta], rb = sm.scal[buf][1][tb];
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int t = q ? tb : ta;
                    const float2 v = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&sm.V[buf][t][n * 8 + p4]));
                    const float be = q ? bb : ba, re = q ? rb : ra;
                    unsigned p1, p2, p3;
                    rc_split(be * v.x - re * ks[n][2 * q], be * v.y - re * ks[n][2 * q + 1], p1, p2, p3);
                    *reinterpret_cast<unsigned*>(&sm.R[0][t][n * 8 + p4]) = p1;
                    *reinterpret_cast<unsigned*>(&sm.R[1][t][n * 8 + p4]) = p2;
                    *reinterpret_cast<unsigned*>(&sm.R[2][t][n * 8 + p4]) = p3;
                }
        }
        cp_async_wait<1>();                                // this chunk's P
        __syncthreads();
        // ---- U = T R: 16 tokens x 8 columns a warp ----
        {
            float u[4] = {0.f, 0.f, 0.f, 0.f}, ul[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int kt = 0; kt < 4; ++kt)
                if (kt <= quad) {
                    unsigned a[3][4], b[3][4];
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl) {
                        rc_a(a[pl], &sm.T[pl][0][0], RC_TLD, quad * 16, kt * 16);
                        rc_b_trans(b[pl], &sm.R[pl][0][0], RC_GD_CLD, kt * 16, 0);
                    }
                    if (warp < 4) rc_mma6(u, ul, a, b, 0);
                    else rc_mma6(u, ul, a, b, 1);
                }
#pragma unroll
            for (int i = 0; i < 4; ++i) u[i] += ul[i];
            const float wa = sm.scal[buf][3][ta], wb = sm.scal[buf][3][tb];
            const int col = (warp >> 2) * 8 + p4;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int t = q ? tb : ta;
                const float w = q ? wb : wa;
                unsigned p1, p2, p3;
                rc_split(u[2 * q], u[2 * q + 1], p1, p2, p3);
                *reinterpret_cast<unsigned*>(&sm.U[0][t][col]) = p1;
                *reinterpret_cast<unsigned*>(&sm.U[1][t][col]) = p2;
                *reinterpret_cast<unsigned*>(&sm.U[2][t][col]) = p3;
                rc_split(u[2 * q] * w, u[2 * q + 1] * w, p1, p2, p3);
                *reinterpret_cast<unsigned*>(&sm.W[0][t][col]) = p1;
                *reinterpret_cast<unsigned*>(&sm.W[1][t][col]) = p2;
                *reinterpret_cast<unsigned*>(&sm.W[2][t][col]) = p3;
            }
        }
        __syncthreads();
        if (c + 1 < chunks) load_planes(sm.T, mine[(size_t)(c + 1) * nh].T);
        if (warp >= 4) {
            // ---- outputs ----
            const float ea = sm.scal[buf][2][ta], eb = sm.scal[buf][2][tb];
#pragma unroll
            for (int n = 0; n < 2; ++n) { ks[n][0] *= ea; ks[n][1] *= ea; ks[n][2] *= eb; ks[n][3] *= eb; }
            float o[2][4];
            rc_zero(o); rc_zero(low);
#pragma unroll
            for (int kt = 0; kt < 4; ++kt)
                if (kt <= quad) {
                    unsigned a[3][4], b[3][4];
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl) {
                        rc_a(a[pl], &sm.P[pl][0][0], RC_TLD, quad * 16, kt * 16);
                        rc_b_trans(b[pl], &sm.U[pl][0][0], RC_GD_CLD, kt * 16, 0);
                    }
                    rc_mma6(o[0], low[0], a, b, 0);
                    rc_mma6(o[1], low[1], a, b, 1);
                }
#pragma unroll
            for (int n = 0; n < 2; ++n)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int at = c * RC_T + (q ? tb : ta);
                    if (at < qlen)
                        *reinterpret_cast<float2*>(out + ((size_t)(t0 + at) * nh + h) * cols + col0 + n * 8 + p4) = 
                            make_float2((o[n][2 * q] + low[n][2 * q]) + ks[n][2 * q], (o[n][2 * q + 1] + low[n][2 * q + 1]) + ks[n][2 * q + 1]);
                }
        } else {
            // ---- the state ----
            const float last = sm.scal[buf][4][0];
            float add[4][4], rest[4][4];
            rc_zero(add); rc_zero(rest);
#pragma unroll
            for (int kt = 0; kt < 4; ++kt) {
                unsigned b[2][4], a[3][4];
#pragma unroll
                for (int q = 0; q < 2; ++q) rc_b_trans(b[q], &sm.K[buf][0][0], RC_LD, kt * 16, r0 + q * 16);
#pragma unroll
                for (int pl = 0; pl < 3; ++pl) rc_a_trans(a[pl], &sm.W[pl][0][0], RC_GD_CLD, kt * 16, 0);
#pragma unroll
                for (int pl = 2; pl >= 0; --pl)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        mma_bf16_16816(pl ? rest[2 * q] : add[2 * q], a[pl], b[q][0], b[q][1]);
                        mma_bf16_16816(pl ? rest[2 * q + 1] : add[2 * q + 1], a[pl], b[q][2], b[q][3]);
                    }
            }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) acc[n][i] = fmaf(last, acc[n][i], add[n][i] + rest[n][i]);
            publish();
        }
    }
    pdl_trigger();
    if (warp < 4) {
#pragma unroll
        for (int n = 0; n < 4; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) S_glob[(size_t)(r0 + n * 8 + p4 + (i & 1)) * cols + (i >> 1) * 8 + g4] = acc[n][i];
    }
}

// ---- host side ------------------------------------------------------------------------------------------
// sequences of at least this many tokens are worth taking (a call may set its own `least`: a sequence alone in its step)
VAPI_EXPORT int vapi_recurrent_chunks_min(int delta) { return delta ? RC_GD_MIN : RC_SS_MIN; }
// bytes of scratch for a delta-rule step of n tokens in num_seqs sequences
VAPI_EXPORT long long vapi_delta_chunks_scratch(int n, int num_seqs, int nh) {
    return ((long long)n / RC_T + num_seqs) * nh * (long long)sizeof(RcPrepared);
}

template <typename K>
static int rc_reserve(K kern, size_t bytes, const char* what) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    return e == cudaSuccess ? 0 : fail(-101, "%s: cannot reserve %zu bytes of shared memory: %s", what, bytes, cudaGetErrorString(e));
}

// The long sequences of a step (see recurrent.cu for the arguments; bfloat16).  Rows of xbc on 16-byte boundaries.
VAPI_EXPORT int vapi_state_space_chunks(const void* xbc, long long xbc_stride, const void* dt, long long dt_stride,
                                        const float* A_log, const float* dt_bias, const float* D, float* state,
                                        long long slot_stride, const int* state_slots, const int* cu_q, const int* positions,
                                        float* out, int num_seqs, int nh, int groups, int rows, int cols, int num_slots,
                                        int least, int* status, cudaStream_t stream) {
    if (num_seqs <= 0) return 0;
    if (least < 1) least = 1;
    if (nh <= 0 || groups <= 0 || nh % groups || rows != RC_ROWS || cols <= 0 || cols % RC_SS_COLS || nh > 65535 || num_seqs > 65535)
        return fail(-1, "state_space_chunks: %d heads over %d groups, state %d x %d (%d rows, columns in multiples of %d)", nh, groups, rows, cols, RC_ROWS, RC_SS_COLS);
    if (((uintptr_t)xbc & 15) != 0 || xbc_stride % 8 != 0 || ((uintptr_t)out & 7) != 0)
        return fail(-1, "state_space_chunks: rows must start on 16-byte boundaries");
    int rc = rc_reserve(state_space_chunks_kernel, sizeof(RcSsSmem), "state_space_chunks");
    if (rc) return rc;
    return check_launch("state_space_chunks", launch_if(false, state_space_chunks_kernel, dim3(cols / RC_SS_COLS, nh, num_seqs), dim3(RC_THREADS),
        sizeof(RcSsSmem), stream, (const __nv_bfloat16*)xbc, xbc_stride, (const __nv_bfloat16*)dt, dt_stride, A_log, dt_bias, D, state,
        slot_stride, state_slots, cu_q, positions, out, nh, groups, cols, num_slots, least, status));
}

// ``scratch``: vapi_delta_chunks_scratch bytes, 16-byte aligned; ``n``: tokens of the step.
VAPI_EXPORT int vapi_gated_delta_chunks(const void* qkv, long long qkv_stride, int q_off, int k_off, int v_off, const void* ab,
                                        long long ab_stride, const float* A_log, const float* dt_bias, float* state,
                                        long long slot_stride, const int* state_slots, const int* cu_q, const int* positions,
                                        float* out, int n, int num_seqs, int nh, int nkv, int rows, int cols, int num_slots,
                                        float norm_eps, void* scratch, int least, int* status, cudaStream_t stream) {
    if (num_seqs <= 0 || n <= 0) return 0;
    if (least < 1) least = 1;
    if (nh <= 0 || nkv <= 0 || nh % nkv || rows != RC_ROWS || cols <= 0 || cols % RC_GD_COLS || nh > 65535 || num_seqs > 65535)
        return fail(-1, "gated_delta_chunks: %d heads over %d, state %d x %d (%d rows, columns in multiples of %d)", nh, nkv, rows, cols, RC_ROWS, RC_GD_COLS);
    if ((((uintptr_t)qkv | (uintptr_t)scratch) & 15) != 0 || qkv_stride % 8 || q_off % 8 || k_off % 8 || v_off % 8 || ((uintptr_t)out & 7) != 0 || !scratch)
        return fail(-1, "gated_delta_chunks: rows must start on 16-byte boundaries");
    int rc = rc_reserve(delta_chunks_kernel, sizeof(RcGdSmem), "gated_delta_chunks");
    if (rc) return rc;
    rc = check_launch("gated_delta_chunks: prepare", launch(delta_prepare_kernel, dim3(n / RC_T + num_seqs, nh), dim3(128), 0, stream,
        (const __nv_bfloat16*)qkv, qkv_stride, q_off, k_off, (const __nv_bfloat16*)ab, ab_stride, A_log, dt_bias, cu_q, (RcPrepared*)scratch,
        num_seqs, nh, nkv, norm_eps, least));
    if (rc) return rc;
    return check_launch("gated_delta_chunks", launch_if(false, delta_chunks_kernel, dim3(cols / RC_GD_COLS, nh, num_seqs), dim3(RC_THREADS),
        sizeof(RcGdSmem), stream, (const __nv_bfloat16*)qkv, qkv_stride, q_off, k_off, v_off, (const RcPrepared*)scratch, state, slot_stride,
        state_slots, cu_q, positions, out, nh, nkv, cols, num_slots, least, status));
}

VAPI_EXPORT const char* vapi_last_error() { return error_buffer(); }
