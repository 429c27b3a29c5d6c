// The two recurrences over a prompt's portion: the same sums in the same order as gated_delta_kernel and
// state_space_kernel (a token's bits do not depend on which kernel walked over it), arranged for many tokens.
//
// What bounds a walk is one warp's way from token to token: for the delta rule the chain decay, four dependent FMAs, three
// shuffles, the write; for the state space the issue of 24 packed operations a column, token and lane.  There are no more
// than about one warp's worth of columns for each of the chip's schedulers, so nothing else may stand in that way:
//  * four warps of a block only stage (the next tokens' rows in 16-byte pieces, norms, decay, write strength) into one half
//    of a double buffer, while the walking warps, one a scheduler, read the other half and do nothing but steps;
//  * the read-outs, which no later step needs, are added over the lanes for eight tokens at once (7 shuffles, not 24);
//  * rows stay in their own type in shared memory: half the bytes of what bounds a step next, the loads from there.
// 2,000 tokens, 128 rows, one sequence, bfloat16: delta rule (16 heads of 128 columns) 655 us in gated_delta_kernel, 317
// here; state space (64 heads of 64 columns) 726 us in state_space_kernel, 250 here.  Measured beside it: two columns a
// thread for the delta rule (half the warps) 373 us; one column a thread for the state space 303 to 380 us; one block an SM
// (more registers) within 2 % for one sequence, but 244 against 191 us for five of 300 tokens; the read-out by four more warps that
// follow with a state of their own 303 against 289 us (captured): what is left is the chain itself.  At the 128 registers that two
// blocks leave a thread the delta rule keeps 16 to 56 bytes of it in local memory and the float state space of 128 rows 28.
#pragma once
#include "common.cuh"

namespace vapi {

constexpr int WALK_TC = 16;                                   // tokens per half of the buffer
constexpr int WALK_STAGERS = 8 * WALK_TC;                     // threads that stage: eight a token

// RT consecutive elements as they are
template <typename T, int RT>
struct WalkPiece {
    static constexpr int PIECES = RT * (int)sizeof(T) / 16;
    uint4 w[PIECES];
    __device__ __forceinline__ void load(const T* p) {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) w[i] = reinterpret_cast<const uint4*>(p)[i];
    }
    __device__ __forceinline__ void store(T* p) const {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) reinterpret_cast<uint4*>(p)[i] = w[i];
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) w[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    // as float, two a register pair
    __device__ __forceinline__ void floats(float2 (&v)[RT / 2]) const {
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
            const unsigned u[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
            if constexpr (sizeof(T) == 2) {
#pragma unroll
                for (int j = 0; j < 4; ++j) v[4 * i + j] = make_float2(__uint_as_float(u[j] << 16), __uint_as_float(u[j] & 0xffff0000u));
            } else {
                v[2 * i] = make_float2(__uint_as_float(u[0]), __uint_as_float(u[1]));
                v[2 * i + 1] = make_float2(__uint_as_float(u[2]), __uint_as_float(u[3]));
            }
        }
    }
};
__device__ __forceinline__ float walk_sum8(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v;
}
// v[i] of the eight lanes of a column added up for i = 0 .. 7, in the order of walk_sum8: lane i keeps the i-th sum.  Seven
// shuffles where eight sums one by one take 24.
__device__ __forceinline__ float walk_sum8_each(const float (&v)[8], int sl) {
    float a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = ((sl & 4) ? v[i + 4] : v[i]) + __shfl_xor_sync(0xffffffffu, (sl & 4) ? v[i] : v[i + 4], 4);
#pragma unroll
    for (int i = 0; i < 2; ++i) b[i] = ((sl & 2) ? a[i + 2] : a[i]) + __shfl_xor_sync(0xffffffffu, (sl & 2) ? a[i] : a[i + 2], 2);
    return ((sl & 1) ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, (sl & 1) ? b[0] : b[1], 1);
}
__device__ __forceinline__ float walk_softplus(float z) { return z > 20.f ? z : log1pf(expf(z)); }

// A column of the state is shared by eight neighbouring lanes of RT consecutive rows each; NC columns a thread, WW walking warps.
template <typename T, int RT, int NC, int WW>
struct WalkShape {
    static constexpr int CPB = WW * 4 * NC;                   // columns of a block
    static constexpr int LANE = RT + 16 / (int)sizeof(T);     // from one lane's rows to the next lane's (banks)
    static constexpr int ROW = 8 * LANE;                      // a row vector in shared memory
    static constexpr int THREADS = 32 * WW + WALK_STAGERS;
};

template <typename T, int RT, int NC, int WW>
struct alignas(16) DeltaStage {
    T k[WALK_TC][WalkShape<T, RT, NC, WW>::ROW], q[WALK_TC][WalkShape<T, RT, NC, WW>::ROW];
    float4 unit[WALK_TC];                                     // decay, write strength, unit-norm factors of k and q
    float qk[WALK_TC];
    float v[WALK_TC][WalkShape<T, RT, NC, WW>::CPB];
};

// (`rows` is 8 RT: its root is taken at run time, as in gated_delta_kernel)
template <typename T, int RT, int NC, int WW>
__global__ void __launch_bounds__(WalkShape<T, RT, NC, WW>::THREADS, 2)
gated_delta_prompt_kernel(const T* __restrict__ qkv, long long qkv_stride, int q_off, int k_off, int v_off,
                          const T* __restrict__ ab, long long ab_stride, const float* __restrict__ A_log,
                          const float* __restrict__ dt_bias, float* __restrict__ state, long long slot_stride,
                          const int* __restrict__ state_slots, const int* __restrict__ cu_q,
                          const int* __restrict__ positions, float* __restrict__ out, int nh, int nkv, int rows, int cols,
                          int num_slots, float norm_eps, int* __restrict__ status) {
    using Shape = WalkShape<T, RT, NC, WW>;
    using Stage = DeltaStage<T, RT, NC, WW>;
    constexpr int ROWS = 8 * RT, CPB = Shape::CPB, LANE = Shape::LANE, VPT = CPB / 8;
    __shared__ Stage stage[2];
    const int s = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * CPB;
    const int t0 = cu_q[s], qlen = cu_q[s + 1] - t0;
    if (qlen <= 0) return;
    const int slot = state_slots[s];
    if (slot < 0 || slot >= num_slots) {
        if (threadIdx.x == 0 && status) atomicExch(status, 3);
        return;
    }
    const bool fresh = positions[t0] == 0;
    const bool walks = threadIdx.x < 32 * WW;
    const int tid = walks ? threadIdx.x : threadIdx.x - 32 * WW;
    const int sl = tid & 7;
    pdl_wait();

    // staging: eight threads a token, each RT rows of k and of q and CPB / 8 columns of v
    const int g = h / (nh / nkv);
    const float decay_rate = expf(A_log[h]), bias = dt_bias[h], q_scale = rsqrtf((float)rows);
    auto fill = [&](Stage& st, int first) {
        const int tt = tid >> 3;
        const size_t t = (size_t)(t0 + first + tt);
        const T* row = qkv + t * qkv_stride;
        WalkPiece<T, RT> kp, qp;
        float2 kv[RT / 2], qv[RT / 2];
        float vv[VPT], a = 0.f, b = 0.f;
        kp.clear();
        qp.clear();
#pragma unroll
        for (int c = 0; c < VPT; ++c) vv[c] = 0.f;
        if (first + tt < qlen) {                              // (nothing steps over what is staged behind the portion)
            kp.load(row + k_off + g * ROWS + sl * RT);
            qp.load(row + q_off + g * ROWS + sl * RT);
#pragma unroll
            for (int c = 0; c < VPT; ++c) vv[c] = to_f32(row[v_off + h * cols + col0 + sl * VPT + c]);
            if (sl == 1) {
                a = to_f32(ab[t * ab_stride + h]);
                b = to_f32(ab[t * ab_stride + nh + h]);
            }
        }
        kp.store(&st.k[tt][sl * LANE]);
        qp.store(&st.q[tt][sl * LANE]);
#pragma unroll
        for (int c = 0; c < VPT; ++c) st.v[tt][sl * VPT + c] = vv[c];
        kp.floats(kv);
        qp.floats(qv);
        if (sl == 1) {
            st.unit[tt].x = expf(-decay_rate * walk_softplus(a + bias));
            st.unit[tt].y = 1.f / (1.f + expf(-b));
        }
        float ssk = 0.f, ssq = 0.f, dot = 0.f;
#pragma unroll
        for (int r = 0; r < RT / 2; ++r) {
            ssk = fmaf(kv[r].y, kv[r].y, fmaf(kv[r].x, kv[r].x, ssk));
            ssq = fmaf(qv[r].y, qv[r].y, fmaf(qv[r].x, qv[r].x, ssq));
            dot = fmaf(kv[r].y, qv[r].y, fmaf(kv[r].x, qv[r].x, dot));
        }
        ssk = walk_sum8(ssk);
        ssq = walk_sum8(ssq);
        dot = walk_sum8(dot);
        if (sl == 0) {
            const float k_inv = rsqrtf(ssk + norm_eps), q_inv = rsqrtf(ssq + norm_eps) * q_scale;
            st.unit[tt].z = k_inv;
            st.unit[tt].w = q_inv;
            st.qk[tt] = dot * k_inv * q_inv;
        }
    };

    // walking: this thread's rows of its columns, two floats a register pair
    const int c0 = (tid >> 3) * NC;                           // its columns within the block
    float* S_glob = state + (size_t)slot * slot_stride + ((size_t)h * ROWS + sl * RT) * cols + col0 + c0;
    float2 S2[NC][RT / 2];
    if (walks) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int r = 0; r < RT; r += 2) {
                S2[c][r / 2].x = fresh ? 0.f : S_glob[(size_t)r * cols + c];
                S2[c][r / 2].y = fresh ? 0.f : S_glob[(size_t)(r + 1) * cols + c];
            }
    } else {
        fill(stage[0], 0);
    }
    __syncthreads();
    for (int first = 0; first < qlen; first += WALK_TC) {
        const Stage& st = stage[(first / WALK_TC) & 1];
        if (!walks) {
            if (first + WALK_TC < qlen) fill(stage[(first / WALK_TC + 1) & 1], first + WALK_TC);
        } else {
            const int count = min(WALK_TC, qlen - first);
            WalkPiece<T, RT> kn, qn;
            kn.load(&st.k[0][sl * LANE]);
            float4 un = st.unit[0];
            // one token: its decay, read-out (this lane's share of it, `qp`) and write (`u`)
            auto step = [&](int tt, int next, float (&qp)[NC], float (&u)[NC]) {
                float2 kc[RT / 2], qc[RT / 2];
                kn.floats(kc);
                const float4 unit = un;
                kn.load(&st.k[next][sl * LANE]);
                qn.load(&st.q[tt][sl * LANE]);
                un = st.unit[next];
                const float2 g2 = make_float2(unit.x, unit.x);
                float ksum[NC], vv[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    vv[c] = st.v[tt][c0 + c];
                    float2 ks[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
                    for (int r4 = 0; r4 < RT / 4; ++r4) {
                        S2[c][2 * r4] = __fmul2_rn(S2[c][2 * r4], g2);
                        S2[c][2 * r4 + 1] = __fmul2_rn(S2[c][2 * r4 + 1], g2);
                        ks[0] = __ffma2_rn(kc[2 * r4], S2[c][2 * r4], ks[0]);
                        ks[1] = __ffma2_rn(kc[2 * r4 + 1], S2[c][2 * r4 + 1], ks[1]);
                    }
                    ksum[c] = (ks[0].x + ks[0].y) + (ks[1].x + ks[1].y);
                }
#pragma unroll
                for (int c = 0; c < NC; ++c) ksum[c] = walk_sum8(ksum[c]) * unit.z;
                // (the read-out of the decayed state: in the shadow of those shuffles)
                qn.floats(qc);
                float2 qs[NC][2];
#pragma unroll
                for (int c = 0; c < NC; ++c) qs[c][0] = qs[c][1] = make_float2(0.f, 0.f);
#pragma unroll
                for (int r4 = 0; r4 < RT / 4; ++r4)
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        qs[c][0] = __ffma2_rn(qc[2 * r4], S2[c][2 * r4], qs[c][0]);
                        qs[c][1] = __ffma2_rn(qc[2 * r4 + 1], S2[c][2 * r4 + 1], qs[c][1]);
                    }
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    qp[c] = (qs[c][0].x + qs[c][0].y) + (qs[c][1].x + qs[c][1].y);
                    u[c] = unit.y * (vv[c] - ksum[c]);
                    const float2 uk = make_float2(u[c] * unit.z, u[c] * unit.z);
#pragma unroll
                    for (int r = 0; r < RT / 2; ++r) S2[c][r] = __ffma2_rn(kc[r], uk, S2[c][r]);
                }
            };
            const int whole = count & ~7;
            for (int done = 0; done < whole; done += 8) {
                float qp[NC][8], mine[NC];                    // the lanes' shares of eight read-outs; u of this lane's token of the eight
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float share[NC], u[NC];
                    step(done + j, j < 7 ? done + j + 1 : min(done + j + 1, WALK_TC - 1), share, u);
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        qp[c][j] = share[c];
                        if (j == 0 || j == sl) mine[c] = u[c];
                    }
                }
                const float qk = st.qk[done + sl], q_inv = st.unit[done + sl].w;
#pragma unroll
                for (int c = 0; c < NC; ++c)
                    out[((size_t)(t0 + first + done + sl) * nh + h) * cols + col0 + c0 + c] = fmaf(qk, mine[c], walk_sum8_each(qp[c], sl) * q_inv);
            }
            // The last few, fewer than eight, one by one: a step over a token that is not there would not leave the state as it is, whatever
            // is staged for it (a unit norm over zeros with an epsilon of 0, an infinity in the state).  A sequence of one token beside a
            // portion takes one step, not eight: 60 of them beside 17, 16 heads of 128 x 128, bfloat16 112 us, so 74.
#pragma unroll 1
            for (int done = whole; done < count; ++done) {
                float share[NC], u[NC];
                step(done, min(done + 1, WALK_TC - 1), share, u);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float qsum = walk_sum8(share[c]) * st.unit[done].w;
                    if (sl == 0) out[((size_t)(t0 + first + done) * nh + h) * cols + col0 + c0 + c] = fmaf(st.qk[done], u[c], qsum);
                }
            }
        }
        __syncthreads();                                      // this half is free, the other one is staged
    }
    pdl_trigger();                                            // (the next kernel is let go when the walk is over)
    if (walks) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int r = 0; r < RT; r += 2) {
                S_glob[(size_t)r * cols + c] = S2[c][r / 2].x;
                S_glob[(size_t)(r + 1) * cols + c] = S2[c][r / 2].y;
            }
    }
}

template <typename T, int RT, int NC, int WW>
struct alignas(16) SpaceStage {
    T B[WALK_TC][WalkShape<T, RT, NC, WW>::ROW], C[WALK_TC][WalkShape<T, RT, NC, WW>::ROW];
    float4 unit[WALK_TC];                                     // decay, step, B . C
    float x[WALK_TC][WalkShape<T, RT, NC, WW>::CPB];
};

// (NC columns a thread share the loads of B and C)
template <typename T, int RT, int NC, int WW>
__global__ void __launch_bounds__(WalkShape<T, RT, NC, WW>::THREADS, 2)
state_space_prompt_kernel(const T* __restrict__ xbc, long long xbc_stride, const T* __restrict__ dt, long long dt_stride,
                          const float* __restrict__ A_log, const float* __restrict__ dt_bias, const float* __restrict__ D,
                          float* __restrict__ state, long long slot_stride, const int* __restrict__ state_slots,
                          const int* __restrict__ cu_q, const int* __restrict__ positions, float* __restrict__ out, int nh,
                          int groups, int cols, int num_slots, int* __restrict__ status) {
    using Shape = WalkShape<T, RT, NC, WW>;
    using Stage = SpaceStage<T, RT, NC, WW>;
    constexpr int ROWS = 8 * RT, CPB = Shape::CPB, LANE = Shape::LANE, VPT = CPB / 8;
    __shared__ Stage stage[2];
    const int s = blockIdx.z, h = blockIdx.y, col0 = blockIdx.x * CPB;
    const int t0 = cu_q[s], qlen = cu_q[s + 1] - t0;
    if (qlen <= 0) return;
    const int slot = state_slots[s];
    if (slot < 0 || slot >= num_slots) {
        if (threadIdx.x == 0 && status) atomicExch(status, 3);
        return;
    }
    const bool fresh = positions[t0] == 0;
    const bool walks = threadIdx.x < 32 * WW;
    const int tid = walks ? threadIdx.x : threadIdx.x - 32 * WW;
    const int sl = tid & 7;
    pdl_wait();

    const int g = h / (nh / groups);
    const float rate = expf(A_log[h]), bias = dt_bias[h], skip = D[h];
    const int b_off = nh * cols + g * ROWS, c_off = nh * cols + groups * ROWS + g * ROWS;
    auto fill = [&](Stage& st, int first) {
        const int tt = tid >> 3;
        const bool there = first + tt < qlen;
        const size_t t = (size_t)(t0 + first + (there ? tt : 0));
        const T* row = xbc + t * xbc_stride;
        WalkPiece<T, RT> bp, cp;
        float2 bv[RT / 2], cv[RT / 2];
        float xv[VPT], d = 0.f;
        bp.load(row + b_off + sl * RT);
        cp.load(row + c_off + sl * RT);
#pragma unroll
        for (int c = 0; c < VPT; ++c) xv[c] = to_f32(row[h * cols + col0 + sl * VPT + c]);
        if (sl == 1) d = to_f32(dt[t * dt_stride + h]);
        if (!there) {                                         // behind the portion: a step that leaves the state as it is
            bp.clear();
            cp.clear();
#pragma unroll
            for (int c = 0; c < VPT; ++c) xv[c] = 0.f;
        }
        bp.store(&st.B[tt][sl * LANE]);
        cp.store(&st.C[tt][sl * LANE]);
#pragma unroll
        for (int c = 0; c < VPT; ++c) st.x[tt][sl * VPT + c] = xv[c];
        bp.floats(bv);
        cp.floats(cv);
        if (sl == 1) {
            const float step = walk_softplus(d + bias);
            st.unit[tt].x = there ? expf(-rate * step) : 1.f;
            st.unit[tt].y = there ? step : 0.f;
        }
        float dot = 0.f;
#pragma unroll
        for (int r = 0; r < RT / 2; ++r) dot = fmaf(bv[r].y, cv[r].y, fmaf(bv[r].x, cv[r].x, dot));
        dot = walk_sum8(dot);
        if (sl == 0) st.unit[tt].z = dot;
    };

    const int c0 = (tid >> 3) * NC;
    float* S_glob = state + (size_t)slot * slot_stride + ((size_t)h * ROWS + sl * RT) * cols + col0 + c0;
    float2 S2[NC][RT / 2];
    if (walks) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int r = 0; r < RT; r += 2) {
                S2[c][r / 2].x = fresh ? 0.f : S_glob[(size_t)r * cols + c];
                S2[c][r / 2].y = fresh ? 0.f : S_glob[(size_t)(r + 1) * cols + c];
            }
    } else {
        fill(stage[0], 0);
    }
    __syncthreads();
    for (int first = 0; first < qlen; first += WALK_TC) {
        const Stage& st = stage[(first / WALK_TC) & 1];
        if (!walks) {
            if (first + WALK_TC < qlen) fill(stage[(first / WALK_TC + 1) & 1], first + WALK_TC);
        } else {
            const int count = min(WALK_TC, qlen - first);
            for (int t8 = 0; t8 < count; t8 += 8) {
                float cp[NC][8];                              // the lanes' shares of eight read-outs
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int tt = t8 + j;
                    const float2 unit = *reinterpret_cast<const float2*>(&st.unit[tt]);
                    const float2 dec2 = make_float2(unit.x, unit.x);
                    WalkPiece<T, RT> bp, cq;
                    float2 bv[RT / 2], cv[RT / 2];
                    bp.load(&st.B[tt][sl * LANE]);
                    cq.load(&st.C[tt][sl * LANE]);
                    bp.floats(bv);
                    cq.floats(cv);
                    float2 cs[NC][2], sx2[NC];
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        const float sxv = unit.y * st.x[tt][c0 + c];
                        sx2[c] = make_float2(sxv, sxv);
                        cs[c][0] = cs[c][1] = make_float2(0.f, 0.f);
                    }
#pragma unroll
                    for (int r4 = 0; r4 < RT / 4; ++r4)
#pragma unroll
                        for (int c = 0; c < NC; ++c) {
                            cs[c][0] = __ffma2_rn(cv[2 * r4], S2[c][2 * r4], cs[c][0]);
                            cs[c][1] = __ffma2_rn(cv[2 * r4 + 1], S2[c][2 * r4 + 1], cs[c][1]);
                            S2[c][2 * r4] = __ffma2_rn(dec2, S2[c][2 * r4], __fmul2_rn(bv[2 * r4], sx2[c]));
                            S2[c][2 * r4 + 1] = __ffma2_rn(dec2, S2[c][2 * r4 + 1], __fmul2_rn(bv[2 * r4 + 1], sx2[c]));
                        }
#pragma unroll
                    for (int c = 0; c < NC; ++c) cp[c][j] = (cs[c][0].x + cs[c][0].y) + (cs[c][1].x + cs[c][1].y);
                }
                const float4 unit = st.unit[t8 + sl];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const float xv = st.x[t8 + sl][c0 + c], sxv = unit.y * xv;
                    const float csum = walk_sum8_each(cp[c], sl);
                    if (t8 + sl < count)
                        out[((size_t)(t0 + first + t8 + sl) * nh + h) * cols + col0 + c0 + c] = fmaf(unit.x, csum, fmaf(unit.z, sxv, skip * xv));
                }
            }
        }
        __syncthreads();
    }
    pdl_trigger();
    if (walks) {
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int r = 0; r < RT; r += 2) {
                S_glob[(size_t)r * cols + c] = S2[c][r / 2].x;
                S_glob[(size_t)(r + 1) * cols + c] = S2[c][r / 2].y;
            }
    }
}

// Whether rows of `src` (16-byte pieces of the row vectors) can be taken by the kernels above.
inline bool walk_aligned(const void* src, long long stride, int dtype, int a_off, int b_off) {
    const int e = dtype == VAPI_BF16 ? 8 : 4;
    return ((uintptr_t)src % 16) == 0 && stride % e == 0 && a_off % e == 0 && b_off % e == 0;
}

}  // namespace vapi
