// Paged GQA attention for prompt portions of the true 32-bit path: float queries, keys and values, head_dim 64, pages whose
// size is a multiple of 64.  Same rows, masks and partial results as the general kernel of attention.cu, which it replaces
// for steps of more than 16 rows per (sequence, kv head): 1,024 tokens, 32 / 8 heads, took that kernel 403 us, almost all of it
// float FMAs fed from shared memory.
//
// Both products run on the tensor cores without giving up float: a float is the exact sum of three bfloat16 (24 bits), and of
// the nine products the six of weight 2^-16 and above are taken (the rest is at most 2^-24 of the term; see linear_f32.cu).
// The leading products and the five small ones have accumulators of their own, and a tile's P.V is added to the output by
// float FMAs: a tensor core cuts off what it adds to an accumulator, so the leading products' chains are kept to four instructions (the
// small ones, of 2^-8 and less, come to twenty).  Maximum, exponentials and sums are float as before.
//
// Portions of sequences of up to 36 tokens would be a little faster on the general kernel (17 tokens, 32 / 8 heads: 7.6 us against 11.4), but its
// results are further from exact (1.3e-7 against 7.6e-8 of their 2-norm), so they stay here.
//
// A block of four warps owns 64 rows and walks the 64-key tiles any of them can see: the tile's floats come by asynchronous copies
// while the tile before is multiplied, all threads split them into planes (128-byte rows, 16-byte pieces swizzled), a warp
// takes 16 rows.  106 KB of shared memory and two blocks a multiprocessor, so that one block splits while the other
// multiplies.  A tile with an infinity or a NaN, which have no such planes, or with magnitudes whose products could overflow is computed by FMAs.
#pragma once
#include "attention_mma.cuh"
#include "attention_tc.cuh"        // ft_tile

namespace vapi {

constexpr int FF_ROWS = 64, FF_BK = 64, FF_HD = 64, FF_THREADS = 128;
constexpr int FF_PLANE = FF_BK * FF_HD * 2;
constexpr size_t FF_SMEM = 9 * FF_PLANE + 2 * FF_BK * FF_HD * 4 + 128;     // planes of Q, K, V; floats of K, V
// From here on a tile is computed by FMAs: below 2^60 a score, and below 2^120 a sum of 64 values, stays finite in every partial
// sum (one that overflows takes the others with it: plus infinity of x1 y1 and minus infinity of x1 y2 are NaN, a float product infinity).
constexpr float FF_LIMIT_QK = 1.152921504606846976e18f, FF_LIMIT_V = 1.329227995784915873e36f;

// four floats of a row (piece c4 of 16 bytes of float) into the three planes; the largest magnitude so far
__device__ __forceinline__ float ff_store(unsigned char* planes, int row, int c4, float4 v, float top) {
    uint2 p1, p2, p3;
    split_f32x2(v.x, v.y, p1.x, p2.x, p3.x);
    split_f32x2(v.z, v.w, p1.y, p2.y, p3.y);
    unsigned char* at = planes + row * 128 + ((((c4 >> 1) ^ (row & 7)) << 4) | ((c4 & 1) << 3));
    *reinterpret_cast<uint2*>(at) = p1;
    *reinterpret_cast<uint2*>(at + FF_PLANE) = p2;
    *reinterpret_cast<uint2*>(at + 2 * FF_PLANE) = p3;
    return absmax_nan(absmax_nan(absmax_nan(absmax_nan(top, v.x), v.y), v.z), v.w);
}
__device__ __forceinline__ const unsigned char* ff_at(const unsigned char* plane, int row, int piece) {
    return plane + row * 128 + ((piece ^ (row & 7)) << 4);
}
// the six products: the leading one into acc, the others into low
__device__ __forceinline__ void ff_mma6(float (&acc)[4], float (&low)[4], const unsigned (&a)[3][4], const unsigned (&b)[3][4], int half) {
    mma_bf16_16816(low, a[2], b[0][2 * half], b[0][2 * half + 1]);
    mma_bf16_16816(low, a[0], b[2][2 * half], b[2][2 * half + 1]);
    mma_bf16_16816(low, a[1], b[1][2 * half], b[1][2 * half + 1]);
    mma_bf16_16816(low, a[1], b[0][2 * half], b[0][2 * half + 1]);
    mma_bf16_16816(low, a[0], b[1][2 * half], b[1][2 * half + 1]);
    mma_bf16_16816(acc, a[0], b[0][2 * half], b[0][2 * half + 1]);
}

__global__ void __launch_bounds__(FF_THREADS, 2)
flash_f32_kernel(const float* q, long long q_row_stride, const float* cache, const int* __restrict__ block_table, int table_stride,
                 const int* __restrict__ cu_q, const int* __restrict__ seqlens_k, float* out, float* part_o, float* part_ml,
                 int num_seqs, int nh, int nkv, int page_size, int num_pages, float scale, int window, int splits, int* status) {
    extern __shared__ unsigned char ff_smem_raw[];
    unsigned char* sQ = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ff_smem_raw) + 127) & ~(uintptr_t)127);
    unsigned char *sK = sQ + 3 * FF_PLANE, *sV = sK + 3 * FF_PLANE;
    float *fK = reinterpret_cast<float*>(sV + 3 * FF_PLANE), *fV = fK + FF_BK * FF_HD;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g4 = lane >> 2, p4 = (lane & 3) * 2, mat = lane >> 3, r8 = lane & 7;
    const int g = (int)blockIdx.x % nkv, sp = blockIdx.y, n_rep = nh / nkv;      // (heads side by side: the longest tiles of all start first)
    pdl_trigger();
    int s = 0, tile = 0;
    const bool mine = ft_tile(cu_q, num_seqs, 1, n_rep, FF_ROWS, (int)blockIdx.x / nkv, s, tile);
    pdl_wait();
    if (!mine) return;
    const int q0 = cu_q[s], qlen = cu_q[s + 1] - q0, klen = seqlens_k[s];
    const int rows_total = qlen * n_rep, tile_start = tile * FF_ROWS;
    const int last_row = min(rows_total, tile_start + FF_ROWS) - 1, base_pos = klen - qlen;
    const int p_min = base_pos + tile_start / n_rep, p_max = base_pos + last_row / n_rep;
    const int key_lo = window > 0 ? max(0, p_min - window + 1) : 0;
    const int kt_lo = key_lo / FF_BK, kt_hi = p_max / FF_BK;
    const int share = (kt_hi - kt_lo + splits) / splits;
    const int kt_begin = kt_lo + sp * share, kt_end = min(kt_hi + 1, kt_begin + share);

    // this lane's two rows
    int pos[2];
    const float* qrow[2];
    long long grow[2];
    bool ok[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int rr = tile_start + warp * 16 + i * 8 + g4;
        ok[i] = rr < rows_total;
        const int tok = ok[i] ? rr / n_rep : 0, h = g * n_rep + (ok[i] ? rr - tok * n_rep : 0);
        pos[i] = ok[i] ? base_pos + tok : -1;                       // -1: sees nothing
        qrow[i] = q + (size_t)(q0 + tok) * q_row_stride + (size_t)h * FF_HD;
        grow[i] = (long long)(q0 + tok) * nh + h;
    }
    const bool busy = tile_start + warp * 16 < rows_total;          // (a warp without rows helps to split and multiplies nothing)
    const int* bt = block_table + (size_t)s * table_stride;
    auto load = [&](int kt) {
        int page = bt[(kt * FF_BK) / page_size];
        const bool good = page >= 0 && page < num_pages;
        if (!good) {
            if (tid == 0 && status) atomicExch(status, 4);
            page = 0;
        }
        const float* k = cache + ((size_t)page * 2 * nkv + g) * page_size * FF_HD + (size_t)((kt * FF_BK) % page_size) * FF_HD;
        const float* v = k + (size_t)nkv * page_size * FF_HD;
        for (int i = tid; i < FF_BK * FF_HD / 4; i += FF_THREADS) {
            const int j = kt * FF_BK + (i >> 4);
            const int bytes = good && j >= key_lo && j <= p_max && j < klen ? 16 : 0;      // keys that no row of the tile can see stay zero
            cp_async_16(fK + i * 4, k + i * 4, bytes);
            cp_async_16(fV + i * 4, v + i * 4, bytes);
        }
        cp_async_commit();
    };
    if (kt_begin < kt_end) load(kt_begin);
    float qtop = 0.f;
    for (int i = tid; i < FF_ROWS * FF_HD / 4; i += FF_THREADS) {
        const int lr = i >> 4, c4 = i & 15, rr = tile_start + lr;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (rr < rows_total) {
            const int tok = rr / n_rep, h = g * n_rep + (rr - tok * n_rep);
            v = *reinterpret_cast<const float4*>(q + (size_t)(q0 + tok) * q_row_stride + (size_t)h * FF_HD + c4 * 4);
            v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
        }
        qtop = ff_store(sQ, lr, c4, v, qtop);
    }

    float o[8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int n = 0; n < 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.f;
    for (int kt = kt_begin; kt < kt_end; ++kt) {
        cp_async_wait<0>();
        __syncthreads();                                            // the tile's floats are here, the planes of the last tile have been read
        float top = qtop, vtop = 0.f;
#pragma unroll 4
        for (int i = tid; i < FF_BK * FF_HD / 4; i += FF_THREADS) {
            top = ff_store(sK, i >> 4, i & 15, *reinterpret_cast<const float4*>(fK + i * 4), top);
            vtop = ff_store(sV, i >> 4, i & 15, *reinterpret_cast<const float4*>(fV + i * 4), vtop);
        }
        const bool plain = __syncthreads_or(!(top < FF_LIMIT_QK && vtop < FF_LIMIT_V)) != 0;
        if (!plain && kt + 1 < kt_end) load(kt + 1);

        if (!busy && !plain) continue;
        float sc[8][4], low[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            sc[n][0] = sc[n][1] = sc[n][2] = sc[n][3] = 0.f;
            low[n][0] = low[n][1] = low[n][2] = low[n][3] = 0.f;
        }
        if (!plain) {
#pragma unroll
            for (int k = 0; k < FF_HD / 16; ++k) {
                unsigned a[3][4], b[3][4];
#pragma unroll
                for (int pl = 0; pl < 3; ++pl)
                    ldmatrix_x4(a[pl][0], a[pl][1], a[pl][2], a[pl][3], ff_at(sQ + pl * FF_PLANE, warp * 16 + (lane & 15), k * 2 + (lane >> 4)));
#pragma unroll
                for (int j = 0; j < 4; ++j) {
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl)
                        ldmatrix_x4(b[pl][0], b[pl][1], b[pl][2], b[pl][3], ff_at(sK + pl * FF_PLANE, j * 16 + (mat >> 1) * 8 + r8, k * 2 + (mat & 1)));
                    ff_mma6(sc[2 * j], low[2 * j], a, b, 0);
                    ff_mma6(sc[2 * j + 1], low[2 * j + 1], a, b, 1);
                }
            }
        } else {
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float* kr = fK + (n * 8 + p4 + (i & 1)) * FF_HD;
                    float d = 0.f;
                    if (ok[i >> 1])
#pragma unroll 1
                        for (int c = 0; c < FF_HD; ++c) d = fmaf(qrow[i >> 1][c] * scale, kr[c], d);
                    sc[n][i] = d;
                }
        }
        float alpha[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {                               // rows g4 and g4 + 8
            float mx = m[i];
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int x = 2 * i; x < 2 * i + 2; ++x) {
                    const int j = kt * FF_BK + n * 8 + p4 + (x & 1);
                    const bool vis = j <= pos[i] && j < klen && (window <= 0 || j > pos[i] - window);
                    sc[n][x] = vis ? sc[n][x] + low[n][x] : -INFINITY;
                    mx = fmaxf(mx, sc[n][x]);
                }
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
            alpha[i] = mx == -INFINITY ? 1.f : expf(m[i] - mx);     // (-inf before the first visible key: 0)
            float sum = 0.f;
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int x = 2 * i; x < 2 * i + 2; ++x) {
                    const int j = kt * FF_BK + n * 8 + p4 + (x & 1);
                    const bool vis = j <= pos[i] && j < klen && (window <= 0 || j > pos[i] - window);
                    const float p = vis && mx != -INFINITY ? expf(sc[n][x] - mx) : 0.f;
                    sc[n][x] = p;
                    sum += p;
                }
            l[i] = l[i] * alpha[i] + sum;                           // (this lane's keys; the four lanes of a row are added at the end)
            m[i] = mx;
        }
        float pv[8][4];
#pragma unroll
        for (int n = 0; n < 8; ++n) {
            pv[n][0] = pv[n][1] = pv[n][2] = pv[n][3] = 0.f;
            low[n][0] = low[n][1] = low[n][2] = low[n][3] = 0.f;
        }
        if (!plain) {
#pragma unroll
            for (int k = 0; k < FF_BK / 16; ++k) {
                unsigned a[3][4], b[3][4];
                split_f32x2(sc[2 * k][0], sc[2 * k][1], a[0][0], a[1][0], a[2][0]);
                split_f32x2(sc[2 * k][2], sc[2 * k][3], a[0][1], a[1][1], a[2][1]);
                split_f32x2(sc[2 * k + 1][0], sc[2 * k + 1][1], a[0][2], a[1][2], a[2][2]);
                split_f32x2(sc[2 * k + 1][2], sc[2 * k + 1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
#pragma unroll
                    for (int pl = 0; pl < 3; ++pl)
                        ldmatrix_x4_trans(b[pl][0], b[pl][1], b[pl][2], b[pl][3], ff_at(sV + pl * FF_PLANE, k * 16 + (mat & 1) * 8 + r8, j * 2 + (mat >> 1)));
                    ff_mma6(pv[2 * j], low[2 * j], a, b, 0);
                    ff_mma6(pv[2 * j + 1], low[2 * j + 1], a, b, 1);
                }
            }
        } else {
            float* P = reinterpret_cast<float*>(sK);                // [64][64], over the keys' planes
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) P[(warp * 16 + (i >> 1) * 8 + g4) * FF_BK + n * 8 + p4 + (i & 1)] = sc[n][i];
            __syncthreads();
#pragma unroll
            for (int n = 0; n < 8; ++n)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float* pr = P + (warp * 16 + (i >> 1) * 8 + g4) * FF_BK;
                    float d = 0.f;
#pragma unroll 1
                    for (int k = 0; k < FF_BK; ++k) {
                        const int j = kt * FF_BK + k, at = pos[i >> 1];
                        if (j <= at && j < klen && (window <= 0 || j > at - window)) d = fmaf(pr[k], fV[k * FF_HD + n * 8 + p4 + (i & 1)], d);
                    }
                    pv[n][i] = d;
                }
            __syncthreads();                                        // the floats have been read
            if (kt + 1 < kt_end) load(kt + 1);
        }
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) o[n][i] = fmaf(alpha[i >> 1], o[n][i], pv[n][i] + low[n][i]);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 1);
        l[i] += __shfl_xor_sync(0xffffffffu, l[i], 2);
        if (!ok[i]) continue;
        const float inv = splits > 1 ? 1.f : (l[i] > 0.f ? 1.f / l[i] : 0.f);
        float* dst = splits > 1 ? part_o + (grow[i] * splits + sp) * FF_HD : out + grow[i] * FF_HD;
#pragma unroll
        for (int n = 0; n < 8; ++n) *reinterpret_cast<float2*>(dst + n * 8 + p4) = make_float2(o[n][2 * i] * inv, o[n][2 * i + 1] * inv);
        if (splits > 1 && (lane & 3) == 0) {
            part_ml[(grow[i] * splits + sp) * 2] = m[i];
            part_ml[(grow[i] * splits + sp) * 2 + 1] = l[i];
        }
    }
}

static int launch_flash_f32(const void* q, long long q_row_stride, const void* cache, const int* block_table, int table_stride,
                            const int* cu_q, const int* seqlens_k, void* out, float* part_o, float* part_ml, int n, int num_seqs,
                            int max_q, int nh, int nkv, int page_size, int num_pages, float scale, int window, int splits,
                            int* status, cudaStream_t stream) {
    const int n_rep = nh / nkv;
    const long long longest = ((long long)max_q * n_rep + FF_ROWS - 1) / FF_ROWS, whole = (long long)n * n_rep / FF_ROWS + num_seqs;
    const long long tiles = longest * num_seqs < whole ? longest * num_seqs : whole;
    if (tiles * nkv > 0x7fffffffLL || nkv > 65535 || (long long)num_seqs * splits > 65535)
        return fail(-1, "paged_attention: %d kv heads or %d sequences x %d splits exceed the grid", nkv, num_seqs, splits);
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(flash_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FF_SMEM);
        if (e != cudaSuccess) return fail(-101, "paged_attention: cannot reserve %zu bytes of shared memory: %s", FF_SMEM, cudaGetErrorString(e));
        attr_set = true;
    }
    return check_launch("paged_attention (float)", launch(flash_f32_kernel, dim3((unsigned)(tiles * nkv), splits), dim3(FF_THREADS), FF_SMEM, stream,
        (const float*)q, q_row_stride, (const float*)cache, block_table, table_stride, cu_q, seqlens_k, (float*)out, part_o, part_ml,
        num_seqs, nh, nkv, page_size, num_pages, scale, window, splits, status));
}

// ---------------------------------------------------------------------------------------------
// Decode steps of the same path: one token a sequence, at most four q heads a kv head.  What there is to do is to read keys and
// values once, so the kernel is built around those loads: a block owns a (sequence, kv head, slice of the keys) and takes 128 keys
// a time.  Scores: a quad of lanes a key, 16 bytes of its row a lane and load, the sixteen floats of every q row that go with them
// in registers, two exchanges a row.  Softmax: a warp a q row.  P.V: 32 keys a warp, two elements a lane, the loads under way
// before the softmax; the four warps' sums are added in their order.  No staging of keys or values.  Pages whose size is a
// multiple of 32.
// (The general kernel copies both through shared memory and keeps four of its sixteen rows busy: 26 us for 8 sequences
// of 1,024 keys, 32 / 8 heads, against 11 here; the bytes take 5.)
constexpr int DF_KEYS = 128, DF_ROWS = 4, DF_THREADS = 128;

__global__ void __launch_bounds__(DF_THREADS, 3)
decode_f32_kernel(const float* q, long long q_row_stride, const float* cache, const int* __restrict__ block_table, int table_stride,
                  const int* __restrict__ cu_q, const int* __restrict__ seqlens_k, float* out, float* part_o, float* part_ml,
                  int nh, int nkv, int page_size, int num_pages, float scale, int window, int splits, int* status) {
    __shared__ __align__(16) float sc[DF_KEYS][DF_ROWS];              // scores, then weights
    __shared__ float m_s[DF_ROWS], l_s[DF_ROWS], alpha_s[DF_ROWS];
    __shared__ float red[4][DF_ROWS][FF_HD];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, sub = lane & 3;
    const int s = blockIdx.x, g = blockIdx.y, sp = blockIdx.z, n_rep = nh / nkv;
    pdl_trigger();
    const int q0 = cu_q[s], qlen = cu_q[s + 1] - q0, klen = seqlens_k[s];
    const int* bt = block_table + (size_t)s * table_stride;
    // the same slices of 32-key tiles as the general kernel's
    const int key_lo = window > 0 ? max(0, klen - window) : 0;
    const int kt_lo = key_lo / 32, kt_hi = (klen - 1) / 32, share = (kt_hi - kt_lo + splits) / splits;
    const int k_begin = (kt_lo + sp * share) * 32, k_end = min(klen, (kt_lo + (sp + 1) * share) * 32);
    pdl_wait();
    if (qlen <= 0) return;
    float4 qv[DF_ROWS][4];
#pragma unroll
    for (int r = 0; r < DF_ROWS; ++r)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (r < n_rep) v = *reinterpret_cast<const float4*>(q + (size_t)q0 * q_row_stride + (size_t)(g * n_rep + r) * FF_HD + (sub + 4 * i) * 4);
            qv[r][i] = make_float4(v.x * scale, v.y * scale, v.z * scale, v.w * scale);
        }
    if (tid < DF_ROWS) { m_s[tid] = -INFINITY; l_s[tid] = 0.f; }
    float2 acc[DF_ROWS];
#pragma unroll
    for (int r = 0; r < DF_ROWS; ++r) acc[r] = make_float2(0.f, 0.f);
    for (int base = k_begin; base < k_end; base += DF_KEYS) {
        // this warp's 32 keys lie in one page; those that there are to read are first .. last - 1 of them
        const int j0 = base + warp * 32;
        int first = max(key_lo - j0, 0), last = min(k_end - j0, 32);
        const float* rows = cache;
        if (first < last) {
            const int pi = j0 / page_size, page = bt[pi];
            if (page < 0 || page >= num_pages) {
                if (lane == 0 && status) atomicExch(status, 4);
                last = first = 0;
            } else {
                rows = cache + ((size_t)page * 2 * nkv + g) * page_size * FF_HD + (size_t)(j0 - pi * page_size) * FF_HD;
            }
        }
        float4 kv[4][4];
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int k = it * 8 + (lane >> 2);
            const float* row = rows + k * FF_HD;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                kv[it][i] = k >= first && k < last ? *reinterpret_cast<const float4*>(row + (sub + 4 * i) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();                                              // the last weights have been read
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            float d[DF_ROWS];
#pragma unroll
            for (int r = 0; r < DF_ROWS; ++r) {
                float t = 0.f;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    t = fmaf(qv[r][i].x, kv[it][i].x, t);
                    t = fmaf(qv[r][i].y, kv[it][i].y, t);
                    t = fmaf(qv[r][i].z, kv[it][i].z, t);
                    t = fmaf(qv[r][i].w, kv[it][i].w, t);
                }
                t += __shfl_xor_sync(0xffffffffu, t, 1);
                d[r] = t + __shfl_xor_sync(0xffffffffu, t, 2);
            }
            const int k = it * 8 + (lane >> 2);
            // (a lane of the quad for each q row)
            const float mine = sub == 0 ? d[0] : sub == 1 ? d[1] : sub == 2 ? d[2] : d[3];
            sc[warp * 32 + k][sub] = k >= max(key_lo - j0, 0) && j0 + k < k_end ? mine : -INFINITY;
        }
        float2 vv[32];
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            vv[i] = i >= first && i < last ? *reinterpret_cast<const float2*>(rows + ((size_t)nkv * page_size + i) * FF_HD + lane * 2) : make_float2(0.f, 0.f);
        }
        __syncthreads();
        {
            const int r = warp;
            float v[4], mx = m_s[r];
#pragma unroll
            for (int i = 0; i < 4; ++i) { v[i] = sc[lane + 32 * i][r]; mx = fmaxf(mx, v[i]); }
            mx = warp_max(mx);
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float p = v[i] == -INFINITY ? 0.f : expf(v[i] - mx);
                sc[lane + 32 * i][r] = p;
                sum += p;
            }
            sum = warp_sum(sum);
            __syncwarp();
            if (lane == 0) {
                const float a = mx == -INFINITY ? 1.f : expf(m_s[r] - mx);
                alpha_s[r] = a;
                l_s[r] = l_s[r] * a + sum;
                m_s[r] = mx;
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < DF_ROWS; ++r) { acc[r].x *= alpha_s[r]; acc[r].y *= alpha_s[r]; }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            const float4 p = *reinterpret_cast<const float4*>(&sc[warp * 32 + i][0]);
            acc[0].x = fmaf(p.x, vv[i].x, acc[0].x); acc[0].y = fmaf(p.x, vv[i].y, acc[0].y);
            acc[1].x = fmaf(p.y, vv[i].x, acc[1].x); acc[1].y = fmaf(p.y, vv[i].y, acc[1].y);
            acc[2].x = fmaf(p.z, vv[i].x, acc[2].x); acc[2].y = fmaf(p.z, vv[i].y, acc[2].y);
            acc[3].x = fmaf(p.w, vv[i].x, acc[3].x); acc[3].y = fmaf(p.w, vv[i].y, acc[3].y);
        }
    }
#pragma unroll
    for (int r = 0; r < DF_ROWS; ++r) *reinterpret_cast<float2*>(&red[warp][r][lane * 2]) = acc[r];
    __syncthreads();
    for (int i = tid; i < n_rep * FF_HD; i += DF_THREADS) {
        const int r = i / FF_HD, c = i - r * FF_HD;
        const float o = (red[0][r][c] + red[1][r][c]) + (red[2][r][c] + red[3][r][c]), l = l_s[r];
        const size_t row = (size_t)q0 * nh + g * n_rep + r;
        if (splits == 1) {
            out[row * FF_HD + c] = o * (l > 0.f ? 1.f / l : 0.f);
        } else {
            part_o[(row * splits + sp) * FF_HD + c] = o;
            if (c == 0) { part_ml[(row * splits + sp) * 2] = m_s[r]; part_ml[(row * splits + sp) * 2 + 1] = l; }
        }
    }
}

static int launch_decode_f32(const void* q, long long q_row_stride, const void* cache, const int* block_table, int table_stride,
                             const int* cu_q, const int* seqlens_k, void* out, float* part_o, float* part_ml, int num_seqs, int nh,
                             int nkv, int page_size, int num_pages, float scale, int window, int splits, int* status, cudaStream_t stream) {
    if (nkv > 65535 || (long long)num_seqs * splits > 65535)
        return fail(-1, "paged_attention: %d kv heads or %d sequences x %d splits exceed the grid", nkv, num_seqs, splits);
    return check_launch("paged_attention (float, decode)", launch(decode_f32_kernel, dim3(num_seqs, nkv, splits), dim3(DF_THREADS), 0, stream,
        (const float*)q, q_row_stride, (const float*)cache, block_table, table_stride, cu_q, seqlens_k, (float*)out, part_o, part_ml,
        nh, nkv, page_size, num_pages, scale, window, splits, status));
}

}  // namespace vapi
