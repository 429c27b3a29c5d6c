// Paged GQA attention for prompt portions of the true 32-bit path: float queries, keys and values, head_dim 64, pages whose
// size is a multiple of 64.  Same rows, masks and partial results as the general kernel of attention.cu, which it replaces
// for steps of more than 16 rows per (sequence, kv head): 1,024 tokens, 32 / 8 heads, took that kernel 403 us, almost all of it
// float FMAs fed from shared memory.
//
// Both products run on the tensor cores without giving up float: a float is the exact sum of three bfloat16 (24 bits), and of
// the nine products the six of weight 2^-16 and above are taken (the rest is below 2^-25 of the term; see linear_f32.cu).
// The leading products and the five small ones have accumulators of their own, and a tile's P.V is added to the output by
// float FMAs: a tensor core cuts off what it adds to an accumulator, so chains are kept to four instructions.  Maximum,
// exponentials and sums are float as before.
//
// A block of four warps owns 64 rows and walks the 64-key tiles any of them can see: the tile's floats come by asynchronous copies
// while the tile before is multiplied, all threads split them into planes (128-byte rows, 16-byte pieces swizzled), a warp
// takes 16 rows.  106 KB of shared memory and two blocks a multiprocessor, so that one block splits while the other
// multiplies.  A tile with an infinity, a NaN or a magnitude of 2^127 and more, which have no such planes, is computed by FMAs.
#pragma once
#include "attention_mma.cuh"
#include "attention_tc.cuh"        // ft_tile

namespace vapi {

constexpr int FF_ROWS = 64, FF_BK = 64, FF_HD = 64, FF_THREADS = 128;
constexpr int FF_PLANE = FF_BK * FF_HD * 2;
constexpr size_t FF_SMEM = 9 * FF_PLANE + 2 * FF_BK * FF_HD * 4 + 128;     // planes of Q, K, V; floats of K, V
constexpr float FF_LIMIT = 1.7014118346046923e38f;                         // 2^127

__device__ __forceinline__ void ff_split2(float a, float b, unsigned& p1, unsigned& p2, unsigned& p3) {
    p1 = pack_bf16(a, b);
    a -= __uint_as_float(p1 << 16);
    b -= __uint_as_float(p1 & 0xffff0000u);
    p2 = pack_bf16(a, b);
    a -= __uint_as_float(p2 << 16);
    b -= __uint_as_float(p2 & 0xffff0000u);
    p3 = pack_bf16(a, b);
}
__device__ __forceinline__ float ff_absmax(float m, float x) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(m), "f"(fabsf(x)));
    return r;
}
// four floats of a row (piece c4 of 16 bytes of float) into the three planes; the largest magnitude so far
__device__ __forceinline__ float ff_store(unsigned char* planes, int row, int c4, float4 v, float top) {
    uint2 p1, p2, p3;
    ff_split2(v.x, v.y, p1.x, p2.x, p3.x);
    ff_split2(v.z, v.w, p1.y, p2.y, p3.y);
    unsigned char* at = planes + row * 128 + ((((c4 >> 1) ^ (row & 7)) << 4) | ((c4 & 1) << 3));
    *reinterpret_cast<uint2*>(at) = p1;
    *reinterpret_cast<uint2*>(at + FF_PLANE) = p2;
    *reinterpret_cast<uint2*>(at + 2 * FF_PLANE) = p3;
    return ff_absmax(ff_absmax(ff_absmax(ff_absmax(top, v.x), v.y), v.z), v.w);
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
    const int g = blockIdx.y, sp = blockIdx.z, n_rep = nh / nkv;
    pdl_trigger();
    int s = 0, tile = 0;
    const bool mine = ft_tile(cu_q, num_seqs, 1, n_rep, FF_ROWS, (int)blockIdx.x, s, tile);
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
        float top = qtop;
#pragma unroll 4
        for (int i = tid; i < FF_BK * FF_HD / 4; i += FF_THREADS) {
            top = ff_store(sK, i >> 4, i & 15, *reinterpret_cast<const float4*>(fK + i * 4), top);
            top = ff_store(sV, i >> 4, i & 15, *reinterpret_cast<const float4*>(fV + i * 4), top);
        }
        const bool plain = __syncthreads_or(!(top < FF_LIMIT)) != 0;
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
                ff_split2(sc[2 * k][0], sc[2 * k][1], a[0][0], a[1][0], a[2][0]);
                ff_split2(sc[2 * k][2], sc[2 * k][3], a[0][1], a[1][1], a[2][1]);
                ff_split2(sc[2 * k + 1][0], sc[2 * k + 1][1], a[0][2], a[1][2], a[2][2]);
                ff_split2(sc[2 * k + 1][2], sc[2 * k + 1][3], a[0][3], a[1][3], a[2][3]);
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
                    for (int k = 0; k < FF_BK; ++k) d = fmaf(pr[k], fV[k * FF_HD + n * 8 + p4 + (i & 1)], d);
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
    if (tiles > 0x7fffffffLL || nkv > 65535 || (long long)num_seqs * splits > 65535)
        return fail(-1, "paged_attention: %d kv heads or %d sequences x %d splits exceed the grid", nkv, num_seqs, splits);
    static bool attr_set = false;
    if (!attr_set) {
        cudaError_t e = cudaFuncSetAttribute(flash_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FF_SMEM);
        if (e != cudaSuccess) return fail(-101, "paged_attention: cannot reserve %zu bytes of shared memory: %s", FF_SMEM, cudaGetErrorString(e));
        attr_set = true;
    }
    return check_launch("paged_attention (float)", launch(flash_f32_kernel, dim3((unsigned)tiles, nkv, splits), dim3(FF_THREADS), FF_SMEM, stream,
        (const float*)q, q_row_stride, (const float*)cache, block_table, table_stride, cu_q, seqlens_k, (float*)out, part_o, part_ml,
        num_seqs, nh, nkv, page_size, num_pages, scale, window, splits, status));
}

}  // namespace vapi
