// Rotary position tables for a step, and the fused per-head q/k RMSNorm + RoPE +
// paged K/V write that follows the q/k/v projection.
//
// Reference behaviour: inv_freq_i = 1 / theta^(2i/d) and angle = p * inv_freq_i in
// float (crates/vapi-backend-candle/src/models/lfm2.rs:163-183); per-head RMSNorm of
// q and k, then rotate-half RoPE (pairs (i, i + d/2)), then the roped-normed k and
// the raw v go to the token's cache slot (lfm2.rs:343-375).  Here the angles, the
// norm and the rotation are float end to end with one rounding at the store.
#include "common.cuh"

using namespace vapi;

// cos/sin rows for the step's tokens: [n, half] each, float.
__global__ void rope_cos_sin_kernel(const int* __restrict__ positions,
                                    const float* __restrict__ inv_freq,
                                    float* __restrict__ cosr, float* __restrict__ sinr,
                                    int n, int half) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_trigger();
    pdl_wait();
    if (i >= n * half) return;
    const int t = i / half, j = i - t * half;
    const float a = (float)positions[t] * inv_freq[j];
    cosr[i] = cosf(a);
    sinr[i] = sinf(a);
}

VAPI_EXPORT int vapi_rope_cos_sin(const int* positions, const float* inv_freq, float* cosr,
                                  float* sinr, int n, int half, cudaStream_t stream) {
    if (n <= 0 || half <= 0) return 0;
    const int total = n * half;
    return check_launch("rope_cos_sin", launch(rope_cos_sin_kernel, (total + 255) / 256, 256, 0, stream,
                                                 positions, inv_freq, cosr, sinr, n, half));
}

// One warp per (token, head).  Heads are laid out in a qkv row as
// [q heads | k heads | v heads], each head_dim wide.
//   q: norm (if qw) -> rope (if cosr) -> written back in place
//   k: norm (if kw) -> rope (if cosr) -> written to the cache slot (if cache)
//   v: copied to the cache slot (if cache)
// Cache layer layout: [num_pages, 2 (k,v), n_kv, page_size, head_dim].
constexpr int QK_WARPS = 4;
constexpr int QK_MAX_D = 256;

template <typename T>
__global__ void qk_norm_rope_write_kernel(T* __restrict__ qkv, const float* __restrict__ qw,
                                          const float* __restrict__ kw, float eps,
                                          const float* __restrict__ cosr,
                                          const float* __restrict__ sinr, int rot,
                                          T* __restrict__ cache,
                                          const int* __restrict__ slot_mapping, int n, int nh,
                                          int nkv, int d, int page_size, int num_pages,
                                          int* __restrict__ status) {
    __shared__ float sh[QK_WARPS][QK_MAX_D];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int heads = nh + 2 * nkv;
    const long long item = (long long)blockIdx.x * QK_WARPS + warp;
    pdl_trigger();
    if (item >= (long long)n * heads) {
        pdl_wait();
        return;
    }
    const int t = (int)(item / heads), h = (int)(item - (long long)t * heads);
    const int slot_pre = (cache && h >= nh) ? slot_mapping[t] : 0;     // host-copied index data: safe before the wait
    pdl_wait();
    T* src = qkv + (size_t)t * heads * d + (size_t)h * d;
    const bool is_q = h < nh, is_k = !is_q && h < nh + nkv;
    const float* w = is_q ? qw : (is_k ? kw : nullptr);
    const bool rope = (is_q || is_k) && cosr != nullptr;
    float* s = sh[warp];

    float ss = 0.f;
    for (int i = lane; i < d; i += 32) {
        const float v = to_f32(src[i]);
        s[i] = v;
        ss += v * v;
    }
    float inv = 1.f;
    if (w) {
        ss = warp_sum(ss);
        inv = rsqrtf(ss / (float)d + eps);
    }
    __syncwarp();

    T* dst = nullptr;
    if (is_q) {
        dst = src;
    } else if (cache) {
        const int slot = slot_pre;
        const int page = slot / page_size, off = slot - page * page_size;
        if (slot < 0 || page >= num_pages) {
            if (lane == 0 && status) atomicExch(status, 2);
            return;
        }
        const int g = is_k ? h - nh : h - nh - nkv;
        dst = cache + ((((size_t)page * 2 + (is_k ? 0 : 1)) * nkv + g) * page_size + off) * d;
    }
    if (!dst) return;

    const int half = rot >> 1;
    for (int i = lane; i < d; i += 32) {
        float v = w ? s[i] * inv * w[i] : s[i];
        if (rope && i < rot) {
            const int j = i < half ? i : i - half;
            const int pi = i < half ? i + half : i - half;
            const float pv = w ? s[pi] * inv * w[pi] : s[pi];
            const float c = cosr[(size_t)t * half + j], sn = sinr[(size_t)t * half + j];
            v = i < half ? v * c - pv * sn : v * c + pv * sn;
        }
        dst[i] = from_f32<T>(v);
    }
}

// The same work with 16-byte accesses, for a rotation over the whole head (rot == d) and a
// half head that 16-byte groups tile evenly: a group of G = (d/2) / VEC lanes (a power of two)
// takes one (token, head); each lane holds VEC elements of the first half and their rotation
// partners in the second half, so no shared memory is needed.
template <typename T> struct Pack16;
template <> struct Pack16<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
        const float4 f = *reinterpret_cast<const float4*>(p);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    }
    static __device__ __forceinline__ void store(float* p, const float (&v)[4]) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    }
};
template <> struct Pack16<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[8]) {
        const uint4 u = *reinterpret_cast<const uint4*>(p);
        const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w[i]));
            v[2 * i] = f.x;
            v[2 * i + 1] = f.y;
        }
    }
    static __device__ __forceinline__ void store(__nv_bfloat16* p, const float (&v)[8]) {
        unsigned w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            __nv_bfloat162 a = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
            w[i] = *reinterpret_cast<unsigned*>(&a);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
    }
};

template <typename T>
__global__ void qk_norm_rope_write_vec_kernel(T* __restrict__ qkv, const float* __restrict__ qw,
                                              const float* __restrict__ kw, float eps,
                                              const float* __restrict__ cosr,
                                              const float* __restrict__ sinr, T* __restrict__ cache,
                                              const int* __restrict__ slot_mapping, int n, int nh,
                                              int nkv, int d, int page_size, int num_pages, int G,
                                              int* __restrict__ status) {
    constexpr int VEC = Pack16<T>::N;
    const int heads = nh + 2 * nkv, half = d >> 1;
    const long long gl = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long item = gl / G;
    const int sub = (int)(gl - item * G);
    const bool active = item < (long long)n * heads;     // whole groups are active or not
    const int t = active ? (int)(item / heads) : 0, h = active ? (int)(item - (long long)t * heads) : 0;
    pdl_trigger();
    const bool is_q = h < nh, is_k = !is_q && h < nh + nkv;
    const int slot = (active && cache && !is_q) ? slot_mapping[t] : 0;     // host-copied index data
    const float* w = is_q ? qw : (is_k ? kw : nullptr);
    const bool rope = (is_q || is_k) && cosr != nullptr;
    const int e = sub * VEC;                               // this lane's elements: e.. and half+e..
    float wl[VEC], wh[VEC];
    if (w) {
#pragma unroll
        for (int i = 0; i < VEC; i += 4) {
            const float4 a = *reinterpret_cast<const float4*>(w + e + i);
            const float4 b = *reinterpret_cast<const float4*>(w + half + e + i);
            wl[i] = a.x; wl[i + 1] = a.y; wl[i + 2] = a.z; wl[i + 3] = a.w;
            wh[i] = b.x; wh[i + 1] = b.y; wh[i + 2] = b.z; wh[i + 3] = b.w;
        }
    }
    pdl_wait();         // the row and the cos/sin tables come from kernels of this step
    float c[VEC], sn[VEC];
    if (rope && active) {
#pragma unroll
        for (int i = 0; i < VEC; i += 4) {
            const float4 a = *reinterpret_cast<const float4*>(cosr + (size_t)t * half + e + i);
            const float4 b = *reinterpret_cast<const float4*>(sinr + (size_t)t * half + e + i);
            c[i] = a.x; c[i + 1] = a.y; c[i + 2] = a.z; c[i + 3] = a.w;
            sn[i] = b.x; sn[i + 1] = b.y; sn[i + 2] = b.z; sn[i + 3] = b.w;
        }
    }
    T* src = qkv + (size_t)t * heads * d + (size_t)h * d;
    float lo[VEC], hi[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) lo[i] = hi[i] = 0.f;
    if (active) {
        Pack16<T>::load(src + e, lo);
        Pack16<T>::load(src + half + e, hi);
    }
    float inv = 1.f;
    if (qw || kw) {     // (uniform over the warp: every lane takes part in the shuffles)
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < VEC; ++i) ss += lo[i] * lo[i] + hi[i] * hi[i];
        for (int o = G >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        inv = rsqrtf(ss / (float)d + eps);
    }
    if (!active) return;
    T* dst = nullptr;
    if (is_q) {
        dst = src;
    } else if (cache) {
        const int page = slot / page_size, off = slot - page * page_size;
        if (slot < 0 || page >= num_pages) {
            if (sub == 0 && status) atomicExch(status, 2);
            return;
        }
        const int g = is_k ? h - nh : h - nh - nkv;
        dst = cache + ((((size_t)page * 2 + (is_k ? 0 : 1)) * nkv + g) * page_size + off) * d;
    }
    if (!dst) return;
    if (w) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            lo[i] = lo[i] * inv * wl[i];
            hi[i] = hi[i] * inv * wh[i];
        }
    }
    if (rope) {
#pragma unroll
        for (int i = 0; i < VEC; ++i) {
            const float a = lo[i], b = hi[i];
            lo[i] = a * c[i] - b * sn[i];
            hi[i] = b * c[i] + a * sn[i];
        }
    }
    Pack16<T>::store(dst + e, lo);
    Pack16<T>::store(dst + half + e, hi);
}

VAPI_EXPORT int vapi_qk_norm_rope_write(void* qkv, int dtype, const float* qw, const float* kw,
                                        float eps, const float* cosr, const float* sinr, int rot,
                                        void* cache, const int* slot_mapping, int n, int nh,
                                        int nkv, int d, int page_size, int num_pages,
                                        int* status, cudaStream_t stream) {
    if (n <= 0) return 0;
    if (d <= 0 || d > QK_MAX_D || (d % 2) != 0)
        return fail(-1, "qk_norm_rope_write: head_dim %d is not an even size up to %d", d, QK_MAX_D);
    if (cosr && (rot <= 0 || rot > d || (rot % 2) != 0))
        return fail(-1, "qk_norm_rope_write: rotary width %d does not fit head_dim %d", rot, d);
    if (nh <= 0 || nkv < 0) return fail(-1, "qk_norm_rope_write: bad head counts %d/%d", nh, nkv);
    if (cache && (page_size <= 0 || num_pages <= 0 || !slot_mapping))
        return fail(-1, "qk_norm_rope_write: cache given without pages or slot mapping");
    const long long items = (long long)n * (nh + 2 * nkv);
    const int blocks = (int)((items + QK_WARPS - 1) / QK_WARPS);
    cudaError_t e;
    {
        // 16-byte form: whole-head rotation (or none) and half a head tiled by 16-byte groups
        const int vec = dtype == VAPI_BF16 ? 8 : 4;
        const int half = d / 2;
        const int G = half % vec == 0 ? half / vec : 0;
        if ((dtype == VAPI_BF16 || dtype == VAPI_F32) && (!cosr || rot == d) && G >= 1 && G <= 32 && (G & (G - 1)) == 0) {
            const long long lanes = items * G;
            const int vblocks = (int)((lanes + 127) / 128);
            if (dtype == VAPI_F32)
                e = launch(qk_norm_rope_write_vec_kernel<float>, vblocks, 128, 0, stream, (float*)qkv, qw, kw, eps,
                           cosr, sinr, (float*)cache, slot_mapping, n, nh, nkv, d, page_size, num_pages, G, status);
            else
                e = launch(qk_norm_rope_write_vec_kernel<__nv_bfloat16>, vblocks, 128, 0, stream,
                           (__nv_bfloat16*)qkv, qw, kw, eps, cosr, sinr, (__nv_bfloat16*)cache, slot_mapping, n,
                           nh, nkv, d, page_size, num_pages, G, status);
            return check_launch("qk_norm_rope_write", e);
        }
    }
    if (dtype == VAPI_F32)
        e = launch(qk_norm_rope_write_kernel<float>, blocks, QK_WARPS * 32, 0, stream,
                   (float*)qkv, qw, kw, eps, cosr, sinr, rot, (float*)cache, slot_mapping, n, nh, nkv, d,
                   page_size, num_pages, status);
    else if (dtype == VAPI_BF16)
        e = launch(qk_norm_rope_write_kernel<__nv_bfloat16>, blocks, QK_WARPS * 32, 0, stream,
                   (__nv_bfloat16*)qkv, qw, kw, eps, cosr, sinr, rot, (__nv_bfloat16*)cache,
                   slot_mapping, n, nh, nkv, d, page_size, num_pages, status);
    else
        return fail(-2, "qk_norm_rope_write: unsupported dtype %d", dtype);
    return check_launch("qk_norm_rope_write", e);
}


// cos/sin rows from per-pair frequencies that the host has already scaled (a frequency
// interpolation such as YaRN changes the frequencies and multiplies both tables by one number).
__global__ void rope_cos_sin_scaled_kernel(const int* __restrict__ positions, const float* __restrict__ freq,
                                           float mult, float* __restrict__ cosr, float* __restrict__ sinr,
                                           int n, int half) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_trigger();
    pdl_wait();
    if (i >= n * half) return;
    const int t = i / half, j = i - t * half;
    const float a = (float)positions[t] * freq[j];
    cosr[i] = cosf(a) * mult;
    sinr[i] = sinf(a) * mult;
}

VAPI_EXPORT int vapi_rope_cos_sin_scaled(const int* positions, const float* freq, float mult, float* cosr,
                                         float* sinr, int n, int half, cudaStream_t stream) {
    if (n <= 0 || half <= 0) return 0;
    const int total = n * half;
    return check_launch("rope_cos_sin_scaled", launch(rope_cos_sin_scaled_kernel, (total + 255) / 256, 256, 0, stream,
                                                        positions, freq, mult, cosr, sinr, n, half));
}

// The general form of the kernel above: keys of width dk and values of width dv in a row
// [q heads x dk | k heads x dk | v heads x dv | anything else] of `row_stride` elements; the rotation
// pairs either (i, i + rot/2) (rotate-half) or (2i, 2i+1) (interleaved) over the first `rot`
// elements of a head; a cache page holds the keys [nkv, page_size, dk] and then the values
// [nkv, page_size, dv].  One warp per (token, head).
template <typename T>
__global__ void qk_norm_rope_write_split_kernel(T* __restrict__ qkv, long long row_stride, const float* __restrict__ qw,
                                                const float* __restrict__ kw, float eps,
                                                const float* __restrict__ cosr, const float* __restrict__ sinr,
                                                int rot, int interleaved, T* __restrict__ cache,
                                                const int* __restrict__ slot_mapping, int n, int nh, int nkv,
                                                int dk, int dv, int page_size, int num_pages,
                                                int* __restrict__ status, const int* __restrict__ positions,
                                                float qt_coef, int qt_every) {
    __shared__ float sh[QK_WARPS][QK_MAX_D];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int heads = nh + 2 * nkv;
    const long long item = (long long)blockIdx.x * QK_WARPS + warp;
    pdl_trigger();
    if (item >= (long long)n * heads) {
        pdl_wait();
        return;
    }
    const int t = (int)(item / heads), h = (int)(item - (long long)t * heads);
    const int slot = (cache && h >= nh) ? slot_mapping[t] : 0;
    pdl_wait();
    const bool is_q = h < nh, is_k = !is_q && h < nh + nkv;
    const int d = (is_q || is_k) ? dk : dv;
    T* src = qkv + (size_t)t * row_stride + (is_q || is_k ? (size_t)h * dk : (size_t)(nh + nkv) * dk + (size_t)(h - nh - nkv) * dv);
    const float* w = is_q ? qw : (is_k ? kw : nullptr);
    const bool rope = (is_q || is_k) && cosr != nullptr;
    // a query temperature: q at position p is multiplied by 1 + coef * ln(floor((p + 1) / every) + 1)
    const float q_mult = (is_q && qt_every > 0) ? 1.f + qt_coef * logf((float)((positions[t] + 1) / qt_every + 1)) : 1.f;
    float* s = sh[warp];
    float ss = 0.f;
    for (int i = lane; i < d; i += 32) {
        const float v = to_f32(src[i]);
        s[i] = v;
        ss += v * v;
    }
    float inv = 1.f;
    if (w) {
        ss = warp_sum(ss);
        inv = rsqrtf(ss / (float)d + eps);
    }
    __syncwarp();
    T* dst = nullptr;
    if (is_q) {
        if (!w && !rope && q_mult == 1.f) return;      // nothing changes a query that is neither normed, rotated nor scaled
        dst = src;
    } else if (cache) {
        const int page = slot / page_size, off = slot - page * page_size;
        if (slot < 0 || page >= num_pages) {
            if (lane == 0 && status) atomicExch(status, 2);
            return;
        }
        const size_t page_elems = (size_t)nkv * page_size * (dk + dv);
        dst = is_k ? cache + (size_t)page * page_elems + ((size_t)(h - nh) * page_size + off) * dk
                   : cache + (size_t)page * page_elems + (size_t)nkv * page_size * dk + ((size_t)(h - nh - nkv) * page_size + off) * dv;
    }
    if (!dst) return;
    const int half = rot >> 1;
    for (int i = lane; i < d; i += 32) {
        float v = w ? s[i] * inv * w[i] : s[i];
        if (rope && i < rot) {
            int j, pi;
            bool first;
            if (interleaved) {
                j = i >> 1; first = (i & 1) == 0; pi = i ^ 1;
            } else {
                first = i < half; j = first ? i : i - half; pi = first ? i + half : i - half;
            }
            const float pv = w ? s[pi] * inv * w[pi] : s[pi];
            const float c = cosr[(size_t)t * half + j], sn = sinr[(size_t)t * half + j];
            v = first ? v * c - pv * sn : v * c + pv * sn;
        }
        dst[i] = from_f32<T>(v * q_mult);
    }
}

// The same for heads of 64: a lane has the elements `lane` and `lane + 32` in registers, and an element's partner in the rotation is
// the neighbouring lane's (interleaved pairs) or its own other one (halves of 32), so nothing goes through shared memory, and a
// warp's loads are all on their way at once.  The sums in the same order.  2,000 tokens of 32 / 8 heads in bfloat16: 34.9 us, so 26.1.
template <typename T>
__global__ void __launch_bounds__(256)
qk_norm_rope_write_split64_kernel(T* __restrict__ qkv, long long row_stride, const float* __restrict__ qw,
                                  const float* __restrict__ kw, float eps, const float* __restrict__ cosr,
                                  const float* __restrict__ sinr, int rot, int interleaved, T* __restrict__ cache,
                                  const int* __restrict__ slot_mapping, int n, int nh, int nkv, int page_size, int num_pages,
                                  int* __restrict__ status, const int* __restrict__ positions, float qt_coef, int qt_every) {
    constexpr int D = 64;
    const int lane = threadIdx.x & 31, heads = nh + 2 * nkv;
    const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    pdl_trigger();
    if (item >= n * heads) {
        pdl_wait();
        return;
    }
    const int t = item / heads, h = item - t * heads;
    const int slot = (cache && h >= nh) ? slot_mapping[t] : 0;
    const bool is_q = h < nh, is_k = !is_q && h < nh + nkv;
    const float* w = is_q ? qw : (is_k ? kw : nullptr);
    const bool rope = (is_q || is_k) && cosr != nullptr;
    // a query temperature: q at position p is multiplied by 1 + coef * ln(floor((p + 1) / every) + 1)
    const float q_mult = (is_q && qt_every > 0) ? 1.f + qt_coef * logf((float)((positions[t] + 1) / qt_every + 1)) : 1.f;
    const float w0 = w ? w[lane] : 1.f, w1 = w ? w[lane + 32] : 1.f;
    pdl_wait();
    T* src = qkv + (size_t)t * row_stride + (size_t)h * D;
    float v0 = to_f32(src[lane]), v1 = to_f32(src[lane + 32]);
    const int half = rot >> 1;
    // of element i: the pair's index, and whether it is the first of its pair
    const int j0 = interleaved ? lane >> 1 : lane, j1 = interleaved ? (lane + 32) >> 1 : lane;
    const bool r0 = rope && lane < rot, r1 = rope && lane + 32 < rot;
    float c0 = 1.f, s0 = 0.f, c1 = 1.f, s1 = 0.f;
    if (r0) { c0 = cosr[(size_t)t * half + j0]; s0 = sinr[(size_t)t * half + j0]; }
    if (r1) { c1 = cosr[(size_t)t * half + j1]; s1 = sinr[(size_t)t * half + j1]; }
    T* dst = nullptr;
    if (is_q) {
        if (!w && !rope && q_mult == 1.f) return;      // nothing changes a query that is neither normed, rotated nor scaled
        dst = src;
    } else if (cache) {
        const int page = slot / page_size, off = slot - page * page_size;
        if (slot < 0 || page >= num_pages) {
            if (lane == 0 && status) atomicExch(status, 2);
            return;
        }
        const size_t page_elems = (size_t)nkv * page_size * (2 * D);
        dst = is_k ? cache + (size_t)page * page_elems + ((size_t)(h - nh) * page_size + off) * D
                   : cache + (size_t)page * page_elems + (size_t)nkv * page_size * D + ((size_t)(h - nh - nkv) * page_size + off) * D;
    }
    if (!dst) return;
    if (w) {
        float ss = 0.f;
        ss += v0 * v0;
        ss += v1 * v1;
        ss = warp_sum(ss);
        const float inv = rsqrtf(ss / (float)D + eps);
        v0 = v0 * inv * w0;
        v1 = v1 * inv * w1;
    }
    if (rope) {                                        // (the same for the whole warp)
        const float p0 = interleaved ? __shfl_xor_sync(0xffffffffu, v0, 1) : v1, p1 = interleaved ? __shfl_xor_sync(0xffffffffu, v1, 1) : v0;
        const bool first0 = interleaved ? (lane & 1) == 0 : true, first1 = interleaved ? (lane & 1) == 0 : false;
        const float a0 = first0 ? v0 * c0 - p0 * s0 : v0 * c0 + p0 * s0, a1 = first1 ? v1 * c1 - p1 * s1 : v1 * c1 + p1 * s1;
        if (r0) v0 = a0;
        if (r1) v1 = a1;
    }
    dst[lane] = from_f32<T>(v0 * q_mult);
    dst[lane + 32] = from_f32<T>(v1 * q_mult);
}

// The same work where the RMS norm of q (and of k) runs over the whole projection of a token, all heads at
// once, with a weight per element of the projection (qw [nh * dk], kw [nkv * dk]); eps inside the root.  One
// block per token: every thread adds up its share of the squares of q and of k in a fixed order, the block
// sums them, and then the warps share out the heads: q is normed (and rotated) in place, k and v go to the
// page.  The sums depend on the token's row alone, never on what else is in the step.
template <typename T>
__global__ void qk_norm_whole_write_split_kernel(T* __restrict__ qkv, long long row_stride, const float* __restrict__ qw,
                                                 const float* __restrict__ kw, float eps,
                                                 const float* __restrict__ cosr, const float* __restrict__ sinr,
                                                 int rot, int interleaved, T* __restrict__ cache,
                                                 const int* __restrict__ slot_mapping, int n, int nh, int nkv,
                                                 int dk, int dv, int page_size, int num_pages,
                                                 int* __restrict__ status) {
    __shared__ float sh[QK_WARPS][QK_MAX_D];
    __shared__ float red[33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x;
    pdl_trigger();
    if (t >= n) {
        pdl_wait();
        return;
    }
    const int slot = cache ? slot_mapping[t] : 0;
    pdl_wait();
    T* row = qkv + (size_t)t * row_stride;
    const int q_len = nh * dk, k_len = nkv * dk;
    float ssq = 0.f, ssk = 0.f;
    for (int i = threadIdx.x; i < q_len; i += blockDim.x) {
        const float v = to_f32(row[i]);
        ssq = fmaf(v, v, ssq);
    }
    for (int i = threadIdx.x; i < k_len; i += blockDim.x) {
        const float v = to_f32(row[q_len + i]);
        ssk = fmaf(v, v, ssk);
    }
    ssq = block_sum(ssq, red);
    ssk = block_sum(ssk, red);
    const float inv_q = qw ? rsqrtf(ssq / (float)q_len + eps) : 1.f;
    const float inv_k = kw ? rsqrtf(ssk / (float)max(k_len, 1) + eps) : 1.f;
    int page = 0, off = 0;
    if (cache) {
        page = slot / page_size;
        off = slot - page * page_size;
        if (slot < 0 || page >= num_pages) {
            if (threadIdx.x == 0 && status) atomicExch(status, 2);
            return;
        }
    }
    const int heads = nh + 2 * nkv;
    const int half = rot >> 1;
    const size_t page_elems = (size_t)nkv * page_size * (dk + dv);
    float* s = sh[warp];
    for (int h = warp; h < heads; h += QK_WARPS) {
        const bool is_q = h < nh, is_k = !is_q && h < nh + nkv;
        const int d = (is_q || is_k) ? dk : dv;
        T* src = row + (is_q || is_k ? (size_t)h * dk : (size_t)(nh + nkv) * dk + (size_t)(h - nh - nkv) * dv);
        const float* w = is_q ? (qw ? qw + (size_t)h * dk : nullptr) : (is_k && kw ? kw + (size_t)(h - nh) * dk : nullptr);
        const float inv = is_q ? inv_q : inv_k;
        const bool rope = (is_q || is_k) && cosr != nullptr;
        T* dst = nullptr;
        if (is_q) dst = src;
        else if (cache)
            dst = is_k ? cache + (size_t)page * page_elems + ((size_t)(h - nh) * page_size + off) * dk
                       : cache + (size_t)page * page_elems + (size_t)nkv * page_size * dk + ((size_t)(h - nh - nkv) * page_size + off) * dv;
        if (!dst) continue;
        __syncwarp();
        for (int i = lane; i < d; i += 32) s[i] = to_f32(src[i]);
        __syncwarp();
        for (int i = lane; i < d; i += 32) {
            float v = w ? s[i] * inv * w[i] : s[i];
            if (rope && i < rot) {
                int j, pi;
                bool first;
                if (interleaved) {
                    j = i >> 1; first = (i & 1) == 0; pi = i ^ 1;
                } else {
                    first = i < half; j = first ? i : i - half; pi = first ? i + half : i - half;
                }
                const float pv = w ? s[pi] * inv * w[pi] : s[pi];
                const float c = cosr[(size_t)t * half + j], sn = sinr[(size_t)t * half + j];
                v = first ? v * c - pv * sn : v * c + pv * sn;
            }
            dst[i] = from_f32<T>(v);
        }
    }
}


VAPI_EXPORT int vapi_qk_norm_rope_write_split(void* qkv, long long row_stride, int dtype, const float* qw, const float* kw,
                                              float eps, const float* cosr, const float* sinr, int rot, int interleaved,
                                              void* cache, const int* slot_mapping, int n, int nh, int nkv, int dk,
                                              int dv, int page_size, int num_pages, int whole, int* status,
                                              cudaStream_t stream, const int* positions, float qt_coef, int qt_every) {
    if (n <= 0) return 0;
    if (qt_every < 0 || (qt_every > 0 && (!positions || whole)))
        return fail(-1, "qk_norm_rope_write_split: a query temperature needs the positions and norms per head");
    if (dk <= 0 || dk > QK_MAX_D || dv <= 0 || dv > QK_MAX_D)
        return fail(-1, "qk_norm_rope_write_split: head sizes %d/%d are outside 1..%d", dk, dv, QK_MAX_D);
    if (cosr && (rot <= 0 || rot > dk || (rot % 2) != 0))
        return fail(-1, "qk_norm_rope_write_split: rotary width %d does not fit head size %d", rot, dk);
    if (nh <= 0 || nkv < 0) return fail(-1, "qk_norm_rope_write_split: bad head counts %d/%d", nh, nkv);
    if (row_stride < (long long)(nh + nkv) * dk + (long long)nkv * dv)
        return fail(-1, "qk_norm_rope_write_split: a row of %lld elements cannot hold the heads", row_stride);
    if (cache && (page_size <= 0 || num_pages <= 0 || !slot_mapping))
        return fail(-1, "qk_norm_rope_write_split: cache given without pages or slot mapping");
    const long long items = (long long)n * (nh + 2 * nkv);
    const int blocks = (int)((items + QK_WARPS - 1) / QK_WARPS);
    cudaError_t e;
    if (whole) {                 // the norms run over a token's whole q and k: a block per token
        if (dtype == VAPI_F32)
            e = launch(qk_norm_whole_write_split_kernel<float>, n, QK_WARPS * 32, 0, stream, (float*)qkv, row_stride, qw, kw,
                       eps, cosr, sinr, rot, interleaved, (float*)cache, slot_mapping, n, nh, nkv, dk, dv, page_size,
                       num_pages, status);
        else if (dtype == VAPI_BF16)
            e = launch(qk_norm_whole_write_split_kernel<__nv_bfloat16>, n, QK_WARPS * 32, 0, stream, (__nv_bfloat16*)qkv,
                       row_stride, qw, kw, eps, cosr, sinr, rot, interleaved, (__nv_bfloat16*)cache, slot_mapping, n, nh,
                       nkv, dk, dv, page_size, num_pages, status);
        else
            return fail(-2, "qk_norm_rope_write_split: unsupported dtype %d", dtype);
        return check_launch("qk_norm_rope_write_split (whole projection)", e);
    }
    if (dk == 64 && dv == 64 && (!cosr || interleaved || rot == 64) && items <= 0x7fffffffLL - 8 && (dtype == VAPI_F32 || dtype == VAPI_BF16)) {
        const int blocks64 = (int)((items + 7) / 8);
#define QK_64(T)                                                                                                              \
    launch(qk_norm_rope_write_split64_kernel<T>, blocks64, 256, 0, stream, (T*)qkv, row_stride, qw, kw, eps, cosr, sinr, rot, \
           interleaved, (T*)cache, slot_mapping, n, nh, nkv, page_size, num_pages, status, positions, qt_coef, qt_every)
        e = dtype == VAPI_F32 ? QK_64(float) : QK_64(__nv_bfloat16);
#undef QK_64
        return check_launch("qk_norm_rope_write_split", e);
    }
    if (dtype == VAPI_F32)
        e = launch(qk_norm_rope_write_split_kernel<float>, blocks, QK_WARPS * 32, 0, stream, (float*)qkv, row_stride, qw, kw, eps,
                   cosr, sinr, rot, interleaved, (float*)cache, slot_mapping, n, nh, nkv, dk, dv, page_size, num_pages, status,
                   positions, qt_coef, qt_every);
    else if (dtype == VAPI_BF16)
        e = launch(qk_norm_rope_write_split_kernel<__nv_bfloat16>, blocks, QK_WARPS * 32, 0, stream, (__nv_bfloat16*)qkv,
                   row_stride, qw, kw, eps, cosr, sinr, rot, interleaved, (__nv_bfloat16*)cache, slot_mapping, n, nh, nkv,
                   dk, dv, page_size, num_pages, status, positions, qt_coef, qt_every);
    else
        return fail(-2, "qk_norm_rope_write_split: unsupported dtype %d", dtype);
    return check_launch("qk_norm_rope_write_split", e);
}

VAPI_EXPORT const char* vapi_last_error() { return error_buffer(); }
