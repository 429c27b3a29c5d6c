// Building blocks for kernels on the fifth-generation tensor cores (sm_100a): mbarriers with
// bounded waits, TMA tile loads, shared-memory matrix descriptors, tcgen05.mma / commit / ld / st,
// and the host-side tensor-map encoder (taken from the driver at run time, so nothing links
// against libcuda).  Shared by linear_tc.cu and attention_tc.cuh.
#pragma once
#include "common.cuh"
#include <cuda.h>
#include <unordered_map>

namespace vapi {

// polls of an mbarrier before a role gives up (about a second); the caller records a status
// and drains instead of hanging
constexpr unsigned TC5_WAIT_LIMIT = 1u << 24;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// bounded wait on a phase parity; false when the limit ran out
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity) {
    for (unsigned i = 0; i < TC5_WAIT_LIMIT; ++i) {
        unsigned done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
    }
    return false;
}
// the same for a role of a block, which also ends when another role has given up
__device__ __forceinline__ bool mbar_wait_role(unsigned bar, unsigned parity, volatile int* abort_flag, unsigned polls = TC5_WAIT_LIMIT) {
    for (unsigned i = 0; i < polls; ++i) {
        unsigned done;
        asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.b32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(bar), "r"(parity) : "memory");
        if (done) return true;
        if ((i & 0xFFF) == 0xFFF && *abort_flag) break;
    }
    *abort_flag = 1;
    return false;
}
__device__ __forceinline__ void tma_load_2d(unsigned dst, const CUtensorMap* map, unsigned bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                 ::"r"(dst), "l"(map), "r"(bar), "r"(x), "r"(y) : "memory");
}
// shared-memory matrix descriptor: K-major tile of rows of 128 bytes, 128-byte swizzle,
// 8-row groups 1024 bytes apart
__device__ __forceinline__ unsigned long long umma_desc(unsigned smem_addr) {
    unsigned long long d = 0;
    d |= (unsigned long long)((smem_addr >> 4) & 0x3FFF);        // start address
    d |= (unsigned long long)1 << 16;                             // leading byte offset (unused with swizzle)
    d |= (unsigned long long)(1024 >> 4) << 32;                   // stride byte offset: 8 rows * 128 B
    d |= (unsigned long long)1 << 46;                             // descriptor version of this architecture
    d |= (unsigned long long)2 << 61;                             // 128-byte swizzle
    return d;
}
__device__ __forceinline__ void umma_f16(unsigned tmem_d, unsigned long long da, unsigned long long db, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n}"
                 ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(accumulate), "r"(0u) : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(unsigned taddr, float (&v)[16]) {
    unsigned r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
// the same without waiting for the data: issue several, then tmem_ld_wait() once
__device__ __forceinline__ void tmem_ld16_nowait(unsigned taddr, unsigned (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// make shared-memory writes of this thread visible to the async proxy (TMA, tcgen05.mma)
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc5_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc5_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 16 consecutive 32-bit columns of this thread's tensor-memory lane, stored from registers
__device__ __forceinline__ void tmem_st16(unsigned taddr, const float (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
                   "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
                   "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7])), "r"(__float_as_uint(v[8])),
                   "r"(__float_as_uint(v[9])), "r"(__float_as_uint(v[10])), "r"(__float_as_uint(v[11])),
                   "r"(__float_as_uint(v[12])), "r"(__float_as_uint(v[13])), "r"(__float_as_uint(v[14])),
                   "r"(__float_as_uint(v[15])) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// Shared-memory matrix descriptor of an operand whose M/N dimension is the contiguous one
// ("MN-major"): rows of 128 bytes each hold 64 consecutive M/N elements of one k, 128-byte
// swizzle, groups of 8 k-rows 1024 bytes apart.  (A [keys][head_dim] tile of V is this for P.V.)
__device__ __forceinline__ unsigned long long umma_desc_mn(unsigned smem_addr) {
    unsigned long long d = 0;
    d |= (unsigned long long)((smem_addr >> 4) & 0x3FFF);
    d |= (unsigned long long)(1024 >> 4) << 16;                   // leading byte offset: next 64 M/N elements (unused at 64)
    d |= (unsigned long long)(1024 >> 4) << 32;                   // stride byte offset: next group of 8 k-rows
    d |= (unsigned long long)1 << 46;
    d |= (unsigned long long)2 << 61;
    return d;
}

// Two floats as three pairs of bfloat16 that add up to them, high plane first (a in the low half of a pair).  A float has 24 significant bits, a
// bfloat16 eight: the differences are exact, and the last one has at most seven bits left.
__device__ __forceinline__ void split_f32x2(float a, float b, unsigned& p1, unsigned& p2, unsigned& p3) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    p1 = *reinterpret_cast<unsigned*>(&v);
    a -= __uint_as_float(p1 << 16);
    b -= __uint_as_float(p1 & 0xffff0000u);
    v = __floats2bfloat162_rn(a, b);
    p2 = *reinterpret_cast<unsigned*>(&v);
    a -= __uint_as_float(p2 << 16);
    b -= __uint_as_float(p2 & 0xffff0000u);
    v = __floats2bfloat162_rn(a, b);
    p3 = *reinterpret_cast<unsigned*>(&v);
}
// the larger magnitude; a NaN stays one
__device__ __forceinline__ float absmax_nan(float m, float x) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(m), "f"(fabsf(x)));
    return r;
}

// ---- host side -------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)ptr;
    }
    return fn;
}

// A tensor map's arguments; the map is a function of these alone.
struct MapKey {
    const void* p;
    long long rows, k;
    int box, promotion;
    bool operator==(const MapKey& o) const { return p == o.p && rows == o.rows && k == o.k && box == o.box && promotion == o.promotion; }
};
struct MapHash {
    size_t operator()(const MapKey& m) const {
        return std::hash<const void*>()(m.p) ^ (std::hash<long long>()(m.rows) * 31) ^ (std::hash<long long>()(m.k) * 131) ^
               (size_t)(m.box * 8 + m.promotion);
    }
};
static std::unordered_map<MapKey, CUtensorMap, MapHash>& kept_maps() {
    static thread_local std::unordered_map<MapKey, CUtensorMap, MapHash> kept;
    return kept;
}

// A [rows][K] bfloat16 matrix, K contiguous, tiled in boxes of 64 k x box_rows rows, 128-byte swizzle.  keep: for weights, the map is encoded
// once for each thread and not at every call (the driver's encoder takes about a microsecond, and a step of a few tokens is bound by what
// its launches cost the host).  Tokens lie at other addresses from step to step, in other numbers: kept, they would only fill the table.
static int kmajor_map(CUtensorMap* out, const char* what, const void* ptr, long long rows, long long K, int box_rows,
                      CUtensorMapL2promotion promotion, bool keep) {
    auto& kept = kept_maps();
    const MapKey key{ptr, rows, K, box_rows, (int)promotion};
    if (keep) {
        const auto it = kept.find(key);
        if (it != kept.end()) { *out = it->second; return 0; }
    }
    EncodeTiledFn fn = encode_fn();
    if (!fn) return fail(-102, "%s: cuTensorMapEncodeTiled is not available from the driver", what);
    if (((uintptr_t)ptr & 15) != 0 || (K * 2) % 16 != 0)
        return fail(-1, "%s: operand address or row pitch is not 16-byte aligned (K=%lld)", what, K);
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, promotion, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(-103, "%s: cuTensorMapEncodeTiled failed with %d", what, (int)r);
    if (keep) {
        if (kept.size() > 4096) kept.clear();
        try { kept.emplace(key, *out); } catch (...) {}      // (no memory for it: encoded again next time; callers in C know no exceptions)
    }
    return 0;
}

}  // namespace vapi
