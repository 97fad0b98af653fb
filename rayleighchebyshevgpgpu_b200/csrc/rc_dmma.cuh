// rc_dmma.cuh -- FP64 tensor-pipe and cp.async primitives of the tall-skinny products
// (rc_gemm.cu, rc_xt.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace rcb {

__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(c0), "+d"(c1)
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16-byte (two rows) or 8-byte (one row) asynchronous copy global -> shared; bytes beyond
// src_bytes are zero-filled (src_bytes = 0 reads nothing).
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async8(void* dst, const void* src, int src_bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}
__device__ __forceinline__ void cp_async_wait0() { cp_async_wait<0>(); }

// ---- a ring of shared-memory stages filled by one producer warp ------------------------
// full[b] completes when stage b has landed, empty[b] when every consumer warp is done with it. The copies
// are bulk copies (16-byte aligned addresses and sizes), counted in bytes by full[b], or, for data that is
// only 8-byte aligned, cp.async, each lane's arrival following its copies.
__device__ __forceinline__ void mbar_init(uint32_t bar, unsigned count) {
    asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared.b64 t, [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_tx(uint32_t bar, unsigned bytes) {
    asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.expect_tx.shared.b64 t, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, unsigned bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// One tile of a 2-D tensor map, starting at (x, y): x a multiple of 16 bytes, dst of 128. What lies outside reads
// as zero, and the whole tile's bytes are counted.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c, int x, int y, int z,
                                            uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(dst),
        "l"(map), "r"(c), "r"(x), "r"(y), "r"(z), "r"(bar)
        : "memory");
}
// Wait for the phase of the given parity. Bounded (each try suspends for a while by itself): false when the
// limit ran out (6 s: a try takes 1.5 us), which only a lost copy could cause.
constexpr int kMbarTries = 1 << 22;
__device__ __forceinline__ bool mbar_wait(uint32_t bar, unsigned parity) {
    for (int i = 0; i < kMbarTries; ++i) {
        unsigned ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// The same by a whole warp, with one answer for all its lanes.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, unsigned parity) {
    return __all_sync(~0u, mbar_wait(bar, parity));
}

// The driver's cuTensorMapEncodeTiled, through the runtime (no link-time dependency on libcuda), or null.
typedef CUresult (*TensorMapEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                      const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                      CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline TensorMapEncodeFn tensor_map_encode() {
    static TensorMapEncodeFn fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            f = nullptr;
        return (TensorMapEncodeFn)f;
    }();
    return fn;
}

// A tensor map of doubles: `inner` consecutive ones in each of `outer` rows, `ld` apart (ld even, p 16-byte
// aligned), tiles of box_inner x box_outer, not swizzled. False when the driver refuses it.
inline bool tma_map_2d(CUtensorMap* map, const double* p, int64_t inner, int64_t outer, int64_t ld, int box_inner,
                       int box_outer) {
    const TensorMapEncodeFn fn = tensor_map_encode();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)inner, (cuuint64_t)outer};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * sizeof(double)};
    const cuuint32_t box[2] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer}, es[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<double*>(p), dims, strides, box, es,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// A tensor map of 4-D blocks of 32-bit words, dims[0] of them a multiple of 4 (what lies outside reads as zero): dense,
// or the last dimension `outer` words apart.
inline bool tma_map_words_4d(CUtensorMap* map, const void* p, const int64_t (&dims)[4], const int (&box)[4],
                             int64_t outer = 0) {
    const TensorMapEncodeFn fn = tensor_map_encode();
    if (!fn) return false;
    cuuint64_t d[4], st[3];
    cuuint32_t b[4], es[4] = {1, 1, 1, 1};
    for (int k = 0; k < 4; ++k) {
        d[k] = (cuuint64_t)dims[k];
        b[k] = (cuuint32_t)box[k];
        if (k < 3) st[k] = (k ? st[k - 1] : 4) * d[k];
    }
    if (outer) st[2] = (cuuint64_t)outer * 4;
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_INT32, 4, const_cast<void*>(p), d, st, b, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) ==
           CUDA_SUCCESS;
}

}  // namespace rcb
