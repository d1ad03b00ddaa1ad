// What the TMA-staged back-projection kernels share: mbarrier waits (bounded), the box
// loads of the filtered-view ring, shared-memory taps, the floor-by-magic-constant trick,
// the global-memory bilinear fallback and the ring's tensor map.
#pragma once

#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>
#include <type_traits>

#include "mr_common.cuh"

namespace mr {

constexpr int ST_BOX_H = 8;                   // rows per TMA box
constexpr float MAGIC = 12582912.0f;          // 1.5 * 2^23
constexpr int MAGIC_BITS = 0x4B400000;
#define kMagic2 make_float2(MAGIC, MAGIC)
#define kNeg2 make_float2(-1.f, -1.f)

enum : int { MODE_STAGED = 0, MODE_GLOBAL = 1, MODE_SKIP = 2 };

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_arrive_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait: gives up after `limit` polls and reports it (never spins forever).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* status) {
    for (int it = 0; it < (1 << 22); ++it)
        if (mbar_try_wait(bar, parity)) return true;
    if (status) atomicExch(status, MR_ERR_TIMEOUT);
    return false;
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
        " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ unsigned short lds_u16(uint32_t addr) {
    unsigned short u;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(u) : "r"(addr));
    return u;
}
// a - c, rounded to nearest, for a 16-bit value a (raw BF16 / FP16 bits) and an FP32 c
template <typename T>
__device__ __forceinline__ float sub16_f32(unsigned short a, float c) {
    float d;
    if constexpr (std::is_same<T, __nv_bfloat16>::value)
        asm("sub.rn.f32.bf16 %0, %1, %2;" : "=f"(d) : "h"(a), "f"(c));
    else
        asm("sub.rn.f32.f16 %0, %1, %2;" : "=f"(d) : "h"(a), "f"(c));
    return d;
}

template <typename T>
__device__ __forceinline__ float lds_elem(uint32_t addr);
template <>
__device__ __forceinline__ float lds_elem<float>(uint32_t addr) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(addr));
    return v;
}
template <>
__device__ __forceinline__ float lds_elem<__nv_bfloat16>(uint32_t addr) {
    unsigned short u;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(u) : "r"(addr));
    return __uint_as_float(static_cast<uint32_t>(u) << 16);
}
template <>
__device__ __forceinline__ float lds_elem<__half>(uint32_t addr) {
    unsigned short u;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(u) : "r"(addr));
    return __half2float(__ushort_as_half(u));
}

// Global-memory bilinear (fallback for footprints larger than a stage); (row, col) counts
// from detector pixel (row_at, col_at).
template <typename T>
__device__ __forceinline__ float bilerp_global(const T* __restrict__ q, int R, int C, int pitch,
                                               float row, float col, int row_at = 0, int col_at = 0) {
    row = fminf(fmaxf(row, (float)(-2 - row_at)), (float)(R + 1 - row_at));
    col = fminf(fmaxf(col, (float)(-2 - col_at)), (float)(C + 1 - col_at));
    const float r0f = floorf(row), c0f = floorf(col);
    const float fr = row - r0f, fc = col - c0f;
    const int r0 = (int)r0f + row_at, c0 = (int)c0f + col_at;
    const bool rin0 = (unsigned)r0 < (unsigned)R, rin1 = (unsigned)(r0 + 1) < (unsigned)R;
    const bool cin0 = (unsigned)c0 < (unsigned)C, cin1 = (unsigned)(c0 + 1) < (unsigned)C;
    const T* p = q + (ptrdiff_t)r0 * pitch + c0;
    const float q00 = (rin0 && cin0) ? ld_elem(p) : 0.f;
    const float q01 = (rin0 && cin1) ? ld_elem(p + 1) : 0.f;
    const float q10 = (rin1 && cin0) ? ld_elem(p + pitch) : 0.f;
    const float q11 = (rin1 && cin1) ? ld_elem(p + pitch + 1) : 0.f;
    const float a = fmaf(fc, q01 - q00, q00);
    const float b = fmaf(fc, q11 - q10, q10);
    return fmaf(fr, b - a, a);
}

// ---------------------------------------------------------------- host side
inline PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

// Tensor map of the ring for boxes of box_w columns x ST_BOX_H rows of one slot.
template <typename T>
inline int make_ring_map(const mr_ring* ring, int box_w, CUtensorMap* map) {
    auto fn = encode_fn();
    if (!fn) return MR_ERR_CUDA;
    const CUtensorMapDataType dt = sizeof(T) == 4 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32
                                   : (std::is_same<T, __half>::value ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                                                     : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16);
    const cuuint64_t dims[3] = {(cuuint64_t)ring->cols, (cuuint64_t)ring->rows, (cuuint64_t)ring->n_slots};
    const cuuint64_t strides[2] = {(cuuint64_t)ring->col_pitch * sizeof(T),
                                   (cuuint64_t)ring->slot_stride * sizeof(T)};
    const cuuint32_t box[3] = {(cuuint32_t)box_w, (cuuint32_t)ST_BOX_H, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(map, dt, 3, ring->data, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? MR_OK : MR_ERR_INVALID;
}

inline int check_staged_ring(const mr_ring* ring) {
    if (!ring || !ring->data) return MR_ERR_INVALID;
    if (ring->rows <= 0 || ring->cols <= 0 || ring->col_pitch < ring->cols || ring->n_slots <= 0)
        return MR_ERR_INVALID;
    if (ring->slot_stride < (int64_t)ring->rows * ring->col_pitch) return MR_ERR_INVALID;
    if (ring->kind != MR_CONE && ring->kind != MR_PARALLEL) return MR_ERR_INVALID;
    if ((reinterpret_cast<uintptr_t>(ring->data) & 15) != 0) return MR_ERR_INVALID;
    const int esz = ring->dtype == MR_F32 ? 4 : 2;
    if (ring->dtype != MR_F32 && ring->dtype != MR_BF16 && ring->dtype != MR_F16) return MR_ERR_INVALID;
    if ((ring->col_pitch * esz) % 16 || (ring->slot_stride * esz) % 16) return MR_ERR_INVALID;
    return MR_OK;
}

}  // namespace mr
