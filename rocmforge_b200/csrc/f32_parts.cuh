// Float32 numbers as three bfloat16 parts, for the tensor cores: what the 32-bit product and the 32-bit prompt attention share.
#pragma once
#include "tcgen05_common.cuh"

#define FS_BK 32                                   // floats of a 128-byte row: what one TMA box of a float32 matrix is wide

__device__ __forceinline__ void fs_st8(uint32_t taddr, const uint32_t* r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
// Two numbers into their three parts, each pair packed with the first in the lower half.
__device__ __forceinline__ float2 fs_sub2(float2 a, uint32_t bx, uint32_t by) {
    float2 r;
    asm("{\n\t.reg .b64 a, b, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tsub.rn.f32x2 d, a, b;\n\tmov.b64 {%0, %1}, d;\n\t}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "r"(bx), "r"(by));
    return r;
}
__device__ __forceinline__ void fs_split2(float a, float b, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    p1 = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
    const float2 r = fs_sub2(make_float2(a, b), __float_as_uint(a) & 0xffff0000u, __float_as_uint(b) & 0xffff0000u);
    p2 = pack_bf16x2(r.x, r.y);
    const float2 q = fs_sub2(r, p2 << 16, p2 & 0xffff0000u);
    p3 = pack_bf16x2(q.x, q.y);
}
__device__ __forceinline__ float4 fs_lds(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

// Float32 matrix [rows, cols] with row stride ld (elements); box = box_rows x 32 numbers, 128-byte swizzle.
static int fs_map(CUtensorMap* map, const void* base, long long rows, long long cols, long long ld, int box_rows) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) return RF_ERR_UNSUPPORTED;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 4};
    cuuint32_t box[2] = {FS_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : RF_ERR_BAD_ARG;
}
