// Fragments of the warp-level tensor-core product (mma.sync m16n8k16, bfloat16 in, float32 out) and what feeds them: asynchronous
// 16-byte copies to shared memory, ldmatrix, and the cut of a float32 number into the sum of two or three bfloat16 ones.
#pragma once

#include "common.cuh"

namespace lily {
namespace mma16 {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// 16 bytes, both ends 16-byte aligned; zeros when `in` is false (src is not read then)
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool in) {
    const int bytes = in ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3) : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Two numbers as pairs of bfloat16: x = hi + lo to 16 bits.
__device__ __forceinline__ void split2(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 back = __bfloat1622float2(h);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - back.x, y - back.y);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    lo = *reinterpret_cast<const uint32_t*>(&l);
}
// The same as three pairs, whose sum they are (an infinity becomes a NaN).
__device__ __forceinline__ void split3(float x, float y, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 back = __bfloat1622float2(h);
    hi = *reinterpret_cast<const uint32_t*>(&h);
    split2(x - back.x, y - back.y, mid, lo);
}

// The second and the first number of a pair of bfloat16.
__device__ __forceinline__ float upper(uint32_t pair) { return __uint_as_float(pair & 0xffff0000u); }
__device__ __forceinline__ float lower(uint32_t pair) { return __uint_as_float(pair << 16); }

// Runs of 16 products' sums onto their totals by rounded additions: the tensor cores cut what they add to an accumulator off, so a total
// kept in one would drift by half a last bit a product.
template <int N>
__device__ __forceinline__ void add(float (*total)[4], const float (&sum)[N][4]) {
#pragma unroll
    for (int j = 0; j < N; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) total[j][q] += sum[j][q];
}

}  // namespace mma16
}  // namespace lily
