// Fragments of the mma.sync attention kernels (attention.cu, tq_attn.cu): scores and P.V with the f16 rows of the cache as B operands
// and q / the probabilities carried as two f16 terms in the upper and lower half of the 16 MMA rows.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace sk {

constexpr float MASKED = -1.0e30f;

__device__ __forceinline__ void mma_f16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// (x, y) -> f16 high parts packed, f16 low parts (x - hi(x)) packed
__device__ __forceinline__ void split_pack(float x, float y, uint32_t& hi, uint32_t& lo) {
    const __half hx = __float2half_rn(x), hy = __float2half_rn(y);
    const __half lx = __float2half_rn(x - __half2float(hx)), ly = __float2half_rn(y - __half2float(hy));
    hi = (uint32_t) __half_as_ushort(hx) | ((uint32_t) __half_as_ushort(hy) << 16);
    lo = (uint32_t) __half_as_ushort(lx) | ((uint32_t) __half_as_ushort(ly) << 16);
}
constexpr float LOG2E = 1.4426950408889634f;
// exp(x) for x <= 0 through the ex2 unit (relative error ~1e-7 after the fp32 pre-scale)
__device__ __forceinline__ float fast_exp(float x) { return exp2f(x * LOG2E); }

// key splits of a decode attention: one wave of CTAs, each with at least one 16-key tile per warp (attention.cu)
int decode_splits(int batch, int kv_heads, int max_kv_len);
// partial records {max, sum, acc[d]} of `rows` heads, `splits` each, folded into out[rows][d] (attention.cu); d 64 or 128
int32_t launch_attn_merge(const float* part, float* out, int rows, int d, int splits, cudaStream_t s);

}  // namespace sk
