// fp32 values as three bf16 parts (hi + mid + lo, each rounded to nearest: 24 significant bits, fp32's exponent range): what the tensor-core
// kernels for fp32 operands (attention_split.cu, linear_split.cu) cut their operands into.
#pragma once
#include "common.cuh"

namespace b2 {

// two values -> their three bf16 parts, packed (first value in the low half). A value that bf16 does not hold (an infinity, a NaN, a magnitude of
// 2^128 (1 - 2^-9) and more, which rounds to infinity) has NaN among its parts, and NaN is then what every sum of products that it enters comes
// to, whatever the other operand. So the kernels take a sum that is NaN for one they cannot do, and do it over in plain fp32 from the
// operands themselves (linear_split.cu, attention_split.cu): infinite results, scores of -inf and large finite values come out as they
// would from fp32 products.
__device__ __forceinline__ void split3(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = pack_bf16(a, b);
    const float a1 = a - bf16_lo(hi), b1 = b - bf16_hi(hi);
    mid = pack_bf16(a1, b1);
    lo = pack_bf16(a1 - bf16_lo(mid), b1 - bf16_hi(mid));
}
__device__ __forceinline__ void split8(const float (&x)[8], uint4& hi, uint4& mid, uint4& lo) {
    split3(x[0], x[1], hi.x, mid.x, lo.x);
    split3(x[2], x[3], hi.y, mid.y, lo.y);
    split3(x[4], x[5], hi.z, mid.z, lo.z);
    split3(x[6], x[7], hi.w, mid.w, lo.w);
}
// 8 floats of a row of `n`, from d on (entries past the end are zero)
__device__ __forceinline__ void load8(const float* p, int d, int n, bool vec, float (&x)[8]) {
    if (vec && d + 8 <= n) {
        const float4 a = *reinterpret_cast<const float4*>(p + d), b = *reinterpret_cast<const float4*>(p + d + 4);
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = d + e < n ? p[d + e] : 0.f;
    }
}

// The six products of two split operands in rising size, so that an accumulator is small while the small ones join it: (lo, hi) (hi, lo) (mid, mid)
// (mid, hi) (hi, mid) (hi, hi); two bits each, first product lowest. What is left out lies below 2^-25 of the operands' product.
constexpr uint32_t SPLIT_A = 2u | 0u << 2 | 1u << 4 | 1u << 6 | 0u << 8 | 0u << 10, SPLIT_B = 0u | 2u << 2 | 1u << 4 | 0u << 6 | 1u << 8 | 0u << 10;

__device__ __forceinline__ void tma_load_3d(void* dst, const void* tmap, uint64_t* bar, int c0, int c1, int c2) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
                 ::"r"(smem_u32(dst)), "l"(tmap), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}

}  // namespace b2
