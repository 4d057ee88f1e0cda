// Device helpers of the prefill's element-wise kernels: eight columns per thread, and the split, tiled form of a GEMM's inputs.
#pragma once

#include "prefill.cuh"

namespace ib {

__device__ __forceinline__ void pf_enter() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

struct F8 { float v[8]; };
__device__ __forceinline__ F8 pf_load8(const float *p) {
    const float4 a = __ldcg(reinterpret_cast<const float4 *>(p)), b = __ldcg(reinterpret_cast<const float4 *>(p) + 1);
    return F8{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
__device__ __forceinline__ void pf_store8(float *p, const F8 &f) {
    reinterpret_cast<float4 *>(p)[0] = make_float4(f.v[0], f.v[1], f.v[2], f.v[3]);
    reinterpret_cast<float4 *>(p)[1] = make_float4(f.v[4], f.v[5], f.v[6], f.v[7]);
}
// the same for a caller's buffer, which may be aligned to 4 bytes only
__device__ __forceinline__ F8 pf_load8u(const float *p) {
    if (((uintptr_t)p & 15) == 0) return pf_load8(p);
    F8 f;
#pragma unroll
    for (int i = 0; i < 8; i++) f.v[i] = __ldcg(p + i);
    return f;
}
__device__ __forceinline__ void pf_add8(F8 &a, const F8 &b) {
#pragma unroll
    for (int i = 0; i < 8; i++) a.v[i] += b.v[i];
}

// Columns c .. c + 7 (c % 8 == 0) of token t into the split, tiled inputs of the next GEMM, with the sums of the 32-column
// sub-blocks: four neighbouring lanes hold one sub-block (all 32 lanes of the warp take part).
__device__ __forceinline__ void pf_emit8(__half *xt, uint32_t t, uint32_t c, uint32_t cols, const F8 &f) {
    const size_t base = (size_t)(t / PF_CHUNK) * pf_x_halves(cols);
    const uint32_t tc = t % PF_CHUNK;
    uint32_t h[4], l[4];
    constexpr int order[8] = {0, 2, 1, 3, 4, 6, 5, 7};   // pf_x_index
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float a = f.v[order[2 * i]], b = f.v[order[2 * i + 1]];
        const __half2 hh = __floats2half2_rn(a, b);
        const float2 back = __half22float2(hh);
        const __half2 ll = __floats2half2_rn(a - back.x, b - back.y);
        h[i] = *reinterpret_cast<const uint32_t *>(&hh);
        l[i] = *reinterpret_cast<const uint32_t *>(&ll);
        sum += f.v[2 * i] + f.v[2 * i + 1];
    }
    const size_t at = base + pf_x_index(tc, c);
    *reinterpret_cast<uint4 *>(xt + at) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(xt + at + PF_X_LO) = make_uint4(l[0], l[1], l[2], l[3]);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const size_t sat = base + pf_s_index(tc, c >> 5, cols);
    if ((c & 31) == 0) {
        const __half sh = __float2half_rn(sum);
        xt[sat] = sh;
        xt[sat + PF_S_LO] = __float2half_rn(sum - __half2float(sh));
    }
    if ((c & 255) == 8) {   // the eight zero halves of the block's row of sums
        *reinterpret_cast<uint4 *>(xt + sat + 64) = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4 *>(xt + sat + PF_S_LO + 64) = make_uint4(0, 0, 0, 0);
    }
}

}  // namespace ib
