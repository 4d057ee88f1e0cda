// Device helpers shared by the quantized GEMV kernels: the block-fixed-point activation form, dp4a wrappers and
// the per-format 64-weight "unit" dot products.
#pragma once

#include "common.cuh"

namespace ib {

constexpr int PACK_THREADS = 512;        // threads that take part in the activation prologue of the streaming kernel
constexpr uint32_t GEMV_MAX_COLS = 32768;

// Activation form in shared memory, for `cols` columns (a multiple of 32):
//   ACT_LIMBS int8 limbs a0, a1 [cols] each;  f32 scale s/32512 per 32 columns;  f32 sum of the quantized x per 16 columns
//   x ~= (s/32512) * (256 a0 + a1)     (resolution 1.5e-5 * max|x| of the 32-group: 16-bit block fixed point)
// The 16-column sums (used for the k-quants' minimums and the Q6_K -32 terms) are sums of the QUANTIZED values, so that
// sum_k w_k a_k is evaluated exactly for the a_k the dot products see; the only error of a GEMV is sum_k w_k (a_k - x_k),
// 2e-5 .. 1e-4 relative.  (A third limb - 24-bit fixed point - costs a third more dp4a and 16 more registers per lane: 583
// against 619 tok/s on the 8B architecture; the logits of the 1B architecture then differ from the f32 oracle's by 7e-4
// instead of 2.7e-3 max-abs, at a tolerance of 2e-2.)
constexpr int ACT_LIMBS = 2;
__host__ __device__ inline size_t act_smem_bytes(uint32_t cols) { return (size_t)cols * ACT_LIMBS + cols / 32 * 4 + cols / 16 * 4; }

struct Act {
    const uint8_t *base;
    uint32_t cols;
    __device__ __forceinline__ const uint4 *limb(int k) const { return reinterpret_cast<const uint4 *>(base + (size_t)k * cols); }
    __device__ __forceinline__ const float *sc() const { return reinterpret_cast<const float *>(base + (size_t)ACT_LIMBS * cols); }
    __device__ __forceinline__ const float *sx16() const { return sc() + cols / 32; }
};

__device__ __forceinline__ int dp4a_ss(uint32_t a, uint32_t b, int c) { return __dp4a((int)a, (int)b, c); }
__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {
    int d;
    asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// The integer dot products of the two limbs -> the dot product in units of the group's scale.  256 d0 + d1 is formed as an
// integer (at most 2^28 for every format's longest chain) and converted once: exact up to the conversion's rounding.
static_assert(ACT_LIMBS == 2, "the dot products combine two limbs");
__device__ __forceinline__ int limb_sum(int d0, int d1) { return d0 * 256 + d1; }
__device__ __forceinline__ float limb_combine(const int *d) { return (float)limb_sum(d[0], d[1]); }
__device__ __forceinline__ float h2f(uint32_t bits16) { return __half2float(__ushort_as_half((unsigned short)bits16)); }

__device__ __forceinline__ void named_barrier(int id, int nthreads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory"); }

__device__ __forceinline__ unsigned long long argmax_key(float v, uint32_t idx) {
    uint32_t u = __float_as_uint(v);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((unsigned long long)u << 32) | (unsigned long long)(0xFFFFFFFFu - idx);  // ties -> lowest index
}

// -------------------------------------------------------------------------------------------------
// prologue: (optional RMSNorm) + conversion of x into the limb form in shared memory.
// Called by the first PACK_THREADS threads of the CTA; synchronises them on named barrier 1.
// A thread owns runs of 16 consecutive columns (run number tid + 256 i): the 16-column sum needs no shuffle, the
// 32-column maximum one shuffle with the neighbour lane, and the 16 conversions are independent of each other.
// -------------------------------------------------------------------------------------------------
constexpr int PACK_RUNS = 2;   // runs of 16 columns kept in registers per thread (covers 16384 columns with 512 threads)

struct PackRegs {
    float4 x[PACK_RUNS][4];
};

// Issues the loads of this thread's norm weights.  They are weights, so a kernel may call this before it waits for
// its predecessor.
__device__ __forceinline__ void pack_prefetch_norm(const float *__restrict__ norm_w, uint32_t cols, float4 (&g)[4]) {
    const uint32_t run = threadIdx.x;   // only the first run's weights are kept (cols <= 4096); wider rows re-fetch
    if (norm_w && run < cols / 16) {
        const float4 *w4 = reinterpret_cast<const float4 *>(norm_w) + 4 * run;
#pragma unroll
        for (int j = 0; j < 4; j++) g[j] = __ldg(w4 + j);
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) g[j] = make_float4(1.f, 1.f, 1.f, 1.f);
    }
}

constexpr float ACT_STEPS = 32512.0f;   // = 127 * 256: the largest |x| of a group is so many units, a0 = +-127, a1 = 0

// Four columns -> their bytes of the two limbs; `inv` = ACT_STEPS / largest |x| of the group; `s0`, `s1` += the limbs.
// One multiply-add rounds to an integer: added to 1.5 * 2^23 the value sits in the low bits of the float, in two's complement.
// It is formed 128 too high, so that its bits 8-15 are a0 rounded to nearest and its low byte is a1 + 128.
__device__ __forceinline__ void pack_four(const float (&e)[4], float inv, uint32_t &w0, uint32_t &w1, int &s0, int &s1) {
    constexpr float MAGIC = 12582912.0f + 128.0f;
    uint32_t b[4];
#pragma unroll
    for (int k = 0; k < 4; k++) b[k] = __float_as_uint(fmaf(e[k], inv, MAGIC));
    w0 = __byte_perm(__byte_perm(b[0], b[1], 0x0051), __byte_perm(b[2], b[3], 0x0051), 0x5410);
    w1 = __byte_perm(__byte_perm(b[0], b[1], 0x0040), __byte_perm(b[2], b[3], 0x0040), 0x5410) ^ 0x80808080u;
    s0 = dp4a_ss(w0, 0x01010101u, s0);
    s1 = dp4a_ss(w1, 0x01010101u, s1);
}

// The larger of two, or NaN where one of them is: a NaN among a group's columns has to reach the group's scale, because the limbs
// cannot carry one (fmaxf drops it, and a row's sum then comes out finite).
__device__ __forceinline__ float max_nan(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float abs_max(const float4 &v) { return max_nan(max_nan(fabsf(v.x), fabsf(v.y)), max_nan(fabsf(v.z), fabsf(v.w))); }

// Units per 1 of x for a group whose largest |x| is `amax`.  f32 cannot hold ACT_STEPS / amax below 2^-113: groups far below 1 are brought
// nearer first, and without a branch (one, never taken, cost 0.7 % of a token of the 1B architecture).  __fdividef is 2 ulp: the limbs absorb
// it, the largest |x| still rounds to ACT_STEPS.
template <int N>
__device__ __forceinline__ float pack_units(float4 (&v)[N], float amax) {
    const float k = amax < 0x1p-100f ? 0x1p64f : 1.0f;
#pragma unroll
    for (int j = 0; j < N; j++) { v[j].x *= k; v[j].y *= k; v[j].z *= k; v[j].w *= k; }
    return amax > 0.f ? __fdividef(ACT_STEPS, amax * k) : 0.f;
}

__device__ __forceinline__ void pack_run(float4 (&v)[4], uint32_t run, uint32_t cols, uint8_t *smem, bool store) {
    const int lane = threadIdx.x & 31;
    int s0 = 0, s1 = 0;
    float amax = max_nan(max_nan(abs_max(v[0]), abs_max(v[1])), max_nan(abs_max(v[2]), abs_max(v[3])));
    amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 1));   // the other half of the 32-column group
    const float inv = pack_units(v, amax);
    uint32_t w0[4], w1[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const float e[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
        pack_four(e, inv, w0[j], w1[j], s0, s1);
    }
    if (store) {
        uint4 *l0 = reinterpret_cast<uint4 *>(smem), *l1 = reinterpret_cast<uint4 *>(smem + cols);
        float *sc = reinterpret_cast<float *>(smem + ACT_LIMBS * cols), *sx16 = sc + cols / 32;
        l0[run] = make_uint4(w0[0], w0[1], w0[2], w0[3]);
        l1[run] = make_uint4(w1[0], w1[1], w1[2], w1[3]);
        if ((lane & 1) == 0) sc[run >> 1] = amax * (1.0f / ACT_STEPS);
        sx16[run] = (float)limb_sum(s0, s1) * (amax * (1.0f / ACT_STEPS));
    }
}

// `g` holds the norm weights of the thread's first run (from pack_prefetch_norm).
template <int NT = PACK_THREADS>
__device__ __forceinline__ void pack_activation(uint8_t *smem, uint32_t cols, const float *__restrict__ x, const float *__restrict__ norm_w, float eps,
                                                float *red /* [NT/32 + 1] */, const float4 (&g)[4]) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nruns = cols / 16;    // cols is a multiple of 32, so runs pair up inside a warp
    const float4 *x4 = reinterpret_cast<const float4 *>(x);
    const float4 *w4 = reinterpret_cast<const float4 *>(norm_w);
    PackRegs r;
#pragma unroll
    for (int i = 0; i < PACK_RUNS; i++) {
        const uint32_t run = tid + NT * i;
#pragma unroll
        for (int j = 0; j < 4; j++) r.x[i][j] = run < nruns ? __ldcg(x4 + 4 * run + j) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    float rms = 1.0f;
    if (norm_w) {
        // crates/inferi-shaders/src/rms_norm.rs:112-120
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < PACK_RUNS; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) ss += (r.x[i][j].x * r.x[i][j].x + r.x[i][j].y * r.x[i][j].y) + (r.x[i][j].z * r.x[i][j].z + r.x[i][j].w * r.x[i][j].w);
        for (uint32_t run = tid + NT * PACK_RUNS; run < nruns; run += NT)   // rows wider than the registers hold
            for (int j = 0; j < 4; j++) {
                const float4 v = __ldcg(x4 + 4 * run + j);
                ss += (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w);
            }
#pragma unroll
        for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) red[warp] = ss;
        named_barrier(1, NT);
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < NT / 32; w++) t += red[w];
        rms = 1.0f / sqrtf(t / (float)cols + eps);
    }
#pragma unroll
    for (int i = 0; i < PACK_RUNS; i++) {
        const uint32_t run = tid + NT * i;
        if ((uint32_t)(warp * 32 + NT * i) < nruns) {   // warp-uniform: both lanes of a 32-column group are present
            const bool ok = run < nruns;
            if (norm_w && ok) {
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float4 w = (i == 0) ? g[j] : __ldg(w4 + 4 * run + j);
                    float4 &v = r.x[i][j];
                    v.x = (v.x * rms) * w.x; v.y = (v.y * rms) * w.y; v.z = (v.z * rms) * w.z; v.w = (v.w * rms) * w.w;
                }
            }
            pack_run(r.x[i], run, cols, smem, ok);
        }
    }
    for (uint32_t base = warp * 32 + NT * PACK_RUNS; base < nruns; base += NT) {   // rows wider than the registers hold
        const uint32_t run = base + lane;
        const bool ok = run < nruns;
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[j] = ok ? __ldcg(x4 + 4 * run + j) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (norm_w && ok) {
                const float4 w = __ldg(w4 + 4 * run + j);
                v[j].x = (v[j].x * rms) * w.x; v[j].y = (v[j].y * rms) * w.y; v[j].z = (v[j].z * rms) * w.z; v[j].w = (v[j].w * rms) * w.w;
            }
        }
        pack_run(v, run, cols, smem, ok);
    }
    named_barrier(1, NT);
}

}  // namespace ib
