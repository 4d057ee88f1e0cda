// Stand-alone element-wise ops of the token loop (RMSNorm, RoPE, SwiGLU, residual add, arg-max).
// Inside the model these are fused into GEMV prologues/epilogues; the stand-alone kernels serve the
// op-level API that mirrors crates/inferi/src/ops/{rms_norm,rope,silu}.rs and context.rs:516-530.
//
// All of them are launched with programmatic dependent launch: each lets its successor start at once and waits for its
// predecessor before it touches an operand, so that in a chain of op calls the next kernel's launch and set-up overlap the
// previous kernel's tail (worth 1-2 us per launch where a kernel itself takes 2 us).
#include "common.cuh"

#include <math.h>
#include <string.h>

namespace ib {

__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... KArgs, typename... Args>
static int32_t launch_op(ib_ctx *ctx, cudaStream_t s, void (*kernel)(KArgs...), uint32_t grid, uint32_t block, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    IB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, (KArgs)args...));
    ctx->launches++;
    return IB_OK;
}

// ---- RMSNorm: crates/inferi-shaders/src/rms_norm.rs:78-121 ----
// One CTA; latency bound (one load, a block reduction, one store).  The first RMS_KEEP values of a thread stay in registers,
// so the vector is read once and the loads of x and w are all in flight together.
constexpr uint32_t RMS_KEEP = 4;
__global__ void __launch_bounds__(1024) rms_norm_kernel(float *out, const float *x, const float *w, uint32_t n, float eps) {
    __shared__ float red[32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5, step = blockDim.x;
    pdl_enter();
    float v[RMS_KEEP], g[RMS_KEEP];
#pragma unroll
    for (uint32_t k = 0; k < RMS_KEEP; k++) {
        const uint32_t i = tid + k * step;
        v[k] = i < n ? x[i] : 0.f;
        g[k] = i < n ? w[i] : 0.f;
    }
    float ss = 0.f;
#pragma unroll
    for (uint32_t k = 0; k < RMS_KEEP; k++) ss += v[k] * v[k];
    for (uint32_t i = tid + RMS_KEEP * step; i < n; i += step) ss += x[i] * x[i];
#pragma unroll
    for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    float t = lane < nwarps ? red[lane] : 0.f;
#pragma unroll
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    const float rms = 1.0f / sqrtf(t / (float)n + eps);
#pragma unroll
    for (uint32_t k = 0; k < RMS_KEEP; k++) {
        const uint32_t i = tid + k * step;
        if (i < n) out[i] = (v[k] * rms) * g[k];
    }
    for (uint32_t i = tid + RMS_KEEP * step; i < n; i += step) out[i] = (x[i] * rms) * w[i];
}

int32_t launch_rms_norm(ib_ctx *ctx, cudaStream_t s, float *out, const float *x, const float *w, uint32_t n, float eps) {
    return launch_op(ctx, s, rms_norm_kernel, 1, n >= 2048 ? 1024 : (n >= 1024 ? 512 : 128), out, x, w, n, eps);
}

// ---- RoPE: crates/inferi-shaders/src/rope.rs:51-92 (Original), :97-141 (NeoX) ----
// The per-dimension frequencies theta_j = base^(-2j/head_size) are computed on the host with the C library's
// powf and passed by value, so that device and host agree on them bit for bit.  They are a model's constants: a thread keeps those of the
// last model it launched for (32 powf are a third of the launch).
struct RopeTheta { float t[128]; };

__global__ void rope_kernel(int variant, float *q, uint32_t q_len, float *k, uint32_t kv_dim, uint32_t head_size, uint32_t pos,
                            const RopeTheta th) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_enter();
    if (i >= q_len / 2) return;
    const uint32_t half = head_size / 2;
    uint32_t i0, i1, j;
    if (variant == IB_ROPE_ORIGINAL) { i0 = 2 * i; i1 = i0 + 1; j = ((2 * i) % head_size) / 2; }
    else { const uint32_t head = i / half; j = i % half; i0 = head * head_size + j; i1 = i0 + half; }
    float sn, cs;
    sincosf((float)pos * th.t[j], &sn, &cs);
    float x = q[i0], y = q[i1];
    q[i0] = cs * x - sn * y;
    q[i1] = sn * x + cs * y;
    if (i0 < kv_dim) {
        x = k[i0]; y = k[i1];
        k[i0] = cs * x - sn * y;
        k[i1] = sn * x + cs * y;
    }
}

int32_t launch_rope(ib_ctx *ctx, cudaStream_t s, int variant, float *q, uint32_t q_len, float *k, uint32_t kv_dim, uint32_t head_size, uint32_t pos,
                    float base_freq) {
    static thread_local RopeTheta th;
    static thread_local float of_base;
    static thread_local uint32_t of_size = 0;
    if (of_size != head_size || memcmp(&of_base, &base_freq, sizeof of_base)) {
        for (uint32_t j = 0; j < head_size / 2; j++) th.t[j] = powf(base_freq, -(float)(2 * j) / (float)head_size);
        of_base = base_freq;
        of_size = head_size;
    }
    const uint32_t n = q_len / 2;
    return launch_op(ctx, s, rope_kernel, (n + 127) / 128, 128, variant, q, q_len, k, kv_dim, head_size, pos, th);
}

// ---- SwiGLU: crates/inferi-shaders/src/silu.rs:24-53 ----
__global__ void silu_mul_kernel(float *h1, const float *h2, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_enter();
    if (i < n) {
        const float a = h1[i];
        h1[i] = h2[i] * (a / (1.0f + expf(-a)));
    }
}
int32_t launch_silu_mul(ib_ctx *ctx, cudaStream_t s, float *h1, const float *h2, uint32_t n) {
    return launch_op(ctx, s, silu_mul_kernel, (n + 255) / 256, 256, h1, h2, n);
}

// ---- residual add: crates/inferi/src/context.rs:516-530 ----
__global__ void add_assign_kernel(float *a, const float *b, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    pdl_enter();
    if (i < n) a[i] += b[i];
}
int32_t launch_add_assign(ib_ctx *ctx, cudaStream_t s, float *a, const float *b, uint32_t n) {
    return launch_op(ctx, s, add_assign_kernel, (n + 255) / 256, 256, a, b, n);
}

// ---- greedy arg-max: crates/inferi/src/models/sampler.rs:54-56; lowest index on ties ----
__device__ __forceinline__ unsigned long long amax_key(float v, uint32_t idx) {
    uint32_t u = __float_as_uint(v);
    u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ((unsigned long long)u << 32) | (unsigned long long)(0xFFFFFFFFu - idx);
}

constexpr int ARGMAX_MAX_CTAS = 1024;

__global__ void __launch_bounds__(256) argmax_kernel(const float *x, uint32_t n, unsigned long long *slots, unsigned int *counter, uint32_t *out) {
    __shared__ unsigned long long sm[8];
    __shared__ bool is_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long best = 0ull;
    pdl_enter();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) best = max(best, amax_key(x[i], i));
#pragma unroll
    for (int o = 16; o; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (lane == 0) sm[warp] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 0; w < 8; w++) best = max(best, sm[w]);
        slots[blockIdx.x] = best;
        __threadfence();
        is_last = (atomicAdd(counter, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (is_last) {
        __threadfence();
        best = 0ull;
        for (uint32_t i = threadIdx.x; i < gridDim.x; i += blockDim.x) best = max(best, __ldcg(slots + i));
#pragma unroll
        for (int o = 16; o; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
        __syncthreads();
        if (lane == 0) sm[warp] = best;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 0; w < 8; w++) best = max(best, sm[w]);
            *out = 0xFFFFFFFFu - (uint32_t)(best & 0xFFFFFFFFull);
            *counter = 0u;
        }
    }
}

int32_t ensure_argmax_scratch(ib_ctx *ctx) {
    if (!ctx->argmax_scratch) {
        IB_CHECK_CUDA(cudaMalloc(&ctx->argmax_scratch, sizeof(unsigned long long) * ARGMAX_MAX_CTAS));
        IB_CHECK_CUDA(cudaMalloc(&ctx->argmax_counter, sizeof(unsigned int)));
        IB_CHECK_CUDA(cudaMemset(ctx->argmax_counter, 0, sizeof(unsigned int)));
    }
    return IB_OK;
}

int32_t launch_argmax(ib_ctx *ctx, cudaStream_t s, const float *x, uint32_t n, uint32_t *out) {
    int32_t rc = ensure_argmax_scratch(ctx);
    if (rc) return rc;
    int grid = (int)((n + 1023) / 1024);
    if (grid > ctx->sm_count * 2) grid = ctx->sm_count * 2;
    if (grid < 1) grid = 1;
    return launch_op(ctx, s, argmax_kernel, (uint32_t)grid, 256, x, n, ctx->argmax_scratch, ctx->argmax_counter, out);
}

}  // namespace ib
