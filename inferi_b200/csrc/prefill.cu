// Prompt prefill: the element-wise kernels between the GEMMs, and the GEMM entry point of the op API.
//
// The prompt's tokens go through every matrix together, as GEMMs on the 5th-generation tensor cores (prefill_gemm.cu),
// instead of one by one through the decode path.  The reference has no prefill: `ChatLlama2::forward` forces the prompt
// through the decode path token by token (crates/inferi-chat/src/chat_llama2.rs:137-155,
// crates/inferi-chat/src/sampler.rs:102-107), which reads every weight once per prompt token.
//
// Between two GEMMs there is one kernel: it adds up the GEMM's partial planes, does what the layer asks for (residual and the
// next norm; rotation and cache append; SwiGLU) and writes the next GEMM's inputs already split into two f16 and in the
// tensor core's tile layout.  All of them are launched with programmatic dependent launch.  They are bound by L2 latency
// and traffic: eight columns per thread, so that every access is 16 or 32 bytes.
#include "prefill_emit.cuh"

namespace ib {

// Rows r .. r + 7 of token t, added up over the tile's planes in plane order (deterministic); DEPTH planes are requested at a time.
template <int DEPTH = 2>
__device__ __forceinline__ F8 pf_sum8(const PfPlanes &g, uint32_t t, uint32_t r) {
    const size_t at = (size_t)t * g.rows + r, plane = (size_t)g.n * g.rows;
    F8 v = pf_load8u(g.plane0 + at);
    const uint32_t np = g.sk.pieces(g.sk.row_tile(r) * g.chunks + t / PF_CHUNK);
    for (uint32_t s = 1; s < np; s += DEPTH) {
        F8 a[DEPTH];
#pragma unroll
        for (int k = 0; k < DEPTH; k++)
            if (s + k < np) a[k] = pf_load8(g.planes + (s - 1 + k) * plane + at);
#pragma unroll
        for (int k = 0; k < DEPTH; k++)
            if (s + k < np) pf_add8(v, a[k]);
    }
    return v;
}

// X[t][c] = dequantized embedding row of token t (crates/inferi/src/models/llama2/transformer.rs:367-374, chat_llama2.rs:217-220)
__global__ void prefill_embed_kernel(QDesc embd, const uint32_t *tokens, uint32_t n, uint32_t hidden, uint32_t vocab, float *X) {
    pf_enter();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)n * hidden; i += (size_t)gridDim.x * blockDim.x) {
        const uint32_t t = (uint32_t)(i / hidden), c = (uint32_t)(i % hidden);
        uint32_t tok = tokens[t];
        if (tok >= vocab) tok = vocab - 1;
        X[i] = dequant_at(embd, embd.w + (size_t)tok * embd.row_bytes, c);
    }
}

// X += the planes of the GEMM before (where there is one), then y = (X * rsqrt(mean(X^2) + eps)) * w
// (crates/inferi-shaders/src/rms_norm.rs:112-120) as the next GEMM's inputs; without NORM y = X.  TOK tokens per CTA, a warp's lanes shared out to them: the
// inputs' layout holds 8 tokens' 8 columns side by side, and a warp of one token writes 16 bytes of every 128.  With NORM the row stays in registers
// between the two (PF_KEEP * 8 columns per thread; what is longer is read again).  Rows n .. n rounded up to 16 are zero-filled.
constexpr int PF_ROW_THREADS = 512, PF_KEEP = 4;
// Two tokens per CTA: a token's lanes are twice those of four, and the second half continues the first one's sums, so that the bits are those of four.
template <int TOK, int DEPTH, bool NORM>
__global__ void __launch_bounds__(PF_ROW_THREADS, TOK == 2 ? 2 : 1) prefill_norm_split_kernel(float *X, const PfPlanes add, uint32_t has_add, const float *w, float eps, uint32_t n, uint32_t cols,
                                                                            __half *xt) {
    constexpr uint32_t PARTS = TOK == 2 ? 2 : 1, LANES = 32 / (TOK * PARTS), WARPS = PF_ROW_THREADS / 32, STEP = WARPS * LANES * 8, HELD = PF_KEEP / PARTS;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, which = lane / (LANES * PARTS), part = lane / LANES % PARTS, t = blockIdx.x * TOK + which;
    const uint32_t c0 = (warp * LANES + lane % LANES) * 8;   // cols % 256 == 0: whole warps
    const bool there = t < n;
    pf_enter();
    float *x = X + (size_t)t * cols;
    const F8 zero = {{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}};
    F8 keep[PF_KEEP];
    auto fetch = [&](uint32_t c) {
        F8 v = zero;
        if (there) {
            v = pf_load8u(x + c);
            if (has_add) {
                pf_add8(v, pf_sum8<DEPTH>(add, t, c));
                pf_store8(x + c, v);
            }
        }
        return v;
    };
    if constexpr (!NORM) {   // (blockIdx.y: so many of the columns)
        const uint32_t c1 = c0 + blockIdx.y * PF_KEEP * STEP;
#pragma unroll
        for (int k = 0; k < PF_KEEP; k++)
            if (c1 + k * STEP < cols) keep[k] = fetch(c1 + k * STEP);
#pragma unroll
        for (int k = 0; k < PF_KEEP; k++)
            if (c1 + k * STEP < cols) pf_emit8(xt, t, c1 + k * STEP, cols, keep[k]);
    } else {
        __shared__ float red[WARPS][TOK];
        float ss = 0.f;
        auto square = [&](const F8 &v) {
#pragma unroll
            for (int i = 0; i < 8; i++) ss += v.v[i] * v.v[i];
        };
        // The lane's pieces: at c0 + (k0 + k) * STEP, k < HELD, up to the row's end or the half's, for all lanes of a warp alike (pf_emit8).  Two halves: cols is
        // a multiple of 2 STEP.
        const uint32_t k0 = PARTS == 1 ? 0 : part * (cols / STEP / 2), end = PARTS == 1 ? cols : c0 + (k0 + cols / STEP / 2) * STEP;
#pragma unroll
        for (uint32_t k = 0; k < HELD; k++)
            if (c0 + (k0 + k) * STEP < end) keep[k] = fetch(c0 + (k0 + k) * STEP);
#pragma unroll
        for (uint32_t p = 0; p < PARTS; p++) {
            if (p) ss = __shfl_sync(0xffffffffu, ss, lane - LANES * part);   // (the second half goes on where the first one ended)
#pragma unroll
            for (uint32_t k = 0; k < HELD; k++)
                if (p == part && c0 + (k0 + k) * STEP < end) square(keep[k]);
        }
        if (PARTS == 1)
            for (uint32_t c = c0 + HELD * STEP; c < cols; c += STEP) square(fetch(c));
#pragma unroll
        for (uint32_t o = LANES / 2; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (part == PARTS - 1 && lane % LANES == 0) red[warp][which] = ss;
        __syncthreads();
        float tot = 0.f;
#pragma unroll
        for (uint32_t i = 0; i < WARPS; i++) tot += red[i][which];
        const float rms = 1.0f / sqrtf(tot / (float)cols + eps);
        auto emit = [&](uint32_t c, F8 v) {
            const F8 g = pf_load8(w + c);
#pragma unroll
            for (int i = 0; i < 8; i++) v.v[i] = there ? (v.v[i] * rms) * g.v[i] : 0.f;
            pf_emit8(xt, t, c, cols, v);
        };
#pragma unroll
        for (uint32_t k = 0; k < HELD; k++)
            if (c0 + (k0 + k) * STEP < end) emit(c0 + (k0 + k) * STEP, keep[k]);
        if (PARTS == 1)
            for (uint32_t c = c0 + HELD * STEP; c < cols; c += STEP) emit(c, there ? pf_load8u(x + c) : zero);
    }
}

__global__ void __launch_bounds__(256) prefill_residual_kernel(float *X, const PfPlanes add) {
    pf_enter();
    const uint32_t per = add.rows / 8, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= add.n * per) return;
    const uint32_t t = i / per, r = (i - t * per) * 8;
    F8 v = pf_load8(X + (size_t)t * add.rows + r);
    pf_add8(v, pf_sum8(add, t, r));
    pf_store8(X + (size_t)t * add.rows + r, v);
}

__global__ void __launch_bounds__(256) prefill_finish_kernel(float *out, const PfPlanes add) {
    pf_enter();
    const uint32_t per = add.rows / 8, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= add.n * per) return;
    const uint32_t t = i / per, r = (i - t * per) * 8;
    if (add.sk.pieces(add.sk.row_tile(r) * add.chunks + t / PF_CHUNK) == 1) return;
    const F8 v = pf_sum8(add, t, r);   // plane 0 is `out`
    float *o = out + (size_t)t * add.rows + r;
    if (((uintptr_t)o & 15) == 0) { pf_store8(o, v); return; }
#pragma unroll
    for (int k = 0; k < 8; k++) o[k] = v.v[k];
}

// The same, one column per thread and eight planes requested at a time: for results of few columns and dozens of planes
__global__ void __launch_bounds__(256) prefill_finish_narrow_kernel(float *out, const PfPlanes add) {
    pf_enter();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= add.n * add.rows) return;
    const uint32_t t = i / add.rows, r = i - t * add.rows, np = add.sk.pieces(add.sk.row_tile(r) * add.chunks + t / PF_CHUNK);
    if (np == 1) return;
    const size_t plane = (size_t)add.n * add.rows;
    const float *p = add.planes + i;
    float v = __ldcg(out + i);
    uint32_t s = 1;
    for (; s + 8 <= np; s += 8) {
        float a[8];
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = __ldcg(p + (s - 1 + k) * plane);
#pragma unroll
        for (int k = 0; k < 8; k++) v += a[k];
    }
    for (; s < np; s++) v += __ldcg(p + (s - 1) * plane);
    out[i] = v;
}

// A warp: 8 tokens x 32 columns, which are whole lines of the next GEMM's inputs (a warp of one token's 256 columns writes 16 bytes of each of 32 lines)
__global__ void __launch_bounds__(256) prefill_swiglu_kernel(const PfPlanes gu, __half *xt) {
    pf_enter();
    const uint32_t F = gu.rows / 2, per = F / 256, lane = threadIdx.x & 31, group = blockIdx.x / per;   // F % 256 == 0
    const uint32_t t = group * 8 + (lane >> 2), c = (blockIdx.x - group * per) * 256 + (threadIdx.x >> 5) * 32 + (lane & 3) * 8;
    F8 y = {{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}};
    if (t < gu.n) {
        const F8 a = pf_sum8(gu, t, c), b = pf_sum8(gu, t, F + c);
#pragma unroll
        for (int k = 0; k < 8; k++) y.v[k] = b.v[k] * (a.v[k] / (1.0f + expf(-a.v[k])));   // crates/inferi-shaders/src/silu.rs:16-19,46-52
    }
    pf_emit8(xt, t, c, F, y);
}

// Eight rows (four rotation pairs) of q, k or v of one token: bias (transformer.rs:434-442), rotation of adjacent pairs
// (crates/inferi-shaders/src/rope.rs:75-91, the angle as the decode path forms it), q out or cache append.
template <int DEPTH>
__global__ void __launch_bounds__(256) prefill_qkv_kernel(const PfQkv p) {
    pf_enter();
    const uint32_t per = (p.q_dim + 2 * p.kv_dim) / 8, i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n * per) return;
    const uint32_t t = i / per;
    uint32_t r = (i - t * per) * 8, which = 0;
    if (r >= p.q_dim) { r -= p.q_dim; which = 1; if (r >= p.kv_dim) { r -= p.kv_dim; which = 2; } }
    F8 v = pf_sum8<DEPTH>(which == 0 ? p.g[0] : (which == 1 ? p.g[1] : p.g[2]), t, (which == 0 ? p.row0[0] : (which == 1 ? p.row0[1] : p.row0[2])) + r);
    const float *bias = which == 0 ? p.bias[0] : (which == 1 ? p.bias[1] : p.bias[2]);
    if (bias) pf_add8(v, F8{{bias[r], bias[r + 1], bias[r + 2], bias[r + 3], bias[r + 4], bias[r + 5], bias[r + 6], bias[r + 7]}});
    if (which < 2) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float sn, cs;
            sincosf((float)(p.pos0 + t) * p.theta[((r + 2 * k) % p.head_size) >> 1], &sn, &cs);
            const float x = v.v[2 * k], y = v.v[2 * k + 1];
            v.v[2 * k] = cs * x - sn * y;
            v.v[2 * k + 1] = sn * x + cs * y;
        }
    }
    if (which == 0) { pf_store8(p.q + (size_t)t * p.q_dim + r, v); return; }
    void *cache = which == 1 ? p.k_cache : p.v_cache;
    const size_t off = (size_t)(p.pos0 + t) * p.kv_dim + r;
    if (p.kv_dtype == IB_KV_F16) {
        uint32_t h[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const __half2 hh = __floats2half2_rn(v.v[2 * k], v.v[2 * k + 1]);
            h[k] = *reinterpret_cast<const uint32_t *>(&hh);
        }
        *reinterpret_cast<uint4 *>(reinterpret_cast<__half *>(cache) + off) = make_uint4(h[0], h[1], h[2], h[3]);
    } else pf_store8(reinterpret_cast<float *>(cache) + off, v);
}

// ---------------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------------
template <typename... KArgs, typename... Args>
static int32_t pf_launch(ib_ctx *ctx, cudaStream_t s, void (*kernel)(KArgs...), dim3 grid, uint32_t block, const Args &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
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

int32_t launch_prefill_embed(ib_ctx *ctx, cudaStream_t s, const ib_qtensor *embd, const uint32_t *tokens_dev, uint32_t n, uint32_t vocab, float *X) {
    const QDesc e{embd->dev, embd->row_bytes, (uint32_t)embd->qtype, embd->layout, embd->nb};
    const uint32_t hidden = (uint32_t)embd->cols;
    return pf_launch(ctx, s, prefill_embed_kernel, (uint32_t)(((size_t)n * hidden + 255) / 256), 256, e, tokens_dev, n, hidden, vocab, X);
}

// Where tiles are cut into many pieces (few tokens: a tile has few units of work, and they are dealt out), four of their planes are requested at a time.
// A layer, us, two / four / eight: 2048 hidden, 9 tokens 73.5 / 70.7 / 71.0, 45 80.8 / 78.7 / 80.6, 100 91.8 / 87.0 / 88.1, 300 151.0 / 148.4 / 152.2; 4096 hidden, 9
// 126.7 / 124.7 / 127.1, 128 164.4 / 162.0 / 159.8.  (In every kernel alike, also where a tile has a plane or two, four were slower.)
constexpr int PF_DEEP = 4;
static bool pf_deep(const StreamK &sk) { return prefill_max_pieces(sk) > 3; }

// Tokens from which several share a CTA.  With a norm two, of which two CTAs fit an SM: a layer, one / four / two tokens per CTA, us: 4096 hidden, 512 tokens 351.2 / 349.1 /
// 346.7, 600 (152 CTAs of four: two waves) 410.8 / 416.9 / 407.5, 1021 658.0 / 654.0 / 652.7; 2048 hidden, 512 199.2 / 190.7 / 189.1, 1021 336.6 / 329.4 / 326.9.  Their halves
// need rows of 2048 or 4096 columns; four for others that a CTA holds in its registers; longer rows, read twice, took 64.1 us instead of 58.5 (2048 x 8192
// Q4_K, 700 tokens, the GEMM with its inputs), a layer of 8192 hidden at 600 tokens 706 instead of 687.  Without a norm nothing is held, and rows are shared
// out to CTAs of 4096 columns: 2048 x 1024, 1000 tokens 21.0 us (one token per CTA 25.6), x 8192, 700 55.5 (58.4), x 14336, 700 91.0 (94.6; with four whole rows
// per CTA 102.5: 176 CTAs of 148 at a time).
constexpr uint32_t PF_MANY_TOKENS = 512;
int32_t launch_prefill_norm_split(ib_ctx *ctx, cudaStream_t s, float *X, const PfPlanes *add, const float *w, float eps, uint32_t n, uint32_t cols, __half *xt) {
    constexpr uint32_t held = PF_KEEP * PF_ROW_THREADS * 8;   // columns that a CTA holds in its registers
    const uint32_t rows = (n + 15) & ~15u;
    const PfPlanes planes = add ? *add : PfPlanes{};
    auto launch = [&](auto kernel, uint32_t tokens) {
        const dim3 grid(rows / tokens, w ? 1 : (cols + held / tokens - 1) / (held / tokens));
        return pf_launch(ctx, s, kernel, grid, PF_ROW_THREADS, X, planes, add ? 1u : 0u, w, eps, n, cols, xt);
    };
    const bool many = n >= PF_MANY_TOKENS;
    if (!w) return many ? launch(prefill_norm_split_kernel<4, 2, false>, 4) : launch(prefill_norm_split_kernel<1, 2, false>, 1);
    if (many && cols <= held / 4)
        return cols % (held / 8) == 0 ? launch(prefill_norm_split_kernel<2, 2, true>, 2) : launch(prefill_norm_split_kernel<4, 2, true>, 4);
    return add && pf_deep(add->sk) ? launch(prefill_norm_split_kernel<1, PF_DEEP, true>, 1) : launch(prefill_norm_split_kernel<1, 2, true>, 1);
}

static uint32_t pf_grid(size_t threads) { return (uint32_t)((threads + 255) / 256); }

int32_t launch_prefill_residual(ib_ctx *ctx, cudaStream_t s, float *X, const PfPlanes &add) {
    return pf_launch(ctx, s, prefill_residual_kernel, pf_grid((size_t)add.n * add.rows / 8), 256, X, add);
}
int32_t launch_prefill_finish(ib_ctx *ctx, cudaStream_t s, float *out, const PfPlanes &add) {
    // A matrix of few rows is cut into dozens of pieces, and threads of eight columns each are then too few to bring the planes in
    // (Q4_K 512 x 14336, 38 planes, the whole GEMM, eight columns / one: 64 tokens 42.9 / 22.8 us, 128 tokens 44.3 / 24.7,
    // 300 tokens 43.1 / 34.3).  Where eight columns each are a CTA per SM they do as well.
    const size_t columns = (size_t)add.n * add.rows;
    if (prefill_max_pieces(add.sk) > 8 && columns < (size_t)8 * 256 * (uint32_t)ctx->sm_count) return pf_launch(ctx, s, prefill_finish_narrow_kernel, pf_grid(columns), 256, out, add);
    return pf_launch(ctx, s, prefill_finish_kernel, pf_grid(columns / 8), 256, out, add);
}
int32_t launch_prefill_swiglu(ib_ctx *ctx, cudaStream_t s, const PfPlanes &gu, __half *xt) {
    return pf_launch(ctx, s, prefill_swiglu_kernel, ((gu.n + 15) & ~15u) / 8 * (gu.rows / 512), 256, gu, xt);
}
int32_t launch_prefill_qkv(ib_ctx *ctx, cudaStream_t s, const PfQkv &p) {
    const bool deep = pf_deep(p.g[0].sk) || pf_deep(p.g[1].sk) || pf_deep(p.g[2].sk);
    return pf_launch(ctx, s, deep ? prefill_qkv_kernel<PF_DEEP> : prefill_qkv_kernel<2>, pf_grid((size_t)p.n * (p.q_dim + 2 * p.kv_dim) / 8), 256, p);
}

}  // namespace ib

using namespace ib;

extern "C" int32_t ib_gemm_quant(ib_ctx *ctx, void *stream, float *out_dev, const ib_qtensor *m, const float *x_dev, uint32_t n) {
    IB_REQUIRE(ctx && m && out_dev && x_dev, "ib_gemm_quant: null argument");
    IB_REQUIRE(m->ctx->device == ctx->device, "ib_gemm_quant: tensor lives on device %d, context on %d", m->ctx->device, ctx->device);
    IB_REQUIRE(n >= 1, "ib_gemm_quant: no rows");
    // Q6_K and Q8_0 matrices whose rows are wider than the GEMV takes are not in the re-tiled layout: re-tiled into the scratch by every
    // call, one read and one write of the matrix ahead of a GEMM that reads it at least once more.  (Rows that the layout cannot hold, Q6_K of
    // no multiple of 8 blocks, are refused.)
    ib_qtensor tiled = *m;
    const bool retile = m->layout == LAYOUT_GGUF && (m->qtype == IB_Q6_K || m->qtype == IB_Q8_0) && m->nb % 8 == 0;
    if (retile) {
        tiled.layout = LAYOUT_SOA;
        tiled.dev = nullptr;
    }
    if (!prefill_gemm_eligible(&tiled))
        return set_error(IB_ERR_UNSUPPORTED, "ib_gemm_quant: %llux%llu of type %d (the tensor-core path takes Q8_0/Q4_K/Q5_K/Q6_K with rows %% 128 == 0 and cols %% 256 == 0)",
                         (unsigned long long)m->rows, (unsigned long long)m->cols, m->qtype);
    int prev = -1;
    cudaGetDevice(&prev);
    IB_REQUIRE(cudaSetDevice(ctx->device) == cudaSuccess, "cudaSetDevice failed");
    cudaStream_t s = (cudaStream_t)stream;
    const uint32_t rows = (uint32_t)m->rows, cols = (uint32_t)m->cols;
    // a pass: what the layers of a prompt take, and less where the split planes of a tall matrix would grow beyond 512 MiB
    uint32_t pass = n < PREFILL_MAX_TOKENS ? n : PREFILL_MAX_TOKENS;
    if (pass > ctx->tc_pass) pass = ctx->tc_pass;
    auto bytes_of = [&](uint32_t nc, size_t &half_bytes) {
        const StreamK sk = prefill_streamk(ctx, rows, cols, nc);
        half_bytes = (nc + PF_CHUNK - 1) / PF_CHUNK * pf_x_halves(cols) * sizeof(__half);
        return half_bytes + (((size_t)(prefill_max_pieces(sk) - 1) * nc * rows * sizeof(float) + 255) & ~(size_t)255);
    };
    auto shorter = [](uint32_t p) { return (p / 2 + PF_CHUNK - 1) / PF_CHUNK * PF_CHUNK; };
    size_t half_bytes = 0;
    while (pass > PF_CHUNK && bytes_of(pass, half_bytes) > ((size_t)512 << 20)) pass = shorter(pass);
    size_t need, tiled_at;
    int32_t rc = IB_OK;
    for (;; pass = shorter(pass)) {
        need = bytes_of(pass, half_bytes);
        if (n % pass) {   // the last, shorter pass may split its tiles further
            size_t hb = 0;
            const size_t last = bytes_of(n % pass, hb) - hb + half_bytes;
            if (last > need) need = last;
        }
        tiled_at = need;
        if (retile) need += m->rows * tiled.row_bytes;
        if (need <= ctx->tc_scratch_bytes) break;
        // growing the scratch: wait for work that may still use the old one
        cudaError_t e = cudaDeviceSynchronize();
        if (e == cudaSuccess && ctx->tc_scratch) e = cudaFree(ctx->tc_scratch);
        ctx->tc_scratch = nullptr;
        ctx->tc_scratch_bytes = 0;
        if (e == cudaSuccess) e = cudaMalloc(&ctx->tc_scratch, need);
        if (e == cudaSuccess) {
            ctx->tc_scratch_bytes = need;
            break;
        }
        cudaGetLastError();
        ctx->tc_scratch = nullptr;
        if (e == cudaErrorMemoryAllocation && pass > PF_CHUNK) {   // shorter passes rather than none
            ctx->tc_pass = shorter(pass);
            continue;
        }
        rc = set_error(e == cudaErrorMemoryAllocation ? IB_ERR_OOM : IB_ERR_CUDA, "ib_gemm_quant: scratch of %llu bytes: %s", (unsigned long long)need, cudaGetErrorString(e));
        break;
    }
    __half *xt = reinterpret_cast<__half *>(ctx->tc_scratch);
    float *planes = reinterpret_cast<float *>((uint8_t *)ctx->tc_scratch + half_bytes);
    if (retile && rc == IB_OK) {
        tiled.dev = (uint8_t *)ctx->tc_scratch + tiled_at;
        rc = retile_to_soa(ctx, s, m->qtype, m->dev, tiled.dev, m->rows, m->nb);
    }
    const ib_qtensor *w = &tiled;
    for (uint32_t t0 = 0; rc == IB_OK && t0 < n; t0 += pass) {
        const uint32_t nc = n - t0 < pass ? n - t0 : pass;
        const StreamK sk = prefill_streamk(ctx, rows, cols, nc);
        float *out = out_dev + (size_t)t0 * rows;   // plane 0 of every tile
        rc = launch_prefill_norm_split(ctx, s, const_cast<float *>(x_dev) + (size_t)t0 * cols, nullptr, nullptr, 0.f, nc, cols, xt);
        if (rc == IB_OK) rc = launch_prefill_gemm(ctx, s, PrefillPart{&w, 1, out, planes, sk}, xt, nc, !retile);
        if (rc == IB_OK && prefill_max_pieces(sk) > 1) rc = launch_prefill_finish(ctx, s, out, PfPlanes{out, planes, sk, rows, (nc + PF_CHUNK - 1) / PF_CHUNK, nc});
    }
    if (prev >= 0 && prev != ctx->device) cudaSetDevice(prev);
    return rc;
}
