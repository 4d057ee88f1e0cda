// Causal attention of a prompt: every query of the pass over the cache rows up to its own position.
//
// Semantics follow `run_cpu` of crates/inferi-shaders/src/fused_attention.rs:191-245, as the decode kernels do: score =
// q.k / sqrt(head_size), softmax over positions 0 .. pos0 + t, weighted sum of V; the cache is f16.  The reference has no
// counterpart: it feeds a prompt token by token.
//
// One CTA: 16 tokens x the 4 query heads of a kv head = 64 score rows; a warp is one head.  Tiles of 64 positions of K and V go
// through shared memory once for all 64 rows (the decode kernel, one query per CTA, read the cache once per query: 34 ms of
// the 66 ms of a 1021-token prompt of the 8B architecture).  The products run on the tensor cores with mma.sync: at these sizes
// (a few tiles per CTA) a warp-level MMA whose operands and sums stay in registers has the shorter critical path, and the
// softmax works on the accumulators in place.
// Precision: K and V are exact in f16; q and the probabilities (f32) are split into two f16 (hi + lo, ~22 bits) and take two
// MMAs each; sums are f32.
//
// Short prompts in long contexts have few (16-token tile, kv head) pairs: the positions are then divided among the CTAs of a
// thread-block cluster (up to 8), which leave (max, sum, accumulator) in their own shared memory and merge row by row through
// distributed shared memory.  The result goes out as the next GEMM's inputs, split and tiled.
#include "prefill_emit.cuh"

#include <cooperative_groups.h>

namespace ib {

namespace cg = cooperative_groups;

constexpr int PA_TOK = 16, PA_HEADS = 4, PA_ROWS = PA_TOK * PA_HEADS, PA_KV = 64, PA_THREADS = 128;

struct PaParams {
    const float *q;          // [n][q_dim], rotated
    const __half *k, *v;     // this layer's cache [max_pos][kv_dim]
    __half *xt;              // the next GEMM's inputs: q_dim columns
    uint32_t n, pos0, q_dim, kv_dim, splits;
};

__device__ __forceinline__ void pa_mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void pa_ldm(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void pa_ldm_t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void pa_cp16(uint32_t dst, const void *src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src)); }
// (a, b) = hi + lo as packed f16 pairs
__device__ __forceinline__ void pa_split(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    const float2 f = __half22float2(h);
    const __half2 l = __floats2half2_rn(a - f.x, b - f.y);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = *reinterpret_cast<const uint32_t *>(&l);
}

template <int HS>
__global__ void __launch_bounds__(PA_THREADS) prefill_attention_kernel(const PaParams p) {
    constexpr int CH = HS / 8;                       // 16-byte chunks of a cache row
    constexpr uint32_t TILE = PA_KV * HS * 2;        // bytes of a K (or V) tile
    extern __shared__ __align__(128) uint8_t smem[];   // [2 stages][K, V]; at the end [64 rows][HS] f32 partials
    __shared__ float sm_m[PA_ROWS], sm_l[PA_ROWS];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t kvh = blockIdx.y, tt = gridDim.z - 1 - blockIdx.z, t0 = tt * PA_TOK;   // longest rows first
    const uint32_t S = p.splits, rank = blockIdx.x;   // the cluster runs along x
    const uint32_t last = p.pos0 + min(t0 + PA_TOK, p.n);              // positions 0 .. last - 1 matter to this tile
    const uint32_t tiles = (last + PA_KV - 1) / PA_KV, k_beg = rank * tiles / S, k_end = (rank + 1) * tiles / S;
    const uint32_t sm = (uint32_t)__cvta_generic_to_shared(smem);
    pf_enter();

    // 16-byte chunk `c` of row `r` sits at chunk c ^ (r & 7): the eight rows of an ldmatrix fall into different banks
    auto at = [&](uint32_t r, uint32_t c) { return r * (HS * 2) + (((c & ~7u) | ((c ^ r) & 7u)) << 4); };
    auto load_tile = [&](uint32_t kt, uint32_t stage) {
        const uint32_t base = sm + stage * 2 * TILE;
#pragma unroll
        for (int i = 0; i < PA_KV * CH / PA_THREADS; i++) {
            const uint32_t e = tid + i * PA_THREADS, r = e / CH, c = e % CH, pos = min(kt * PA_KV + r, last - 1);   // rows past the end repeat the last one (masked)
            const size_t g = (size_t)pos * p.kv_dim + kvh * HS + c * 8;
            pa_cp16(base + at(r, c), p.k + g);
            pa_cp16(base + TILE + at(r, c), p.v + g);
        }
        asm volatile("cp.async.commit_group;");
    };
    if (k_beg < k_end) load_tile(k_beg, 0);

    // the warp's 16 query rows (tokens t0 .. t0 + 15 of head kvh * 4 + warp) as A fragments, scaled into the exponent's base 2
    const uint32_t r_lo = lane >> 2, c2 = 2 * (lane & 3);
    uint32_t qh[HS / 16][4], ql[HS / 16][4];
    {
        const float scale = 1.4426950408889634f / sqrtf((float)HS);
        const uint32_t ta = min(t0 + r_lo, p.n - 1), tb = min(t0 + r_lo + 8, p.n - 1);
        const float *qa = p.q + (size_t)ta * p.q_dim + (kvh * PA_HEADS + warp) * HS + c2, *qb = p.q + (size_t)tb * p.q_dim + (kvh * PA_HEADS + warp) * HS + c2;
#pragma unroll
        for (int k = 0; k < HS / 16; k++) {
            const float2 x0 = __ldcg(reinterpret_cast<const float2 *>(qa + 16 * k)), x1 = __ldcg(reinterpret_cast<const float2 *>(qb + 16 * k));
            const float2 x2 = __ldcg(reinterpret_cast<const float2 *>(qa + 16 * k + 8)), x3 = __ldcg(reinterpret_cast<const float2 *>(qb + 16 * k + 8));
            pa_split(x0.x * scale, x0.y * scale, qh[k][0], ql[k][0]);
            pa_split(x1.x * scale, x1.y * scale, qh[k][1], ql[k][1]);
            pa_split(x2.x * scale, x2.y * scale, qh[k][2], ql[k][2]);
            pa_split(x3.x * scale, x3.y * scale, qh[k][3], ql[k][3]);
        }
    }
    const uint32_t lim_a = p.pos0 + t0 + r_lo, lim_b = lim_a + 8;   // last position each of the thread's two rows sees
    float O[HS / 8][4], m_a = -INFINITY, m_b = -INFINITY, l_a = 0.f, l_b = 0.f;
#pragma unroll
    for (int i = 0; i < HS / 8; i++) O[i][0] = O[i][1] = O[i][2] = O[i][3] = 0.f;

    for (uint32_t kt = k_beg; kt < k_end; kt++) {
        const uint32_t stage = (kt - k_beg) & 1, ks = sm + stage * 2 * TILE, vs = ks + TILE;
        if (kt + 1 < k_end) {
            load_tile(kt + 1, stage ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        float s[PA_KV / 8][4];
#pragma unroll
        for (int i = 0; i < PA_KV / 8; i++) s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f;
#pragma unroll
        for (int k = 0; k < HS / 16; k++) {
#pragma unroll
            for (int np = 0; np < PA_KV / 16; np++) {
                uint32_t b[4];
                pa_ldm(b, ks + at(16 * np + (lane & 7) + ((lane >> 4) << 3), 2 * k + ((lane >> 3) & 1)));
                pa_mma(s[2 * np], qh[k], b[0], b[1]);
                pa_mma(s[2 * np + 1], qh[k], b[2], b[3]);
                pa_mma(s[2 * np], ql[k], b[0], b[1]);
                pa_mma(s[2 * np + 1], ql[k], b[2], b[3]);
            }
        }
        if (kt * PA_KV + PA_KV - 1 > p.pos0 + t0) {   // the tile reaches beyond the first token's position
#pragma unroll
            for (int i = 0; i < PA_KV / 8; i++) {
                const uint32_t pos = kt * PA_KV + 8 * i + c2;
                if (pos > lim_a) s[i][0] = -INFINITY;
                if (pos + 1 > lim_a) s[i][1] = -INFINITY;
                if (pos > lim_b) s[i][2] = -INFINITY;
                if (pos + 1 > lim_b) s[i][3] = -INFINITY;
            }
        }
        float x_a = s[0][0], x_b = s[0][2];
#pragma unroll
        for (int i = 0; i < PA_KV / 8; i++) {
            x_a = fmaxf(x_a, fmaxf(s[i][0], s[i][1]));
            x_b = fmaxf(x_b, fmaxf(s[i][2], s[i][3]));
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            x_a = fmaxf(x_a, __shfl_xor_sync(0xffffffffu, x_a, o));
            x_b = fmaxf(x_b, __shfl_xor_sync(0xffffffffu, x_b, o));
        }
        // (a row that has seen no valid position yet keeps the maximum -inf; its weights are exp2(-inf - 0) = 0)
        const float n_a = fmaxf(m_a, x_a), n_b = fmaxf(m_b, x_b), f_a = n_a == -INFINITY ? 0.f : n_a, f_b = n_b == -INFINITY ? 0.f : n_b;
        const float w_a = exp2f(m_a - f_a), w_b = exp2f(m_b - f_b);
        m_a = n_a; m_b = n_b;
        l_a *= w_a; l_b *= w_b;
#pragma unroll
        for (int i = 0; i < HS / 8; i++) { O[i][0] *= w_a; O[i][1] *= w_a; O[i][2] *= w_b; O[i][3] *= w_b; }
#pragma unroll
        for (int k = 0; k < PA_KV / 16; k++) {
            uint32_t ph[4], pl[4];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float (&x)[4] = s[2 * k + h];
                x[0] = exp2f(x[0] - f_a); x[1] = exp2f(x[1] - f_a); x[2] = exp2f(x[2] - f_b); x[3] = exp2f(x[3] - f_b);
                l_a += x[0] + x[1];
                l_b += x[2] + x[3];
                pa_split(x[0], x[1], ph[2 * h], pl[2 * h]);
                pa_split(x[2], x[3], ph[2 * h + 1], pl[2 * h + 1]);
            }
#pragma unroll
            for (int dn = 0; dn < HS / 16; dn++) {
                uint32_t b[4];
                pa_ldm_t(b, vs + at(16 * k + (lane & 7) + (((lane >> 3) & 1) << 3), 2 * dn + (lane >> 4)));
                pa_mma(O[2 * dn], ph, b[0], b[1]);
                pa_mma(O[2 * dn + 1], ph, b[2], b[3]);
                pa_mma(O[2 * dn], pl, b[0], b[1]);
                pa_mma(O[2 * dn + 1], pl, b[2], b[3]);
            }
        }
        __syncthreads();   // the stage may be refilled
    }

    // partials to shared memory: row = head * 16 + token; 16-byte groups are swizzled by the row (a warp stores eight rows at once)
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
        l_a += __shfl_xor_sync(0xffffffffu, l_a, o);
        l_b += __shfl_xor_sync(0xffffffffu, l_b, o);
    }
    float *part = reinterpret_cast<float *>(smem);
    auto o_at = [](uint32_t r, uint32_t c) { return r * HS + (((c >> 2) ^ (r & 7)) << 2) + (c & 3); };
    const uint32_t ra = warp * PA_TOK + r_lo, rb = ra + 8;
#pragma unroll
    for (int i = 0; i < HS / 8; i++) {
        *reinterpret_cast<float2 *>(part + o_at(ra, 8 * i + c2)) = make_float2(O[i][0], O[i][1]);
        *reinterpret_cast<float2 *>(part + o_at(rb, 8 * i + c2)) = make_float2(O[i][2], O[i][3]);
    }
    if ((lane & 3) == 0) { sm_m[ra] = m_a; sm_l[ra] = l_a; sm_m[rb] = m_b; sm_l[rb] = l_b; }
    cg::cluster_group cluster = cg::this_cluster();
    if (S > 1) cluster.sync(); else __syncthreads();

    // merge and emit: the CTA's share of the rows, eight columns per thread (four neighbouring lanes: a 32-column sub-block)
    for (uint32_t e = rank * PA_THREADS + tid; e < PA_ROWS * CH; e += S * PA_THREADS) {
        const uint32_t r = e / CH, c = (e % CH) * 8, t = t0 + r % PA_TOK, head = kvh * PA_HEADS + r / PA_TOK;
        F8 y = {{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}};
        float mx = -INFINITY, sum = 0.f;
        for (uint32_t k = 0; k < S; k++) mx = fmaxf(mx, S > 1 ? *cluster.map_shared_rank(&sm_m[r], k) : sm_m[r]);
        for (uint32_t k = 0; k < S; k++) {
            const float *o = S > 1 ? cluster.map_shared_rank(part, k) : part;
            const float mk = S > 1 ? *cluster.map_shared_rank(&sm_m[r], k) : sm_m[r];
            const float w = mk == -INFINITY ? 0.f : exp2f(mk - mx);
            sum += w * (S > 1 ? *cluster.map_shared_rank(&sm_l[r], k) : sm_l[r]);
            const float4 a = *reinterpret_cast<const float4 *>(o + o_at(r, c)), b = *reinterpret_cast<const float4 *>(o + o_at(r, c + 4));
            y.v[0] += w * a.x; y.v[1] += w * a.y; y.v[2] += w * a.z; y.v[3] += w * a.w;
            y.v[4] += w * b.x; y.v[5] += w * b.y; y.v[6] += w * b.z; y.v[7] += w * b.w;
        }
        const float inv = t < p.n ? 1.0f / sum : 0.f;   // padding rows (up to a multiple of 16 tokens) are zero
#pragma unroll
        for (int i = 0; i < 8; i++) y.v[i] *= inv;
        pf_emit8(p.xt, t, head * HS + c, p.q_dim, y);
    }
    if (S > 1) cluster.sync();   // nobody leaves while its partials are being read
}

template <int HS>
static int32_t pa_launch(ib_ctx *ctx, cudaStream_t s, PaParams &p, uint32_t n_kv) {
    static bool attr_set[16] = {false};
    constexpr int smem = 2 * 2 * PA_KV * HS * 2;
    static_assert(smem >= PA_ROWS * HS * 4, "the partials reuse the tiles' memory");
    if (!attr_set[ctx->device & 15]) {
        IB_CHECK_CUDA(cudaFuncSetAttribute(prefill_attention_kernel<HS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
        attr_set[ctx->device & 15] = true;
    }
    // CTAs along the positions of one tile: as many as it takes to give every SM two CTAs, but no fewer than two tiles of
    // positions each (a CTA's set-up and the merge cost about as much as two tiles)
    const uint32_t token_tiles = (p.n + PA_TOK - 1) / PA_TOK, base = token_tiles * n_kv, tiles = (p.pos0 + p.n + PA_KV - 1) / PA_KV;
    p.splits = 1;
    while (p.splits < 8 && base * p.splits < 2u * (uint32_t)ctx->sm_count && tiles >= 4 * p.splits) p.splits *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.splits, n_kv, token_tiles);
    cfg.blockDim = dim3(PA_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    IB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, prefill_attention_kernel<HS>, (const PaParams)p));
    ctx->launches++;
    return IB_OK;
}

int32_t launch_prefill_attention(ib_ctx *ctx, cudaStream_t s, const float *q, const void *k_cache, const void *v_cache, uint32_t n, uint32_t pos0, uint32_t n_kv, uint32_t head_size,
                                 __half *xt) {
    PaParams p = {};
    p.q = q; p.k = (const __half *)k_cache; p.v = (const __half *)v_cache; p.xt = xt;
    p.n = n; p.pos0 = pos0; p.q_dim = n_kv * PA_HEADS * head_size; p.kv_dim = n_kv * head_size;
    switch (head_size) {
    case 128: return pa_launch<128>(ctx, s, p, n_kv);
    case 64: return pa_launch<64>(ctx, s, p, n_kv);
    default: return set_error(IB_ERR_UNSUPPORTED, "prefill attention: head_size=%u (supported: 64, 128)", head_size);
    }
}

}  // namespace ib
