// Grouped-query decode attention over the KV cache: split-K flash-decoding with a log-sum-exp merge.
//
// Replaces crates/inferi-shaders/src/fused_attention.rs:63-241 (fused_attention, <= 2048 positions) and
// :374-617 (flash_attention) and their launcher crates/inferi/src/ops/batched_multiquery_attention.rs:27-77.
// Semantics follow `run_cpu` (:191-245): score = q.k / sqrt(head_size), softmax over positions 0..=pos, weighted
// sum of V.  Cache rows are [position, kv_dim] (fused_attention.rs:107-108), f32 as in the reference or f16.
//
// A group of up to four query heads of one kv head shares the slices' K and V rows (the reference reads them once per query head, one workgroup each);
// eight heads are two groups, which read the same rows.  One CTA per (group, position slice) leaves an un-normalised partial (max, sum,
// accumulator): many slices in global memory, where the last CTA of a group to arrive merges them and none waits for another; few slices
// in the shared memory of the first CTA of their cluster, whose barrier they meet at (attention_group.cuh).  The split follows from the
// position on the device, so the same launch (and the same CUDA graph node) serves every context length of its regime.
#include "attention_group.cuh"

namespace ib {

size_t attn_scratch_bytes(const ib_attn_params &p, uint32_t max_splits) {
    const size_t n_kv = p.n_heads / p.kv_mul;
    return n_kv * max_splits * p.kv_mul * (p.head_size + 2) * sizeof(float);
}

// The merging CTA keeps the weights of ATTN_MAX_SLICES slices.  (Head size 64: half as many.  Only one to three groups of heads could use more; whether
// they gain by it has not been measured.)
static uint32_t attn_slice_limit(const ib_attn_params &p) { return 2 * p.head_size < ATTN_MAX_SLICES ? 2 * p.head_size : ATTN_MAX_SLICES; }

uint32_t attn_max_splits(const ib_ctx *ctx, const ib_attn_params &p) {
    const uint32_t groups = attn_groups(p);
    uint32_t s = (uint32_t)(ctx->sm_count * 3) / (groups ? groups : 1);   // three CTAs fit one SM: one wave
    if (s < 1) s = 1;
    const uint32_t most = attn_slice_limit(p);
    return s < most ? s : most;
}

// CTAs per cluster, one cluster per kv head.  Short: 8 while that is three (head size 128: two) on every SM, and from there on as many as fit
// with one per SM (head size 64, 400 positions: 26 kv heads 4.8 us in clusters of 8, 6.6 in clusters of 4; 64 heads 8.1 and 6.8).
// Middle: its CTAs need an SM each and their clusters a GPC with so many free ones; on more than two thirds of the SMs some clusters wait
// for others (12 kv heads x 8 CTAs fit; 16 x 8 take twice the time: 13.4 us against 8.9 as 16 x 4 at 2048 positions).  Fewer than 4 CTAs per kv head: no middle regime.
static uint32_t attn_cluster_ctas(const ib_ctx *ctx, const ib_attn_params &p, uint32_t regime) {
    const uint32_t n_kv = attn_groups(p), room = (uint32_t)ctx->sm_count * 2 / (regime == ATTN_MIDDLE ? 3 : 2);
    uint32_t c = ATTN_CLUSTER_MAX;
    if (regime == ATTN_SHORT && c * n_kv <= (p.head_size == 128 ? 2 : 3) * (uint32_t)ctx->sm_count) return c;
    while (c > 1 && c * n_kv > room) c /= 2;
    return regime == ATTN_MIDDLE && (c < 4 || c * n_kv > room) ? 0u : c;
}

// Up to how many positions per CTA of a kv head's cluster a regime is the fastest.  A cluster regime's time hardly depends on the number
// of kv heads, the long one's does: with few heads it has more CTAs per head.  Measured us per launch, short / middle / long:
//   head size 64:   4 kv heads  5.3 / 6.2 / 6.5 at 1536 positions, 6.1 / 6.6 / 7.0 at 2048;  8 heads  4.4 / 5.7 / 6.6 at 640, 4.9 / 5.9 / 6.8 at
//                   1024, 6.7 / 6.3 / 7.6 at 1536;  16 (middle in clusters of 4)  5.0 / 6.0 / 7.0 at 768, 6.8 / 6.8 / 7.9 at 1024.
//                   Middle against long, launches back to back (caches that stay in L2): 8.3 / 7.4 at 5000 with 4 heads (12.3 / 9.2 at 10000),
//                   7.6 / 7.5 at 4000 with 8 (10.9 / 9.2 at 8000, 17.4 / 12.3 at 16000), 8.4 / 8.3 at 5000 with 12 (14.0 / 12.4 at 12000), 7.6 /
//                   6.9 at 2000 with 16.  Inside a token graph the middle regime leaves SMs for the next launch's CTAs, which is worth up to 1.3 us
//                   (1B architecture, a layer of a token, 2000 positions: 26.5 / 27.9 us, 3000: 27.5 / 28.6): the limits lie that much further.
//   head size 128:  8 kv heads  3.6 / 4.1 / 4.2 at 128, 4.0 / 4.2 / 4.5 at 192, 4.2 / 4.1 / 4.4 at 224, 5.0 / 4.5 / 6.2 at 512.
//                   Middle against long: 6.8 / 6.1 at 2000 with 2 heads, 6.9 / 6.2 at 1800 with 4, 7.0 / 7.2 at 1800 with 8 (8.9 / 8.6 at 3000),
//                   8.0 / 8.9 at 2500 with 12;  16 heads  5.7 / 6.1 at 600, 7.1 / 6.6 at 1000.  In the graph (a layer of the 8B shapes): 45.6 / 46.9
//                   at 1900, 48.7 / 48.0 at 2700;  4 heads  28.3 / 29.9 at 1600.
// The middle regime's ends are those of the token graph (for head size 64 beyond 3000 positions: the crossing back to back, moved by that margin).  Launches outside it, which take the same ones, would cross over earlier by the
// figures above: up to 0.9 us of 8 between 4000 and 6400 positions of up to 8 heads of 64, 0.7 of 7 below 2560 positions of 2 to 4 heads of 128.
// Groups of one or two heads and the f32 cache have no middle regime; short / long, us: f16, head size 128, 8 x 2 heads 2.9 / 3.7 at 200 positions, 4.3 / 4.1 at
// 450, 16 x 1 4.3 / 4.5 at 450 (6.1 / 5.6 at 900); head size 64, 8 x 2 3.2 / 3.6 at 500 (4.2 / 3.9 at 600).  f32, head size 128, 8 x 4 4.6 / 5.0 at 200,
// 6.4 / 5.1 at 450, 8 x 8 3.7 / 4.1 at 60, 6.0 / 5.0 at 200, 16 x 1 4.0 / 4.2 at 200, 4.6 / 4.3 at 260; head size 64, 8 x 4 2.9 / 3.5 at 200, 4.2 / 4.0 at 450, 8 x 1 3.8 / 3.8 at 380.
// (2 to 4 heads of 128 end at 2560, 8 at 2400: the latter was measured in the graph up to its crossing, the former at 1600 only.)
uint32_t attn_regime_positions(const ib_ctx *ctx, const AttnLaunch &a, uint32_t regime) {
    if (ctx->sm_count == 0) return 0u;
    if (regime == ATTN_LONG) return a.p.kv_mul <= 2 ? ATTN_ALONE : 0u;
    const bool has_middle = a.kv_dtype == IB_KV_F16 && a.p.kv_mul >= ATTN_GROUP;
    const uint32_t n_kv = attn_groups(a.p), middle = has_middle ? attn_cluster_ctas(ctx, a.p, ATTN_MIDDLE) : 0u;
    const uint32_t c = regime == ATTN_MIDDLE ? middle : attn_cluster_ctas(ctx, a.p, regime);
    const bool wide = a.p.head_size == 128;
    if (regime == ATTN_MIDDLE) return c * (wide ? (c < 8 ? 256 : (n_kv <= 4 ? 320 : (n_kv <= 8 ? 300 : 384))) : (c < 8 ? 512 : (n_kv <= 8 ? 800 : 1400)));
    if (!has_middle) return c * (wide ? (a.kv_dtype == IB_KV_F16 ? 48 : (a.p.kv_mul > ATTN_GROUP ? 16 : 32)) : (a.kv_dtype == IB_KV_F16 ? 64 : 48));
    if (middle == 0 || c < 8) return c * (wide && middle ? 24 : 64);
    return c * (wide ? 24 : (middle < 8 ? 96 : (n_kv <= 4 ? 256 : 128)));
}

static bool attn_aligned(const float *q, const float *out) { return ((uintptr_t)q % 16) == 0 && ((uintptr_t)out % 16) == 0; }

template <int HS, int KVM, typename T, uint32_t REGIME, bool ALIGNED = true>
static int32_t launch_group(ib_ctx *ctx, cudaStream_t s, const AttnArgs &args, dim3 grid) {
    constexpr uint32_t smem = attn_smem_floats(HS, KVM, REGIME) * sizeof(float);
    static_assert(smem + 4096 <= 49152, "dynamic and static shared memory without opting in");
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(attn_warps(HS, REGIME) * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = REGIME != ATTN_LONG ? grid.y : 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = args.pdl ? 2 : 1;
    IB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, attn_group_kernel<HS, KVM, T, REGIME, ALIGNED>, args));
    ctx->launches++;
    return IB_OK;
}

template <int HS, int KVM, typename T>
static int32_t launch_regime(ib_ctx *ctx, cudaStream_t s, const AttnArgs &args, dim3 grid, uint32_t regime) {
    if (!attn_aligned(args.q, args.out)) return launch_group<HS, KVM, T, ATTN_LONG, false>(ctx, s, args, grid);
    if constexpr (KVM == (int)ATTN_GROUP && sizeof(T) == 2)
        if (regime == ATTN_MIDDLE) return launch_group<HS, KVM, T, ATTN_MIDDLE>(ctx, s, args, grid);
    return regime == ATTN_SHORT ? launch_group<HS, KVM, T, ATTN_SHORT>(ctx, s, args, grid) : launch_group<HS, KVM, T, ATTN_LONG>(ctx, s, args, grid);
}

template <int HS, typename T>
static int32_t launch_heads(ib_ctx *ctx, cudaStream_t s, const AttnArgs &args, dim3 grid, uint32_t regime) {
    switch (args.p.kv_mul) {
    case 1: return launch_regime<HS, 1, T>(ctx, s, args, grid, regime);
    case 2: return launch_regime<HS, 2, T>(ctx, s, args, grid, regime);
    case 4: case 8: return launch_regime<HS, 4, T>(ctx, s, args, grid, regime);
    default: return set_error(IB_ERR_UNSUPPORTED, "attention: kv_mul=%u (supported: 1, 2, 4, 8)", args.p.kv_mul);
    }
}

int32_t launch_attention(ib_ctx *ctx, cudaStream_t s, const AttnLaunch &a) {
    const ib_attn_params &p = a.p;
    IB_REQUIRE(p.kv_mul >= 1 && p.n_heads % p.kv_mul == 0, "attention: n_heads=%u is not a multiple of kv_mul=%u", p.n_heads, p.kv_mul);
    const uint32_t n_kv = p.n_heads / p.kv_mul;
    IB_REQUIRE(p.kv_dim == n_kv * p.head_size, "attention: kv_dim=%u != n_kv_heads*head_size=%u", p.kv_dim, n_kv * p.head_size);
    IB_REQUIRE(a.pos_ptr || p.pos < p.seq_len, "attention: pos=%u outside the cache of %u rows", p.pos, p.seq_len);
    IB_REQUIRE(a.max_splits >= 1 && a.max_splits <= attn_slice_limit(p), "attention: %u position slices (1 to %u)", a.max_splits, attn_slice_limit(p));
    IB_REQUIRE(((uintptr_t)a.k_cache % 16) == 0 && ((uintptr_t)a.v_cache % 16) == 0, "attention: the caches must be 16-byte aligned");
    if (p.head_size != 64 && p.head_size != 128) return set_error(IB_ERR_UNSUPPORTED, "attention: head_size=%u (supported: 64, 128)", p.head_size);
    if (p.kv_mul != 1 && p.kv_mul != 2 && p.kv_mul != 4 && p.kv_mul != 8) return set_error(IB_ERR_UNSUPPORTED, "attention: kv_mul=%u (supported: 1, 2, 4, 8)", p.kv_mul);
    AttnArgs args{p, a.pos_ptr, a.q, a.k_cache, a.v_cache, a.out, a.scratch, a.counters, a.max_splits, a.pdl, 0u};
    // A launch that serves many positions (a graph node) is told the regime they are in.  A caller's q or output off the 16-byte boundaries: the long
    // one, whatever the position.
    const bool aligned = attn_aligned(a.q, a.out);
    uint32_t regime = aligned ? a.regime : ATTN_LONG;
    if (!a.pos_ptr && aligned) {
        uint32_t positions[3];
        for (uint32_t r : {ATTN_LONG, ATTN_SHORT, ATTN_MIDDLE}) positions[r] = attn_regime_positions(ctx, a, r);
        regime = attn_regime_of(positions, (uint64_t)p.pos + 1);
    }
    uint32_t splits = a.max_splits, per;
    if (regime != ATTN_LONG) args.cluster = splits = attn_cluster_ctas(ctx, p, regime);
    if (!a.pos_ptr) {   // with a host-known position only the slices that will do work are launched
        attn_plan(p.pos + 1, a.max_splits, args.cluster, attn_warps(p.head_size, regime), p.kv_mul, splits, per);
        if (regime != ATTN_LONG) args.cluster = splits;
    }
    const dim3 grid(attn_groups(p), splits);
    const bool f16 = a.kv_dtype == IB_KV_F16;
    if (p.head_size == 128) return f16 ? launch_heads<128, __half>(ctx, s, args, grid, regime) : launch_heads<128, float>(ctx, s, args, grid, regime);
    return f16 ? launch_heads<64, __half>(ctx, s, args, grid, regime) : launch_heads<64, float>(ctx, s, args, grid, regime);
}

}  // namespace ib

// -------------------------------------------------------------------------------------------------------------------
// ib_attention_static: decode attention for callers that must not allocate.
//
// Some hosts of this library run where device allocation is off limits once set-up is over: a real-time audio/serving
// thread that may not take the allocator's locks, a plugin whose host application owns the memory budget, code running
// inside a region where cudaMalloc would synchronise the device.  ib_attention() grows a scratch buffer with cudaMalloc
// on demand and needs a context (whose creation allocates); this variant needs neither.  Its split-K scratch is the
// fixed array below, part of the library image: every GPU that loads the library carries these ~1 MiB until the process
// exits, whether or not the entry point is ever called.
// -------------------------------------------------------------------------------------------------------------------
namespace ib {
constexpr uint32_t STATIC_ATTN_FLOATS = 262144;    // 1 MiB of partials: bounds n_heads * (head_size + 2) * splits
constexpr uint32_t STATIC_ATTN_KV_HEADS = 256;     // arrival counters: two per kv head at most (attn_groups)
constexpr uint32_t STATIC_ATTN_MAX_SPLITS = 32;
constexpr int STATIC_ATTN_MAX_DEVICES = 64;
}  // namespace ib

static __device__ __align__(256) float g_static_attn_scratch[ib::STATIC_ATTN_FLOATS];
static __device__ __align__(256) unsigned int g_static_attn_counters[2 * ib::STATIC_ATTN_KV_HEADS];

// Device addresses of the two arrays, looked up once per device.  In host code the array names above are only
// host-side stand-ins for the symbols; the addresses a kernel can use come from cudaGetSymbolAddress, called with the
// device in question current.
static float *g_static_scratch_addr[ib::STATIC_ATTN_MAX_DEVICES];
static unsigned int *g_static_counters_addr[ib::STATIC_ATTN_MAX_DEVICES];

extern "C" int32_t ib_attention_static(void *stream, const ib_attn_params *params, const float *q_dev, const void *k_cache_dev,
                                       const void *v_cache_dev, int32_t kv_dtype, float *out_dev) {
    using namespace ib;
    IB_REQUIRE(params && q_dev && k_cache_dev && v_cache_dev && out_dev, "ib_attention_static: null argument");
    IB_REQUIRE(kv_dtype == IB_KV_F32 || kv_dtype == IB_KV_F16, "ib_attention_static: unknown kv dtype %d", kv_dtype);
    const ib_attn_params &p = *params;
    IB_REQUIRE(p.kv_mul >= 1 && p.n_heads >= p.kv_mul && p.n_heads % p.kv_mul == 0 && p.head_size > 0, "ib_attention_static: bad head counts");
    const uint32_t n_kv = p.n_heads / p.kv_mul;
    const uint64_t per_split = (uint64_t)p.n_heads * (p.head_size + 2);   // floats one split of all heads leaves behind
    if (n_kv > STATIC_ATTN_KV_HEADS || per_split > STATIC_ATTN_FLOATS)
        return set_error(IB_ERR_UNSUPPORTED,
                         "ib_attention_static: %u heads of %u exceed the built-in scratch (n_heads * (head_size + 2) <= %u, kv heads <= %u); "
                         "use ib_attention, which allocates",
                         p.n_heads, p.head_size, STATIC_ATTN_FLOATS, STATIC_ATTN_KV_HEADS);
    uint32_t splits = (uint32_t)(STATIC_ATTN_FLOATS / per_split);
    if (splits > STATIC_ATTN_MAX_SPLITS) splits = STATIC_ATTN_MAX_SPLITS;

    int dev = -1;
    IB_CHECK_CUDA(cudaGetDevice(&dev));
    IB_REQUIRE(dev >= 0 && dev < STATIC_ATTN_MAX_DEVICES, "ib_attention_static: device ordinal %d not supported", dev);
    if (!g_static_scratch_addr[dev]) {
        // first call on this device: resolve the symbols.  With lazy module loading this is also the moment the driver loads
        // the module that holds the arrays (which may allocate and synchronise): make this call during set-up.
        float *s = nullptr;
        unsigned int *c = nullptr;
        IB_CHECK_CUDA(cudaGetSymbolAddress((void **)&s, g_static_attn_scratch));
        IB_CHECK_CUDA(cudaGetSymbolAddress((void **)&c, g_static_attn_counters));
        g_static_counters_addr[dev] = c;
        g_static_scratch_addr[dev] = s;
    }
    ib_ctx local;                 // plain bookkeeping struct on the stack: launch_attention only counts launches in it
    local.device = dev;
    AttnLaunch a = {};
    a.p = p;
    a.q = q_dev; a.k_cache = k_cache_dev; a.v_cache = v_cache_dev; a.kv_dtype = kv_dtype; a.out = out_dev;
    a.scratch = g_static_scratch_addr[dev];
    a.counters = g_static_counters_addr[dev];   // zero when the library is loaded; the kernel puts every counter back to zero
    a.max_splits = splits;
    a.pdl = 2;
    return launch_attention(&local, (cudaStream_t)stream, a);
}
