// Decode attention: one launch's device side.  One CTA per (group of query heads, position slice), un-normalised partials, the last CTA of a group to
// arrive merges them; crates/inferi-shaders/src/fused_attention.rs:63-241 and :374-617 are what it replaces.  A group is up to four query heads
// of one kv head (eight are two groups, which read the same rows: the second time from L2), head size 64 or 128, an f16 or f32 cache.
// Built for a short critical path at small contexts and for few instructions per cache row at long ones:
//  * a lane holds 8 elements of a cache row and the matching 8 elements of the group's query vectors: 16 lanes a row of 128, 8 lanes a row of 64;
//    a warp iteration covers 8 rows (4 of f32 at head size 128: their registers; more of one or two heads, attn_steps);
//  * the per-lane partial scores of the step go through a halving exchange (each shuffle moves one value and
//    leaves half as many to reduce) instead of a butterfly per score: afterwards every lane owns exactly one
//    (row, head) score - two or four lanes the same one where a step has fewer scores than lanes - so exp() is evaluated once per score;
//  * the probabilities travel back to the lanes through 128 bytes of shared memory per warp;
//  * multiply-adds are issued as packed pairs (fma.rn.f32x2);
//  * the loop body is small (no 8-step unrolling): at short contexts the kernel runs its code once, and the time goes
//    to instruction fetch if the code is long.
#pragma once

#include "attention.cuh"

#include <cooperative_groups.h>

namespace ib {

constexpr uint32_t ATTN_GROUP = 4;   // query heads of a group, at most
__host__ __device__ constexpr uint32_t attn_groups(const ib_attn_params &p) { return p.n_heads / (p.kv_mul < ATTN_GROUP ? p.kv_mul : ATTN_GROUP); }

constexpr uint32_t ATTN_ROWS_PER_WARP_STEP = 8;
// Three ways to split a kv head's positions, by context length:
//  * short: the slices are the CTAs of one thread-block cluster, 4 warps each.  They leave their partials in the shared memory of the
//    cluster's first CTA (distributed shared memory) and meet at the cluster barrier; the first CTA merges from its own shared
//    memory.  Publishing the partials through global memory, counting arrivals with an atomic and reading them back are three L2
//    round trips (~2.6 us of a ~6 us kernel at these lengths); the cluster barrier is one hardware barrier.
//  * middle: the same with 8 or 16 warps per CTA, which hold the row loop at a few iterations.
//  * long: many CTAs of 4 warps (one wave of 3 per SM), merged through global memory.  Slices: one warp step of every warp (32
//    positions) each while there are at most 16 of them, then 16 slices that grow to 128 positions, then slices of 128
//    positions up to the launch's maximum, then longer ones.  Measured us per launch at 2500 / 4096 / 8192 / 16384 positions of 8 heads of
//    128: this plan 8.7 / 9.2 / 12.0 / 17.6, 32 positions each throughout 8.2 / 9.3 / 12.0 / 17.7, at least 256 each 9.8 / 9.9 / 13.0 / 17.7
//    (the merge fetches sixteen slices per L2 round trip; when it fetched eight, 32 each cost 12.6 at 2048 where the plan cost 9.2).
// Clusters have at most 8 CTAs: eight clusters of 16 - one per kv head of the Llama-3 models - do not all fit the GPU at once.
constexpr uint32_t ATTN_CLUSTER_MAX = 8, ATTN_MAX_SLICES = 256;
__host__ __device__ constexpr int attn_warps(uint32_t hs, uint32_t regime) { return regime != ATTN_MIDDLE ? ATTN_WARPS : (hs == 128 ? 8 : 16); }   // (head size 128 needs 196 registers a thread)
// Steps of a warp iteration: what of a slice is in flight, twice.  Four heads have registers for 8 rows (f32 at head size 128: 4); fewer heads need more rows, or
// long contexts wait for them (us, with the 8 rows of four heads / so: f16, head size 64, 30000 positions, 16 x 1 heads 36.2 / 26.3, 16 x 2 38.2 / 26.9, 5000 positions
// 9.8 / 8.3, 10.3 / 8.7; f32, 30000 positions of 16 x 1, head size 64 42.5 / 40.2, 128 78.6 / 73.9).  Eight steps of one f16 head: 25.0, but 11.1 / 10.5 at 8000.
__host__ __device__ constexpr int attn_steps(int hs, int heads, int bytes, uint32_t regime) {
    if (regime == ATTN_LONG && (bytes == 2 ? hs == 64 && heads <= 2 : heads == 1)) return 4;
    return bytes == 2 ? hs / 32 : 2;
}
constexpr uint32_t ATTN_MIN_PER_SPLIT = ATTN_WARPS * ATTN_ROWS_PER_WARP_STEP, ATTN_KNEE = 16, ATTN_KNEE_PER = 128;
// Rows of one or two heads that one CTA is as fast with as two that merge (60 rows, 16 x 1 heads of 128: 2.4 us, 2.7 as two).  It belongs to the long regime: a cluster
// starts when all of its CTAs find room at one time (a layer of a token, 32 x 1 heads of 64, 20 positions: 24.7 us, 25.2 as the one busy CTA of a cluster).
constexpr uint32_t ATTN_ALONE = 64;
__host__ __device__ __forceinline__ void attn_plan(uint32_t total, uint32_t max_splits, uint32_t cluster, uint32_t warps, uint32_t heads, uint32_t &nsplit, uint32_t &per) {
    if (heads <= 2 && total <= ATTN_ALONE) {
        nsplit = 1;
        per = total;
    } else if (cluster) {
        nsplit = (total + warps * ATTN_ROWS_PER_WARP_STEP - 1) / (warps * ATTN_ROWS_PER_WARP_STEP);
        if (nsplit > cluster) nsplit = cluster;
        per = (total + nsplit - 1) / nsplit;
        nsplit = (total + per - 1) / per;
    } else {
        attn_split_plan(total, max_splits, nsplit, per, ATTN_MIN_PER_SPLIT, ATTN_KNEE, ATTN_KNEE_PER);
    }
}

__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
    unsigned long long ra, rb, rc, rd;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(rc) : "f"(c.x), "f"(c.y));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(ra), "l"(rb), "l"(rc));
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
    return d;
}

// Halving exchange over the L lanes of a row: on entry every lane holds N partial sums (one per (step, head)); after the
// round with lane distance o the lanes whose bit o is set keep the upper half of the values, the others the lower half,
// each added to the partner's copy.  After log2(L) rounds (N == L) lane li of the row holds the complete sum number li.
template <int N>
__device__ __forceinline__ void halve_exchange(float (&v)[N], int lane, int o) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < N / 2; i++) {
        const float keep = up ? v[i + N / 2] : v[i];
        const float send = up ? v[i] : v[i + N / 2];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
}

// N consecutive floats of shared memory (aligned to all of them)
template <int N>
__device__ __forceinline__ void load_few(float (&f)[N], const float *p) {
    if constexpr (N == 4) {
        const float4 v = *reinterpret_cast<const float4 *>(p);
        f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
    } else if constexpr (N == 2) {
        const float2 v = *reinterpret_cast<const float2 *>(p);
        f[0] = v.x; f[1] = v.y;
    } else f[0] = p[0];
}

// o += w * p[0 .. N-1];  p[0 .. N-1] = w * o: in pairs where there are any (p is 8-byte aligned then)
template <int N>
__device__ __forceinline__ void add_scaled(float (&o)[N], float w, const float *p) {
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int e = 0; e < N; e += 2) {
            const float2 v = *reinterpret_cast<const float2 *>(p + e);
            o[e] += w * v.x;
            o[e + 1] += w * v.y;
        }
    } else {
#pragma unroll
        for (int e = 0; e < N; e++) o[e] += w * p[e];
    }
}
template <int N>
__device__ __forceinline__ void store_scaled(float *p, const float (&o)[N], float w) {
    if constexpr (N % 2 == 0) {
#pragma unroll
        for (int e = 0; e < N; e += 2) *reinterpret_cast<float2 *>(p + e) = make_float2(o[e] * w, o[e + 1] * w);
    } else {
#pragma unroll
        for (int e = 0; e < N; e++) p[e] = o[e] * w;
    }
}

// A warp's accumulators meet in shared memory, by row groups (lanes of one cache row) where there is room: adding the groups up with shuffles
// first is 64 instructions per round that every launch fetches and runs once.  (Many warps: they are added up first.)
__host__ __device__ constexpr uint32_t attn_row_groups(uint32_t hs, uint32_t regime) { return regime == ATTN_MIDDLE ? 1 : 256 / hs; }
// floats of dynamic shared memory: the warps' accumulators, and with clusters the slices' partials (in the first CTA)
__host__ __device__ constexpr uint32_t attn_smem_floats(uint32_t hs, uint32_t kvm, uint32_t regime) {
    return attn_warps(hs, regime) * attn_row_groups(hs, regime) * kvm * hs + (regime != ATTN_LONG ? ATTN_CLUSTER_MAX * kvm * (hs + 2) : 0);
}
// The caller's output: in pairs, or one by one where it is aligned to 4 bytes only
template <int N>
__device__ __forceinline__ void store_out(float *p, const float (&o)[N], float w, bool pairs) {
    if (pairs) store_scaled(p, o, w);
    else {
#pragma unroll
        for (int e = 0; e < N; e++) p[e] = o[e] * w;
    }
}

// A lane's 8 elements of a cache row: one 16-byte load of f16, two of f32 (each of them 16 bytes of every lane side by side).  FIRST * li: where its
// elements 0-3 are in the row; SECOND: how far behind them 4-7 are.  (load: from the lane's elements on)
template <typename T, int HS> struct LaneRow;
template <int HS> struct LaneRow<__half, HS> {
    static constexpr uint32_t FIRST = 8, SECOND = 4;
    uint4 r;
    __device__ __forceinline__ void load(const __half *p) { r = __ldcg(reinterpret_cast<const uint4 *>(p)); }
    __device__ __forceinline__ void get(float2 (&f)[4]) const {
        const __half2 *h = reinterpret_cast<const __half2 *>(&r);
#pragma unroll
        for (int j = 0; j < 4; j++) f[j] = __half22float2(h[j]);
    }
};
template <int HS> struct LaneRow<float, HS> {
    static constexpr uint32_t FIRST = 4, SECOND = HS / 2;
    float4 a, b;
    __device__ __forceinline__ void load(const float *p) {
        a = __ldcg(reinterpret_cast<const float4 *>(p));
        b = __ldcg(reinterpret_cast<const float4 *>(p + SECOND));
    }
    __device__ __forceinline__ void get(float2 (&f)[4]) const {
        f[0] = make_float2(a.x, a.y); f[1] = make_float2(a.z, a.w);
        f[2] = make_float2(b.x, b.y); f[3] = make_float2(b.z, b.w);
    }
};
constexpr int attn_log2(int n) { return n <= 1 ? 0 : 1 + attn_log2(n / 2); }

// ALIGNED: q and out are on 16-byte boundaries.  (A run-time choice made launches of 200 to 250 positions of 8 x 4 heads of 128 0.2 of 3.7 us slower: code.)
template <int HS, int KVM, typename T, uint32_t REGIME, bool ALIGNED>
__global__ void __launch_bounds__(attn_warps(HS, REGIME) * 32, REGIME == ATTN_MIDDLE ? 1 : 3) attn_group_kernel(const AttnArgs a) {
    constexpr int EPL = 8;
    constexpr bool CLUSTER = REGIME != ATTN_LONG;
    constexpr int W = attn_warps(HS, REGIME), THREADS = W * 32;
    constexpr int L = HS / EPL;          // lanes per cache row
    constexpr int RPW = 32 / L;          // rows per warp step
    constexpr int STEPS = attn_steps(HS, KVM, sizeof(T), REGIME);   // steps per warp iteration
    constexpr int ROWS = STEPS * RPW;
    constexpr int N = STEPS * KVM;       // partial scores per lane and iteration; L / N lanes end up with the same complete one
    static_assert(N <= L && (N & (N - 1)) == 0, "lane layout");
    constexpr int DUP = attn_log2(L / N), FROM_S = 1 << (DUP + attn_log2(KVM));   // the lane's bits: [row group][step][head][copy]
    constexpr int G = attn_row_groups(HS, REGIME);
    static_assert(G == 1 || G == RPW, "row groups of a warp");
    extern __shared__ __align__(16) float sm_acc[];   // [W][G][KVM][HS]
    float *sm_cl = sm_acc + W * G * KVM * HS;         // clusters: [slices][KVM][HS + 2]
    __shared__ float sm_m[W * KVM], sm_l[W * KVM];
    __shared__ __align__(16) float sm_p[W][32];
    __shared__ __align__(16) float sm_alpha[W][4];
    __shared__ uint32_t sm_last;

    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    // Another CTA's shared memory may be written only once that CTA has started: everyone arrives here, and waits ahead of the first
    // remote store (or of leaving), behind the rows.
    if constexpr (CLUSTER) cluster.barrier_arrive();
    // Behind any kernel (pdl 2), the long regime lets its successor start with the last of its own rows: an attention launch that
    // starts earlier takes the SMs' free slots unevenly and itself ends later (4 kv heads of 128, 4096 positions, back to back: 10.2 us
    // against 11.4).  In a token graph the successor fills a whole SM and cannot.
    const bool late = !CLUSTER && a.pdl == 2;
    if (a.pdl && !late) asm volatile("griddepcontrol.launch_dependents;");
    const bool early = a.pdl == 1;   // rows may be requested ahead of the wait
    if (a.pdl == 2) asm volatile("griddepcontrol.wait;" ::: "memory");
    // The position was written at the end of the previous token, not by the predecessor: it can be read before the wait.
    const uint32_t kvh = blockIdx.x, split = blockIdx.y;   // (kvh: the group's number)
    const uint32_t total = (a.pos_ptr ? *a.pos_ptr : a.p.pos) + 1;
    uint32_t nsplit, per;
    attn_plan(total, a.max_splits, CLUSTER ? a.cluster : 0u, W, KVM, nsplit, per);
    if (split >= nsplit) {
        if constexpr (CLUSTER) {
            cluster.barrier_wait();
            if (nsplit > 1) cluster.sync();   // the barrier of the working CTAs below
        }
        return;
    }
    const uint32_t t0 = split * per, t1 = min(total, t0 + per);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane / L, li = lane % L;
    const uint32_t kv_dim = a.p.kv_dim;
    const uint32_t cache_head = KVM == (int)ATTN_GROUP ? kvh >> (a.p.kv_mul > ATTN_GROUP ? 1 : 0) : kvh;   // (eight heads: two groups)
    const uint32_t at0 = LaneRow<T, HS>::FIRST * li, at1 = at0 + LaneRow<T, HS>::SECOND;
    // The lane's offset: part of the pointers that the loop starts from (f16, 19000 positions of 16 heads of 64: 27.3 us, 27.6 if added per load), but not in the
    // long regime of head size 128, which has no registers left (10000 positions of 8 heads: 13.87 us, 14.00 if it is).
    constexpr bool FOLDED = HS != 128 || REGIME != ATTN_LONG;
    const uint32_t in_base = FOLDED ? at0 : 0u, in_load = FOLDED ? 0u : at0;
    const T *kc = reinterpret_cast<const T *>(a.kc) + (size_t)cache_head * HS + in_base;
    const T *vc = reinterpret_cast<const T *>(a.vc) + (size_t)cache_head * HS + in_base;
    const float scale = 1.0f / sqrtf((float)HS);

    // First iteration: the predecessor (the q/k/v kernel) writes this token's q and the newest cache row (position
    // total - 1); every older row is from earlier tokens.  So the older rows are requested before the wait for the
    // predecessor, q and the newest row after it: the cache round trip overlaps the predecessor's tail.
    LaneRow<T, HS> kraw[STEPS], vraw[STEPS];
    const uint32_t base0 = t0 + warp * ROWS;
    if (base0 < t1) {
#pragma unroll
        for (int s = 0; s < STEPS; s++) {
            const uint32_t t = base0 + s * RPW + g, tc = t < t1 ? t : t1 - 1;
            if (tc + 1 != total || !early) {
                kraw[s].load(kc + (size_t)tc * kv_dim + in_load);
                vraw[s].load(vc + (size_t)tc * kv_dim + in_load);
            }
        }
    }
    if (early) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (base0 < t1) {
#pragma unroll
            for (int s = 0; s < STEPS; s++) {
                const uint32_t t = base0 + s * RPW + g, tc = t < t1 ? t : t1 - 1;
                if (tc + 1 == total) {
                    kraw[s].load(kc + (size_t)tc * kv_dim + in_load);
                    vraw[s].load(vc + (size_t)tc * kv_dim + in_load);
                }
            }
        }
    }
    float2 q2[KVM][EPL / 2];
#pragma unroll
    for (int m = 0; m < KVM; m++) {
        const float *qp = a.q + (size_t)(kvh * KVM + m) * HS;
        float4 x, y;
        if constexpr (ALIGNED) {
            x = __ldcg(reinterpret_cast<const float4 *>(qp + at0));
            y = __ldcg(reinterpret_cast<const float4 *>(qp + at1));
        } else {
            x = make_float4(__ldcg(qp + at0), __ldcg(qp + at0 + 1), __ldcg(qp + at0 + 2), __ldcg(qp + at0 + 3));
            y = make_float4(__ldcg(qp + at1), __ldcg(qp + at1 + 1), __ldcg(qp + at1 + 2), __ldcg(qp + at1 + 3));
        }
        q2[m][0] = make_float2(x.x, x.y); q2[m][1] = make_float2(x.z, x.w);
        q2[m][2] = make_float2(y.x, y.y); q2[m][3] = make_float2(y.z, y.w);
    }

    // running maximum and sum of the head this lane scores (m_own); accumulators of all four heads for the lane's 8 elements
    const int s_own = (li >> DUP) / KVM;   // (and head (li >> DUP) % KVM)
    const bool owner = (li & ((1 << DUP) - 1)) == 0;
    float M = -INFINITY, l = 0.f;
    float2 acc[KVM][EPL / 2];
#pragma unroll
    for (int m = 0; m < KVM; m++)
#pragma unroll
        for (int j = 0; j < EPL / 2; j++) acc[m][j] = make_float2(0.f, 0.f);

    // The rows of the next iteration are requested before the current ones are used: a slice is then one cache round
    // trip plus arithmetic, however many iterations it has, and twice the bytes are in flight per warp.
    LaneRow<T, HS> knext[STEPS], vnext[STEPS];
#pragma unroll 1
    for (uint32_t base = base0; base < t1; base += W * ROWS) {
        const uint32_t nbase = base + W * ROWS;
        if (late && nbase >= t1) asm volatile("griddepcontrol.launch_dependents;");
        if (nbase < t1) {
#pragma unroll
            for (int s = 0; s < STEPS; s++) {
                const uint32_t t = nbase + s * RPW + g, tc = t < t1 ? t : t1 - 1;
                knext[s].load(kc + (size_t)tc * kv_dim + in_load);
                vnext[s].load(vc + (size_t)tc * kv_dim + in_load);
            }
        }
        // partial scores of the lane's 8 elements: v[s * KVM + m]
        float v[N];
#pragma unroll
        for (int s = 0; s < STEPS; s++) {
            float2 k2[EPL / 2];
            kraw[s].get(k2);
#pragma unroll
            for (int m = 0; m < KVM; m++) {
                float2 d = make_float2(0.f, 0.f);
#pragma unroll
                for (int j = 0; j < EPL / 2; j++) d = ffma2(q2[m][j], k2[j], d);
                v[s * KVM + m] = d.x + d.y;
            }
        }
        // complete sums: lane li of the row ends up with score number li >> DUP = s_own * KVM + m_own
        constexpr int H = L / 2;   // the first round's distance
        if constexpr (N == 16) {
            halve_exchange<16>(v, lane, H);
            halve_exchange<8>(reinterpret_cast<float (&)[8]>(v), lane, H / 2);
            halve_exchange<4>(reinterpret_cast<float (&)[4]>(v), lane, H / 4);
            halve_exchange<2>(reinterpret_cast<float (&)[2]>(v), lane, H / 8);
        } else if constexpr (N == 8) {
            halve_exchange<8>(v, lane, H);
            halve_exchange<4>(reinterpret_cast<float (&)[4]>(v), lane, H / 2);
            halve_exchange<2>(reinterpret_cast<float (&)[2]>(v), lane, H / 4);
        } else if constexpr (N == 4) {
            halve_exchange<4>(v, lane, H);
            halve_exchange<2>(reinterpret_cast<float (&)[2]>(v), lane, H / 2);
        } else halve_exchange<2>(v, lane, H);
#pragma unroll
        for (int o = (1 << DUP) / 2; o; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
        const bool valid = (base + s_own * RPW + g) < t1;
        const float sc = valid ? v[0] * scale : -INFINITY;
        // block maximum of the head over the warp's rows
        float bm = sc;
#pragma unroll
        for (int o = FROM_S; o < 32; o <<= 1) bm = fmaxf(bm, __shfl_xor_sync(0xffffffffu, bm, o));
        const float Mn = fmaxf(M, bm);   // finite: row `base` (step 0, group 0) is valid
        const float alpha = expf(M - Mn), pe = expf(sc - Mn);
        M = Mn;
        l = l * alpha + pe;
        __syncwarp();   // the previous iteration's reads of sm_p are done
        if (owner) {
            sm_p[warp][g * N + (li >> DUP)] = pe;   // index g * N + s * KVM + m
            if (lane < FROM_S) sm_alpha[warp][lane >> DUP] = alpha;   // group 0, step 0: m_own
        }
        __syncwarp();
        float alv[KVM];
        load_few<KVM>(alv, sm_alpha[warp]);
#pragma unroll
        for (int m = 0; m < KVM; m++)
#pragma unroll
            for (int j = 0; j < EPL / 2; j++) { acc[m][j].x *= alv[m]; acc[m][j].y *= alv[m]; }
#pragma unroll
        for (int s = 0; s < STEPS; s++) {
            float pv[KVM];
            load_few<KVM>(pv, &sm_p[warp][g * N + s * KVM]);
            float2 v2[EPL / 2];
            vraw[s].get(v2);
#pragma unroll
            for (int m = 0; m < KVM; m++)
#pragma unroll
                for (int j = 0; j < EPL / 2; j++) acc[m][j] = ffma2(make_float2(pv[m], pv[m]), v2[j], acc[m][j]);
        }
        if (nbase < t1) {
#pragma unroll
            for (int s = 0; s < STEPS; s++) { kraw[s] = knext[s]; vraw[s] = vnext[s]; }
        }
    }

    // the row groups of the warp (lanes with the same li) and the warps of the block
    if constexpr (G == 1) {
#pragma unroll
        for (int o = L; o < 32; o <<= 1) {
#pragma unroll
            for (int m = 0; m < KVM; m++)
#pragma unroll
                for (int j = 0; j < EPL / 2; j++) {
                    acc[m][j].x += __shfl_xor_sync(0xffffffffu, acc[m][j].x, o);
                    acc[m][j].y += __shfl_xor_sync(0xffffffffu, acc[m][j].y, o);
                }
        }
    }
#pragma unroll
    for (int o = FROM_S; o < 32; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);   // the lanes that score the same head
    if (G > 1 || g == 0) {
        float *dst = &sm_acc[(warp * G + (G > 1 ? g : 0)) * KVM * HS];
#pragma unroll
        for (int m = 0; m < KVM; m++) {
            *reinterpret_cast<float4 *>(dst + m * HS + at0) = make_float4(acc[m][0].x, acc[m][0].y, acc[m][1].x, acc[m][1].y);
            *reinterpret_cast<float4 *>(dst + m * HS + at1) = make_float4(acc[m][2].x, acc[m][2].y, acc[m][3].x, acc[m][3].y);
        }
    }
    if (owner && lane < FROM_S) { sm_m[warp * KVM + (lane >> DUP)] = M; sm_l[warp * KVM + (lane >> DUP)] = l; }
    __syncthreads();

    // every thread owns PER consecutive outputs of one head (16 warps at head size 64: half of the threads one each)
    constexpr uint32_t slot = HS + 2;
    constexpr int PER = KVM * HS >= THREADS ? KVM * HS / THREADS : 1;
    const bool has = KVM * HS >= THREADS || tid * PER < KVM * HS;
    const int at = has ? tid * PER : 0, m_out = at / HS, d_out = at % HS;
    // partials in global memory: the accumulators [kv head][slice][KVM][HS], behind them all (max, sum) pairs [kv head][slice][KVM]
    float *part = a.scratch + ((size_t)kvh * a.max_splits + split) * KVM * HS;
    float2 *part_ml = reinterpret_cast<float2 *>(a.scratch + (size_t)gridDim.x * a.max_splits * KVM * HS) + (size_t)kvh * a.max_splits * KVM;
    float *out = a.out + (size_t)(kvh * KVM + m_out) * HS + d_out;
    {
        // A warp's outputs are of one head, so its lanes share out the weights: lane w has that of warp w.  (Every thread evaluating every
        // warp's and every slice's weight: 7.9 us instead of 6.9 at 3000 positions of 8 heads of 64, 7.7 instead of 7.2 at 2000 of 128.)
        static_assert((W & (W - 1)) == 0 && W <= 32 && (32 * PER) <= HS && HS % (32 * PER) == 0, "outputs of a warp");
        const float mw = sm_m[(lane & (W - 1)) * KVM + m_out];
        float mx = mw;
#pragma unroll
        for (int x = 1; x < W; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
        const float wt = merge_weight(mw, mx);
        float ls = wt * sm_l[(lane & (W - 1)) * KVM + m_out];
#pragma unroll
        for (int x = 1; x < W; x <<= 1) ls += __shfl_xor_sync(0xffffffffu, ls, x);
        float o[PER];
#pragma unroll
        for (int e = 0; e < PER; e++) o[e] = 0.f;
#pragma unroll
        for (int w = 0; w < W; w++) {
            const float ww = __shfl_sync(0xffffffffu, wt, w);
            float a[PER];
#pragma unroll
            for (int e = 0; e < PER; e++) a[e] = 0.f;
#pragma unroll
            for (int k = 0; k < G; k++) add_scaled(a, 1.0f, &sm_acc[((w * G + k) * KVM + m_out) * HS + d_out]);
#pragma unroll
            for (int e = 0; e < PER; e++) o[e] += ww * a[e];
        }
        if (nsplit == 1) {
            if (has) store_out(out, o, 1.0f / ls, ALIGNED);
            if constexpr (CLUSTER) cluster.barrier_wait();
            return;
        }
        if constexpr (CLUSTER) {
            // the partial goes into the first CTA's shared memory; after the cluster barrier that CTA merges the slices
            cluster.barrier_wait();
            if (has) {
                float *dst = cluster.map_shared_rank(sm_cl, 0) + ((size_t)split * KVM + m_out) * slot;
                store_scaled(dst + d_out, o, 1.0f);
                if (d_out == 0) *reinterpret_cast<float2 *>(dst + HS) = make_float2(mx, ls);
            }
            cluster.sync();
            if (split != 0 || !has) return;   // (whole warps: a warp has outputs or none)
            // (the lanes share out the slices' weights like the warps' above)
            const uint32_t sl = lane & (ATTN_CLUSTER_MAX - 1);
            const float2 ml = sl < nsplit ? *reinterpret_cast<const float2 *>(&sm_cl[(sl * KVM + m_out) * slot + HS]) : make_float2(-INFINITY, 0.f);
            float cm = ml.x;
#pragma unroll
            for (int x = 1; x < (int)ATTN_CLUSTER_MAX; x <<= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, x));
            const float ws = merge_weight(ml.x, cm);
            float lsum = ws * ml.y, acc[PER];
#pragma unroll
            for (int x = 1; x < (int)ATTN_CLUSTER_MAX; x <<= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, x);
#pragma unroll
            for (int e = 0; e < PER; e++) acc[e] = 0.f;
            for (uint32_t s = 0; s < nsplit; s++) add_scaled(acc, __shfl_sync(0xffffffffu, ws, s), sm_cl + (s * KVM + m_out) * slot + d_out);
            store_out(out, acc, 1.0f / lsum, ALIGNED);
            return;
        } else {
            if (has) store_scaled(part + m_out * HS + d_out, o, 1.0f);
            if (has && d_out == 0) part_ml[split * KVM + m_out] = make_float2(mx, ls);
        }
    }
    if constexpr (!CLUSTER) {

    // The block's partial is published by one release/acquire arrival of thread 0: the barrier before it orders the other
    // threads' stores ahead of the release, the barrier after it orders their reads of the other blocks' partials (from
    // L2) behind the acquire.
    __syncthreads();
    if (tid == 0) {
        uint32_t old;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(a.counters + kvh) : "memory");
        sm_last = (old == nsplit - 1) ? 1u : 0u;
    }
    __syncthreads();
    if (sm_last == 0u) return;
    // Merge of the kv head's partials.  A warp's outputs are of one head: its lanes fetch the slices' (max, sum) pairs together and share out
    // the weights, which then lie in shared memory (the accumulators there have been used); the accumulators come sixteen slices per
    // L2 round trip, the first of them requested ahead of the weights.  Eight slices at a time with their pairs and a running maximum:
    // 21.4 us instead of 17.9 at 16384 positions of 8 heads of 128, 18.9 instead of 13.9 at 20000 of 64.
    constexpr uint32_t AT_ONCE = 16;
    static_assert(W * ATTN_MAX_SLICES <= attn_smem_floats(HS, KVM, REGIME), "the weights fit the accumulators' place");
    float *sm_w = sm_acc + warp * ATTN_MAX_SLICES;
    const float *mine = a.scratch + (size_t)kvh * a.max_splits * KVM * HS + m_out * HS + d_out;
    float dat[AT_ONCE][PER];
    auto fetch = [&](uint32_t s0) {
#pragma unroll
        for (uint32_t j = 0; j < AT_ONCE; j++) {
            const float *ps = mine + (size_t)min(s0 + j, nsplit - 1) * (KVM * HS);   // (slices past the last one have weight 0)
            if constexpr (PER == 4) {
                const float4 v = __ldcg(reinterpret_cast<const float4 *>(ps));
                dat[j][0] = v.x; dat[j][1] = v.y; dat[j][2] = v.z; dat[j][3] = v.w;
            } else if constexpr (PER == 2) {
                const float2 v = __ldcg(reinterpret_cast<const float2 *>(ps));
                dat[j][0] = v.x; dat[j][1] = v.y;
            } else dat[j][0] = __ldcg(ps);
        }
    };
    fetch(0);
    constexpr uint32_t PAIRS = ATTN_MAX_SLICES / 32;
    float2 ml[PAIRS];
    float cm = -INFINITY;
#pragma unroll
    for (uint32_t i = 0; i < PAIRS; i++) {
        const uint32_t s = 32 * i + lane;
        ml[i] = s < nsplit ? __ldcg(part_ml + s * KVM + m_out) : make_float2(-INFINITY, 0.f);
        cm = fmaxf(cm, ml[i].x);
    }
#pragma unroll
    for (int x = 16; x; x >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, x));
    float ls = 0.f;
#pragma unroll
    for (uint32_t i = 0; i < PAIRS; i++) {
        if (32 * i >= nsplit) break;
        const float wt = merge_weight(ml[i].x, cm);
        ls += wt * ml[i].y;
        sm_w[32 * i + lane] = wt;
    }
#pragma unroll
    for (int x = 16; x; x >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, x);
    __syncwarp();
    float o[PER];
#pragma unroll
    for (int e = 0; e < PER; e++) o[e] = 0.f;
#pragma unroll 1
    for (uint32_t s0 = 0;;) {
#pragma unroll
        for (uint32_t j = 0; j < AT_ONCE; j++) {
            const float wt = sm_w[s0 + j];
#pragma unroll
            for (int e = 0; e < PER; e++) o[e] += wt * dat[j][e];
        }
        s0 += AT_ONCE;
        if (s0 >= nsplit) break;
        fetch(s0);
    }
    if (has) store_out(out, o, 1.0f / ls, ALIGNED);
    if (tid == 0) a.counters[kvh] = 0u;
    }
}

}  // namespace ib
