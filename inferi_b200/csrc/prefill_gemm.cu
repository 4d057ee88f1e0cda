// The GEMM of the prompt prefill: out^T tile = W tile (256 rows of a quantized matrix) x X^T (up to 128 tokens), on the
// 5th-generation tensor cores (tcgen05.mma, f32 accumulators in tensor memory) of a pair of SMs; few tokens: 128 rows on one SM.
//
// Exact integer weights.  A k-quant weight is w = d * (sc * q) - dmin * m with d, dmin one f16 (pair) per 256 columns and
// row, sc a 6- or 8-bit integer, q a small integer (crates/inferi/src/quantization.rs:227-402).  sc * q is an integer; per
// 256-column block
//     sum_k w_k x_k = d * P - Z,   P = sum_k (sc * q)_k x_k,   Z = sum_sb (dmin * m_sb) * S_sb,   S_sb = sum_{k in sb} x_k
//   Q4_K, Q5_K: sc * q <= 63 * 31 < 2048 is exact in one f16: 2 MMAs per 16 columns (the inputs are split into two f16, hi
//     and lo); Z is a small MMA of the sub-blocks' minimums with the inputs' sub-block sums (both split, 3 MMAs per block).
//   Q6_K: |sc * (q - 32)| <= 4096 is the sum of its f16 rounding and a remainder of at most 1, both exact: 3 MMAs per 16
//     columns (remainder x lo is below f32 resolution).  No minimums.
//   Q8_0: w = d * q with d per 32 columns; d * q (19 bits) is the sum of its f16 rounding and an f16 remainder: 3 MMAs.
// The weights' operand lives in TENSOR MEMORY: a producer thread owns one row (a tensor-memory lane), turns the row's 64
// columns into 32 packed f16 pairs in registers and stores them with one tcgen05.st; nothing of the weights goes back to shared
// memory (through shared memory the tile cost a write, a proxy fence that every warp waited for, and 64 bytes a clock of
// operand reads next to the inputs' 64).
//
// Two SMs per tile (cta_group::2).  Each makes the operand of its 128 rows and keeps their sums; the inputs of the 128 tokens are
// shared, half of them in either's shared memory.  On one SM a 256-column block of 128 rows took 131 KB of inputs from L2 for 2240
// clocks of MMAs, and L2 delivers 72 bytes a nanosecond to an SM: 9.5 of at most 10.7 TB/s, 4000 clocks a block.  Now 2490 (Q4_K).
// Measured, one SM / two: Q4_K 14336 x 4096, 900 tokens 218 / 185 us; with Q6_K's conversions (below) 4096 x 14336, 1000 tokens 383 /
// 288; a prompt of 1021 tokens of the 8B architecture 39.8 / 33.1 ms, of 128 tokens 6.24 / 5.36.  With few tokens L2 has little to deliver, and one
// SM per tile (PAIR = false, cta_group::1) is the faster way: prefill_streamk.
//
// Who does what (19 warps, one CTA per SM; the MMAs of both are issued by the first):
//   warps 0-7    producers: two warpgroups, each two of the block's four 64-column chunks
//   warps 8-15   fold: when a block's P is complete, Y += d * P into registers (64 accumulators a thread); at the end of the
//                tile's K range Y -= Z and the store, [token][row]
//   warp 16      MMA issue (one thread); warp 17 requests the inputs' tiles, warp 18 the raw blocks (tiled TMA copies)
// They hand over through mbarriers only.  P is double-buffered, so a block's MMAs run while the previous block is folded.
// Tensor memory (512 columns): P0, P1, Z of 128 columns each and 128 columns of operand slots (Q4_K / Q5_K: three stages of
// 32 columns and two slots of minimums), or, without Z, 256 columns of operand slots (four stages of 64).
//
// The (tile, 256-column block) units of the launch are dealt out as equal contiguous ranges over one wave of CTAs (StreamK
// in prefill.cuh); a tile whose K range falls to several CTAs gets one partial plane per CTA, added in CTA order by the
// element-wise kernel behind the GEMM.
//
// Every wait is bounded; a wait that gives up raises the context's error word and the kernel returns after freeing its tensor memory.
#include "prefill.cuh"

#include <cuda.h>   // CUtensorMap and the enumerations of cuTensorMapEncodeTiled (the entry point is looked up at run time)

namespace ib {

constexpr int PG_PRODUCERS = 8, PG_FOLD = 8, PG_W_MMA = 16, PG_W_X = 17, PG_W_RAW = 18;
constexpr int PG_THREADS = 19 * 32;
constexpr uint32_t PG_DSLOTS = 8;   // slots of the blocks' scales, each taken from the request of the raw block to the fold (more than the raw stages and the fold's delay)
constexpr uint32_t PG_XSTAGES_MAX = 16;   // a stage holds the tokens' 64 columns, hi and lo: few tokens, small stages, more of them (launch)
constexpr uint32_t PG_STILE = PF_CHUNK * 16 * 2;        // ... of 128 tokens x 16 sub-block sums
constexpr uint32_t PG_SMEM_LIMIT = 227 * 1024;
constexpr uint32_t PG_LBO = 128, PG_SBO = 2048, PG_SSBO = 512;   // core matrices of the inputs' tiles and of the sums' tiles
// tensor memory columns
constexpr uint32_t PG_P = 0, PG_Z = 256, PG_A4 = 384, PG_M4 = 480, PG_A6 = 256;

enum PgFormat : int { PG_Q4K = 0, PG_Q5K = 1, PG_Q6K = 2, PG_Q80 = 3 };
constexpr bool pg_has_min(int f) { return f == PG_Q4K || f == PG_Q5K; }
constexpr uint32_t pg_slots(int f) { return pg_has_min(f) ? 3u : 4u; }
// A raw stage holds one 256-column block of each of the tile's 128 rows.  The row strides are odd multiples of 16 bytes: the
// 16-byte reads of 8 consecutive rows fall into different bank groups.  Q6_K: four arrays (low bits, high bits, scales, d).
constexpr uint32_t PG_Q6_QL = 0, PG_Q6_QH = 128 * 144, PG_Q6_SC = PG_Q6_QH + 128 * 80, PG_Q6_D = PG_Q6_SC + 128 * 16;
constexpr uint32_t pg_raw_bytes(int f) { return f == PG_Q4K ? 128 * 144u : f == PG_Q5K ? 128 * 176u : f == PG_Q6K ? PG_Q6_D + 128 * 16u : 128 * 272u; }
// Shared memory: raw blocks (PG_RAW stages), sums, scales, barriers; the rest is the inputs' ring.  Four raw blocks are 74 KB in
// flight per SM for Q4_K, enough to stream at the HBM's rate; the inputs come from L2 with ~1.5 us between request and
// arrival, so what bounds a small ring is its depth.
constexpr uint32_t pg_raw_stages(int f) { return f == PG_Q4K ? 4u : (f == PG_Q5K ? 3u : 2u); }
constexpr uint32_t pg_fixed_smem(int f) {
    return pg_raw_stages(f) * pg_raw_bytes(f) + (pg_has_min(f) ? 2 * 2 * PG_STILE : 0u) + PG_DSLOTS * 512 + 640 + 1024;
}

struct PgMaps { CUtensorMap m[PF_MAX_SEGS][3]; };

// ---- small wrappers ----
__device__ __forceinline__ uint32_t pg_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long pg_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void pg_bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void pg_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void pg_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool pg_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool pg_test(uint32_t bar, uint32_t parity) {   // does not suspend the thread
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait.  The clock is only looked at after many tries: reading %globaltimer stalls the thread for about a microsecond,
// longer than most waits here.
__device__ __noinline__ bool pg_wait_long(uint32_t bar, uint32_t parity, unsigned long long limit, uint32_t *err, uint32_t code) {
    unsigned long long t0 = 0;
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 1024; i++)
            if (pg_try(bar, parity)) return true;
        const unsigned long long t = pg_ns();
        if (t0 == 0) t0 = t;
        else if (t - t0 > limit) break;
    }
    if (err) {
        *(volatile uint32_t *)err = code;
        __threadfence_system();
    }
    return false;
}
__device__ __forceinline__ bool pg_wait(uint32_t bar, uint32_t parity, const PgParams &p, uint32_t code) {
    return pg_try(bar, parity) || pg_wait_long(bar, parity, p.wait_ns, p.err, code);
}
// the same for a whole warp: the result is warp-uniform
__device__ __forceinline__ bool pg_wait_warp(uint32_t bar, uint32_t parity, const PgParams &p, uint32_t code) { return __all_sync(0xffffffffu, pg_wait(bar, parity, p, code)); }
// One lane of a converged warp.  The single-thread roles run as whole warps and elect a lane only around the instruction itself: with
// the loop inside a `lane == 0` branch the compiler cannot keep descriptors and addresses in uniform registers, and an MMA
// cost 60 clocks of issue, a commit 190.
__device__ __forceinline__ bool pg_elect() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ uint4 pg_lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 pg_lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t pg_lds16(uint32_t a) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ float pg_h2f(uint32_t bits16) { return __half2float(__ushort_as_half((unsigned short)bits16)); }
__device__ __forceinline__ __half2 pg_h2(uint32_t bits) { return *reinterpret_cast<const __half2 *>(&bits); }
__device__ __forceinline__ uint32_t pg_bits(__half2 h) { return *reinterpret_cast<const uint32_t *>(&h); }

__device__ __forceinline__ void pg_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void pg_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 16 consecutive tensor-memory columns of the warp's 32 lanes
__device__ __forceinline__ void pg_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
                   "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void pg_st16(uint32_t taddr, const uint32_t *r) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
                 "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void pg_st1(uint32_t taddr, uint32_t v) { asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%1], {%0};" ::"r"(v), "r"(taddr) : "memory"); }
__device__ __forceinline__ void pg_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void pg_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory descriptor of a K-major tile without swizzle: core matrices of 8 rows x 16 bytes, `lbo` bytes between core
// matrices that are neighbours along K, `sbo` bytes between 8-row groups; bits 46-47: the descriptor version of this architecture.
__device__ __forceinline__ uint64_t pg_desc(uint32_t smem_addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((smem_addr & 0x3FFFFu) >> 4) | (uint64_t)((lbo >> 4) & 0x3FFFu) << 16 | (uint64_t)((sbo >> 4) & 0x3FFFu) << 32 | (uint64_t)1 << 46;
}
// Instruction descriptor of kind::f16: f16 A and B (both K-major), f32 accumulator, M x N.
__device__ __forceinline__ uint32_t pg_idesc(uint32_t M, uint32_t N) { return (1u << 4) | ((N >> 3) << 17) | ((M >> 4) << 24); }
// D[128 x N] (+)= A (tensor memory, 16 columns of f16 = 8 columns of 32 bits) x B (shared memory).  PAIR: D[256 x N] on both SMs of the
// pair: each has its 128 rows of A and D in its own tensor memory and half of B's N rows in its own shared memory, at the same places.
template <bool PAIR>
__device__ __forceinline__ void pg_mma(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    if constexpr (PAIR)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem),
                     "l"(b_desc), "r"(idesc), "r"(accumulate)
                     : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem),
                     "l"(b_desc), "r"(idesc), "r"(accumulate)
                     : "memory");
}
// arrives, when the MMAs issued so far are done, on the barrier (PAIR: on the barrier at this place in both CTAs)
template <bool PAIR>
__device__ __forceinline__ void pg_commit(uint32_t bar) {
    if constexpr (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"((uint16_t)3) : "memory");
    else asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// the whole tensor memory; its address is left at shared address `at`
template <bool PAIR>
__device__ __forceinline__ void pg_alloc(uint32_t at) {
    if constexpr (PAIR) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(at), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
}
template <bool PAIR>
__device__ __forceinline__ void pg_dealloc(uint32_t tmem) {
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}
// ---- between the two CTAs ----
// (Arrivals and waits keep the default scope also across the pair: what those barriers order is tensor memory and bulk copies.  Waits that
// acquire, or arrivals that release, at cluster scope make every launch 1.1 to 1.5 times as long.  Plain shared memory - the blocks' scales - is
// ordered inside the CTA that it lies in, by rawempty, pdone and dempty.)
template <bool PAIR>
__device__ __forceinline__ uint32_t pg_leader(uint32_t addr) {   // the same place in the pair's first CTA
    uint32_t a = addr;
    if constexpr (PAIR) asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(addr));
    return a;
}
template <bool PAIR>
__device__ __forceinline__ void pg_arrive_leader(uint32_t addr) {   // addr: from pg_leader
    if constexpr (PAIR) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
    else pg_arrive(addr);
}
template <bool PAIR>
__device__ __forceinline__ void pg_sync() {
    if constexpr (PAIR) {
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    } else __syncthreads();
}
__device__ __forceinline__ void pg_tma2d(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t bar, uint64_t policy) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar), "l"(policy)
                 : "memory");
}
__device__ __forceinline__ void pg_bulk(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// ---- the producers' conversions: a row's raw bytes -> packed f16 pairs of exact integers ----
// Four consecutive weights are stored in the order 0, 2, 1, 3 (the two even bytes of a word first): masking a word leaves
// bytes 0 and 2 in the low halves of an f16 pair, so a pair costs one logic operation (or two with more bits) and one packed f16
// operation, no byte permute.  The inputs' tiles are written in the same order (pf_x_index).
constexpr uint32_t PG_MAGIC = 0x64006400u;   // f16 pair (1024, 1024): OR-ing an integer below 1024 into the mantissa adds it

// 64 columns (sub-blocks 2c and 2c + 1) of a Q4_K / Q5_K block: (1024 + q) * sc - 1024 * sc = q * sc; the high nibbles stay in
// place: (1024 + 16 q) * (sc / 16) - 64 * sc.  One rounding of an exact result: exact.
template <bool Q5>
__device__ __forceinline__ void pg_convert_k(const uint4 &q0, const uint4 &q1, const uint4 &h0, const uint4 &h1, uint32_t c, float sc_lo, float sc_hi, uint32_t (&r)[32]) {
    const uint32_t qw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w}, hw[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    const __half2 s0 = __float2half2_rn(sc_lo), o0 = __float2half2_rn(-1024.0f * sc_lo), s1 = __float2half2_rn(sc_hi * 0.0625f), o1 = __float2half2_rn(-64.0f * sc_hi);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t w = qw[i], w8 = w >> 8;
        uint32_t le = (w & 0x000F000Fu) | PG_MAGIC, lo = (w8 & 0x000F000Fu) | PG_MAGIC, he = (w & 0x00F000F0u) | PG_MAGIC, ho = (w8 & 0x00F000F0u) | PG_MAGIC;
        if (Q5) {
            const uint32_t t = hw[i] >> (2 * c);   // bit 0 of a byte: fifth bit of the low-nibble weight, bit 1: of the high-nibble weight
            le |= (t << 4) & 0x00100010u;
            lo |= (t >> 4) & 0x00100010u;
            he |= (t << 7) & 0x01000100u;
            ho |= (t >> 1) & 0x01000100u;
        }
        r[2 * i] = pg_bits(__hfma2(pg_h2(le), s0, o0));
        r[2 * i + 1] = pg_bits(__hfma2(pg_h2(lo), s0, o0));
        r[16 + 2 * i] = pg_bits(__hfma2(pg_h2(he), s1, o1));
        r[16 + 2 * i + 1] = pg_bits(__hfma2(pg_h2(ho), s1, o1));
    }
}

// 32 columns (group g of a half block) of Q6_K: a = f16(sc * (q - 32)), b = the remainder.  Groups 2 and 3 use the high
// nibbles in place: 16 * (q - 32) times sc / 16.
template <int G>
__device__ __forceinline__ void pg_convert_q6(const uint4 &l0, const uint4 &l1, const uint4 &h0, const uint4 &h1, float sc0, float sc1, uint32_t (&a)[16], uint32_t (&b)[16]) {
    constexpr bool HI = G >= 2;
    constexpr int SH = (G & 1) ? 2 : 4;
    constexpr uint32_t LM = HI ? 0x00F000F0u : 0x000F000Fu, HM = HI ? 0x03000300u : 0x00300030u;
    const uint32_t lw[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w}, hw[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
    const __half2 off = __float2half2_rn(HI ? -1536.0f : -1056.0f);
    const __half2 s[2] = {__float2half2_rn(HI ? sc0 * 0.0625f : sc0), __float2half2_rn(HI ? sc1 * 0.0625f : sc1)};
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t w = lw[i], w8 = w >> 8, h = hw[i] << SH, h8 = SH == 4 ? hw[i] >> 4 : hw[i] >> 6;
        const __half2 e = __hadd2(pg_h2((w & LM) | (h & HM) | PG_MAGIC), off), o = __hadd2(pg_h2((w8 & LM) | (h8 & HM) | PG_MAGIC), off);
        const __half2 sc = s[i >> 2];
        const __half2 pe = __hmul2(e, sc), po = __hmul2(o, sc);
        a[2 * i] = pg_bits(pe);
        a[2 * i + 1] = pg_bits(po);
        b[2 * i] = pg_bits(__hfma2(e, sc, __hneg2(pe)));
        b[2 * i + 1] = pg_bits(__hfma2(o, sc, __hneg2(po)));
    }
}

// 32 columns (one block) of Q8_0: a = f16(d * q), b = the remainder
__device__ __forceinline__ void pg_convert_q8(const uint4 &q0, const uint4 &q1, __half2 d, uint32_t (&a)[16], uint32_t (&b)[16]) {
    const uint32_t qw[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
    const __half2 off = __float2half2_rn(-1152.0f);
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const uint32_t u = qw[i] ^ 0x80808080u;
        const __half2 e = __hadd2(pg_h2((u & 0x00FF00FFu) | PG_MAGIC), off), o = __hadd2(pg_h2(((u >> 8) & 0x00FF00FFu) | PG_MAGIC), off);
        const __half2 pe = __hmul2(e, d), po = __hmul2(o, d);
        a[2 * i] = pg_bits(pe);
        a[2 * i + 1] = pg_bits(po);
        b[2 * i] = pg_bits(__hfma2(e, d, __hneg2(pe)));
        b[2 * i + 1] = pg_bits(__hfma2(o, d, __hneg2(po)));
    }
}

// Scales and minimums of sub-blocks 2c and 2c + 1 of a Q4_K / Q5_K header (get_scale_min_k4, quantization.rs:394-402), one byte each
__device__ __forceinline__ void pg_scales(const uint4 &hdr, uint32_t c, uint32_t &sc2, uint32_t &m2) {
    const uint32_t sh = 16 * (c & 1), y = hdr.y >> sh, z = hdr.z >> sh, w = hdr.w >> sh;
    if (c < 2) {
        sc2 = y & 0x3F3Fu;
        m2 = z & 0x3F3Fu;
    } else {
        sc2 = (w & 0x0F0Fu) | ((y >> 2) & 0x3030u);
        m2 = ((w >> 4) & 0x0F0Fu) | ((z >> 2) & 0x3030u);
    }
}

// The current unit of a role's walk over its CTA's range, carried forward by additions
struct PgCursor {
    uint32_t rt, chunk, kb;   // row tile (128 rows, of a pair 256), chunk of 128 tokens, 256-column block
    __device__ __forceinline__ void init(const PgParams &p, uint32_t u) {
        const uint32_t tile = u / p.sk.nb;
        kb = u - tile * p.sk.nb;
        rt = tile / p.chunks;
        chunk = tile - rt * p.chunks;
    }
    __device__ __forceinline__ void next(const PgParams &p) {
        if (++kb == p.sk.nb) {
            kb = 0;
            if (++chunk == p.chunks) { chunk = 0; rt++; }
        }
    }
    __device__ __forceinline__ uint32_t tile(const PgParams &p) const { return rt * p.chunks + chunk; }
    __device__ __forceinline__ uint32_t tokens(const PgParams &p) const { return chunk + 1 == p.chunks ? p.n - chunk * PF_CHUNK : (uint32_t)PF_CHUNK; }
};
__device__ __forceinline__ uint32_t pg_pad(uint32_t n) { return (n + 15) & ~15u; }

// One CTA's work, number `cta` of the launch's CTAs of this format
template <int FMT, bool PAIR>
__device__ __forceinline__ void pg_gemm(const PgParams &p, const PgMaps &maps, const uint32_t cta) {
    constexpr bool MIN = pg_has_min(FMT), SCALED = FMT != PG_Q80;   // (Q8_0's operands carry their scales)
    constexpr uint32_t CTAS = PAIR ? 2 : 1;
    constexpr uint32_t NS = pg_slots(FMT), R = pg_raw_stages(FMT), RAW = pg_raw_bytes(FMT), A0 = MIN ? PG_A4 : PG_A6, ACOLS = MIN ? 32 : 64;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const uint32_t xst = pg_smem(smem);                                            // inputs' stages (hi, lo)
    const uint32_t XS = p.x_stages, XTILE = p.x_tile, sst = xst + XS * 2 * XTILE;   // sub-block sums (hi, lo): a slot per block
    const uint32_t SS = (XS + 6) / 4, STILE = XTILE / 4;                            // ... that the ring's XS stages can touch (4 SS >= XS + 3)
    const uint32_t raw0 = (sst + (MIN ? SS * 2 * STILE : 0) + 127) & ~127u;          // raw blocks
    uint8_t *tail = smem + (raw0 - xst) + R * RAW;
    float *dsm = reinterpret_cast<float *>(tail);                                   // [PG_DSLOTS][128] a block's scale of every row
    uint64_t *bars = reinterpret_cast<uint64_t *>(tail + PG_DSLOTS * 512);
    uint32_t nb = pg_smem(bars);
    auto take = [&](uint32_t n) { const uint32_t b = nb; nb += 8 * n; return b; };
    const uint32_t b_rawfull = take(R), b_rawempty = take(R), b_afull = take(NS), b_aempty = take(NS), b_xfull = take(PG_XSTAGES_MAX), b_xempty = take(PG_XSTAGES_MAX);
    const uint32_t b_pdone = take(PG_DSLOTS), b_dempty = take(PG_DSLOTS), b_pfree = take(2);
    const uint32_t b_zdone = take(1), b_zfree = take(1), s_tmem = nb;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const StreamK sk = p.sk;
    const uint32_t range = PAIR ? cta >> 1 : cta, rank = PAIR ? cta & 1 : 0;   // pairs: clusters of two CTAs along x
    const uint32_t u0 = sk.first_unit(range), nunits = sk.first_unit(range + 1) - u0;

    asm volatile("griddepcontrol.launch_dependents;");
    if (warp == 0) {
        // A lane per barrier.  What the MMA warp waits for counts both CTAs and lives in the first one; the MMAs' completion arrives in both.
        constexpr uint32_t X0 = 2 * R + 2 * NS, P0 = X0 + 2 * PG_XSTAGES_MAX;
        for (uint32_t i = lane; i < P0 + 2 * PG_DSLOTS + 4; i += 32) {
            uint32_t count = 1;
            if (i >= R && i < 2 * R) count = PG_PRODUCERS;                                                // rawempty
            else if (i >= 2 * R && i < 2 * R + NS) count = CTAS * PG_PRODUCERS / 2;                       // afull
            else if (i >= X0 && i < X0 + PG_XSTAGES_MAX) count = rank == 0 ? CTAS : 1;                    // xfull: the bytes, and word of the other CTA's
            else if (i >= P0 && i < P0 + PG_DSLOTS) count = SCALED ? 2 : 1;                               // pdone: the MMAs, and the scales
            else if (i >= P0 + PG_DSLOTS && i < P0 + 2 * PG_DSLOTS) count = PG_FOLD;                      // dempty
            else if (i >= P0 + 2 * PG_DSLOTS && i != P0 + 2 * PG_DSLOTS + 2) count = CTAS * PG_FOLD;      // pfree, zfree
            pg_bar_init(b_rawfull + 8 * i, count);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == PG_W_MMA) pg_alloc<PAIR>(s_tmem);
    pg_fence_before();
    pg_sync<PAIR>();
    pg_fence_after();
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(s_tmem));
    bool ok = true;

    if (warp < PG_PRODUCERS) {
        // ===== producers: thread = row; warpgroup `wg` makes chunks 2 wg and 2 wg + 1 of every block =====
        const uint32_t row = tid & 127, wg = warp >> 2, tl = tmem + ((uint32_t)((warp & 3) * 32) << 16), lead_afull = pg_leader<PAIR>(b_afull);
        if (MIN && wg == 0) {   // columns 4..7 of the minimums' operands (sub-blocks 8..15 of a K = 16 MMA) stay zero
            for (uint32_t m = 0; m < 4; m++)
                for (uint32_t c = 4; c < 8; c++) pg_st1(tl + PG_M4 + 8 * m + c, 0u);
        }
        PgCursor cur;
        cur.init(p, u0);
        uint32_t slot = 0, rpar = 0;
        for (uint32_t j = 0; j < nunits && ok; j++) {
            if (!(ok = pg_wait_warp(b_rawfull + 8 * slot, rpar, p, 8))) break;
            const uint32_t raw = raw0 + slot * RAW;
            // The quants are read where they are converted, not all at the unit's start: registers that wait for their turn are
            // registers that the conversions of other words cannot overlap in (Q6_K 4096 x 14336, 1000 tokens: 291 us against 383).
            uint4 hdr = make_uint4(0, 0, 0, 0), f0, f1, g0 = hdr, g1 = hdr;
            uint2 sc8 = make_uint2(0, 0);
            float d = 1.0f;
            if constexpr (MIN) {
                const uint32_t blk = raw + row * (FMT == PG_Q4K ? 144 : 176);
                hdr = pg_lds128(blk);
                if (FMT == PG_Q5K) { g0 = pg_lds128(blk + 16); g1 = pg_lds128(blk + 32); }
                d = pg_h2f(hdr.x & 0xFFFFu);
            } else if constexpr (FMT == PG_Q6K) {
                const uint32_t qh = raw + PG_Q6_QH + row * 80 + 32 * wg;
                g0 = pg_lds128(qh); g1 = pg_lds128(qh + 16);
                sc8 = pg_lds64(raw + PG_Q6_SC + row * 16 + 8 * wg);
                d = pg_h2f(pg_lds16(raw + PG_Q6_D + row * 16 + 2 * (cur.kb & 7)));
            } else {
                sc8 = pg_lds64(raw + row * 272 + 256 + 8 * wg);   // f16 scales of the warpgroup's four blocks
            }
#pragma unroll
            for (uint32_t cc = 0; cc < 2; cc++) {
                const uint32_t c = 2 * wg + cc, st = 4 * j + c, as = st % NS, use = st / NS, ta = tl + A0 + as * ACOLS;
                if constexpr (MIN) {
                    uint32_t sc2, m2, r[32];
                    pg_scales(hdr, c, sc2, m2);
                    const uint32_t qs = raw + row * (FMT == PG_Q4K ? 144 : 176) + (FMT == PG_Q4K ? 16 : 48) + 32 * c;
                    f0 = pg_lds128(qs); f1 = pg_lds128(qs + 16);
                    pg_convert_k<FMT == PG_Q5K>(f0, f1, g0, g1, c, (float)(sc2 & 0xFFu), (float)(sc2 >> 8), r);
                    const float dmin = pg_h2f(hdr.x >> 16), m0 = dmin * (float)(m2 & 0xFFu), m1 = dmin * (float)(m2 >> 8);
                    const __half2 mh = __floats2half2_rn(m0, m1);
                    const float2 back = __half22float2(mh);
                    const __half2 ml = __floats2half2_rn(m0 - back.x, m1 - back.y);
                    if (cc == 1) {   // the thread's raw bytes are in registers
                        __syncwarp();
                        if (lane == 0) pg_arrive(b_rawempty + 8 * slot);
                    }
                    if (use && !(ok = pg_wait_warp(b_aempty + 8 * as, (use - 1) & 1, p, 8))) break;
                    pg_fence_after();
                    pg_st16(ta, r);
                    pg_st16(ta + 16, r + 16);
                    // the slot of the minimums is free: block j - 2's were read ahead of the stage (of block j - 1) just waited for
                    pg_st1(tl + PG_M4 + 16 * (j & 1) + c, pg_bits(mh));
                    pg_st1(tl + PG_M4 + 16 * (j & 1) + 8 + c, pg_bits(ml));
                } else {
                    uint32_t a[16], b[16];
                    if constexpr (FMT == PG_Q6K) {
                        const uint32_t sw = cc ? sc8.y : sc8.x;
                        auto sc = [&](uint32_t k) { return (float)(int)(int8_t)((sw >> (8 * k)) & 0xFFu); };
                        const uint32_t ql = raw + PG_Q6_QL + row * 144 + 64 * wg;
                        f0 = pg_lds128(ql); f1 = pg_lds128(ql + 16);
                        if (cc == 0) pg_convert_q6<0>(f0, f1, g0, g1, sc(0), sc(1), a, b);
                        else pg_convert_q6<2>(f0, f1, g0, g1, sc(0), sc(1), a, b);
                        if (use && !(ok = pg_wait_warp(b_aempty + 8 * as, (use - 1) & 1, p, 8))) break;
                        pg_fence_after();
                        pg_st16(ta, a);
                        pg_st16(ta + 32, b);
                        f0 = pg_lds128(ql + 32); f1 = pg_lds128(ql + 48);
                        if (cc == 0) pg_convert_q6<1>(f0, f1, g0, g1, sc(2), sc(3), a, b);
                        else pg_convert_q6<3>(f0, f1, g0, g1, sc(2), sc(3), a, b);
                    } else {
                        const __half2 dd = pg_h2(cc ? sc8.y : sc8.x);
                        const uint32_t qs = raw + row * 272 + 64 * c;
                        f0 = pg_lds128(qs); f1 = pg_lds128(qs + 16);
                        pg_convert_q8(f0, f1, __low2half2(dd), a, b);
                        if (use && !(ok = pg_wait_warp(b_aempty + 8 * as, (use - 1) & 1, p, 8))) break;
                        pg_fence_after();
                        pg_st16(ta, a);
                        pg_st16(ta + 32, b);
                        f0 = pg_lds128(qs + 32); f1 = pg_lds128(qs + 48);
                        pg_convert_q8(f0, f1, __high2half2(dd), a, b);
                    }
                    if (cc == 1) {
                        __syncwarp();
                        if (lane == 0) pg_arrive(b_rawempty + 8 * slot);
                    }
                    pg_st16(ta + 16, a);
                    pg_st16(ta + 48, b);
                }
                if (SCALED && cc == 0 && wg == 0) dsm[(j & (PG_DSLOTS - 1)) * 128 + row] = d;   // for the fold warps (the raw block was requested when the slot was free)
                pg_wait_st();
                pg_fence_before();
                __syncwarp();
                if (lane == 0) pg_arrive_leader<PAIR>(lead_afull + 8 * as);
            }
            if (++slot == R) { slot = 0; rpar ^= 1u; }
            cur.next(p);
        }
        pg_fence_before();
    } else if (warp < PG_PRODUCERS + PG_FOLD) {
        // ===== fold: thread = row (tensor-memory lane), 64 of the tokens =====
        const uint32_t row = (warp & 3) * 32 + lane, half = (warp - PG_PRODUCERS) >> 2, tl = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 64 * half;
        const uint32_t lead_pfree = pg_leader<PAIR>(b_pfree), lead_zfree = pg_leader<PAIR>(b_zfree);
        float Y[64];
#pragma unroll
        for (int i = 0; i < 64; i++) Y[i] = 0.f;
        PgCursor cur;
        cur.init(p, u0);
        uint32_t seg = 0;
        for (uint32_t j = 0; j < nunits; j++) {
            const uint32_t chunk = cur.chunk, nt = cur.tokens(p), groups = pg_pad(nt) / 16;
            auto fold = [&](uint32_t col, float f) {
#pragma unroll
                for (uint32_t g = 0; g < 4; g++)
                    if (4 * half + g < groups) {
                        uint32_t r[16];
                        pg_ld16(tl + col + 16 * g, r);
                        pg_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; i++) Y[16 * g + i] = fmaf(f, __uint_as_float(r[i]), Y[16 * g + i]);
                    }
            };
            const uint32_t pb = j & 1, ds = j & (PG_DSLOTS - 1);
            const bool end = cur.kb + 1 == sk.nb || j + 1 == nunits;
            if (!(ok = pg_wait_warp(b_pdone + 8 * ds, (j / PG_DSLOTS) & 1, p, 10))) break;
            pg_fence_after();
            float d = 1.0f;
            if constexpr (SCALED) {
                d = dsm[ds * 128 + row];
                __syncwarp();
                if (lane == 0) pg_arrive(b_dempty + 8 * ds);
            }
            fold(PG_P + 128 * pb, d);
            pg_fence_before();
            __syncwarp();
            if (lane == 0) pg_arrive_leader<PAIR>(lead_pfree + 8 * pb);
            if (end) {
                if (MIN) {
                    if (!(ok = pg_wait_warp(b_zdone, seg & 1, p, 10))) break;
                    pg_fence_after();
                    fold(PG_Z, -1.0f);
                    pg_fence_before();
                    __syncwarp();
                    if (lane == 0) pg_arrive_leader<PAIR>(lead_zfree);
                }
                seg++;
                const uint32_t piece = range - sk.range_of(cur.tile(p) * sk.nb), rt = CTAS * cur.rt + rank;   // (a pair's last tile may lack its second half)
                float *out = (piece == 0 ? p.plane0 : p.planes + (size_t)(piece - 1) * p.n * p.rows) + (size_t)(chunk * PF_CHUNK + 64 * half) * p.rows + rt * 128 + row;
                const uint32_t count = rt * 128 < p.rows && nt > 64 * half ? nt - 64 * half : 0;
                // (straight stores where 16 tokens are there: this code runs once or twice per launch, and its length is what it costs)
#pragma unroll
                for (uint32_t g = 0; g < 4; g++) {
                    if (count >= 16 * g + 16) {
#pragma unroll
                        for (uint32_t t = 0; t < 16; t++, out += p.rows) *out = Y[16 * g + t];
                    } else {
#pragma unroll
                        for (uint32_t t = 0; t < 16; t++, out += p.rows)
                            if (16 * g + t < count) *out = Y[16 * g + t];
                    }
                }
                if (j + 1 < nunits) {
#pragma unroll
                    for (uint32_t t = 0; t < 64; t++) Y[t] = 0.f;
                }
            }
            cur.next(p);
        }
    } else if (PAIR && warp == PG_W_MMA && rank != 0) {
        // ===== the second CTA issues no MMAs: it tells the first one when its half of a stage's inputs is there =====
        const uint32_t lead_xfull = pg_leader<PAIR>(b_xfull);
        uint32_t xs = 0, par = 0;
        for (uint32_t i = 0; i < 4 * nunits && ok; i++) {
            if (!(ok = pg_wait_warp(b_xfull + 8 * xs, par, p, 9))) break;
            if (pg_elect()) pg_arrive_leader<PAIR>(lead_xfull + 8 * xs);
            __syncwarp();
            if (++xs == XS) { xs = 0; par ^= 1u; }
        }
    } else if (warp == PG_W_MMA) {
        // ===== MMA issue: one elected lane; descriptors differ from the first stage's only in the start-address field =====
        const uint64_t xd0 = pg_desc(xst, PG_LBO, PG_SBO), sd0 = pg_desc(sst, PG_LBO, PG_SSBO);
        PgCursor cur;
        cur.init(p, u0);
        // The tensor pipe queues about six MMAs (400 clocks at 128 tokens), and this warp's instructions between two stages have to
        // fit in that.  So everything the next stage needs - whether its barriers are complete, the next block's descriptor -
        // is asked for ahead of the current stage's MMAs.  A block's sums arrive with its first inputs and its minimums with
        // its weights: the minimums' MMAs at the end of the block wait for nothing of their own.
        const uint32_t id_full = pg_idesc(128 * CTAS, PF_CHUNK), id_last = pg_idesc(128 * CTAS, pg_pad(p.n - (p.chunks - 1) * PF_CHUNK));
        const uint32_t xstep = 2 * XTILE >> 4, sstep = 2 * STILE >> 4, xlo = PF_X_LO * 2 >> 4, slo = PF_S_LO * 2 >> 4;
        const uint32_t bx_end = b_xfull + 8 * XS, sd_end = (uint32_t)sd0 + SS * sstep, x_empty = b_xempty - b_xfull, a_empty = b_aempty - b_afull;
        const uint32_t x_hi32 = (uint32_t)(xd0 >> 32), s_hi32 = (uint32_t)(sd0 >> 32);
        // carried by additions: full barrier, parity and low descriptor word (start address) of the inputs' stage; barrier, parity and column of the weights'
        uint32_t bx = b_xfull, xpar = 0, xd = (uint32_t)xd0, ba = b_afull, apar = 0, a = tmem + A0, sd = (uint32_t)sd0, seg = 0;
        uint32_t idesc = cur.chunk + 1 == p.chunks ? id_last : id_full, P = tmem + PG_P, bp = b_pfree, ppar = 1, bd = b_pdone;
        bool begin = true, end = cur.kb + 1 == sk.nb || nunits == 1, ready = false;
        auto desc = [](uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; };
        for (uint32_t j = 0; j < nunits; j++) {
            uint32_t idesc_next = idesc;
            bool begin_next = false, end_next = true;
#pragma unroll
            for (uint32_t c = 0; c < 4; c++) {
                if (!ready) {
                    // (the first two blocks find the P buffers free: waiting for the parity before the first phase succeeds)
                    if (c == 0 && !(ok = pg_wait_warp(bp, ppar, p, 9))) break;
                    if (!(ok = __all_sync(0xffffffffu, pg_wait(bx, xpar, p, 9) && pg_wait(ba, apar, p, 9)))) break;
                }
                if (MIN && c == 3 && begin && seg && !(ok = pg_wait_warp(b_zfree, (seg - 1) & 1, p, 9))) break;
                pg_fence_after();
                const uint32_t xh = xd, col = a, cx = bx + x_empty, ca = ba + a_empty;
                xd += xstep;
                bx += 8;
                if (bx == bx_end) { bx = b_xfull; xd = (uint32_t)xd0; xpar ^= 1u; }
                a += ACOLS;
                ba += 8;
                if (ba == b_afull + 8 * NS) { ba = b_afull; a = tmem + A0; apar ^= 1u; }
                bool next = pg_test(bx, xpar) & pg_test(ba, apar);
                if (c == 3) next &= pg_test(bp ^ (b_pfree ^ (b_pfree + 8)), bp == b_pfree ? ppar : ppar ^ 1u);
                if (c == 2) {
                    cur.next(p);
                    begin_next = cur.kb == 0;
                    end_next = cur.kb + 1 == sk.nb || j + 2 >= nunits;
                    idesc_next = cur.chunk + 1 == p.chunks ? id_last : id_full;
                }
                if (pg_elect()) {
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++) {
                        const uint32_t ko = kk * (2 * PG_LBO >> 4);
                        pg_mma<PAIR>(P, col + 8 * kk, desc(x_hi32, xh + ko), idesc, !(c == 0 && kk == 0));   // every block starts a new P
                        pg_mma<PAIR>(P, col + 8 * kk, desc(x_hi32, xh + xlo + ko), idesc, 1);
                        if (!MIN) pg_mma<PAIR>(P, col + 32 + 8 * kk, desc(x_hi32, xh + ko), idesc, 1);
                    }
                    if (c == 3) pg_commit<PAIR>(bd);
                    if (MIN && c == 3) {
                        // the block's minimums x sums: hi * hi, hi * lo, lo * hi
                        const uint32_t m = tmem + PG_M4 + 16 * (j & 1);
                        pg_mma<PAIR>(tmem + PG_Z, m, desc(s_hi32, sd), idesc, !begin);
                        pg_mma<PAIR>(tmem + PG_Z, m, desc(s_hi32, sd + slo), idesc, 1);
                        pg_mma<PAIR>(tmem + PG_Z, m + 8, desc(s_hi32, sd), idesc, 1);
                        if (end) pg_commit<PAIR>(b_zdone);
                    }
                    pg_commit<PAIR>(ca);
                    pg_commit<PAIR>(cx);
                }
                __syncwarp();
                ready = __all_sync(0xffffffffu, next);
            }
            if (!ok) break;
            sd += sstep;
            if (sd == sd_end) sd = (uint32_t)sd0;
            if (end) seg++;
            idesc = idesc_next;
            begin = begin_next;
            end = end_next;
            P ^= (PG_P ^ (PG_P + 128));
            if (bp == b_pfree) bp = b_pfree + 8;
            else { bp = b_pfree; ppar ^= 1u; }
            bd = bd + 8 == b_dempty ? b_pdone : bd + 8;
        }
    } else if (warp == PG_W_X) {
        // ===== the tokens' inputs, of a pair this CTA's half of them (a bulk copy per 64 columns) and, per block, of their sub-block sums =====
        asm volatile("griddepcontrol.wait;" ::: "memory");   // the previous kernel writes them
        PgCursor cur;
        cur.init(p, u0);
        uint32_t xs = 0, use = 0, ss = 0;
        for (uint32_t j = 0; j < nunits && ok; j++) {
            const uint32_t tokens = pg_pad(cur.tokens(p)) / CTAS;
            const __half *x = p.x + (size_t)cur.chunk * p.x_chunk;
            for (uint32_t c = 0; c < 4; c++) {
                if (use && !(ok = pg_wait_warp(b_xempty + 8 * xs, (use - 1) & 1, p, 8))) break;
                const uint32_t full = b_xfull + 8 * xs, dst = xst + xs * 2 * XTILE, bytes = tokens * 256;
                const size_t at = (size_t)(4 * cur.kb + c) * (PF_CHUNK * 128) + rank * tokens * 128;
                if (pg_elect()) {
                    const bool sums = MIN && c == 0;   // (their slot's last reader was issued ahead of the stage just waited for)
                    pg_expect(full, bytes + (sums ? bytes / 4 : 0));
                    pg_bulk(dst, x + at, bytes, full);
                    if (sums) pg_bulk(sst + ss * 2 * STILE, x + (size_t)2 * PF_CHUNK * sk.nb * 256 + (size_t)cur.kb * (PF_CHUNK * 32) + rank * tokens * 32, bytes / 4, full);
                }
                __syncwarp();
                if (++xs == XS) { xs = 0; use++; }
            }
            if (!ok) break;
            if (++ss == SS) ss = 0;
            cur.next(p);
        }
    } else if (warp == PG_W_RAW) {
        // ===== the raw blocks: one 256-column block of each of the tile's 128 rows per step.  They are weights: requested ahead
        // of the wait for the previous kernel.  Q6_K keeps a block's low bits, high bits, scales and d in four places of the row
        // group: four boxes, the first two 16 bytes wider than their field, which gives the rows their conflict-free strides of
        // 144 and 80 bytes (the extra bytes are the row's own next bytes and are never read). =====
        PgCursor cur;
        cur.init(p, u0);
        // One chunk of tokens reads every weight once, a second comes back to it soon: as the first to be evicted from L2 the weights leave the planes and
        // the inputs there for the kernels that follow (a prompt of 128 tokens of the 8B architecture 5.18 -> 4.96 ms; a layer at 140 tokens 225 -> 217 us,
        // 2048 hidden at 256 tokens 127 -> 123).  Three chunks: no difference; four: a layer 464 -> 482 us.
        uint64_t policy;
        if (p.chunks <= 2) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
        else asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(policy));
        uint32_t slot = 0, use = 0;
        for (uint32_t j = 0; j < nunits + (SCALED ? R : 0) && ok; j++) {
            if (use) {
                if (!(ok = pg_wait_warp(b_rawempty + 8 * slot, (use - 1) & 1, p, 8))) break;
                // Block j - R has been read, so its scales are there too: this warp says so on the producers' behalf (they are short of time).
                if (SCALED && pg_elect()) pg_arrive(b_pdone + 8 * ((j - R) & (PG_DSLOTS - 1)));
                __syncwarp();
            }
            if (SCALED && j >= nunits) {
                if (++slot == R) { slot = 0; use++; }
                continue;
            }
            if (SCALED && j >= PG_DSLOTS && !(ok = pg_wait_warp(b_dempty + 8 * (j & (PG_DSLOTS - 1)), (j / PG_DSLOTS - 1) & 1, p, 8))) break;   // its scales' slot is free
            const uint32_t rt = CTAS * cur.rt + rank, s = rt >= p.tile0[2] ? 2 : (rt >= p.tile0[1] ? 1 : 0), y = (rt - p.tile0[s]) * 128;
            const uint32_t full = b_rawfull + 8 * slot, dst = raw0 + slot * RAW;
            const CUtensorMap *m = maps.m[s];
            if (pg_elect()) {
                pg_expect(full, FMT == PG_Q6K ? 128u * (144 + 80 + 16 + 16) : RAW);
                if (FMT == PG_Q6K) {
                    const uint32_t x0 = (cur.kb >> 3) * 1680, bb = cur.kb & 7;
                    pg_tma2d(dst + PG_Q6_QL, m + 0, x0 + 128 * bb, y, full, policy);
                    pg_tma2d(dst + PG_Q6_QH, m + 1, x0 + 1024 + 64 * bb, y, full, policy);
                    pg_tma2d(dst + PG_Q6_SC, m + 2, x0 + 1536 + 16 * bb, y, full, policy);
                    pg_tma2d(dst + PG_Q6_D, m + 2, x0 + 1664, y, full, policy);
                } else {
                    // Q8_0: 272 bytes = 136 elements of two bytes (a box is at most 256 elements wide)
                    pg_tma2d(dst, m, FMT == PG_Q80 ? cur.kb * 136 : cur.kb * (FMT == PG_Q4K ? 144 : 176), y, full, policy);
                }
            }
            __syncwarp();
            if (++slot == R) { slot = 0; use++; }
            cur.next(p);
        }
    }
    if (!ok) {
        // a wait gave up: bulk copies of this CTA may still be in flight; give them time to land before the CTA ends
        const unsigned long long t0 = pg_ns();
        while (pg_ns() - t0 < 100000ull) {}
    }
    if (warp == PG_W_MMA && ok) {
        // The last MMAs' commits arrive in shared memory, a pair's in both CTAs': let them, before a CTA can end.
        const uint32_t last = 4 * nunits - 1;
        pg_wait_warp(b_aempty + 8 * (last % NS), (last / NS) & 1, p, 9);
        pg_wait_warp(b_xempty + 8 * (last % XS), (last / XS) & 1, p, 9);
    }
    __syncwarp();
    pg_fence_before();
    pg_sync<PAIR>();   // the other CTA's shared and tensor memory are in use until here
    if (warp == PG_W_MMA) pg_dealloc<PAIR>(tmem);
}

template <int FMT, bool PAIR>
__global__ void __launch_bounds__(PG_THREADS, 1) prefill_gemm_kernel(const __grid_constant__ PgParams p, const __grid_constant__ PgMaps maps) {
    pg_gemm<FMT, PAIR>(p, maps, blockIdx.x);
}
// Matrices of two formats with the same inputs (q and k beside v in most files): the first CTAs take the one, the others the other, each its
// format's path.  As a launch of its own v's few tiles took a start and an end of a GEMM, and were cut into so many pieces that adding them up was
// most of the kernel behind it.
template <int A, int B, bool PAIR>
__global__ void __launch_bounds__(PG_THREADS, 1) prefill_gemm_mixed_kernel(const __grid_constant__ PgParams pa, const __grid_constant__ PgMaps ma,
                                                                           const __grid_constant__ PgParams pb, const __grid_constant__ PgMaps mb) {
    const uint32_t first = (PAIR ? 2 : 1) * pa.sk.ranges;
    if (blockIdx.x < first) pg_gemm<A, PAIR>(pa, ma, blockIdx.x);
    else pg_gemm<B, PAIR>(pb, mb, blockIdx.x - first);
}

// ---------------------------------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------------------------------
static uint32_t pg_units(uint32_t rows, uint32_t nb, uint32_t n, bool pair) {
    const uint32_t tile = pair ? 256 : 128;
    return (rows + tile - 1) / tile * ((n + PF_CHUNK - 1) / PF_CHUNK) * nb;
}
static uint32_t pg_most(const ib_ctx *ctx, bool pair) { return pair ? (ctx->sm_count >= 2 ? (uint32_t)ctx->sm_count / 2 : 1u) : (uint32_t)ctx->sm_count; }

StreamK prefill_streamk(const ib_ctx *ctx, uint32_t rows, uint32_t cols, uint32_t n) {
    StreamK sk;
    sk.nb = cols / 256;
    // One SM or a pair per tile.  A pair's start and end (its launch, tensor memory, meetings and remote arrivals) cost a launch about a
    // microsecond more, what it saves is L2 traffic of the inputs: nothing up to 16 tokens (us, one SM / pair: Q4_K 512 x 1024 10.0 / 10.1, 4096 x
    // 4096 17.2 / 18.6, 28672 x 4096 39.0 / 41.3), little where no CTA has more than a unit (1152 x 4096, 64 tokens 14.8 / 16.6; 256 x 2048 10.3 /
    // 12.0).  Beyond, pairs are the faster ones or equal (4096 x 4096, 40 tokens 20.4 / 19.3).
    const bool pair = n > PF_SINGLE_TOKENS || (n > PF_SINGLE_ALWAYS && (rows >> 7) * sk.nb > (uint32_t)ctx->sm_count);
    sk.row_log2 = pair ? 8 : 7;
    sk.total = pg_units(rows, sk.nb, n, pair);
    const uint32_t most = pg_most(ctx, pair);
    sk.ranges = sk.total < most ? sk.total : most;
    return sk;
}
// The same for a launch of two groups of rows of different formats: the ranges are dealt out so that the slower group ends as early as it can.  A
// unit of Q6_K (three products a weight) takes 3100 clocks, of Q4_K or Q5_K 2490.
void prefill_streamk_mixed(const ib_ctx *ctx, uint32_t rows_a, uint32_t rows_b, uint32_t cols, uint32_t n, StreamK &a, StreamK &b) {
    const StreamK all = prefill_streamk(ctx, rows_a + rows_b, cols, n);   // (one SM or two per tile)
    const bool pair = all.row_log2 == 8;
    a = b = all;
    a.total = pg_units(rows_a, all.nb, n, pair);
    b.total = pg_units(rows_b, all.nb, n, pair);
    const uint32_t most = pg_most(ctx, pair);
    uint32_t best = 0xFFFFFFFFu;
    for (uint32_t r = 1; r < most; r++) {
        const uint32_t ra = r < a.total ? r : a.total, rb = most - r < b.total ? most - r : b.total;
        const uint32_t ta = (a.total + ra - 1) / ra * 249, tb = (b.total + rb - 1) / rb * 310, t = ta > tb ? ta : tb;
        if (t < best) {
            best = t;
            a.ranges = ra;
            b.ranges = rb;
        }
    }
}
// Most planes a tile needs: a range of `len` units cut into pieces of at least floor(total / ranges) units each
uint32_t prefill_max_pieces(const StreamK &sk) {
    const uint32_t least = sk.total / sk.ranges;
    const uint32_t most = (sk.nb - 1) / least + 2;   // nb consecutive units touch at most this many ranges of that length
    return most < sk.ranges ? most : sk.ranges;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static EncodeTiledFn encode_tiled() {
    static EncodeTiledFn fn = [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) ptr = nullptr;
        return (EncodeTiledFn)ptr;
    }();
    return fn;
}

static int pg_format(const ib_qtensor *m) {
    switch (m->qtype) {
    case IB_Q4_K: return PG_Q4K;
    case IB_Q5_K: return PG_Q5K;
    case IB_Q6_K: return m->layout == LAYOUT_SOA ? PG_Q6K : -1;
    case IB_Q8_0: return m->layout == LAYOUT_SOA ? PG_Q80 : -1;
    default: return -1;
    }
}

bool prefill_gemm_eligible(const ib_qtensor *m) {
    return m->rows % 128 == 0 && m->cols % 256 == 0 && pg_format(m) >= 0 && ((uintptr_t)m->dev % 16) == 0 && m->row_bytes % 16 == 0;
}

// The matrix as a 2-D byte array [rows][row_bytes]; a box = one field of one block of 128 consecutive rows
static int32_t pg_encode(const ib_qtensor *m, int fmt, CUtensorMap *maps) {
    EncodeTiledFn encode = encode_tiled();
    IB_REQUIRE(encode, "prefill GEMM: the driver does not export cuTensorMapEncodeTiled");
    static const uint32_t widths[4][3] = {{144, 0, 0}, {176, 0, 0}, {144, 80, 16}, {136, 0, 0}};
    const cuuint32_t unit = fmt == PG_Q80 ? 2 : 1, estr[2] = {1, 1};
    const cuuint64_t dims[2] = {(cuuint64_t)m->row_bytes / unit, (cuuint64_t)m->rows}, strides[1] = {(cuuint64_t)m->row_bytes};
    for (int i = 0; i < 3 && widths[fmt][i]; i++) {
        const cuuint32_t box[2] = {widths[fmt][i], 128};
        const CUresult cr = encode(&maps[i], unit == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void *)m->dev, dims, strides, box, estr,
                                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        IB_REQUIRE(cr == CUDA_SUCCESS, "prefill GEMM: cuTensorMapEncodeTiled failed with %d", (int)cr);
    }
    return IB_OK;
}

// The inputs' ring of a launch; returns the shared memory that it takes
template <int FMT, bool PAIR>
static uint32_t pg_ring(PgParams &p) {
    constexpr uint32_t room = PG_SMEM_LIMIT - pg_fixed_smem(FMT);
    static_assert(room >= 3 * (PAIR ? PF_CHUNK / 2 : PF_SINGLE_TOKENS) * 256, "shared memory");
    p.x_tile = ((p.n < PF_CHUNK ? p.n : PF_CHUNK) + 15) / 16 * (PAIR ? 8 : 16) * 128;   // 64 columns of a CTA's (padded) tokens of a chunk
    p.x_stages = room / (2 * p.x_tile) < PG_XSTAGES_MAX ? room / (2 * p.x_tile) : PG_XSTAGES_MAX;
    return pg_fixed_smem(FMT) + p.x_stages * 2 * p.x_tile;
}

template <bool PAIR, typename... KArgs, typename... Args>
static int32_t pg_launch_kernel(ib_ctx *ctx, cudaStream_t s, void (*kernel)(KArgs...), bool &attr_set, uint32_t ranges, uint32_t smem, bool early, const Args &...args) {
    if (!attr_set) {
        IB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PG_SMEM_LIMIT));
        attr_set = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((PAIR ? 2 : 1) * ranges);
    cfg.blockDim = dim3(PG_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (PAIR) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = 2;
        attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
        cfg.numAttrs++;
    }
    if (early) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
        cfg.numAttrs++;
    }
    IB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    ctx->launches++;
    return IB_OK;
}

template <int FMT, bool PAIR>
static int32_t pg_launch(ib_ctx *ctx, cudaStream_t s, PgParams &p, const PgMaps &maps, bool early) {
    static bool attr_set[16] = {};
    const uint32_t smem = pg_ring<FMT, PAIR>(p);
    return pg_launch_kernel<PAIR>(ctx, s, prefill_gemm_kernel<FMT, PAIR>, attr_set[ctx->device & 15], p.sk.ranges, smem, early, p, maps);
}

template <int FMT>
static int32_t pg_launch_rows(ib_ctx *ctx, cudaStream_t s, PgParams &p, const PgMaps &maps, bool early) {
    return p.sk.row_log2 == 8 ? pg_launch<FMT, true>(ctx, s, p, maps, early) : pg_launch<FMT, false>(ctx, s, p, maps, early);
}

template <int A, bool PAIR>
static int32_t pg_launch_mixed(ib_ctx *ctx, cudaStream_t s, PgParams &pa, const PgMaps &ma, PgParams &pb, const PgMaps &mb) {
    static bool attr_set[16] = {};
    const uint32_t sa = pg_ring<A, PAIR>(pa), sb = pg_ring<PG_Q6K, PAIR>(pb);
    return pg_launch_kernel<PAIR>(ctx, s, prefill_gemm_mixed_kernel<A, PG_Q6K, PAIR>, attr_set[ctx->device & 15], pa.sk.ranges + pb.sk.ranges, sa > sb ? sa : sb, true, pa, ma, pb, mb);
}

// What a launch (or its part of one format) is told
static int32_t pg_describe(const ib_ctx *ctx, const PrefillPart &w, const __half *x, uint32_t n, PgParams &p, PgMaps &maps) {
    IB_REQUIRE(w.n_mats >= 1 && w.n_mats <= PF_MAX_SEGS, "prefill GEMM: %u matrices", w.n_mats);
    IB_REQUIRE(w.sk.total < (1u << 24), "prefill GEMM: %u units of work are too many for one launch", w.sk.total);
    IB_REQUIRE(((uintptr_t)x % 16) == 0, "prefill GEMM: the input tiles must be 16-byte aligned for the bulk copies");
    const int fmt = pg_format(w.mats[0]);
    p = PgParams{};
    uint32_t tiles = 0;
    for (uint32_t i = 0; i < PF_MAX_SEGS; i++) {
        p.tile0[i] = i < w.n_mats ? tiles : 0xFFFFFFFFu;
        if (i >= w.n_mats) continue;
        const ib_qtensor *m = w.mats[i];
        IB_REQUIRE(pg_format(m) == fmt && m->cols == w.mats[0]->cols, "prefill GEMM: the matrices of a launch differ in type or width");
        const int32_t rc = pg_encode(m, fmt, maps.m[i]);
        if (rc) return rc;
        tiles += (uint32_t)m->rows / 128;
    }
    p.rows = tiles * 128;
    p.n = n; p.chunks = (n + PF_CHUNK - 1) / PF_CHUNK; p.x = x; p.x_chunk = pf_x_halves((uint32_t)w.mats[0]->cols);
    p.plane0 = w.plane0; p.planes = w.planes; p.sk = w.sk; p.err = ctx->err_dev; p.wait_ns = ctx->wait_limit_ns;
    return IB_OK;
}

int32_t launch_prefill_gemm(ib_ctx *ctx, cudaStream_t s, const PrefillPart &w, const __half *x, uint32_t n, bool early) {
    PgParams p;
    PgMaps maps;
    const int32_t rc = pg_describe(ctx, w, x, n, p, maps);
    if (rc) return rc;
    switch (pg_format(w.mats[0])) {
    case PG_Q4K: return pg_launch_rows<PG_Q4K>(ctx, s, p, maps, early);
    case PG_Q5K: return pg_launch_rows<PG_Q5K>(ctx, s, p, maps, early);
    case PG_Q6K: return pg_launch_rows<PG_Q6K>(ctx, s, p, maps, early);
    case PG_Q80: return pg_launch_rows<PG_Q80>(ctx, s, p, maps, early);
    default: return set_error(IB_ERR_UNSUPPORTED, "prefill GEMM: a matrix of type %d", w.mats[0]->qtype);
    }
}

// Longer passes have v enough to do by itself.  A layer, us, two launches / one: 2048 hidden (q4_k and q6_k), 30 tokens 84.2 / 78.4, 128 99.7 / 96.4, 256
// 132.6 / 128.8, 300 152.1 / 152.9, 384 162.9 / 163.5; 4096 hidden 30 tokens 139.7 / 129.9, 128 168.2 / 166.8, 300 334.5 / 326.2, 384 369.2 / 365.7, 500
// 471.0 / 470.4.
bool prefill_mixable(const ib_qtensor *a, const ib_qtensor *b, uint32_t n) {
    const int fa = pg_format(a);
    return (fa == PG_Q4K || fa == PG_Q5K) && pg_format(b) == PG_Q6K && a->cols == b->cols && n <= (a->cols >= 4096 ? 3 : 2) * PF_CHUNK;
}
int32_t launch_prefill_gemm_mixed(ib_ctx *ctx, cudaStream_t s, const PrefillPart &a, const PrefillPart &b, const __half *x, uint32_t n) {
    IB_REQUIRE(prefill_mixable(a.mats[0], b.mats[0], n) && a.sk.row_log2 == b.sk.row_log2, "prefill GEMM: these matrices cannot share a launch");
    PgParams pa, pb;
    PgMaps ma, mb;
    int32_t rc = pg_describe(ctx, a, x, n, pa, ma);
    if (rc == IB_OK) rc = pg_describe(ctx, b, x, n, pb, mb);
    if (rc) return rc;
    const bool pair = a.sk.row_log2 == 8;
    if (pg_format(a.mats[0]) == PG_Q4K) return pair ? pg_launch_mixed<PG_Q4K, true>(ctx, s, pa, ma, pb, mb) : pg_launch_mixed<PG_Q4K, false>(ctx, s, pa, ma, pb, mb);
    return pair ? pg_launch_mixed<PG_Q5K, true>(ctx, s, pa, ma, pb, mb) : pg_launch_mixed<PG_Q5K, false>(ctx, s, pa, ma, pb, mb);
}

}  // namespace ib
