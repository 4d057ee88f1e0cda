// Device-side building blocks of the streaming quantized GEMV (gemv_stream.cu): mbarrier / bulk-copy wrappers with bounded
// waits, the byte-balanced row split, the per-format 64-weight unit dot products and the row-pair epilogues.
#pragma once

#include "gemv_common.cuh"

namespace ib {


constexpr int CW = 16;                          // consumer warps
constexpr int PIPES = 2;                        // pipelines: a producer warp, part of the ring and of the consumers, an epilogue warp
constexpr int W_PRODUCER = CW, W_EPILOGUE = CW + PIPES;
constexpr int STREAM_THREADS = (CW + 2 * PIPES) * 32;   // 20 warps: 5 per scheduler at 96 registers fill its register file
constexpr int PT_MAX = 16;                      // row pairs per tile

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)   // a waiting warp sleeps for a while instead of spinning through issue slots
        : "memory");
    return ok != 0;
}
// Bounded wait: returns false (and raises *err) if the phase does not complete within `limit_ns` (a context setting).
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// The clock is read (about a microsecond) and the limit applied only after many tries, out of line: what the loops of the kernel
// carry is the few instructions of the first ones.
__device__ __noinline__ bool mbar_wait_long(uint32_t bar, uint32_t parity, uint32_t *err, uint32_t code, unsigned long long limit_ns) {
    const unsigned long long t0 = global_ns();
    for (;;) {
        for (int i = 0; i < 256; i++)
            if (mbar_try_wait(bar, parity)) return true;
        if (global_ns() - t0 > limit_ns) break;
    }
    if (err) {
        *(volatile uint32_t *)err = code;   // mapped host memory: a plain store, made visible system-wide
        __threadfence_system();
    }
    return false;
}
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t *err, uint32_t code, unsigned long long limit_ns) {
#pragma unroll 1
    for (int i = 0; i < 64; i++)
        if (mbar_try_wait(bar, parity)) return true;
    return mbar_wait_long(bar, parity, err, code, limit_ns);
}
// A tagged word of the tensor-parallel exchange: waits (bounded) until the word carries `tag`, returns its value.
__device__ __forceinline__ float wait_tagged(const uint2 *w, uint32_t tag, uint32_t *err, unsigned long long limit_ns) {
    uint2 v;
    asm volatile("ld.relaxed.sys.global.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(w) : "memory");
    if (v.y != tag) {
        const unsigned long long t0 = global_ns();
        for (;;) {
#pragma unroll 1
            for (int i = 0; i < 64 && v.y != tag; i++) asm volatile("ld.relaxed.sys.global.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(w) : "memory");
            if (v.y == tag) break;
            if (global_ns() - t0 > limit_ns) {
                if (err) {
                    *(volatile uint32_t *)err = 3;
                    __threadfence_system();
                }
                break;
            }
        }
    }
    return __uint_as_float(v.x);
}

__device__ __forceinline__ uint32_t ld_acquire_gpu(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// the same bounded wait on a counter that only this GPU's CTAs advance
__device__ __forceinline__ bool wait_counter_gpu(const uint32_t *flag, uint32_t target, uint32_t *err, uint32_t code, unsigned long long limit_ns) {
    if ((int32_t)(ld_acquire_gpu(flag) - target) >= 0) return true;
    const unsigned long long t0 = global_ns();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 64; i++)
            if ((int32_t)(ld_acquire_gpu(flag) - target) >= 0) return true;
        if (global_ns() - t0 > limit_ns) break;
    }
    if (err) {
        *(volatile uint32_t *)err = code;
        __threadfence_system();
    }
    return false;
}

// `policy`: an L2 eviction policy from evict_first_policy()
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar, uint64_t policy) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst), "l"(src), "r"(bytes),
                 "r"(bar), "l"(policy)
                 : "memory");
}
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}

// Shared-memory loads by 32-bit shared address (no generic-address arithmetic in the inner loop).  volatile: they stay
// between the mbarrier wait before them and the arrival after them.
__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
    return v;
}

// ---- this CTA's share of the work: per segment a contiguous range of row pairs, balanced by bytes ----
// (three scalar sets instead of arrays: indexing them with a run-time segment number would put them in local memory)
struct Share {
    uint32_t a0, a1, a2, b0, b1, b2;   // pair range per segment
    uint32_t t0, t1, t2;               // pairs per tile
    uint32_t nseg;
    __device__ __forceinline__ uint32_t a(uint32_t s) const { return s == 0 ? a0 : (s == 1 ? a1 : a2); }
    __device__ __forceinline__ uint32_t b(uint32_t s) const { return s == 0 ? b0 : (s == 1 ? b1 : b2); }
    __device__ __forceinline__ uint32_t pt(uint32_t s) const { return s == 0 ? t0 : (s == 1 ? t1 : t2); }
};

// What the split needs, from the host: nothing here divides (a handful of 32-bit divisions at its start cost every launch a microsecond
// before its first copy).  All byte counts are in units of 16 bytes.
//
// A CTA works on one weight format: where a launch mixes formats (q, k, v of most files), the CTAs are dealt out to the runs of segments of one
// format ("groups") in proportion to their bytes.  Rounded to whole CTAs that is at most 3 % off where a group has 33 of them.  With CTAs that went
// from one format to the next on the way, through code that switched between them, a 1B-architecture token took 405 instead of 397 us, an 8B one
// 1323 instead of 1307: a launch fetched twice the code, and loaded its operands a second time behind the first tile.
struct ShareGeom {
    uint64_t scale[3];     // per group: its bytes / its pipelines in units of 2^-32, rounded up
    uint32_t base[3];      // where the group begins in the launch's bytes
    uint32_t cta0[3];      // its first CTA (0xFFFFFFFF: no such group)
    uint32_t seg0[3];      // its first segment
    uint32_t start[3];     // where a segment begins in the launch's bytes
    uint32_t cost16[3];    // bytes per pair
    uint32_t inv[3];       // 2^32 / cost16, rounded up
};
// The first pair that belongs to the part of the launch behind byte `at`.  Neighbours call it with the same `at`, so their ranges meet
// whatever the product's rounding does; it never decreases, gives 0 at the segment's start and all pairs at its end.
__host__ __device__ __forceinline__ uint32_t share_pair(uint32_t at, uint32_t start, uint32_t cost16, uint32_t inv, uint32_t pairs) {
    if (at <= start) return 0;
    const uint32_t n = (uint32_t)(((uint64_t)(at - start + cost16 - 1) * inv) >> 32);
    return n < pairs ? n : pairs;
}
__host__ __device__ __forceinline__ uint32_t share_byte(uint64_t scale, uint32_t me) { return (uint32_t)((me * scale) >> 32); }
__device__ __forceinline__ uint32_t share_group(const ShareGeom &g, uint32_t cta) { return cta >= g.cta0[2] ? 2u : (cta >= g.cta0[1] ? 1u : 0u); }
// `scale`, `base`: the group's; `me`: the pipeline's number among its group's
__device__ __forceinline__ void make_share(const ShareGeom &g, const uint32_t (&pairs)[3], const uint32_t (&pt)[3], uint32_t nseg, uint64_t scale, uint32_t base, uint32_t me, Share &sh) {
    const uint32_t lo = base + share_byte(scale, me), hi = base + share_byte(scale, me + 1);
    sh.nseg = nseg;
    sh.a0 = share_pair(lo, g.start[0], g.cost16[0], g.inv[0], pairs[0]);
    sh.b0 = share_pair(hi, g.start[0], g.cost16[0], g.inv[0], pairs[0]);
    sh.a1 = share_pair(lo, g.start[1], g.cost16[1], g.inv[1], pairs[1]);
    sh.b1 = share_pair(hi, g.start[1], g.cost16[1], g.inv[1], pairs[1]);
    sh.a2 = share_pair(lo, g.start[2], g.cost16[2], g.inv[2], pairs[2]);
    sh.b2 = share_pair(hi, g.start[2], g.cost16[2], g.inv[2], pairs[2]);
    sh.t0 = pt[0];
    sh.t1 = pt[1];
    sh.t2 = pt[2];
}

struct TileCursor {
    uint32_t seg, next, end, pt;   // segment, first pair of the next tile, end of the segment's range, pairs per tile
    __device__ __forceinline__ void enter(const Share &sh) {
        while (seg < sh.nseg) {
            next = sh.a(seg); end = sh.b(seg); pt = sh.pt(seg);
            if (next < end) break;
            seg++;
        }
    }
    __device__ __forceinline__ void init(const Share &sh) { seg = 0; next = end = pt = 0; enter(sh); }
    __device__ __forceinline__ bool valid(const Share &sh) const { return seg < sh.nseg; }
    __device__ __forceinline__ uint32_t count(const Share &) const { return (end - next) < pt ? (end - next) : pt; }
    __device__ __forceinline__ void advance(const Share &sh) {
        next += count(sh);
        if (next >= end) { seg++; enter(sh); }
    }
};

// -------------------------------------------------------------------------------------------------
// The dot products, on the integer tensor path (mma.sync m16n8k32, 8-bit operands, 32-bit accumulators).
//
// A warp works on 8 rows x 256 columns (a "block") at a time: lane (g, t) = (lane >> 2, lane & 3) reads 64 weights of row g
// and ends up with the integer dot products of unit t of that row: 64 columns with their sub-block scales, both activation
// limbs.  Four mma per block and format:
//  * the 16 rows of the A operand are two stretches, X and Y, of the same 8 weight rows (X in rows 0-7, Y in rows 8-15), so a
//    lane's A registers are simply what it read from row g;
//  * a sub-block must not be summed with its neighbours, so every sub-block gets its own pair of B columns (limb 0, limb 1) and
//    a column holds activations only in the k slots of its sub-block, zeros elsewhere.  The four column pairs serve two
//    sub-blocks of X and two of Y; the accumulators where a row meets the other stretch's columns are not used;
//  * accumulator columns 2t, 2t+1 land in lane t: a select between the X and the Y rows leaves every lane with one unit.
// The order of the k slots is free as long as A and B agree; it is chosen so that a lane's bytes are consecutive in memory.
// Rows of more than 16 blocks are so long that 8 of them are a third to a half of the ring; they are worked on 4 rows x 512 columns
// at a time.  The A rows are then stretch X of the 4 rows, stretch Y of the 4 rows - both of one block - and the same of the next
// block, which has B columns of its own: 8 mma with half of the results used, and everything else as before (with 8-row tiles HBM
// waited for the consumers: two tiles fill the ring and land together; with 8-row products of 4-row tiles the consumers became the
// limit).
// Per 64 weights this issues 4 mma and 16 masks where byte dot products took 32 dp4a, and the row sum needs 2 shuffles per
// 8 rows instead of 5 per 2 rows.  HBM delivers 64 Q4_K weights per lane and scheduler every ~195 clocks; the dot products took
// about 250, these take about 100.
// -------------------------------------------------------------------------------------------------
constexpr int NB_MAX = 4;   // blocks of 256 columns per consumer warp

// c = a . b, or c += a . b
#define IB_MMA(NAME, TYPE)                                                                                                               \
    __device__ __forceinline__ void NAME(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {     \
        asm("mma.sync.aligned.m16n8k32.row.col.s32." TYPE ".s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"            \
            : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])                                                                             \
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));                                                             \
    }                                                                                                                                    \
    __device__ __forceinline__ void NAME##_add(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) { \
        asm("mma.sync.aligned.m16n8k32.row.col.s32." TYPE ".s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"                \
            : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])                                                                             \
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));                                                                     \
    }
IB_MMA(mma_u8, "u8")
IB_MMA(mma_s8, "s8")
#undef IB_MMA

// Everything that depends only on the lane and the warp's first block: byte offsets inside a row, shifts, masks.
struct LaneConst {
    uint32_t o0, o1, o2, o3;   // byte offsets inside a row
    uint32_t sh, ma, mb, mc;   // scale extraction: byte selector, masks
    uint32_t h0, h1;           // Q5_K: shifts of the fifth bits
    uint32_t sc, sx;           // shared addresses of the unit's activation scales and 16-column sums
    bool first;                // this lane's unit is in accumulator rows 0-7
};

// The lane's unit of a step: activation scales and sums, ready for the format's formula.  At most two steps per warp: kept in
// registers (8 rows at a time); longer rows read them from shared memory for every dot product.
struct UnitAct { float s[4], x[4]; };

// A byte of `w` (the `sel`-th, see byte_selector) as a float: behind the exponent of 2^23 its value is the float's low bits.  A byte
// permute and an addition on the floating-point pipe; extracting and converting it are two instructions of the integer pipe, which is
// what the dot products are short of (it takes a warp instruction every other clock).
constexpr uint32_t BYTE_SELECTOR = 0x7440u;   // + the byte's number
__device__ __forceinline__ float byte_to_float(uint32_t w, uint32_t sel, float bias = 8388608.0f) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, sel)) - bias;
}

// 6-bit (scale, min) pairs of sub-blocks 2t and 2t+1 of a Q4_K / Q5_K header, as bytes scale 2t, scale 2t+1, min 2t, min 2t+1, without a
// branch on t (the lanes of a warp differ in t): lanes with t < 2 carry masks (0x3F.., 0, 0), the others (0, 0x30.., 0x0F..), and both
// read the same half of the header's words (crates/inferi/src/quantization.rs:394-402).
__device__ __forceinline__ uint32_t kquant_scales_lane(const uint4 &hdr, const LaneConst &lc) {
    const uint32_t p = __byte_perm(hdr.y, hdr.z, lc.sh), q = __byte_perm(hdr.w, hdr.w >> 4, lc.sh);
    return (p & lc.ma) | ((p >> 2) & lc.mb) | (q & lc.mc);
}
// d * (sc_lo * lo + sc_hi * hi) - dmin * (m_lo * x_lo + m_hi * x_hi) for the 64 columns of a unit of a Q4_K / Q5_K block;
// `lo`, `hi`: the integer dot products, a.s their units, a.x the sums of the columns
__device__ __forceinline__ float kquant_finish(const uint4 &hdr, const LaneConst &lc, float lo, float hi, const float s0, const float s1, const float x0, const float x1) {
    const uint32_t k = kquant_scales_lane(hdr, lc);
    const float2 dm = __half22float2(*reinterpret_cast<const __half2 *>(&hdr.x));
    const float a = byte_to_float(k, BYTE_SELECTOR) * (s0 * lo) + byte_to_float(k, BYTE_SELECTOR + 1) * (s1 * hi);
    const float b = byte_to_float(k, BYTE_SELECTOR + 2) * x0 + byte_to_float(k, BYTE_SELECTOR + 3) * x1;
    return dm.x * a - dm.y * b;
}
// scales of columns 64u .. +31 and +32 .. +63 of the block and the sums of the same columns; `hi_unit`: what a high dot product counts
template <bool FOUR>
__device__ __forceinline__ void kquant_unit(const LaneConst &lc, uint32_t i, float hi_unit, UnitAct &a) {
    const uint2 s = lds64(lc.sc + (FOUR ? 64 : 32) * i);
    const uint4 x = lds128(lc.sx + (FOUR ? 128 : 64) * i);
    a.s[0] = __uint_as_float(s.x);
    a.s[1] = __uint_as_float(s.y) * hi_unit;
    a.x[0] = __uint_as_float(x.x) + __uint_as_float(x.y);
    a.x[1] = __uint_as_float(x.z) + __uint_as_float(x.w);
}
// this lane's unit out of the accumulators (4 rows: `e` has the products with the second block's operand)
template <bool FOUR>
__device__ __forceinline__ float unit_of(const int (&c)[4], const int (&e)[4], bool first) {
    const int lower = limb_sum(c[0], c[1]), upper = FOUR ? limb_sum(e[2], e[3]) : limb_sum(c[2], c[3]);
    return (float)(first ? lower : upper);
}
// Which rows and units a lane works on.  `sx`: the stretch in its lower A row (the upper one holds the other stretch, or the same
// stretch of the next block); `own`: its unit is in the lower A rows; `u`: the unit, of block `next` (0, 1) of the step.
struct LaneUnit { uint32_t sx, u, next; bool own; };
template <bool FOUR>
__device__ __forceinline__ LaneUnit lane_unit(uint32_t g, uint32_t t, bool swap) {
    LaneUnit l;
    l.sx = (FOUR ? g >> 2 : 0u) ^ (swap ? 1u : 0u);
    l.own = (t >> 1) == l.sx;
    l.next = FOUR && !l.own ? 1u : 0u;
    l.u = l.next ? t ^ 2u : t;
    return l;
}

// Per format:  init: the lane's constants for the warp's first block `blk` (rows `stride` bytes apart);  operand: the B registers
// of block `blk` (`limb`: shared address of limb (g & 1) of the activations: B column g belongs to unit g >> 1, limb g & 1; the
// second block of a 4-row step has the units of X and Y exchanged: pass g ^ 4);  dot: step `i` (a block, or two) of the row at
// shared address `row`, operands `b`, `b2` -> the lane's unit of that row;  unit: the activations' side of step i.
template <uint32_t QT> struct Frag;

// Rows whose stride is close to a multiple of the 128 bytes of a shared-memory wavefront all start at the same bank: every other
// row then reads its stretch Y first, so that the two rows a wavefront serves use both halves of the banks.
__device__ __forceinline__ bool swap_stretches(uint32_t g, uint32_t stride) { return (g & 1) && ((stride + 32) & 127) < 64; }

// Q4_K and Q5_K: X = the 64 quant bytes of units 0 and 1 (each 32 bytes: low nibbles sub-block 2t, high nibbles 2t+1), Y = units
// 2 and 3; lane t holds 16 bytes of unit (t >> 1) of either.
template <bool FOUR>
__device__ __forceinline__ void kquant_init(uint32_t g, uint32_t t, uint32_t stride, uint32_t block_bytes, uint32_t quants_at, uint32_t blk, LaneConst &lc) {
    const LaneUnit l = lane_unit<FOUR>(g, t, swap_stretches(g, stride));
    const uint32_t at = blk * block_bytes;
    lc.o0 = at + l.next * block_bytes;
    lc.o1 = at + quants_at + 16 * t + 64 * l.sx;
    lc.o2 = FOUR ? lc.o1 + block_bytes : at + quants_at + 16 * t + 64 * (1 - l.sx);
    lc.first = l.own;
    lc.sh = l.u & 1 ? 0x7632u : 0x5410u;   // bytes 2 and 3, or 0 and 1, of either operand
    lc.ma = l.u < 2 ? 0x3F3F3F3Fu : 0u;
    lc.mb = l.u < 2 ? 0u : 0x30303030u;
    lc.mc = l.u < 2 ? 0u : 0x0F0F0F0Fu;
    lc.o3 = at + 16 + 16 * (t & 1);   // Q5_K: the fifth bits of this lane's 16 columns, bit 2u / 2u+1 of a byte for unit u
    lc.h0 = 2 * (t >> 1) + 4 * l.sx;
    lc.h1 = FOUR ? lc.h0 : 2 * (t >> 1) + 4 * (1 - l.sx);
    lc.sc += 4 * (8 * (blk + l.next) + 2 * l.u);
    lc.sx += 4 * (16 * (blk + l.next) + 4 * l.u);
}
__device__ __forceinline__ void load_operand(uint32_t lo_at, uint32_t hi_at, uint32_t (&b)[8]) {
    const uint4 lo = lds128(lo_at), hi = lds128(hi_at);
    b[0] = lo.x; b[1] = lo.y; b[2] = lo.z; b[3] = lo.w;
    b[4] = hi.x; b[5] = hi.y; b[6] = hi.z; b[7] = hi.w;
}
// `zeros`: shared address of 16 bytes of zeros, what a lane's slots outside its column's sub-block hold
__device__ __forceinline__ void kquant_operand(uint32_t g, uint32_t t, uint32_t limb, uint32_t zeros, uint32_t blk, uint32_t (&b)[8]) {
    const uint32_t q = g >> 1, at = limb + 256 * blk + 64 * q + 16 * (t & 1);
    const bool has = (t >> 1) == (q & 1);
    load_operand(has ? at : zeros, has ? at + 32 : zeros, b);
}

template <> struct Frag<IB_Q4_K> {
    template <bool FOUR>
    static __device__ __forceinline__ void unit(const LaneConst &lc, uint32_t i, UnitAct &a) { kquant_unit<FOUR>(lc, i, 1.0f / 16.0f, a); }
    template <bool FOUR>
    static __device__ __forceinline__ void init(uint32_t g, uint32_t t, uint32_t stride, uint32_t blk, LaneConst &lc) { kquant_init<FOUR>(g, t, stride, 144, 16, blk, lc); }
    static __device__ __forceinline__ void operand(uint32_t g, uint32_t t, uint32_t limb, uint32_t zeros, uint32_t blk, uint32_t (&b)[8]) { kquant_operand(g, t, limb, zeros, blk, b); }
    template <bool FOUR>
    static __device__ __forceinline__ float dot(uint32_t row, const LaneConst &lc, uint32_t i, const uint32_t (&b)[8], const uint32_t (&b2)[8], const UnitAct &a) {
        constexpr uint32_t LO = 0x0F0F0F0Fu, HI = 0xF0F0F0F0u, STEP = FOUR ? 2 * 144 : 144;   // high nibbles are used in place: 16 q
        const uint4 v = lds128(row + lc.o1 + STEP * i), w = lds128(row + lc.o2 + STEP * i), hdr = lds128(row + lc.o0 + STEP * i);
        int L[4], H[4], L2[4], H2[4];
        mma_u8(L, v.x & LO, w.x & LO, v.y & LO, w.y & LO, b[0], b[1]);
        mma_u8(H, v.x & HI, w.x & HI, v.y & HI, w.y & HI, b[4], b[5]);
        if (FOUR) mma_u8(L2, v.x & LO, w.x & LO, v.y & LO, w.y & LO, b2[0], b2[1]);
        if (FOUR) mma_u8(H2, v.x & HI, w.x & HI, v.y & HI, w.y & HI, b2[4], b2[5]);
        mma_u8_add(L, v.z & LO, w.z & LO, v.w & LO, w.w & LO, b[2], b[3]);
        mma_u8_add(H, v.z & HI, w.z & HI, v.w & HI, w.w & HI, b[6], b[7]);
        if (FOUR) mma_u8_add(L2, v.z & LO, w.z & LO, v.w & LO, w.w & LO, b2[2], b2[3]);
        if (FOUR) mma_u8_add(H2, v.z & HI, w.z & HI, v.w & HI, w.w & HI, b2[6], b2[7]);
        return kquant_finish(hdr, lc, unit_of<FOUR>(L, L2, lc.first), unit_of<FOUR>(H, H2, lc.first), a.s[0], a.s[1], a.x[0], a.x[1]);
    }
};

template <> struct Frag<IB_Q5_K> {
    template <bool FOUR>
    static __device__ __forceinline__ void unit(const LaneConst &lc, uint32_t i, UnitAct &a) { kquant_unit<FOUR>(lc, i, 1.0f, a); }
    template <bool FOUR>
    static __device__ __forceinline__ void init(uint32_t g, uint32_t t, uint32_t stride, uint32_t blk, LaneConst &lc) { kquant_init<FOUR>(g, t, stride, 176, 48, blk, lc); }
    static __device__ __forceinline__ void operand(uint32_t g, uint32_t t, uint32_t limb, uint32_t zeros, uint32_t blk, uint32_t (&b)[8]) { kquant_operand(g, t, limb, zeros, blk, b); }
    static __device__ __forceinline__ uint32_t lo5(uint32_t q, uint32_t h) { return (q & 0x0F0F0F0Fu) | ((h << 4) & 0x10101010u); }
    static __device__ __forceinline__ uint32_t hi5(uint32_t q, uint32_t h) { return ((q >> 4) & 0x0F0F0F0Fu) | ((h << 3) & 0x10101010u); }
    template <bool FOUR>
    static __device__ __forceinline__ float dot(uint32_t row, const LaneConst &lc, uint32_t i, const uint32_t (&b)[8], const uint32_t (&b2)[8], const UnitAct &a) {
        constexpr uint32_t STEP = FOUR ? 2 * 176 : 176;
        const uint4 v = lds128(row + lc.o1 + STEP * i), w = lds128(row + lc.o2 + STEP * i), h = lds128(row + lc.o3 + STEP * i);
        const uint4 k = FOUR ? lds128(row + lc.o3 + STEP * i + 176) : h, hdr = lds128(row + lc.o0 + STEP * i);
        const uint32_t hv[4] = {h.x >> lc.h0, h.y >> lc.h0, h.z >> lc.h0, h.w >> lc.h0}, hw[4] = {k.x >> lc.h1, k.y >> lc.h1, k.z >> lc.h1, k.w >> lc.h1};
        int L[4], H[4], L2[4], H2[4];
        const uint32_t vv[4] = {v.x, v.y, v.z, v.w}, ww[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
            const uint32_t l0 = lo5(vv[j], hv[j]), l1 = lo5(ww[j], hw[j]), l2 = lo5(vv[j + 1], hv[j + 1]), l3 = lo5(ww[j + 1], hw[j + 1]);
            const uint32_t h0 = hi5(vv[j], hv[j]), h1 = hi5(ww[j], hw[j]), h2 = hi5(vv[j + 1], hv[j + 1]), h3 = hi5(ww[j + 1], hw[j + 1]);
            if (j == 0) {
                mma_u8(L, l0, l1, l2, l3, b[0], b[1]);
                mma_u8(H, h0, h1, h2, h3, b[4], b[5]);
                if (FOUR) mma_u8(L2, l0, l1, l2, l3, b2[0], b2[1]);
                if (FOUR) mma_u8(H2, h0, h1, h2, h3, b2[4], b2[5]);
            } else {
                mma_u8_add(L, l0, l1, l2, l3, b[2], b[3]);
                mma_u8_add(H, h0, h1, h2, h3, b[6], b[7]);
                if (FOUR) mma_u8_add(L2, l0, l1, l2, l3, b2[2], b2[3]);
                if (FOUR) mma_u8_add(H2, h0, h1, h2, h3, b2[6], b2[7]);
            }
        }
        return kquant_finish(hdr, lc, unit_of<FOUR>(L, L2, lc.first), unit_of<FOUR>(H, H2, lc.first), a.s[0], a.s[1], a.x[0], a.x[1]);
    }
};

// Q6_K rows are stored as groups of 8 blocks: [8 x 128 ql][8 x 64 qh][8 x 16 scales][8 x 2 d] = 1680 bytes per 2048 columns.
// X / Y = halves 0 / 1 of a block (128 columns; their 32-byte ql segments hold columns +0 and +64, and +32 and +96).  A scale
// covers 16 columns, so each of the four 32-column stretches of a half is a product of its own; lane t holds 8 of its columns.
// Unit t: half i = t >> 1, 16-column half h = t & 1 of all four stretches.
template <> struct Frag<IB_Q6_K> {
    template <bool FOUR>
    static __device__ __forceinline__ void init(uint32_t g, uint32_t t, uint32_t, uint32_t blk, LaneConst &lc) {
        const LaneUnit l = lane_unit<FOUR>(g, t, false);
        const uint32_t grp = (blk >> 3) * 1680, bb = blk & 7;   // a warp's blocks never straddle a group: their number divides 8
        lc.o0 = grp + 128 * bb + 8 * t + (FOUR ? 64 * l.sx : 0);
        lc.o1 = grp + 1024 + 64 * bb + 8 * t + (FOUR ? 32 * l.sx : 0);
        lc.o2 = grp + 1536 + 16 * (bb + l.next) + 8 * (l.u >> 1);
        lc.o3 = grp + 1664 + 2 * (bb + l.next);
        lc.sh = BYTE_SELECTOR + (l.u & 1);
        lc.ma = lc.mb = lc.mc = lc.h0 = lc.h1 = 0;
        lc.first = l.own;
        lc.sc += 4 * (8 * (blk + l.next) + 4 * (l.u >> 1));
        lc.sx += 4 * (16 * (blk + l.next) + 8 * (l.u >> 1) + (l.u & 1));
    }
    static __device__ __forceinline__ void operand(uint32_t g, uint32_t t, uint32_t limb, uint32_t zeros, uint32_t blk, uint32_t (&b)[8]) {
        const uint32_t i = g >> 2, h = (g >> 1) & 1;
        const uint32_t at = limb + 256 * blk + 128 * i + 16 * h + 8 * (t & 1);
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const uint2 v = lds64((t >> 1) == h ? at + 32 * s : zeros);
            b[2 * s] = v.x;
            b[2 * s + 1] = v.y;
        }
    }
    template <bool FOUR>
    static __device__ __forceinline__ void unit(const LaneConst &lc, uint32_t i, UnitAct &a) {
        constexpr uint32_t K = FOUR ? 2 : 1;
        const uint4 s = lds128(lc.sc + 32 * K * i);
        a.s[0] = __uint_as_float(s.x); a.s[1] = __uint_as_float(s.y); a.s[2] = __uint_as_float(s.z); a.s[3] = __uint_as_float(s.w);
#pragma unroll
        for (int k = 0; k < 4; k++) a.x[k] = -32.0f * __uint_as_float(lds32(lc.sx + 64 * K * i + 8 * k));
    }
    // crates/inferi/src/quantization.rs:237-246: 4 low bits from ql, 2 high bits from qh.  `h`: the two bits in bits 4-5 of each
    // byte, bits 6-7 clear; bits 0-3 are dropped
    static __device__ __forceinline__ uint32_t join(uint32_t q, uint32_t h) { return (q & 0x0F0F0F0Fu) | (h & 0xF0F0F0F0u); }
    template <bool FOUR>
    static __device__ __forceinline__ float dot(uint32_t row, const LaneConst &lc, uint32_t i, const uint32_t (&b)[8], const uint32_t (&b2)[8], const UnitAct &a) {
        constexpr uint32_t K = FOUR ? 2 : 1;   // the upper A rows: the other half, 64 (32) bytes on, or the next block, 128 (64) bytes on
        const uint32_t q0 = row + lc.o0 + 128 * K * i, h0 = row + lc.o1 + 64 * K * i;
        const uint2 hx = lds64(h0), hy = lds64(h0 + 32 * K);
        const uint2 ax = lds64(q0), ay = lds64(q0 + 64 * K), bx = lds64(q0 + 32), by = lds64(q0 + 32 + 64 * K);
        constexpr uint32_t M = 0x33333333u;
        int D[4][4], E[4][4];
#pragma unroll
        for (int s = 0; s < 2; s++) {   // the two 32-byte segments: columns +0, +64 and +32, +96 of a half
            const uint2 x = s ? bx : ax, y = s ? by : ay;
            const uint32_t e0 = (s ? hx.x >> 2 : hx.x) & M, e1 = (s ? hy.x >> 2 : hy.x) & M, e2 = (s ? hx.y >> 2 : hx.y) & M, e3 = (s ? hy.y >> 2 : hy.y) & M;
            const uint32_t l0 = join(x.x, e0 << 4), l1 = join(y.x, e1 << 4), l2 = join(x.y, e2 << 4), l3 = join(y.y, e3 << 4);
            const uint32_t u0 = join(x.x >> 4, e0), u1 = join(y.x >> 4, e1), u2 = join(x.y >> 4, e2), u3 = join(y.y >> 4, e3);
            mma_u8(D[s], l0, l1, l2, l3, b[2 * s], b[2 * s + 1]);
            mma_u8(D[s + 2], u0, u1, u2, u3, b[2 * s + 4], b[2 * s + 5]);
            if (FOUR) mma_u8(E[s], l0, l1, l2, l3, b2[2 * s], b2[2 * s + 1]);
            if (FOUR) mma_u8(E[s + 2], u0, u1, u2, u3, b2[2 * s + 4], b2[2 * s + 5]);
        }
        const uint2 scw = lds64(row + lc.o2 + 16 * K * i);   // scales[8 half .. +7]: stretch s is byte 2s + h
        const float d = h2f(lds16(row + lc.o3 + 2 * K * i));
        const uint32_t sa = scw.x ^ 0x80808080u, sb = scw.y ^ 0x80808080u;   // signed bytes, 128 too high
        constexpr float BIAS = 8388608.0f + 128.0f;
        const float w[4] = {byte_to_float(sa, lc.sh, BIAS), byte_to_float(sa, lc.sh + 2, BIAS), byte_to_float(sb, lc.sh, BIAS), byte_to_float(sb, lc.sh + 2, BIAS)};
        float v = 0.f;
#pragma unroll
        for (int k = 0; k < 4; k++) v += w[k] * (a.s[k] * unit_of<FOUR>(D[k], E[k], lc.first) + a.x[k]);
        return d * v;
    }
};

// Q8_0 rows are stored as groups of 8 blocks: [8 x 32 quants][8 x 2 scale] = 272 bytes per 256 columns.  Two products: X, Y =
// blocks 0-1, 2-3 of the group and 4-5, 6-7; unit t is blocks t and 4 + t.
template <> struct Frag<IB_Q8_0> {
    template <bool FOUR>
    static __device__ __forceinline__ void unit(const LaneConst &lc, uint32_t i, UnitAct &a) {
        a.s[0] = __uint_as_float(lds32(lc.sc + (FOUR ? 64 : 32) * i));
        a.s[1] = __uint_as_float(lds32(lc.sc + (FOUR ? 64 : 32) * i + 16));
    }
    template <bool FOUR>
    static __device__ __forceinline__ void init(uint32_t g, uint32_t t, uint32_t stride, uint32_t blk, LaneConst &lc) {
        const LaneUnit l = lane_unit<FOUR>(g, t, swap_stretches(g, stride));
        lc.o0 = 272 * (blk + l.next) + 256 + 2 * l.u;
        lc.o1 = 272 * blk + 16 * t + 64 * l.sx;
        lc.o2 = FOUR ? lc.o1 + 272 : 272 * blk + 16 * t + 64 * (1 - l.sx);
        lc.o3 = lc.sh = lc.ma = lc.mb = lc.mc = lc.h0 = lc.h1 = 0;
        lc.first = l.own;
        lc.sc += 4 * (8 * (blk + l.next) + l.u);
    }
    static __device__ __forceinline__ void operand(uint32_t g, uint32_t t, uint32_t limb, uint32_t zeros, uint32_t blk, uint32_t (&b)[8]) {
        const uint32_t q = g >> 1, at = limb + 256 * blk + 32 * q + 16 * (t & 1);
        const bool has = (t >> 1) == (q & 1);
        load_operand(has ? at : zeros, has ? at + 128 : zeros, b);
    }
    template <bool FOUR>
    static __device__ __forceinline__ float dot(uint32_t row, const LaneConst &lc, uint32_t i, const uint32_t (&b)[8], const uint32_t (&b2)[8], const UnitAct &a) {
        constexpr uint32_t K = FOUR ? 2 : 1;
        const uint32_t p = row + lc.o1 + 272 * K * i, c = row + lc.o2 + 272 * K * i;
        const uint4 v = lds128(p), w = lds128(c), y = lds128(p + 128), z = lds128(c + 128);
        const float d0 = h2f(lds16(row + lc.o0 + 272 * K * i)), d1 = h2f(lds16(row + lc.o0 + 272 * K * i + 8));
        int P[4], Q[4], P2[4], Q2[4];
        mma_s8(P, v.x, w.x, v.y, w.y, b[0], b[1]);
        mma_s8(Q, y.x, z.x, y.y, z.y, b[4], b[5]);
        if (FOUR) mma_s8(P2, v.x, w.x, v.y, w.y, b2[0], b2[1]);
        if (FOUR) mma_s8(Q2, y.x, z.x, y.y, z.y, b2[4], b2[5]);
        mma_s8_add(P, v.z, w.z, v.w, w.w, b[2], b[3]);
        mma_s8_add(Q, y.z, z.z, y.w, z.w, b[6], b[7]);
        if (FOUR) mma_s8_add(P2, v.z, w.z, v.w, w.w, b2[2], b2[3]);
        if (FOUR) mma_s8_add(Q2, y.z, z.z, y.w, z.w, b2[6], b2[7]);
        return d0 * (a.s[0] * unit_of<FOUR>(P, P2, lc.first)) + d1 * (a.s[1] * unit_of<FOUR>(Q, Q2, lc.first));
    }
};

constexpr uint32_t QT_MIXED = 0xFFu;   // kernel instance for launches whose segments differ in format: every CTA takes the path of its own

// How a launch's rows are split over the consumer warps: NB blocks of 256 columns per warp, CG warps side by side cover a row and
// form a stream, RG such streams share the tiles.  One or two blocks per warp where half of the warps then cover a row (one stream
// per pipeline; short rows leave room for two), four for longer rows - 8 rows at a time as long as three such tiles fit the ring
// (`long8`), else tiles of 4 rows: two of them at a time where the ring holds five, so that a step's successor is there when it ends, and the format
// and the number of tiles make it pay (4096 x 14336 Q4_K 10.6 -> 9.8 us, 4096 x 10240 Q6_K 10.0 -> 9.4; with a ring of four, 4096 x 14336 Q6_K 11.5 -> 12.0; the
// rule and its figures are beside the launcher), one otherwise.
// 8 rows of one or two blocks per warp, of up to four, 4 rows of up to four, 8 rows of up to four out of two tiles of 4
constexpr uint32_t ROWS8 = 0, ROWS8_LONG = 1, ROWS4 = 2, ROWS8_PAIR = 3;
struct Split { uint32_t NB, CG, RG, mode; };
inline Split split_of(uint32_t cols, bool long8) {
    const uint32_t blocks = cols / 256;
    Split s;
    s.NB = blocks <= 8 ? 1 : (blocks <= 16 ? 2 : NB_MAX);
    s.mode = s.NB < NB_MAX ? ROWS8 : (long8 ? ROWS8_LONG : ROWS4);
    s.CG = (blocks + s.NB - 1) / s.NB;
    s.RG = s.CG <= 4 ? 4 : (s.CG <= 8 ? 2 : 1);   // 1, or a multiple of the pipelines
    return s;
}

// -------------------------------------------------------------------------------------------------
// Prologue of the streaming kernel, run by the 16 consumer warps: y = x * w -> limb form in
// shared memory.  The RMS factor is NOT applied here: it is one scalar for the whole vector, the GEMV is linear, so the
// epilogue warp multiplies the finished row sums by it.  That takes the sum-of-squares reduction off the consumers'
// critical path: every warp leaves its part of the sum in red[warp], arrives on `ss_bar` and carries on; only the
// epilogue warp waits there.
// -------------------------------------------------------------------------------------------------
// A thread converts 8 consecutive columns at a time (a 32-column group is four lanes, a 16-column sum two): with 4096 columns
// all 512 threads take part - with 16 columns per thread half of them did, for twice as long.  `g`: the norm weights of
// the thread's first group, fetched ahead of the wait for the previous kernel.
__device__ __forceinline__ void pack_prefetch_norm8(const float *__restrict__ norm_w, uint32_t cols, float4 (&g)[2]) {
    const uint32_t grp = threadIdx.x;
    if (norm_w && grp < cols / 8) {
        g[0] = __ldg(reinterpret_cast<const float4 *>(norm_w) + 2 * grp);
        g[1] = __ldg(reinterpret_cast<const float4 *>(norm_w) + 2 * grp + 1);
    } else g[0] = g[1] = make_float4(1.f, 1.f, 1.f, 1.f);
}
// Eight floats past L1 (the previous kernel has just written them).  As two 16-byte loads a warp fetches every 32-byte sector
// twice, and all SMs want the same sectors at once.  `whole`: 32-byte aligned.
__device__ __forceinline__ void load_8(const float4 *p, bool whole, float4 &a, float4 &b) {
    if (whole)
        asm volatile("ld.global.cg.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                     : "l"(p)
                     : "memory");
    else {
        a = __ldcg(p);
        b = __ldcg(p + 1);
    }
}
// GROUPS: groups of 8 columns per thread, all in flight at once: 4096 columns each.
template <uint32_t GROUPS>
__device__ __forceinline__ void pack_stream(uint8_t *smem, uint32_t cols, const float *__restrict__ x, const float *__restrict__ norm_w, float *red,
                                            uint32_t ss_bar, const float4 (&g)[2]) {
    constexpr uint32_t NT = PACK_THREADS;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, groups = cols / 8;   // cols is a multiple of 256: whole warps
    const float4 *x4 = reinterpret_cast<const float4 *>(x), *w4 = reinterpret_cast<const float4 *>(norm_w);
    const bool whole = ((uintptr_t)x & 31) == 0;
    float4 r[GROUPS][2];
#pragma unroll
    for (uint32_t i = 0; i < GROUPS; i++) {
        const uint32_t grp = tid + NT * i;
        r[i][0] = r[i][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (grp < groups) load_8(x4 + 2 * grp, whole, r[i][0], r[i][1]);
    }
    if (norm_w) {
        // crates/inferi-shaders/src/rms_norm.rs:112-120: the sum of squares; the factor itself is applied by the epilogue warp
        float ss = 0.f;
#pragma unroll
        for (uint32_t i = 0; i < GROUPS; i++)
#pragma unroll
            for (int j = 0; j < 2; j++) ss += (r[i][j].x * r[i][j].x + r[i][j].y * r[i][j].y) + (r[i][j].z * r[i][j].z + r[i][j].w * r[i][j].w);
#pragma unroll
        for (int o = 16; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) {
            red[warp] = ss;
            mbar_arrive(ss_bar);   // a release: the epilogue warp's wait sees red[warp]
        }
    }
    float *sc = reinterpret_cast<float *>(smem + ACT_LIMBS * cols), *sx16 = sc + cols / 32;
#pragma unroll
    for (uint32_t i = 0; i < GROUPS; i++) {
        const uint32_t grp = tid + NT * i;
        if (warp * 32 + NT * i >= groups) continue;   // warp-uniform
        const bool ok = grp < groups;
        float4 (&v)[2] = r[i];
        if (norm_w && ok) {
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const float4 w = i == 0 ? g[j] : __ldg(w4 + 2 * grp + j);
                v[j].x *= w.x; v[j].y *= w.y; v[j].z *= w.z; v[j].w *= w.w;
            }
        }
        float amax = max_nan(abs_max(v[0]), abs_max(v[1]));
        amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = max_nan(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const float inv = pack_units(v, amax);
        uint32_t w0[2], w1[2];
        int s0 = 0, s1 = 0;
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const float e[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
            pack_four(e, inv, w0[j], w1[j], s0, s1);
        }
        int sum = limb_sum(s0, s1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        if (ok) {
            const uint32_t run = grp >> 1;
            *reinterpret_cast<uint2 *>(smem + 8 * grp) = make_uint2(w0[0], w0[1]);
            *reinterpret_cast<uint2 *>(smem + cols + 8 * grp) = make_uint2(w1[0], w1[1]);
            if ((grp & 3) == 0) sc[grp >> 2] = amax * (1.0f / ACT_STEPS);
            if ((grp & 1) == 0) sx16[run] = (float)sum * (amax * (1.0f / ACT_STEPS));
        }
    }
    named_barrier(1, PACK_THREADS);
}

// What the epilogue of a pair reads from memory: the residual, or the rotation of a q / k pair.  Requested ahead of the wait for
// the dot products.
__device__ __forceinline__ float2 epilogue_prefetch(const GemvParams &p, uint32_t s, uint32_t pair) {
    if (p.epi == EPI_RESIDUAL) return __ldcg(reinterpret_cast<const float2 *>(p.resid + 2 * pair));
    if (p.epi == EPI_QKV && s < 2) return __ldcg(p.rope_cs + (((2 * pair) % p.head_size) >> 1));
    return make_float2(0.f, 0.f);
}

// EPI_PUSH, out of line (as what else only some launches do: a launch fetches its code from L2, and what lies between the parts that it
// runs is fetched with them): row-split matrix of a tensor-parallel model, this rank's partial goes straight into every rank's memory
// ({value, tag} words: see GemvParams).
__device__ __noinline__ void push_pair(const GemvParams &p, uint32_t r0, float a, float b) {
    const uint32_t tag = (*p.epoch_ptr) * p.xchg_per_epoch + p.push_use;
    const uint4 w = make_uint4(__float_as_uint(a), tag, __float_as_uint(b), tag);
#pragma unroll 1
    for (uint32_t rk = 0; rk < p.tp; rk++) *reinterpret_cast<uint4 *>(p.push_dst[rk] + r0) = w;
}

// ---- epilogue of one row pair (run by an epilogue warp only, so the kind of epilogue is a run-time switch: one kernel
// instance per weight format serves every role in the token graph and stays in the instruction cache) ----
// `pre`: from epilogue_prefetch;  `pos`: the token's position (EPI_QKV).
__device__ __forceinline__ void epilogue(const GemvParams &p, uint32_t s, uint32_t pair, float a, float b, unsigned long long &best, float2 pre, uint32_t pos) {
    const uint32_t epi = p.epi;
    if (epi == EPI_SWIGLU) {
        // crates/inferi-shaders/src/silu.rs:16-19,46-52: a = gate row, b = up row
        p.seg[0].out[pair] = b * (a / (1.0f + expf(-a)));
        return;
    }
    const uint32_t r0 = 2 * pair;
    if (epi == EPI_STORE) {
        *reinterpret_cast<float2 *>(p.seg[s].out + r0) = make_float2(a, b);
    } else if (epi == EPI_RESIDUAL) {
        *reinterpret_cast<float2 *>(p.seg[s].out + r0) = make_float2(pre.x + a, pre.y + b);
    } else if (epi == EPI_QKV) {
        if (p.bias[s]) {
            const float2 bv = __ldg(reinterpret_cast<const float2 *>(p.bias[s] + r0));
            a += bv.x;
            b += bv.y;
        }
        if (s < 2) {
            // crates/inferi-shaders/src/rope.rs:75-91 (adjacent pairs)
            const float x = a, y = b;
            a = pre.x * x - pre.y * y;
            b = pre.y * x + pre.x * y;
        }
        if (s == 0) {
            *reinterpret_cast<float2 *>(p.seg[0].out + r0) = make_float2(a, b);
        } else {
            void *cache = (s == 1) ? p.k_cache : p.v_cache;
            const size_t off = (size_t)pos * p.kv_dim + r0;
            if (p.kv_dtype == IB_KV_F16) reinterpret_cast<__half2 *>(cache)[off >> 1] = __floats2half2_rn(a, b);
            else reinterpret_cast<float2 *>(cache)[off >> 1] = make_float2(a, b);
        }
    } else if (epi == EPI_PUSH) {
        push_pair(p, r0, a, b);
    } else if (epi == EPI_ARGMAX) {
        if (p.seg[0].out) *reinterpret_cast<float2 *>(p.seg[0].out + r0) = make_float2(a, b);
        best = max(best, max(argmax_key(a, p.row_offset + r0), argmax_key(b, p.row_offset + r0 + 1)));
    }
}

}  // namespace ib
