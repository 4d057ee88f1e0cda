// Streaming quantized GEMV for sm_100a: the kernel of the token loop.
//
// Replaces the reference shaders crates/inferi-shaders/src/gemv_quant_{q8_0x2,q4_k,q5_k,q6_kx2}.rs (one 32-thread
// workgroup per 4 rows, 4-byte scattered loads) and their launcher crates/inferi/src/ops/gemv_quant.rs:183-341.
//
// One persistent CTA per SM of sixteen consumer warps, as two pipelines (one where all warps are needed for one row).  Each has:
//  * A producer warp that streams rows from HBM into its part of a shared-memory ring with bulk asynchronous copies
//    (cp.async.bulk, one copy per tile of contiguous row pairs, completion on an mbarrier).  It starts before the kernel
//    waits for its predecessor (programmatic dependent launch): weights never depend on the previous kernel, so the ring
//    fills while that kernel is still finishing.
//  * Its consumer warps split a row's columns in blocks of 256 and work on eight rows at a time.  A warp's activations - two
//    int8 limbs per column, see gemv_common.cuh - stay in registers for the whole kernel as operands of integer mma, so
//    the inner loop touches shared memory for weights and scales only (gemv_stream.cuh).
//  * Per-warp partial row sums meet in shared memory; the epilogue warp adds them in a fixed order and runs the epilogue
//    (store / residual add / SwiGLU / RoPE + KV append / arg-max).  No warp ever waits for another one except through the ring.
// What bounds it: a launch that streams, HBM and the dot products alike (gate/up of an 8B model, 66 MB, with the RMSNorm ahead of it: 13.6 us);
// every launch carries 3 us that no byte moves in - the input vector from L2, its packing, the B operands, the first tile's products and the
// last tile's epilogue, one after the other - which is most of a short one (4096 x 4096 Q4_K, 9.4 MB: 4.3 us).  Byte dot products on
// lanes that each own 64 columns, one producer and one epilogue warp: 15.5 and 5.8 us; there a tile took about 0.9 us whatever its size
// (a producer's or an epilogue's latency per tile), and the dot products as long as HBM.
// A launch starts with its code and its parameters in no near cache, so what it runs first is kept short: the split is multiplications by
// constants of the host, the producers make their own barriers ready and copy without meeting the other warps, every line of the
// parameters is touched by another warp at once, and what only some launches do (arg-max, the ranks' exchange) lies out of the way.  From
// a CTA's start to its first copy 1.1 us instead of 1.8-2.2, and decoding 21.4 instead of 23.2 ms per 16 tokens of an 8B model, 13.1 instead of
// 14.4 ms per 32 of a 1B model.
// Every wait on an mbarrier is bounded; a wait that gives up raises the context's error word and carries on.
#include "gemv_stream.cuh"

#include <stdlib.h>

namespace ib {


struct StreamGeom {
    ShareGeom share;       // the pipelines' byte-balanced ranges
    uint32_t nseg;         // 1 where gate and up rows travel together
    uint32_t stages, stage_bytes, act_off, part_off, bar_off;
    // the launch's tiles in hand-out order: per segment the pairs, the pairs per tile and the bytes per pair
    uint32_t seg_pairs[3], seg_pt[3], seg_cost[3], meta_off;
    uint32_t NB, CG, RG, mode;   // see Split
    uint32_t P;            // pipelines
    uint32_t ahead;        // stages: how far the first round of copies runs ahead of their arrival
    uint32_t width_log2;   // lanes of the epilogue warp: groups of so many (log2) pairs share the addition of the pairs' partial sums
    uint32_t cg_inv;       // 2^16 / CG, rounded up
    uint32_t unit;   // tiles are claimed from a counter, so many at a time; 0: every CTA streams its own byte-balanced range of pairs
    uint32_t head;   // counter hand-out: so many tiles of every pipeline are its own by position
};

// Counter hand-out (one segment only): tile number -> (segment 0, first pair, pairs); pairs == 0 past the last tile.
__device__ __forceinline__ uint4 tile_of(const StreamGeom &g, uint32_t t) {
    const uint32_t np = g.seg_pairs[0], pt = g.seg_pt[0], first = t * pt;
    if (first >= np) return make_uint4(0, 0, 0, 0);
    return make_uint4(0, first, (np - first) < pt ? (np - first) : pt, 0);
}

// ---- consumer side ----
struct Consumer {
    uint32_t ring;        // shared address of the ring
    uint32_t part;        // shared address of this column group's partial sums of the first stage
    uint32_t meta;        // shared address of [stages] (segment, first pair, pairs, -) descriptors written by the producer
    uint32_t bar0, S, stage_bytes;
    uint32_t zeros;            // shared address of 16 zero bytes
    uint32_t stream, RG, pt;   // the stream's stages: stream, stream + RG, ... < S; pairs per tile
    uint32_t blk, nb;          // the warp's first block of 256 columns, blocks
    uint32_t stride;           // bytes of a row
    int lane;
};

// Partial sums of a stage: [column group][2 * pair + row of the pair], so that the epilogue warp's lanes (one pair each) read
// consecutive pairs of words.
constexpr uint32_t PART_STAGE_FLOATS = 2 * CW * PT_MAX;

// A consumer warp.  The tiles of a CTA go round-robin to RG streams of CG warps each, so that the streams' waits, loads and
// reductions overlap.  Per tile a warp waits for the weights, leaves its columns' part of every row sum in the stage's partial
// block, 8 rows at a time, and arrives on the stage's "done" barrier.  It never waits for another consumer warp: adding up the
// column groups and everything that follows is the epilogue warp's work.
template <uint32_t QT, uint32_t MODE>
__device__ __forceinline__ void consume_tiles(const GemvParams &p, const Consumer &c, const Act &A) {
    const uint32_t g = c.lane >> 2, t = c.lane & 3, stride = c.stride;
    using F = Frag<QT>;
    LaneConst lc;
    constexpr bool FOUR = MODE == ROWS4;
    constexpr uint32_t NB = MODE == ROWS8 ? 2 : NB_MAX;
    uint32_t B[NB][8];
    UnitAct ua[2];
    const bool swiglu = p.epi == EPI_SWIGLU;   // a "pair" is gate row r + up row r: 4 gate rows, then their 4 up rows, at a time
    const uint32_t act = smem_u32(A.base), sc0 = act + ACT_LIMBS * A.cols, sx0 = sc0 + A.cols / 8;
    // The lane's activations go into registers in the order of the format's B operand before the first tile is waited for: the copy of that
    // tile and this load overlap.
    lc.sc = sc0;
    lc.sx = sx0;
    F::template init<FOUR>(g, t, stride, c.blk, lc);
    // (the same value, so told that it can be had again from the other one: a register that long rows spill otherwise, 4096 x 6144 6.60 us, 6.33 so)
    if constexpr (QT == IB_Q5_K && (MODE == ROWS8_LONG || MODE == ROWS8_PAIR)) lc.h1 = lc.h0 ^ 4u;
#pragma unroll
    for (uint32_t i = 0; i < NB; i++) {
        if (i < c.nb) F::operand(FOUR && (i & 1) ? g ^ 4 : g, t, act + (g & 1) * A.cols, c.zeros, c.blk + i, B[i]);
        else
            for (int k = 0; k < 8; k++) B[i][k] = 0;
    }
    if (MODE == ROWS8) {
        F::template unit<FOUR>(lc, 0, ua[0]);
        if (c.nb == 2) F::template unit<FOUR>(lc, 1, ua[1]);
    }
    constexpr bool PAIR = MODE == ROWS8_PAIR;
    constexpr uint32_t together = FOUR || PAIR ? 4 : 8, half = together / 2;   // rows of a tile at a time; gate/up: gate rows, then their up rows
    const uint32_t add = swiglu ? half : together, row_of = g & (add - 1), b_off = swiglu && (g & half) ? c.pt * stride : 0;   // the up rows follow a full tile's gate rows
    const uint32_t part0 = c.part + 4 * (swiglu ? 2 * row_of + ((g & half) ? 1 : 0) : row_of), out_step = 4 * together;
    const bool writer = t == 0 && (PAIR || g < together);
    uint32_t st = c.stream, par = 0, ring = c.ring;   // ring: address of stage st
    // a row's up to four blocks: straight-line code where they are four, so that the blocks' loads and products overlap
    auto long_dot = [&](uint32_t row) {
        float v = 0.f;
        if (c.nb == NB_MAX) {
#pragma unroll
            for (uint32_t i = 0; i < NB_MAX; i++) {
                F::template unit<false>(lc, i, ua[i & 1]);
                v += F::template dot<false>(row, lc, i, B[i & (NB - 1)], B[i & (NB - 1)], ua[i & 1]);
            }
        } else {
#pragma unroll
            for (uint32_t i = 0; i < NB_MAX - 1; i++)
                if (i < c.nb) {
                    F::template unit<false>(lc, i, ua[0]);
                    v += F::template dot<false>(row, lc, i, B[i & (NB - 1)], B[i & (NB - 1)], ua[0]);
                }
        }
        return v;
    };
    auto next_stage = [&]() {
        st += c.RG;
        ring += c.stage_bytes;
        if (st >= c.S) {
            st = c.stream;
            ring = c.ring;
            par ^= 1u;
        }
    };
#pragma unroll 1
    for (;;) {
        if (!mbar_wait(c.bar0 + 8 * st, par, p.err, 1, p.wait_ns)) return;   // the error word is raised; give up on this CTA's rows
        const uint4 tm = lds128(c.meta + 16 * st);
        const uint32_t n = tm.z;
        if (n == 0) {   // no tiles left
            if (c.lane == 0) mbar_arrive(c.bar0 + 8 * (2 * c.S + st));
            break;
        }
        if constexpr (PAIR) {
            // Two tiles of 4 rows as 8 rows: the lower lanes' rows are this tile's, the upper ones' the next one's, which may be the end.  The ring
            // keeps its four stages (and HBM its pace: with two tiles of 8 rows both land together).
            const uint32_t st_a = st, ring_a = ring;
            next_stage();
            if (!mbar_wait(c.bar0 + 8 * st, par, p.err, 1, p.wait_ns)) return;
            const uint32_t n_b = lds128(c.meta + 16 * st).z;
            const bool b = (g & 4) && n_b;
            const uint32_t rows = swiglu ? (b ? n_b : n) : 2 * (b ? n_b : n), row = (b ? ring : ring_a) + b_off + (row_of < rows ? row_of : rows - 1) * stride;
            float v = long_dot(row);
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            if (writer) asm volatile("st.shared.f32 [%0], %1;" ::"r"(part0 + (g & 4 ? st : st_a) * (4 * PART_STAGE_FLOATS)), "f"(v) : "memory");
            __syncwarp();
            if (c.lane < 2) mbar_arrive(c.bar0 + 8 * (2 * c.S + (c.lane ? st : st_a)));
            if (n_b == 0) break;
            next_stage();
            continue;
        }
        const uint32_t base = ring + b_off, rows = swiglu ? n : 2 * n;
        uint32_t out = part0 + st * (4 * PART_STAGE_FLOATS);
        for (uint32_t r = row_of, first = 0; first < rows; first += add, r += add, out += out_step) {
            // rows past the tile's last one repeat it: what they give is not used
            const uint32_t row = base + (r < rows ? r : rows - 1) * stride;
            float v = 0.f;
            // straight-line code: the steps' loads and products overlap
            if constexpr (FOUR) {
                // `lc.first` differs between formats (swap_stretches).  Where it does not hold, the lane's units are in the second
                // block of a step, which the last step may lack.
                F::template unit<true>(lc, 0, ua[0]);
                v = F::template dot<true>(row, lc, 0, B[0], B[1], ua[0]);
                if (c.nb == 1 && !lc.first) v = 0.f;
                if (c.nb > 2) {
                    F::template unit<true>(lc, 1, ua[1]);
                    const float y = F::template dot<true>(row, lc, 1, B[2], B[3], ua[1]);
                    v += c.nb == 3 && !lc.first ? 0.f : y;
                }
            } else if constexpr (MODE == ROWS8_LONG) {
                v = long_dot(row);
            } else {
                v = F::template dot<false>(row, lc, 0, B[0], B[0], ua[0]);
                if (c.nb == 2) v += F::template dot<false>(row, lc, 1, B[1], B[1], ua[1]);
            }
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            v += __shfl_xor_sync(0xffffffffu, v, 2);
            if (FOUR) v += __shfl_xor_sync(0xffffffffu, v, 16);
            if (writer) asm volatile("st.shared.f32 [%0], %1;" ::"r"(out), "f"(v) : "memory");
        }
        __syncwarp();   // the lanes' partials are ordered before lane 0's arrival (a release)
        if (c.lane == 0) mbar_arrive(c.bar0 + 8 * (2 * c.S + st));   // this warp is done with the stage: weights read, partials left
        next_stage();
    }
}

// The epilogue warp: per tile it waits until every consumer warp has left its partials, adds up the column groups in a
// fixed order (bitwise deterministic results), hands the stage back to the producer and runs the epilogue of the tile's
// row pairs, one pair per lane.
__device__ __forceinline__ void finish_tiles(const GemvParams &p, const StreamGeom &geo, uint32_t part, uint32_t meta, uint32_t bar0, uint32_t pipe,
                                             uint32_t lane, const float *red, unsigned long long &best) {
    const uint32_t S = geo.stages, CG = geo.CG, width = 1u << geo.width_log2, slices = 32u >> geo.width_log2;   // lanes: `slices` groups of `width` pairs
    const uint32_t pr = lane & (width - 1), slice = lane >> geo.width_log2;
    uint32_t st = pipe, par = 0;
    float rms = 1.0f;
    if (p.norm_w) {
        // RMSNorm factor of the input vector (crates/inferi-shaders/src/rms_norm.rs:112-120): the consumer warps left
        // their parts of the sum of squares in `red`; added in a fixed order
        if (!mbar_wait(bar0 + 8 * (3 * S), 0, p.err, 6, p.wait_ns)) return;
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < PACK_THREADS / 32; w++) t += red[w];
        rms = 1.0f / sqrtf(t / (float)p.cols + p.eps);
    }
    const bool reads = p.epi == EPI_RESIDUAL || p.epi == EPI_QKV;
    const uint32_t pos = p.epi == EPI_QKV ? __ldcg(p.pos_ptr) : 0u;
#pragma unroll 1
    for (;;) {
        // what the epilogue reads is requested before the wait for the dot products: the L2 round trip overlaps it
        float2 pre = make_float2(0.f, 0.f);
        if (reads) {
            if (!mbar_wait(bar0 + 8 * st, par, p.err, 1, p.wait_ns)) return;
            const uint4 tm = lds128(meta + 16 * st);
            if (lane < tm.z) pre = epilogue_prefetch(p, tm.x, tm.y + lane);
        }
        if (!mbar_wait(bar0 + 8 * (2 * S + st), par, p.err, 5, p.wait_ns)) return;   // (implies the tile's announcement)
        const uint4 tm = lds128(meta + 16 * st);
        const uint32_t s = tm.x, first_pair = tm.y, n = tm.z;
        if (n == 0) break;
        const bool mine = lane < n;
        float va = 0.f, vb = 0.f;
        const uint32_t at = part + 4 * (st * PART_STAGE_FLOATS + 2 * pr);
#pragma unroll 2
        for (uint32_t g = slice; g < CG; g += slices) {
            const uint2 v = lds64(at + 4 * (g * 2 * PT_MAX));
            va += __uint_as_float(v.x);
            vb += __uint_as_float(v.y);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(bar0 + 8 * (S + st));   // partials read: the producer may refill the stage
#pragma unroll
        for (uint32_t o = 16; o; o >>= 1)
            if (o >= width) {
                va += __shfl_xor_sync(0xffffffffu, va, o);
                vb += __shfl_xor_sync(0xffffffffu, vb, o);
            }
        if (mine) epilogue(p, s, first_pair + lane, va * rms, vb * rms, best, pre, pos);
        st += geo.P;
        if (st >= S) {
            st = pipe;
            par ^= 1u;
        }
    }
}

// Tensor parallel: the previous row-split GEMV of every rank leaves its partial sums in this rank's slots.  The sum (x + the partials
// in rank order, so every rank gets the same bits) is formed once per rank: an epilogue warp adds up the groups of 32 columns that
// fall to its CTA and stores them as the new residual stream; the consumer warps of all CTAs wait until every group is there.  (Each
// CTA adding up the whole vector for itself was N x 16 KiB of L2 reads per CTA: at 8 ranks more than its share of the weights.)
__device__ __noinline__ void reduce_partials(const GemvParams &p, uint32_t lane) {
    const uint32_t tag = (*p.epoch_ptr) * p.xchg_per_epoch + p.reduce_use;
    uint32_t cnt = 0;
#pragma unroll 1
    for (uint32_t grp = blockIdx.x; grp < p.cols / 32; grp += gridDim.x) {
        const uint32_t col = grp * 32 + lane;
        float v = __ldcg(p.x + col);
        // on a time-out the error word is raised and the launch runs to its end on whatever is there
#pragma unroll 1
        for (uint32_t rk = 0; rk < p.tp; rk++) v += wait_tagged(p.reduce_src + (size_t)rk * p.cols + col, tag, p.err, p.wait_ns);
        p.x_out[col] = v;
        cnt++;
    }
    __threadfence();
    __syncwarp();
    if (lane == 0 && cnt) asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p.reduce_done), "r"(cnt) : "memory");
}

// EPI_ARGMAX: `best` of an epilogue warp's lanes becomes its pipeline's candidate; the last of the launch's `slots` pipelines to arrive
// folds all of them (none waits for another).
__device__ __noinline__ void finish_argmax(const GemvParams &p, unsigned long long best, uint32_t slot, uint32_t slots, uint32_t lane) {
#pragma unroll 1
    for (int o = 16; o; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    uint32_t last = 0;
    if (lane == 0) {
        p.argmax_slots[slot] = best;
        __threadfence();
        last = (atomicAdd(p.argmax_counter, 1u) == slots - 1) ? 1u : 0u;
    }
    last = __shfl_sync(0xffffffffu, last, 0);
    if (!last) return;
    __threadfence();
    unsigned long long b = 0ull;
    for (uint32_t i = lane; i < slots; i += 32) b = max(b, __ldcg(p.argmax_slots + i));
#pragma unroll 1
    for (int o = 16; o; o >>= 1) b = max(b, __shfl_xor_sync(0xffffffffu, b, o));
    if (lane == 0) {
        *p.argmax_out = 0xFFFFFFFFu - (uint32_t)(b & 0xFFFFFFFFull);
        *p.argmax_counter = 0u;
        if (p.tp > 1) {
            // sharded vocabulary: every rank gets this rank's candidate; the end-of-token kernel folds them
#pragma unroll 1
            for (uint32_t rk = 0; rk < p.tp; rk++) *p.amax_dst[rk] = b;
            __threadfence_system();
#pragma unroll 1
            for (uint32_t rk = 0; rk < p.tp; rk++) atomicAdd_system(p.amax_flag[rk], 1u);
        }
    }
}

// One 4-byte word of every 64 bytes of the launch's parameters, each by another consumer warp: a launch's parameters are in no cache when it
// starts, and a warp that comes to them one after the other waits for every line.
__device__ __forceinline__ void touch_parameters(const GemvParams &p, const StreamGeom &geo, uint32_t warp) {
    constexpr uint32_t LP = (sizeof(GemvParams) + 63) / 64, LG = (sizeof(StreamGeom) + 63) / 64;
    static_assert(LP + LG <= CW, "a consumer warp per line (the producers do not come here)");
    uint32_t v = 0;
    if (warp < LP) v = reinterpret_cast<const uint32_t *>(&p)[16 * warp];
    else if (warp < LP + LG) v = reinterpret_cast<const uint32_t *>(&geo)[16 * (warp - LP)];
    asm volatile("" ::"r"(v));
}

// ---- the kernel ----
// Shared-memory barriers: full[S] (the producer's expect_tx arrival + the copy's bytes), empty[S] (one arrival: the
// epilogue warp has read the stage's partials, which implies that every consumer warp is done with its weights),
// done[S] (one arrival per consumer warp of the tile's stream), ss (one arrival per consumer warp: its part of the input's sum of squares).
// One instance per weight format (and one for launches that mix them); what the launch does with the row sums is a run-time switch in the
// epilogue warp, so that the launches of a token graph share their code.
template <uint32_t QT, uint32_t MODE>
__global__ void __launch_bounds__(STREAM_THREADS, 1) gemv_stream_kernel(const __grid_constant__ GemvParams p, const __grid_constant__ StreamGeom geo) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float red[PACK_THREADS / 32 + 1];
    __shared__ uint4 zeros;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int BAR_START = 2;   // named barrier: the mbarriers are ready

    uint8_t *act_sm = smem + geo.act_off;
    const uint32_t part = smem_u32(smem + geo.part_off);                        // [stages][CW][2 * PT_MAX] floats
    const uint32_t bar0 = smem_u32(smem + geo.bar_off);                         // full[stages], empty[stages], done[stages]
    const uint32_t S = geo.stages;
    const uint32_t CG = geo.CG, RG = geo.RG, active = CG * RG;   // consumer warps with work

    if (warp >= W_PRODUCER && warp < W_EPILOGUE) {
        // A pipeline's producer makes its stages' barriers ready and goes on to its first copies; the other warps wait for both producers.
        if ((uint32_t)lane < S && (lane & (geo.P - 1)) == warp - W_PRODUCER) {
            mbar_init(bar0 + 8 * lane, 1);
            mbar_init(bar0 + 8 * (S + lane), 1);
            mbar_init(bar0 + 8 * (2 * S + lane), CG);
        }
        if (lane == 31 && warp == W_PRODUCER) mbar_init(bar0 + 8 * (3 * S), CW);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        __syncwarp();
        asm volatile("bar.arrive %0, %1;" ::"r"(BAR_START), "r"(STREAM_THREADS) : "memory");
        // ================= producer warp: picks tiles and streams them =================
        // With many tiles per CTA they are handed out through a counter in global memory, so that a CTA which starts late
        // (its SM was the last to be freed by the previous kernel) or runs slowly takes fewer of them.  With few tiles per
        // CTA a tile is too coarse a unit for that: every pipeline then streams its own byte-balanced range of row pairs, cut
        // into tiles.  Either way the slot's descriptor tells the other warps what the tile is.  One lane picks, waits for
        // the slot, announces the tile and issues its bulk copies.
        // A tile costs this lane 0.4-0.7 us, most of it between issuing a copy and being able to prepare the next one, and a
        // claim another 0.6: with one producer per SM that, not HBM, was the pace of the launches that stream.  Hence two pipelines.
        const uint32_t pipe = warp - W_PRODUCER;
        if (pipe >= geo.P || lane != 0) return;
        uint4 *meta = reinterpret_cast<uint4 *>(smem + geo.meta_off);
        const bool dyn = geo.unit != 0, swiglu = p.epi == EPI_SWIGLU;
        const uint32_t pipes = gridDim.x * geo.P, me = blockIdx.x * geo.P + pipe;
        Share sh;
        TileCursor tc;
        // counter hand-out: a pipeline's first tiles are its own by position (no round trip before the first copy), every
        // later unit of tiles is claimed
        uint32_t held = 0, t = 0;
        if (dyn) {
            held = geo.head;
            t = me * held;
        } else {
            uint64_t scale = geo.share.scale[0];
            uint32_t base = 0, number = me;
            if constexpr (QT == QT_MIXED) {   // (one format, one group)
                const uint32_t group = share_group(geo.share, blockIdx.x);
                scale = geo.share.scale[group];
                base = geo.share.base[group];
                number -= geo.share.cta0[group] * geo.P;
            }
            make_share(geo.share, geo.seg_pairs, geo.seg_pt, geo.nseg, scale, base, number, sh);
            tc.init(sh);
        }
        uint32_t cost = swiglu ? (uint32_t)p.seg[0].row_bytes : geo.seg_cost[0], cost_b = (uint32_t)p.seg[1].row_bytes, cur = 0;
        const uint8_t *w = p.seg[0].w, *wb = p.seg[1].w;
        // The weights of a token pass through L2 once; as the first to be evicted they leave the rest of it - the code of the token's
        // other kernels, the cache, the activations - in place (attention in the first layer of a token, after the classifier's
        // hundreds of megabytes: 13.5 us instead of 5).
        const uint64_t policy = evict_first_policy();
        uint32_t st = pipe, ring = smem_u32(smem), par = 1, ends = 0;   // par: parity of the slot's previous use ("1" before the first one); ends: end markers, one per stream
        bool first_round = true, gave_up = false;
        for (;;) {
            uint4 tm = make_uint4(0, 0, 0, 0);
            if (dyn) {
                if (held == 0) {
                    t = geo.head * pipes + geo.unit * atomicAdd(p.tile_claim, 1u);
                    held = geo.unit;
                }
                tm = tile_of(geo, t);
            } else if (tc.valid(sh)) tm = make_uint4(tc.seg, tc.next, tc.count(sh), 0);
            const uint32_t n = tm.z, full = bar0 + 8 * st;
            // Slot free?  In the first round every slot is; there the copies in flight are kept to what the memory system's latency
            // needs: a ring-full of them would only queue up, and the input vector's few kilobytes behind them.
            if (!first_round ? !mbar_wait(bar0 + 8 * (S + st), par, p.err, 2, p.wait_ns)
                             : (st >= geo.ahead && !mbar_wait(bar0 + 8 * (st - geo.ahead), 0, p.err, 1, p.wait_ns))) {
                gave_up = true;
                break;
            }
            meta[st] = tm;
            if (n == 0) {
                // no tiles left: tell the others, and let the last pipeline to get here clear the counters for their next use
                mbar_arrive(full);
                if (++ends == geo.RG / geo.P) break;
            } else {
                if (tm.x != cur) {
                    cur = tm.x;
                    cost = cur == 1 ? geo.seg_cost[1] : geo.seg_cost[2];
                    w = cur == 1 ? p.seg[1].w : p.seg[2].w;
                }
                if (!first_round) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // the consumers' reads of the slot come first
                const uint32_t ba = n * cost, bb = swiglu ? n * cost_b : 0u, dst = ring + st * geo.stage_bytes;
                mbar_expect_tx(full, ba + bb);
                bulk_g2s(dst, w + (size_t)tm.y * cost, ba, full, policy);
                if (swiglu) bulk_g2s(dst + geo.seg_pt[0] * cost, wb + (size_t)tm.y * cost_b, bb, full, policy);
                if (!dyn) tc.advance(sh);
                else { t++; held--; }
            }
            st += geo.P;
            if (st >= S) {
                st = pipe;
                par ^= 1u;
                first_round = false;
            }
        }
        if (gave_up) {
            // The copies in flight write into this CTA's shared memory: let them land (bounded, like every wait) before the CTA can end.
            // A stage's last announcement is this round's up to `st` and the previous round's from there on.
            for (uint32_t s = pipe; s < S && (s < st || !first_round); s += geo.P) mbar_wait(bar0 + 8 * s, s < st ? par ^ 1u : par, nullptr, 1, p.wait_ns);
        }
        // Every pipeline gets here, one that gave up too: a launch that ended early must not leave counts behind for the next one that
        // is given these counters.
        if (dyn && atomicAdd(p.tile_claim + 1, 1u) == pipes - 1) {
            p.tile_claim[0] = 0u;
            p.tile_claim[1] = 0u;
        }
        return;
    }

    touch_parameters(p, geo, warp);
    if (threadIdx.x == 0) zeros = make_uint4(0, 0, 0, 0);
    named_barrier(BAR_START, STREAM_THREADS);

    if (warp >= W_EPILOGUE) {
        // ================= epilogue warp =================
        if (p.pdl) asm volatile("griddepcontrol.launch_dependents;");
        const uint32_t pipe = warp - W_EPILOGUE;
        if (pipe >= geo.P) return;
        // outputs (and the residual it reads) are touched by the previous kernels of the stream: wait for them like the consumers do
        if (p.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");
        if (p.reduce_src && pipe == 0) reduce_partials(p, lane);
        unsigned long long best = 0ull;
        finish_tiles(p, geo, part, smem_u32(smem + geo.meta_off), bar0, pipe, lane, red, best);
        if (p.epi == EPI_ARGMAX) finish_argmax(p, best, blockIdx.x * geo.P + pipe, gridDim.x * geo.P, lane);
        return;
    }

    // ================= consumer warps =================
    Consumer c;
    const uint32_t stream = (warp * geo.cg_inv) >> 16, cg = warp - stream * CG, blocks = p.cols / 256;
    c.zeros = smem_u32(&zeros); c.meta = smem_u32(smem + geo.meta_off); c.bar0 = bar0; c.S = S; c.lane = lane;
    c.part = part + 4 * (cg * 2 * PT_MAX);
    c.stream = stream; c.RG = RG; c.pt = geo.seg_pt[0];
    c.ring = smem_u32(smem) + stream * geo.stage_bytes;
    c.stage_bytes = geo.stage_bytes * RG;   // from one of the stream's stages to the next
    c.blk = cg * geo.NB;
    c.nb = blocks - c.blk < geo.NB ? blocks - c.blk : geo.NB;
    const uint32_t seg0 = QT == QT_MIXED ? geo.share.seg0[share_group(geo.share, blockIdx.x)] : 0;
    c.stride = (uint32_t)p.seg[seg0].row_bytes;
    const Act A{act_sm, p.cols};
    float4 norm_g[2];
    pack_prefetch_norm8(p.norm_w, p.cols, norm_g);   // weights: fetched while the previous kernel is still running
    if (p.pdl) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (p.reduce_src) {
        // tensor parallel: the reduced residual stream is complete once the epilogue warps of all CTAs have stored their groups
        if (threadIdx.x == 0) wait_counter_gpu(p.reduce_done, ((*p.epoch_ptr) * p.xchg_per_epoch + p.reduce_use) * (p.cols / 32), p.err, 7, p.wait_ns);
        named_barrier(1, PACK_THREADS);
    }
    pack_stream<MODE == ROWS8 ? 1 : 4>(act_sm, p.cols, p.reduce_src ? p.x_out : p.x, p.norm_w, red, bar0 + 8 * (3 * S), norm_g);
    if ((uint32_t)warp >= active) return;
    if constexpr (QT != QT_MIXED) consume_tiles<QT, MODE>(p, c, A);
    else
        switch (p.seg[seg0].qtype) {   // of all the CTA's tiles
        case IB_Q4_K: consume_tiles<IB_Q4_K, MODE>(p, c, A); break;
        case IB_Q6_K: consume_tiles<IB_Q6_K, MODE>(p, c, A); break;
        case IB_Q5_K: consume_tiles<IB_Q5_K, MODE>(p, c, A); break;
        default: consume_tiles<IB_Q8_0, MODE>(p, c, A); break;
        }
}

// -------------------------------------------------------------------------------------------------
// host side
// -------------------------------------------------------------------------------------------------
// AHEAD_BYTES: about HBM's latency times an SM's share of its rate; with the ring-full in flight a Q8_0 4096 x 4096 launch takes 5.7 us
// instead of 5.3.  TILE_BYTES: a tile's fixed costs (waits, operands' latency, epilogue) spread over so much; gate/up of a 1B model
// 6.6 us at half of it.
constexpr uint32_t AHEAD_BYTES = 73728;
constexpr uint32_t TILE_BYTES = 40960, UNIT_BYTES = 40960, MIN_STAGES = 3, MAX_STAGES = 12;
constexpr size_t STREAM_SMEM_BUDGET = 226 * 1024;   // one CTA per SM

bool gemv_stream_eligible(const GemvParams &p) {
    if (p.cols % 256 || p.cols > 256 * NB_MAX * CW) return false;
    for (uint32_t s = 0; s < p.nseg; s++) {
        const uint32_t q = p.seg[s].qtype;
        if (q != IB_Q4_K && q != IB_Q5_K && q != IB_Q6_K && q != IB_Q8_0) return false;
        if (p.seg[s].row_bytes % 16) return false;
    }
    return true;
}

template <uint32_t QT, uint32_t MODE>
static int32_t launch_stream_rows(ib_ctx *ctx, cudaStream_t stream, const GemvParams &p, int grid, const StreamGeom &geo, size_t smem) {
    static bool attr_set[16] = {false};
    if (!attr_set[ctx->device & 15]) {
        IB_CHECK_CUDA(cudaFuncSetAttribute(gemv_stream_kernel<QT, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STREAM_SMEM_BUDGET));
        attr_set[ctx->device & 15] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(STREAM_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.pdl ? 1 : 0;
    IB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, gemv_stream_kernel<QT, MODE>, p, geo));
    ctx->launches++;
    return IB_OK;
}

template <uint32_t QT>
static int32_t launch_stream_inst(ib_ctx *ctx, cudaStream_t stream, const GemvParams &p, int grid, const StreamGeom &geo, size_t smem) {
    switch (geo.mode) {
    case ROWS4: return launch_stream_rows<QT, ROWS4>(ctx, stream, p, grid, geo, smem);
    case ROWS8_PAIR: return launch_stream_rows<QT, ROWS8_PAIR>(ctx, stream, p, grid, geo, smem);
    case ROWS8_LONG: return launch_stream_rows<QT, ROWS8_LONG>(ctx, stream, p, grid, geo, smem);
    default: return launch_stream_rows<QT, ROWS8>(ctx, stream, p, grid, geo, smem);
    }
}

// Which instance serves a launch: the one of its format, or the one whose CTAs each take the path of their own.
static int32_t launch_stream_format(ib_ctx *ctx, cudaStream_t stream, const GemvParams &p, int grid, const StreamGeom &geo, size_t smem) {
    uint32_t qt = p.seg[0].qtype;
    for (uint32_t s = 0; s < p.nseg; s++)
        if (p.seg[s].qtype != qt) qt = QT_MIXED;
    switch (qt) {
    case IB_Q4_K: return launch_stream_inst<IB_Q4_K>(ctx, stream, p, grid, geo, smem);
    case IB_Q6_K: return launch_stream_inst<IB_Q6_K>(ctx, stream, p, grid, geo, smem);
    case IB_Q5_K: return launch_stream_inst<IB_Q5_K>(ctx, stream, p, grid, geo, smem);
    case IB_Q8_0: return launch_stream_inst<IB_Q8_0>(ctx, stream, p, grid, geo, smem);
    default: return launch_stream_inst<QT_MIXED>(ctx, stream, p, grid, geo, smem);
    }
}

// The CTAs of every group of segments of one format (ShareGeom), in proportion to its bytes; a group has a CTA at least (every segment has
// two row pairs, so the grid has a CTA for each).
static void deal_ctas(ShareGeom &g, const GemvParams &p, uint32_t nseg, const uint32_t (&pairs)[3], uint32_t total16, uint32_t grid, uint32_t P) {
    uint32_t n = 0, bytes[3] = {0, 0, 0}, ctas[3] = {0, 0, 0}, used = 0;
    for (uint32_t s = 0; s < nseg; s++) {
        if (s == 0 || p.seg[s].qtype != p.seg[s - 1].qtype) {
            g.seg0[n] = s;
            g.base[n++] = g.start[s];
        }
        bytes[n - 1] += pairs[s] * g.cost16[s];
    }
    for (uint32_t i = 0; i < n; i++) {
        ctas[i] = (uint32_t)((uint64_t)bytes[i] * grid / total16);
        if (ctas[i] < 1) ctas[i] = 1;
        used += ctas[i];
    }
    // rounded down: to the group whose CTAs have most; a group that was given its one CTA: from the group that misses it least
    for (; used != grid; used += used < grid ? 1 : -1) {
        uint32_t best = 0;
        for (uint32_t i = 1; i < n; i++) {
            if (used < grid ? (uint64_t)bytes[i] * ctas[best] > (uint64_t)bytes[best] * ctas[i]
                            : ctas[best] < 2 || (ctas[i] > 1 && (uint64_t)bytes[i] * (ctas[best] - 1) < (uint64_t)bytes[best] * (ctas[i] - 1)))
                best = i;
        }
        ctas[best] += used < grid ? 1 : -1;
    }
    uint32_t at = 0;
    for (uint32_t i = 0; i < 3; i++) {
        g.cta0[i] = i < n ? at : 0xFFFFFFFFu;
        if (i >= n) {
            g.scale[i] = 0;
            g.base[i] = g.seg0[i] = 0;
            continue;
        }
        const uint32_t pipes = ctas[i] * P;
        g.scale[i] = (((uint64_t)bytes[i] << 32) + pipes - 1) / pipes;
        at += ctas[i];
    }
}

int32_t launch_gemv_stream(ib_ctx *ctx, cudaStream_t stream, const GemvParams &p) {
    uint32_t max_cost = 0, pairs = 0;
    if (p.epi == EPI_SWIGLU) {
        max_cost = (uint32_t)(p.seg[0].row_bytes + p.seg[1].row_bytes);
        pairs = p.seg[0].rows;
    } else {
        for (uint32_t s = 0; s < p.nseg; s++) {
            const uint32_t c = (uint32_t)(2 * p.seg[s].row_bytes);
            if (c > max_cost) max_cost = c;
            pairs += p.seg[s].rows / 2;
        }
    }
    // Tile = whole groups of 8 (4) rows: as many as fit TILE_BYTES and no more than a third of the ring, and at most about a stream's
    // share of the launch - one tile of it rather than two (4096 x 4096 Q4_K 4.77 -> 4.61 us, 3072 x 2048 4.05 -> 3.70).  As many stages as fit beside the activations.
    int grid = ctx->sm_count;       // one persistent CTA per SM
    if ((uint32_t)grid > pairs) grid = (int)pairs;
    if (grid < 1) grid = 1;
    const size_t act = (act_smem_bytes(p.cols) + 127) & ~(size_t)127;
    const size_t per_stage = PART_STAGE_FLOATS * 4 + 3 * 8 + 16;   // partials, barriers, tile descriptor
    const size_t room = STREAM_SMEM_BUDGET - act - 256;
    const uint32_t max_stage = (uint32_t)(room / MIN_STAGES - per_stage) & ~127u;
    Split split = split_of(p.cols, 4 * max_cost <= max_stage);
    if (max_cost > max_stage)
        return set_error(IB_ERR_UNSUPPORTED, "gemv: a row pair of %u bytes with %u columns does not fit the streaming kernel's ring", max_cost, p.cols);
    auto pairs_per_tile = [&](uint32_t cost) {
        uint32_t pt = split.mode == ROWS4 ? 2 : 4;
        while (pt * 2 <= PT_MAX && pt * 2 * cost <= TILE_BYTES && pt * (uint32_t)grid * split.RG < pairs) pt *= 2;
        while (pt > 1 && pt * cost > max_stage) pt--;
        return pt;
    };
    StreamGeom geo;
    uint32_t stage_data = 0, tiles = 0, most_pt = 0;
    for (uint32_t s = 0; s < 3; s++) {
        geo.seg_pairs[s] = 0;
        geo.seg_pt[s] = 1;
        geo.seg_cost[s] = 16;
        const bool swiglu = p.epi == EPI_SWIGLU;
        if (s >= (swiglu ? 1u : p.nseg)) continue;
        const uint32_t cost = swiglu ? max_cost : (uint32_t)(2 * p.seg[s].row_bytes);
        const uint32_t pt = pairs_per_tile(cost);
        geo.seg_cost[s] = cost;
        geo.seg_pt[s] = pt;
        geo.seg_pairs[s] = swiglu ? p.seg[0].rows : p.seg[s].rows / 2;
        tiles += (geo.seg_pairs[s] + pt - 1) / pt;
        if (pt * cost > stage_data) stage_data = pt * cost;
        if (pt > most_pt) most_pt = pt;
    }
    uint32_t total16 = 0;
    for (uint32_t s = 0; s < 3; s++) {
        geo.share.start[s] = total16;
        geo.share.cost16[s] = geo.seg_cost[s] / 16;
        geo.share.inv[s] = (uint32_t)(0xFFFFFFFFull / geo.share.cost16[s] + 1);
        total16 += geo.seg_pairs[s] * geo.share.cost16[s];
    }
    geo.nseg = p.epi == EPI_SWIGLU ? 1u : p.nseg;
    geo.stage_bytes = (stage_data + 127) & ~127u;
    uint32_t S = (uint32_t)(room / (geo.stage_bytes + per_stage));
    if (S > MAX_STAGES) S = MAX_STAGES;
    // A stage always serves the same stream: the barriers' parities only order uses that one and the same warp waits for.
    while (split.RG > S) split.RG /= 2;
    S -= S % split.RG;
    // Two tiles at a time: where CTAs have more of them than that takes to pay.  us, one / two at a time: Q4_K of 14336 columns, 592 rows (a tile per CTA)
    // 4.84 / 4.99, 800 5.68 / 5.60, 2000 7.82 / 7.15; Q5_K of 12288, 592 rows 4.52 / 5.09, 1500 6.67 / 6.77, 2000 (3.4 tiles per CTA) 7.77 / 7.45; Q6_K of
    // 10240, 1180 5.28 / 5.49, 2000 7.07 / 6.94.  Q8_0, which has the fewest instructions per byte, waits for a second tile in vain: 8704 columns, 800 rows
    // 4.57 / 5.17, 2960 7.75 / 8.64.
    bool q4_k = true, q8_0 = false;
    for (uint32_t s = 0; s < p.nseg; s++) {
        q4_k = q4_k && p.seg[s].qtype == IB_Q4_K;
        q8_0 = q8_0 || p.seg[s].qtype == IB_Q8_0;
    }
    const bool pays = !q8_0 && tiles > (q4_k ? 1 : 3) * (uint32_t)grid;
    if (split.mode == ROWS4 && most_pt == 2 && S >= 5 * split.RG && pays) {
        split.mode = ROWS8_PAIR;
        geo.stage_bytes = stage_data;   // the rows of two tiles follow one another: eight rows then start at different banks where their stride lets them
    }
    geo.NB = split.NB;
    geo.mode = split.mode;
    geo.CG = split.CG;
    geo.RG = split.RG;
    geo.P = split.RG < (uint32_t)PIPES ? 1u : (uint32_t)PIPES;
    uint32_t most = geo.seg_pt[0] > geo.seg_pt[1] ? geo.seg_pt[0] : geo.seg_pt[1], width = 1;
    most = geo.seg_pt[2] > most ? geo.seg_pt[2] : most;
    while (width < most) width *= 2;
    geo.width_log2 = 0;
    while ((1u << geo.width_log2) < width) geo.width_log2++;
    geo.cg_inv = (65536 + split.CG - 1) / split.CG;
    deal_ctas(geo.share, p, geo.nseg, geo.seg_pairs, total16, (uint32_t)grid, geo.P);
    geo.ahead = (AHEAD_BYTES / geo.stage_bytes) / geo.P * geo.P;
    if (geo.ahead < geo.P) geo.ahead = geo.P;
    geo.stages = S;
    geo.act_off = S * geo.stage_bytes;
    geo.part_off = (uint32_t)(geo.act_off + act);
    geo.bar_off = geo.part_off + S * PART_STAGE_FLOATS * 4;
    geo.meta_off = (geo.bar_off + (3 * S + 1) * 8 + 15) & ~15u;
    const size_t total = geo.meta_off + S * 16;
    // Hand-out: launches of one segment with enough tiles per CTA give every pipeline three quarters of its share by position and let
    // the pipelines claim the rest from a counter, in units of about UNIT_BYTES (a claim takes about as long as such a unit's copy).
    // Everything else: static byte-balanced ranges.
    geo.unit = geo.head = 0;
    const bool single = p.epi == EPI_SWIGLU || p.nseg == 1;
    uint32_t unit = UNIT_BYTES / geo.stage_bytes;
    if (unit < 1) unit = 1;
    if (single && tiles >= 6 * unit * (uint32_t)grid) {
        geo.unit = unit;
        geo.head = tiles / ((uint32_t)grid * geo.P) * 3 / 4;
    }
    // the counters through which this launch's CTAs share out the tiles: consecutive launches overlap (programmatic
    // dependent launch), so they take different pairs of a small ring; the last CTA of a launch clears its pair
    GemvParams q = p;
    q.tile_claim = ctx->stream_counters + 2 * (ctx->stream_seq++ % IB_STREAM_COUNTER_PAIRS);
    IB_REQUIRE(q.epi <= EPI_PUSH, "gemv: unknown epilogue %u", q.epi);
    return launch_stream_format(ctx, stream, q, grid, geo, total);
}

}  // namespace ib
