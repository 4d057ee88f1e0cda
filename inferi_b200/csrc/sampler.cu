// On-device token sampling: temperature, softmax, multinomial and top-p (nucleus) sampling.
//
// Replaces `Sampler::sample`, `sample_mult` and `sample_topp` (crates/inferi/src/models/sampler.rs:32-130) and the CPU
// softmax they call (crates/inferi/src/ops/softmax.rs:130-143).  The reference reads all logits back and samples on the
// host with an unseeded `rand::random()`; here the logits stay on the device and the coin of a position is a pure
// function of (seed, position), so a sequence can be reproduced.
//
//   x_i = logit_i / temperature;  p_i = exp(x_i - max x) / sum          (softmax.rs:134-142)
//   multinomial: first i with coin < p_0 + ... + p_i, else n - 1         (sampler.rs:62-77)
//   top-p: candidates p_i >= (1 - topp) / (n - 1), sorted by descending p (stable: ascending index on ties), cut after
//          the first prefix whose sum exceeds topp, then first i with coin * prefix_sum < running sum (sampler.rs:84-129)
//
// The launch is ONE thread-block cluster of 16 CTAs (8 where the device cannot place 16; one CTA for small vocabularies).  Every CTA holds a contiguous
// slice of the vocabulary in shared memory; what the CTAs have to tell one another (maximum, sum, histograms) goes
// through distributed shared memory and the cluster barrier, so the whole of it is one launch without a round trip to
// L2.  The work is a few passes over some hundred KB: with one CTA those passes alone took 100 us, and the sort of the
// candidates (thousands for a language model's distribution) several hundred.
//
// Nothing is sorted here but a few dozen elements.  Both steps of top-p ask for the element at which the running sum of the sorted candidates
// crosses a bound, and that is a selection: a histogram of probability mass over the top bits of p (2048 bins, sixteen
// per factor of two) finds the bin of the crossing.  The first CTA adds up the histograms of the cluster (only the bins between the candidates'
// bound and the largest p) and finds both bins: where topp is exceeded, and where the coin falls.  The coin's bound is coin times a running sum
// inside the first bin, known up to that bin's mass, and mostly one bin holds whatever it turns out to be.  The elements of both are listed
// in one pass, cut into finer bins where they are more than a warp sorts, and the first CTA ends the launch: five cluster barriers.  Where the coin's bin is not
// certain, or a bin holds more elements than the list (flat distributions), the general way follows: bound by bound, cutting a bin into
// finer ones; when all bits are used up its elements are equal and are taken in index order.
//
// Masses are added as integers in units of 2^-52 (p's f32 mantissa fits), so the sums are exact, independent of the
// order in which the atomics happen, and at least as close to the real sums as the sequential f32 ones.
//
// What bounds it: latency (cluster barriers and the passes between them), not bytes: 513 KB of logits.  128256 tokens
// of a language model's distribution, top-p 0.95: 14.6 us per launch; with every bound searched for in turn (eleven barriers), divisions for every token, and
// loads one after the other 26.4; with one CTA and a sort 515 us.  20.5 against 44 us where the bin holds 1500 elements.  Multinomial 8.7 us (11.3).
#include "common.cuh"

#include <cooperative_groups.h>
#include <math.h>

namespace ib {

namespace cg = cooperative_groups;

constexpr int SAMPLE_THREADS = 1024, SAMPLE_WARPS = SAMPLE_THREADS / 32;
constexpr uint32_t SAMPLE_MAX_CLUSTER = 16;
// Vocabularies up to this size are one CTA's work: its barriers are a third of a cluster's, and a pass over them is four elements a thread.
// us per call, 1 / 16 CTAs, top-p: 512 tokens 7.2 / 10.2, 2048 9.9 / 13.3, 4096 9.6 / 10.7, 8192 11.1 / 10.5, 16384 17.2 / 11.2, 32000 27.4 / 11.9; multinomial:
// 512 3.7 / 6.0, 4096 5.1 / 6.2, 8192 6.4 / 6.2.
constexpr uint32_t SAMPLE_ONE_CTA = 4096;
constexpr uint32_t SAMPLE_BINS = 2048, SAMPLE_TOP_SHIFT = 19;   // p <= 1: bits(p) >> 19 <= 0x7F0
constexpr uint32_t SAMPLE_LIST = 4096;                          // elements of a bin that are ordered in shared memory
constexpr uint32_t SAMPLE_SLICE_MAX = 32768;                    // floats of a slice that fit shared memory beside the rest; longer slices live in global memory

struct SampleShared {
    uint2 hist[SAMPLE_BINS];                        // this CTA's histogram of mass: 64-bit sums as two words (see mass_add); later its elements of the bins of interest
    unsigned long long tot[SAMPLE_BINS];            // first CTA: the cluster's histogram
    unsigned long long list[SAMPLE_LIST];           // first CTA: the elements of one bin, key = (~bits(p), index)
    float xf[2][SAMPLE_MAX_CLUSTER];                // one word from every CTA of the cluster
    unsigned long long xu[2][SAMPLE_MAX_CLUSTER];
    unsigned long long red[SAMPLE_WARPS];
    unsigned long long base, answer, cum;           // first CTA: mass ahead of the bin; the crossing element's key and running sum
    unsigned long long base1, mass1, total;         // first CTA: mass ahead of and in the bin of the coin, mass of all candidates
    uint4 plan;                                     // every CTA: the two bins whose elements the first CTA wants, and whether it wants them (sample_plan)
    unsigned long long few[32], fine_base;          // first CTA: the elements of a finer bin, mass ahead of it
    uint32_t count, prefix, found, slot, bin_lo, bin_hi, n, fine, n_few;
};

// coin of a position: splitmix64 of (seed, position), top 24 bits -> [0, 1)
__host__ __device__ inline float sample_coin(uint64_t seed, uint32_t pos) {
    uint64_t z = seed + 0x9E3779B97F4A7C15ull * ((uint64_t)pos + 1ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z = z ^ (z >> 31);
    return (float)(uint32_t)(z >> 40) * (1.0f / 16777216.0f);
}

// p in units of 2^-52 (p in [0, 1]; exact for p >= 2^-29, rounded down below, but never to nothing: a coin of 0 falls to the first token
// whose p is above 0, however small).  A p that is no number - the logits held one, or an infinity - has no mass.
__device__ __forceinline__ unsigned long long mass_of(float p) {
    const uint32_t b = __float_as_uint(p), e = b >> 23;
    if (!(p > 0.f)) return 0ull;
    const unsigned long long m = (b & 0x7FFFFFu) | 0x800000u;
    const int s = (int)e - 98;   // value = m * 2^(e - 150)
    return s >= 0 ? m << s : (s > -24 ? m >> -s : 1ull);
}
// 64-bit shared-memory sum out of two native 32-bit atomics: whoever makes the low word wrap carries the one
__device__ __forceinline__ void mass_add(SampleShared &S, uint32_t bin, unsigned long long q) {
    const uint32_t l = (uint32_t)q;
    const uint32_t old = atomicAdd(&S.hist[bin].x, l);
    const uint32_t h = (uint32_t)(q >> 32) + ((uint32_t)(old + l) < old ? 1u : 0u);
    if (h) atomicAdd(&S.hist[bin].y, h);
}

__device__ __forceinline__ unsigned long long hist_sum(uint2 h) { return ((unsigned long long)h.y << 32) + h.x; }

template <typename T> __device__ __forceinline__ T shfl_down_t(T v, int o) { return __shfl_down_sync(0xffffffffu, v, o); }

// Inclusive scan over the block in thread order; *total gets the sum.  Ends with a barrier.
__device__ __forceinline__ unsigned long long block_scan(unsigned long long v, SampleShared &S, unsigned long long *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) S.red[warp] = v;
    __syncthreads();
    unsigned long long w = S.red[lane];   // SAMPLE_WARPS == 32
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += t;
    }
    *total = __shfl_sync(0xffffffffu, w, 31);
    const unsigned long long ahead = __shfl_sync(0xffffffffu, w, warp ? warp - 1 : 0);
    __syncthreads();
    return v + (warp ? ahead : 0ull);
}

// Ascending bitonic sort of list[0 .. cap) (cap a power of two <= SAMPLE_LIST).  Up to 1024 keys a thread holds one and the
// exchanges inside a warp are shuffles.
__device__ __forceinline__ void sort_list(unsigned long long *list, uint32_t cap) {
    const uint32_t tid = threadIdx.x;
    if (cap <= SAMPLE_THREADS) {
        unsigned long long v = tid < cap ? list[tid] : ~0ull;
        for (uint32_t k = 2; k <= cap; k <<= 1)
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                unsigned long long o;
                if (j >= 32) {
                    __syncthreads();
                    if (tid < cap) list[tid] = v;
                    __syncthreads();
                    o = tid < cap ? list[tid ^ j] : ~0ull;
                } else o = __shfl_xor_sync(0xffffffffu, v, j);
                const bool keep_min = ((tid & k) == 0) == ((tid & j) == 0);
                v = keep_min ? (v < o ? v : o) : (v < o ? o : v);
            }
        __syncthreads();
        if (tid < cap) list[tid] = v;
        __syncthreads();
        return;
    }
    for (uint32_t k = 2; k <= cap; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t t = tid; t < cap / 2; t += SAMPLE_THREADS) {
                const uint32_t a = ((t & ~(j - 1)) << 1) | (t & (j - 1)), b = a | j;
                const unsigned long long x = list[a], y = list[b];
                if ((x > y) == ((a & k) == 0)) { list[a] = y; list[b] = x; }
            }
            __syncthreads();
        }
}

__device__ __forceinline__ unsigned long long sort_warp(unsigned long long v, uint32_t lane) {
#pragma unroll
    for (uint32_t k = 2; k <= 32; k <<= 1)
#pragma unroll
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            const unsigned long long o = __shfl_xor_sync(0xffffffffu, v, j);
            const bool keep_min = ((lane & k) == 0) == ((lane & j) == 0);
            v = keep_min ? (v < o ? v : o) : (v < o ? o : v);
        }
    return v;
}
__device__ __forceinline__ uint32_t key_bin(unsigned long long key) { return (~(uint32_t)(key >> 32)) >> SAMPLE_TOP_SHIFT; }
__device__ __forceinline__ unsigned long long key_mass(unsigned long long key) { return mass_of(__uint_as_float(~(uint32_t)(key >> 32))); }
__device__ __forceinline__ unsigned long long scaled_mass(float f, unsigned long long m) { return (unsigned long long)((double)f * (double)m); }

// The element of `bin` among list[0 .. m) at which `base` + the running mass (descending p, ascending index) exceeds X, by finer bins of the next 11
// bits -> S.cum, S.answer.  False where more than 32 elements share the finer bin.  Called by a whole CTA; ends with a barrier.
__device__ __forceinline__ bool pick_in_bin(SampleShared &S, uint32_t m, uint32_t bin, unsigned long long base, unsigned long long X) {
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    constexpr uint32_t SHIFT = SAMPLE_TOP_SHIFT - 11;
    for (uint32_t b = tid; b < SAMPLE_BINS; b += SAMPLE_THREADS) S.hist[b] = make_uint2(0u, 0u);
    if (tid == 0) S.n_few = 0u;
    __syncthreads();
    for (uint32_t i = tid; i < m; i += SAMPLE_THREADS) {
        const unsigned long long key = S.list[i];
        if (key_bin(key) == bin) mass_add(S, (~(uint32_t)(key >> 32) >> SHIFT) & (SAMPLE_BINS - 1), key_mass(key));
    }
    __syncthreads();
    const uint32_t bin_a = SAMPLE_BINS - 1 - 2 * tid, bin_b = bin_a - 1;
    unsigned long long all;
    const unsigned long long a = hist_sum(S.hist[bin_a]), b = hist_sum(S.hist[bin_b]), upto = base + block_scan(a + b, S, &all), before = upto - a - b;
    if (X >= before && X < upto) {
        const bool second = X >= before + a;
        S.fine = second ? bin_b : bin_a;
        S.fine_base = second ? before + a : before;
    }
    __syncthreads();
    const uint32_t fine = S.fine;
    for (uint32_t i = tid; i < m; i += SAMPLE_THREADS) {
        const unsigned long long key = S.list[i];
        if (key_bin(key) == bin && ((~(uint32_t)(key >> 32) >> SHIFT) & (SAMPLE_BINS - 1)) == fine) {
            const uint32_t at = atomicAdd(&S.n_few, 1u);
            if (at < 32) S.few[at] = key;
        }
    }
    __syncthreads();
    const uint32_t n = S.n_few;
    if (n > 32) return false;
    if (tid < 32) {
        const unsigned long long key = sort_warp(lane < n ? S.few[lane] : ~0ull, lane);
        unsigned long long run = lane < n ? key_mass(key) : 0ull;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long t = __shfl_up_sync(0xffffffffu, run, o);
            if ((int)lane >= o) run += t;
        }
        run += S.fine_base;
        const uint32_t hit = __ballot_sync(0xffffffffu, lane < n && X < run);
        if ((int)lane == __ffs(hit) - 1) {
            S.cum = run;
            S.answer = key;
        }
    }
    __syncthreads();
    return true;
}

// AT_ONCE: elements per thread whose loads and arithmetic overlap; a slice is one round of them where there is an instance wide enough.
// `probs` [n]: scratch for slices that do not fit shared memory (null otherwise).  `pos_ptr` / `seed`: the coin
// (sample_coin); with pos_ptr == null `coin_in` is used.  Writes the token to *out (and to *out2 if non-null).
template <uint32_t AT_ONCE>
__global__ void __launch_bounds__(SAMPLE_THREADS) sample_kernel(const float *__restrict__ logits, uint32_t n, uint32_t slice, float temperature, float topp,
                                                                uint64_t seed, const uint32_t *pos_ptr, float coin_in, float *probs, uint32_t *out,
                                                                uint32_t *out2, uint32_t pdl) {
    extern __shared__ __align__(16) uint8_t smem[];
    SampleShared &S = *reinterpret_cast<SampleShared *>(smem);
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t C = cluster.num_blocks(), rank = cluster.block_rank(), tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    SampleShared &first = *cluster.map_shared_rank(&S, 0);
    auto barrier = [&]() { if (C > 1) cluster.sync(); else __syncthreads(); };

    cluster.barrier_arrive();   // every CTA of the cluster runs: needed before its shared memory is written from outside
    const bool nucleus = !(topp <= 0.f || topp >= 1.f);
    if (nucleus) {
        for (uint32_t b = tid; b < SAMPLE_BINS; b += SAMPLE_THREADS) {
            S.hist[b] = make_uint2(0u, 0u);
            if (rank == 0) S.tot[b] = 0ull;
        }
        if (tid == 0) { S.count = 0u; S.found = 0u; S.n = 0u; }
    }
    if (pdl) {
        asm volatile("griddepcontrol.launch_dependents;");
        asm volatile("griddepcontrol.wait;" ::: "memory");
    }
    const float coin = pos_ptr ? sample_coin(seed, *pos_ptr) : coin_in;
    const uint32_t i0 = min(n, rank * slice), len = min(n, i0 + slice) - i0;
    float *P = probs ? probs + i0 : reinterpret_cast<float *>(smem + sizeof(SampleShared));
    constexpr uint32_t STEP = AT_ONCE * SAMPLE_THREADS;

    // x = logits / temperature, softmax (softmax.rs:134-142)
    float mx = -INFINITY;
    for (uint32_t base = tid; base < len; base += STEP) {
        float v[AT_ONCE];
#pragma unroll
        for (uint32_t k = 0; k < AT_ONCE; k++) v[k] = base + k * SAMPLE_THREADS < len ? __ldcg(logits + i0 + base + k * SAMPLE_THREADS) : -INFINITY;
#pragma unroll
        for (uint32_t k = 0; k < AT_ONCE; k++) {
            const float x = __fdiv_rn(v[k], temperature);
            if (base + k * SAMPLE_THREADS < len) P[base + k * SAMPLE_THREADS] = x;
            mx = fmaxf(mx, x);
        }
    }
    // one f32 per CTA -> every CTA; `op` folds warps, then CTAs, in a fixed order
    auto exchange = [&](float v, int which, auto op) {
        float *red = reinterpret_cast<float *>(S.red);
#pragma unroll
        for (int o = 16; o; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
        if (lane == 0) red[warp] = v;
        __syncthreads();
        if (warp == 0) {
            v = red[lane];
#pragma unroll
            for (int o = 16; o; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
            if ((uint32_t)lane < C) *cluster.map_shared_rank(&S.xf[which][rank], lane) = v;
        }
        barrier();
        v = S.xf[which][0];
        for (uint32_t r = 1; r < C; r++) v = op(v, S.xf[which][r]);
        return v;
    };
    cluster.barrier_wait();
    mx = exchange(mx, 0, [](float a, float b) { return fmaxf(a, b); });
    float s = 0.f;
    for (uint32_t base = tid; base < len; base += STEP) {
#pragma unroll
        for (uint32_t k = 0; k < AT_ONCE; k++) {
            const uint32_t i = base + k * SAMPLE_THREADS;
            if (i < len) {
                const float e = expf(P[i] - mx);
                P[i] = e;
                s += e;
            }
        }
    }
    const float sum = exchange(s, 1, [](float a, float b) { return a + b; });
    auto done = [&](uint32_t token) {
        *out = token;
        if (out2) *out2 = token;
    };

    if (!nucleus) {
        // sampler.rs:62-77: the slices' masses, then the slice that holds the crossing looks for it.  A thread adds up consecutive elements, an odd
        // number of them: a warp's reads of one element each then fall to different banks.
        const uint32_t per = ((len + SAMPLE_THREADS - 1) / SAMPLE_THREADS) | 1u, a = min(len, tid * per), b = min(len, a + per);
        unsigned long long mine = 0ull, total, ahead = 0ull;
        constexpr uint32_t TOGETHER = AT_ONCE == 1 ? 1 : AT_ONCE + 1;   // (places and one more: the odd number)
        for (uint32_t base = a; base < b; base += TOGETHER) {
#pragma unroll
            for (uint32_t k = 0; k < TOGETHER; k++)
                if (base + k < b) {
                    const float p = __fdiv_rn(P[base + k], sum);
                    P[base + k] = p;
                    mine += mass_of(p);
                }
        }
        const unsigned long long upto = block_scan(mine, S, &total);
        if (tid < C) *cluster.map_shared_rank(&S.xu[0][rank], tid) = total;
        barrier();
        const unsigned long long X = (unsigned long long)((double)coin * 4503599627370496.0);
        for (uint32_t r = 0; r < rank; r++) ahead += S.xu[0][r];
        unsigned long long run = ahead + upto - mine;
        if (X >= run && X < run + mine) {
            for (uint32_t i = a; i < b; i++) {
                run += mass_of(P[i]);
                if (X < run) { done(i0 + i); break; }
            }
        }
        if (rank == C - 1 && tid == 0 && X >= ahead + total) done(n - 1);
        return;
    }

    // sampler.rs:84-129
    const float cutoff = __fdiv_rn(1.0f - topp, (float)n - 1.0f);
    // P becomes p where an element is a candidate, -e elsewhere.  Most of a language model's tokens are no candidates, and in places that no warp
    // shares: every thread notes which of its elements may be (the exact test is on the rounded p), and the divisions go to those.
    const float clearly_less = cutoff * sum * 0.999f;
    for (uint32_t base = 0; base < len; base += STEP) {
        uint32_t may = 0;
#pragma unroll
        for (uint32_t k = 0; k < AT_ONCE; k++) {
            const uint32_t i = base + k * SAMPLE_THREADS + tid;
            if (i < len) {
                const float e = P[i];
                if (e >= clearly_less) may |= 1u << k;
                else P[i] = -e;
            }
        }
        while (__any_sync(0xffffffffu, may != 0u)) {
            const uint32_t i = base + (may ? __ffs(may) - 1 : 0) * SAMPLE_THREADS + tid;
            const float e = may ? P[i] : 0.f, p = may ? __fdiv_rn(e, sum) : -1.f;
            const bool cand = p >= cutoff;
            if (may) P[i] = cand ? p : -e;
            may &= may - 1;
            const uint32_t bin = min(__float_as_uint(p) >> SAMPLE_TOP_SHIFT, SAMPLE_BINS - 1), act = __ballot_sync(0xffffffffu, cand);
            if (act == 0u) continue;
            // flat distributions: a warp whose 32 candidates share a bin adds them up first
            int same = 0;
            if (act == 0xffffffffu) __match_all_sync(0xffffffffu, bin, &same);
            unsigned long long q = cand ? mass_of(p) : 0ull;
            if (same) {
#pragma unroll
                for (int o = 16; o; o >>= 1) q += __shfl_xor_sync(0xffffffffu, q, o);
                if (lane == 0) mass_add(S, bin, q);
            } else if (cand) mass_add(S, bin, q);
        }
    }

    // Both answers - the running sum at which topp is exceeded (`cum`), and the element at which coin * cum is - lie in two bins that the first
    // CTA finds from the cluster's histogram: the coin's bound is known up to the mass of the first one, and mostly that leaves one bin.
    // The elements of both go into the first CTA's list, are ordered once, and the first CTA ends the launch.
    const unsigned long long X0 = (unsigned long long)((double)topp * 4503599627370496.0);
    constexpr uint32_t NO_BIN = 0xFFFFFFFFu;
    barrier();
    if (rank == 0) {
        const uint32_t lo = __float_as_uint(cutoff) >> SAMPLE_TOP_SHIFT, hi = min(__float_as_uint(__fdiv_rn(1.0f, sum)) >> SAMPLE_TOP_SHIFT, SAMPLE_BINS - 1);   // (the largest e is 1)
        const uint32_t lanes = C >= 4 ? 4 : 1, items = hi >= lo ? (hi - lo + 1) * lanes : 0;
        for (uint32_t base = 0; base < items; base += SAMPLE_THREADS) {
            const uint32_t it = base + tid, bin = lo + it / lanes;
            unsigned long long v = 0ull;
            uint2 h[4] = {};
#pragma unroll
            for (uint32_t k = 0; k < 4; k++)
                if (it < items && it % lanes + k * lanes < C) h[k] = cluster.map_shared_rank(&S, it % lanes + k * lanes)->hist[bin];
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) v += hist_sum(h[k]);
            if (lanes == 4) {
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
            }
            if (it < items && it % lanes == 0) S.tot[bin] = v;
        }
        __syncthreads();
        unsigned long long total;
        const uint32_t bin_a = SAMPLE_BINS - 1 - 2 * tid, bin_b = bin_a - 1;   // counted from the largest
        const unsigned long long a = S.tot[bin_a], b = S.tot[bin_b], upto = block_scan(a + b, S, &total), before = upto - a - b;
        if (X0 >= before && X0 < upto) {
            const bool second = X0 >= before + a;
            S.prefix = second ? bin_b : bin_a;
            S.base = second ? before + a : before;
            S.found = 1u;
        }
        __syncthreads();
        const bool found = S.found != 0u;
        // cum lies in (base, base + the bin's mass]; not found: the candidates do not reach topp, all of them are in
        const unsigned long long c0 = found ? S.base + 1 : total, c1 = found ? S.base + S.tot[S.prefix] : total;
        const unsigned long long X1[2] = {scaled_mass(coin, c0), scaled_mass(coin, c1)};
#pragma unroll
        for (int w = 0; w < 2; w++)
            if (X1[w] >= before && X1[w] < upto) {
                const bool second = X1[w] >= before + a;
                if (w == 0) S.bin_lo = second ? bin_b : bin_a;
                else {
                    S.bin_hi = second ? bin_b : bin_a;
                    S.base1 = second ? before + a : before;
                    S.mass1 = second ? b : a;
                }
            }
        if (tid == 0) S.total = total;
        __syncthreads();
        // (no candidates, a bound that two bins may hold, or more elements than the list has room for - at least a bin's mass over its largest p: the general way)
        if (tid < C) {
            const uint32_t bin0 = found ? S.prefix : NO_BIN, bin1 = S.bin_hi;
            bool plain = total != 0ull && S.bin_lo == bin1;
            if (plain) {
                auto least = [](unsigned long long mass, uint32_t bin) { return (float)mass / (float)mass_of(__uint_as_float(((bin + 1) << SAMPLE_TOP_SHIFT) - 1)); };
                plain = least(S.mass1, bin1) + (found && bin0 != bin1 ? least(S.tot[bin0], bin0) : 0.f) <= (float)(C == 1 ? SAMPLE_BINS : SAMPLE_LIST);
            }
            cluster.map_shared_rank(&S, tid)->plan = make_uint4(bin0, bin1, plain ? 1u : 0u, 0u);
        }
    }
    barrier();
    if (S.plan.z) {
        const uint32_t bin0 = S.plan.x, bin1 = S.plan.y;
        unsigned long long *staged = reinterpret_cast<unsigned long long *>(S.hist);   // (the first CTA has read it)
        for (uint32_t base = tid; base < len; base += STEP) {
#pragma unroll
            for (uint32_t k = 0; k < AT_ONCE; k++) {
                const uint32_t i = base + k * SAMPLE_THREADS;
                const uint32_t bits = i < len ? __float_as_uint(P[i]) : 0x80000000u, bin = bits >> SAMPLE_TOP_SHIFT;   // (no candidate: the sign)
                if (bin == bin0 || bin == bin1) {
                    const uint32_t at = atomicAdd(&S.n, 1u);
                    if (at < SAMPLE_BINS) staged[at] = ((unsigned long long)(~bits) << 32) | (i0 + i);
                }
            }
        }
        __syncthreads();
        const uint32_t mine = S.n;
        if (tid == 0 && mine) S.slot = atomicAdd(&first.count, mine <= SAMPLE_BINS ? mine : SAMPLE_LIST + 1u);
        __syncthreads();
        if (mine && mine <= SAMPLE_BINS) {
            const uint32_t at = S.slot;
            for (uint32_t i = tid; i < mine; i += SAMPLE_THREADS)
                if (at + i < SAMPLE_LIST) first.list[at + i] = staged[i];
        }
        barrier();
        const uint32_t m = first.count;
        if (m <= SAMPLE_LIST) {
            cluster.barrier_arrive();   // the first CTA's words have been read
            if (rank != 0) return;
            const bool found = bin0 != NO_BIN;
            const unsigned long long base1 = S.base1, cum_all = S.total;
            if (m > 32 && (!found || pick_in_bin(S, m, bin0, S.base, X0)) &&
                pick_in_bin(S, m, bin1, base1, scaled_mass(coin, found ? S.cum : cum_all))) {
                if (tid == 0) done((uint32_t)S.answer);
                cluster.barrier_wait();
                return;
            }
            const unsigned long long base0 = S.base - (bin0 != bin1 ? S.mass1 : 0ull);   // both bins in one order: the coin's bin comes first, its mass is in front
            if (m <= 32) {
                if (warp == 0) {
                    const unsigned long long key = sort_warp(lane < (int)m ? S.list[lane] : ~0ull, lane), q = lane < (int)m ? key_mass(key) : 0ull;
                    unsigned long long run = q;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const unsigned long long t = __shfl_up_sync(0xffffffffu, run, o);
                        if (lane >= o) run += t;
                    }
                    const uint32_t bin = lane < (int)m ? key_bin(key) : NO_BIN - 1u, at = __ballot_sync(0xffffffffu, found && bin == bin0 && X0 < base0 + run);
                    const unsigned long long cum = found ? __shfl_sync(0xffffffffu, base0 + run, at ? __ffs(at) - 1 : 0) : S.total, X1 = scaled_mass(coin, cum);
                    const uint32_t hit = __ballot_sync(0xffffffffu, bin == bin1 && X1 < base1 + run);
                    if (lane == __ffs(hit) - 1) done((uint32_t)key);
                }
            } else {
                uint32_t cap = 64;
                while (cap < m) cap <<= 1;
                for (uint32_t i = m + tid; i < cap; i += SAMPLE_THREADS) S.list[i] = ~0ull;
                __syncthreads();
                sort_list(S.list, cap);
                const uint32_t per = (m + SAMPLE_THREADS - 1) / SAMPLE_THREADS, a = min(m, tid * per), b = min(m, a + per);
                unsigned long long mass = 0ull, all;
                for (uint32_t i = a; i < b; i++) mass += key_mass(S.list[i]);
                const unsigned long long before = block_scan(mass, S, &all) - mass;
                if (found && X0 >= base0 + before && X0 < base0 + before + mass) {
                    unsigned long long run = base0 + before;
                    for (uint32_t i = a; i < b; i++) {
                        run += key_mass(S.list[i]);
                        if (X0 < run && key_bin(S.list[i]) == bin0) { S.cum = run; break; }
                    }
                }
                __syncthreads();
                const unsigned long long X1 = scaled_mass(coin, found ? S.cum : S.total);
                if (X1 >= base1 + before && X1 < base1 + before + mass) {
                    unsigned long long run = base1 + before;
                    for (uint32_t i = a; i < b; i++) {
                        run += key_mass(S.list[i]);
                        if (X1 < run) { done((uint32_t)S.list[i]); break; }
                    }
                }
            }
            cluster.barrier_wait();
            return;
        }
        // more elements than the list holds
        barrier();   // (everyone has read the first CTA's words)
        if (tid == 0) S.count = 0u;
        for (uint32_t b = tid; b < SAMPLE_BINS; b += SAMPLE_THREADS) S.hist[b] = make_uint2(0u, 0u);
        __syncthreads();
        for (uint32_t i = tid; i < len; i += SAMPLE_THREADS)
            if (P[i] >= cutoff) mass_add(S, min(__float_as_uint(P[i]) >> SAMPLE_TOP_SHIFT, SAMPLE_BINS - 1), mass_of(P[i]));
    }
    if (tid == 0) S.found = 0u;

    // the cluster's histogram in the first CTA: every CTA adds up its share of the bins over the CTAs
    auto gather_bins = [&]() {
        barrier();
        if (C == 1) {
            for (uint32_t b = tid; b < SAMPLE_BINS; b += SAMPLE_THREADS) S.tot[b] = hist_sum(S.hist[b]);
            __syncthreads();
            return;
        }
        const uint32_t lanes = C / 2, share = SAMPLE_BINS / C, bin = rank * share + tid / lanes, r0 = tid % lanes;   // share * lanes == SAMPLE_THREADS
        unsigned long long v = 0ull;
#pragma unroll
        for (uint32_t k = 0; k < 2; k++) {
            v += hist_sum(cluster.map_shared_rank(&S, r0 + k * lanes)->hist[bin]);
        }
        for (uint32_t o = lanes / 2; o; o >>= 1) v += shfl_down_t(v, o);
        if (r0 == 0) first.tot[bin] = v;
        barrier();
    };
    // first CTA: the bin, counted from the largest, at which base + running mass exceeds X -> S.prefix, S.base, S.found
    auto find_bin = [&](unsigned long long base, unsigned long long X, uint32_t prefix_above, unsigned long long *total) {
        const unsigned long long a = S.tot[SAMPLE_BINS - 1 - 2 * tid], b = S.tot[SAMPLE_BINS - 2 - 2 * tid];
        const unsigned long long upto = base + block_scan(a + b, S, total), before = upto - a - b;
        if (tid == 0) S.count = 0u;
        if (X >= before && X < upto) {
            const bool second = X >= before + a;
            S.prefix = prefix_above | (SAMPLE_BINS - 1 - 2 * tid - (second ? 1u : 0u));
            S.base = second ? before + a : before;
            S.found = 1u;
        }
        __syncthreads();
    };

    if (S.plan.z) gather_bins();   // (else the first CTA's sums of before are still those of all candidates)
    unsigned long long X = X0, total = 0ull;
    uint32_t listed = 0xFFFFFFFFu, listed_m = 0;   // the top-level bin whose elements are in the list, ordered, and their number
    // Query 0: where the running sum exceeds topp (only that running sum matters: `cum`); query 1: where it exceeds coin * cum.
    for (int query = 0; query < 2; query++) {
        if (rank == 0) {
            find_bin(0ull, X, 0u, &total);
            if (!S.found && tid == 0) S.cum = total;   // query 0 only: the candidates do not reach topp, all of them are in
        }
        barrier();
        const uint32_t found = first.found;
        if (query == 0 && !found) {
            // (no candidate at all - (1 - topp) / (n - 1) above the largest probability, e.g. n = 2 with a small topp: the reference
            // subtracts 1 from an unsigned zero there (sampler.rs:108); defined here as the arg-max, lowest index on ties)
            if (first.cum == 0ull) {
                unsigned long long b = 0ull;
                for (uint32_t i = tid; i < len; i += SAMPLE_THREADS) {
                    const unsigned long long k = ((unsigned long long)__float_as_uint(__fdiv_rn(-P[i], sum)) << 32) | (0xFFFFFFFFu - (i0 + i));   // p >= 0: bits order like values
                    b = k > b ? k : b;
                }
#pragma unroll
                for (int o = 16; o; o >>= 1) { const unsigned long long t = __shfl_xor_sync(0xffffffffu, b, o); b = t > b ? t : b; }
                if (lane == 0) S.red[warp] = b;
                __syncthreads();
                if (tid == 0) {
                    for (int w = 1; w < SAMPLE_WARPS; w++) b = S.red[w] > b ? S.red[w] : b;
                    first.xu[1][rank] = b;
                }
                barrier();
                if (rank == 0 && tid == 0) {
                    for (uint32_t r = 0; r < C; r++) b = S.xu[1][r] > b ? S.xu[1][r] : b;
                    done(0xFFFFFFFFu - (uint32_t)b);
                }
                return;
            }
        } else {
            uint32_t shift = SAMPLE_TOP_SHIFT;
            for (;;) {
                const uint32_t prefix = first.prefix;
                const bool have = shift == SAMPLE_TOP_SHIFT && prefix == listed;
                if (!have) {
                    // the bin's elements into the first CTA's list
                    auto in_bin = [&](uint32_t i) {
                        const float p = P[i];
                        const uint32_t bits = __float_as_uint(p);
                        return p >= cutoff && (shift == SAMPLE_TOP_SHIFT ? min(bits >> shift, SAMPLE_BINS - 1) : bits >> shift) == prefix;
                    };
                    uint32_t c = 0;
                    for (uint32_t i = tid; i < len; i += SAMPLE_THREADS) c += in_bin(i);
                    unsigned long long mine;
                    const uint32_t at0 = (uint32_t)block_scan(c, S, &mine) - c;
                    if (tid == 0 && mine) S.slot = atomicAdd(&first.count, (uint32_t)mine);
                    __syncthreads();
                    if (c) {
                        uint32_t at = S.slot + at0;
                        for (uint32_t i = tid; i < len; i += SAMPLE_THREADS)
                            if (in_bin(i)) {
                                if (at < SAMPLE_LIST) first.list[at] = ((unsigned long long)(~__float_as_uint(P[i])) << 32) | (i0 + i);
                                at++;
                            }
                    }
                    if (tid < C) *cluster.map_shared_rank(&S.xu[1][rank], tid) = mine;
                    barrier();
                }
                const uint32_t m = have ? listed_m : first.count;
                if (m <= SAMPLE_LIST) {
                    if (rank == 0) {
                        uint32_t cap = 1;
                        while (cap < m) cap <<= 1;
                        if (!have) {
                            for (uint32_t i = m + tid; i < cap; i += SAMPLE_THREADS) S.list[i] = ~0ull;
                            __syncthreads();
                            sort_list(S.list, cap);
                        }
                        const uint32_t per = (m + SAMPLE_THREADS - 1) / SAMPLE_THREADS, a = min(m, tid * per), b = min(m, a + per);
                        auto q_at = [&](uint32_t i) { return mass_of(__uint_as_float(~(uint32_t)(S.list[i] >> 32))); };
                        unsigned long long mine = 0ull, all;
                        for (uint32_t i = a; i < b; i++) mine += q_at(i);
                        unsigned long long run = S.base + block_scan(mine, S, &all) - mine;
                        if (X >= run && X < run + mine) {
                            for (uint32_t i = a; i < b; i++) {
                                run += q_at(i);
                                if (X < run) { S.cum = run; S.answer = S.list[i]; break; }
                            }
                        }
                        __syncthreads();
                        if (query == 1 && tid == 0) done((uint32_t)S.answer);
                    }
                    listed = shift == SAMPLE_TOP_SHIFT ? prefix : 0xFFFFFFFFu;
                    listed_m = m;
                    break;
                }
                if (shift == 0) {
                    // more equal elements than the list holds: number k of them in index order
                    const unsigned long long q = mass_of(__uint_as_float(prefix)), b0 = first.base, k = (X - b0) / q;
                    if (query == 0) {
                        if (rank == 0 && tid == 0) S.cum = b0 + (k + 1) * q;
                        barrier();   // (everyone has read the first CTA's words)
                    } else {
                        unsigned long long ahead = 0ull, mine;
                        for (uint32_t r = 0; r < rank; r++) ahead += S.xu[1][r];
                        const uint32_t per = (len + SAMPLE_THREADS - 1) / SAMPLE_THREADS, a = min(len, tid * per), b = min(len, a + per);
                        uint32_t c = 0;
                        for (uint32_t i = a; i < b; i++) c += __float_as_uint(P[i]) == prefix;
                        unsigned long long at = ahead + block_scan(c, S, &mine) - c;
                        for (uint32_t i = a; i < b; i++)
                            if (__float_as_uint(P[i]) == prefix && at++ == k) done(i0 + i);
                    }
                    listed = 0xFFFFFFFFu;
                    break;
                }
                // finer bins inside this one
                const uint32_t next = shift > 11 ? shift - 11 : 0, width = shift - next;
                for (uint32_t b = tid; b < SAMPLE_BINS; b += SAMPLE_THREADS) S.hist[b] = make_uint2(0u, 0u);
                __syncthreads();
                for (uint32_t i = tid; i < len; i += SAMPLE_THREADS) {
                    const float p = P[i];
                    const uint32_t bits = __float_as_uint(p);
                    if (p >= cutoff && bits >> shift == prefix) mass_add(S, (bits >> next) & ((1u << width) - 1u), mass_of(p));
                }
                gather_bins();
                if (rank == 0) find_bin(S.base, X, prefix << width, &total);
                shift = next;
                barrier();
            }
        }
        if (query == 0) {
            // the second bound, known to the first CTA; the top-level histogram is needed again if finer ones took its place
            barrier();
            X = scaled_mass(coin, first.cum);
            if (listed == 0xFFFFFFFFu && found) {
                for (uint32_t b = tid; b < SAMPLE_BINS; b += SAMPLE_THREADS) S.hist[b] = make_uint2(0u, 0u);
                __syncthreads();
                for (uint32_t i = tid; i < len; i += SAMPLE_THREADS)
                    if (P[i] >= cutoff) mass_add(S, min(__float_as_uint(P[i]) >> SAMPLE_TOP_SHIFT, SAMPLE_BINS - 1), mass_of(P[i]));
                gather_bins();
            }
        }
    }
    barrier();   // no CTA leaves while another may still read its shared memory
}

// Scratch a launch needs in global memory (0 for vocabularies whose slices fit shared memory: up to 262144 tokens on clusters of 8)
size_t sample_scratch_bytes(uint32_t n) { return (n + 7) / 8 <= SAMPLE_SLICE_MAX ? 0 : sizeof(float) * (size_t)n; }

int32_t launch_sample(ib_ctx *ctx, cudaStream_t s, const float *logits, uint32_t n, float temperature, float topp, uint64_t seed, const uint32_t *pos_ptr,
                      float coin, float *probs, uint32_t *out, uint32_t *out2, uint32_t pdl) {
    // The instance that a slice fits with the fewest idle places: places cost instructions, a second round another trip to L2 (us per call, top-p,
    // 5 / 8 / 10 places: 32000 tokens, 2 a thread, 13.0 / 14.3 / 15.3; 128256, 8 a thread, 16.1 / 14.6 / 15.6; 152000, 10 a thread, 15.7 / 18.0 / 15.4).
    using Kernel = void (*)(const float *, uint32_t, uint32_t, float, float, uint64_t, const uint32_t *, float, float *, uint32_t *, uint32_t *, uint32_t);
    static constexpr Kernel kernels[] = {sample_kernel<1>, sample_kernel<2>, sample_kernel<3>, sample_kernel<4>, sample_kernel<5>, sample_kernel<6>, sample_kernel<7>, sample_kernel<8>, sample_kernel<9>, sample_kernel<10>};
    constexpr uint32_t INSTANCES = sizeof(kernels) / sizeof(kernels[0]);
    static uint32_t cluster_size[16] = {0};
    const size_t smem_max = sizeof(SampleShared) + SAMPLE_SLICE_MAX * sizeof(float);
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    cfg.blockDim = dim3(SAMPLE_THREADS);
    cfg.stream = s;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    uint32_t &C = cluster_size[ctx->device & 15];
    if (!C) {
        for (Kernel k : kernels) {
            IB_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max));
            IB_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        }
        // 16 CTAs of one cluster have to fit one graphics-processing cluster of the device
        int fit = 0;
        attr[0].val.clusterDim.x = SAMPLE_MAX_CLUSTER;
        cfg.gridDim = dim3(SAMPLE_MAX_CLUSTER);
        cfg.numAttrs = 1;
        cfg.dynamicSmemBytes = smem_max;
        C = (cudaOccupancyMaxActiveClusters(&fit, kernels[0], &cfg) == cudaSuccess && fit > 0) ? SAMPLE_MAX_CLUSTER : 8u;
        cudaGetLastError();
    }
    const uint32_t ctas = n <= SAMPLE_ONE_CTA ? 1u : C, slice = (n + ctas - 1) / ctas;
    attr[0].val.clusterDim.x = ctas;
    cfg.gridDim = dim3(ctas);
    cfg.dynamicSmemBytes = sizeof(SampleShared) + (probs ? 0 : slice * sizeof(float));
    cfg.numAttrs = pdl ? 2 : 1;
    const uint32_t places = (slice + SAMPLE_THREADS - 1) / SAMPLE_THREADS, fits = places < 1 ? 0 : places - 1;
    IB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernels[fits < INSTANCES ? fits : INSTANCES - 1], logits, n, slice, temperature, topp, seed, pos_ptr, coin, probs, out, out2, pdl));
    ctx->launches++;
    return IB_OK;
}

}  // namespace ib

extern "C" int32_t ib_sample(ib_ctx *ctx, void *stream, const float *logits_dev, uint32_t n, float temperature, float topp, float coin, uint32_t *out_dev) {
    using namespace ib;
    IB_REQUIRE(ctx && logits_dev && out_dev, "ib_sample: null argument");
    IB_REQUIRE(cudaSetDevice(ctx->device) == cudaSuccess, "cudaSetDevice failed");
    IB_REQUIRE(n >= 2 && n <= (1u << 22), "ib_sample: n=%u outside [2, 4194304]", n);
    IB_REQUIRE(coin >= 0.f && coin < 1.f, "ib_sample: coin=%f outside [0, 1)", (double)coin);
    IB_REQUIRE(temperature >= 0.f, "ib_sample: negative temperature");
    if (temperature == 0.f) return launch_argmax(ctx, (cudaStream_t)stream, logits_dev, n, out_dev);   // sampler.rs:33-35
    // stream-ordered scratch for the vocabularies that need it
    float *scratch = nullptr;
    const size_t bytes = sample_scratch_bytes(n);
    if (bytes) IB_CHECK_CUDA(cudaMallocAsync((void **)&scratch, bytes, (cudaStream_t)stream));
    const int32_t rc = launch_sample(ctx, (cudaStream_t)stream, logits_dev, n, temperature, topp, 0, nullptr, coin, scratch, out_dev, nullptr, 0);
    if (scratch) cudaFreeAsync(scratch, (cudaStream_t)stream);
    return rc;
}
