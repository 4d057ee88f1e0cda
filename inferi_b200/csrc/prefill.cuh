// Prompt prefill on the tensor cores: what the model code (llama.cu), the GEMM (prefill_gemm.cu) and the element-wise kernels
// around it (prefill.cu) share.
#pragma once

#include "token.cuh"

namespace ib {

constexpr uint32_t PF_CHUNK = 128;             // tokens per GEMM tile (the N of the MMA)
// Tokens that go through the layers together; longer prompts go in passes.  Two passes cost hardly more than a pass of twice the length would
// (two layers of the 8B shapes: 1024 tokens 2.45 ms, 2000 tokens 5.28), and the buffers grow by 41 MB per 128 tokens of these shapes.
constexpr uint32_t PREFILL_MAX_TOKENS = 1024;
constexpr uint32_t PF_MAX_SEGS = 3;            // matrices of one GEMM launch

// A tile of the prefill GEMM is 256 rows on a pair of SMs that share the tokens' inputs, or 128 rows on one SM: up to 16 tokens, and up to 64
// where no SM gets more than one unit of work (prefill_streamk).
constexpr uint32_t PF_SINGLE_ALWAYS = 16, PF_SINGLE_TOKENS = 64;

// How a prefill GEMM's work is handed out: the units (row tile, chunk of 128 tokens, 256-column block), in that order, are
// cut into contiguous, equally long ranges - one per CTA or pair of CTAs of a grid that fills the GPU exactly once, whatever the
// matrix's shape (a grid of tiles x K slices was 1.5 waves for the FFN matrices).  The K range of a tile (= row tile and
// chunk) can then fall to several ranges; each CTA or pair writes its partial sums to the plane numbered by its position among the
// tile's, and the element-wise kernel behind the GEMM adds a tile's planes in that order.
struct StreamK {
    uint32_t ranges, nb, total, row_log2;   // ranges, 256-column blocks per row, units = tiles * nb, rows of a tile (log2)
    // 32-bit arithmetic: the launcher keeps total below 2^24
    __host__ __device__ uint32_t first_unit(uint32_t c) const { return c * total / ranges; }
    __host__ __device__ uint32_t range_of(uint32_t u) const { return ((u + 1) * ranges - 1) / total; }
    __host__ __device__ uint32_t pieces(uint32_t tile) const { return range_of(tile * nb + nb - 1) - range_of(tile * nb) + 1; }
    __host__ __device__ uint32_t row_tile(uint32_t row) const { return row >> row_log2; }
};
StreamK prefill_streamk(const ib_ctx *ctx, uint32_t rows, uint32_t cols, uint32_t n);
// a launch that two groups of rows of different formats share: the split of each.  (Never more pieces per tile than as launches of their own.)
void prefill_streamk_mixed(const ib_ctx *ctx, uint32_t rows_a, uint32_t rows_b, uint32_t cols, uint32_t n, StreamK &a, StreamK &b);
uint32_t prefill_max_pieces(const StreamK &sk);   // bound of the planes that any tile needs

struct PgParams {
    uint32_t tile0[PF_MAX_SEGS];   // first row tile of each matrix (0xFFFFFFFF: not there)
    uint32_t rows, n, chunks;      // rows of all matrices together, tokens, chunks of 128 tokens
    const __half *x;               // the tokens' inputs split into two f16, tiled (pf_x_index); per chunk x_chunk halves
    size_t x_chunk;
    float *plane0, *planes;        // [n][rows] the first range's sums of every tile; [piece - 1][n][rows] the others'
    uint32_t x_stages, x_tile;     // ring of the inputs: stages, bytes of a stage's hi (= lo) half (set by the launcher)
    StreamK sk;
    uint32_t *err;
    unsigned long long wait_ns;
};

// ---- the tokens' inputs in global memory, laid out the way the tensor core reads them from shared memory ----
// Per chunk of 128 tokens: one tile of 128 token rows per 64 columns in the K-major core-matrix layout (8 rows x 16 bytes),
// the eight hi core matrices of a group of 8 tokens (1 KiB) followed by its eight lo ones, so that what a stage needs of any range
// of groups is one bulk copy (a copying warp's turn takes about 430 clocks whatever it copies).  Four consecutive columns are
// stored in the order 0, 2, 1, 3, the order in which the producers unpack the weights.
constexpr uint32_t PF_X_LO = 512, PF_S_LO = 128;   // halves from an element's hi part to its lo part: of the inputs, of the sums
__host__ __device__ inline uint32_t pf_x_index(uint32_t t, uint32_t c) {   // halves inside the chunk; t: token inside the chunk
    const uint32_t k = (c & 4u) | ((c & 1u) << 1) | ((c >> 1) & 1u);
    return (c >> 6) * (PF_CHUNK * 128) + (t >> 3) * 1024 + ((c & 63) >> 3) * 64 + (t & 7) * 8 + k;
}
// Behind the input tiles of a chunk sit the tiles of its sub-block sums: per 256 columns one tile of 128 token rows x 16 halves
// in the same core-matrix layout (the sums of the block's eight 32-column sub-blocks, then eight zeros), hi and lo by groups of 8
// tokens like the inputs.  The k-quant GEMM multiplies them with the sub-blocks' minimums.
__host__ __device__ inline uint32_t pf_s_index(uint32_t t, uint32_t sb, uint32_t cols) {
    return 2 * PF_CHUNK * cols + (sb >> 3) * (PF_CHUNK * 32) + (t >> 3) * 256 + (t & 7) * 8 + (sb & 7);
}
__host__ __device__ inline size_t pf_x_halves(uint32_t cols) { return (size_t)2 * (PF_CHUNK + 8) * cols; }   // halves per chunk

bool prefill_gemm_eligible(const ib_qtensor *m);
// What one format's matrices of a GEMM launch are and give: plane0 / planes = partial sums of W x_t over the tile's K ranges.  The matrices have the
// same type and width; their rows follow one another.
struct PrefillPart {
    const ib_qtensor *const *mats;
    uint32_t n_mats;
    float *plane0, *planes;
    StreamK sk;
};
// x: the layout above, token rows n .. (n rounded up to 16) - 1 of the last chunk zero; early: the weights may be read before the stream's previous
// kernels are done
int32_t launch_prefill_gemm(ib_ctx *ctx, cudaStream_t s, const PrefillPart &w, const __half *x, uint32_t n, bool early = true);
// two formats with the same inputs in one launch: Q4_K or Q5_K, and Q6_K, where that is the faster way for n tokens
bool prefill_mixable(const ib_qtensor *a, const ib_qtensor *b, uint32_t n);
int32_t launch_prefill_gemm_mixed(ib_ctx *ctx, cudaStream_t s, const PrefillPart &a, const PrefillPart &b, const __half *x, uint32_t n);

// One GEMM launch's result, as the element-wise kernels read it
struct PfPlanes {
    const float *plane0, *planes;
    StreamK sk;
    uint32_t rows, chunks, n;
};

int32_t launch_prefill_embed(ib_ctx *ctx, cudaStream_t s, const ib_qtensor *embd, const uint32_t *tokens_dev, uint32_t n, uint32_t vocab, float *X);
// X += the planes (if any); y = RMSNorm(X) with weights w (null: y = X), split and tiled into xt
int32_t launch_prefill_norm_split(ib_ctx *ctx, cudaStream_t s, float *X, const PfPlanes *add, const float *w, float eps, uint32_t n, uint32_t cols, __half *xt);
// X += the planes
int32_t launch_prefill_residual(ib_ctx *ctx, cudaStream_t s, float *X, const PfPlanes &add);
// out += the planes behind plane 0 (= out): completes a GEMM whose plane 0 was its output
int32_t launch_prefill_finish(ib_ctx *ctx, cudaStream_t s, float *out, const PfPlanes &add);
// y = up * silu(gate), split and tiled: gate = rows 0 .. F-1, up = rows F .. 2F-1 of one launch
int32_t launch_prefill_swiglu(ib_ctx *ctx, cudaStream_t s, const PfPlanes &gu, __half *xt);

struct PfQkv {
    PfPlanes g[3];                   // the launches that q, k and v came from (two or three may be the same launch) ...
    uint32_t row0[3];                // ... and the row of the launch at which each starts
    const float *bias[3];
    uint32_t n, q_dim, kv_dim, head_size, pos0, kv_dtype;
    const float *theta;              // [head_size / 2]
    float *q;                        // [n][q_dim]
    void *k_cache, *v_cache;         // this layer's cache [max_pos][kv_dim]
};
// causal attention of n queries at positions pos0 .. pos0 + n - 1 (four query heads per kv head, f16 cache that already holds their
// rows); the result as the next GEMM's inputs
int32_t launch_prefill_attention(ib_ctx *ctx, cudaStream_t s, const float *q, const void *k_cache, const void *v_cache, uint32_t n, uint32_t pos0, uint32_t n_kv, uint32_t head_size,
                                 __half *xt);
// bias, rotation, q out and cache append
int32_t launch_prefill_qkv(ib_ctx *ctx, cudaStream_t s, const PfQkv &p);

}  // namespace ib
