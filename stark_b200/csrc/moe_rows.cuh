// Prompt rows of the routed-expert decoder (moe_rows.cu): the f32 conventions of a token (moe_model.cu), many rows at once.
#pragma once
#include <algorithm>

#include "moe_math.cuh"
#include "qmv.cuh"

namespace sb {

constexpr uint32_t kMoeRowsMax = 512;    // rows of one pass
constexpr uint32_t kMoeRowsChunk = 16;   // rows that share one reading of a weight record
constexpr uint32_t kRowsMeta = 12;       // floats beside a row's slice: 2^-s, three unused, the sums of its eight sub-blocks

// Input rows of a contraction, slice by slice (split_slice): f16 head and remainder of slice * 2^s, 2^-s and sums.
struct RowsOperand {
    __half *split = nullptr;   // [rows][2][columns]
    float *meta = nullptr;     // [rows][columns / 256][kRowsMeta]
    float *scale = nullptr;    // [rows] what a row's sums are multiplied with: the norm's scale (nullptr: nothing)
    uint32_t columns = 0;
};

// Spans of the attention's working memory for rows that see up to `rows` of the cache, which a token divides into `splits`.
inline uint32_t moe_rows_spans(uint32_t splits, uint32_t rows) { return std::min(splits, (rows + kMinSpan - 1u) / kMinSpan); }
// Floats of it that a row takes.
size_t moe_rows_part(uint32_t q_heads, uint32_t spans);

// Rows of a pass sorted by the expert they go to.  A tile is up to kMoeRowsChunk pairs (row, selection slot) of one expert.
struct MoeRowLists {
    uint32_t *ids = nullptr;     // [rows][active] selected experts
    float *probs = nullptr;      // [rows][active]
    float *scores = nullptr;     // [rows][experts]
    uint32_t *pairs = nullptr;   // [rows * active] row * active + slot, by expert
    uint32_t *tiles = nullptr;   // [0] their number; then {expert, first pair, pairs} each
    static uint32_t max_tiles(uint32_t rows, uint32_t active, uint32_t experts) {
        return (rows * active < experts ? rows * active : experts) + rows * active / kMoeRowsChunk;
    }
};

// out[row][r] = W x[row] for the rows of a pass (Q8_0, re-tiled).
stark_b200_status rows_q8_launch(const QMatrix *w, const RowsOperand &x, float *out, uint32_t rows, cudaStream_t stream);
// out[pair][block * w->rows + r] = W[expert + block * experts] x[pair / divisor] for the pairs of the lists and the bank's
// blocks (Q4_K, re-tiled; 2 blocks: a fused [gate; up] bank).
stark_b200_status rows_q4k_experts_launch(const QMatrix *w, uint32_t blocks, const RowsOperand &x, uint32_t divisor, float *out,
                                          const MoeRowLists &lists, uint32_t rows, uint32_t active, cudaStream_t stream);

// x = rows of the Q8_0 token table; the operand is rms_norm(x, w).
stark_b200_status moe_rows_embed_launch(const uint32_t *tokens, const uint8_t *table, float *x, const float *w, float eps,
                                        const RowsOperand &out, uint32_t rows, cudaStream_t stream);
// Per-head norm and rope of the query heads in place, keys and values into the cache rows first_pos ...
stark_b200_status moe_rows_heads_launch(float *qkv, const float *q_norm, const float *k_norm, float *keys, float *values,
                                        uint32_t q_heads, uint32_t kv_heads, float eps, float theta, uint32_t first_pos,
                                        uint32_t rows, cudaStream_t stream);
// Causal attention of the rows as operand rows, in spans as tokens divide the cache (`splits`); as many rows at once as `part`
// has room for.
stark_b200_status moe_rows_attention_launch(const float *qkv, const float *keys, const float *values, float *part, size_t part_floats,
                                            uint32_t q_heads, uint32_t kv_heads, uint32_t splits, uint32_t first_pos,
                                            const RowsOperand &out, uint32_t rows, cudaStream_t stream);
// x += update[row] (probs == nullptr) or the mixture of the row's expert outputs in selection order; the operand is
// rms_norm(x, w).
stark_b200_status moe_rows_add_norm_launch(float *x, const float *update, const float *probs, uint32_t active, const float *w,
                                           float eps, const RowsOperand &out, uint32_t rows, cudaStream_t stream);
// Scores of every expert over rms_norm(x, norm) (its scales beside the operand `normed`), selection and weights; the last row's
// selection also goes to last_ids [2 active] (ids, ids + experts).
stark_b200_status moe_rows_route_launch(const float *router, const float *x, const float *norm, const RowsOperand &normed,
                                        uint32_t experts, uint32_t active, const MoeRowLists &lists, uint32_t *last_ids,
                                        uint32_t rows, cudaStream_t stream);
stark_b200_status moe_rows_lists_launch(const MoeRowLists &lists, uint32_t rows, uint32_t active, uint32_t experts,
                                        cudaStream_t stream);
// The operand is silu(gate) * up of every pair.
stark_b200_status moe_rows_gate_launch(const float *gate_up, const RowsOperand &out, uint32_t pairs, cudaStream_t stream);

}  // namespace sb
