// Prompt rows of the routed-expert decoder (moe_rows.cu): the f32 conventions of a token (moe_model.cu), many rows at once.
#pragma once
#include "qmv.cuh"

namespace sb {

constexpr uint32_t kMoeRowsMax = 512;    // rows of one pass
constexpr uint32_t kMoeRowsWidest = 12288;  // columns of the widest row
constexpr uint32_t kMoeRowsChunk = 16;   // rows that share one reading of a weight record

// Input rows of a contraction: every row as f16 head and f16 remainder of row * 2^s (s by the row's largest element),
// 2^-s, and the sums of 32 consecutive elements of row * 2^s.
struct RowsOperand {
    __half *split = nullptr;    // [rows][2][columns]
    float *unscale = nullptr;   // [rows]
    float *sums = nullptr;      // [rows][columns / 32]
    uint32_t columns = 0;
    static size_t bytes(size_t rows, size_t columns) { return rows * (columns * 4u + columns / 8u + 4u); }
};

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
                                        uint32_t q_heads, uint32_t kv_heads, uint32_t dim, float eps, float theta,
                                        uint32_t first_pos, uint32_t rows, cudaStream_t stream);
// Merges the spans of every head (moe_attention_merge_kernel) and splits the row.
stark_b200_status moe_rows_merge_launch(const float *part, uint32_t heads, uint32_t splits, const RowsOperand &out,
                                        uint32_t rows, cudaStream_t stream);
// x += update[row] (probs == nullptr) or the mixture of the row's expert outputs in selection order; then, with w, the norm as
// an operand and, where `normed` is given, as f32 rows.
stark_b200_status moe_rows_add_norm_launch(float *x, const float *update, const float *probs, uint32_t active, const float *w,
                                           float eps, float *normed, const RowsOperand &out, uint32_t rows, uint32_t hidden,
                                           cudaStream_t stream);
// Scores of every expert, selection and weights; the last row's selection also goes to last_ids [2 active] (ids, ids + experts).
stark_b200_status moe_rows_route_launch(const float *router, const float *normed, uint32_t hidden, uint32_t experts,
                                        uint32_t active, const MoeRowLists &lists, uint32_t *last_ids, uint32_t rows,
                                        cudaStream_t stream);
stark_b200_status moe_rows_lists_launch(const MoeRowLists &lists, uint32_t rows, uint32_t active, uint32_t experts,
                                        cudaStream_t stream);
// The operand is silu(gate) * up of every pair.
stark_b200_status moe_rows_gate_launch(const float *gate_up, uint32_t inter, const RowsOperand &out, uint32_t pairs,
                                       cudaStream_t stream);

}  // namespace sb
