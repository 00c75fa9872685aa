// What a token of the routed-expert decoder launches per layer where its matrices are re-tiled (moe_token.cu).
#pragma once
#include "qmv.cuh"

namespace sb {

constexpr uint32_t kEpSkip = 0xffffffffu;  // expert id of a selection slot another rank owns

// Whether the token kernels take these matrices: formats of 16 x 256 records, rows that fit the warps of a CTA.
bool token_q8_supports(const QMatrix *w);
bool token_gate_up_supports(const QMatrix *w);
bool token_down_supports(const QMatrix *w);

// out = W rms_norm(x, norm) where norm is given, else W x; with `residual` (which may be `out`), that + residual.
stark_b200_status token_q8_launch(const QMatrix *w, const float *x, const float *norm, float eps, const float *residual,
                                  float *out, bool pdl, cudaStream_t stream);

// Causal attention of the token at *position over spans of the cache, and the spans' merge.  `raw`: qkv holds the projection
// as the matvec left it, and the kernel norms and rotates the heads and writes the cache row; else both are done.
stark_b200_status token_attention_launch(const uint32_t *position, const float *qkv, bool raw, float *keys, float *values,
                                         float *part, uint32_t splits, uint32_t q_heads, uint32_t kv_heads, uint32_t context,
                                         const float *q_norm, const float *k_norm, float eps, float theta, bool pdl,
                                         cudaStream_t stream);
stark_b200_status token_merge_launch(const uint32_t *position, const float *part, float *out, uint32_t splits, uint32_t q_heads,
                                     uint32_t context, bool pdl, cudaStream_t stream);

// scores[e] = router[e] . rms_norm(x, norm)
stark_b200_status token_router_launch(const float *router, const float *x, const float *norm, float eps, float *scores,
                                      uint32_t hidden, uint32_t experts, bool pdl, cudaStream_t stream);

// The selection over the scores (top-k by value, lower index first; softmax over the selected) and, for every selected expert,
// act[slot] = silu(gate) * up of rms_norm(x, norm).  ids [2 active] and probs [active] as the older selection leaves them.
struct TokenSelection {
    const float *scores;
    uint32_t experts, active;
    uint32_t *ids;
    float *probs;
    uint32_t *ids_global;           // expert parallel: the selection in the model's numbering, else nullptr
    uint32_t ep_first, ep_local;    // expert parallel: the experts of this rank
};
stark_b200_status token_gate_up_launch(const QMatrix *w, const TokenSelection &sel, const float *x, const float *norm, float eps,
                                       float *act, bool pdl, cudaStream_t stream);
// out[slot] = down[ids[slot]] act[slot]
stark_b200_status token_down_launch(const QMatrix *w, const uint32_t *ids, uint32_t active, const float *act, float *out, bool pdl,
                                    cudaStream_t stream);
// x += sum_r probs[r] * rows[r], r ascending from zero; probs == nullptr: x += rows.
stark_b200_status token_mix_launch(float *x, const float *rows, const float *probs, uint32_t active, uint32_t hidden, bool pdl,
                                   cudaStream_t stream);

}  // namespace sb
