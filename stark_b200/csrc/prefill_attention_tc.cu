// Causal attention of a prompt pass on the sm_100a tensor cores (tcgen05.mma, accumulators in tensor memory):
// the same arithmetic as prefill_attention_kernel (attention_single_pass.rs:11-133: scores q.k in f32 scaled by
// 1/sqrt(d), softmax in f32, probabilities into the second product as bf16 hi + lo, output rounded to bf16), in the
// shape the tensor core wants.
//
// One CTA owns 128 rows of one query head and walks the keys in steps of 128 (two pages of the cache), in two passes:
//   pass 1   S = Q K^T per step, only to find every row's maximum; left out where the head norms bound the scores (PrefillAttnArgs)
//   pass 2   S again, P = exp2(S - max) (already final: no accumulator is ever rescaled), O += P V.
// The second look at the keys costs a quarter more tensor-core work and removes the read-modify-write of the output
// accumulator that an online softmax needs whenever a maximum moves.  Roles:
//   warps 0-7   softmax: thread = row (tensor-memory lane) x half of the step's keys; tcgen05.ld of S in 32-column
//               pieces, mask by the row's causal limit, maximum (pass 1) or exp2 / row sum / bf16 hi + lo stored to tensor
//               memory, the A operand of the second product (pass 2); at the end the read-out of O
//   warp 8      one thread: TMA loads -- Q once, then per step the K tile (and in pass 2 the V tile) as four
//               [64 keys x 64 dims] boxes straight from the paged cache
//   warp 9      owns tensor memory (S twice, so that step j + 1 is multiplied while step j is exponentiated, O and P);
//               one thread issues the MMAs: S = Q K^T with both operands K-major, O += P V with V as an MN-major
//               operand (its rows are keys, the contraction index), and commits them to the barriers
// Every wait is bounded; a wait that runs out sets the error word, the CTA drains and frees its tensor memory.
//
// What bounds it: the chain of a step through the softmax warps (about nine instructions for two probabilities, two warps a scheduler),
// beside 1 536 tensor-core cycles.  4 096 rows of the 8b shape, a layer: 571 000 cycles with P in shared memory and two passes, 524 000 with P in
// tensor memory, masks out of line and sums in four chains, 515 000 with paired f32 instructions, 398 000 in one pass (336 -> 234 us).
// Three stages instead of two and four score tiles in pass 1 changed nothing alone.
//
// Few rows over many keys (SPLIT): 16 heads of one row block are 16 CTAs that walk the whole cache one after another.  The
// keys are then divided among the CTAs of a cluster: they exchange the rows' maxima between the passes, so that every CTA's
// probabilities are final too, and add up accumulators and row sums at the end, in rank order.
#include <cuda.h>

#include <algorithm>

#include "context.cuh"
#include "device_math.cuh"
#include "prefill.cuh"
#include "softmax_tc.cuh"
#include "tc05.cuh"
#include "thin_tile.cuh"
#include "tunables.cuh"

namespace sb {

namespace {

constexpr uint32_t kBox = 64u * 128u;       // [64 rows][64 elements] bf16 in 128-byte swizzled lines: 8 KB
constexpr uint32_t kBlock = 2u * kBox;      // 128 rows x 64 elements: 16 KB
constexpr uint32_t kOperand = 2u * kBlock;  // 128 x 128: 32 KB
constexpr uint32_t kSoftmaxWarps = 8, kTcThreads = (kSoftmaxWarps + 2u) * 32u;
// shared memory: Q | K, three stages | V, three stages | barriers (512 B) | exchange words [2][128] f32
constexpr uint32_t kDepth = 3;
constexpr uint32_t kQOff = 0, kKOff = kOperand, kVOff = kKOff + kDepth * kOperand, kBarOff = kVOff + kDepth * kOperand;
constexpr uint32_t kSumsOff = kVOff + kOperand;  // SPLIT, at the end: the row sums, behind the shares of O
constexpr uint32_t kTcSmem = kBarOff + 2048u /* barriers, exchange words */ + 1024u /* alignment */;
constexpr uint32_t kTcTmemColumns = 512;  // S twice (2 x 128), O (128), P as pairs of bf16: 64 columns hi, 64 lo
constexpr uint32_t kPColumn = 384;
// D f32, A and B bf16, M 128, N 128; the second product takes B (V) MN-major
constexpr uint32_t kIdescS = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kIdescPV = kIdescS | (1u << 16);

// A bound (in powers of two) up to which it may stand in for a row's maximum: probabilities then lie above 2^-96, a row's largest too,
// so that every one that counts beside it is a normal f32 -- the same relative precision as behind the maximum itself.
constexpr float kMostBound = 48.0f;

struct TcAttnParams {
    uint16_t *out;
    const int32_t *block_table;
    uint32_t m, first_pos, q_heads, kv_heads, gqa, num_blocks;
    float scale_log2;  // log2(e) / sqrt(d)
    float bound;       // no score times scale_log2 is larger (0: unknown); it stands in for the rows' maxima
    uint32_t *error_word;
    uint32_t stop_after;  // 0 whole kernel; 1 set-up and tensor memory only; 2 pass 1 only (no MN-major operand)
};

constexpr uint32_t kPartPitch = 128u + 4u;  // floats between the rows of a CTA's share of O, in place of the K and V stages

template <bool SPLIT>
__global__ void __launch_bounds__(kTcThreads, 1)
prefill_attention_tc_kernel(const __grid_constant__ CUtensorMap q_map, const __grid_constant__ CUtensorMap k_map,
                            const __grid_constant__ CUtensorMap v_map, const TcAttnParams p) {
    extern __shared__ uint8_t tc_smem_raw[];
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(tc_smem_raw) + 1023u) & ~(uintptr_t)1023u);
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kBarOff);
    uint64_t *q_full = bars, *s_full = bars + 1, *s_free = bars + 3, *p_full = bars + 5, *p_free = bars + 6, *o_full = bars + 7;
    uint64_t *m_full = bars + 8, *m_free = bars + 12;  // pass 1: all of tensor memory is four score tiles
    uint64_t *k_full = bars + 16, *k_empty = k_full + kDepth, *v_full = k_empty + kDepth, *v_empty = v_full + kDepth;
    uint64_t *a_full = v_empty + kDepth, *a_empty = a_full + 2u * kDepth;  // pass 1: the K and V stages together are one ring of K tiles
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(a_empty + 2u * kDepth);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    float *exchange = reinterpret_cast<float *>(smem + kBarOff + 512u);  // what the two warps of a row tell each other
    float *part_sums = reinterpret_cast<float *>(smem + kSumsOff);  // SPLIT: the row sums [2][128], at the end

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t head = blockIdx.x, kvh = head / p.gqa;
    // causal: late row blocks read the most keys, so they are issued first
    const uint32_t row0 = (gridDim.y - 1u - blockIdx.y) * 128u;
    const uint32_t last_row = min(p.m, row0 + 128u) - 1u;
    const uint32_t all_steps = (p.first_pos + last_row) / 128u + 1u;
    const uint32_t split = SPLIT ? gridDim.z : 1u, rank = SPLIT ? blockIdx.z : 0u;  // the cluster is the grid's z
    const uint32_t step0 = all_steps * rank / split, steps = all_steps * (rank + 1u) / split - step0;  // possibly none
    const uint32_t passes = p.stop_after == 2u ? 1u : 2u, first_steps = p.bound > 0.0f ? 0u : steps;  // of pass 1

    if (tid == 0) {
        mbar_init(q_full, 1);
        for (uint32_t s = 0; s < 2; ++s) {
            mbar_init(&s_full[s], 1);
            mbar_init(&s_free[s], kSoftmaxWarps);
        }
        for (uint32_t s = 0; s < 4; ++s) {
            mbar_init(&m_full[s], 1);
            mbar_init(&m_free[s], kSoftmaxWarps);
        }
        for (uint32_t s = 0; s < kDepth; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (uint32_t s = 0; s < 2u * kDepth; ++s) {
            mbar_init(&a_full[s], 1);
            mbar_init(&a_empty[s], 1);
        }
        mbar_init(p_full, kSoftmaxWarps);
        mbar_init(p_free, 1);
        mbar_init(o_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == kSoftmaxWarps + 1u) tmem_alloc(tmem_slot, kTcTmemColumns);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();
    pdl_wait();  // the rows and the cache rows appended for them
    // the maxima are the softmax warps' business: the other two arrive ahead and collect the barrier at their end
    const bool bystander = SPLIT && warp >= kSoftmaxWarps && !(p.bound > 0.0f);
    if (bystander) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    auto give_up = [&]() {
        *abort_flag = 1;
        atomicOr(p.error_word, kErrMbarTimeout);
    };

    if (p.stop_after == 1u) {
        // nothing between allocation and release
    } else if (warp == kSoftmaxWarps) {
        // ------------------------------------------------ tiles by TMA
        if (lane == 0) {
            mbar_arrive_expect_tx(q_full, kOperand);
            tma_load_2d(smem + kQOff, &q_map, head * 128u, row0, q_full);
            tma_load_2d(smem + kQOff + kBlock, &q_map, head * 128u + 64u, row0, q_full);
            // a page past the allocated ones is read out of bounds: the copy engine fills zeros
            auto page_row = [&](uint32_t page) -> uint32_t {
                return page < p.num_blocks ? ((uint32_t)p.block_table[page] * p.kv_heads + kvh) * kPageTokens
                                           : p.num_blocks * p.kv_heads * kPageTokens;
            };
            auto load_tile = [&](uint8_t *dst, const CUtensorMap *map, uint32_t y0, uint32_t y1, uint64_t *bar) {
                mbar_arrive_expect_tx(bar, kOperand);
                tma_load_2d(dst, map, 0u, y0, bar);
                tma_load_2d(dst + kBox, map, 0u, y1, bar);
                tma_load_2d(dst + kBlock, map, 64u, y0, bar);
                tma_load_2d(dst + kBlock + kBox, map, 64u, y1, bar);
            };
            uint32_t ks = 0, kph = 1, vs = 0, vph = 1;  // a fresh barrier passes a wait on parity 1
            bool ok = true;
            {   // pass 1: K tiles only
                uint32_t as = 0, aph = 1;
                for (uint32_t j = 0; j < first_steps && ok; ++j) {
                    if (!(ok = mbar_wait_bounded(&a_empty[as], aph, abort_flag))) break;
                    load_tile(smem + kKOff + as * kOperand, &k_map, page_row(2u * (step0 + j)), page_row(2u * (step0 + j) + 1u), &a_full[as]);
                    if (++as == 2u * kDepth) as = 0, aph ^= 1u;
                }
                // pass 2 loads into the same memory: every stage's last pass-1 tile must have been multiplied
                for (uint32_t s = 0; s < 2u * kDepth && ok && passes == 2u; ++s) {
                    const uint32_t uses = first_steps > s ? (first_steps - s + 2u * kDepth - 1u) / (2u * kDepth) : 0u;
                    if (uses) ok = mbar_wait_bounded(&a_empty[s], (uses - 1u) & 1u, abort_flag);
                }
            }
            for (uint32_t pass = 1; pass < passes && ok; ++pass) {
                for (uint32_t j = 0; j < steps && ok; ++j) {
                    const uint32_t y0 = page_row(2u * (step0 + j)), y1 = page_row(2u * (step0 + j) + 1u);
                    if (!(ok = mbar_wait_bounded(&k_empty[ks], kph, abort_flag))) break;
                    load_tile(smem + kKOff + ks * kOperand, &k_map, y0, y1, &k_full[ks]);
                    if (++ks == kDepth) ks = 0, kph ^= 1u;
                    if (pass == 1u) {
                        if (!(ok = mbar_wait_bounded(&v_empty[vs], vph, abort_flag))) break;
                        load_tile(smem + kVOff + vs * kOperand, &v_map, y0, y1, &v_full[vs]);
                        if (++vs == kDepth) vs = 0, vph ^= 1u;
                    }
                }
            }
            if (!ok) give_up();
        }
    } else if (warp == kSoftmaxWarps + 1u) {
        // ------------------------------------------------ tensor-core issue
        if (lane == 0) {
            bool ok = mbar_wait_bounded(q_full, 0, abort_flag);
            uint32_t ks = 0, kph = 0, vs = 0, vph = 0, g = 0;  // g counts score tiles: buffer g & 1
            const uint32_t q_addr = smem_u32(smem + kQOff);
            auto scores = [&](uint64_t *full, uint64_t *empty, uint32_t slots, uint64_t *tile_full, uint64_t *tile_free, uint32_t tiles) {
                const uint32_t b = g % tiles, use = g / tiles;
                ok = ok && mbar_wait_bounded(&full[ks], kph, abort_flag) &&
                     mbar_wait_bounded(&tile_free[b], (use & 1u) ^ 1u, abort_flag);  // the softmax warps are done with use - 1
                if (!ok) return;
                tc_fence_after();
                const uint32_t k_addr = smem_u32(smem + kKOff + ks * kOperand);
#pragma unroll
                for (uint32_t i = 0; i < 8u; ++i) {  // 16 dims a step; 64 dims a block
                    const uint32_t at = (i >> 2) * kBlock + (i & 3u) * 32u;
                    umma_f16(tmem_base + b * 128u, smem_desc_sw128(q_addr + at), smem_desc_sw128(k_addr + at), kIdescS,
                             i != 0u ? 1u : 0u);
                }
                umma_commit(&empty[ks]);
                umma_commit(&tile_full[b]);
                if (++ks == slots) ks = 0, kph ^= 1u;
                ++g;
            };
            for (uint32_t j = 0; j < first_steps && ok; ++j) scores(a_full, a_empty, 2u * kDepth, m_full, m_free, 4u);
            ks = 0, kph = 0, g = 0;
            if (passes == 2u) {
                for (uint32_t b = 0; b < 4u && ok; ++b)  // O and P take the place of score tiles that have been read
                    if (first_steps > b) ok = mbar_wait_bounded(&m_free[b], ((first_steps - b + 3u) / 4u - 1u) & 1u, abort_flag);
                tc_fence_after();
                for (uint32_t j = 0; j <= steps && ok; ++j) {
                    if (j < steps) scores(k_full, k_empty, kDepth, s_full, s_free, 2u);  // step j is multiplied while step j - 1 is exponentiated
                    if (j == 0u || !ok) continue;
                    const uint32_t t = j - 1u;
                    ok = mbar_wait_bounded(p_full, t & 1u, abort_flag) && mbar_wait_bounded(&v_full[vs], vph, abort_flag);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t v_addr = smem_u32(smem + kVOff + vs * kOperand);
#pragma unroll
                    for (uint32_t i = 0; i < 8u; ++i) {  // 16 keys a step
                        const uint64_t vdesc = smem_desc_sw128_mn(v_addr + i * 2048u, kBlock);
                        umma_f16_ts(tmem_base + 256u, tmem_base + kPColumn + 8u * i, vdesc, kIdescPV, (t | i) != 0u ? 1u : 0u);
                        umma_f16_ts(tmem_base + 256u, tmem_base + kPColumn + 64u + 8u * i, vdesc, kIdescPV, 1u);
                    }
                    umma_commit(&v_empty[vs]);
                    umma_commit(p_free);
                    if (++vs == kDepth) vs = 0, vph ^= 1u;
                }
            }
            if (!ok) give_up();
            umma_commit(o_full);  // also on the give-up path: the softmax warps wait on it
        }
    } else {
        // ------------------------------------------------ softmax: thread = row (tensor-memory lane) x half of the keys
        // Warps w and w + 4 share the 32 rows of lane group w & 3 (a warp reaches only the lanes of its index modulo
        // 4) and take the step's keys 0-63 and 64-127: twice the warps that issue exponentials and conversions.
        const uint32_t sub = warp & 3u, half = warp >> 2;
        const uint32_t r = 32u * sub + lane, row = row0 + r;
        const uint32_t pos = p.first_pos + min(row, p.m - 1u);  // last key this row may see
        const uint32_t lanes = (32u * sub) << 16, col0 = 64u * half;
        float mrow = -INFINITY;
        uint32_t g = 0;
        bool ok = true;
        for (uint32_t j = 0; j < first_steps && ok; ++j) {
            const uint32_t b = j & 3u;
            if (!(ok = mbar_wait_bounded(&m_full[b], (j >> 2) & 1u, abort_flag))) break;
            tc_fence_after();
            uint32_t v[2][32];
#pragma unroll
            for (uint32_t c = 0; c < 2u; ++c) tmem_ld_32x32_issue(tmem_base + lanes + b * 128u + col0 + 32u * c, v[c]);
#pragma unroll
            for (uint32_t c = 0; c < 2u; ++c) {
                tmem_ld_wait_32(v[c]);
                hide_keys(v[c], (step0 + j) * 128u + col0 + 32u * c, pos);
                mrow = fmaxf(mrow, largest(v[c]) * p.scale_log2);  // the scale is positive: it commutes with the maximum
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&m_free[b]);
        }
        // the row's maximum over both halves of the keys
        if (p.bound > 0.0f) {
            mrow = p.bound;
        } else {
            exchange[half * 128u + r] = mrow;
            if constexpr (SPLIT) {
                __syncwarp();
                thin_cluster_sync();
                mrow = thin_fold(&exchange[r], split, mrow, [](float a, float b) { return fmaxf(a, b); });
            } else {
                named_bar_sync(1, kSoftmaxWarps * 32u);
                mrow = fmaxf(mrow, exchange[(half ^ 1u) * 128u + r]);
                named_bar_sync(1, kSoftmaxWarps * 32u);  // everybody has read: the words are free for the row sums
            }
        }
        float l = 0.0f;
        float2 sums[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
        if (passes == 2u) {
            for (uint32_t j = 0; j < steps && ok; ++j, ++g) {
                const uint32_t b = g & 1u;
                if (!(ok = mbar_wait_bounded(&s_full[b], (g >> 1) & 1u, abort_flag))) break;
                tc_fence_after();
                uint32_t v[2][32], hi[2][16], lo[2][16];
                tmem_ld_32x32_issue(tmem_base + lanes + b * 128u + col0, v[0]);
                tmem_ld_32x32_issue(tmem_base + lanes + b * 128u + col0 + 32u, v[1]);
                tmem_ld_wait_32(v[0]);
                tmem_ld_wait_32(v[1]);
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&s_free[b]);
#pragma unroll
                for (uint32_t c = 0; c < 2u; ++c) {
                    hide_keys(v[c], (step0 + j) * 128u + col0 + 32u * c, pos);
                    probabilities(v[c], p.scale_log2, mrow, sums, hi[c], lo[c]);
                }
                // the previous step's second product must have read P before it is overwritten; the warp goes on as one
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(p_free, (j & 1u) ^ 1u, abort_flag));
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (uint32_t c = 0; c < 2u; ++c) {  // 32 keys = 16 columns of pairs
                    tmem_st_32x16(tmem_base + lanes + kPColumn + half * 32u + c * 16u, hi[c]);
                    tmem_st_32x16(tmem_base + lanes + kPColumn + 64u + half * 32u + c * 16u, lo[c]);
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_full);
            }
            l = (sums[0].x + sums[0].y) + (sums[1].x + sums[1].y);
            // the row's sum over both halves
            if constexpr (!SPLIT) {
                exchange[half * 128u + r] = l;
                named_bar_sync(1, kSoftmaxWarps * 32u);
                l = exchange[r] + exchange[128u + r];
            }
            // ---- read-out of O: this warp's 64 of the 128 dims
            const bool o_ok = mbar_wait_bounded(o_full, 0, abort_flag);
            if (!o_ok && lane == 0) atomicOr(p.error_word, kErrMbarTimeout);
            tc_fence_after();
            if constexpr (SPLIT) part_sums[half * 128u + r] = l;  // every read of P has completed
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
            uint16_t *dst = p.out + ((size_t)row * p.q_heads + head) * kHeadDim + col0;
            uint32_t v[2][32];
#pragma unroll
            for (uint32_t c = 0; c < 2u; ++c) tmem_ld_32x32_issue(tmem_base + lanes + 256u + col0 + 32u * c, v[c]);
#pragma unroll
            for (uint32_t c = 0; c < 2u; ++c) {
                tmem_ld_wait_32(v[c]);
                if constexpr (SPLIT) {  // every read of the stages has completed
                    if (!steps)
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[c][i] = 0u;
                    thin_store(reinterpret_cast<float *>(smem + kKOff) + r * kPartPitch + col0 + 32u * c, v[c]);
                } else if (row < p.m && o_ok && ok) {
                    uint32_t packed[16];
#pragma unroll
                    for (int i = 0; i < 32; i += 2)
                        packed[i >> 1] = f32x2_to_bf16x2(__uint_as_float(v[c][i]) * inv, __uint_as_float(v[c][i + 1]) * inv);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        reinterpret_cast<uint4 *>(dst + 32u * c)[q] =
                            make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
                }
            }
        }
        if (!ok && lane == 0) give_up();
    }
    tc_fence_before();
    if constexpr (SPLIT) {
        __syncwarp();
        if (bystander) asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        thin_cluster_sync();
        const uint32_t rows_each = 128u / split;
        const float *part = reinterpret_cast<const float *>(smem + kKOff);
#pragma unroll 1
        for (uint32_t i = tid; i < rows_each * 32u; i += kTcThreads) {
            const uint32_t r = rank * rows_each + i / 32u, column = i % 32u * 4u;
            if (row0 + r >= p.m) break;
            const float l = thin_fold(&part_sums[r], split, 0.0f, [](float a, float b) { return a + b; });
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
            const float4 o = thin_sum(part + r * kPartPitch + column, split);
            *reinterpret_cast<uint2 *>(p.out + ((size_t)(row0 + r) * p.q_heads + head) * kHeadDim + column) =
                make_uint2(f32x2_to_bf16x2(o.x * inv, o.y * inv), f32x2_to_bf16x2(o.z * inv, o.w * inv));
        }
        __syncwarp();
        thin_cluster_leave();
    } else {
        __syncthreads();
    }
    if (warp == kSoftmaxWarps + 1u) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTcTmemColumns);
    }
}

}  // namespace

bool prefill_attention_tc_supports(const PrefillAttnArgs &a) {
    return a.num_blocks != 0 && a.m > 16u && a.kv_heads != 0 && a.q_heads % a.kv_heads == 0 &&
           (reinterpret_cast<uintptr_t>(a.qkv) & 15u) == 0 && encode_tiled() != nullptr;
}

stark_b200_status prefill_attention_tc_launch(const PrefillAttnArgs &a, cudaStream_t stream) {
    if (!a.qkv || !a.kv.keys || !a.kv.values || !a.block_table || !a.out || a.m == 0) return STARK_B200_INVALID_ARGUMENT;
    if (!prefill_attention_tc_supports(a)) return STARK_B200_UNSUPPORTED;
    DeviceContext *ctx = device_context();
    if (!ctx) return STARK_B200_DEVICE_FAILURE;
    EncodeTiledFn encode = encode_tiled();
    const uint32_t heads = a.q_heads + 2u * a.kv_heads;
    CUtensorMap q_map, k_map, v_map;
    const cuuint32_t elem[2] = {1u, 1u};
    {
        // the query heads of the pass's rows: [m][heads * 128], the q heads first in every row
        const cuuint64_t dims[2] = {(cuuint64_t)a.q_heads * kHeadDim, a.m};
        const cuuint64_t strides[1] = {(cuuint64_t)heads * kHeadDim * 2u};
        const cuuint32_t box[2] = {64u, 128u};
        if (encode(&q_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t *>(a.qkv), dims, strides, box, elem,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return STARK_B200_DEVICE_FAILURE;
    }
    {
        // the paged cache of the layer as rows of one head's 128 dims: [(page, kv head, token)][128]
        const cuuint64_t dims[2] = {kHeadDim, (cuuint64_t)a.num_blocks * a.kv_heads * kPageTokens};
        const cuuint64_t strides[1] = {(cuuint64_t)kHeadDim * 2u};
        const cuuint32_t box[2] = {64u, kPageTokens};
        for (int which = 0; which < 2; ++which)
            if (encode(which ? &v_map : &k_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, which ? a.kv.values : a.kv.keys, dims,
                       strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                       CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return STARK_B200_DEVICE_FAILURE;
    }
    TcAttnParams p{};
    p.out = a.out;
    p.block_table = a.block_table;
    p.m = a.m;
    p.first_pos = a.first_pos;
    p.q_heads = a.q_heads;
    p.kv_heads = a.kv_heads;
    p.gqa = a.q_heads / a.kv_heads;
    p.num_blocks = a.num_blocks;
    p.scale_log2 = a.scale * 1.4426950408889634f;
    p.bound = tunables().prefill_attn_tc == 1u && a.score_bound > 0.0f && a.score_bound * 1.4426950408889634f <= kMostBound ? a.score_bound * 1.4426950408889634f : 0.0f;
    p.error_word = ctx->error_word;
    p.stop_after = tunables().attn_tc_stop_after;
    // 77 rows behind 1 024 (16 heads, 28 layers): 2.87 ms with one CTA a row block, 2.72 with two, 2.50 with four, 2.86 with eight
    // (whose 16 clusters do not fit at once).
    const uint32_t split = p.stop_after ? 1u : thin_split((a.whole_heads ? a.whole_heads : a.q_heads) * ((a.m + 127u) / 128u), (a.first_pos + a.m - 1u) / 128u + 1u);
    const auto kernel = split > 1u ? prefill_attention_tc_kernel<true> : prefill_attention_tc_kernel<false>;
    static SmemOptIn once[2];
    if (stark_b200_status s = ensure_dynamic_smem(kernel, (int)kTcSmem, once[split > 1u])) return s;
    return thin_launch(kernel, dim3(a.q_heads, (a.m + 127u) / 128u, split), kTcThreads, kTcSmem, stream, q_map, k_map, v_map, p);
}

}  // namespace sb
