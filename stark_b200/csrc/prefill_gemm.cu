// Y[M, N] = X[M, K] W[N, K]^T for a 4-bit affine group-64 matrix, many rows at a time: the prompt-chunk
// contraction of the token loop on the sm_100a tensor cores (tcgen05.mma, accumulators in tensor memory).
//
// One CTA owns a tile of 256 rows x 256 output features and walks K in steps of one quantization group (64):
//   warp 0      one thread: TMA loads of the two 128-row activation boxes of the step (bf16, 128-byte swizzle)
//   warp 1      allocates tensor memory (all 512 columns: two 128 x 256 f32 accumulators); one thread issues
//               2 x 4 tcgen05.mma (128 x 256 x 16) per step and commits them to the barrier that frees the stage
//   warps 2-9   the dequantizing prologue: warp d turns two records (16 features x 64 columns, 576 bytes each,
//               read straight from the re-tiled matrix the matvec kernels stream) into bf16 rows of the B operand --
//               codes become exact bf16 integers (shift, lop3 and one bf16 subtract per pair), then
//               bf16(scale * q + bias) in one bf16 FMA per pair -- written in the swizzled K-major layout the
//               tensor core reads.  The same warps run the epilogue: tcgen05.ld of the accumulators, bf16 rounding,
//               residual add or SwiGLU, 64-byte row segments to global memory.
// Rounding points are those of the one-row path (f32 accumulation, one bf16 rounding of the product, then the
// epilogue's own roundings); the operand W is rounded to bf16, the activations' type, as the reference's own
// tiled GEMM does, where the one-row path keeps scale * q + bias in f32: inside the per-operator tolerance.
// The tile is as wide as tensor memory allows because the activation tile is what the step re-reads from L2 (once
// per feature tile) and what the tensor core re-reads from shared memory: at 256 features a step moves 41 KB from
// L2 and 160 KB through shared memory for 1024 tensor-core cycles (156 B/cycle of the 128 B/cycle an SM has, the
// binding limit), at 128 features 37 KB and 112 KB for 512 cycles.
// Every wait is bounded; a wait that runs out sets the error word, the CTA drains and frees its tensor memory.
#include <cuda.h>

#include <algorithm>

#include "a4_record.cuh"
#include "device_math.cuh"
#include "pair_gemm.cuh"
#include "prefill.cuh"
#include "tc05.cuh"
#include "thin_tile.cuh"
#include "tunables.cuh"

namespace sb {

namespace {

constexpr uint32_t kBM = 256, kBN = 256, kBK = 64;
constexpr uint32_t kStages = 3;
constexpr uint32_t kABox = 128u * 128u;            // one 128-row x 64-column bf16 box: 16 KB
constexpr uint32_t kAStage = 2u * kABox;           // 32 KB
constexpr uint32_t kBStage = kBN * 128u;           // 32 KB
constexpr uint32_t kStageBytes = kAStage + kBStage;
constexpr uint32_t kDequantWarps = 8;
constexpr uint32_t kGemmThreads = (2u + kDequantWarps) * 32u;
constexpr uint32_t kTmemColumns = 512;             // two 128 x 256 f32 accumulators: all of tensor memory
constexpr uint32_t kGemmSmem = kStages * kStageBytes + 1024u /* alignment */ + 256u /* barriers */;

struct GemmParams {
    const uint8_t *w;
    uint32_t row_tiles, groups, rows;
    uint32_t m;
    uint16_t *out;
    uint32_t ld_out;
    uint32_t epilogue;
    uint32_t *error_word;
    // tensor parallel: the same place in the other ranks' row buffers (peer mappings); the epilogue stores every
    // output segment there as well, tile by tile, so the all-gather of the column slices rides under the contraction
    uint16_t *peer_out[kMaxExchangeRanks];
    uint32_t peers;
    uint32_t stop_after;  // 0: the whole kernel.  1: set-up and tensor-memory allocation only; 2: + operand staging
                          // (no tensor-core work); 3: + tcgen05.mma (accumulators not read).  A bring-up aid: a
                          // fault in one kind of instruction is located by the first stage that shows it.
};

// Instruction descriptor: D f32, A bf16 (activations), B bf16 (dequantized weights), both K-major, M 128, N 256.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kBN >> 3) << 17) | ((128u >> 4) << 24);

// One record (16 features x 64 columns) into rows [16 d, 16 d + 16) of the B stage: two 16-byte chunks of a lane in each of its two rows.
__device__ inline void dequant_record_to_smem(const RecordRegs &r, uint8_t *b_stage, uint32_t d, uint32_t lane) {
    const uint32_t g = lane >> 2, t = lane & 3u;
    uint4 v[4];
    dequant_record(r, v);
    // row R of the stage starts at R * 128; its 16-byte chunk c sits at chunk position c ^ (R & 7)
    const uint32_t r_lo = 16u * d + g, r_hi = r_lo + 8u;  // both have (R & 7) == g
    uint8_t *p_lo = b_stage + r_lo * 128u, *p_hi = b_stage + r_hi * 128u;
    const uint32_t c0 = ((2u * t) ^ g) * 16u, c1 = ((2u * t + 1u) ^ g) * 16u;
    *reinterpret_cast<uint4 *>(p_lo + c0) = v[0];
    *reinterpret_cast<uint4 *>(p_lo + c1) = v[1];
    *reinterpret_cast<uint4 *>(p_hi + c0) = v[2];
    *reinterpret_cast<uint4 *>(p_hi + c1) = v[3];
}

// 32 columns of a warp's 32 accumulator rows, from storage row f0 of the matrix: bf16 rounding, residual add or SwiGLU, to this rank's
// buffer and the other ranks'.  `scratch`: the warp's own 32 rows of 80 bytes.
__device__ __forceinline__ void store_block(const GemmParams &p, uint32_t row, uint32_t f0, const uint32_t (&acc)[32], uint8_t *scratch,
                                            uint32_t lane, bool acc_ok) {
    const bool row_ok = row < p.m;
    if (p.epilogue == kEpiSwiGlu) {
        // storage tiles alternate up / gate (pair_halves): columns 0-15 up rows, 16-31 the gate rows
        // of the same logical rows.  gated_act_mul.rs:80-95: silu in f32 -> bf16, product -> bf16
        uint32_t packed[8];
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            float o2[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float up = bf16_round(__uint_as_float(acc[i + e]));
                const float gate = bf16_round(__uint_as_float(acc[16 + i + e]));
                const float activated = bf16_round(gate / (1.0f + expf(-1.0f * gate)));
                o2[e] = up * activated;
            }
            packed[i >> 1] = f32x2_to_bf16x2(o2[0], o2[1]);
        }
        const uint32_t o0 = (f0 / 32u) * 16u;  // logical row of the pair
        if (row_ok && o0 + 16u <= p.rows / 2u) {
            uint4 *dst = reinterpret_cast<uint4 *>(p.out + (size_t)row * p.ld_out + o0);
            dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
        }
        if (p.peers && acc_ok) {
            // The same 32 x 16 block to the other ranks.  A lane holds 32 bytes of ITS row: stored from here, one
            // instruction would touch 32 rows with 16 bytes each, and over NVLink every such fragment is a packet
            // of its own.  Through the warp's scratch rows (48-byte pitch: conflict-free) the lanes regroup
            // so that two neighbours write one row's 32 contiguous bytes.
            uint4 *mine = reinterpret_cast<uint4 *>(scratch + lane * 48u);
            mine[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            mine[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
            __syncwarp();
#pragma unroll
            for (uint32_t j = 0; j < 2u; ++j) {
                const uint32_t r = 16u * j + (lane >> 1), q = lane & 1u;
                const uint4 v = *reinterpret_cast<const uint4 *>(scratch + r * 48u + q * 16u);
                const uint32_t prow = row - lane + r;
                if (prow < p.m && o0 + 16u <= p.rows / 2u) {
                    const size_t at = (size_t)prow * p.ld_out + o0 + q * 8u;
#pragma unroll
                    for (uint32_t k = 0; k + 1u < kMaxExchangeRanks; ++k) {
                        if (k >= p.peers) break;
                        *reinterpret_cast<uint4 *>(p.peer_out[k] + at) = v;
                    }
                }
            }
            __syncwarp();
        }
    } else {
        const bool cols_ok = f0 + 32u <= p.rows;
        uint16_t *dst16 = p.out + (size_t)row * p.ld_out + f0;
        uint32_t packed[16];
        if (p.epilogue == kEpiResidual && row_ok && cols_ok) {
            const uint4 *src = reinterpret_cast<const uint4 *>(dst16);
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4) {
                const uint4 rv = src[q4];
                const uint32_t rr[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = q4 * 8 + e * 2;
                    const uint32_t y2 = f32x2_to_bf16x2(__uint_as_float(acc[i]), __uint_as_float(acc[i + 1]));
                    packed[q4 * 4 + e] = f32x2_to_bf16x2(__uint_as_float(y2 << 16) + __uint_as_float(rr[e] << 16),
                                                         __uint_as_float(y2 & 0xffff0000u) +
                                                             __uint_as_float(rr[e] & 0xffff0000u));
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < 32; i += 2)
                packed[i >> 1] = f32x2_to_bf16x2(__uint_as_float(acc[i]), __uint_as_float(acc[i + 1]));
        }
        if (row_ok && cols_ok) {
            uint4 *dst = reinterpret_cast<uint4 *>(dst16);
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4)
                dst[q4] = make_uint4(packed[4 * q4], packed[4 * q4 + 1], packed[4 * q4 + 2], packed[4 * q4 + 3]);
        }
        if (p.peers && acc_ok) {
            // to the other ranks, regrouped through the warp's scratch rows (80-byte pitch) so that four
            // neighbouring lanes write one row's 64 contiguous bytes (see the gated branch)
            uint4 *mine = reinterpret_cast<uint4 *>(scratch + lane * 80u);
#pragma unroll
            for (int q4 = 0; q4 < 4; ++q4)
                mine[q4] = make_uint4(packed[4 * q4], packed[4 * q4 + 1], packed[4 * q4 + 2], packed[4 * q4 + 3]);
            __syncwarp();
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {
                const uint32_t r = 8u * j + (lane >> 2), q = lane & 3u;
                const uint4 v = *reinterpret_cast<const uint4 *>(scratch + r * 80u + q * 16u);
                const uint32_t prow = row - lane + r;
                if (prow < p.m && cols_ok) {
                    const size_t at = (size_t)prow * p.ld_out + f0 + q * 8u;
#pragma unroll
                    for (uint32_t k = 0; k + 1u < kMaxExchangeRanks; ++k) {
                        if (k >= p.peers) break;
                        *reinterpret_cast<uint4 *>(p.peer_out[k] + at) = v;
                    }
                }
            }
            __syncwarp();
        }
    }
}

// HALVES = 2: a CTA owns 256 rows (two 128-row accumulators over one dequantized weight tile).  HALVES = 1: 128
// rows -- twice the CTAs, each amortizing its dequantization over half the rows -- for contractions too narrow to
// fill the SMs with 256-row tiles (a 1 024-feature slice of o or down under tensor parallelism, a 1 024-row pass).
template <uint32_t HALVES>
__global__ void __launch_bounds__(kGemmThreads, 1)
prefill_gemm_a4_kernel(const __grid_constant__ CUtensorMap x_map, const GemmParams p) {
    extern __shared__ uint8_t gemm_smem_raw[];
    // operand stages need 1024-byte alignment (swizzle atom = 8 rows x 128 bytes)
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gemm_smem_raw) + 1023u) & ~(uintptr_t)1023u);
    uint8_t *stages = smem;
    uint64_t *bars = reinterpret_cast<uint64_t *>(smem + kStages * kStageBytes);
    uint64_t *full_a = bars, *full_b = bars + kStages, *empty = bars + 2 * kStages, *acc_full = bars + 3 * kStages;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bars + 3 * kStages + 1);
    volatile uint32_t *abort_flag = tmem_slot + 1;

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t n_tile0 = blockIdx.x * (kBN / 16u);  // first 16-row storage tile of this CTA
    const uint32_t m0 = blockIdx.y * (128u * HALVES);

    if (tid == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(&full_a[s], 1);
            mbar_init(&full_b[s], kDequantWarps);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, kTmemColumns);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const uint32_t stop = p.stop_after;

    if (stop == 1u) {
        // nothing between allocation and release
    } else if (warp == 0) {
        // ------------------------------------------------ activation tiles by TMA
        if (lane == 0) {
            uint32_t slot = 0, phase = 1;  // a fresh barrier passes a wait on parity 1
            for (uint32_t kg = 0; kg < p.groups; ++kg) {
                if (!mbar_wait_bounded(&empty[slot], phase, abort_flag)) {
                    *abort_flag = 1;
                    atomicOr(p.error_word, kErrMbarTimeout);
                    break;
                }
                uint8_t *a_stage = stages + slot * kStageBytes;
                mbar_arrive_expect_tx(&full_a[slot], HALVES * kABox);
                tma_load_2d(a_stage, &x_map, kg * kBK, m0, &full_a[slot]);
                if (HALVES == 2u) tma_load_2d(a_stage + kABox, &x_map, kg * kBK, m0 + 128u, &full_a[slot]);
                if (++slot == kStages) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ tensor-core issue
        if (lane == 0) {
            uint32_t slot = 0, phase = 0;
            bool ok = true;
            for (uint32_t kg = 0; kg < p.groups && ok; ++kg) {
                ok = mbar_wait_bounded(&full_a[slot], phase, abort_flag) && mbar_wait_bounded(&full_b[slot], phase, abort_flag);
                if (!ok) {
                    *abort_flag = 1;
                    atomicOr(p.error_word, kErrMbarTimeout);
                    break;
                }
                if (stop == 2u) {  // staging only: hand the stage back without touching the tensor core
                    mbar_arrive(&empty[slot]);
                    if (++slot == kStages) {
                        slot = 0;
                        phase ^= 1u;
                    }
                    continue;
                }
                tc_fence_after();
                const uint32_t a_addr = smem_u32(stages + slot * kStageBytes);
                const uint32_t b_addr = a_addr + kAStage;
#pragma unroll
                for (uint32_t half = 0; half < HALVES; ++half) {
#pragma unroll
                    for (uint32_t k4 = 0; k4 < kBK / 16u; ++k4) {
                        const uint64_t adesc = smem_desc_sw128(a_addr + half * kABox + k4 * 32u);
                        const uint64_t bdesc = smem_desc_sw128(b_addr + k4 * 32u);
                        umma_f16(tmem_base + half * kBN, adesc, bdesc, kIdesc, (kg | k4) != 0u ? 1u : 0u);
                    }
                }
                umma_commit(&empty[slot]);  // arrives when the MMAs reading this stage are done
                if (++slot == kStages) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
            if (stop == 2u) mbar_arrive(acc_full);
            else umma_commit(acc_full);  // also on the give-up path: the epilogue warps wait on it
        }
    } else {
        // ------------------------------------------------ dequantizing prologue (one record per warp per step)
        const uint32_t d = warp - 2u;
        const uint32_t tile = n_tile0 + d;  // and tile + 8: rows 16 d .. and 128 + 16 d .. of the B stage
        uint32_t slot = 0, phase = 1;
        constexpr uint32_t kAhead = 4;  // steps requested ahead of use (global latency >> one step)
        RecordRegs ring[kAhead][2];
#pragma unroll
        for (uint32_t i = 0; i < kAhead; ++i) {
            ring[i][0] = load_record(p.w, i < p.groups ? tile : 0xffffffffu, p.row_tiles, p.groups, i, lane);
            ring[i][1] = load_record(p.w, i < p.groups ? tile + 8u : 0xffffffffu, p.row_tiles, p.groups, i, lane);
        }
        bool ok = true;
        for (uint32_t kb = 0; kb < p.groups && ok; kb += kAhead) {
#pragma unroll
            for (uint32_t i = 0; i < kAhead; ++i) {
                const uint32_t kg = kb + i;
                if (kg >= p.groups) break;
                const RecordRegs cur0 = ring[i][0], cur1 = ring[i][1];
                const uint32_t next = kg + kAhead;
                ring[i][0] = load_record(p.w, next < p.groups ? tile : 0xffffffffu, p.row_tiles, p.groups,
                                         next < p.groups ? next : 0u, lane);
                ring[i][1] = load_record(p.w, next < p.groups ? tile + 8u : 0xffffffffu, p.row_tiles, p.groups,
                                         next < p.groups ? next : 0u, lane);
                if (!mbar_wait_bounded(&empty[slot], phase, abort_flag)) {
                    if (lane == 0) {
                        *abort_flag = 1;
                        atomicOr(p.error_word, kErrMbarTimeout);
                    }
                    ok = false;
                    break;
                }
                dequant_record_to_smem(cur0, stages + slot * kStageBytes + kAStage, d, lane);
                dequant_record_to_smem(cur1, stages + slot * kStageBytes + kAStage, d + 8u, lane);
                proxy_fence_async();  // the tensor core reads shared memory through the async proxy
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_b[slot]);
                if (++slot == kStages) {
                    slot = 0;
                    phase ^= 1u;
                }
            }
        }

        // ------------------------------------------------ epilogue: warp -> (sub-partition, accumulator half)
        // (with one accumulator the two warps of a sub-partition share its columns instead)
        const uint32_t sub = warp & 3u, half = HALVES == 2u ? d >> 2 : 0u;
        const uint32_t c_first = HALVES == 2u ? 0u : (d >> 2) * (kBN / 64u), c_count = kBN / 32u / (3u - HALVES);
        const bool acc_ok = mbar_wait_bounded(acc_full, 0, abort_flag);
        if (!acc_ok && lane == 0) atomicOr(p.error_word, kErrMbarTimeout);
        tc_fence_after();
        // every tensor-core read of the operand stages has completed: their first bytes serve as 4 KB of scratch per warp
        uint8_t *scratch = stages + d * 4096u;
        const uint32_t row = m0 + half * 128u + sub * 32u + lane;  // this thread's row of the output
#pragma unroll 1
        for (uint32_t c = c_first; c < (stop == 0u ? c_first + c_count : 0u); ++c) {
            uint32_t acc[32];
            tmem_ld_32x32(tmem_base + ((sub * 32u) << 16) + half * kBN + c * 32u, acc);
            // columns of the accumulator are storage rows of the matrix: feature = 16 * tile + r
            store_block(p, row, n_tile0 * 16u + c * 32u, acc, scratch, lane, acc_ok);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kTmemColumns);
    }
}

// The contraction over weights that lie in memory as bf16 rows (pair_gemm.cuh).  Same values, same order of sums as the kernel above: the same bits.
__global__ void __launch_bounds__(kPairThreads, 1)
prefill_gemm_pair_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const GemmParams p) {
    extern __shared__ uint8_t gemm_smem_raw[];
    pair_gemm(x_map, w_map, p.groups, (p.m + kPairRows - 1u) / kPairRows, (p.row_tiles * 16u + kPairFeatures - 1u) / kPairFeatures,
              p.error_word, gemm_smem_raw, [&](uint32_t row, uint32_t f0, const uint32_t (&acc)[32], uint8_t *scratch, uint32_t lane) {
                  store_block(p, row, f0, acc, scratch, lane, true);
              });
}

// ---------------------------------------------------------------------------------------- one or two row tiles
// 128 rows x WIDTH features, K divided among the CTAs of a cluster (thin_tile.cuh); two CTAs to an SM.  The roles are those of
// the kernel above; with 64 features a step has four records, and the dequantizing warps take steps in turn.  Set-up, the
// first records and their requests run under the launch before this one.
template <uint32_t WIDTH>
struct Thin {
    static constexpr uint32_t kStage = kABox + WIDTH * 128u, kDepth = WIDTH == 64u ? 4u : 3u;
    static constexpr uint32_t kSmem = kDepth * kStage + 1024u + 256u;
    static constexpr uint32_t kRecords = WIDTH / 16u, kTurns = kDequantWarps / kRecords;
    static constexpr uint32_t kPitch = WIDTH + 4u;  // floats between the rows of the accumulator tile
    static constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((WIDTH >> 3) << 17) | ((128u >> 4) << 24);
    static_assert(128u * kPitch * 4u <= kDepth * kStage, "the accumulator tile takes the place of the stages");
};

template <uint32_t WIDTH>
__global__ void __launch_bounds__(kGemmThreads, 2)
prefill_gemm_a4_thin_kernel(const __grid_constant__ CUtensorMap x_map, const GemmParams p) {
    using T = Thin<WIDTH>;
    extern __shared__ uint8_t gemm_smem_raw[];
    uint8_t *stages = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gemm_smem_raw) + 1023u) & ~(uintptr_t)1023u);
    uint64_t *bars = reinterpret_cast<uint64_t *>(stages + T::kDepth * T::kStage);
    uint64_t *full_a = bars, *full_b = bars + T::kDepth, *empty = bars + 2 * T::kDepth, *acc_full = bars + 3 * T::kDepth;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    float *tile_sums = reinterpret_cast<float *>(stages);

    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t n_tile0 = blockIdx.x * (WIDTH / 16u), m0 = blockIdx.y * 128u;
    const uint32_t split = gridDim.z, rank = blockIdx.z;  // the cluster is the grid's z
    const uint32_t first = p.groups * rank / split, steps = p.groups * (rank + 1u) / split - first;

    if (tid == 0) {
        for (uint32_t s = 0; s < T::kDepth; ++s) {
            mbar_init(&full_a[s], 1);
            mbar_init(&full_b[s], T::kRecords);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, WIDTH);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const auto failed = [&] {
        *abort_flag = 1;
        atomicOr(p.error_word, kErrMbarTimeout);
    };
    pdl_launch_dependents();  // behind the allocation: what starts now cannot take tensor memory from a CTA that waits for it

    if (warp == 0) {
        if (lane == 0) {
            pdl_wait();  // the activations come from the launch before this one
            for (uint32_t i = 0; i < steps; ++i) {
                const uint32_t slot = i % T::kDepth;
                if (!mbar_wait_bounded(&empty[slot], (i / T::kDepth & 1u) ^ 1u, abort_flag)) {
                    failed();
                    break;
                }
                mbar_arrive_expect_tx(&full_a[slot], kABox);
                tma_load_2d(stages + slot * T::kStage, &x_map, (first + i) * kBK, m0, &full_a[slot]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            for (uint32_t i = 0; i < steps; ++i) {
                const uint32_t slot = i % T::kDepth, phase = i / T::kDepth & 1u;
                if (!(mbar_wait_bounded(&full_a[slot], phase, abort_flag) && mbar_wait_bounded(&full_b[slot], phase, abort_flag))) {
                    failed();
                    break;
                }
                tc_fence_after();
                const uint32_t a_addr = smem_u32(stages + slot * T::kStage), b_addr = a_addr + kABox;
#pragma unroll
                for (uint32_t k4 = 0; k4 < kBK / 16u; ++k4)
                    umma_f16(tmem_base, smem_desc_sw128(a_addr + k4 * 32u), smem_desc_sw128(b_addr + k4 * 32u), T::kIdesc,
                             (i | k4) != 0u ? 1u : 0u);
                umma_commit(&empty[slot]);
            }
            umma_commit(acc_full);  // also on the give-up path: the warps below wait on it
        }
    } else {
        const uint32_t d = warp - 2u, tile = n_tile0 + d % T::kRecords;
        constexpr uint32_t kAhead = 3;  // of this warp's steps: more spill at two CTAs an SM
        RecordRegs ring[kAhead];
        const auto fetch = [&](uint32_t i) {
            return load_record(p.w, i < steps ? tile : 0xffffffffu, p.row_tiles, p.groups, i < steps ? first + i : 0u, lane);
        };
        const uint32_t turn = d / T::kRecords;
#pragma unroll
        for (uint32_t j = 0; j < kAhead; ++j) ring[j] = fetch(turn + j * T::kTurns);
        bool ok = true;
#pragma unroll 1
        for (uint32_t base = turn; base < steps && ok; base += kAhead * T::kTurns) {
#pragma unroll
            for (uint32_t j = 0; j < kAhead; ++j) {
                const uint32_t i = base + j * T::kTurns, slot = i % T::kDepth;
                if (i >= steps) break;
                const RecordRegs cur = ring[j];
                ring[j] = fetch(i + kAhead * T::kTurns);
                if (!mbar_wait_bounded(&empty[slot], (i / T::kDepth & 1u) ^ 1u, abort_flag)) {
                    if (lane == 0) failed();
                    ok = false;
                    break;
                }
                dequant_record_to_smem(cur, stages + slot * T::kStage + kABox, d % T::kRecords, lane);
                proxy_fence_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full_b[slot]);
            }
        }
        if (!mbar_wait_bounded(acc_full, 0, abort_flag) && lane == 0) atomicOr(p.error_word, kErrMbarTimeout);
        tc_fence_after();
        // every read of the stages has completed: the accumulators take their place
        const uint32_t sub = warp & 3u;
#pragma unroll 1
        for (uint32_t c = (d >> 2) * (WIDTH / 64u); c < ((d >> 2) + 1u) * (WIDTH / 64u); ++c) {
            uint32_t acc[32];
            tmem_ld_32x32(tmem_base + ((sub * 32u) << 16) + c * 32u, acc);
            thin_store(tile_sums + (sub * 32u + lane) * T::kPitch + c * 32u, acc);
        }
    }
    __syncwarp();
    tc_fence_before();
    thin_cluster_sync();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, WIDTH);
    }
    pdl_wait();  // the residual rows
    const uint32_t rows_each = 128u / split, f0 = n_tile0 * 16u;
    if (p.epilogue == kEpiSwiGlu) {
        // 16 up columns, then the 16 gate columns of the same units: four units a thread
        constexpr uint32_t kQuads = WIDTH / 8u;
#pragma unroll 1
        for (uint32_t i = tid; i < rows_each * kQuads; i += kGemmThreads) {
            const uint32_t r = rank * rows_each + i / kQuads, q = i % kQuads, column = q / 4u * 32u + q % 4u * 4u;
            const uint32_t unit = (f0 + column) / 32u * 16u + q % 4u * 4u;
            if (m0 + r >= p.m || unit >= p.rows / 2u) continue;
            const float *at = tile_sums + r * T::kPitch + column;
            const float4 up4 = thin_sum(at, split), gate4 = thin_sum(at + 16, split);
            const float ups[4] = {up4.x, up4.y, up4.z, up4.w}, gates[4] = {gate4.x, gate4.y, gate4.z, gate4.w};
            float o[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float gate = bf16_round(gates[e]);
                o[e] = bf16_round(ups[e]) * bf16_round(gate / (1.0f + expf(-1.0f * gate)));
            }
            *reinterpret_cast<uint2 *>(p.out + (size_t)(m0 + r) * p.ld_out + unit) =
                make_uint2(f32x2_to_bf16x2(o[0], o[1]), f32x2_to_bf16x2(o[2], o[3]));
        }
    } else {
        constexpr uint32_t kQuads = WIDTH / 4u;
#pragma unroll 1
        for (uint32_t i = tid; i < rows_each * kQuads; i += kGemmThreads) {
            const uint32_t r = rank * rows_each + i / kQuads, column = i % kQuads * 4u;
            if (m0 + r >= p.m || f0 + column >= p.rows) continue;
            uint2 *dst = reinterpret_cast<uint2 *>(p.out + (size_t)(m0 + r) * p.ld_out + f0 + column);
            uint2 res = make_uint2(0u, 0u);
            if (p.epilogue == kEpiResidual) res = *dst;
            const float4 v = thin_sum(tile_sums + r * T::kPitch + column, split);
            uint2 y = make_uint2(f32x2_to_bf16x2(v.x, v.y), f32x2_to_bf16x2(v.z, v.w));
            if (p.epilogue == kEpiResidual) {
                y.x = f32x2_to_bf16x2(__uint_as_float(y.x << 16) + __uint_as_float(res.x << 16),
                                      __uint_as_float(y.x & 0xffff0000u) + __uint_as_float(res.x & 0xffff0000u));
                y.y = f32x2_to_bf16x2(__uint_as_float(y.y << 16) + __uint_as_float(res.y << 16),
                                      __uint_as_float(y.y & 0xffff0000u) + __uint_as_float(res.y & 0xffff0000u));
            }
            *dst = y;
        }
    }
    __syncwarp();
    thin_cluster_leave();
}

// ---------------------------------------------------------------------------------------- host side

// Estimated us of the 256-feature tiles.  Over packed weights a step of 64 columns and wave of 256 rows takes 1.15, of 128 rows 0.75: the
// dequantizing warps bound it.  Over unpacked ones a step of a round of pairs takes 0.4 (all SMs at the power limit), behind the
// unpacking of 2.56 bytes a weight at 5 TB/s.  Measured, prompts of the 8b shape, packed and unpacked: 700 rows 17.1 and 17.4 ms, 1 000
// rows 21.8 and 21.1, 3 000 rows 56.5 and 51.5; of the 0.6b shape 1 000 rows 4.70 and 4.22, 3 500 rows 12.3 and 9.8.
struct WideTimes {
    float packed, unpacked;
};
WideTimes wide_times(uint32_t features, uint32_t m, uint32_t groups) {
    const uint32_t tiles = (features + kBN - 1u) / kBN, sms = 148u, tall = tiles * ((m + 255u) / 256u);
    const float waves_256 = (float)((tall + sms - 1u) / sms), waves_128 = (float)((tiles * ((m + 127u) / 128u) + sms - 1u) / sms);
    const float k = (float)groups, unpack = 2.5625f * 64.0f * k * (float)features / 5.0e6f, rounds = (float)((tall + sms / 2u - 1u) / (sms / 2u));
    return {4.0f + k * std::min(1.15f * waves_256, 0.75f * waves_128), 8.0f + unpack + k * 0.4f * rounds};
}
// Setting gemm_unpack: 0 never, 1 by estimated times, 2 always.
bool takes_unpacked(const WideTimes &t, uint32_t m) {
    const uint32_t mode = tunables().gemm_unpack;
    if (mode == 0u || m <= kPrefillSmallRows || tunables().gemm_stop_after) return false;
    return mode == 2u || t.unpacked < t.packed;
}

// Setting gemm_thin: 0 never, 1 by estimated times, width + split that tile.  256-feature tiles take 1.15 us a step and wave of
// 256 rows, 0.75 of 128 rows; measured, 77 rows: 1024 x 3072 39.6 -> 7.3 us, 4096 x 12288 136 -> 23, 6144 x 1024 gated 28.5 ->
// 10; 301 rows: 41.4 -> 11.0, 141 -> 66, 29.2 -> 16; from about 600 rows the wide tiles fill the SMs and win.
ThinTile thin_tile(const GemmArgs &a) {
    const uint32_t mode = tunables().gemm_thin, groups = a.w->groups, features = a.whole_rows ? a.whole_rows : a.w->rows;
    if (mode == 0u || tunables().gemm_stop_after) return {};
    if (mode > 1u) return forced_thin_tile(mode, groups);
    const WideTimes t = wide_times(features, a.m, groups);
    const float wide = a.may_unpack && takes_unpacked(t, a.m) ? std::min(t.packed, t.unpacked) : t.packed;
    return pick_thin_tile(features, a.m, groups, wide, ThinSteps{{0.52f, 0.6f}, {0.6f, 0.85f}});
}

}  // namespace

size_t prefill_gemm_unpacked_bytes(const GemmArgs &a) {
    const QMatrix *w = a.w;
    if (!w || w->format != kFmtAffine4 || thin_tile(a).width) return 0;
    return takes_unpacked(wide_times(a.whole_rows ? a.whole_rows : w->rows, a.m, w->groups), a.m) ? (size_t)w->row_tiles * 16u * w->columns * 2u : 0u;
}

bool prefill_gemm_wide(const GemmArgs &a) { return !thin_tile(a).width; }

stark_b200_status prefill_gemm_launch(const GemmArgs &a, cudaStream_t stream) {
    const QMatrix *w = a.w;
    if (!w || !a.x || !a.out || a.m == 0 || a.m > a.x_rows) return STARK_B200_INVALID_ARGUMENT;
    if (w->format != kFmtAffine4) return STARK_B200_UNSUPPORTED;
    if (a.epilogue != kEpiStore && a.epilogue != kEpiResidual && a.epilogue != kEpiSwiGlu) return STARK_B200_UNSUPPORTED;
    // a pair-ordered [up; gate] matrix stores its rows interleaved: only the SwiGLU epilogue puts them back
    if ((a.epilogue == kEpiSwiGlu) != (w->pair_halves != 0)) return STARK_B200_INVALID_ARGUMENT;
    if (w->rows % 32u != 0) return STARK_B200_UNSUPPORTED;  // the epilogue writes whole 32-feature segments
    if ((reinterpret_cast<uintptr_t>(a.x) & 15u) || (reinterpret_cast<uintptr_t>(a.out) & 15u) || (a.ld_out % 8u) != 0)
        return STARK_B200_INVALID_ARGUMENT;
    // A handful of rows is a weight stream, not a contraction: the several-rows matvec reads the matrix once at the
    // pace of the one-token path.
    if (a.peers > kMaxExchangeRanks) return STARK_B200_INVALID_ARGUMENT;
    for (uint32_t r = 0; r < a.peers; ++r)
        if (!a.peer_out[r] || (reinterpret_cast<uintptr_t>(a.peer_out[r]) & 15u)) return STARK_B200_INVALID_ARGUMENT;
    if (a.peers && a.m <= kPrefillSmallRows) return STARK_B200_UNSUPPORTED;  // only the 256-feature tiles store to peers
    if (tunables().rows_matvec && qmv_multi_supports(w, a.m, false)) {
        QmvMultiArgs q{};
        q.matrix = w;
        q.x = a.x;
        q.x_stride = w->columns;
        q.m = a.m;
        q.y = a.out;
        q.y_stride = a.ld_out;
        q.epilogue = a.epilogue;
        q.error_word = a.error_word;
        q.pdl = true;  // the kernel awaits its predecessor itself, after its weight ring has begun to fill
        return qmv_multi_launch(q, stream);
    }
    EncodeTiledFn encode = encode_tiled();
    if (!encode) return STARK_B200_UNSUPPORTED;

    CUtensorMap map;
    const cuuint64_t dims[2] = {w->columns, a.x_rows};
    const cuuint64_t strides[1] = {(cuuint64_t)w->columns * 2u};
    const cuuint32_t box[2] = {kBK, 128u};
    const cuuint32_t elem[2] = {1u, 1u};
    if (encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t *>(a.x), dims, strides, box, elem,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return STARK_B200_DEVICE_FAILURE;

    GemmParams p{};
    p.w = w->data;
    p.row_tiles = w->row_tiles;
    p.groups = w->groups;
    p.rows = w->rows;
    p.m = a.m;
    p.out = a.out;
    p.ld_out = a.ld_out;
    p.epilogue = a.epilogue;
    p.error_word = a.error_word;
    p.peers = a.peers;
    for (uint32_t r = 0; r < a.peers; ++r) p.peer_out[r] = a.peer_out[r];
    p.stop_after = tunables().gemm_stop_after;
    static SmemOptIn once;
    const uint32_t feature_tiles = (w->row_tiles * 16u + kBN - 1u) / kBN;
    // Tile height by waves over the SMs: a 128-row tile takes 0.87 of a 256-row tile's time (measured: it
    // dequantizes the same weight tile for half the rows), so it pays only where 256-row tiles leave more than
    // half of the SMs idle.
    const uint32_t sms = 148u, full = feature_tiles * ((a.m + kBM - 1u) / kBM), halved = feature_tiles * ((a.m + 127u) / 128u);
    const float cost_full = (float)((full + sms - 1u) / sms), cost_half = 0.87f * (float)((halved + sms - 1u) / sms);
    const uint32_t mode = tunables().gemm_half_tiles;  // 0 never, 1 by the rule above, 2 always
    const ThinTile thin = thin_tile(a);
    if (thin.width) {
        if (a.peers) return STARK_B200_UNSUPPORTED;
        const auto kernel = thin.width == 64u ? prefill_gemm_a4_thin_kernel<64> : prefill_gemm_a4_thin_kernel<128>;
        const uint32_t smem = thin.width == 64u ? Thin<64>::kSmem : Thin<128>::kSmem;
        static SmemOptIn once_thin[2];
        if (stark_b200_status s = ensure_dynamic_smem(kernel, (int)smem, once_thin[thin.width / 128u])) return s;
        return thin_launch(kernel, dim3((w->rows + thin.width - 1u) / thin.width, (a.m + 127u) / 128u, thin.split), kGemmThreads,
                           smem, stream, map, p);
    }
    if (a.unpacked) {
        CUtensorMap w_map;
        const cuuint64_t w_dims[2] = {w->columns, w->row_tiles * 16u};
        const cuuint32_t w_box[2] = {kBK, kPairFeatures / 2u};
        if (encode(&w_map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t *>(a.unpacked), w_dims, strides, w_box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return STARK_B200_DEVICE_FAILURE;
        static SmemOptIn once_pair;
        if (stark_b200_status s = ensure_dynamic_smem(prefill_gemm_pair_kernel, (int)kPairSmem, once_pair)) return s;
        if (stark_b200_status s = pair_launch(prefill_gemm_pair_kernel, w->row_tiles * 16u, a.m, sms, stream, map, w_map, p)) return s;
    } else if (mode == 2u || (mode == 1u && cost_half < cost_full)) {
        static SmemOptIn once_half;
        if (stark_b200_status s = ensure_dynamic_smem(prefill_gemm_a4_kernel<1>, (int)kGemmSmem, once_half)) return s;
        prefill_gemm_a4_kernel<1><<<dim3(feature_tiles, (a.m + 127u) / 128u), kGemmThreads, kGemmSmem, stream>>>(map, p);
    } else {
        if (stark_b200_status s = ensure_dynamic_smem(prefill_gemm_a4_kernel<2>, (int)kGemmSmem, once)) return s;
        prefill_gemm_a4_kernel<2><<<dim3(feature_tiles, (a.m + kBM - 1u) / kBM), kGemmThreads, kGemmSmem, stream>>>(map, p);
    }
    SB_CUDA(cudaGetLastError());
    return STARK_B200_OK;
}

}  // namespace sb
