// Y[M, N] = X[M, K] W[N, K]^T over a bf16 matrix, many rows at a time, on the sm_100a tensor cores (tcgen05.mma,
// accumulators in tensor memory): the prompt-pass contraction of the layered decoders.
//
// Three forms: tiles of 256 rows x 256 features on pairs of SMs (pair_gemm.cuh); where those leave SMs idle, of 128 rows x 256 features, one
// a CTA (below); for few tiles, narrow ones with K on a cluster (thin_tile.cuh).  Each walks K in steps of 64.
//   warp 0      one thread: TMA loads of the step's activation boxes and of the weight box, all bf16 in 128-byte
//               swizzled lines; rows and columns past the ends arrive as zeros
//   warp 1      owns tensor memory; one thread issues the MMAs and commits them to the barrier that frees the stage
//   warps 2-9   the epilogue: bias, then f32 or bf16 rows, or the gate of 16 gate / 16 up columns in turn (columns in front
//               of the gated ones stored as bf16 rows), or a scaled add to f32 rows (the residual stream)
// Every wait is bounded; a wait that runs out sets the error word, the CTA drains and frees its tensor memory.
#include <cuda.h>

#include <algorithm>

#include "layered.cuh"
#include "layered_math.cuh"
#include "pair_gemm.cuh"
#include "tc05.cuh"
#include "thin_tile.cuh"
#include "tunables.cuh"

namespace sb {

namespace {

constexpr uint32_t kBN = 256, kBK = 64;
constexpr uint32_t kABox = 128u * 128u;  // 128 rows x 64 bf16
constexpr uint32_t kBStage = kBN * 128u;
constexpr uint32_t kEpilogueWarps = 8, kGemmThreads = (2u + kEpilogueWarps) * 32u;

constexpr uint32_t kStageBytes = kABox + kBStage, kDepth = 4, kTileSmem = kDepth * kStageBytes + 1024u + 256u;

// D f32, A and B bf16, both K-major, M 128, N 256
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kBN >> 3) << 17) | ((128u >> 4) << 24);

struct GemmB16Params {
    uint32_t steps, m, out_cols, ld_out;
    void *out;
    const float *bias;
    Gate gate;
    uint32_t stored_cols, ld_stored;
    uint16_t *stored_out;
    const float *scale;
    uint32_t *error_word;
};

// 32 f32 values as bf16 into a row, 16-byte aligned.
__device__ inline void store_row32(uint16_t *dst, const uint32_t (&acc)[32]) {
    uint32_t packed[16];
#pragma unroll
    for (int i = 0; i < 32; i += 2) packed[i >> 1] = f32x2_to_bf16x2(__uint_as_float(acc[i]), __uint_as_float(acc[i + 1]));
#pragma unroll
    for (int q = 0; q < 4; ++q)
        reinterpret_cast<uint4 *>(dst)[q] = make_uint4(packed[4 * q], packed[4 * q + 1], packed[4 * q + 2], packed[4 * q + 3]);
}

// 32 columns from f0 of one row's accumulators.
template <uint32_t KIND>
__device__ __forceinline__ void store_block(const GemmB16Params &p, uint32_t row, bool row_ok, uint32_t f0, uint32_t (&acc)[32]) {
    const bool whole = f0 + 32u <= p.out_cols;
    if (p.bias) {  // biases come with gated and stored layers whose widths are whole blocks
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            const float4 b = __ldg(reinterpret_cast<const float4 *>(p.bias + f0 + i));
            acc[i] = __float_as_uint(__uint_as_float(acc[i]) + b.x);
            acc[i + 1] = __float_as_uint(__uint_as_float(acc[i + 1]) + b.y);
            acc[i + 2] = __float_as_uint(__uint_as_float(acc[i + 2]) + b.z);
            acc[i + 3] = __float_as_uint(__uint_as_float(acc[i + 3]) + b.w);
        }
    }
    if (!row_ok) return;
    if (KIND == kGemmGate) {
        if (f0 < p.stored_cols) {
            store_row32(p.stored_out + (size_t)row * p.ld_stored + f0, acc);
            return;
        }
        uint32_t packed[8];
#pragma unroll
        for (int i = 0; i < 16; i += 2)
            packed[i >> 1] = f32x2_to_bf16x2(gated(p.gate, __uint_as_float(acc[i]), __uint_as_float(acc[16 + i])),
                                             gated(p.gate, __uint_as_float(acc[i + 1]), __uint_as_float(acc[17 + i])));
        uint4 *dst = reinterpret_cast<uint4 *>(static_cast<uint16_t *>(p.out) + (size_t)row * p.ld_out + (f0 - p.stored_cols) / 2u);
        dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
    } else if (KIND == kGemmBf16) {
        store_row32(static_cast<uint16_t *>(p.out) + (size_t)row * p.ld_out + f0, acc);
    } else if (KIND == kGemmResidual) {
        float4 *dst = reinterpret_cast<float4 *>(static_cast<float *>(p.out) + (size_t)row * p.ld_out + f0);
        const float4 *scale = reinterpret_cast<const float4 *>(p.scale + f0);
        float4 v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = dst[q];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float4 g = __ldg(scale + q);
            v[q].x = fmaf(g.x, __uint_as_float(acc[4 * q]), v[q].x);
            v[q].y = fmaf(g.y, __uint_as_float(acc[4 * q + 1]), v[q].y);
            v[q].z = fmaf(g.z, __uint_as_float(acc[4 * q + 2]), v[q].z);
            v[q].w = fmaf(g.w, __uint_as_float(acc[4 * q + 3]), v[q].w);
            dst[q] = v[q];
        }
    } else {
        float *dst = static_cast<float *>(p.out) + (size_t)row * p.ld_out + f0;
        if (whole && p.ld_out % 4u == 0) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
                reinterpret_cast<uint4 *>(dst)[q] = make_uint4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
        } else {
#pragma unroll
            for (uint32_t i = 0; i < 32u; ++i)
                if (f0 + i < p.out_cols) dst[i] = __uint_as_float(acc[i]);
        }
    }
}

template <uint32_t KIND>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_b16_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const GemmB16Params p) {
    extern __shared__ uint8_t gemm_b16_smem[];
    uint8_t *stages = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gemm_b16_smem) + 1023u) & ~(uintptr_t)1023u);
    uint64_t *bars = reinterpret_cast<uint64_t *>(stages + kDepth * kStageBytes);
    uint64_t *full = bars, *empty = bars + kDepth, *acc_full = bars + 2 * kDepth;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    // row tiles are the fast index: a wave of CTAs then shares few weight tiles, so the weights stream from memory once
    // while the activations of a pass stay in L2
    const uint32_t n0 = blockIdx.y * kBN, m0 = blockIdx.x * 128u;

    if (tid == 0) {
        for (uint32_t s = 0; s < kDepth; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(tmem_slot, kBN);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t slot = 0, phase = 1;  // a fresh barrier passes a wait on parity 1
            for (uint32_t k = 0; k < p.steps; ++k) {
                if (!mbar_wait_bounded(&empty[slot], phase, abort_flag)) {
                    *abort_flag = 1;
                    atomicOr(p.error_word, kErrMbarTimeout);
                    break;
                }
                uint8_t *stage = stages + slot * kStageBytes;
                mbar_arrive_expect_tx(&full[slot], kStageBytes);
                tma_load_2d(stage, &x_map, k * kBK, m0, &full[slot]);
                tma_load_2d(stage + kABox, &w_map, k * kBK, n0, &full[slot]);
                if (++slot == kDepth) slot = 0, phase ^= 1u;
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            uint32_t slot = 0, phase = 0;
            for (uint32_t k = 0; k < p.steps; ++k) {
                if (!mbar_wait_bounded(&full[slot], phase, abort_flag)) {
                    *abort_flag = 1;
                    atomicOr(p.error_word, kErrMbarTimeout);
                    break;
                }
                tc_fence_after();
                const uint32_t a_addr = smem_u32(stages + slot * kStageBytes), b_addr = a_addr + kABox;
#pragma unroll
                for (uint32_t k4 = 0; k4 < kBK / 16u; ++k4)
                    umma_f16(tmem_base, smem_desc_sw128(a_addr + k4 * 32u), smem_desc_sw128(b_addr + k4 * 32u), kIdesc, (k | k4) != 0u ? 1u : 0u);
                umma_commit(&empty[slot]);
                if (++slot == kDepth) slot = 0, phase ^= 1u;
            }
            umma_commit(acc_full);  // also on the give-up path: the epilogue warps wait on it
        }
    } else {
        // two warps share a sub-partition's columns
        const uint32_t d = warp - 2u, sub = warp & 3u, c_first = (d >> 2) * (kBN / 64u), c_count = kBN / 64u;
        const bool acc_ok = mbar_wait_bounded(acc_full, 0, abort_flag);
        if (!acc_ok && lane == 0) atomicOr(p.error_word, kErrMbarTimeout);
        tc_fence_after();
        const uint32_t row = m0 + sub * 32u + lane;
        const bool row_ok = row < p.m && acc_ok;
#pragma unroll 1
        for (uint32_t c = c_first; c < c_first + c_count; ++c) {
            const uint32_t f0 = n0 + c * 32u;
            if (f0 >= p.out_cols) break;
            uint32_t acc[32];
            tmem_ld_32x32(tmem_base + ((sub * 32u) << 16) + c * 32u, acc);
            store_block<KIND>(p, row, row_ok, f0, acc);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, kBN);
    }
}

// Many tiles: pairs of SMs (pair_gemm.cuh).
template <uint32_t KIND>
__global__ void __launch_bounds__(kPairThreads, 1)
gemm_b16_pair_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const GemmB16Params p) {
    extern __shared__ uint8_t gemm_b16_smem[];
    pair_gemm(x_map, w_map, p.steps, (p.m + kPairRows - 1u) / kPairRows, (p.out_cols + kPairFeatures - 1u) / kPairFeatures, p.error_word,
              gemm_b16_smem, [&](uint32_t row, uint32_t f0, uint32_t (&acc)[32], uint8_t *, uint32_t) {
                  if (f0 < p.out_cols) store_block<KIND>(p, row, row < p.m, f0, acc);
              });
}

// One or two row tiles: 128 rows x WIDTH features, K divided among the CTAs of a cluster (thin_tile.cuh), two CTAs to an SM.
// The first stages' weights are requested before the wait on the launch before this one.
template <uint32_t WIDTH>
struct Thin {
    static constexpr uint32_t kStage = kABox + WIDTH * 128u, kDepth = WIDTH == 64u ? 4u : 3u;
    static constexpr uint32_t kSmem = kDepth * kStage + 1024u + 256u;
    static constexpr uint32_t kPitch = WIDTH + 4u;  // floats between the rows of the accumulator tile
    static constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((WIDTH >> 3) << 17) | ((128u >> 4) << 24);
    static_assert(128u * kPitch * 4u <= kDepth * kStage, "the accumulator tile takes the place of the stages");
};

__device__ inline uint2 bf16_quad(const float4 &v) { return make_uint2(f32x2_to_bf16x2(v.x, v.y), f32x2_to_bf16x2(v.z, v.w)); }

template <uint32_t WIDTH, uint32_t KIND>
__global__ void __launch_bounds__(kGemmThreads, 2)
gemm_b16_thin_kernel(const __grid_constant__ CUtensorMap x_map, const __grid_constant__ CUtensorMap w_map, const GemmB16Params p) {
    using T = Thin<WIDTH>;
    extern __shared__ uint8_t gemm_b16_smem[];
    uint8_t *stages = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(gemm_b16_smem) + 1023u) & ~(uintptr_t)1023u);
    uint64_t *bars = reinterpret_cast<uint64_t *>(stages + T::kDepth * T::kStage);
    uint64_t *full = bars, *empty = bars + T::kDepth, *acc_full = bars + 2 * T::kDepth;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_full + 1);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    float *tile_sums = reinterpret_cast<float *>(stages);
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t n0 = blockIdx.y * WIDTH, m0 = blockIdx.x * 128u;
    const uint32_t split = gridDim.z, rank = blockIdx.z;  // the cluster is the grid's z
    const uint32_t first = p.steps * rank / split, steps = p.steps * (rank + 1u) / split - first;

    if (tid == 0) {
        for (uint32_t s = 0; s < T::kDepth; ++s) {
            mbar_init(&full[s], 1);
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
            const auto weights = [&](uint32_t i) {
                const uint32_t slot = i % T::kDepth;
                mbar_arrive_expect_tx(&full[slot], T::kStage);
                tma_load_2d(stages + slot * T::kStage + kABox, &w_map, (first + i) * kBK, n0, &full[slot]);
            };
            const uint32_t ahead = min(steps, T::kDepth);
            for (uint32_t i = 0; i < ahead; ++i) weights(i);
            pdl_wait();  // the activations come from the launch before this one
            for (uint32_t i = 0; i < steps; ++i) {
                const uint32_t slot = i % T::kDepth;
                if (i >= ahead) {
                    if (!mbar_wait_bounded(&empty[slot], (i / T::kDepth & 1u) ^ 1u, abort_flag)) {
                        failed();
                        break;
                    }
                    weights(i);
                }
                tma_load_2d(stages + slot * T::kStage, &x_map, (first + i) * kBK, m0, &full[slot]);
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            for (uint32_t i = 0; i < steps; ++i) {
                const uint32_t slot = i % T::kDepth;
                if (!mbar_wait_bounded(&full[slot], i / T::kDepth & 1u, abort_flag)) {
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
        const uint32_t d = warp - 2u, sub = warp & 3u;
        if (!mbar_wait_bounded(acc_full, 0, abort_flag) && lane == 0) atomicOr(p.error_word, kErrMbarTimeout);
        tc_fence_after();
        // every read of the stages has completed: the accumulators take their place
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
    const bool ok = *abort_flag == 0u;
    // four columns and the four 16 further on (a gated block's gate and up columns) a thread
    constexpr uint32_t kItems = WIDTH / 8u;
    const uint32_t rows_each = 128u / split;
#pragma unroll 1
    for (uint32_t i = tid; i < rows_each * kItems; i += kGemmThreads) {
        const uint32_t r = rank * rows_each + i / kItems, q = i % kItems, column = q / 4u * 32u + q % 4u * 4u;
        const uint32_t row = m0 + r, block = n0 + q / 4u * 32u;
        if (row >= p.m || block >= p.out_cols || !ok) continue;
        float4 v[2];
#pragma unroll
        for (uint32_t h = 0; h < 2u; ++h) {
            v[h] = thin_sum(tile_sums + r * T::kPitch + column + 16u * h, split);
            if (p.bias) {
                const float4 b = __ldg(reinterpret_cast<const float4 *>(p.bias + n0 + column + 16u * h));
                v[h].x += b.x, v[h].y += b.y, v[h].z += b.z, v[h].w += b.w;
            }
        }
        if (KIND == kGemmGate && block >= p.stored_cols) {
            const float4 o = make_float4(gated(p.gate, v[0].x, v[1].x), gated(p.gate, v[0].y, v[1].y), gated(p.gate, v[0].z, v[1].z),
                                         gated(p.gate, v[0].w, v[1].w));
            *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(p.out) + (size_t)row * p.ld_out + (block - p.stored_cols) / 2u +
                                       q % 4u * 4u) = bf16_quad(o);
            continue;
        }
#pragma unroll
        for (uint32_t h = 0; h < 2u; ++h) {
            const uint32_t f = n0 + column + 16u * h;
            if (KIND == kGemmGate) {
                *reinterpret_cast<uint2 *>(p.stored_out + (size_t)row * p.ld_stored + f) = bf16_quad(v[h]);
            } else if (KIND == kGemmBf16) {
                *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(p.out) + (size_t)row * p.ld_out + f) = bf16_quad(v[h]);
            } else if (KIND == kGemmResidual) {
                float4 *dst = reinterpret_cast<float4 *>(static_cast<float *>(p.out) + (size_t)row * p.ld_out + f);
                const float4 g = __ldg(reinterpret_cast<const float4 *>(p.scale + f));
                float4 x = *dst;
                x.x = fmaf(g.x, v[h].x, x.x), x.y = fmaf(g.y, v[h].y, x.y), x.z = fmaf(g.z, v[h].z, x.z), x.w = fmaf(g.w, v[h].w, x.w);
                *dst = x;
            } else {
                float *dst = static_cast<float *>(p.out) + (size_t)row * p.ld_out + f;
                if (f + 4u <= p.out_cols && p.ld_out % 4u == 0) {
                    *reinterpret_cast<float4 *>(dst) = v[h];
                } else {
                    const float e[4] = {v[h].x, v[h].y, v[h].z, v[h].w};
#pragma unroll
                    for (uint32_t j = 0; j < 4u; ++j)
                        if (f + j < p.out_cols) dst[j] = e[j];
                }
            }
        }
    }
    __syncwarp();
    thin_cluster_leave();
}

template <uint32_t WIDTH>
stark_b200_status launch_thin(const GemmB16Args &a, const CUtensorMap &x_map, const CUtensorMap &w_map, const GemmB16Params &p,
                              uint32_t split, cudaStream_t stream) {
    auto kernel = a.kind == kGemmBf16
                      ? gemm_b16_thin_kernel<WIDTH, kGemmBf16>
                      : (a.kind == kGemmF32 ? gemm_b16_thin_kernel<WIDTH, kGemmF32>
                                            : (a.kind == kGemmGate ? gemm_b16_thin_kernel<WIDTH, kGemmGate> : gemm_b16_thin_kernel<WIDTH, kGemmResidual>));
    static SmemOptIn once[4];
    if (stark_b200_status st = ensure_dynamic_smem(kernel, (int)Thin<WIDTH>::kSmem, once[a.kind])) return st;
    return thin_launch(kernel, dim3((a.m + 127u) / 128u, (a.out_cols + WIDTH - 1u) / WIDTH, split), kGemmThreads, Thin<WIDTH>::kSmem,
                       stream, x_map, w_map, p);
}

stark_b200_status launch(const GemmB16Args &a, const CUtensorMap &x_map, const CUtensorMap &w_map, const GemmB16Params &p,
                         cudaStream_t stream) {
    auto kernel = a.kind == kGemmBf16
                      ? gemm_b16_kernel<kGemmBf16>
                      : (a.kind == kGemmF32 ? gemm_b16_kernel<kGemmF32>
                                            : (a.kind == kGemmGate ? gemm_b16_kernel<kGemmGate> : gemm_b16_kernel<kGemmResidual>));
    static SmemOptIn once[4];
    if (stark_b200_status st = ensure_dynamic_smem(kernel, (int)kTileSmem, once[a.kind])) return st;
    kernel<<<dim3((a.m + 127u) / 128u, (a.out_cols + kBN - 1u) / kBN), kGemmThreads, kTileSmem, stream>>>(x_map, w_map, p);
    SB_CUDA(cudaGetLastError());
    return STARK_B200_OK;
}

stark_b200_status launch_pairs(const GemmB16Args &a, const CUtensorMap &x_map, const CUtensorMap &w_map, const GemmB16Params &p,
                               cudaStream_t stream) {
    auto kernel = a.kind == kGemmBf16
                      ? gemm_b16_pair_kernel<kGemmBf16>
                      : (a.kind == kGemmF32 ? gemm_b16_pair_kernel<kGemmF32>
                                            : (a.kind == kGemmGate ? gemm_b16_pair_kernel<kGemmGate> : gemm_b16_pair_kernel<kGemmResidual>));
    static SmemOptIn once[4];
    if (stark_b200_status st = ensure_dynamic_smem(kernel, (int)kPairSmem, once[a.kind])) return st;
    return pair_launch(kernel, a.out_cols, a.m, 148u, stream, x_map, w_map, p);
}

// Setting gemm_thin as in prefill_gemm.cu.  256-feature tiles take 0.66 us a step and wave of 256 rows, 0.38 of 128 rows;
// measured, 77 rows: 1024 x 3072 20.3 -> 6.2 us, 4096 x 12288 71.8 -> 21.6, 6144 x 1024 gated 14.4 -> 8.9; 400 rows: 22.0 ->
// 9.5, 76.5 -> 50.9; 1024 x 2048 at 1 537 rows 17.8 -> 14.0.
ThinTile thin_tile(const GemmB16Args &a, uint32_t waves_256, uint32_t waves_128) {
    const uint32_t mode = tunables().gemm_thin, steps = a.w.cols / kBK;
    if (mode == 0u) return {};
    if (mode > 1u) return forced_thin_tile(mode, steps);
    const float wide = 5.0f + (float)steps * std::min(0.66f * (float)waves_256, 0.38f * (float)waves_128);
    return pick_thin_tile(a.out_cols, a.m, steps, wide, ThinSteps{{0.29f, 0.4f}, {0.34f, 0.55f}});
}

}  // namespace

stark_b200_status gemm_b16_launch(const GemmB16Args &a, cudaStream_t stream) {
    if (!a.w.data || !a.x || !a.out || a.m == 0 || a.m > a.x_rows || a.w.cols % kBK || a.ld_x % 8u || a.ld_x < a.w.cols ||
        a.out_cols > a.w.rows || (reinterpret_cast<uintptr_t>(a.x) & 15u))
        return STARK_B200_INVALID_ARGUMENT;
    // vector stores and bias reads work on whole 32-column blocks; only a bare f32 output may end inside one
    if ((a.kind != kGemmF32 || a.bias) && (a.out_cols % 32u || a.ld_out % 16u)) return STARK_B200_INVALID_ARGUMENT;
    if (a.kind == kGemmGate && a.stored_cols && (!a.stored_out || a.stored_cols % 32u || a.ld_stored % 16u)) return STARK_B200_INVALID_ARGUMENT;
    if (a.kind == kGemmResidual && (!a.scale || a.bias)) return STARK_B200_INVALID_ARGUMENT;
    DeviceContext *ctx = device_context();
    EncodeTiledFn encode = encode_tiled();
    if (!ctx || !encode) return STARK_B200_DEVICE_FAILURE;
    const cuuint32_t elem[2] = {1u, 1u};
    CUtensorMap x_map, w_map;
    auto make = [&](CUtensorMap *map, const uint16_t *base, uint32_t rows, uint32_t ld, uint32_t box_rows) {
        const cuuint64_t dims[2] = {a.w.cols, rows}, strides[1] = {(cuuint64_t)ld * 2u};
        const cuuint32_t box[2] = {kBK, box_rows};
        return encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t *>(base), dims, strides, box, elem,
                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
    };
    // 256-row tiles on pairs of SMs unless 128-row tiles fill the SMs so much better that it pays for their loading the weight tile once per
    // 128 rows.  One 256-row tile a CTA, which pairs replaced: 2 500 rows of pomelix-0.6b 7.00 -> 6.61 ms, of guvulorn-0.6b 8.17 -> 7.85
    const uint32_t wide = (a.out_cols + kBN - 1u) / kBN, tall = (a.m + 255u) / 256u, flat = (a.m + 127u) / 128u;
    const uint32_t waves2 = (wide * tall + 147u) / 148u * 2u, waves1 = (wide * flat + 147u) / 148u;
    const ThinTile thin = thin_tile(a, waves2 / 2u, waves1);
    const bool pairs = !thin.width && (tunables().gemm_pairs == 1u ? waves1 * 5u >= waves2 * 4u : tunables().gemm_pairs > 1u);
    if (!make(&x_map, a.x, a.x_rows, a.ld_x, 128u) ||
        !make(&w_map, a.w.data, a.w.rows, a.w.pitch(), thin.width ? thin.width : (pairs ? kPairFeatures / 2u : kBN)))
        return STARK_B200_DEVICE_FAILURE;
    const GemmB16Params p{a.w.cols / kBK, a.m, a.out_cols, a.ld_out, a.out, a.bias, a.gate, a.kind == kGemmGate ? a.stored_cols : 0u,
                          a.ld_stored, a.stored_out, a.scale, ctx->error_word};
    if (thin.width)
        return thin.width == 64u ? launch_thin<64>(a, x_map, w_map, p, thin.split, stream) : launch_thin<128>(a, x_map, w_map, p, thin.split, stream);
    if (pairs) return launch_pairs(a, x_map, w_map, p, stream);
    return launch(a, x_map, w_map, p, stream);
}

}  // namespace sb
