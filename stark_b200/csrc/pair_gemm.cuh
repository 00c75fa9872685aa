// Y[M, N] = X[M, K] W[N, K]^T over bf16 rows for passes of many rows: the contraction loop on pairs of SMs (tcgen05 cta_group::2) that the
// prompt contractions of both decoder families share (prefill_gemm.cu, gemm_b16.cu).
//
// A pair of CTAs (one cluster, one CTA an SM, as many pairs as the GPU holds) walks tiles of 256 rows x 256 features.  Each CTA loads
// 128 of the rows and 128 of the features per step of 64 columns (cp.async.bulk.tensor, no multicast); the even CTA issues one MMA of
// M = 256 over both, and each CTA's tensor memory receives its 128 rows x 256 accumulators.  Two accumulators a CTA: while the epilogue
// warps empty one, the tensor cores fill the other.
//   warp 0      one thread: loads; a stage of either CTA counts on the even CTA's barrier
//   warp 1      owns tensor memory; in the even CTA one thread issues the MMAs and commits them to the barriers of both
//   warps 2-9   epilogue: warp -> (32 rows, half of the columns), 32 columns at a time
// What this replaces is one CTA per 256 x 256 tile: all of its tensor memory held one tile, so set-up, the first loads and the epilogue
// (20 000 of a tile's 90 000 cycles at K = 4096) ran with idle tensor cores, and it moved 64 KB a step and SM through L2 where
// this moves the same for twice the features of half the rows.
// Every wait is bounded; one that runs out sets the error word, both CTAs drain and free their tensor memory.
#pragma once
#include <algorithm>

#include "tc05.cuh"

namespace sb {

constexpr uint32_t kPairEpilogueWarps = 8, kPairThreads = (2u + kPairEpilogueWarps) * 32u;
constexpr uint32_t kPairScratch = 32u * 80u;  // bytes of an epilogue warp's scratch rows

constexpr uint32_t kPairRows = 256, kPairFeatures = 256;
constexpr uint32_t kPairBox = 128u * 128u, kPairStage = 2u * kPairBox, kPairDepth = 6;  // 128 rows or features x 64 columns of bf16
constexpr uint32_t kPairSmem = kPairDepth * kPairStage + kPairEpilogueWarps * kPairScratch + 256u + 1024u;
// D f32, A and B bf16, both K-major, M 256, N 256
constexpr uint32_t kPairIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((kPairFeatures >> 3) << 17) | ((kPairRows >> 4) << 24);

__device__ inline uint32_t pair_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// The address of the same place in the even CTA.
__device__ inline uint32_t pair_even(const void *p) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(a) : "r"(smem_u32(p)));
    return a;
}
__device__ inline void pair_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ inline void pair_load_2d(void *dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ inline void pair_mma(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the barrier of both CTAs when the MMAs issued so far are done.
__device__ inline void pair_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3u)
                 : "memory");
}
__device__ inline void pair_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ inline bool pair_wait(uint64_t *bar, uint32_t parity, volatile uint32_t *abort_flag, uint32_t *error_word) {
    for (uint32_t it = 0; it < (1u << 22); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        if (it > 64u) {
            if (*abort_flag) return false;
            __nanosleep(64);
        }
    }
    *abort_flag = 1;
    atomicOr(error_word, kErrMbarTimeout);
    return false;
}

// epilogue(row, column, acc, scratch, lane): 32 columns from `column` of the whole warp's 32 rows, lane `lane` holding those of `row`.
template <typename Epilogue>
__device__ __forceinline__ void pair_gemm(const CUtensorMap &x_map, const CUtensorMap &w_map, uint32_t steps, uint32_t row_tiles,
                                          uint32_t column_tiles, uint32_t *error_word, uint8_t *smem_raw, Epilogue &&epilogue) {
    uint8_t *stages = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023u) & ~(uintptr_t)1023u);
    uint8_t *scratch = stages + kPairDepth * kPairStage;
    uint64_t *full = reinterpret_cast<uint64_t *>(scratch + kPairEpilogueWarps * kPairScratch);
    uint64_t *empty = full + kPairDepth, *acc_full = empty + kPairDepth, *acc_empty = acc_full + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(acc_empty + 2);
    volatile uint32_t *abort_flag = tmem_slot + 1;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, rank = pair_rank();
    const uint32_t pairs = gridDim.x / 2u, pair = blockIdx.x / 2u, tiles = row_tiles * column_tiles;

    if (tid == 0) {
        for (uint32_t s = 0; s < kPairDepth; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (uint32_t b = 0; b < 2u; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 2u * kPairEpilogueWarps);
        }
        *abort_flag = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    pair_sync();  // the other CTA's barriers exist
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();  // behind the allocation: what starts now cannot take tensor memory from a CTA that waits for it
    pdl_wait();  // rows, weights unpacked for this launch and the residual come from the launches before

    // row tiles are the fast index: the pairs then share few tiles of weights, which stream from memory once, while the rows stay in L2
    if (warp == 0) {
        if (lane == 0) {
            uint32_t slot = 0, phase = 1, used = 0;  // a fresh barrier passes a wait on parity 1
            bool ok = true;
            for (uint32_t t = pair; t < tiles && ok; t += pairs) {
                const uint32_t m0 = t % row_tiles * kPairRows + rank * 128u, n0 = t / row_tiles * kPairFeatures + rank * 128u;
                for (uint32_t k = 0; k < steps; ++k) {
                    if (!(ok = pair_wait(&empty[slot], phase, abort_flag, error_word))) break;
                    uint8_t *stage = stages + slot * kPairStage;
                    const uint32_t bar = pair_even(&full[slot]);
                    if (rank == 0) mbar_arrive_expect_tx(&full[slot], 2u * kPairStage);
                    pair_load_2d(stage, &x_map, k * 64u, m0, bar);
                    pair_load_2d(stage + kPairBox, &w_map, k * 64u, n0, bar);
                    ++used;
                    if (++slot == kPairDepth) slot = 0, phase ^= 1u;
                }
            }
            // nobody leaves while the other CTA's commits are on their way here: every stage used is handed back first
            for (uint32_t s = 0; s < min(used, kPairDepth) && ok; ++s) {
                slot = (slot + kPairDepth - 1u) % kPairDepth;
                if (slot == kPairDepth - 1u) phase ^= 1u;
                ok = pair_wait(&empty[slot], phase ^ 1u, abort_flag, error_word);
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            uint32_t slot = 0, phase = 0, i = 0;
            bool ok = true;
            for (uint32_t t = pair; t < tiles && ok; t += pairs, ++i) {
                const uint32_t buffer = i & 1u, acc = tmem_base + buffer * 256u;
                if (!(ok = pair_wait(&acc_empty[buffer], (i >> 1 & 1u) ^ 1u, abort_flag, error_word))) break;
                tc_fence_after();
                for (uint32_t k = 0; k < steps; ++k) {
                    if (!(ok = pair_wait(&full[slot], phase, abort_flag, error_word))) break;
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(stages + slot * kPairStage);
#pragma unroll
                    for (uint32_t k4 = 0; k4 < 4u; ++k4)
                        pair_mma(acc, smem_desc_sw128(a_addr + k4 * 32u), smem_desc_sw128(a_addr + kPairBox + k4 * 32u), kPairIdesc,
                                 (k | k4) != 0u ? 1u : 0u);
                    pair_commit(&empty[slot]);
                    if (++slot == kPairDepth) slot = 0, phase ^= 1u;
                }
                pair_commit(&acc_full[buffer]);  // also on the give-up path: the epilogue warps wait on it
            }
        }
    } else {
        const uint32_t d = warp - 2u, sub = warp & 3u, half = d >> 2;
        uint32_t i = 0;
        for (uint32_t t = pair; t < tiles; t += pairs, ++i) {
            const uint32_t buffer = i & 1u;
            if (!__all_sync(0xffffffffu, pair_wait(&acc_full[buffer], i >> 1 & 1u, abort_flag, error_word))) break;
            tc_fence_after();
            const uint32_t row = t % row_tiles * kPairRows + rank * 128u + sub * 32u + lane, n0 = t / row_tiles * kPairFeatures;
#pragma unroll 1
            for (uint32_t c = half * 4u; c < half * 4u + 4u; ++c) {
                uint32_t acc[32];
                __syncwarp();  // behind the stores of the block before, where a ragged tile's lanes part
                tmem_ld_32x32(tmem_base + ((sub * 32u) << 16) + buffer * 256u + c * 32u, acc);
                if (c + 1u == half * 4u + 4u) {  // this warp's share of the accumulator is in registers
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) pair_arrive(pair_even(&acc_empty[buffer]));
                }
                epilogue(row, n0 + c * 32u, acc, scratch + d * kPairScratch, lane);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    pair_sync();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
        __syncwarp();
    }
    pair_sync();  // the release takes both CTAs: neither leaves before it is done
}

template <typename Kernel, typename... Args>
inline stark_b200_status pair_launch(Kernel kernel, uint32_t out_cols, uint32_t m, uint32_t sms, cudaStream_t stream, Args... args) {
    const uint32_t tiles = (m + kPairRows - 1u) / kPairRows * ((out_cols + kPairFeatures - 1u) / kPairFeatures);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2u * std::min(tiles, sms / 2u));
    cfg.blockDim = dim3(kPairThreads);
    cfg.dynamicSmemBytes = kPairSmem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    SB_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    return STARK_B200_OK;
}

}  // namespace sb
