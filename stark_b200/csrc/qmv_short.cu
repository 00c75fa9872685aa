// y = W x over a 4-bit affine group-64 matrix that is small enough to be requested whole before the wait on the launch before
// it: the projections of a small model's token.
//
// The streaming kernel (qmv.cu) fills the register file with two CTAs an SM, so its ring starts to fill when the launch before
// it ends; on a matrix of 1 to 4 MB that start-up, two block barriers of the prologue and the hand-off between warps are most
// of its time.  Here a CTA of eight warps owns one row tile (one [up; gate] pair of tiles) and all of K; a warp owns a slice of
// the columns: it requests its records at once, stages the slice itself (f16 by an exact power of two of its own), multiplies,
// and leaves its partial rows.  Two block barriers with the norm (its sum of squares), one without.  Arithmetic and rounding
// points are the streaming kernel's: exact integer codes times f16 on mma.sync, f32 sums, scale and bias per group in f32.
// A token of the 0.6b shape (28 layers, 500 rows of cache): 0.683 -> 0.657 ms.
#include <algorithm>

#include "device_math.cuh"
#include "qmv.cuh"
#include "tunables.cuh"

namespace sb {

namespace {

constexpr uint32_t kWarps = 8, kThreads = kWarps * 32;
constexpr uint32_t kMostRecords = 8;  // of a warp's slice: two 16-byte chunks of the row a lane

struct ShortParams {
    const uint8_t *w;
    uint32_t rows, groups, pair_halves, slice;  // slice: records of a warp's columns in shared memory
    const uint16_t *x, *norm, *resid;
    float eps;
    uint32_t epilogue;
    uint16_t *y;
};

// A warp's records, its columns as f16 and their sums by group.
__host__ __device__ inline uint32_t slice_bytes(uint32_t slice, uint32_t tiles) {
    return (slice * (tiles * kA4RecordBytes + 128u + 4u) + 15u) & ~15u;
}

// TILES = 2: the up and the gate tile of 16 units.
template <int TILES, bool NORM>
__global__ void __launch_bounds__(kThreads) qmv_a4_short_kernel(const ShortParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float part[kWarps][TILES * 16], squares[kWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, tile0 = blockIdx.x * TILES;
    const uint32_t first = p.groups * warp / kWarps, count = p.groups * (warp + 1u) / kWarps - first;
    uint8_t *stage = smem + warp * slice_bytes(p.slice, TILES);
    uint8_t *xs = stage + p.slice * TILES * kA4RecordBytes;
    float *sums = reinterpret_cast<float *>(xs + p.slice * 128u);
    pdl_launch_dependents();
#pragma unroll
    for (int tile = 0; tile < TILES; ++tile) {
        const uint8_t *src = p.w + ((size_t)(tile0 + tile) * p.groups + first) * kA4RecordBytes;
        for (uint32_t off = lane * 16u; off < count * kA4RecordBytes; off += 512u)
            cp_async16(stage + tile * p.slice * kA4RecordBytes + off, src + off);
    }
    cp_async_commit();
    uint4 nw[2];
    if (NORM)
#pragma unroll
        for (uint32_t r = 0; r < 2u; ++r) {
            const uint32_t c = lane + 32u * r;
            if (c >= count * 8u) continue;
            nw[r] = reinterpret_cast<const uint4 *>(p.norm + first * 64u)[c];
        }
    pdl_wait();
    const uint32_t row = tile_row0(tile0, p.pair_halves, p.rows) + lane;  // what this lane of warp 0 stores
    float residual = 0.0f;
    if (warp == 0 && lane < 16u && p.epilogue == kEpiResidual && row < p.rows) residual = bf16_bits_to_f32(p.resid[row]);
    float f[2][8];
#pragma unroll
    for (uint32_t r = 0; r < 2u; ++r) {
        const uint32_t c = lane + 32u * r;
        const uint4 v = c < count * 8u ? reinterpret_cast<const uint4 *>(p.x + first * 64u)[c] : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t w4[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) f[r][2 * i] = __uint_as_float(w4[i] << 16), f[r][2 * i + 1] = __uint_as_float(w4[i] & 0xffff0000u);
    }
    if (NORM) {
        float s = 0.0f;
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 8; ++i) s = fmaf(f[r][i], f[r][i], s);
        s = warp_sum(s);
        if (lane == 0) squares[warp] = s;
        __syncthreads();
        s = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < kWarps; ++w) s += squares[w];
        const float rms_inv = 1.0f / sqrtf(s / (float)(p.groups * 64u) + p.eps);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (lane + 32u * r >= count * 8u) continue;  // its entries are zeros, the weights were not read
            const uint32_t n4[4] = {nw[r].x, nw[r].y, nw[r].z, nw[r].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {  // bf16(normalized) * bf16(weight), product rounded to bf16 (normalization.rs:157-161)
                const uint32_t n2 = f32x2_to_bf16x2(f[r][2 * i] * rms_inv, f[r][2 * i + 1] * rms_inv);
                const uint32_t p2 = f32x2_to_bf16x2(__uint_as_float(n2 << 16) * __uint_as_float(n4[i] << 16),
                                                    __uint_as_float(n2 & 0xffff0000u) * __uint_as_float(n4[i] & 0xffff0000u));
                f[r][2 * i] = __uint_as_float(p2 << 16), f[r][2 * i + 1] = __uint_as_float(p2 & 0xffff0000u);
            }
        }
    }
    // exact power-of-two scale: the slice's largest element lands in [2^14, 2^15)
    uint32_t top = 0;
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int i = 0; i < 8; ++i) top = max(top, __float_as_uint(f[r][i]) & 0x7fffffffu);
    top = __reduce_max_sync(0xffffffffu, top);
    int shift = max(-100, min(100, 14 - ((int)(top >> 23) - 127)));
    if (top == 0u || top >= 0x7f800000u) shift = 0;
    const float scale = __uint_as_float((uint32_t)(shift + 127) << 23), unscale = __uint_as_float((uint32_t)(127 - shift) << 23);
#pragma unroll
    for (uint32_t r = 0; r < 2u; ++r) {
        const uint32_t c = lane + 32u * r;
        float s = 0.0f;
        uint32_t h[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            s += f[r][2 * i], s += f[r][2 * i + 1];
            const __half2 v = __floats2half2_rn(f[r][2 * i] * scale, f[r][2 * i + 1] * scale);
            h[i] = *reinterpret_cast<const uint32_t *>(&v);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (c < count * 8u) {
            reinterpret_cast<uint4 *>(xs)[c] = make_uint4(h[0], h[1], h[2], h[3]);
            if ((lane & 7u) == 0) sums[c >> 3] = s;
        }
    }
    cp_async_wait<0>();
    __syncwarp();

    const uint32_t g = lane >> 2, t = lane & 3u;
    float dot[TILES][2] = {}, bias[TILES][2] = {};
#pragma unroll 2
    for (uint32_t k = 0; k < count; ++k) {
        const uint4 xa = *reinterpret_cast<const uint4 *>(xs + k * 128u + t * 32u), xb = *reinterpret_cast<const uint4 *>(xs + k * 128u + t * 32u + 16u);
        const uint32_t xw[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
        const float sum = sums[k];
#pragma unroll
        for (int tile = 0; tile < TILES; ++tile) {
            const uint8_t *rec = stage + (tile * p.slice + k) * kA4RecordBytes;
            const uint4 q = *reinterpret_cast<const uint4 *>(rec + lane * 16u);
            const uint32_t sw = *reinterpret_cast<const uint32_t *>(rec + 512u + 4u * g), bw = *reinterpret_cast<const uint32_t *>(rec + 544u + 4u * g);
            const uint32_t words[4] = {q.x, q.y, q.z, q.w};
            float c[2][4] = {};  // two chains of two products
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t a[4];
                dequant_a4_word<0>(words[j], a);
                mma_m16n8k16_f16(c[j & 1], a, xw[2 * j], xw[2 * j + 1]);
            }
            dot[tile][0] = fmaf(__uint_as_float(sw << 16), c[0][0] + c[1][0], dot[tile][0]);
            dot[tile][1] = fmaf(__uint_as_float(sw & 0xffff0000u), c[0][2] + c[1][2], dot[tile][1]);
            bias[tile][0] = fmaf(__uint_as_float(bw << 16), sum, bias[tile][0]);
            bias[tile][1] = fmaf(__uint_as_float(bw & 0xffff0000u), sum, bias[tile][1]);
        }
    }
    if (t == 0)
#pragma unroll
        for (int tile = 0; tile < TILES; ++tile)
#pragma unroll
            for (int h = 0; h < 2; ++h) part[warp][tile * 16 + h * 8 + g] = fmaf(dot[tile][h], unscale, bias[tile][h]);
    __syncthreads();
    if (warp != 0 || lane >= 16u * TILES) return;
    float v = 0.0f;
#pragma unroll
    for (uint32_t w = 0; w < kWarps; ++w) v += part[w][lane];
    if (TILES == 2) {  // gated_act_mul.rs:80-95: silu in f32 -> bf16, product of two bf16 -> bf16
        const float gate = bf16_round(__shfl_down_sync(0xffffffffu, v, 16));
        const uint32_t unit = blockIdx.x * 16u + lane;
        if (lane < 16u && unit < p.rows / 2u)
            p.y[unit] = f32_to_bf16_bits(bf16_round(v) * bf16_round(gate / (1.0f + expf(-1.0f * gate))));
    } else if (row < p.rows) {
        p.y[row] = p.epilogue == kEpiResidual ? f32_to_bf16_bits(bf16_round(v) + residual) : f32_to_bf16_bits(v);
    }
}

uint32_t short_slice(const QMatrix *m) { return (m->groups + kWarps - 1u) / kWarps; }
uint32_t short_smem(const QMatrix *m, uint32_t tiles) {
    return kWarps * slice_bytes(short_slice(m), tiles);
}

}  // namespace

// One wave of CTAs whose records all fit the SMs beside a launch that waits: at most four an SM and 150 KB of them; rows of up
// to 4 096 values (two chunks a lane).  No more than 4 MB: 4096 x 4096 (9.4 MB) takes 5.5 us against 4.9 streamed, twenty of
// them in turn in a graph, and the qkv and o projections of the 8b shape leave its token where it was.  Setting qmv_short: 0 never.
// A bare row takes it with one CTA an SM at most: twenty in turn in a graph, 2368 x 1024 (148 CTAs) 2.21 -> 1.53 us, but 2560 x
// 1024 (160) 2.51 -> 3.08 and 4096 x 1024 2.68 -> 3.27.  Behind a norm or gated, two an SM are about even: with one at most a
// sampled answer on the 0.6b shape takes 10.9 ms (11.1), a prompt behind a prefix 2.44 (2.40).
constexpr size_t kShortBytes = 4u << 20;
bool qmv_short_takes(const QmvArgs &a) {
    const QMatrix *m = a.matrix;
    const bool pair = a.epilogue == kEpiSwiGlu;
    if (!tunables().qmv_short || a.io_type != STARK_B200_BF16 || a.exchange || a.trace || m->bytes > kShortBytes ||
        m->groups > kWarps * kMostRecords)
        return false;
    if (a.prologue != kProPlain && !(a.prologue == kProRmsNorm && a.norm_weight_bf16)) return false;
    if (!pair && a.epilogue != kEpiStore && a.epilogue != kEpiResidual) return false;
    if (pair && m->row_tiles % 2u) return false;
    const uint32_t each = (m->row_tiles / (pair ? 2u : 1u) + 147u) / 148u;
    if (each > 1u && !pair && a.prologue == kProPlain) return false;
    return each <= 4u && each * short_smem(m, pair ? 2u : 1u) <= 150u * 1024u;
}

stark_b200_status qmv_short_launch(const QmvArgs &a, cudaStream_t stream) {
    const QMatrix *m = a.matrix;
    const bool pair = a.epilogue == kEpiSwiGlu, norm = a.prologue == kProRmsNorm;
    const uint32_t smem = short_smem(m, pair ? 2u : 1u), grid = m->row_tiles / (pair ? 2u : 1u);
    void (*const kernels[4])(ShortParams) = {qmv_a4_short_kernel<1, false>, qmv_a4_short_kernel<1, true>, qmv_a4_short_kernel<2, false>,
                                             qmv_a4_short_kernel<2, true>};
    const int slot = (pair ? 2 : 0) + (norm ? 1 : 0);
    static SmemOptIn once[4];
    if (stark_b200_status s = ensure_dynamic_smem(kernels[slot], 150 * 1024, once[slot])) return s;
    if (a.out_grid) *a.out_grid = grid;
    const ShortParams p{m->data, m->rows, m->groups, m->pair_halves, short_slice(m), static_cast<const uint16_t *>(a.x), a.norm_weight_bf16,
                        static_cast<const uint16_t *>(a.resid), a.eps, a.epilogue, static_cast<uint16_t *>(a.y)};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.pdl ? 1 : 0;
    SB_CUDA(cudaLaunchKernelEx(&cfg, kernels[slot], p));
    return STARK_B200_OK;
}

}  // namespace sb
