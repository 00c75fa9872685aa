// y = W x (one row, or up to eight) over a 4-bit affine group-64 matrix of any size: the matvecs of a token, of a draft step and of a
// pass of a few rows.
//
// A CTA of eight warps owns whole row tiles; a warp owns one eighth of the columns (of every 64 * 8 * NG of them), streams the records of
// its columns through a ring of its own (cp.async, two half items ahead, the first requested before the wait on the launch before), stages
// its own columns of the input and leaves its partial rows in shared memory.  So a warp waits for nobody but its own copies, the input
// needs no barrier beyond the norm's one, and the sums over the warps cost one barrier per round of tiles.
//   one row      the row as f16 scaled by an exact power of two per warp (largest element in [2^14, 2^15)), codes as f16 256 + q and
//                16 + q (six instructions for eight codes; exact integers take nine)
//   eight rows   rows are the eight columns; rows as they are, codes as bf16 128 + q
// The group's scale multiplies its sum in f32; its bias and the codes' offset go through one 16 x 8 x 8 product for four groups.
// Rounding points are those of the reference's chain (normalization.rs:13-191, gated_act_mul.rs:80-95).
//
// What bounds it: not memory (a matrix that stays in L2 takes the same time, 11.3 us for 24576 x 4096 against 11.4 cold) but the path
// into the SMs -- cp.async brings 24576 x 4096 in 11.4 us, bulk copies in 12.6, the shared ring of qmv.cu in 13.4, twenty and more in turn
// in a graph -- and, in a token, the start: code that the SM fetches anew.  So the launches of a token share one instance (the norm is a
// branch, the second half of an item a loop), and a ring of two beats one of five with an instance of its own: o 4.9 -> 3.0 us, [up; gate]
// 14.1 -> 13.1, a token of the 8b shape 1.75 -> 1.65 ms (1.76 with the shared ring).  Only the read-out, a launch a token, has a ring of five.
// 54 KB and at most 104 registers a thread: two CTAs and one of the attention fit an SM.
#include <algorithm>

#include "device_math.cuh"
#include "qmv.cuh"
#include "tunables.cuh"

namespace sb {

namespace {

constexpr uint32_t kWarps = 8, kThreads = kWarps * 32, kCtas = 2;  // CTAs an SM

struct SliceParams {
    const uint8_t *w;
    uint32_t rows, row_tiles, groups, chunks, pair_halves, unit_tiles;
    uint32_t m, x_stride, y_stride;
    const uint16_t *x;
    uint16_t *y;
    const uint16_t *resid;
    const float *norm;          // eight rows
    const uint16_t *norm_b16;   // one row
    float eps;
    uint32_t epilogue;
    float *partial_max;
    uint32_t *partial_index;
    TraceSlot *trace;
};

// NG: groups of a warp's slice.  A half item is half of a warp's 8 (NG = 6: 6) records of one or more tiles.
template <int NG, bool MULTI>
struct Slice {
    static constexpr int kTiles = NG >= 6 ? 1 : 8 / NG;           // of an item
    static constexpr int kHalf = NG * kTiles / 2;                 // records of half an item
    static constexpr int kHalfTiles = NG >= 6 ? 1 : kTiles / 2;   // tiles a half touches
    static constexpr int kHalfGroups = NG >= 6 ? NG / 2 : NG;     // groups of each of them
    static constexpr uint32_t kHalfBytes = kHalf * kA4RecordBytes;
    static constexpr uint32_t kRound = !MULTI ? 8 : (NG == 2 ? 4 : 2);  // tiles between two sums over the warps: whole items
    static constexpr uint32_t kTileFloats = 16u * (MULTI ? 8u : 1u);
    static constexpr uint32_t kStageX = kWarps * NG * 128u;       // one row: f16 columns; eight rows: the norm's weights in bf16
    static constexpr uint32_t kPart = 2u * kRound * kWarps * kTileFloats * 4u;
    static constexpr uint32_t smem(uint32_t depth) { return kWarps * depth * kHalfBytes + kStageX + kPart + 256u; }
};

// Without `volatile`: the compiler may order independent products.  ZERO: the sums start at zero.
template <bool ZERO>
__device__ inline void product_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (ZERO)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <bool ZERO>
__device__ inline void product_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    if (ZERO)
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
            : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.0f));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
            : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
            : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ inline void product_k8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(b0));
}
// f32 as three bf16 terms, 24 bits in all; the term `which` of two values as a pair.
__device__ inline uint32_t bf16_term(float a, float b, uint32_t which) {
    uint32_t hi = f32x2_to_bf16x2(a, b);
#pragma unroll
    for (uint32_t i = 0; i < 2u; ++i) {
        if (i == which) break;
        a -= __uint_as_float(hi << 16), b -= __uint_as_float(hi & 0xffff0000u);
        hi = f32x2_to_bf16x2(a, b);
    }
    return hi;
}

// DEPTH: half items of a warp's ring.  NORM: eight rows only.
template <int NG, bool MULTI, bool NORM, int DEPTH>
__global__ void __launch_bounds__(kThreads) __maxnreg__(MULTI ? 128 : 104) qmv_a4_slice_kernel(const SliceParams p) {
    using S = Slice<NG, MULTI>;
    const bool norm = MULTI ? NORM : p.norm_b16 != nullptr;  // one row: one piece of code, which the launches of a token share
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    uint8_t *xs = smem + warp * NG * 128u;
    float *part = reinterpret_cast<float *>(smem + S::kStageX);
    float *squares = part + S::kPart / 4u;                                       // [8 rows][8 warps]
    uint8_t *ring = smem + S::kStageX + S::kPart + 256u + warp * DEPTH * S::kHalfBytes;

    const uint32_t units = p.row_tiles / p.unit_tiles;
    const uint32_t t0 = (uint32_t)(((uint64_t)blockIdx.x * units) / gridDim.x) * p.unit_tiles;
    const uint32_t t1 = (uint32_t)(((uint64_t)(blockIdx.x + 1) * units) / gridDim.x) * p.unit_tiles;
    const uint32_t items = (t1 - t0 + S::kTiles - 1u) / S::kTiles;  // of one chunk of columns
    const uint32_t halves = 2u * items * p.chunks;

    pdl_launch_dependents();
    if (tid == 0 && p.trace) trace_min(&p.trace->start), trace_max(&p.trace->start_last);

    // What the warp requests next: half `ahead_half` of the records of its columns of tile `ahead`; one group of copies a half.
    const size_t tile_stride = (size_t)p.groups * kA4RecordBytes, chunk_stride = (size_t)kWarps * NG * kA4RecordBytes;
    const uint8_t *chunk_at = p.w + t0 * tile_stride + warp * NG * kA4RecordBytes + lane * 16u, *ahead_at = chunk_at;
    uint32_t ahead = t0, ahead_half = 0, left = halves;
    const auto request = [&](uint32_t slot) {
        if (left) {
            --left;
            uint8_t *dst = ring + slot * S::kHalfBytes + lane * 16u;
            constexpr uint32_t kRun = S::kHalfGroups * kA4RecordBytes;
#pragma unroll
            for (uint32_t i = 0; i < (uint32_t)S::kHalfTiles; ++i)
                if (ahead + i < t1)
#pragma unroll
                    for (uint32_t off = 0; off < kRun; off += 512u)
                        if (off + 512u <= kRun || lane * 16u + off < kRun) cp_async16(dst + i * kRun + off, ahead_at + i * tile_stride + off);
            if (NG >= 6 && ahead_half == 0) {
                ahead_half = 1, ahead_at += kRun;
            } else {
                if (NG >= 6) ahead_half = 0, ahead_at -= kRun;
                ahead += S::kHalfTiles, ahead_at += S::kHalfTiles * tile_stride;
                if (ahead == t0 + items * S::kTiles) ahead = t0, ahead_at = chunk_at += chunk_stride;
            }
        }
        cp_async_commit();
    };
    // Two half items before the wait, the others when the input is here: a CTA that starts late does not queue it behind them.
    constexpr uint32_t kEarly = 2;
#pragma unroll 1
    for (uint32_t s = 0; s < kEarly; ++s) request(s);
    const auto request_others = [&] {
#pragma unroll 1
        for (uint32_t s = kEarly; s < DEPTH; ++s) request(s);
    };

    // ------------------------------------------------------------------ the input
    constexpr uint32_t kChunks = NG * 8u;  // of eight columns, of the slice
    uint32_t xf[MULTI ? NG : 1][8];        // eight rows: fragments of row g
    // Per group the bias and what the codes' offset adds leave through one more product of 16 x 8 x 8: k 0-3 the biases of the half's
    // groups times the sums of their inputs, k 4-7 their scales times -offset times the sums; sums as three bf16 terms, which are
    // three columns (one row) or three products (eight rows).
    constexpr int kOffsets = NG >= 6 ? 2 : 1, kTerms = MULTI ? 3 : 1;
    uint32_t offsets[kOffsets][kTerms];
    const float offset_factor = t < 2u ? 1.0f : (MULTI ? -128.0f : -256.0f);
    const uint32_t offset_pair = 2u * (t & 1u);  // this lane's two groups of a half
    float unscale = 1.0f;
    __shared__ float group_sums[kWarps][NG];  // one row: sums by group
    float *sums = group_sums[warp];

    // One row, chunk c of columns: f16 by an exact power of two of the warp's own, and the sums by group.
    const auto stage_row = [&](const uint4 (&raw)[2], const uint4 (&nw)[2], bool normed, float rms_inv) {
        float f[2][8];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t w4[4] = {raw[r].x, raw[r].y, raw[r].z, raw[r].w}, n4[4] = {nw[r].x, nw[r].y, nw[r].z, nw[r].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float a = __uint_as_float(w4[i] << 16), b = __uint_as_float(w4[i] & 0xffff0000u);
                if (normed) {  // bf16(normalized) * bf16(weight), product rounded to bf16
                    const uint32_t n2 = f32x2_to_bf16x2(a * rms_inv, b * rms_inv);
                    const uint32_t p2 = f32x2_to_bf16x2(__uint_as_float(n2 << 16) * __uint_as_float(n4[i] << 16),
                                                        __uint_as_float(n2 & 0xffff0000u) * __uint_as_float(n4[i] & 0xffff0000u));
                    a = __uint_as_float(p2 << 16), b = __uint_as_float(p2 & 0xffff0000u);
                }
                f[r][2 * i] = a, f[r][2 * i + 1] = b;
            }
        }
        uint32_t top = 0;
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int i = 0; i < 8; ++i) top = max(top, __float_as_uint(f[r][i]) & 0x7fffffffu);
        top = __reduce_max_sync(0xffffffffu, top);
        int shift = max(-100, min(100, 14 - ((int)(top >> 23) - 127)));
        if (top == 0u || top >= 0x7f800000u) shift = 0;
        const float scale = __uint_as_float((uint32_t)(shift + 127) << 23);
        unscale = __uint_as_float((uint32_t)(127 - shift) << 23);
#pragma unroll
        for (uint32_t r = 0; r < 2u; ++r) {
            const uint32_t c = lane + 32u * r;
            float s = 0.0f;
            uint32_t h[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s += f[r][2 * i], s += f[r][2 * i + 1];
                asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(h[i]) : "f"(f[r][2 * i + 1] * scale), "f"(f[r][2 * i] * scale));
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (c < kChunks) {
                reinterpret_cast<uint4 *>(xs)[c] = make_uint4(h[0], h[1], h[2], h[3]);
                if ((lane & 7u) == 0) sums[c >> 3] = s;
            }
        }
        __syncwarp();
#pragma unroll
        for (int o = 0; o < kOffsets; ++o) {
            float v[2];
#pragma unroll
            for (uint32_t e = 0; e < 2u; ++e)
                v[e] = offset_pair + e < (uint32_t)S::kHalfGroups ? sums[o * S::kHalfGroups + offset_pair + e] * scale * offset_factor : 0.0f;
            offsets[o][0] = g < 3u ? bf16_term(v[0], v[1], g) : 0u;
        }
    };
    const auto load_row = [&](uint32_t chunk, uint4 (&raw)[2]) {
#pragma unroll
        for (uint32_t r = 0; r < 2u; ++r) {
            const uint32_t c = lane + 32u * r;
            raw[r] = c < kChunks ? reinterpret_cast<const uint4 *>(p.x + (chunk * kWarps + warp) * NG * 64u)[c] : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    uint4 raw[2] = {};
    if (!MULTI) {
        uint4 nw[2] = {};
        if (norm)
#pragma unroll
            for (uint32_t r = 0; r < 2u; ++r) {
                const uint32_t c = lane + 32u * r;
                if (c < kChunks) nw[r] = __ldg(reinterpret_cast<const uint4 *>(p.norm_b16 + warp * NG * 64u) + c);
            }
        pdl_wait();
        if (tid == 0 && p.trace) trace_min(&p.trace->ready), trace_max(&p.trace->ready_last);
        load_row(0, raw);
        float rms_inv = 1.0f;
        if (norm) {
            float s = 0.0f;
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t w4[4] = {raw[r].x, raw[r].y, raw[r].z, raw[r].w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float a = __uint_as_float(w4[i] << 16), b = __uint_as_float(w4[i] & 0xffff0000u);
                    s = fmaf(a, a, s), s = fmaf(b, b, s);
                }
            }
            s = warp_sum(s);
            if (lane == 0) squares[warp] = s;
            request_others();
            __syncthreads();
            s = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < kWarps; ++i) s += squares[i];
            rms_inv = 1.0f / sqrtf(s / (float)(p.groups * 64u) + p.eps);
        }
        stage_row(raw, nw, norm, rms_inv);
        if (!norm) request_others();
        if (p.chunks > 1u) load_row(1, raw);
    } else {
        if (norm) {
            for (uint32_t c = lane; c < kChunks; c += 32u) {
                const float4 *src = reinterpret_cast<const float4 *>(p.norm + warp * NG * 64u) + 2u * c;
                const float4 a = __ldg(src), b = __ldg(src + 1);
                reinterpret_cast<uint4 *>(xs)[c] =
                    make_uint4(f32x2_to_bf16x2(a.x, a.y), f32x2_to_bf16x2(a.z, a.w), f32x2_to_bf16x2(b.x, b.y), f32x2_to_bf16x2(b.z, b.w));
            }
            __syncwarp();
        }
        pdl_wait();
        // fragments straight from memory: lane (g, t) takes columns 16 t .. 16 t + 15 of every group of row g (rows past the last: row 0)
        const uint16_t *row = p.x + (size_t)(g < p.m ? g : 0u) * p.x_stride + warp * NG * 64u + t * 16u;
#pragma unroll
        for (int k = 0; k < NG; ++k) {
            const uint4 a = reinterpret_cast<const uint4 *>(row + k * 64)[0], b = reinterpret_cast<const uint4 *>(row + k * 64)[1];
            xf[k][0] = a.x, xf[k][1] = a.y, xf[k][2] = a.z, xf[k][3] = a.w, xf[k][4] = b.x, xf[k][5] = b.y, xf[k][6] = b.z, xf[k][7] = b.w;
        }
        if (norm) {
            float s = 0.0f;
#pragma unroll
            for (int k = 0; k < NG; ++k)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float a = __uint_as_float(xf[k][i] << 16), b = __uint_as_float(xf[k][i] & 0xffff0000u);
                    s = fmaf(a, a, s), s = fmaf(b, b, s);
                }
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            if (t == 0) squares[g * kWarps + warp] = s;
            request_others();
            __syncthreads();
            s = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < kWarps; ++i) s += squares[g * kWarps + i];
            const float rms_inv = 1.0f / sqrtf(s / (float)(p.groups * 64u) + p.eps);
#pragma unroll
            for (int k = 0; k < NG; ++k) {
                const uint4 a = reinterpret_cast<const uint4 *>(xs + k * 128 + t * 32u)[0], b = reinterpret_cast<const uint4 *>(xs + k * 128 + t * 32u)[1];
                const uint32_t n8[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t n2 = f32x2_to_bf16x2(__uint_as_float(xf[k][i] << 16) * rms_inv, __uint_as_float(xf[k][i] & 0xffff0000u) * rms_inv);
                    xf[k][i] = f32x2_to_bf16x2(__uint_as_float(n2 << 16) * __uint_as_float(n8[i] << 16),
                                               __uint_as_float(n2 & 0xffff0000u) * __uint_as_float(n8[i] & 0xffff0000u));
                }
            }
        }
        if (!norm) request_others();
        float sum[NG];  // of this lane's row, by group
#pragma unroll
        for (int k = 0; k < NG; ++k) {
            float s = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) s += __uint_as_float(xf[k][i] << 16), s += __uint_as_float(xf[k][i] & 0xffff0000u);
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            sum[k] = s + __shfl_xor_sync(0xffffffffu, s, 2);
        }
#pragma unroll
        for (int o = 0; o < kOffsets; ++o) {
            float v[2] = {0.0f, 0.0f};
#pragma unroll
            for (int k = 0; k < S::kHalfGroups; ++k) {
                if ((uint32_t)k == offset_pair) v[0] = sum[o * S::kHalfGroups + k] * offset_factor;
                if ((uint32_t)k == offset_pair + 1u) v[1] = sum[o * S::kHalfGroups + k] * offset_factor;
            }
#pragma unroll
            for (uint32_t i = 0; i < 3u; ++i) offsets[o][i] = bf16_term(v[0], v[1], i);
        }
    }

    if (tid == 0 && p.trace) trace_max(&p.trace->compute);
    // ------------------------------------------------------------------ main loop
    uint16_t residual = 0;  // of the element this thread stores first
    if (!MULTI && p.epilogue == kEpiResidual && tid < (t1 - t0) * 16u && tid < S::kRound * 16u) {
        const uint32_t row = tile_row0(t0 + tid / 16u, p.pair_halves, p.rows) + tid % 16u;
        if (row < p.rows) residual = p.resid[row];
    }
    float best = -INFINITY;  // kEpiLogits: of the rows this thread stores
    uint32_t best_index = 0xffffffffu;
    uint32_t slot = 0;
    // of the second product: scales of rows g + 8 count a sixteenth, biases whole
    const __nv_bfloat162 sixteenth = __float2bfloat162_rn(t < 2u ? 1.0f : 0.0625f);
    constexpr uint32_t kRoundItems = S::kRound / S::kTiles;
    uint32_t buffer = 0;
    // more than one chunk of columns: the launcher gives every CTA no more than a round of tiles
    for (uint32_t first = 0; first < items; first += kRoundItems, buffer ^= 1u) {
        const uint32_t last = min(items, first + kRoundItems);
        float *sum_at = part + buffer * S::kRound * kWarps * S::kTileFloats;
        for (uint32_t chunk = 0; chunk < p.chunks; ++chunk) {
            if (!MULTI && chunk) {
                const uint4 none[2] = {};
                __syncwarp();  // the columns before these have been read
                stage_row(raw, none, false, 1.0f);
                if (chunk + 1u < p.chunks) load_row(chunk + 1u, raw);
            }
            for (uint32_t item = first; item < last; ++item) {
                float acc[S::kHalfTiles][4], bias[S::kHalfTiles][4];
#pragma unroll MULTI ? 2 : 1  // one row: half the code, which every launch fetches anew
                for (int half = 0; half < 2; ++half) {
                    if (NG < 6 || half == 0)
#pragma unroll
                        for (int i = 0; i < S::kHalfTiles; ++i)
#pragma unroll
                            for (int e = 0; e < 4; ++e) acc[i][e] = bias[i][e] = 0.0f;
                    cp_async_wait<DEPTH - 1>();
                    __syncwarp();
                    const uint8_t *rec0 = ring + slot * S::kHalfBytes;
                    // the half's records are independent chains of four products: they run side by side, product by product
                    uint4 q[S::kHalf];
                    uint32_t sw[S::kHalf];
                    float c[S::kHalf][4];
#pragma unroll
                    for (int k = 0; k < S::kHalf; ++k) {
                        q[k] = *reinterpret_cast<const uint4 *>(rec0 + k * kA4RecordBytes + lane * 16u);
                        sw[k] = *reinterpret_cast<const uint32_t *>(rec0 + k * kA4RecordBytes + 512u + 4u * g);
                    }
                    // biases (t < 2) or scales of the lane's two groups, rows g and g + 8 of each
                    uint32_t pw[S::kHalfTiles][2];
#pragma unroll
                    for (int i = 0; i < S::kHalfTiles; ++i)
#pragma unroll
                        for (uint32_t e = 0; e < 2u; ++e)
                            pw[i][e] = *reinterpret_cast<const uint32_t *>(
                                rec0 + (i * S::kHalfGroups + min(offset_pair + e, S::kHalfGroups - 1u)) * kA4RecordBytes + (t < 2u ? 544u : 512u) + 4u * g);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int k = 0; k < S::kHalf; ++k) {
                            const int group = NG >= 6 ? half * S::kHalfGroups + k : k % S::kHalfGroups;
                            const uint32_t word = j == 0 ? q[k].x : (j == 1 ? q[k].y : (j == 2 ? q[k].z : q[k].w));
                            if constexpr (MULTI) {
                                const uint32_t magic = 0x43004300u, mask = 0x000f000fu;  // bf16 pair (128 + q, 128 + q')
                                const uint32_t a0 = lop3_and_or(word, mask, magic), a1 = lop3_and_or(word >> 4, mask, magic);
                                const uint32_t a2 = lop3_and_or(word >> 8, mask, magic), a3 = lop3_and_or(word >> 12, mask, magic);
                                if (j == 0) product_bf16<true>(c[k], a0, a1, a2, a3, xf[group][0], xf[group][1]);
                                else product_bf16<false>(c[k], a0, a1, a2, a3, xf[group][2 * j], xf[group][2 * j + 1]);
                            } else {
                                const uint2 x2 = *reinterpret_cast<const uint2 *>(xs + group * 128 + t * 32u + j * 8u);
                                // f16 pairs: row g 256 + q (a unit of 256 is four last places), row g + 8 sixteen times 16 + q
                                const uint32_t lo = word << 2, hi = word >> 6, magic = 0x5c005c00u;
                                const uint32_t a0 = lop3_and_or(lo, 0x003c003cu, magic), a1 = lop3_and_or(lo, 0x03c003c0u, magic);
                                const uint32_t a2 = lop3_and_or(hi, 0x003c003cu, magic), a3 = lop3_and_or(hi, 0x03c003c0u, magic);
                                if (j == 0) product_f16<true>(c[k], a0, a1, a2, a3, x2.x, x2.y);
                                else product_f16<false>(c[k], a0, a1, a2, a3, x2.x, x2.y);
                            }
                        }
#pragma unroll
                    for (int i = 0; i < S::kHalfTiles; ++i) {
                        const uint32_t p0 = __byte_perm(pw[i][0], pw[i][1], 0x5410);
                        uint32_t p1 = __byte_perm(pw[i][0], pw[i][1], 0x7632);
                        if constexpr (MULTI) {
#pragma unroll
                            for (int e = 0; e < 3; ++e) product_k8(acc[i], p0, p1, offsets[NG >= 6 ? half : 0][e]);
                        } else {
                            // row g + 8: offset 16 where row g has 256
                            const __nv_bfloat162 v = __hmul2(*reinterpret_cast<const __nv_bfloat162 *>(&p1), sixteenth);
                            p1 = *reinterpret_cast<const uint32_t *>(&v);
                            product_k8(bias[i], p0, p1, NG >= 6 && half ? offsets[kOffsets - 1][0] : offsets[0][0]);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < S::kHalf; ++k) {
                        const int i = k / S::kHalfGroups;
                        const float s0 = __uint_as_float(sw[k] << 16), s1 = __uint_as_float(sw[k] & 0xffff0000u);
                        acc[i][0] = fmaf(s0, c[k][0], acc[i][0]);
                        acc[i][2] = fmaf(s1, c[k][2], acc[i][2]);
                        if constexpr (MULTI) {
                            acc[i][1] = fmaf(s0, c[k][1], acc[i][1]);
                            acc[i][3] = fmaf(s1, c[k][3], acc[i][3]);
                        }
                    }
                    __syncwarp();  // every lane has its records in registers
                    request(slot);
                    if (++slot == DEPTH) slot = 0;
                    if (NG >= 6 && half == 0) continue;
#pragma unroll
                    for (int i = 0; i < S::kHalfTiles; ++i) {
                        const uint32_t tile = (item - first) * S::kTiles + (NG >= 6 ? 0 : half * S::kHalfTiles) + i;
                        float *at = sum_at + (tile * kWarps + warp) * S::kTileFloats;
                        if constexpr (MULTI) {
                            *reinterpret_cast<float2 *>(at + g * 8u + 2u * t) = make_float2(acc[i][0], acc[i][1]);
                            *reinterpret_cast<float2 *>(at + (g + 8u) * 8u + 2u * t) = make_float2(acc[i][2], acc[i][3]);
                        } else {
                            // columns 0, 1 (t = 0) and 2 (t = 1) hold the terms of the second product
                            float lo = bias[i][0] + bias[i][1], hi = bias[i][2] + bias[i][3];
                            lo += __shfl_down_sync(0xffffffffu, lo, 1), hi += __shfl_down_sync(0xffffffffu, hi, 1);
                            if (t == 0) {
                                lo = (acc[i][0] + lo) * unscale, hi = fmaf(acc[i][2], 0.0625f, hi) * unscale;
                                at[g] = chunk ? at[g] + lo : lo;
                                at[g + 8u] = chunk ? at[g + 8u] + hi : hi;
                            }
                        }
                    }
                }
            }
        }
        __syncthreads();
        // ---------------------------------------------------------------- sums over the warps, epilogue
        const uint32_t tile0 = t0 + first * S::kTiles, tiles = min(t1 - tile0, S::kRound);
        constexpr uint32_t kWide = MULTI ? 8u : 1u;
        const auto total = [&](uint32_t tile, uint32_t at) {
            const float *src = sum_at + tile * kWarps * S::kTileFloats + at;
            float v = 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < kWarps; ++i) v += src[i * S::kTileFloats];
            return v;
        };
        if (p.epilogue == kEpiSwiGlu) {
            for (uint32_t i = tid; i < tiles / 2u * 16u * kWide; i += kThreads) {
                const uint32_t unit = i / (16u * kWide), e = i % (16u * kWide), r = MULTI ? e / 8u : e, xr = MULTI ? e % 8u : 0u;
                const float up = bf16_round(total(2u * unit, e)), gate = bf16_round(total(2u * unit + 1u, e));
                const uint32_t orow = (tile0 / 2u + unit) * 16u + r;
                if (xr < p.m && orow < p.rows / 2u)
                    p.y[(size_t)xr * p.y_stride + orow] = f32_to_bf16_bits(up * bf16_round(gate / (1.0f + expf(-1.0f * gate))));
            }
        } else {
            for (uint32_t i = tid; i < tiles * 16u * kWide; i += kThreads) {
                const uint32_t tile = i / (16u * kWide), e = i % (16u * kWide), r = MULTI ? e / 8u : e, xr = MULTI ? e % 8u : 0u;
                const uint32_t row = tile_row0(tile0 + tile, p.pair_halves, p.rows) + r;
                if (xr >= p.m || row >= p.rows) continue;
                const float v = total(tile, e);
                uint16_t *dst = p.y + (size_t)xr * p.y_stride + row;
                if (p.epilogue == kEpiResidual) {
                    *dst = f32_to_bf16_bits(bf16_round(v) + bf16_bits_to_f32(!MULTI && first == 0 && i == tid ? residual : p.resid[(size_t)xr * p.y_stride + row]));
                } else {
                    const uint16_t bits = f32_to_bf16_bits(v);
                    *dst = bits;
                    if (p.epilogue == kEpiLogits) {
                        const float lv = bf16_bits_to_f32(bits), key = isfinite(lv) ? lv : INFINITY;  // a non-finite logit must surface
                        if (key > best || (key == best && row < best_index)) best = key, best_index = row;
                    }
                }
            }
        }
    }
    if (tid == 0 && p.trace) trace_max(&p.trace->end);
    if (!MULTI && p.epilogue == kEpiLogits) {  // first index of the maximum over this CTA's rows
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best, o);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, best_index, o);
            if (ov > best || (ov == best && oi < best_index)) best = ov, best_index = oi;
        }
        __shared__ float top[kWarps];
        __shared__ uint32_t top_index[kWarps];
        if (lane == 0) top[warp] = best, top_index[warp] = best_index;
        __syncthreads();
        if (tid == 0) {
            for (uint32_t i = 1; i < kWarps; ++i)
                if (top[i] > best || (top[i] == best && top_index[i] < best_index)) best = top[i], best_index = top_index[i];
            p.partial_max[blockIdx.x] = best;
            p.partial_index[blockIdx.x] = best_index;
        }
    }
}

// Groups of a warp's slice: the most of 8, 6, 4 and 2 that cut the columns into whole chunks; 0: none does.
uint32_t slice_groups(uint32_t groups) {
    for (uint32_t n : {8u, 6u, 4u, 2u})
        if (groups % (kWarps * n) == 0) return n;
    return 0u;
}

uint32_t sm_count() {
    static int cached[64] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (cached[dev] == 0) {
        int n = 0;
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
        cached[dev] = n;
    }
    return (uint32_t)cached[dev];
}

template <int NG, bool MULTI, bool NORM, int DEPTH>
stark_b200_status launch(const SliceParams &p, uint32_t grid, bool pdl, cudaStream_t stream) {
    static SmemOptIn once;
    using S = Slice<NG, MULTI>;
    constexpr uint32_t smem = S::smem(DEPTH);
    if (stark_b200_status s = ensure_dynamic_smem(qmv_a4_slice_kernel<NG, MULTI, NORM, DEPTH>, (int)smem, once)) return s;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    SB_CUDA(cudaLaunchKernelEx(&cfg, qmv_a4_slice_kernel<NG, MULTI, NORM, DEPTH>, p));
    return STARK_B200_OK;
}

template <bool MULTI, bool NORM, int DEPTH>
stark_b200_status launch_slice(const SliceParams &p, uint32_t slice, uint32_t grid, bool pdl, cudaStream_t stream) {
    switch (slice) {
        case 8: return launch<8, MULTI, NORM, DEPTH>(p, grid, pdl, stream);
        case 6: return launch<6, MULTI, NORM, DEPTH>(p, grid, pdl, stream);
        case 4: return launch<4, MULTI, NORM, DEPTH>(p, grid, pdl, stream);
        default: return launch<2, MULTI, NORM, DEPTH>(p, grid, pdl, stream);
    }
}

}  // namespace

bool qmv_slice_takes(const QmvArgs &a) {
    const QMatrix *m = a.matrix;
    if (!tunables().qmv_slice || a.io_type != STARK_B200_BF16 || a.exchange) return false;
    if (a.prologue != kProPlain && !(a.prologue == kProRmsNorm && a.norm_weight_bf16)) return false;
    if (a.epilogue != kEpiStore && a.epilogue != kEpiResidual && a.epilogue != kEpiSwiGlu && a.epilogue != kEpiLogits) return false;
    const uint32_t slice = slice_groups(m->groups);
    if (!slice) return false;
    const uint32_t chunks = m->groups / (kWarps * slice), unit = a.epilogue == kEpiSwiGlu ? 2u : 1u;
    if (m->row_tiles % unit) return false;
    // several chunks: no norm, and no more than a round of tiles a CTA
    if (chunks > 1u && (a.prologue == kProRmsNorm || (m->row_tiles + sm_count() - 1u) / sm_count() + unit > 8u)) return false;
    return true;
}

stark_b200_status qmv_slice_launch(const QmvArgs &a, cudaStream_t stream) {
    const QMatrix *m = a.matrix;
    const uint32_t slice = slice_groups(m->groups);
    SliceParams p{};
    p.w = m->data;
    p.rows = m->rows;
    p.row_tiles = m->row_tiles;
    p.groups = m->groups;
    p.chunks = m->groups / (kWarps * slice);
    p.pair_halves = m->pair_halves;
    p.unit_tiles = a.epilogue == kEpiSwiGlu ? 2u : 1u;
    p.m = 1;
    p.x = static_cast<const uint16_t *>(a.x);
    p.y = static_cast<uint16_t *>(a.y);
    p.resid = static_cast<const uint16_t *>(a.resid);
    p.norm_b16 = a.prologue == kProRmsNorm ? a.norm_weight_bf16 : nullptr;
    p.eps = a.eps;
    p.epilogue = a.epilogue;
    p.partial_max = a.partial_max;
    p.partial_index = a.partial_index;
    p.trace = a.trace;
    const uint32_t grid = std::max(1u, std::min(p.row_tiles / p.unit_tiles, sm_count() * kCtas));
    if (a.out_grid) *a.out_grid = grid;
    return a.epilogue == kEpiLogits ? launch_slice<false, false, 5>(p, slice, grid, a.pdl, stream) : launch_slice<false, false, 2>(p, slice, grid, a.pdl, stream);
}

bool qmv_slice_multi_takes(const QmvMultiArgs &a) {
    const QMatrix *m = a.matrix;
    const uint32_t slice = slice_groups(m->groups);
    return tunables().qmv_slice && slice && m->groups == kWarps * slice;
}

stark_b200_status qmv_slice_multi_launch(const QmvMultiArgs &a, cudaStream_t stream) {
    const QMatrix *m = a.matrix;
    const uint32_t slice = slice_groups(m->groups);
    SliceParams p{};
    p.w = m->data;
    p.rows = m->rows;
    p.row_tiles = m->row_tiles;
    p.groups = m->groups;
    p.chunks = 1;
    p.pair_halves = m->pair_halves;
    p.unit_tiles = a.epilogue == kEpiSwiGlu ? 2u : 1u;
    p.m = a.m;
    p.x = a.x;
    p.x_stride = a.x_stride ? a.x_stride : m->columns;
    p.y = a.y;
    p.y_stride = a.y_stride;
    p.resid = a.y;
    p.norm = a.norm_weight;
    p.eps = a.eps;
    p.epilogue = a.epilogue;
    const uint32_t grid = std::max(1u, std::min(p.row_tiles / p.unit_tiles, sm_count() * kCtas));
    return p.norm ? launch_slice<true, true, 2>(p, slice, grid, a.pdl, stream) : launch_slice<true, false, 2>(p, slice, grid, a.pdl, stream);
}

}  // namespace sb
