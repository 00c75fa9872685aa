// One token of the routed-expert decoder (moe_model.cu) where every matrix is re-tiled.
//
// A layer's matrices are 7 to 14 MB, a microsecond or two of HBM time each, so what a launch costs is its chain: the hand-off
// from the kernel before it, the input row, the products, the sum over the row's warps.  Every kernel here is built to make
// that chain short:
//   - all weight bytes of a CTA are requested at once, before the wait on the kernel before it (the expert banks as soon as
//     the selection is known; the down projection from the selection that gate and up published, checked after its wait);
//   - a warp owns one 16 x 256 record (a few for wide rows) and stages the 256 inputs it needs itself: no block barrier before
//     the products, one between a team's partial rows;
//   - the norm's weights are multiplied in while staging, its scale, a scalar, when the partial rows are added, where the sum
//     of squares arrives the same way;
//   - sums go in the order of moe_math.cuh, which a pass of prompt rows keeps;
//   - the selection is repeated by every warp of gate and up from the scores (two warp reductions a pick) instead of passing
//     through a last CTA's arrival counter.
// 12 layers of the 30B-A3B shape behind 12 to 36 rows: 0.79 -> 0.45 ms a token; a layer 61 -> 32 us, of which the eight kernels
// take 48 us when run one by one on a cold cache (93 before).
#include <algorithm>
#include <cmath>

#include "context.cuh"
#include "moe_math.cuh"
#include "moe_select.cuh"
#include "moe_token.cuh"

namespace sb {

namespace {

constexpr uint32_t kDim = kHeadWidth;
constexpr uint32_t kSliceLine = 512 + 64;   // head or remainder of 256 inputs: two lines 64 B apart modulo 128 B
constexpr uint32_t kSliceBytes = 2 * kSliceLine;
constexpr uint32_t kMaxWarps = kMaxMembers;

// The eight inputs of a lane (8 lane ... + 7 of a slice) as the products read them; returns 2^-s.  xa, xb: sums of the scaled
// slice over the sub-blocks t and t + 4 (32 columns each).
__device__ inline float stage_slice(const float (&v)[8], uint8_t *lines, uint32_t lane, float &xa, float &xb) {
    const SplitSlice s = split_slice(v);
    __syncwarp();  // the slice before this one has been read
    *reinterpret_cast<uint4 *>(lines + lane * 16u) = s.head;
    *reinterpret_cast<uint4 *>(lines + kSliceLine + lane * 16u) = s.rest;
    const uint32_t t = lane & 3u;
    xa = __shfl_sync(0xffffffffu, s.sum, 4u * t);
    xb = __shfl_sync(0xffffffffu, s.sum, 4u * t + 16u);
    __syncwarp();
    return s.down;
}

__device__ inline float quad_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// A record times the staged slice, added to the sums of rows g and g + 8 (on all four lanes of a row).
__device__ inline void q8_record(const uint8_t *rec, const uint8_t *lines, float down, uint32_t lane, float &v0, float &v1) {
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint16_t *meta = reinterpret_cast<const uint16_t *>(rec + 4096u);
    const uint8_t *x = lines + (g & 1u) * kSliceLine + t * 16u;  // column n = g of B: even the head, odd the remainder
    float s0[2] = {0.0f, 0.0f}, s1[2] = {0.0f, 0.0f};
#pragma unroll
    for (uint32_t jb = 0; jb < 8; ++jb) {
        const uint4 w = *reinterpret_cast<const uint4 *>(rec + jb * 512u + lane * 16u);
        const uint4 xv = *reinterpret_cast<const uint4 *>(x + 64u * jb);
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        uint32_t a[4];
        bytes_to_f16<false>(w.x, a[0], a[1]);
        bytes_to_f16<false>(w.y, a[2], a[3]);
        mma_m16n8k16_f16(c, a, xv.x, xv.y);
        bytes_to_f16<false>(w.z, a[0], a[1]);
        bytes_to_f16<false>(w.w, a[2], a[3]);
        mma_m16n8k16_f16(c, a, xv.z, xv.w);
        const bool mine = (jb & 3u) == t;
        s0[jb >> 2] = mine ? c[0] + c[1] : s0[jb >> 2];
        s1[jb >> 2] = mine ? c[2] + c[3] : s1[jb >> 2];
    }
    const float r0 = q8_share(f16_bits_f32(meta[t * 16u + g]), s0[0], f16_bits_f32(meta[(t + 4u) * 16u + g]), s0[1]);
    const float r1 = q8_share(f16_bits_f32(meta[t * 16u + g + 8u]), s1[0], f16_bits_f32(meta[(t + 4u) * 16u + g + 8u]), s1[1]);
    v0 = fmaf(down, quad_sum(r0), v0), v1 = fmaf(down, quad_sum(r1), v1);
}

__device__ inline void q4_record(const uint8_t *rec, const uint8_t *lines, float down, float xa, float xb, uint32_t lane,
                                 float &v0, float &v1) {
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint8_t *x = lines + (g & 1u) * kSliceLine + t * 16u;
    float s0[2] = {0.0f, 0.0f}, s1[2] = {0.0f, 0.0f};
#pragma unroll
    for (uint32_t jb = 0; jb < 8; ++jb) {
        const uint2 w = *reinterpret_cast<const uint2 *>(rec + jb * 256u + lane * 8u);
        const uint4 xv = *reinterpret_cast<const uint4 *>(x + 64u * jb);
        float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        uint32_t a[4];
        dequant_a4_word<0>(w.x, a);
        mma_m16n8k16_f16(c, a, xv.x, xv.y);
        dequant_a4_word<0>(w.y, a);
        mma_m16n8k16_f16(c, a, xv.z, xv.w);
        const bool mine = (jb & 3u) == t;
        s0[jb >> 2] = mine ? c[0] + c[1] : s0[jb >> 2];
        s1[jb >> 2] = mine ? c[2] + c[3] : s1[jb >> 2];
    }
    float dsc[2], dm[2];
    q4k_scales_pair(*reinterpret_cast<const uint4 *>(rec + 2048u + 16u * g), t, dsc, dm);
    const float r0 = q4k_share(dsc[0], s0[0], dsc[1], s0[1], dm[0], xa, dm[1], xb);
    q4k_scales_pair(*reinterpret_cast<const uint4 *>(rec + 2048u + 16u * (g + 8u)), t, dsc, dm);
    const float r1 = q4k_share(dsc[0], s1[0], dsc[1], s1[1], dm[0], xa, dm[1], xb);
    v0 = fmaf(down, quad_sum(r0), v0), v1 = fmaf(down, quad_sum(r1), v1);
}

template <uint32_t BYTES>
__device__ inline void fetch_record(uint8_t *dst, const uint8_t *src, uint32_t lane) {
    for (uint32_t off = lane * 16u; off < BYTES; off += 512u) cp_async16(dst + off, src + off);
}

// How the warps of a CTA share a matrix: `width` warps a row tile (a team), `records` super-blocks each, as Members.
struct Teams {
    uint32_t supers, row_tiles, rows, width, records, teams;
};

struct TokenQ8Params {
    Teams at;
    const uint8_t *data;
    const float *x, *norm, *residual;
    float eps;
    float *out;
};

// Bound by its chain: 11 MB (5120 x 2048) are 1.7 us of HBM time, requested before the wait.
__global__ void __launch_bounds__(kMaxWarps * 32) token_q8_kernel(const TokenQ8Params p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float rows[kMaxWarps][16], squares[kMaxWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, W = p.at.width;
    const uint32_t team = warp / W, member = warp % W, tile = blockIdx.x * p.at.teams + team;
    const bool live = tile < p.at.row_tiles;
    pdl_launch_dependents();
    uint8_t *lines = smem + warp * (kSliceBytes + p.at.records * kB8SuperBytes), *stage = lines + kSliceBytes;
    if (live)
        for (uint32_t r = 0, s = member; r < p.at.records && s < p.at.supers; ++r, s += W)
            fetch_record<kB8SuperBytes>(stage + r * kB8SuperBytes, p.data + ((size_t)tile * p.at.supers + s) * kB8SuperBytes, lane);
    cp_async_commit();
    float w[8];
    if (p.norm && member < p.at.supers) load8(p.norm + member * 256u + lane * 8u, w);
    pdl_wait();
    if (!live) return;  // whole teams
    const uint32_t row = tile * 16u + lane;
    const bool writes = member == 0 && lane < 16u && row < p.at.rows;
    const float add = writes && p.residual ? p.residual[row] : 0.0f;
    float v0 = 0.0f, v1 = 0.0f, square = 0.0f;
    for (uint32_t r = 0, s = member; r < p.at.records && s < p.at.supers; ++r, s += W) {
        float v[8], xa, xb;
        load8(p.x + s * 256u + lane * 8u, v);
        if (p.norm) {
            if (r) load8(p.norm + s * 256u + lane * 8u, w);
            weigh8(v, w, square);
        }
        const float down = stage_slice(v, lines, lane, xa, xb);
        if (r == 0) {
            cp_async_wait<0>();
            __syncwarp();
        }
        q8_record(stage + r * kB8SuperBytes, lines, down, lane, v0, v1);
    }
    if (p.norm) square = warp_sum(square);
    if ((lane & 3u) == 0) rows[warp][lane >> 2] = v0, rows[warp][(lane >> 2) + 8u] = v1;
    if (lane == 0) squares[warp] = square;
    if (W > 1u) named_bar_sync(1 + (int)team, (int)W * 32);
    else __syncwarp();
    if (!writes) return;
    float sum = 0.0f, total = 0.0f;
    for (uint32_t m = 0; m < W; ++m) sum += rows[warp + m][lane], total += squares[warp + m];
    if (p.norm) sum = __fmul_rn(sum, norm_scale(total, p.at.supers * 256u, p.eps));
    p.out[row] = p.residual ? add + sum : sum;
}

constexpr uint32_t kTokenAttnWarps = kStrands;  // a strand a warp

// One CTA per KV head and span; the G query heads of the group are scored against each row once it is read.  Rows that the
// cache held before this token, the angles and the norms are fetched before the wait.
template <int G>
__global__ void __launch_bounds__(kTokenAttnWarps * 32, 2) token_attention_kernel(const uint32_t *position_word, const float *qkv,
                                                                               const bool raw, float *keys, float *values,
                                                                               float *part, uint32_t splits, uint32_t kv_heads,
                                                                               float scale, uint32_t context,
                                                                               const float *q_norm, const float *k_norm,
                                                                               float eps, float theta) {
    __shared__ float sm[kTokenAttnWarps][G], sl[kTokenAttnWarps][G];
    __shared__ __align__(16) float4 sacc[kTokenAttnWarps][G][32];
    __shared__ __align__(16) float heads[G][kDim], fresh[2][kDim];
    pdl_launch_dependents();
    const uint32_t kvh = blockIdx.x, split = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t position = min(*position_word, context - 1u), rows = position + 1u;  // written between tokens only
    const uint32_t span = span_rows(rows, splits), lo = split * span;
    if (lo >= rows) return;  // the first span of every head stays
    const uint32_t hi = min(rows, lo + span);
    const size_t kv_row = (size_t)kv_heads * kDim;
    const uint32_t begin = kvh * kDim;
    const auto load_row = [&](const float *cache, uint32_t t) {
        return reinterpret_cast<const float4 *>(cache + t * kv_row + begin)[lane];
    };
    float4 kv[2] = {}, vv[2] = {};
#pragma unroll
    for (uint32_t j = 0; j < 2u; ++j) {
        const uint32_t t = min(lo + warp + j * kTokenAttnWarps, hi - 1u);  // a row past the end repeats the last one, unused
        if (t != position) kv[j] = load_row(keys, t), vv[j] = load_row(values, t);
    }
    float qn[4], kn[4], cs[2], sn[2];
    const bool newest = hi == rows, key_warp = warp == kTokenAttnWarps - 1u, value_warp = warp == kTokenAttnWarps - 2u;
    if (raw) {
#pragma unroll
        for (int k = 0; k < 4; ++k) qn[k] = q_norm[32 * k + lane], kn[k] = k_norm[32 * k + lane];
        head_angles(position, theta, lane, cs, sn);
    }
    pdl_wait();
    if (raw) {
        const uint32_t q_heads = kv_heads * G;
        float v[4], o[4], f[4];
        if (newest && (key_warp || value_warp)) {
            const float *src = qkv + ((size_t)q_heads + (key_warp ? 0u : kv_heads) + kvh) * kDim;
#pragma unroll
            for (int k = 0; k < 4; ++k) f[k] = src[32 * k + lane];
        }
        if (warp < (uint32_t)G) {
            const float *src = qkv + ((size_t)kvh * G + warp) * kDim;
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = src[32 * k + lane];
            prepare_head(v, qn, cs, sn, eps, o);
#pragma unroll
            for (int k = 0; k < 4; ++k) heads[warp][32 * k + lane] = o[k];
        }
        if (newest && (key_warp || value_warp)) {
            float *dst = (key_warp ? keys : values) + position * kv_row + begin;
            if (key_warp) {
                prepare_head(f, kn, cs, sn, eps, o);
#pragma unroll
                for (int k = 0; k < 4; ++k) f[k] = o[k];
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) fresh[key_warp ? 0 : 1][32 * k + lane] = f[k], dst[32 * k + lane] = f[k];
        }
        __syncthreads();
    }
    const float *q = raw ? &heads[0][0] : qkv + (size_t)kvh * G * kDim;
    float4 qv[G];
#pragma unroll
    for (int g = 0; g < G; ++g) qv[g] = reinterpret_cast<const float4 *>(q + (size_t)g * kDim)[lane];
    float m[G], l[G];
    float4 acc[G];
#pragma unroll
    for (int g = 0; g < G; ++g) m[g] = -INFINITY, l[g] = 0.0f, acc[g] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (uint32_t t0 = lo + warp; t0 < hi; t0 += 2u * kTokenAttnWarps) {
        float dot[2][G];
#pragma unroll
        for (uint32_t j = 0; j < 2u; ++j) {
            const uint32_t t = min(t0 + j * kTokenAttnWarps, hi - 1u);
            if (t == position && raw) {
                kv[j] = reinterpret_cast<const float4 *>(fresh[0])[lane], vv[j] = reinterpret_cast<const float4 *>(fresh[1])[lane];
            } else if (t == position || t0 != lo + warp) {
                kv[j] = load_row(keys, t), vv[j] = load_row(values, t);
            }
        }
#pragma unroll
        for (uint32_t j = 0; j < 2u; ++j)
#pragma unroll
            for (int g = 0; g < G; ++g)
                dot[j][g] = dot4(qv[g], kv[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (uint32_t j = 0; j < 2u; ++j)
#pragma unroll
                for (int g = 0; g < G; ++g) dot[j][g] += __shfl_xor_sync(0xffffffffu, dot[j][g], o);
#pragma unroll
        for (uint32_t j = 0; j < 2u; ++j) {
            if (t0 + j * kTokenAttnWarps >= hi) break;
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float c, e;
                strand_step(m[g], l[g], __fmul_rn(dot[j][g], scale), c, e);
                strand_add(acc[g], c, e, vv[j]);
            }
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (lane == 0) sm[warp][g] = m[g], sl[warp][g] = l[g];
        sacc[warp][g][lane] = acc[g];
    }
    __syncthreads();
    if (warp >= (uint32_t)G) return;
    float gm = -INFINITY;
#pragma unroll
    for (uint32_t w = 0; w < kTokenAttnWarps; ++w) gm = fmaxf(gm, sm[w][warp]);
    float gl = 0.0f;
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (uint32_t w = 0; w < kTokenAttnWarps; ++w) strand_take(gl, a, strand_weight(sm[w][warp], gm), sl[w][warp], sacc[w][warp][lane]);
    float *dst = part + (((size_t)kvh * G + warp) * splits + split) * (kDim + 2u);
    if (lane == 0) dst[0] = gm, dst[1] = gl;
    reinterpret_cast<float2 *>(dst + 2)[lane * 2u] = make_float2(a.x, a.y);
    reinterpret_cast<float2 *>(dst + 2)[lane * 2u + 1u] = make_float2(a.z, a.w);
}

// One CTA per query head; a lane keeps the weights of spans `lane` and `lane + 32`, every warp for itself.
__global__ void __launch_bounds__(kDim) token_merge_kernel(const uint32_t *position_word, const float *part, float *out,
                                                           uint32_t splits, uint32_t context) {
    pdl_launch_dependents();
    const uint32_t h = blockIdx.x, i = threadIdx.x, lane = i & 31u;
    const uint32_t rows = min(*position_word, context - 1u) + 1u, span = span_rows(rows, splits);
    const uint32_t used = (rows + span - 1u) / span;
    const float *src = part + (size_t)h * splits * (kDim + 2u);
    pdl_wait();
    float m[2], l[2];
#pragma unroll
    for (uint32_t j = 0; j < 2u; ++j) {
        const uint32_t s = lane + 32u * j;
        m[j] = s < used ? src[s * (kDim + 2u)] : -INFINITY;
        l[j] = s < used ? src[s * (kDim + 2u) + 1u] : 0.0f;
    }
    float c[2];
    const float total = span_weights(m, l, c);
    float a = 0.0f;
#pragma unroll 8
    for (uint32_t s = 0; s < used; ++s) {
        const float weight = __shfl_sync(0xffffffffu, s < 32u ? c[0] : c[1], s & 31u);
        a = fmaf(src[s * (kDim + 2u) + 2u + i], weight, a);
    }
    out[(size_t)h * kDim + i] = a / total;
}

// One CTA per expert, a warp a member; its router row times the norm's weights is ready before the wait.
__global__ void __launch_bounds__(kMaxWarps * 32) token_router_kernel(const float *router, const float *x, const float *norm,
                                                                      float eps, float *scores, const Members at) {
    __shared__ float part[2][kMaxWarps];
    pdl_launch_dependents();
    const uint32_t lane = threadIdx.x & 31u, member = threadIdx.x >> 5;
    const float *row = router + (size_t)blockIdx.x * at.supers * kSlice;
    float a[8], w[8], v[8], dot = 0.0f, square = 0.0f;
    const auto product = [&](uint32_t s) {
        load8(row + s * kSlice + lane * 8u, a), load8(norm + s * kSlice + lane * 8u, w);
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = __fmul_rn(a[i], w[i]);
    };
    product(member);
    pdl_wait();
    for (uint32_t r = 0, s = member; r < at.records && s < at.supers; ++r, s += at.width) {
        if (r) product(s);
        load8(x + s * kSlice + lane * 8u, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) dot = fmaf(a[i], v[i], dot), square = fmaf(v[i], v[i], square);
    }
    dot = warp_sum(dot), square = warp_sum(square);
    if (lane == 0) part[0][member] = dot, part[1][member] = square;
    __syncthreads();
    if (threadIdx.x) return;
    dot = square = 0.0f;
    for (uint32_t m = 0; m < at.width; ++m) dot += part[0][m], square += part[1][m];
    scores[blockIdx.x] = __fmul_rn(dot, norm_scale(square, at.supers * kSlice, eps));
}

struct TokenGateUpParams {
    Teams at;
    TokenSelection sel;
    const uint8_t *data;
    size_t matrix_bytes;
    const float *x, *norm;
    float eps;
    float *act;
};

// KEYS: the scores a lane holds (experts / 32, rounded up to 4 or 32).  WARPS: the most a CTA has; three CTAs of eight stay on an
// SM, so that the 384 of 8 experts of 768 x 2048 run in one wave.  Bound by HBM latency and the records' bytes behind the
// selection (14.2 MB there).
template <int KEYS, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8 ? 3 : 1) token_gate_up_kernel(const TokenGateUpParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float rows[kMaxWarps][32], squares[kMaxWarps];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, W = p.at.width, slot = blockIdx.y;
    const uint32_t team = warp / W, member = warp % W, tile = blockIdx.x * p.at.teams + team;
    uint8_t *lines = smem + warp * (kSliceBytes + 2u * p.at.records * kQ4SuperBytes), *stage = lines + kSliceBytes;
    float w[8], v[8];
    load8(p.norm + member * 256u + lane * 8u, w);  // the width is no more than the super-blocks
    pdl_wait();
    uint32_t key[KEYS];
#pragma unroll
    for (int j = 0; j < KEYS; ++j)
        key[j] = lane + 32u * j < p.sel.experts ? order_key(p.sel.scores[lane + 32u * j]) : 0u;
    load8(p.x + member * 256u + lane * 8u, v);

    // the selection up to this CTA's slot, by every warp; one warp of the launch goes to its end and publishes it
    const bool publishes = blockIdx.x == 0 && blockIdx.y == 0 && warp == 0;
    const uint32_t picks = publishes ? p.sel.active : slot + 1u;
    uint32_t expert = 0, mine = 0, mine_key = 0;  // of this slot; of selection slot `lane`
    for (uint32_t r = 0; r < picks; ++r) {
        uint32_t top;
        const uint32_t pick = take_first_largest(key, lane, top);
        if (r == slot) expert = pick;
        if (r == lane) mine = pick, mine_key = top;
    }
    if (publishes) {
        const float share = selection_share(key_value(mine_key), p.sel.active, lane);
        if (lane < p.sel.active) {
            p.sel.probs[lane] = share;
            if (p.sel.ids_global) {
                const bool here = mine >= p.sel.ep_first && mine < p.sel.ep_first + p.sel.ep_local;
                p.sel.ids[lane] = here ? mine - p.sel.ep_first : kEpSkip;
                p.sel.ids[p.sel.active + lane] = here ? mine - p.sel.ep_first + p.sel.ep_local : kEpSkip;
                p.sel.ids_global[lane] = mine;
            } else {
                p.sel.ids[lane] = mine;
                p.sel.ids[p.sel.active + lane] = mine + p.sel.experts;
            }
        }
        __threadfence();
    }
    pdl_launch_dependents();  // the down projection reads the ids ahead of its wait
    uint32_t bank = p.sel.experts;
    if (p.sel.ids_global) {
        if (expert < p.sel.ep_first || expert >= p.sel.ep_first + p.sel.ep_local) return;  // the whole CTA
        expert -= p.sel.ep_first, bank = p.sel.ep_local;
    }
    if (tile >= p.at.row_tiles) return;  // whole teams
    const uint8_t *gate = p.data + (size_t)expert * p.matrix_bytes, *up = gate + (size_t)bank * p.matrix_bytes;
    for (uint32_t r = 0, s = member; r < p.at.records && s < p.at.supers; ++r, s += W) {
        const size_t at = ((size_t)tile * p.at.supers + s) * kQ4SuperBytes;
        fetch_record<kQ4SuperBytes>(stage + 2u * r * kQ4SuperBytes, gate + at, lane);
        fetch_record<kQ4SuperBytes>(stage + (2u * r + 1u) * kQ4SuperBytes, up + at, lane);
    }
    cp_async_commit();
    float g0 = 0.0f, g1 = 0.0f, u0 = 0.0f, u1 = 0.0f, square = 0.0f;
    for (uint32_t r = 0, s = member; r < p.at.records && s < p.at.supers; ++r, s += W) {
        float xa, xb;
        if (r) load8(p.norm + s * 256u + lane * 8u, w), load8(p.x + s * 256u + lane * 8u, v);
        weigh8(v, w, square);
        const float down = stage_slice(v, lines, lane, xa, xb);
        if (r == 0) {
            cp_async_wait<0>();
            __syncwarp();
        }
        q4_record(stage + 2u * r * kQ4SuperBytes, lines, down, xa, xb, lane, g0, g1);
        q4_record(stage + (2u * r + 1u) * kQ4SuperBytes, lines, down, xa, xb, lane, u0, u1);
    }
    square = warp_sum(square);
    if ((lane & 3u) == 0) {
        const uint32_t g = lane >> 2;
        rows[warp][g] = g0, rows[warp][g + 8u] = g1, rows[warp][g + 16u] = u0, rows[warp][g + 24u] = u1;
    }
    if (lane == 0) squares[warp] = square;
    if (W > 1u) named_bar_sync(1 + (int)team, (int)W * 32);
    else __syncwarp();
    if (member) return;
    float sum = 0.0f, total = 0.0f;
    for (uint32_t m = 0; m < W; ++m) sum += rows[warp + m][lane], total += squares[warp + m];
    sum = __fmul_rn(sum, norm_scale(total, p.at.supers * 256u, p.eps));
    const float other = __shfl_down_sync(0xffffffffu, sum, 16);  // lanes 0-15: gate rows, 16-31: up rows
    if (lane >= 16u || tile * 16u + lane >= p.at.rows) return;
    p.act[(size_t)slot * p.at.rows + tile * 16u + lane] = gated_value(sum, other);
}

struct TokenDownParams {
    Teams at;
    const uint8_t *data;
    size_t matrix_bytes;
    const uint32_t *ids;
    uint32_t experts;
    const float *x;
    float *out;
};

__global__ void __launch_bounds__(kMaxWarps * 32) token_down_kernel(const TokenDownParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ float rows[kMaxWarps][16];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, W = p.at.width, slot = blockIdx.y;
    const uint32_t team = warp / W, member = warp % W, tile = blockIdx.x * p.at.teams + team;
    uint8_t *lines = smem + warp * (kSliceBytes + p.at.records * kQ4SuperBytes), *stage = lines + kSliceBytes;
    const bool live = tile < p.at.row_tiles;
    pdl_launch_dependents();
    const auto fetch = [&](uint32_t expert) {
        if (live && expert < p.experts)
            for (uint32_t r = 0, s = member; r < p.at.records && s < p.at.supers; ++r, s += W)
                fetch_record<kQ4SuperBytes>(stage + r * kQ4SuperBytes,
                                            p.data + expert * p.matrix_bytes + ((size_t)tile * p.at.supers + s) * kQ4SuperBytes, lane);
        cp_async_commit();
    };
    // The kernel before this one starts it once its selection is published; what is read here is only believed after the
    // wait, when the word is read again.
    const uint32_t early = __shfl_sync(0xffffffffu, *reinterpret_cast<const volatile uint32_t *>(p.ids + slot), 0);
    fetch(early);
    pdl_wait();
    const uint32_t expert = __shfl_sync(0xffffffffu, *reinterpret_cast<const volatile uint32_t *>(p.ids + slot), 0);
    if (expert != early) {
        cp_async_wait<0>();
        __syncwarp();
        fetch(expert);
    }
    if (!live || expert >= p.experts) return;  // whole teams; a slot of another rank
    float v0 = 0.0f, v1 = 0.0f;
    for (uint32_t r = 0, s = member; r < p.at.records && s < p.at.supers; ++r, s += W) {
        float v[8], xa, xb;
        load8(p.x + ((size_t)slot * p.at.supers + s) * 256u + lane * 8u, v);
        const float down = stage_slice(v, lines, lane, xa, xb);
        if (r == 0) {
            cp_async_wait<0>();
            __syncwarp();
        }
        q4_record(stage + r * kQ4SuperBytes, lines, down, xa, xb, lane, v0, v1);
    }
    if ((lane & 3u) == 0) rows[warp][lane >> 2] = v0, rows[warp][(lane >> 2) + 8u] = v1;
    if (W > 1u) named_bar_sync(1 + (int)team, (int)W * 32);
    else __syncwarp();
    if (member || lane >= 16u || tile * 16u + lane >= p.at.rows) return;
    float sum = 0.0f;
    for (uint32_t m = 0; m < W; ++m) sum += rows[warp + m][lane];
    p.out[(size_t)slot * p.at.rows + tile * 16u + lane] = sum;
}

constexpr uint32_t kMixThreads = 128;
__global__ void __launch_bounds__(kMixThreads) token_mix_kernel(float *x, const float *rows, const float *probs, uint32_t active,
                                                                uint32_t hidden) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t i = blockIdx.x * kMixThreads + threadIdx.x;
    if (i >= hidden) return;
    const float before = x[i];
    float r = 0.0f;
    if (probs) {
#pragma unroll 8
        for (uint32_t e = 0; e < active; ++e) r = fmaf(probs[e], rows[(size_t)e * hidden + i], r);
    } else {
        r = rows[i];
    }
    x[i] = before + r;
}

// A warp a super-block up to 16 of them; `warps` per CTA (16 where one team needs more).
Teams teams_of(const QMatrix *w, uint32_t warps) {
    Teams at{};
    const Members m = members_of(w->columns);
    at.supers = m.supers, at.width = m.width, at.records = m.records;
    at.row_tiles = w->row_tiles;
    at.rows = w->rows;
    at.teams = std::max(1u, warps / at.width);
    return at;
}
dim3 teams_grid(const Teams &at, uint32_t slots) { return dim3((at.row_tiles + at.teams - 1u) / at.teams, slots); }
size_t teams_smem(const Teams &at, uint32_t record_bytes) {
    return (size_t)at.teams * at.width * (kSliceBytes + (size_t)at.records * record_bytes);
}

constexpr int kTokenSmem = 227 * 1024 - 4096;  // dynamic, beside the partial rows
// Eight warps a CTA for gate and up, so that the 384 CTAs of 8 x 768 rows spread over the SMs within one or two of each other.
constexpr uint32_t kQ8Warps = 16, kGateUpWarps = 8, kDownWarps = 16;

bool fits(const QMatrix *w, QFormat format, uint32_t warps, uint32_t record_bytes) {
    if (w->format != format || w->columns % 256u || w->columns == 0) return false;
    const Teams at = teams_of(w, warps);
    return at.width <= kMaxWarps && teams_smem(at, record_bytes) <= (size_t)kTokenSmem;
}

}  // namespace

bool token_q8_supports(const QMatrix *w) { return fits(w, kFmtQ8_0T, kQ8Warps, kB8SuperBytes); }
bool token_gate_up_supports(const QMatrix *w) { return fits(w, kFmtQ4_K, kGateUpWarps, 2u * kQ4SuperBytes); }
bool token_down_supports(const QMatrix *w) { return fits(w, kFmtQ4_K, kDownWarps, kQ4SuperBytes); }

stark_b200_status token_q8_launch(const QMatrix *w, const float *x, const float *norm, float eps, const float *residual,
                                  float *out, bool pdl, cudaStream_t stream) {
    static SmemOptIn once;
    if (stark_b200_status s = ensure_dynamic_smem(token_q8_kernel, kTokenSmem, once)) return s;
    const TokenQ8Params p{teams_of(w, kQ8Warps), w->data, x, norm, residual, eps, out};
    return moe_launch(token_q8_kernel, teams_grid(p.at, 1), p.at.teams * p.at.width * 32u, teams_smem(p.at, kB8SuperBytes), pdl, stream, p);
}

stark_b200_status token_attention_launch(const uint32_t *position, const float *qkv, bool raw, float *keys, float *values,
                                         float *part, uint32_t splits, uint32_t q_heads, uint32_t kv_heads, uint32_t context,
                                         const float *q_norm, const float *k_norm, float eps, float theta, bool pdl,
                                         cudaStream_t stream) {
    const uint32_t group = q_heads / kv_heads;
    const auto kernel = group == 8u ? token_attention_kernel<8> : (group == 4u ? token_attention_kernel<4> : token_attention_kernel<2>);
    return moe_launch(kernel, dim3(kv_heads, splits), kTokenAttnWarps * 32u, 0, pdl, stream, position, qkv, raw, keys, values, part,
                  splits, kv_heads, 1.0f / sqrtf((float)kDim), context, q_norm, k_norm, eps, theta);
}

stark_b200_status token_merge_launch(const uint32_t *position, const float *part, float *out, uint32_t splits, uint32_t q_heads,
                                     uint32_t context, bool pdl, cudaStream_t stream) {
    if (splits > 64u) return STARK_B200_INVALID_ARGUMENT;  // two spans a lane
    return moe_launch(token_merge_kernel, q_heads, kDim, 0, pdl, stream, position, part, out, splits, context);
}

stark_b200_status token_router_launch(const float *router, const float *x, const float *norm, float eps, float *scores,
                                      uint32_t hidden, uint32_t experts, bool pdl, cudaStream_t stream) {
    const Members at = members_of(hidden);
    return moe_launch(token_router_kernel, experts, at.width * 32u, 0, pdl, stream, router, x, norm, eps, scores, at);
}

stark_b200_status token_gate_up_launch(const QMatrix *w, const TokenSelection &sel, const float *x, const float *norm, float eps,
                                       float *act, bool pdl, cudaStream_t stream) {
    const Teams at = teams_of(w, kGateUpWarps);
    const int slot = (sel.experts <= 128u ? 0 : 1) + (at.teams * at.width <= kGateUpWarps ? 0 : 2);
    void (*const kernels[4])(TokenGateUpParams) = {token_gate_up_kernel<4, kGateUpWarps>, token_gate_up_kernel<32, kGateUpWarps>,
                                                   token_gate_up_kernel<4, kMaxWarps>, token_gate_up_kernel<32, kMaxWarps>};
    static SmemOptIn once[4];
    if (stark_b200_status s = ensure_dynamic_smem(kernels[slot], kTokenSmem, once[slot])) return s;
    const TokenGateUpParams p{at, sel, w->data, (size_t)at.row_tiles * at.supers * kQ4SuperBytes, x, norm, eps, act};
    return moe_launch(kernels[slot], teams_grid(at, sel.active), at.teams * at.width * 32u, teams_smem(at, 2u * kQ4SuperBytes), pdl, stream, p);
}

stark_b200_status token_down_launch(const QMatrix *w, const uint32_t *ids, uint32_t active, const float *act, float *out, bool pdl,
                                    cudaStream_t stream) {
    static SmemOptIn once;
    if (stark_b200_status s = ensure_dynamic_smem(token_down_kernel, kTokenSmem, once)) return s;
    const Teams at = teams_of(w, kDownWarps);
    const TokenDownParams p{at, w->data, (size_t)at.row_tiles * at.supers * kQ4SuperBytes, ids, w->experts ? w->experts : 1u, act, out};
    return moe_launch(token_down_kernel, teams_grid(at, active), at.teams * at.width * 32u, teams_smem(at, kQ4SuperBytes), pdl, stream, p);
}

stark_b200_status token_mix_launch(float *x, const float *rows, const float *probs, uint32_t active, uint32_t hidden, bool pdl,
                                   cudaStream_t stream) {
    return moe_launch(token_mix_kernel, (hidden + kMixThreads - 1u) / kMixThreads, kMixThreads, 0, pdl, stream, x, rows, probs, active,
                  hidden);
}

}  // namespace sb
