// Prompt rows of the routed-expert decoder: a pass of up to 512 rows through the operators of a token (moe_model.cu), f32
// activations throughout.  The reference batches them in 256-row passes with the rows grouped by expert
// (crates/stark-engine/src/encodable_block/decoder.rs:182-186, mlp/routed.rs:144-256).
//
// A token reads every active weight for one row; a pass reads a weight record once for 16 rows.  The contractions keep the
// token's arithmetic: codes as exact f16 integers on the M side of mma.sync.m16n8k16, an input row as f16 head and remainder
// (~22 bits) in two of the eight N columns -- four rows fill the tile that one row's copies filled -- and the block scales
// applied in f32 to every sub-block's sums.  (tcgen05 accumulates over the whole contraction, so the scales would have to
// go into the weights, which then need a remainder of their own and the input's 22 bits three products instead of two.)
//
// 12 layers of the 30B-A3B shape, 160 rows and the token behind them: 5.9 ms against 112 ms token by token.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "context.cuh"
#include "gguf_math.cuh"
#include "moe_rows.cuh"
#include "moe_select.cuh"

namespace sb {

namespace {

constexpr uint32_t kNt = kMoeRowsChunk / 4u;         // column tiles of four rows
static_assert(kNt == 4u, "run() below has a loop for each");
constexpr uint32_t kLine = 512u + 64u;               // a row's head or remainder of 256 columns: two lines 64 B apart modulo 128 B
constexpr uint32_t kTileLines = kMoeRowsChunk * 2u;  // lines of a stage

struct RowsGemmParams {
    const uint8_t *data;
    uint32_t rows, row_tiles, supers, row_blocks;  // of one matrix; row_blocks: its CTAs
    size_t matrix_bytes;
    const __half *x;
    const float *unscale, *sums;
    float *out;
    uint32_t out_stride;
    uint32_t m;                            // dense: input rows
    const uint32_t *tiles, *pairs;         // experts: see MoeRowLists
    uint32_t divisor, experts;
};

// One CTA: 16 matrix rows a warp times up to 16 input rows, the contraction in steps of 256 columns, copies of the
// next steps in flight.  Bound by issue slots of the tensor-core loop at full tiles (10 instructions per two products) and by
// the weights' bytes where experts have few rows.
template <bool Q4, int STAGES, uint32_t WARPS>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8u ? 2 : 1) rows_gemm_kernel(const RowsGemmParams p) {
    constexpr uint32_t kSuper = Q4 ? kQ4SuperBytes : kB8SuperBytes;
    constexpr uint32_t kStage = WARPS * kSuper + kTileLines * kLine + (Q4 ? kMoeRowsChunk * 32u : 0u);
    extern __shared__ __align__(16) uint8_t rows_smem[];
    __shared__ uint32_t ids[kMoeRowsChunk];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, g = lane >> 2, t = lane & 3u;
    pdl_launch_dependents();
    pdl_wait();
    uint32_t matrix = 0, block = blockIdx.x, count;
    if (p.tiles) {
        if (blockIdx.y >= p.tiles[0]) return;
        const uint32_t *tile = p.tiles + 1u + 3u * blockIdx.y;
        matrix = tile[0] + block / p.row_blocks * p.experts;
        block %= p.row_blocks;
        count = tile[2];
        if (tid < count) ids[tid] = p.pairs[tile[1] + tid];
    } else {
        const uint32_t first = blockIdx.y * kMoeRowsChunk;
        count = min(kMoeRowsChunk, p.m - first);
        if (tid < count) ids[tid] = first + tid;
    }
    __syncthreads();
    const uint32_t row_tile = block * WARPS + warp;
    const bool live = row_tile < p.row_tiles;
    const uint8_t *weights = p.data + (size_t)matrix * p.matrix_bytes + (size_t)row_tile * p.supers * kSuper;
    const size_t columns = (size_t)p.supers * 256u;
    const uint32_t live_nt = (count + 3u) / 4u;

    const auto issue = [&](uint32_t s) {
        if (s < p.supers) {
            uint8_t *stage = rows_smem + (s % STAGES) * kStage;
            if (live)
                for (uint32_t off = lane * 16u; off < kSuper; off += 512u)
                    cp_async16(stage + warp * kSuper + off, weights + (size_t)s * kSuper + off);
            uint8_t *lines = stage + WARPS * kSuper;
            for (uint32_t i = tid; i < count * 64u; i += WARPS * 32u) {
                const uint32_t line = i >> 5, c = i & 31u;
                cp_async16(lines + line * kLine + c * 16u,
                           p.x + ((size_t)(ids[line >> 1] / p.divisor) * 2u + (line & 1u)) * columns + s * 256u + c * 8u);
            }
            if (Q4 && tid < count * 2u)
                cp_async16(lines + kTileLines * kLine + tid * 16u,
                           p.sums + (size_t)(ids[tid >> 1] / p.divisor) * (p.supers * 8u) + s * 8u + (tid & 1u) * 4u);
        }
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) issue(s);

    float acc0[kNt], acc1[kNt];  // matrix rows g and g + 8, input row t of every column tile
#pragma unroll
    for (uint32_t n = 0; n < kNt; ++n) acc0[n] = acc1[n] = 0.0f;
    // The loop for a number of column tiles known to the compiler: their products are independent chains, which a test in
    // between kept apart (a warp waited 2.6 cycles an instruction for the one before it).
    const auto run = [&](auto tiles) {
        constexpr uint32_t NT = decltype(tiles)::value;
        for (uint32_t s = 0; s < p.supers; ++s) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();  // every thread's copies of this step are there, and everybody is done with the step before
            issue(s + STAGES - 1);
            if (!live) continue;
            const uint8_t *rec = rows_smem + (s % STAGES) * kStage + warp * kSuper;
            const uint8_t *lines = rows_smem + (s % STAGES) * kStage + WARPS * kSuper + g * kLine + t * 16u;
            const float *sums = reinterpret_cast<const float *>(rows_smem + (s % STAGES) * kStage + WARPS * kSuper + kTileLines * kLine);
            float dsc0[2], dm0[2], dsc1[2], dm1[2];
            if (Q4) {
                q4k_scales_pair(*reinterpret_cast<const uint4 *>(rec + 2048u + 16u * g), t, dsc0, dm0);
                q4k_scales_pair(*reinterpret_cast<const uint4 *>(rec + 2048u + 16u * (g + 8u)), t, dsc1, dm1);
            }
#pragma unroll
            for (uint32_t jb = 0; jb < 8; ++jb) {
                uint32_t a[8];
                float s0, s1, m0 = 0.0f, m1 = 0.0f;
                if (Q4) {
                    const uint2 w = *reinterpret_cast<const uint2 *>(rec + jb * 256u + lane * 8u);
                    dequant_a4_word<0>(w.x, *reinterpret_cast<uint32_t(*)[4]>(&a[0]));
                    dequant_a4_word<0>(w.y, *reinterpret_cast<uint32_t(*)[4]>(&a[4]));
                    // lane jb mod 4 of the four that share these rows decoded this sub-block's scales
                    const uint32_t from = (lane & ~3u) | (jb & 3u);
                    s0 = __shfl_sync(0xffffffffu, dsc0[jb >> 2], from), s1 = __shfl_sync(0xffffffffu, dsc1[jb >> 2], from);
                    m0 = __shfl_sync(0xffffffffu, dm0[jb >> 2], from), m1 = __shfl_sync(0xffffffffu, dm1[jb >> 2], from);
                } else {
                    const uint4 w = *reinterpret_cast<const uint4 *>(rec + jb * 512u + lane * 16u);
                    bytes_to_f16<false>(w.x, a[0], a[1]);
                    bytes_to_f16<false>(w.y, a[2], a[3]);
                    bytes_to_f16<false>(w.z, a[4], a[5]);
                    bytes_to_f16<false>(w.w, a[6], a[7]);
                    const uint16_t *meta = reinterpret_cast<const uint16_t *>(rec + 4096u);
                    s0 = f16_bits_f32(meta[jb * 16u + g]), s1 = f16_bits_f32(meta[jb * 16u + g + 8u]);
                }
                uint4 xv[NT];
                float c[NT][4];
#pragma unroll
                for (uint32_t n = 0; n < NT; ++n) {
                    xv[n] = *reinterpret_cast<const uint4 *>(lines + n * 8u * kLine + jb * 64u);
                    c[n][0] = c[n][1] = c[n][2] = c[n][3] = 0.0f;
                }
#pragma unroll
                for (uint32_t n = 0; n < NT; ++n) mma_m16n8k16_f16(c[n], *reinterpret_cast<uint32_t(*)[4]>(&a[0]), xv[n].x, xv[n].y);
#pragma unroll
                for (uint32_t n = 0; n < NT; ++n) mma_m16n8k16_f16(c[n], *reinterpret_cast<uint32_t(*)[4]>(&a[4]), xv[n].z, xv[n].w);
#pragma unroll
                for (uint32_t n = 0; n < NT; ++n) {
                    acc0[n] = fmaf(s0, c[n][0] + c[n][1], acc0[n]);
                    acc1[n] = fmaf(s1, c[n][2] + c[n][3], acc1[n]);
                    if (Q4) {
                        const float xs = sums[(n * 4u + t) * 8u + jb];
                        acc0[n] = fmaf(-m0, xs, acc0[n]);
                        acc1[n] = fmaf(-m1, xs, acc1[n]);
                    }
                }
            }
        }
    };
    if (live_nt <= 1u) run(std::integral_constant<uint32_t, 1>());
    else if (live_nt == 2u) run(std::integral_constant<uint32_t, 2>());
    else if (live_nt == 3u) run(std::integral_constant<uint32_t, 3>());
    else run(std::integral_constant<uint32_t, 4>());
    if (!live) return;
    const uint32_t r0 = row_tile * 16u + g, r1 = r0 + 8u;
    const size_t column = p.tiles ? (size_t)(blockIdx.x / p.row_blocks) * p.rows : 0u;
#pragma unroll
    for (uint32_t n = 0; n < kNt; ++n) {
        const uint32_t i = n * 4u + t;
        if (i >= count) continue;
        const uint32_t id = ids[i];
        const float unscale = p.unscale[id / p.divisor];
        float *y = p.out + (size_t)id * p.out_stride + column;
        if (r0 < p.rows) y[r0] = acc0[n] * unscale;
        if (r1 < p.rows) y[r1] = acc1[n] * unscale;
    }
}

template <int THREADS, typename F>
__device__ inline float row_reduce(float v, F f, float *scratch /* [THREADS / 32] */) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = f(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    float r = scratch[0];
#pragma unroll
    for (int w = 1; w < THREADS / 32; ++w) r = f(r, scratch[w]);
    return r;
}

__device__ inline float4 read4(const float *p) { return *reinterpret_cast<const float4 *>(p); }

// One row, in shared memory, as an operand; a thread takes four columns at a time.  The scale is the largest power of two that
// keeps the head in f16's range, as the one-row matvecs choose it; columns are a multiple of 256, so eight lanes hold 32
// consecutive ones.
template <int THREADS>
__device__ inline void split_row(const float *row, float largest, const RowsOperand &out, uint32_t at) {
    int shift = 14 - ((int)((__float_as_uint(largest) >> 23) & 0xffu) - 127);
    shift = max(-100, min(100, shift));
    if (!(largest > 0.0f) || !isfinite(largest)) shift = 0;
    const float scale = __uint_as_float((uint32_t)(shift + 127) << 23);
    __half *head = out.split + (size_t)at * 2u * out.columns, *rest = head + out.columns;
    for (uint32_t i = threadIdx.x * 4u; i < out.columns; i += THREADS * 4u) {
        const float4 r = read4(row + i);
        const float v[4] = {r.x * scale, r.y * scale, r.z * scale, r.w * scale};
        __half2 h[2], l[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            h[j] = __floats2half2_rn(v[2 * j], v[2 * j + 1]);
            l[j] = __floats2half2_rn(v[2 * j] - __low2float(h[j]), v[2 * j + 1] - __high2float(h[j]));
        }
        *reinterpret_cast<uint2 *>(head + i) = make_uint2(*reinterpret_cast<uint32_t *>(&h[0]), *reinterpret_cast<uint32_t *>(&h[1]));
        *reinterpret_cast<uint2 *>(rest + i) = make_uint2(*reinterpret_cast<uint32_t *>(&l[0]), *reinterpret_cast<uint32_t *>(&l[1]));
        float s = (v[0] + v[1]) + (v[2] + v[3]);
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if ((threadIdx.x & 7u) == 0) out.sums[(size_t)at * (out.columns / 32u) + (i >> 5)] = s;
    }
    if (threadIdx.x == 0) out.unscale[at] = __uint_as_float((uint32_t)(127 - shift) << 23);
}

constexpr int kRowThreads = 512;
__device__ inline float larger(float a, float b) { return fmaxf(a, b); }
__device__ inline float added(float a, float b) { return a + b; }

// rms_norm of a row in shared memory (math.rs:18-34), in place, and its operand.  Every thread its own four columns throughout.
__device__ inline void norm_and_split(float *row, const float *w, float eps, float *normed, const RowsOperand &out, uint32_t at,
                                      float *scratch) {
    const uint32_t n = out.columns;
    float s = 0.0f;
    for (uint32_t i = threadIdx.x * 4u; i < n; i += kRowThreads * 4u) {
        const float4 v = read4(row + i);
        s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    }
    const float scale = 1.0f / sqrtf(row_reduce<kRowThreads>(s, added, scratch) / (float)n + eps);
    float mx = 0.0f;
    for (uint32_t i = threadIdx.x * 4u; i < n; i += kRowThreads * 4u) {
        float4 v = read4(row + i);
        const float4 g = read4(w + i);
        v.x = v.x * scale * g.x, v.y = v.y * scale * g.y, v.z = v.z * scale * g.z, v.w = v.w * scale * g.w;
        *reinterpret_cast<float4 *>(row + i) = v;
        if (normed) *reinterpret_cast<float4 *>(normed + i) = v;
        mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
    split_row<kRowThreads>(row, row_reduce<kRowThreads>(mx, larger, scratch), out, at);
}

__global__ void __launch_bounds__(kRowThreads) moe_rows_embed_kernel(const uint32_t *tokens, const uint8_t *table, float *x,
                                                                     const float *w, float eps, const RowsOperand out) {
    extern __shared__ __align__(16) float row[];
    __shared__ float scratch[kRowThreads / 32];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t H = out.columns, at = blockIdx.x;
    const uint8_t *src = table + (size_t)tokens[at] * (H / 32u) * 34u;
    for (uint32_t i = threadIdx.x; i < H; i += kRowThreads) {
        const uint8_t *b = src + (i >> 5) * 34u;
        const float d = __half2float(__ushort_as_half((unsigned short)(b[0] | (b[1] << 8))));
        const float v = d * (float)(int8_t)b[2u + (i & 31u)];
        row[i] = v;
        x[(size_t)at * H + i] = v;
    }
    __syncthreads();
    norm_and_split(row, w, eps, nullptr, out, at, scratch);
}

// moe_heads_kernel for the rows of a pass: one CTA of `dim` threads per head and row.
__global__ void moe_rows_heads_kernel(float *qkv, const float *q_norm, const float *k_norm, float *keys, float *values,
                                      uint32_t q_heads, uint32_t kv_heads, uint32_t dim, float eps, float theta,
                                      uint32_t first_pos) {
    pdl_launch_dependents();
    pdl_wait();
    __shared__ float scratch[32];
    __shared__ float head[256];
    const uint32_t h = blockIdx.x, i = threadIdx.x, position = first_pos + blockIdx.y;
    const size_t kv_row = (size_t)kv_heads * dim;
    float *src = qkv + ((size_t)blockIdx.y * (q_heads + 2u * kv_heads) + h) * dim;
    if (h >= q_heads + kv_heads) {
        values[position * kv_row + (size_t)(h - q_heads - kv_heads) * dim + i] = src[i];
        return;
    }
    const float v = src[i];
    float s = v * v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((i & 31u) == 0) scratch[i >> 5] = s;
    __syncthreads();
    float sum = 0.0f;
    for (uint32_t w = 0; w < dim / 32u; ++w) sum += scratch[w];
    const float scale = 1.0f / sqrtf(sum / (float)dim + eps);
    head[i] = v * scale * (h < q_heads ? q_norm : k_norm)[i];
    __syncthreads();
    const uint32_t half = dim / 2u, pair = i < half ? i : i - half;
    const float angle = (float)position * powf(theta, -((float)(2u * pair)) / (float)dim);
    float sn, cs;
    sincosf(angle, &sn, &cs);
    const float a = head[pair], b = head[pair + half];
    const float out = i < half ? a * cs - b * sn : a * sn + b * cs;
    if (h < q_heads)
        src[i] = out;
    else
        keys[position * kv_row + (size_t)(h - q_heads) * dim + i] = out;
}

// moe_attention_merge_kernel for a whole row, and the row's operand.
__global__ void __launch_bounds__(kRowThreads) moe_rows_merge_kernel(const float *part, uint32_t splits, const RowsOperand out) {
    constexpr uint32_t D = 128;
    extern __shared__ __align__(16) float row[];
    __shared__ float scratch[kRowThreads / 32];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t heads = out.columns / D;
    float mx = 0.0f;
    for (uint32_t i = threadIdx.x; i < out.columns; i += kRowThreads) {
        const float *src = part + ((size_t)blockIdx.x * heads + i / D) * splits * (D + 2u);
        float gm = -INFINITY;
        for (uint32_t s = 0; s < splits; ++s) gm = fmaxf(gm, src[s * (D + 2u)]);
        float l = 0.0f, a = 0.0f;
        for (uint32_t s = 0; s < splits; ++s) {
            const float m = src[s * (D + 2u)];
            const float c = m == -INFINITY ? 0.0f : expf(m - gm);  // an empty span weighs nothing
            l += src[s * (D + 2u) + 1u] * c;
            a += src[s * (D + 2u) + 2u + i % D] * c;
        }
        const float v = a / l;
        row[i] = v;
        mx = fmaxf(mx, fabsf(v));
    }
    split_row<kRowThreads>(row, row_reduce<kRowThreads>(mx, larger, scratch), out, blockIdx.x);
}

__global__ void __launch_bounds__(kRowThreads) moe_rows_add_norm_kernel(float *x, const float *update, const float *probs,
                                                                        uint32_t active, const float *w, float eps, float *normed,
                                                                        const RowsOperand out, uint32_t hidden) {
    extern __shared__ __align__(16) float row[];
    __shared__ float scratch[kRowThreads / 32];
    __shared__ float share[32];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t at = blockIdx.x;
    if (probs && threadIdx.x < active) share[threadIdx.x] = probs[(size_t)at * active + threadIdx.x];
    __syncthreads();
    const float *rows = update + (size_t)at * (probs ? active : 1u) * hidden;
    for (uint32_t i = threadIdx.x * 4u; i < hidden; i += kRowThreads * 4u) {
        float4 *home = reinterpret_cast<float4 *>(x + (size_t)at * hidden + i);
        float4 v = *home, r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (probs) {
#pragma unroll 8
            for (uint32_t e = 0; e < active; ++e) {
                const float4 o = read4(rows + (size_t)e * hidden + i);
                r.x += share[e] * o.x, r.y += share[e] * o.y, r.z += share[e] * o.z, r.w += share[e] * o.w;
            }
        } else {
            r = read4(rows + i);
        }
        v.x += r.x, v.y += r.y, v.z += r.z, v.w += r.w;
        *home = v;
        *reinterpret_cast<float4 *>(row + i) = v;
    }
    if (w) norm_and_split(row, w, eps, normed ? normed + (size_t)at * hidden : nullptr, out, at, scratch);
}

// Router scores of four rows and kRouteWarps experts a CTA: a warp multiplies one router row with the four.  (All experts of
// four rows in one CTA took 40 us: the 1 MB of router rows went by one after another.)
constexpr uint32_t kRouteRows = 4, kRouteWarps = 8;
__global__ void __launch_bounds__(kRouteWarps * 32) moe_rows_scores_kernel(const float *router, const float *normed, uint32_t hidden,
                                                                           uint32_t experts, float *scores, uint32_t rows) {
    pdl_launch_dependents();
    const uint32_t lane = threadIdx.x & 31u, e = blockIdx.y * kRouteWarps + (threadIdx.x >> 5), first = blockIdx.x * kRouteRows;
    if (e >= experts) {
        pdl_wait();
        return;
    }
    const float4 *w = reinterpret_cast<const float4 *>(router + (size_t)e * hidden);
    const float4 *x[kRouteRows];
#pragma unroll
    for (uint32_t r = 0; r < kRouteRows; ++r)
        x[r] = reinterpret_cast<const float4 *>(normed + (size_t)min(first + r, rows - 1u) * hidden);
    constexpr uint32_t kAhead = 4;
    float4 a[kAhead];
    const auto fetch = [&](uint32_t from) {
#pragma unroll
        for (uint32_t j = 0; j < kAhead; ++j)
            if (from + 32u * j < hidden / 4u) a[j] = w[from + 32u * j];
    };
    fetch(lane);
    pdl_wait();
    float s[kRouteRows] = {};
    for (uint32_t from = lane; from < hidden / 4u; from += 32u * kAhead) {
        float4 now[kAhead];
#pragma unroll
        for (uint32_t j = 0; j < kAhead; ++j) now[j] = a[j];
        fetch(from + 32u * kAhead);
#pragma unroll
        for (uint32_t j = 0; j < kAhead; ++j) {
            const uint32_t i = from + 32u * j;
            if (i >= hidden / 4u) break;
#pragma unroll
            for (uint32_t r = 0; r < kRouteRows; ++r) {
                const float4 b = x[r][i];
                s[r] += now[j].x * b.x + now[j].y * b.y + now[j].z * b.z + now[j].w * b.w;
            }
        }
    }
#pragma unroll
    for (uint32_t r = 0; r < kRouteRows; ++r) {
        s[r] = warp_sum(s[r]);
        if (lane == 0 && first + r < rows) scores[(size_t)(first + r) * experts + e] = s[r];
    }
}

// A warp a row: the selection and its weights, as a token makes them (moe_token.cuh).
constexpr uint32_t kSelectWarps = 4;
template <int KEYS>
__global__ void __launch_bounds__(kSelectWarps * 32) moe_rows_select_kernel(const float *scores, uint32_t experts, uint32_t active,
                                                                            uint32_t *ids, float *probs, uint32_t *last_ids,
                                                                            uint32_t rows) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31u, row = blockIdx.x * kSelectWarps + (threadIdx.x >> 5);
    if (row >= rows) return;
    uint32_t key[KEYS];
#pragma unroll
    for (int j = 0; j < KEYS; ++j) key[j] = lane + 32u * j < experts ? order_key(scores[(size_t)row * experts + lane + 32u * j]) : 0u;
    uint32_t chosen = 0, chosen_key = 0;
    for (uint32_t r = 0; r < active; ++r) {
        uint32_t top;
        const uint32_t pick = take_first_largest(key, lane, top);
        if (r == lane) chosen = pick, chosen_key = top;
    }
    const float share = selection_share(key_value(chosen_key), active, lane);
    if (lane < active) {
        ids[(size_t)row * active + lane] = chosen;
        probs[(size_t)row * active + lane] = share;
        if (row + 1u == rows) {
            last_ids[lane] = chosen;
            last_ids[active + lane] = chosen + experts;
        }
    }
}

// Pairs by expert and the tiles over them: a count, a scan and a scatter in one CTA.  The order of an expert's pairs is
// whatever the scatter makes it; a pair's results do not depend on its place in a tile.
constexpr uint32_t kListThreads = 1024;
__global__ void __launch_bounds__(kListThreads) moe_rows_lists_kernel(const uint32_t *ids, uint32_t *pairs, uint32_t *tiles,
                                                                      uint32_t count, uint32_t experts) {
    __shared__ uint32_t counts[1024], starts[1024], sums[2][32];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    counts[tid] = 0;
    __syncthreads();
    for (uint32_t i = tid; i < count; i += kListThreads) atomicAdd(&counts[ids[i]], 1u);
    __syncthreads();
    const uint32_t mine = tid < experts ? counts[tid] : 0u, chunks = (mine + kMoeRowsChunk - 1u) / kMoeRowsChunk;
    uint32_t upto = mine, tiles_upto = chunks;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t a = __shfl_up_sync(0xffffffffu, upto, o), b = __shfl_up_sync(0xffffffffu, tiles_upto, o);
        if (lane >= (uint32_t)o) upto += a, tiles_upto += b;
    }
    if (lane == 31u) sums[0][warp] = upto, sums[1][warp] = tiles_upto;
    __syncthreads();
    for (uint32_t w = 0; w < warp; ++w) upto += sums[0][w], tiles_upto += sums[1][w];
    const uint32_t start = upto - mine;
    starts[tid] = start;
    counts[tid] = 0;
    for (uint32_t c = 0, at = tiles_upto - chunks; c < chunks; ++c, ++at) {
        tiles[1u + 3u * at] = tid;
        tiles[2u + 3u * at] = start + c * kMoeRowsChunk;
        tiles[3u + 3u * at] = min(kMoeRowsChunk, mine - c * kMoeRowsChunk);
    }
    if (tid == kListThreads - 1u) tiles[0] = tiles_upto;
    __syncthreads();
    for (uint32_t i = tid; i < count; i += kListThreads) pairs[starts[ids[i]] + atomicAdd(&counts[ids[i]], 1u)] = i;
}

constexpr int kGateThreads = 256;
__global__ void __launch_bounds__(kGateThreads) moe_rows_gate_kernel(const float *gate_up, const RowsOperand out) {
    extern __shared__ __align__(16) float row[];
    __shared__ float scratch[kGateThreads / 32];
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t I = out.columns;
    const float *gate = gate_up + (size_t)blockIdx.x * 2u * I, *up = gate + I;
    float mx = 0.0f;
    for (uint32_t i = threadIdx.x; i < I; i += kGateThreads) {  // silu with the two-branch sigmoid (math.rs:5-16)
        const float g = gate[i];
        float sg;
        if (g >= 0.0f) {
            sg = 1.0f / (1.0f + expf(-g));
        } else {
            const float e = expf(g);
            sg = e / (1.0f + e);
        }
        const float v = g * sg * up[i];
        row[i] = v;
        mx = fmaxf(mx, fabsf(v));
    }
    split_row<kGateThreads>(row, row_reduce<kGateThreads>(mx, larger, scratch), out, blockIdx.x);
}

// A launch that may start before its predecessor ends: every kernel here awaits it before its first access.
template <typename... Params, typename... Args>
stark_b200_status launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    SB_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
    return STARK_B200_OK;
}

// The kernels that hold a row in shared memory: the widest takes 48 KB beside their own words, more than a launch has unasked.
template <typename... Params, typename... Args>
stark_b200_status launch_row(SmemOptIn &once, void (*kernel)(Params...), dim3 grid, dim3 block, uint32_t columns, cudaStream_t stream,
                             Args... args) {
    if (columns > kMoeRowsWidest) return STARK_B200_UNSUPPORTED;
    if (stark_b200_status s = ensure_dynamic_smem(kernel, (int)kMoeRowsWidest * 4, once)) return s;
    return launch(kernel, grid, block, (size_t)columns * 4u, stream, args...);
}

constexpr size_t gemm_smem(uint32_t stages, uint32_t warps, uint32_t super_bytes, uint32_t sums) {
    return stages * (warps * super_bytes + kTileLines * kLine + sums);
}
constexpr uint32_t kQ4Stages = 3, kQ4Warps = 8;
constexpr size_t kQ4Smem = gemm_smem(kQ4Stages, kQ4Warps, kQ4SuperBytes, kMoeRowsChunk * 32u);

RowsGemmParams gemm_params(const QMatrix *w, uint32_t super_bytes, uint32_t warps, const RowsOperand &x, float *out) {
    RowsGemmParams p{};
    p.data = w->data;
    p.rows = w->rows;
    p.row_tiles = w->row_tiles;
    p.supers = w->columns / 256u;
    p.row_blocks = (w->row_tiles + warps - 1u) / warps;
    p.matrix_bytes = (size_t)w->row_tiles * p.supers * super_bytes;
    p.x = x.split;
    p.unscale = x.unscale;
    p.sums = x.sums;
    p.out = out;
    p.divisor = 1;
    return p;
}

}  // namespace

stark_b200_status rows_q8_launch(const QMatrix *w, const RowsOperand &x, float *out, uint32_t rows, cudaStream_t stream) {
    if (w->format != kFmtQ8_0T || w->columns != x.columns || rows == 0) return STARK_B200_INVALID_ARGUMENT;
    // A few rows of a small matrix are few CTAs of 128 rows (16 for 2 048 x 4 096: 38 us at 11 rows), each a chain of copies: 32
    // rows a CTA then, with twice the steps in flight.
    const uint32_t chunks = (rows + kMoeRowsChunk - 1u) / kMoeRowsChunk;
    const bool narrow = (w->row_tiles + 7u) / 8u * chunks < 148u;
    const uint32_t warps = narrow ? 2u : 8u;
    const size_t smem = gemm_smem(narrow ? 4u : 2u, warps, kB8SuperBytes, 0u);
    const auto kernel = narrow ? rows_gemm_kernel<false, 4, 2> : rows_gemm_kernel<false, 2, 8>;
    static SmemOptIn once[2];
    if (stark_b200_status s = ensure_dynamic_smem(kernel, (int)smem, once[narrow])) return s;
    RowsGemmParams p = gemm_params(w, kB8SuperBytes, warps, x, out);
    p.m = rows;
    p.out_stride = w->rows;
    return launch(kernel, dim3(p.row_blocks, chunks), warps * 32u, smem, stream, p);
}

stark_b200_status rows_q4k_experts_launch(const QMatrix *w, uint32_t blocks, const RowsOperand &x, uint32_t divisor, float *out,
                                          const MoeRowLists &lists, uint32_t rows, uint32_t active, cudaStream_t stream) {
    if (w->format != kFmtQ4_K || w->columns != x.columns || rows == 0 || w->experts % blocks) return STARK_B200_INVALID_ARGUMENT;
    static SmemOptIn once;
    if (stark_b200_status s = ensure_dynamic_smem(rows_gemm_kernel<true, kQ4Stages, kQ4Warps>, (int)kQ4Smem, once)) return s;
    RowsGemmParams p = gemm_params(w, kQ4SuperBytes, kQ4Warps, x, out);
    p.experts = w->experts / blocks;
    p.tiles = lists.tiles;
    p.pairs = lists.pairs;
    p.divisor = divisor;
    p.out_stride = blocks * w->rows;
    return launch(rows_gemm_kernel<true, kQ4Stages, kQ4Warps>, dim3(p.row_blocks * blocks, MoeRowLists::max_tiles(rows, active, p.experts)),
                  kQ4Warps * 32u, kQ4Smem, stream, p);
}

stark_b200_status moe_rows_embed_launch(const uint32_t *tokens, const uint8_t *table, float *x, const float *w, float eps,
                                        const RowsOperand &out, uint32_t rows, cudaStream_t stream) {
    static SmemOptIn once;
    return launch_row(once, moe_rows_embed_kernel, rows, kRowThreads, out.columns, stream, tokens, table, x, w, eps, out);
}

stark_b200_status moe_rows_heads_launch(float *qkv, const float *q_norm, const float *k_norm, float *keys, float *values,
                                        uint32_t q_heads, uint32_t kv_heads, uint32_t dim, float eps, float theta,
                                        uint32_t first_pos, uint32_t rows, cudaStream_t stream) {
    return launch(moe_rows_heads_kernel, dim3(q_heads + 2u * kv_heads, rows), dim, 0, stream, qkv, q_norm, k_norm, keys, values,
                  q_heads, kv_heads, dim, eps, theta, first_pos);
}

stark_b200_status moe_rows_merge_launch(const float *part, uint32_t heads, uint32_t splits, const RowsOperand &out,
                                        uint32_t rows, cudaStream_t stream) {
    if (out.columns != heads * 128u) return STARK_B200_INVALID_ARGUMENT;
    static SmemOptIn once;
    return launch_row(once, moe_rows_merge_kernel, rows, kRowThreads, out.columns, stream, part, splits, out);
}

stark_b200_status moe_rows_add_norm_launch(float *x, const float *update, const float *probs, uint32_t active, const float *w,
                                           float eps, float *normed, const RowsOperand &out, uint32_t rows, uint32_t hidden,
                                           cudaStream_t stream) {
    static SmemOptIn once;
    return launch_row(once, moe_rows_add_norm_kernel, rows, kRowThreads, hidden, stream, x, update, probs, active, w, eps,
                  normed, out, hidden);
}

stark_b200_status moe_rows_route_launch(const float *router, const float *normed, uint32_t hidden, uint32_t experts,
                                        uint32_t active, const MoeRowLists &lists, uint32_t *last_ids, uint32_t rows,
                                        cudaStream_t stream) {
    if (stark_b200_status s = launch(moe_rows_scores_kernel, dim3((rows + kRouteRows - 1u) / kRouteRows, (experts + kRouteWarps - 1u) / kRouteWarps),
                                     kRouteWarps * 32u, 0, stream, router, normed, hidden, experts, lists.scores, rows))
        return s;
    return launch(experts <= 128u ? moe_rows_select_kernel<4> : moe_rows_select_kernel<32>, (rows + kSelectWarps - 1u) / kSelectWarps,
                  kSelectWarps * 32u, 0, stream, lists.scores, experts, active, lists.ids, lists.probs, last_ids, rows);
}

stark_b200_status moe_rows_lists_launch(const MoeRowLists &lists, uint32_t rows, uint32_t active, uint32_t experts,
                                        cudaStream_t stream) {
    return launch(moe_rows_lists_kernel, 1, kListThreads, 0, stream, lists.ids, lists.pairs, lists.tiles, rows * active, experts);
}

stark_b200_status moe_rows_gate_launch(const float *gate_up, uint32_t inter, const RowsOperand &out, uint32_t pairs,
                                       cudaStream_t stream) {
    static SmemOptIn once;
    return launch_row(once, moe_rows_gate_kernel, pairs, kGateThreads, inter, stream, gate_up, out);
}

}  // namespace sb
