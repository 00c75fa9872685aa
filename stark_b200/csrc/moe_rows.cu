// Prompt rows of the routed-expert decoder: a pass of up to 512 rows through the operators of a token (moe_token.cu), f32
// activations throughout.  The reference batches them in 256-row passes with the rows grouped by expert
// (crates/stark-engine/src/encodable_block/decoder.rs:182-186, mlp/routed.rs:144-256).
//
// A token reads every active weight for one row; a pass reads a weight record once for 16 rows.  The contractions keep the
// token's arithmetic: codes as exact f16 integers on the M side of mma.sync.m16n8k16, an input row as f16 head and remainder
// (~22 bits) in two of the eight N columns -- four rows fill the tile that one row's copies filled -- and the block scales
// applied in f32 to every sub-block's sums.  (tcgen05 accumulates over the whole contraction, so the scales would have to
// go into the weights, which then need a remainder of their own and the input's 22 bits three products instead of two.)
//
// Every sum over a row, a slice of 256 columns, a strand of keys or the spans is formed as a token forms it (moe_math.cuh): a
// row's results are the token's, bit for bit.
//
// 12 layers of the 30B-A3B shape, 160 rows and the token behind them: 4.56 ms against 112 ms token by token.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "context.cuh"
#include "moe_rows.cuh"
#include "moe_select.cuh"

namespace sb {

namespace {

constexpr uint32_t kNt = kMoeRowsChunk / 4u;         // column tiles of four rows
static_assert(kNt == 4u, "run() below has a loop for each");
constexpr uint32_t kLine = 512u + 64u;               // a row's head or remainder of 256 columns: two lines 64 B apart modulo 128 B
constexpr uint32_t kTileLines = kMoeRowsChunk * 2u;  // lines of a stage
template <bool Q4>
constexpr uint32_t kMetaBytes = Q4 ? kRowsMeta * 4u : 16u;  // of a row's slice: the scale; the sums behind it

struct RowsGemmParams {
    const uint8_t *data;
    uint32_t rows, row_tiles, row_blocks;  // of one matrix; row_blocks: its CTAs
    Members at;
    size_t matrix_bytes;
    const __half *x;
    const float *meta, *scale;
    float *out;
    uint32_t out_stride;
    uint32_t m;                            // dense: input rows
    const uint32_t *tiles, *pairs;         // experts: see MoeRowLists
    uint32_t divisor, experts;
};

// The slices in the order in which a token adds them up: member by member.  `ends`: the member's last.
__device__ inline uint32_t slice_at(const Members &at, uint32_t step, bool &ends) {
    const uint32_t full = at.supers - (at.records - 1u) * at.width;  // members with `records` slices, the first ones
    const bool late = step >= full * at.records;
    const uint32_t each = at.records - (late ? 1u : 0u), k = late ? step - full * at.records : step;
    ends = k % each + 1u == each;
    return (late ? full : 0u) + k / each + k % each * at.width;
}

// One CTA: 16 matrix rows a warp times up to 16 input rows, the contraction in steps of 256 columns, copies of the
// next steps in flight.  Bound by the latency of the tensor-core loop at full tiles, 16 warps an SM at 128 registers, and by the
// weights' bytes where experts have few rows.  160 rows, 8 of 128 experts: gate and up 151 us, down 82.
// MULTI: members of several slices.
template <bool Q4, int STAGES, uint32_t WARPS, bool MULTI>
__global__ void __launch_bounds__(WARPS * 32, WARPS == 8u && !MULTI ? 2 : 1) rows_gemm_kernel(const RowsGemmParams p) {
    constexpr uint32_t kSuper = Q4 ? kQ4SuperBytes : kB8SuperBytes, kMeta = kMetaBytes<Q4>;
    constexpr uint32_t kStage = WARPS * kSuper + kTileLines * kLine + kMoeRowsChunk * kMeta;
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
    const uint32_t row_tile = block * WARPS + warp, supers = p.at.supers;
    const bool live = row_tile < p.row_tiles;
    const uint8_t *weights = p.data + (size_t)matrix * p.matrix_bytes + (size_t)row_tile * supers * kSuper;
    const size_t columns = (size_t)supers * kSlice;
    const uint32_t live_nt = (count + 3u) / 4u;

    const auto issue = [&](uint32_t step) {
        if (step < supers) {
            bool ends;
            const uint32_t s = MULTI ? slice_at(p.at, step, ends) : step;
            uint8_t *stage = rows_smem + (step % STAGES) * kStage;
            if (live)
                for (uint32_t off = lane * 16u; off < kSuper; off += 512u)
                    cp_async16(stage + warp * kSuper + off, weights + (size_t)s * kSuper + off);
            uint8_t *lines = stage + WARPS * kSuper;
            for (uint32_t i = tid; i < count * 64u; i += WARPS * 32u) {
                const uint32_t line = i >> 5, c = i & 31u;
                cp_async16(lines + line * kLine + c * 16u,
                           p.x + ((size_t)(ids[line >> 1] / p.divisor) * 2u + (line & 1u)) * columns + s * kSlice + c * 8u);
            }
            constexpr uint32_t kChunks = kMeta / 16u;
            for (uint32_t i = tid; i < count * kChunks; i += WARPS * 32u)
                cp_async16(lines + kTileLines * kLine + i * 16u,
                           p.meta + ((size_t)(ids[i / kChunks] / p.divisor) * supers + s) * kRowsMeta + i % kChunks * 4u);
        }
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) issue(s);

    float acc0[kNt], acc1[kNt], part0[kNt], part1[kNt];  // matrix rows g and g + 8, input row t of every column tile; of a member
#pragma unroll
    for (uint32_t n = 0; n < kNt; ++n) acc0[n] = acc1[n] = part0[n] = part1[n] = 0.0f;
    // The loop for a number of column tiles known to the compiler: their products are independent chains, which a test in
    // between kept apart (a warp waited 2.6 cycles an instruction for the one before it).
    const auto run = [&](auto tiles) {
        constexpr uint32_t NT = decltype(tiles)::value;
        for (uint32_t step = 0; step < supers; ++step) {
            cp_async_wait<STAGES - 2>();
            __syncthreads();  // every thread's copies of this step are there, and everybody is done with the step before
            issue(step + STAGES - 1);
            if (!live) continue;
            const uint8_t *stage = rows_smem + (step % STAGES) * kStage, *rec = stage + warp * kSuper;
            const uint8_t *lines = stage + WARPS * kSuper + g * kLine + t * 16u;
            const uint8_t *meta = stage + WARPS * kSuper + kTileLines * kLine + t * kMeta;  // of input row t; 4 kMeta to the next tile's
            float dsc0[2], dm0[2], dsc1[2], dm1[2];
            if (Q4) {
                q4k_scales_pair(*reinterpret_cast<const uint4 *>(rec + 2048u + 16u * g), t, dsc0, dm0);
                q4k_scales_pair(*reinterpret_cast<const uint4 *>(rec + 2048u + 16u * (g + 8u)), t, dsc1, dm1);
            }
            // What sub-blocks q and q + 4 add: the share of lane q of a token's row.
            const auto shares = [&](uint32_t q, float(&r0)[NT], float(&r1)[NT]) {
#pragma unroll
                for (int h = 1; h >= 0; --h) {
                    const uint32_t jb = q + 4u * h;
                    uint32_t a[8];
                    if (Q4) {
                        const uint2 w = *reinterpret_cast<const uint2 *>(rec + jb * 256u + lane * 8u);
                        dequant_a4_word<0>(w.x, *reinterpret_cast<uint32_t(*)[4]>(&a[0]));
                        dequant_a4_word<0>(w.y, *reinterpret_cast<uint32_t(*)[4]>(&a[4]));
                    } else {
                        const uint4 w = *reinterpret_cast<const uint4 *>(rec + jb * 512u + lane * 16u);
                        bytes_to_f16<false>(w.x, a[0], a[1]);
                        bytes_to_f16<false>(w.y, a[2], a[3]);
                        bytes_to_f16<false>(w.z, a[4], a[5]);
                        bytes_to_f16<false>(w.w, a[6], a[7]);
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
                    float s0, s1, m0 = 0.0f, m1 = 0.0f, n0 = 0.0f, n1 = 0.0f;
                    if (Q4) {  // lane q of the four that share these rows decoded these sub-blocks' scales
                        const uint32_t from = (lane & ~3u) | q;
                        s0 = __shfl_sync(0xffffffffu, dsc0[h], from), s1 = __shfl_sync(0xffffffffu, dsc1[h], from);
                        if (h == 1) {
                            m0 = __shfl_sync(0xffffffffu, dm0[0], from), m1 = __shfl_sync(0xffffffffu, dm1[0], from);
                            n0 = __shfl_sync(0xffffffffu, dm0[1], from), n1 = __shfl_sync(0xffffffffu, dm1[1], from);
                        }
                    } else {
                        const uint16_t *scales = reinterpret_cast<const uint16_t *>(rec + 4096u) + jb * 16u + g;
                        s0 = f16_bits_f32(scales[0]), s1 = f16_bits_f32(scales[8]);
                    }
#pragma unroll
                    for (uint32_t n = 0; n < NT; ++n) {
                        const float p0 = c[n][0] + c[n][1], p1 = c[n][2] + c[n][3];
                        if (h == 0) {
                            r0[n] = share_first(s0, p0, r0[n]), r1[n] = share_first(s1, p1, r1[n]);
                        } else if (Q4) {
                            const float *sums = reinterpret_cast<const float *>(meta + 4u * n * kMeta) + 4u + q;
                            r0[n] = q4k_share_second(s0, p0, m0, sums[0], n0, sums[4]);
                            r1[n] = q4k_share_second(s1, p1, m1, sums[0], n1, sums[4]);
                        } else {
                            r0[n] = q8_share_second(s0, p0), r1[n] = q8_share_second(s1, p1);
                        }
                    }
                }
            };
            float sum0[NT] = {}, sum1[NT] = {};
#pragma unroll 1  // two shares at a time: four in one stretch spill
            for (uint32_t q = 0; q < 4u; q += 2u) {
                float a0[NT], a1[NT], b0[NT], b1[NT];
                shares(q, a0, a1);
                shares(q + 1u, b0, b1);
#pragma unroll
                for (uint32_t n = 0; n < NT; ++n) sum0[n] += a0[n] + b0[n], sum1[n] += a1[n] + b1[n];
            }
            bool ends = true;
            if (MULTI) slice_at(p.at, step, ends);
#pragma unroll
            for (uint32_t n = 0; n < NT; ++n) {
                const float down = *reinterpret_cast<const float *>(meta + 4u * n * kMeta);
                if (MULTI) {
                    part0[n] = fmaf(down, sum0[n], part0[n]), part1[n] = fmaf(down, sum1[n], part1[n]);
                    if (ends) acc0[n] += part0[n], acc1[n] += part1[n], part0[n] = part1[n] = 0.0f;
                } else {
                    acc0[n] = __fadd_rn(acc0[n], __fmul_rn(down, sum0[n])), acc1[n] = __fadd_rn(acc1[n], __fmul_rn(down, sum1[n]));
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
        const float scale = p.scale ? p.scale[id / p.divisor] : 1.0f;
        float *y = p.out + (size_t)id * p.out_stride + column;
        if (r0 < p.rows) y[r0] = __fmul_rn(acc0[n], scale);
        if (r1 < p.rows) y[r1] = __fmul_rn(acc1[n], scale);
    }
}

// A slice of an operand row, by one warp.
__device__ inline void store_slice(const RowsOperand &out, uint32_t at, uint32_t s, const float (&v)[8]) {
    const uint32_t lane = threadIdx.x & 31u;
    const SplitSlice split = split_slice(v);
    __half *head = out.split + (size_t)at * 2u * out.columns + s * kSlice + lane * 8u;
    *reinterpret_cast<uint4 *>(head) = split.head;
    *reinterpret_cast<uint4 *>(head + out.columns) = split.rest;
    float *meta = out.meta + ((size_t)at * (out.columns / kSlice) + s) * kRowsMeta;
    if ((lane & 3u) == 0) meta[4u + lane / 4u] = split.sum;
    if (lane == 0) meta[0] = split.down;
}

// rms_norm(row, w) as an operand, a warp a member of the row: `value` gives a lane's eight columns of a slice.
template <typename Value>
__device__ inline void norm_operand(const RowsOperand &out, uint32_t at, const Members &members, const float *w, float eps, Value value) {
    __shared__ float squares[kMaxMembers];
    const uint32_t lane = threadIdx.x & 31u, member = threadIdx.x >> 5;
    float square = 0.0f;
    for (uint32_t s = member; s < members.supers; s += members.width) {
        float v[8], g[8];
        load8(w + s * kSlice + lane * 8u, g);
        value(s, v);
        weigh8(v, g, square);
        store_slice(out, at, s, v);
    }
    square = warp_sum(square);
    if (lane == 0) squares[member] = square;
    __syncthreads();
    if (threadIdx.x) return;
    float total = 0.0f;
    for (uint32_t m = 0; m < members.width; ++m) total += squares[m];
    out.scale[at] = norm_scale(total, out.columns, eps);
}

__device__ inline void store8(float *dst, const float (&v)[8]) {
    reinterpret_cast<float4 *>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
    reinterpret_cast<float4 *>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
}

__global__ void __launch_bounds__(kMaxMembers * 32) moe_rows_embed_kernel(const uint32_t *tokens, const uint8_t *table, float *x,
                                                                          const float *w, float eps, const RowsOperand out,
                                                                          const Members members) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t H = out.columns, at = blockIdx.x, lane = threadIdx.x & 31u;
    const uint8_t *src = table + (size_t)tokens[at] * (H / 32u) * 34u;
    norm_operand(out, at, members, w, eps, [&](uint32_t s, float(&v)[8]) {
        const uint32_t column = s * kSlice + lane * 8u;
        const uint8_t *b = src + (column >> 5) * 34u;
        const float d = __half2float(__ushort_as_half((unsigned short)(b[0] | (b[1] << 8))));
#pragma unroll
        for (uint32_t i = 0; i < 8u; ++i) v[i] = d * (float)(int8_t)b[2u + (column & 31u) + i];
        store8(x + (size_t)at * H + column, v);
    });
}

// Per-head norm and rope of the rows' heads and the cache rows: a warp a head, as a token's attention prepares them.
constexpr uint32_t kHeadWarps = 4;
__global__ void __launch_bounds__(kHeadWarps * 32) moe_rows_heads_kernel(float *qkv, const float *q_norm, const float *k_norm,
                                                                         float *keys, float *values, uint32_t q_heads,
                                                                         uint32_t kv_heads, float eps, float theta, uint32_t first_pos) {
    const uint32_t lane = threadIdx.x & 31u, heads = q_heads + 2u * kv_heads, position = first_pos + blockIdx.y;
    const uint32_t h = blockIdx.x * kHeadWarps + (threadIdx.x >> 5);
    pdl_launch_dependents();
    float norm[4], cs[2], sn[2], v[4], o[4];
    if (h < q_heads + kv_heads) {
#pragma unroll
        for (int k = 0; k < 4; ++k) norm[k] = (h < q_heads ? q_norm : k_norm)[32 * k + lane];
        head_angles(position, theta, lane, cs, sn);
    }
    pdl_wait();
    if (h >= heads) return;
    float *src = qkv + ((size_t)blockIdx.y * heads + h) * kHeadWidth, *dst = src;
    const size_t cache_row = (size_t)position * kv_heads * kHeadWidth;
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = v[k] = src[32 * k + lane];
    if (h < q_heads + kv_heads) prepare_head(v, norm, cs, sn, eps, o);
    if (h >= q_heads + kv_heads) dst = values + cache_row + (size_t)(h - q_heads - kv_heads) * kHeadWidth;
    else if (h >= q_heads) dst = keys + cache_row + (size_t)(h - q_heads) * kHeadWidth;
#pragma unroll
    for (int k = 0; k < 4; ++k) dst[32 * k + lane] = o[k];
}

// G values a lane, each summed over the warp as warp_sum does it: the same pairs in the same order, but a lane goes on with half
// of the values at a time.  Returns value lane / (32 / G).
template <int G>
__device__ inline float group_sums(float (&d)[G], uint32_t lane) {
    int left = G;
#pragma unroll
    for (uint32_t o = 16u; o > 0; o >>= 1) {
        if (left > 1) {
            left /= 2;
#pragma unroll
            for (int i = 0; i < G / 2; ++i)
                if (i < left) {
                    const float got = __shfl_xor_sync(0xffffffffu, lane & o ? d[i] : d[i + left], o);
                    d[i] = (lane & o ? d[i + left] : d[i]) + got;
                }
        } else {
            d[0] += __shfl_xor_sync(0xffffffffu, d[0], o);
        }
    }
    return d[0];
}

// State of a span of a head: its maximum and sum, two unused words, its 128 columns.
constexpr uint32_t kSpanState = kHeadWidth + 4u;

// Attention of a row, `each` spans of a KV head a CTA: as in a token a warp is a strand, which reads a key once for the G query
// heads of the group; 32 / G lanes keep the maximum and sum of a head.  Two keys of a strand go side by side up to their
// scores, and the next two are fetched meanwhile.  A span's strands merge through one of two buffers, so that a barrier a span
// is enough.  Bound by instruction issue and that barrier: 160 rows of 32 heads behind 500 take 201 us, 209 with one key at a time
// and one buffer, 238 with a warp a query head, 350 with every lane computing every weight.
template <int G>
struct SpanBuffer {
    float m[kStrands][G], l[kStrands][G];
    float4 acc[kStrands][G][32];
};
template <int G>
__global__ void __launch_bounds__(kStrands * 32, 2) moe_rows_attention_kernel(const float *qkv, const float *keys, const float *values,
                                                                              float *part, uint32_t first_pos, uint32_t splits,
                                                                              uint32_t each, uint32_t spans, uint32_t kv_heads, float scale) {
    constexpr uint32_t kLanes = 32u / G;
    extern __shared__ __align__(16) uint8_t span_smem[];
    const uint32_t kvh = blockIdx.x, row = blockIdx.z, warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t rows = first_pos + row + 1u, span = span_rows(rows, splits), used = (rows + span - 1u) / span;
    const uint32_t from = blockIdx.y * each, to = min(used, from + each);
    pdl_launch_dependents();
    pdl_wait();
    if (from >= to) return;
    const size_t kv_row = (size_t)kv_heads * kHeadWidth;
    const auto fetch = [&](const float *cache, uint32_t t) {
        return reinterpret_cast<const float4 *>(cache + min(t, rows - 1u) * kv_row + kvh * kHeadWidth)[lane];
    };
    float4 q[G];
#pragma unroll
    for (int g = 0; g < G; ++g)
        q[g] = reinterpret_cast<const float4 *>(qkv + ((size_t)row * kv_heads * (G + 2u) + kvh * G + g) * kHeadWidth)[lane];
    float4 k[2], v[2];
#pragma unroll
    for (uint32_t j = 0; j < 2u; ++j) {
        const uint32_t t = from * span + warp + j * kStrands;
        k[j] = fetch(keys, t), v[j] = fetch(values, t);
    }
    for (uint32_t n = from; n < to; ++n) {
        SpanBuffer<G> &buffer = reinterpret_cast<SpanBuffer<G> *>(span_smem)[n & 1u];
        const uint32_t lo = n * span, hi = min(rows, lo + span);
        float m = -INFINITY, l = 0.0f;
        float4 acc[G];
#pragma unroll
        for (int g = 0; g < G; ++g) acc[g] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (uint32_t t = lo + warp; t < hi; t += 2u * kStrands) {
            float score[2];
            float4 value[2];
            const uint32_t next = t + 2u * kStrands < hi ? t + 2u * kStrands : hi + warp;  // of this span, or the first of the next
#pragma unroll
            for (uint32_t j = 0; j < 2u; ++j) {
                float dot[G];
#pragma unroll
                for (int g = 0; g < G; ++g) dot[g] = dot4(q[g], k[j]);
                value[j] = v[j];
                k[j] = fetch(keys, next + j * kStrands), v[j] = fetch(values, next + j * kStrands);
                score[j] = __fmul_rn(group_sums<G>(dot, lane), scale);
            }
#pragma unroll
            for (uint32_t j = 0; j < 2u; ++j) {
                if (t + j * kStrands >= hi) break;
                float c, e;
                strand_step(m, l, score[j], c, e);
#pragma unroll
                for (int g = 0; g < G; ++g)
                    strand_add(acc[g], __shfl_sync(0xffffffffu, c, g * kLanes), __shfl_sync(0xffffffffu, e, g * kLanes), value[j]);
            }
        }
        if (lane % kLanes == 0) buffer.m[warp][lane / kLanes] = m, buffer.l[warp][lane / kLanes] = l;
#pragma unroll
        for (int g = 0; g < G; ++g) buffer.acc[warp][g][lane] = acc[g];
        __syncthreads();  // the span two before this one was merged ahead of the barrier between them
        if (warp >= (uint32_t)G) continue;
        float top = -INFINITY, sum = 0.0f;
#pragma unroll
        for (uint32_t w = 0; w < kStrands; ++w) top = fmaxf(top, buffer.m[w][warp]);
        float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
        for (uint32_t w = 0; w < kStrands; ++w) strand_take(sum, a, strand_weight(buffer.m[w][warp], top), buffer.l[w][warp], buffer.acc[w][warp][lane]);
        float *dst = part + (((size_t)row * kv_heads * G + kvh * G + warp) * spans + n) * kSpanState;
        if (lane == 0) *reinterpret_cast<float2 *>(dst) = make_float2(top, sum);
        reinterpret_cast<float4 *>(dst)[lane + 1u] = a;
    }
}

// Merges the spans of a row's heads: a slice is two heads, half a warp each.
constexpr uint32_t kMergeWarps = 4;
__global__ void __launch_bounds__(kMergeWarps * 32) moe_rows_merge_kernel(const float *part, uint32_t first_pos, uint32_t splits,
                                                                          uint32_t spans, uint32_t first_row, const RowsOperand out) {
    const uint32_t lane = threadIdx.x & 31u, row = blockIdx.x, heads = out.columns / kHeadWidth;
    const uint32_t s = blockIdx.y * kMergeWarps + (threadIdx.x >> 5);
    const uint32_t rows = first_pos + row + 1u, span = span_rows(rows, splits), used = (rows + span - 1u) / span;
    pdl_launch_dependents();
    pdl_wait();
    if (2u * s >= heads) return;
    const float *src = part + ((size_t)row * heads + 2u * s) * spans * kSpanState;
    float c[2][2], total[2];
#pragma unroll
    for (uint32_t h = 0; h < 2u; ++h) {
        float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.0f, 0.0f};
#pragma unroll
        for (uint32_t j = 0; j < 2u; ++j)
            if (lane + 32u * j < used) {
                const float2 state = *reinterpret_cast<const float2 *>(src + ((size_t)h * spans + lane + 32u * j) * kSpanState);
                m[j] = state.x, l[j] = state.y;
            }
        total[h] = span_weights(m, l, c[h]);
    }
    const bool second = lane >= 16u;
    src += (second ? spans * kSpanState : 0u) + 4u + (lane & 15u) * 8u;
    float v[8] = {};
#pragma unroll 8
    for (uint32_t n = 0; n < used; ++n) {
        const float first_weight = __shfl_sync(0xffffffffu, n < 32u ? c[0][0] : c[0][1], n & 31u);
        const float second_weight = __shfl_sync(0xffffffffu, n < 32u ? c[1][0] : c[1][1], n & 31u);
        const float weight = second ? second_weight : first_weight;
        float a[8];
        load8(src + n * kSpanState, a);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = fmaf(a[i], weight, v[i]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = v[i] / (second ? total[1] : total[0]);
    store_slice(out, first_row + row, s, v);
}

__global__ void __launch_bounds__(kMaxMembers * 32) moe_rows_add_norm_kernel(float *x, const float *update, const float *probs,
                                                                             uint32_t active, const float *w, float eps,
                                                                             const RowsOperand out, const Members members) {
    __shared__ float share[32];
    const uint32_t at = blockIdx.x, lane = threadIdx.x & 31u, hidden = out.columns;
    pdl_launch_dependents();
    pdl_wait();
    if (probs) {
        for (uint32_t e = threadIdx.x; e < active; e += blockDim.x) share[e] = probs[(size_t)at * active + e];
        __syncthreads();
    }
    const float *rows = update + (size_t)at * (probs ? active : 1u) * hidden;
    norm_operand(out, at, members, w, eps, [&](uint32_t s, float(&v)[8]) {
        const uint32_t column = s * kSlice + lane * 8u;
        float *home = x + (size_t)at * hidden + column, r[8], o[8];
        load8(home, v);
        if (probs) {
#pragma unroll
            for (int i = 0; i < 8; ++i) r[i] = 0.0f;
#pragma unroll 8
            for (uint32_t e = 0; e < active; ++e) {
                load8(rows + (size_t)e * hidden + column, o);
#pragma unroll
                for (int i = 0; i < 8; ++i) r[i] = fmaf(share[e], o[i], r[i]);
            }
        } else {
            load8(rows + column, r);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] += r[i];
        store8(home, v);
    });
}

// Router scores of 16 rows and four experts a CTA, a warp a member of the rows: it holds its slice of the four experts' rows
// times the norm's weights, so an input row is read once for four scores.  (All experts of four rows in one CTA took 40 us: the
// 1 MB of router rows went by one after another.)
constexpr uint32_t kRouteRows = 16, kRouteExperts = 4;
__global__ void __launch_bounds__(kMaxMembers * 32) moe_rows_scores_kernel(const float *router, const float *x, const float *norm,
                                                                           const float *scale, uint32_t experts, float *scores,
                                                                           uint32_t rows, const Members at) {
    __shared__ float part[kRouteRows][kRouteExperts][kMaxMembers];
    const uint32_t lane = threadIdx.x & 31u, member = threadIdx.x >> 5, expert0 = blockIdx.x * kRouteExperts, row0 = blockIdx.y * kRouteRows;
    const uint32_t hidden = at.supers * kSlice, count = min(kRouteRows, rows - row0);
    float a[kRouteExperts][8];
    const auto products = [&](uint32_t s) {
        float w[8];
        load8(norm + s * kSlice + lane * 8u, w);
#pragma unroll
        for (uint32_t e = 0; e < kRouteExperts; ++e) {
            load8(router + (size_t)min(expert0 + e, experts - 1u) * hidden + s * kSlice + lane * 8u, a[e]);
#pragma unroll
            for (int i = 0; i < 8; ++i) a[e][i] = __fmul_rn(a[e][i], w[i]);
        }
    };
    pdl_launch_dependents();
    products(member);
    pdl_wait();
#pragma unroll 2
    for (uint32_t row = 0; row < count; ++row) {
        float dot[kRouteExperts] = {};
        for (uint32_t s = member; s < at.supers; s += at.width) {
            float v[8];
            if (at.records > 1u) products(s);
            load8(x + (size_t)(row0 + row) * hidden + s * kSlice + lane * 8u, v);
#pragma unroll
            for (uint32_t e = 0; e < kRouteExperts; ++e)
#pragma unroll
                for (int i = 0; i < 8; ++i) dot[e] = fmaf(a[e][i], v[i], dot[e]);
        }
#pragma unroll
        for (uint32_t e = 0; e < kRouteExperts; ++e) dot[e] = warp_sum(dot[e]);
        if (lane == 0)
#pragma unroll
            for (uint32_t e = 0; e < kRouteExperts; ++e) part[row][e][member] = dot[e];
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < count * kRouteExperts; i += blockDim.x) {
        const uint32_t row = i / kRouteExperts, e = i % kRouteExperts;
        if (expert0 + e >= experts) continue;
        float dot = 0.0f;
        for (uint32_t m = 0; m < at.width; ++m) dot += part[row][e][m];
        scores[(size_t)(row0 + row) * experts + expert0 + e] = __fmul_rn(dot, scale[row0 + row]);
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

// silu(gate) * up of every pair, a warp a slice.
constexpr uint32_t kGateWarps = 8;
__global__ void __launch_bounds__(kGateWarps * 32) moe_rows_gate_kernel(const float *gate_up, const RowsOperand out, uint32_t slices) {
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t lane = threadIdx.x & 31u, i = blockIdx.x * kGateWarps + (threadIdx.x >> 5), each = out.columns / kSlice;
    if (i >= slices) return;
    const float *gates = gate_up + (size_t)(i / each) * 2u * out.columns + i % each * kSlice + lane * 8u;
    float g[8], u[8], v[8];
    load8(gates, g), load8(gates + out.columns, u);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = gated_value(g[j], u[j]);
    store_slice(out, i / each, i % each, v);
}

// Launches that may start before their predecessor ends: every kernel here awaits it before its first access to what it made.
template <typename... Params, typename... Args>
stark_b200_status launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args... args) {
    return moe_launch(kernel, grid, block, smem, true, stream, args...);
}

// CTAs of a pass's attention from which on each takes more than one span.
constexpr uint32_t kAttentionCtas = 1184;

constexpr size_t gemm_smem(uint32_t stages, uint32_t warps, bool q4) {
    return stages * (warps * (q4 ? kQ4SuperBytes : kB8SuperBytes) + kTileLines * kLine + kMoeRowsChunk * (q4 ? kMetaBytes<true> : kMetaBytes<false>));
}
constexpr uint32_t kQ4Stages = 3, kQ4Warps = 8;
constexpr size_t kQ4Smem = gemm_smem(kQ4Stages, kQ4Warps, true);

RowsGemmParams gemm_params(const QMatrix *w, uint32_t super_bytes, uint32_t warps, const RowsOperand &x, float *out) {
    RowsGemmParams p{};
    p.data = w->data;
    p.rows = w->rows;
    p.row_tiles = w->row_tiles;
    p.at = members_of(w->columns);
    p.row_blocks = (w->row_tiles + warps - 1u) / warps;
    p.matrix_bytes = (size_t)w->row_tiles * p.at.supers * super_bytes;
    p.x = x.split;
    p.meta = x.meta;
    p.scale = x.scale;
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
    const size_t smem = gemm_smem(narrow ? 4u : 2u, warps, false);
    RowsGemmParams p = gemm_params(w, kB8SuperBytes, warps, x, out);
    const bool multi = p.at.records > 1u;
    const auto kernel = narrow ? (multi ? rows_gemm_kernel<false, 4, 2, true> : rows_gemm_kernel<false, 4, 2, false>)
                               : (multi ? rows_gemm_kernel<false, 2, 8, true> : rows_gemm_kernel<false, 2, 8, false>);
    static SmemOptIn once[2][2];
    if (stark_b200_status s = ensure_dynamic_smem(kernel, (int)smem, once[narrow][multi])) return s;
    p.m = rows;
    p.out_stride = w->rows;
    return launch(kernel, dim3(p.row_blocks, chunks), warps * 32u, smem, stream, p);
}

stark_b200_status rows_q4k_experts_launch(const QMatrix *w, uint32_t blocks, const RowsOperand &x, uint32_t divisor, float *out,
                                          const MoeRowLists &lists, uint32_t rows, uint32_t active, cudaStream_t stream) {
    if (w->format != kFmtQ4_K || w->columns != x.columns || rows == 0 || w->experts % blocks) return STARK_B200_INVALID_ARGUMENT;
    RowsGemmParams p = gemm_params(w, kQ4SuperBytes, kQ4Warps, x, out);
    const bool multi = p.at.records > 1u;
    const auto kernel = multi ? rows_gemm_kernel<true, kQ4Stages, kQ4Warps, true> : rows_gemm_kernel<true, kQ4Stages, kQ4Warps, false>;
    static SmemOptIn once[2];
    if (stark_b200_status s = ensure_dynamic_smem(kernel, (int)kQ4Smem, once[multi])) return s;
    p.experts = w->experts / blocks;
    p.tiles = lists.tiles;
    p.pairs = lists.pairs;
    p.divisor = divisor;
    p.out_stride = blocks * w->rows;
    return launch(kernel, dim3(p.row_blocks * blocks, MoeRowLists::max_tiles(rows, active, p.experts)),
                  kQ4Warps * 32u, kQ4Smem, stream, p);
}

stark_b200_status moe_rows_embed_launch(const uint32_t *tokens, const uint8_t *table, float *x, const float *w, float eps,
                                        const RowsOperand &out, uint32_t rows, cudaStream_t stream) {
    const Members at = members_of(out.columns);
    return launch(moe_rows_embed_kernel, rows, at.width * 32u, 0, stream, tokens, table, x, w, eps, out, at);
}

stark_b200_status moe_rows_heads_launch(float *qkv, const float *q_norm, const float *k_norm, float *keys, float *values,
                                        uint32_t q_heads, uint32_t kv_heads, float eps, float theta, uint32_t first_pos,
                                        uint32_t rows, cudaStream_t stream) {
    return launch(moe_rows_heads_kernel, dim3((q_heads + 2u * kv_heads + kHeadWarps - 1u) / kHeadWarps, rows), kHeadWarps * 32u, 0, stream,
                  qkv, q_norm, k_norm, keys, values, q_heads, kv_heads, eps, theta, first_pos);
}

stark_b200_status moe_rows_attention_launch(const float *qkv, const float *keys, const float *values, float *part, size_t part_floats,
                                            uint32_t q_heads, uint32_t kv_heads, uint32_t splits, uint32_t first_pos,
                                            const RowsOperand &out, uint32_t rows, cudaStream_t stream) {
    const uint32_t group = q_heads / kv_heads, spans = moe_rows_spans(splits, first_pos + rows);
    const size_t row_floats = moe_rows_part(q_heads, spans);
    if (out.columns != q_heads * kHeadWidth || splits > 64u || part_floats < row_floats) return STARK_B200_INVALID_ARGUMENT;
    const auto kernel = group == 8u ? moe_rows_attention_kernel<8> : (group == 4u ? moe_rows_attention_kernel<4> : moe_rows_attention_kernel<2>);
    const size_t smem = 2u * (group == 8u ? sizeof(SpanBuffer<8>) : (group == 4u ? sizeof(SpanBuffer<4>) : sizeof(SpanBuffer<2>)));
    static SmemOptIn once[3];
    if (stark_b200_status s = ensure_dynamic_smem(kernel, (int)smem, once[group / 4u])) return s;
    const uint32_t batch = (uint32_t)std::min<size_t>(rows, part_floats / row_floats);
    for (uint32_t done = 0; done < rows; done += batch) {
        const uint32_t now = std::min(batch, rows - done), pos = first_pos + done;
        const uint32_t each = std::max(1u, std::min(spans, kv_heads * spans * now / kAttentionCtas));
        if (stark_b200_status s = launch(kernel, dim3(kv_heads, (spans + each - 1u) / each, now), kStrands * 32u, smem, stream,
                                         qkv + (size_t)done * (q_heads + 2u * kv_heads) * kHeadWidth, keys, values, part, pos, splits, each,
                                         spans, kv_heads, 1.0f / sqrtf((float)kHeadWidth)))
            return s;
        if (stark_b200_status s = launch(moe_rows_merge_kernel, dim3(now, (q_heads / 2u + kMergeWarps - 1u) / kMergeWarps), kMergeWarps * 32u, 0, stream,
                                         part, pos, splits, spans, done, out))
            return s;
    }
    return STARK_B200_OK;
}

stark_b200_status moe_rows_add_norm_launch(float *x, const float *update, const float *probs, uint32_t active, const float *w,
                                           float eps, const RowsOperand &out, uint32_t rows, cudaStream_t stream) {
    const Members at = members_of(out.columns);
    return launch(moe_rows_add_norm_kernel, rows, at.width * 32u, 0, stream, x, update, probs, active, w, eps, out, at);
}

stark_b200_status moe_rows_route_launch(const float *router, const float *x, const float *norm, const RowsOperand &normed,
                                        uint32_t experts, uint32_t active, const MoeRowLists &lists, uint32_t *last_ids,
                                        uint32_t rows, cudaStream_t stream) {
    const Members at = members_of(normed.columns);
    if (stark_b200_status s = launch(moe_rows_scores_kernel, dim3((experts + kRouteExperts - 1u) / kRouteExperts, (rows + kRouteRows - 1u) / kRouteRows),
                                     at.width * 32u, 0, stream, router, x, norm, normed.scale, experts, lists.scores, rows, at))
        return s;
    return launch(experts <= 128u ? moe_rows_select_kernel<4> : moe_rows_select_kernel<32>, (rows + kSelectWarps - 1u) / kSelectWarps,
                  kSelectWarps * 32u, 0, stream, lists.scores, experts, active, lists.ids, lists.probs, last_ids, rows);
}

stark_b200_status moe_rows_lists_launch(const MoeRowLists &lists, uint32_t rows, uint32_t active, uint32_t experts,
                                        cudaStream_t stream) {
    return launch(moe_rows_lists_kernel, 1, kListThreads, 0, stream, lists.ids, lists.pairs, lists.tiles, rows * active, experts);
}

stark_b200_status moe_rows_gate_launch(const float *gate_up, const RowsOperand &out, uint32_t pairs, cudaStream_t stream) {
    const uint32_t slices = pairs * (out.columns / kSlice);
    return launch(moe_rows_gate_kernel, (slices + kGateWarps - 1u) / kGateWarps, kGateWarps * 32u, 0, stream, gate_up, out, slices);
}

size_t moe_rows_part(uint32_t q_heads, uint32_t spans) { return (size_t)q_heads * spans * kSpanState; }

}  // namespace sb
