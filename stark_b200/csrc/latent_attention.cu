// Latent attention in its absorbed form: the cache holds one row per position -- the normed latent c and a rotated key
// part all heads share -- and the per-head key and value matrices are applied on the query's and the output's side:
//   score_j = ((W_uk^T q) . c_j + q_rot . r_j) * scale,     out = W_uv (sum_j a_j c_j)
// so a decode step reads rank + rot values per cached row whatever the number of heads.  Three launches:
//   latent_query    per head and 64 latent columns: W_uk^T q, the rotated query part, both times scale * log2(e); one
//                   more CTA per row norms the new latent, rotates the new key part and appends the cache row
//   latent_attend   per span of the cached rows and group of heads: f32 scores, running softmax, weighted latents
//   latent_value    per head and 32 output values: merge of the spans, then W_uv
// Angles, norms, scores and softmax are f32.  A row of a pass attends to the rows up to its own position.
#include "layered.cuh"
#include "layered_math.cuh"

namespace sb {

namespace {

constexpr uint32_t kQueryThreads = 256;
__device__ inline float *partial_of(const LatentArgs &a, uint32_t row, uint32_t head, uint32_t split) {
    return a.partials + (((size_t)row * a.s.heads + head) * a.splits + split) * (a.s.rank_p + 4u);
}

// The new cache row of one position: latent / rms * w, and the key part rotated.  One CTA.
template <typename T, typename C>
__device__ void append_row(const LatentArgs &a, const T *src, uint32_t pos, float *scratch) {
    const LatentShape &s = a.s;
    C *dst = reinterpret_cast<C *>(a.cache) +
             ((size_t)a.block_table[pos / kPageTokens] * kPageTokens + pos % kPageTokens) * s.row();
    float sum = 0.0f;
    for (uint32_t i = threadIdx.x; i < s.rank; i += blockDim.x) {
        const float v = load_value(src + i);
        sum += v * v;
    }
    const float inv = inverse_rms(block_sum(sum, scratch), s.rank, a.eps);
    for (uint32_t i = threadIdx.x; i < s.rank_p; i += blockDim.x)
        store_value(dst + i, i < s.rank ? load_value(src + i) * inv * a.latent_norm[i] : 0.0f);
    for (uint32_t i = threadIdx.x; i < s.rot_p / 2u; i += blockDim.x) {
        float u = load_value(src + s.rank_p + 2u * i), v = load_value(src + s.rank_p + 2u * i + 1u);
        if (i < a.rot.pairs) {
            float sn, cs;
            sincosf((float)pos * a.rot.freq[i], &sn, &cs);
            sn *= a.rot.factor, cs *= a.rot.factor;
            const float u0 = u;
            u = u0 * cs - v * sn;
            v = v * cs + u0 * sn;
        }
        store_value(dst + s.rank_p + 2u * i, u);
        store_value(dst + s.rank_p + 2u * i + 1u, v);
    }
}

// blockIdx.x: (head, 64 latent columns), then one CTA that appends the cache row; blockIdx.y: row
template <typename T, typename C>
__global__ void __launch_bounds__(kQueryThreads) latent_query_kernel(const LatentArgs a) {
    extern __shared__ float q[];                 // [dim_p]
    __shared__ float part[32][64];
    __shared__ float scratch[32];
    const LatentShape &s = a.s;
    const uint32_t blocks = s.rank_p / 64u, head = blockIdx.x / blocks, piece = blockIdx.x % blocks;
    const uint32_t row = blockIdx.y, lane8 = threadIdx.x & 7u, slice = threadIdx.x >> 3;
    // this thread's first weights do not depend on the previous kernel
    const uint16_t *uk = a.uk_uv.data + (size_t)head * s.dim_p * s.rank_p + piece * 64u + lane8 * 8u;
    uint4 w[4];
    if (head < s.heads) {
#pragma unroll
        for (uint32_t j = 0; j < 4u; ++j) {
            const uint32_t d = slice + 32u * j;
            w[j] = d < s.dim_p ? ldg_nc_v4(uk + (size_t)d * s.rank_p) : make_uint4(0u, 0u, 0u, 0u);
        }
    }
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t pos = a.state ? a.state->position : a.first_pos + row;
    const T *src = reinterpret_cast<const T *>(a.qd) + (size_t)row * a.ld_qd;
    if (head >= s.heads) {
        append_row<T, C>(a, src + s.q_width(), pos, scratch);
        return;
    }
    const float factor = a.scale * kLog2e;
    float *dst = a.queries + ((size_t)row * s.heads + head) * s.row();
    const T *qh = src + (size_t)head * s.q_head();
    for (uint32_t i = threadIdx.x; i < s.dim_p; i += kQueryThreads) q[i] = load_value(qh + i);
    if (piece == 0u) {
        for (uint32_t i = threadIdx.x; i < s.rot_p / 2u; i += kQueryThreads) {
            float u = load_value(qh + s.dim_p + 2u * i), v = load_value(qh + s.dim_p + 2u * i + 1u);
            if (i < a.rot.pairs) {
                float sn, cs;
                sincosf((float)pos * a.rot.freq[i], &sn, &cs);
                sn *= a.rot.factor, cs *= a.rot.factor;
                const float u0 = u;
                u = u0 * cs - v * sn;
                v = v * cs + u0 * sn;
            }
            dst[s.rank_p + 2u * i] = u * factor;
            dst[s.rank_p + 2u * i + 1u] = v * factor;
        }
    }
    __syncthreads();
    float acc[8] = {};
    for (uint32_t d0 = 0; d0 < s.dim_p; d0 += 128u) {
#pragma unroll
        for (uint32_t j = 0; j < 4u; ++j) {
            const uint32_t d = d0 + slice + 32u * j;
            if (d >= s.dim_p) break;
            const uint4 v = d0 == 0u ? w[j] : ldg_nc_v4(uk + (size_t)d * s.rank_p);
            const uint32_t words[4] = {v.x, v.y, v.z, v.w};
            const float x = q[d];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                acc[2 * e] = fmaf(__uint_as_float(words[e] << 16), x, acc[2 * e]);
                acc[2 * e + 1] = fmaf(__uint_as_float(words[e] & 0xffff0000u), x, acc[2 * e + 1]);
            }
        }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) part[slice][lane8 * 8u + e] = acc[e];
    __syncthreads();
    if (threadIdx.x < 64u) {
        float sum = 0.0f;
#pragma unroll
        for (uint32_t k = 0; k < 32u; ++k) sum += part[k][threadIdx.x];
        dst[piece * 64u + threadIdx.x] = sum * factor;
    }
}

// blockIdx.x: (head, 32 output values), blockIdx.y: row.
// Bound by its chain of trips to memory, so there is one behind the wait: the weights of this warp's rows up to rank 512 come ahead of
// it, and the spans' partials beside their statistics.  64 values a CTA, half of the weights and all partials behind other trips: 17
// tokens of guvulorn-8b behind 4 000 rows 61.1 -> 58.2 ms with this, 32 values and one trip (4.7 us a layer).
constexpr uint32_t kValueRows = 4, kValueTile = 8u * kValueRows, kAhead = 2, kBatch = 8;
template <typename O>
__global__ void __launch_bounds__(256) latent_value_kernel(const LatentArgs a) {
    extern __shared__ __align__(16) float o[];  // [rank_p], then the pieces of the merge
    __shared__ float weight[kMaxSplits];
    const LatentShape &s = a.s;
    const uint32_t blocks = s.vdim_p / kValueTile, head = blockIdx.x / blocks, piece = blockIdx.x % blocks, row = blockIdx.y;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t value0 = piece * kValueTile + warp * kValueRows;
    const uint16_t *uv = a.uk_uv.data + ((size_t)s.heads * s.dim_p + (size_t)head * s.vdim_p + value0) * s.rank_p;
    auto weights = [&](uint32_t j, uint32_t c) { return c < s.rank_p ? ldg_nc_v4(uv + (size_t)j * s.rank_p + c) : make_uint4(0u, 0u, 0u, 0u); };
    uint4 w[kAhead][kValueRows];
#pragma unroll
    for (uint32_t i = 0; i < kAhead; ++i)
#pragma unroll
        for (uint32_t j = 0; j < kValueRows; ++j) w[i][j] = weights(j, i * 256u + lane * 8u);
    pdl_launch_dependents();
    pdl_wait();
    const float *part = partial_of(a, row, head, 0);
    const uint32_t pitch = s.rank_p + 4u;
    // four columns a thread; where the latent is narrow several threads share the spans of the same four
    const uint32_t quads = s.rank_p / 4u, shares = quads >= 256u ? 1u : 256u / quads;
    float4 x[kBatch];
    auto fetch = [&](uint32_t t, uint32_t k0) {
#pragma unroll
        for (uint32_t i = 0; i < kBatch; ++i) {
            const uint32_t k = k0 + i * shares;
            x[i] = t < quads * shares && k < a.splits ? *reinterpret_cast<const float4 *>(part + (size_t)k * pitch + 4u + t % quads * 4u)
                                                      : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    fetch(threadIdx.x, threadIdx.x / quads);
    // every warp forms the spans' weights exp2(m - max) / sum for itself; the first one leaves them for the columns
    {
        float m[2], l[2], top = -INFINITY, sum = 0.0f;
#pragma unroll
        for (uint32_t j = 0; j < 2u; ++j) {
            const uint32_t k = lane + 32u * j;
            const float2 v = k < a.splits ? *reinterpret_cast<const float2 *>(part + (size_t)k * pitch) : make_float2(-INFINITY, 0.0f);
            m[j] = v.x, l[j] = v.y;
            top = fmaxf(top, v.x);
        }
        top = warp_max(top);
#pragma unroll
        for (uint32_t j = 0; j < 2u; ++j) {
            m[j] = exp2f(m[j] - top);  // 0 for an empty span
            sum = fmaf(m[j], l[j], sum);
        }
        const float inv = 1.0f / warp_sum(sum);
        if (warp == 0u) weight[lane] = m[0] * inv, weight[lane + 32u] = m[1] * inv;
    }
    __syncthreads();
    float4 *pieces = reinterpret_cast<float4 *>(o + s.rank_p);  // [shares][quads]
    for (uint32_t t = threadIdx.x; t < quads * shares; t += 256u) {
        const uint32_t share = t / quads;
        if (t != threadIdx.x) fetch(t, share);
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        for (uint32_t k0 = share; k0 < a.splits; k0 += kBatch * shares) {
            if (k0 != share) fetch(t, k0);
#pragma unroll
            for (uint32_t i = 0; i < kBatch; ++i) {
                if (k0 + i * shares >= a.splits) break;
                const float c = weight[k0 + i * shares];
                v.x = fmaf(c, x[i].x, v.x), v.y = fmaf(c, x[i].y, v.y), v.z = fmaf(c, x[i].z, v.z), v.w = fmaf(c, x[i].w, v.w);
            }
        }
        pieces[t] = v;
    }
    __syncthreads();
    for (uint32_t quad = threadIdx.x; quad < quads; quad += 256u) {
        float4 v = pieces[quad];
        for (uint32_t k = 1; k < shares; ++k) {
            const float4 y = pieces[k * quads + quad];
            v.x += y.x, v.y += y.y, v.z += y.z, v.w += y.w;
        }
        reinterpret_cast<float4 *>(o)[quad] = v;
    }
    __syncthreads();
    float acc[kValueRows] = {};
    auto columns = [&](uint32_t c, const uint4 (&now)[kValueRows]) {
        const float4 l = *reinterpret_cast<const float4 *>(o + c), r = *reinterpret_cast<const float4 *>(o + c + 4u);
#pragma unroll
        for (uint32_t j = 0; j < kValueRows; ++j) {
            const uint4 v = now[j];
            acc[j] = fmaf(__uint_as_float(v.x << 16), l.x, acc[j]);
            acc[j] = fmaf(__uint_as_float(v.x & 0xffff0000u), l.y, acc[j]);
            acc[j] = fmaf(__uint_as_float(v.y << 16), l.z, acc[j]);
            acc[j] = fmaf(__uint_as_float(v.y & 0xffff0000u), l.w, acc[j]);
            acc[j] = fmaf(__uint_as_float(v.z << 16), r.x, acc[j]);
            acc[j] = fmaf(__uint_as_float(v.z & 0xffff0000u), r.y, acc[j]);
            acc[j] = fmaf(__uint_as_float(v.w << 16), r.z, acc[j]);
            acc[j] = fmaf(__uint_as_float(v.w & 0xffff0000u), r.w, acc[j]);
        }
    };
#pragma unroll
    for (uint32_t i = 0; i < kAhead; ++i)
        if (i * 256u + lane * 8u < s.rank_p) columns(i * 256u + lane * 8u, w[i]);
    for (uint32_t c = kAhead * 256u + lane * 8u; c < s.rank_p; c += 256u) {
        uint4 now[kValueRows];
#pragma unroll
        for (uint32_t j = 0; j < kValueRows; ++j) now[j] = weights(j, c);
        columns(c, now);
    }
    O *dst = reinterpret_cast<O *>(a.out) + ((size_t)row * s.heads + head) * s.vdim_p + value0;
#pragma unroll
    for (uint32_t j = 0; j < kValueRows; ++j) {
        const float v = warp_sum(acc[j]);
        if (lane == 0) store_value(dst + j, v);
    }
}

// One CTA per row of a pass: the new cache row, and the rotated part of every query head rotated in place (bf16 rows).
__global__ void __launch_bounds__(256) latent_rotate_append_kernel(const LatentArgs a) {
    extern __shared__ float2 turn[];  // [pairs] (cos, sin)
    __shared__ float scratch[32];
    const LatentShape &s = a.s;
    const uint32_t row = blockIdx.x, pos = a.first_pos + row;
    uint16_t *src = const_cast<uint16_t *>(reinterpret_cast<const uint16_t *>(a.qd)) + (size_t)row * a.ld_qd;
    pdl_launch_dependents();
    for (uint32_t i = threadIdx.x; i < a.rot.pairs; i += 256u) {
        float sn, cs;
        sincosf((float)pos * a.rot.freq[i], &sn, &cs);
        turn[i] = make_float2(cs * a.rot.factor, sn * a.rot.factor);
    }
    pdl_wait();
    append_row<uint16_t, uint16_t>(a, src + s.q_width(), pos, scratch);
    __syncthreads();
    for (uint32_t t = threadIdx.x; t < s.heads * a.rot.pairs; t += 256u) {
        const uint32_t head = t / a.rot.pairs, i = t % a.rot.pairs;
        uint32_t *pair = reinterpret_cast<uint32_t *>(src + (size_t)head * s.q_head() + s.dim_p) + i;
        const float u = __uint_as_float(*pair << 16), v = __uint_as_float(*pair & 0xffff0000u);
        *pair = f32x2_to_bf16x2(u * turn[i].x - v * turn[i].y, v * turn[i].x + u * turn[i].y);
    }
}

stark_b200_status check_args(const LatentArgs &a) {
    if (!latent_shape_supported(a.s)) return STARK_B200_UNSUPPORTED;
    if (!a.qd || !a.cache || !a.block_table || !a.uk_uv.data || a.m == 0 || (a.state && a.m != 1u) || !a.rot.freq ||
        a.splits > kMaxSplits || a.splits == 0)
        return STARK_B200_INVALID_ARGUMENT;
    return STARK_B200_OK;
}

}  // namespace

bool latent_shape_supported(const LatentShape &s) {
    return s.heads != 0 && s.dim != 0 && s.rot_dim % 2u == 0 && s.vdim != 0 && s.rank != 0 &&
           span_attend_supports(s.row(), s.rank_p) && s.dim_p <= 4096u;
}

stark_b200_status latent_query_launch(const LatentArgs &a, cudaStream_t stream) {
    if (stark_b200_status st = check_args(a)) return st;
    if (!a.queries) return STARK_B200_INVALID_ARGUMENT;
    const dim3 grid(a.s.heads * (a.s.rank_p / 64u) + 1u, a.m);
    auto kernel = a.qd_b16 ? (a.cache_f32 ? latent_query_kernel<uint16_t, float> : latent_query_kernel<uint16_t, uint16_t>)
                           : (a.cache_f32 ? latent_query_kernel<float, float> : latent_query_kernel<float, uint16_t>);
    return launch_chained(kernel, grid, dim3(kQueryThreads), a.s.dim_p * 4u, a.pdl, stream, a);
}

stark_b200_status latent_attend_launch(const LatentArgs &a, cudaStream_t stream) {
    if (stark_b200_status st = check_args(a)) return st;
    if (!a.queries || !a.partials) return STARK_B200_INVALID_ARGUMENT;
    if (!a.cache_f32 && latent_attend_mma_supports(a.s)) return latent_attend_mma_launch(a, stream);
    if (a.cluster != 1u) return STARK_B200_INVALID_ARGUMENT;
    SpanAttendArgs g{};  // all heads share the cached rows; their values are the latent columns of the same rows
    g.queries = a.queries, g.heads = a.s.heads, g.key_heads = 1, g.width = a.s.row(), g.out_width = a.s.rank_p;
    g.keys = g.values = a.cache, g.key_pitch = g.value_pitch = a.s.row(), g.cache_f32 = a.cache_f32;
    g.block_table = a.block_table, g.state = a.state, g.first_pos = a.first_pos, g.m = a.m, g.splits = a.splits;
    g.partials = a.partials, g.pdl = a.pdl;
    return span_attend_launch(g, stream);
}

stark_b200_status latent_value_launch(const LatentArgs &a, cudaStream_t stream) {
    if (stark_b200_status st = check_args(a)) return st;
    if (!a.partials || !a.out) return STARK_B200_INVALID_ARGUMENT;
    auto kernel = a.out_b16 ? latent_value_kernel<uint16_t> : latent_value_kernel<float>;
    return launch_chained(kernel, dim3(a.s.heads * (a.s.vdim_p / kValueTile), a.m), dim3(256),
                          a.s.rank_p * 4u + std::max(a.s.rank_p * 4u, 4096u), a.pdl, stream, a);
}

stark_b200_status latent_rotate_append_launch(const LatentArgs &a, cudaStream_t stream) {
    if (stark_b200_status st = check_args(a)) return st;
    if (a.cache_f32 || !a.qd_b16) return STARK_B200_INVALID_ARGUMENT;
    return launch_chained(latent_rotate_append_kernel, dim3(a.m), dim3(256), a.s.rot_p * 4u, true, stream, a);
}

}  // namespace sb
