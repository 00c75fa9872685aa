// The arithmetic of the routed-expert decoder, shared by a token's kernels (moe_token.cu) and a pass's (moe_rows.cu): every sum
// is formed in the same order in both, with its multiply-adds written out, so that prompt rows leave the same bits whether they
// are ingested in a pass, one by one, or by ranks that ingest one by one.
#pragma once
#include "gguf_math.cuh"

namespace sb {

constexpr uint32_t kHeadWidth = 128;
constexpr uint32_t kSlice = 256;      // columns of a record: what one warp stages, eight a lane
constexpr uint32_t kMaxMembers = 16;  // warps that share a row

// How warps share the slices of a row: member m takes slices m, m + width, ...; sums over a row go member by member.
struct Members {
    uint32_t supers, width, records;  // slices; members; the most slices of one
};
__host__ __device__ inline Members members_of(uint32_t columns) {
    Members m{};
    m.supers = columns / kSlice;
    m.records = (m.supers + kMaxMembers - 1u) / kMaxMembers;
    m.width = (m.supers + m.records - 1u) / m.records;
    return m;
}

__device__ inline void load8(const float *src, float (&v)[8]) {
    const float4 a = reinterpret_cast<const float4 *>(src)[0], b = reinterpret_cast<const float4 *>(src)[1];
    v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
}

// A lane's eight values times the norm's weights, and their squares; the norm's own scale is multiplied into the sums.
__device__ inline void weigh8(float (&v)[8], const float (&w)[8], float &square) {
#pragma unroll
    for (int i = 0; i < 8; ++i) square = fmaf(v[i], v[i], square), v[i] = __fmul_rn(v[i], w[i]);
}
__device__ inline float norm_scale(float squares, uint32_t columns, float eps) { return 1.0f / sqrtf(squares / (float)columns + eps); }

// A slice as f16 head and remainder of v * up, up the power of two that brings its largest element to the top of f16's range;
// down = 1 / up.  sum: of v * up over the 32 columns of this lane's sub-block (lanes 4 j ... 4 j + 3 hold sub-block j).
struct SplitSlice {
    uint4 head, rest;
    float down, sum;
};
__device__ inline SplitSlice split_slice(const float (&v)[8]) {
    uint32_t top = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) top = max(top, __float_as_uint(v[i]) & 0x7fffffffu);
    top = __reduce_max_sync(0xffffffffu, top);
    int shift = max(-100, min(100, 14 - ((int)(top >> 23) - 127)));
    if (top == 0u || top >= 0x7f800000u) shift = 0;
    const float up = __uint_as_float((uint32_t)(shift + 127) << 23);
    uint32_t head[4], rest[4];
    SplitSlice s;
    s.sum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = __fmul_rn(v[2 * i], up), b = __fmul_rn(v[2 * i + 1], up);
        const __half2 h = __floats2half2_rn(a, b), r = __floats2half2_rn(a - __low2float(h), b - __high2float(h));
        head[i] = *reinterpret_cast<const uint32_t *>(&h);
        rest[i] = *reinterpret_cast<const uint32_t *>(&r);
        s.sum += a + b;
    }
    s.sum += __shfl_xor_sync(0xffffffffu, s.sum, 1);
    s.sum += __shfl_xor_sync(0xffffffffu, s.sum, 2);
    s.head = make_uint4(head[0], head[1], head[2], head[3]);
    s.rest = make_uint4(rest[0], rest[1], rest[2], rest[3]);
    s.down = __uint_as_float((uint32_t)(127 - shift) << 23);
    return s;
}

// What sub-blocks t and t + 4 add to a row: s0, s1 the products of their codes with the slice, xa, xb the slice's sums there;
// sub-block t + 4 first.  A slice adds down * ((share 0 + share 1) + (share 2 + share 3)).
__device__ inline float q8_share_second(float scale1, float s1) { return __fmul_rn(scale1, s1); }
__device__ inline float q4k_share_second(float scale1, float s1, float min0, float xa, float min1, float xb) {
    return fmaf(scale1, s1, -fmaf(min0, xa, __fmul_rn(min1, xb)));
}
__device__ inline float share_first(float scale0, float s0, float second) { return fmaf(scale0, s0, second); }
__device__ inline float q8_share(float scale0, float s0, float scale1, float s1) { return share_first(scale0, s0, q8_share_second(scale1, s1)); }
__device__ inline float q4k_share(float scale0, float s0, float scale1, float s1, float min0, float xa, float min1, float xb) {
    return share_first(scale0, s0, q4k_share_second(scale1, s1, min0, xa, min1, xb));
}

// silu with the two-branch sigmoid (engine/hybrid/math.rs:5-16), times the up row's value
__device__ inline float gated_value(float gate, float up) {
    float sigmoid;
    if (gate >= 0.0f) {
        sigmoid = 1.0f / (1.0f + expf(-gate));
    } else {
        const float e = expf(gate);
        sigmoid = e / (1.0f + e);
    }
    return __fmul_rn(__fmul_rn(gate, sigmoid), up);
}

// One 128-wide head by one warp: lane L holds elements L, 32 + L, 64 + L, 96 + L, so both halves of a rotation pair sit in one
// lane, and the sums are formed in the order of moe_heads_kernel's four warps: the same bits.
__device__ inline void head_angles(uint32_t position, float theta, uint32_t lane, float (&cs)[2], float (&sn)[2]) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float angle = __fmul_rn((float)position, powf(theta, -((float)(2u * (32u * k + lane))) / (float)kHeadWidth));
        sincosf(angle, &sn[k], &cs[k]);
    }
}
__device__ inline void prepare_head(const float (&v)[4], const float (&norm)[4], const float (&cs)[2], const float (&sn)[2],
                                    float eps, float (&out)[4]) {
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) sum += warp_sum(__fmul_rn(v[k], v[k]));
    const float scale = norm_scale(sum, kHeadWidth, eps);
    float head[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) head[k] = __fmul_rn(__fmul_rn(v[k], scale), norm[k]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const float a = head[k], b = head[k + 2];
        out[k] = fmaf(a, cs[k], -__fmul_rn(b, sn[k]));
        out[k + 2] = fmaf(a, sn[k], __fmul_rn(b, cs[k]));
    }
}

// Attention.  A span of the cache is eight strands (keys lo + w, lo + w + 8, ... are strand w), each with a running softmax; the
// strands of a span merge in order, then the spans.  Strand and span have their four columns a lane and four floats.
constexpr uint32_t kStrands = 8;
constexpr uint32_t kMinSpan = 16;  // cache rows of a span at least: two for every strand

// Cache rows per span, and with it the spans that hold any, of a token that sees `rows` rows.
__host__ __device__ inline uint32_t span_rows(uint32_t rows, uint32_t splits) {
    const uint32_t even = (rows + splits - 1u) / splits;
    return even > kMinSpan ? even : kMinSpan;
}

__device__ inline float dot4(const float4 &a, const float4 &b) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, __fmul_rn(a.x, b.x))));
}
// One more key of a strand: its accumulator is to be scaled by c and takes the key's value times e.
__device__ inline void strand_step(float &m, float &l, float score, float &c, float &e) {
    const float top = fmaxf(m, score);
    c = expf(m - top), e = expf(score - top);
    l = fmaf(l, c, e);
    m = top;
}
__device__ inline void strand_add(float4 &acc, float c, float e, const float4 &v) {
    acc.x = fmaf(acc.x, c, __fmul_rn(e, v.x)), acc.y = fmaf(acc.y, c, __fmul_rn(e, v.y));
    acc.z = fmaf(acc.z, c, __fmul_rn(e, v.z)), acc.w = fmaf(acc.w, c, __fmul_rn(e, v.w));
}
// What a strand weighs in its span, whose maximum is `top` (an empty one nothing), and the merge.
__device__ inline float strand_weight(float m, float top) { return m == -INFINITY ? 0.0f : expf(m - top); }
__device__ inline void strand_take(float &l, float4 &acc, float weight, float strand_l, const float4 &strand) {
    l = fmaf(strand_l, weight, l);
    acc.x = fmaf(strand.x, weight, acc.x), acc.y = fmaf(strand.y, weight, acc.y);
    acc.z = fmaf(strand.z, weight, acc.z), acc.w = fmaf(strand.w, weight, acc.w);
}

// The merge of up to 64 spans of a head: a lane holds the maximum and sum of spans `lane` and `lane + 32`, and gets their
// weights; returns what the weighted columns are divided by.
__device__ inline float span_weights(const float (&m)[2], const float (&l)[2], float (&c)[2]) {
    const float top = warp_max(fmaxf(m[0], m[1]));
#pragma unroll
    for (int j = 0; j < 2; ++j) c[j] = strand_weight(m[j], top);
    return warp_sum(fmaf(l[1], c[1], __fmul_rn(l[0], c[0])));
}

// With `pdl` the launch may start before its predecessor ends; every kernel of the decoder awaits that one by itself.
template <typename... Params, typename... Args>
stark_b200_status moe_launch(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, bool pdl, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    SB_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
    return STARK_B200_OK;
}

}  // namespace sb
