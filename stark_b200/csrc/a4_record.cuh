// A 576-byte record of a re-tiled 4-bit matrix (qmv.cuh) as bf16 weights: the operand of the prompt contractions.
#pragma once
#include "qmv.cuh"

namespace sb {

struct RecordRegs {
    uint4 q;
    uint32_t scales, biases;  // bf16 pairs: rows g and g + 8
};

__device__ inline RecordRegs load_record(const uint8_t *w, uint32_t tile, uint32_t row_tiles, uint32_t groups,
                                         uint32_t kg, uint32_t lane) {
    RecordRegs r;
    if (tile < row_tiles) {
        const uint8_t *rec = w + ((size_t)tile * groups + kg) * kA4RecordBytes;
        r.q = ldg_nc_v4(rec + lane * 16u);
        r.scales = __ldg(reinterpret_cast<const uint32_t *>(rec + 512u + 4u * (lane >> 2)));
        r.biases = __ldg(reinterpret_cast<const uint32_t *>(rec + 544u + 4u * (lane >> 2)));
    } else {  // past the last row tile: zero rows
        r.q = make_uint4(0u, 0u, 0u, 0u);
        r.scales = 0u;
        r.biases = 0u;
    }
    return r;
}

// One record word -> the eight codes as exact bf16 integers, in the fragment order of dequant_a4_word:
// (w >> 4s) & 0x000f000f | 0x43004300 is the bf16 pair (128 + q, 128 + q') -- 0x4300 is 128.0 and the last
// mantissa bit of a bf16 in [128, 256) weighs 1 -- and 128 is then subtracted exactly.
__device__ inline void codes_to_bf16(uint32_t w, __nv_bfloat162 (&q)[4]) {
    const uint32_t magic = 0x43004300u;
    const __nv_bfloat162 k128 = __float2bfloat162_rn(128.0f);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const uint32_t v = lop3_and_or(w >> (4 * s), 0x000f000fu, magic);
        q[s] = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&v), k128);
    }
}
__device__ inline __nv_bfloat162 bf16_pair(uint32_t bits16) {
    const uint32_t v = bits16 | (bits16 << 16);
    return *reinterpret_cast<const __nv_bfloat162 *>(&v);
}

// A lane's share of a record: columns 16 t .. 16 t + 15 of row g (out[0], out[1]) and of row g + 8 (out[2], out[3]).
__device__ inline void dequant_record(const RecordRegs &r, uint4 (&out)[4]) {
    const __nv_bfloat162 s0 = bf16_pair(r.scales & 0xffffu), s1 = bf16_pair(r.scales >> 16);
    const __nv_bfloat162 b0 = bf16_pair(r.biases & 0xffffu), b1 = bf16_pair(r.biases >> 16);
    const uint32_t ww[4] = {r.q.x, r.q.y, r.q.z, r.q.w};
    uint32_t lo_row[8], hi_row[8];  // 16 bf16 values per row
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        __nv_bfloat162 a[4];
        codes_to_bf16(ww[j], a);  // a[0], a[2]: row g, columns 4j + {0,1}, {2,3}; a[1], a[3]: row g + 8
        // bf16(scale * q + bias): one fused multiply-add, one rounding -- the dequantized operand in the
        // activations' type, as the reference's tiled GEMM stages it (gemm.metal:122-203, `threadgroup BT b_shared`)
        const __nv_bfloat162 v0 = __hfma2(a[0], s0, b0);
        const __nv_bfloat162 v2 = __hfma2(a[2], s0, b0);
        const __nv_bfloat162 v1 = __hfma2(a[1], s1, b1);
        const __nv_bfloat162 v3 = __hfma2(a[3], s1, b1);
        lo_row[2 * j] = *reinterpret_cast<const uint32_t *>(&v0);
        lo_row[2 * j + 1] = *reinterpret_cast<const uint32_t *>(&v2);
        hi_row[2 * j] = *reinterpret_cast<const uint32_t *>(&v1);
        hi_row[2 * j + 1] = *reinterpret_cast<const uint32_t *>(&v3);
    }
    out[0] = make_uint4(lo_row[0], lo_row[1], lo_row[2], lo_row[3]);
    out[1] = make_uint4(lo_row[4], lo_row[5], lo_row[6], lo_row[7]);
    out[2] = make_uint4(hi_row[0], hi_row[1], hi_row[2], hi_row[3]);
    out[3] = make_uint4(hi_row[4], hi_row[5], hi_row[6], hi_row[7]);
}

// Matrices as bf16 rows [16 row_tiles][64 groups], in storage order: the values the dequantizing warps of the packed contraction form.
struct UnpackJobs {
    const uint8_t *w[2];
    uint16_t *out[2];
    uint32_t row_tiles[2], groups[2];
};
// Warp `first` of `warps`, two records in flight.  Memory-bound: 0.56 bytes read and 2 written a weight; a record fills 16 whole
// 128-byte lines.
__device__ inline void unpack_records(const uint8_t *w, uint16_t *out, uint32_t row_tiles, uint32_t groups, uint32_t first, uint32_t warps) {
    const uint32_t lane = threadIdx.x & 31u, g = lane >> 2, t = lane & 3u, records = row_tiles * groups, columns = groups * 64u;
    for (; first < records; first += 2u * warps) {
        const uint32_t at[2] = {first, first + warps};
        RecordRegs r[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) r[i] = load_record(w, at[i] < records ? 0u : 1u, 1u, 1u, at[i], lane);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            if (at[i] >= records) break;
            uint4 v[4];
            dequant_record(r[i], v);
            uint16_t *row = out + (size_t)(at[i] / groups * 16u + g) * columns + at[i] % groups * 64u + 16u * t;
            reinterpret_cast<uint4 *>(row)[0] = v[0], reinterpret_cast<uint4 *>(row)[1] = v[1];
            row += (size_t)8u * columns;
            reinterpret_cast<uint4 *>(row)[0] = v[2], reinterpret_cast<uint4 *>(row)[1] = v[3];
        }
    }
}

}  // namespace sb
