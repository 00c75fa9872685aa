// Stochastic sampling over one row of full-vocabulary logits, the device form of the reference's
// unified sampler (crates/stark-engine/src/backends/cpu/kernel/sampling/unified_sampling.rs:15-117):
// finite check -> temperature (with overflow centring) -> top-k / top-p / min-p as ONE prefix of the
// descending (value, then lower index) order -> Gumbel-max with Philox4x32-10 noise keyed by the seed
// (encodable_block/sampling/gumbel.rs:1-85) -> first index of the maximum.
//
// One cluster of CTAs, barriers between its phases in hardware.  Bound by the latency of those phases: a row is
// 0.3 MB.  A row of 151 936 bf16 logits (top-k 20, top-p 0.95) takes 59 us where one logit stands out and 305 us where none
// does, f32 89 and 338; on one CTA that added term by term, 1.2, 12.3, 1.7 and 29 ms.  With filters the row is sorted
// for real (stable LSD radix sort, 8-bit digits), because the reference's cut depends on f32 sums accumulated one after
// another in that order.  The sums keep the bits of that chain
// without running it: between two powers of two every addition moves the sum by a whole number of its units in the
// last place, which depends on the sum only through its parity where a term lies half way between two of them, so
// stretches of terms compose (sum_in_order).
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "cluster_fit.cuh"
#include "context.cuh"
#include "ops.cuh"

namespace sb {

namespace {

namespace cg = cooperative_groups;

constexpr int kSampleThreads = 1024;
constexpr int kSampleWarps = kSampleThreads / 32;

__device__ inline void philox_round(uint32_t (&c)[4], uint32_t k0, uint32_t k1) {
    const uint32_t hi0 = __umulhi(0xD2511F53u, c[0]), lo0 = 0xD2511F53u * c[0];
    const uint32_t hi1 = __umulhi(0xCD9E8D57u, c[2]), lo1 = 0xCD9E8D57u * c[2];
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0, c[1] = lo1, c[2] = n2, c[3] = lo0;
}

__device__ inline float gumbel_at(unsigned long long seed, uint32_t index, uint32_t vocab) {
    // revidx (gumbel.rs:66-80): the counter layout of a 1024-thread group drawing 4 words per counter
    const uint32_t thread_idx = index % 1024u, block_idx = index / 1024u;
    const uint32_t offset = ((vocab + 4095u) / 4096u) * thread_idx + block_idx / 4u, word = block_idx % 4u;
    uint32_t c[4] = {offset, 0u, 0u, 0u};
    uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
    philox_round(c, k0, k1);
#pragma unroll
    for (int i = 0; i < 9; ++i) {
        k0 += 0x9E3779B9u;
        k1 += 0xBB67AE85u;
        philox_round(c, k0, k1);
    }
    const uint32_t w = max(c[word] >> 8, 1u);                  // unit_interval: 24 bits, never 0
    const float u = (float)w * (1.0f / 16777216.0f);
    return -logf(-logf(u));
}

// ascending radix order of this key = descending float order
__device__ inline uint32_t descending_key(float v) {
    const uint32_t u = __float_as_uint(v);
    const uint32_t asc = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
    return ~asc;
}
__device__ inline float key_value(uint32_t key) {
    const uint32_t asc = ~key;
    return __uint_as_float((asc & 0x80000000u) ? (asc & 0x7fffffffu) : ~asc);
}

struct SampleParams {
    const void *logits;
    uint32_t io_type, vocab, flags, top_k;
    unsigned long long seed;
    float temperature, top_p, min_p;
    uint32_t *keys[2], *idx[2];  // [vocab] each (filters only)
    uint32_t *out;
};

template <typename T, typename F>
__device__ inline T block_reduce(T v, F f, T *scratch /* [32] */) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = f(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if ((threadIdx.x & 31u) == 0) scratch[threadIdx.x >> 5] = v;
    __syncthreads();
    T r = scratch[0];
    for (int w = 1; w < kSampleWarps; ++w) r = f(r, scratch[w]);
    return r;
}

// Per-CTA working memory of the sort (dynamic shared memory).
struct SortShared {
    uint32_t counts[kSampleWarps][256];  // of a warp's digits, then where its next element of a digit goes within the CTA's
    uint32_t totals[256];                // of this CTA's digits (read by the others of the cluster)
    uint32_t base[256];                  // where this CTA's first element of a digit goes
    uint32_t scan[32];
};

// Elements [lo, hi) of a row that belong to this CTA of the cluster.
struct Segment {
    uint32_t lo, hi;
};
__device__ inline Segment segment_of(uint32_t V, uint32_t rank, uint32_t ranks) {
    const uint32_t each = (V + ranks - 1u) / ranks;
    return {min(V, rank * each), min(V, (rank + 1u) * each)};
}

// Lanes whose digit is the caller's, live lanes only.  Eight votes; match.any takes as many rounds as there are digits.
__device__ inline uint32_t same_digit(uint32_t digit, bool live) {
    uint32_t peers = __ballot_sync(0xffffffffu, live);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        const uint32_t set = __ballot_sync(0xffffffffu, (digit >> b) & 1u);
        peers &= ((digit >> b) & 1u) ? set : ~set;
    }
    return peers;
}

// Stable LSD radix sort of (key, id) pairs by key, ascending, 8-bit digits, by the CTAs of a cluster; digits below
// `first_pass` are equal in all keys (an even number of passes runs, so the sorted pairs end in buffer 0).  Elements
// keep the order (CTA, warp, lane) of their places.  Other CTAs' elements are read past L1.
//
// Bound by a warp's rounds of 32 elements (ranking, then scattered stores), so by the number of warps: 151 936 pairs take 65 us
// in four passes and 33 us in two on 16 CTAs, and took 1.3 ms in four on one.  Ranking by votes instead of match.any: 27 -> 16 us
// a pass.
__device__ inline void sort_pairs(const cg::cluster_group &cluster, uint32_t *const (&keys)[2], uint32_t *const (&idx)[2], uint32_t V,
                                  uint32_t first_pass, SortShared &sh) {
    constexpr uint32_t kAhead = 5;  // rounds of 32 elements whose loads a warp has in flight
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t rank = cluster.block_rank(), ranks = cluster.num_blocks();
    const Segment mine = segment_of(V, rank, ranks);
    const uint32_t span = (mine.hi - mine.lo + kSampleWarps - 1u) / kSampleWarps;
    const uint32_t lo = min(mine.hi, mine.lo + warp * span), hi = min(mine.hi, lo + span);
    cluster.sync();  // the pairs are written
    for (uint32_t pass = first_pass; pass < 4u; ++pass) {
        const uint32_t from = (pass - first_pass) & 1u, shift = pass * 8u;
        const uint32_t *kin = keys[from], *iin = idx[from];
        uint32_t *kout = keys[from ^ 1u], *iout = idx[from ^ 1u];
        for (uint32_t i = lane; i < 256u; i += 32u) sh.counts[warp][i] = 0;
        __syncwarp();
        for (uint32_t base = lo; base < hi; base += 32u * kAhead) {
            uint32_t key[kAhead];
#pragma unroll
            for (uint32_t r = 0; r < kAhead; ++r) key[r] = base + 32u * r + lane < hi ? __ldcg(kin + base + 32u * r + lane) : 0u;
#pragma unroll
            for (uint32_t r = 0; r < kAhead; ++r)
                if (base + 32u * r + lane < hi) atomicAdd(&sh.counts[warp][(key[r] >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (tid < 256u) {  // exclusive over the CTA's warps
            uint32_t run = 0;
#pragma unroll 8
            for (int w = 0; w < kSampleWarps; ++w) {
                const uint32_t c = sh.counts[w][tid];
                sh.counts[w][tid] = run;
                run += c;
            }
            sh.totals[tid] = run;
        }
        cluster.sync();
        uint32_t before = 0, all = 0;
        if (tid < 256u) {
            for (uint32_t r = 0; r < ranks; ++r) {
                const uint32_t c = *cluster.map_shared_rank(&sh.totals[tid], r);
                before += r < rank ? c : 0u;
                all += c;
            }
        }
        uint32_t incl = all;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += n;
        }
        if (lane == 31u) sh.scan[warp] = incl;
        __syncthreads();
        if (tid < 256u) {
            for (uint32_t w = 0; w < warp; ++w) before += sh.scan[w];
            sh.base[tid] = before + incl - all;
        }
        __syncthreads();
        for (uint32_t base = lo; base < hi; base += 32u * kAhead) {
            uint32_t key[kAhead], id[kAhead];
#pragma unroll
            for (uint32_t r = 0; r < kAhead; ++r) {
                const uint32_t i = base + 32u * r + lane;
                key[r] = i < hi ? __ldcg(kin + i) : 0u;
                id[r] = i < hi ? __ldcg(iin + i) : 0u;
            }
#pragma unroll
            for (uint32_t r = 0; r < kAhead; ++r) {
                const bool live = base + 32u * r + lane < hi;
                const uint32_t digit = (key[r] >> shift) & 255u, peers = same_digit(digit, live);
                const uint32_t place = __popc(peers & ((1u << lane) - 1u));
                uint32_t start = 0;
                if (live) start = sh.counts[warp][digit];
                __syncwarp();
                if (live) {
                    const uint32_t at = sh.base[digit] + start + place;
                    kout[at] = key[r];
                    iout[at] = id[r];
                    if (place == 0) sh.counts[warp][digit] = start + __popc(peers);
                }
                __syncwarp();
            }
        }
        cluster.sync();
    }
}

// What a stretch of additions does to a sum that is a whole number of units in the last place: how many units it moves
// when that number is even, and when it is odd (they differ where a term lies half way and rounds to even).
struct Moves {
    unsigned long long even, odd;
};
__device__ inline Moves then(const Moves &a, const Moves &b) {
    return {a.even + ((a.even & 1u) ? b.odd : b.even), a.odd + ((a.odd & 1u) ? b.even : b.odd)};
}
__device__ inline Moves move_of(float units /* the term over the unit, exact */) {
    const float whole = floorf(units), rest = units - whole;
    const unsigned long long k = (unsigned long long)whole;
    if (rest != 0.5f) return {k + (rest > 0.5f), k + (rest > 0.5f)};
    return {k + (k & 1u), k + !(k & 1u)};
}
__device__ inline Moves shift_up(const Moves &m, int by) {
    return {__shfl_up_sync(0xffffffffu, m.even, by), __shfl_up_sync(0xffffffffu, m.odd, by)};
}

struct SumShared {
    Moves warps[kSampleWarps];
    uint32_t crossing, reached;  // first index where the sum passes a power of two / reaches the threshold
    float value;
};

// sum = term(0); sum = sum + term(i) for i = 1 .. count - 1, every addition rounded to f32: the same bits, by one CTA.
// Terms are not negative and descending, term(0) is a normal number.  Stops where the sum is at least `enough`: `used` is the
// number of terms added by then, or count.  A power of two between two sums ends a stretch: that addition is done as it is, and
// the next stretch starts behind it (at most a few dozen stretches of 8 192 terms for any row).
template <typename Term>
__device__ inline float sum_in_order(Term term, uint32_t count, float enough, uint32_t &used, SumShared &sh) {
    constexpr uint32_t kEach = 8;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    float sum = term(0u);
    used = count;
    if (sum >= enough) {
        used = 1;
        return sum;
    }
    for (uint32_t at = 1; at < count;) {
        const int e = ilogbf(sum);
        const float per_unit = ldexpf(1.0f, 23 - e), unit = ldexpf(1.0f, e - 23);
        const unsigned long long start = (unsigned long long)(sum * per_unit);  // in [2^23, 2^24)
        if (tid == 0) sh.crossing = sh.reached = 0xffffffffu;
        float units[kEach];
        Moves own = {0, 0};
        const uint32_t first = at + tid * kEach;
#pragma unroll
        for (uint32_t j = 0; j < kEach; ++j) {
            units[j] = first + j < count ? term(first + j) * per_unit : 0.0f;
            own = then(own, move_of(units[j]));
        }
        Moves upto = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const Moves n = shift_up(upto, o);
            if (lane >= (uint32_t)o) upto = then(n, upto);
        }
        __syncthreads();
        if (lane == 31u) sh.warps[warp] = upto;
        __syncthreads();
        Moves before = {0, 0}, total = {0, 0};
        for (int w = 0; w < kSampleWarps; ++w) {
            if (w == (int)warp) before = total;
            total = then(total, sh.warps[w]);
        }
        const Moves left = shift_up(upto, 1);
        if (lane) before = then(before, left);
        const unsigned long long all = (start & 1u) ? total.odd : total.even;
        unsigned long long n = start + ((start & 1u) ? before.odd : before.even);
        // the threshold in units: a sum of n units has reached it where n >= enough / unit
        const float need = enough * per_unit;
        const bool can_reach = (float)(start + all) >= need || start + all >= (1ull << 24);
        if (can_reach && n < (1ull << 24)) {
#pragma unroll
            for (uint32_t j = 0; j < kEach; ++j) {
                const Moves m = move_of(units[j]);
                const unsigned long long next = n + ((n & 1u) ? m.odd : m.even);
                if (next >= (1ull << 24)) {  // only the first crossing's value survives below
                    atomicMin(&sh.crossing, first + j);
                    break;
                }
                n = next;
                if ((float)n >= need) {
                    atomicMin(&sh.reached, first + j);
                    break;
                }
            }
        }
        __syncthreads();
        const uint32_t crossing = sh.crossing, reached = sh.reached;
        if (reached < crossing) {
            used = reached + 1u;
            return enough;
        }
        if (crossing == 0xffffffffu) {
            if (all == 0) return sum;  // descending terms: none of the rest moves the sum either
            sum = (float)(start + all) * unit;
            at += kSampleThreads * kEach;
            continue;
        }
        if (crossing >= first && crossing < first + kEach) {  // the thread that stands before it adds it as it is
            unsigned long long here = start + ((start & 1u) ? before.odd : before.even);
#pragma unroll
            for (uint32_t j = 0; j < kEach; ++j) {
                if (first + j == crossing) sh.value = (float)here * unit + units[j] * unit;
                const Moves m = move_of(units[j]);
                here += (here & 1u) ? m.odd : m.even;
            }
        }
        __syncthreads();
        sum = sh.value;
        at = crossing + 1u;
        if (sum >= enough) {
            used = at;
            return sum;
        }
        __syncthreads();  // sh.value is read before the next stretch writes it
    }
    return sum;
}

// Reductions over the CTAs of a cluster through one word a CTA.
__device__ inline bool cluster_any(const cg::cluster_group &cluster, bool mine, uint32_t *word) {
    const int any = __syncthreads_or(mine);
    if (threadIdx.x == 0) *word = any != 0;
    cluster.sync();
    uint32_t r = 0;
    for (uint32_t c = 0; c < cluster.num_blocks(); ++c) r |= *cluster.map_shared_rank(word, c);
    cluster.sync();
    return r != 0;
}

__global__ void __launch_bounds__(kSampleThreads) unified_sampling_kernel(const SampleParams p) {
    extern __shared__ uint8_t dynamic_shared[];
    SortShared &sort = *reinterpret_cast<SortShared *>(dynamic_shared);
    __shared__ SumShared sums;
    __shared__ float fscratch[32];
    __shared__ uint32_t uscratch[32];
    __shared__ uint32_t word;
    __shared__ float best_value;
    __shared__ uint32_t best_index;
    const cg::cluster_group cluster = cg::this_cluster();
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, V = p.vocab;
    const uint32_t rank = cluster.block_rank(), ranks = cluster.num_blocks();
    const Segment mine = segment_of(V, rank, ranks);
    const auto logit = [&](uint32_t i) {
        return p.io_type == STARK_B200_F32 ? reinterpret_cast<const float *>(p.logits)[i]
                                           : bf16_bits_to_f32(reinterpret_cast<const uint16_t *>(p.logits)[i]);
    };

    // ---- finite check (unified_sampling.rs:42-45), and what the temperature does to the row (:59-77) ----
    const float recip = (p.flags & 2u) ? 1.0f / p.temperature : 1.0f;
    bool bad = false, over = false, tiny = false;
    float mx = -INFINITY;
    for (uint32_t i = mine.lo + tid; i < mine.hi; i += kSampleThreads) {
        const float v = logit(i);
        bad |= !isfinite(v);
        over |= !isfinite(v * recip);
        tiny |= v != 0.0f && fabsf(v * recip) < 1.1754944e-38f;
        mx = fmaxf(mx, v);
    }
    if (cluster_any(cluster, bad, &word)) {
        if (rank == 0 && tid == 0) *p.out = 0xffffffffu;
        return;
    }
    const bool center = (p.flags & 2u) && cluster_any(cluster, over, &word);
    float shift = 0.0f;
    if (center) {
        mx = block_reduce(mx, [](float a, float b) { return fmaxf(a, b); }, fscratch);
        if (tid == 0) best_value = mx;
        cluster.sync();
        shift = -INFINITY;
        for (uint32_t r = 0; r < ranks; ++r) shift = fmaxf(shift, *cluster.map_shared_rank(&best_value, r));
        cluster.sync();
    }
    const auto scaled = [&](float v) { return (center ? v - shift : v) * recip; };

    float best = -INFINITY;
    uint32_t bi = 0xffffffffu;
    const auto candidate = [&](float v, uint32_t i) {
        if (p.flags & 1u) v += gumbel_at(p.seed, i, V);
        if (v > best || (v == best && i < bi) || bi == 0xffffffffu) {
            best = v;
            bi = i;
        }
    };
    uint32_t parts = ranks;  // CTAs that hold candidates
    if (p.flags & (4u | 8u | 16u)) {
        // ---- filters (:79-99): sort, sums in order, prefix ----
        // bf16 logits keep their order and their ties under a scaling that neither overflows nor reaches the subnormal numbers:
        // their own 16 bits are sorted (two passes) and scaled afterwards
        const bool half = p.io_type != STARK_B200_F32 && !center && !cluster_any(cluster, tiny, &word);
        for (uint32_t i = mine.lo + tid; i < mine.hi; i += kSampleThreads) {
            const float v = half ? logit(i) : scaled(logit(i));
            p.keys[0][i] = descending_key(v == 0.0f ? 0.0f : v);  // -0 and +0 compare equal: one key for both
            p.idx[0][i] = i;
        }
        sort_pairs(cluster, p.keys, p.idx, V, half ? 2u : 0u, sort);
        if (rank != 0) return;
        const auto value = [&](uint32_t n) {
            const float v = key_value(__ldcg(p.keys[0] + n));
            return half ? v * recip : v;
        };
        const float top = value(0u);
        uint32_t kept = (p.flags & 4u) ? min(p.top_k, V) : V;
        if (p.flags & 16u) {
            const float floor_value = top + logf(p.min_p);
            uint32_t first = kept;  // the first below the floor: values descend, so the ones before it are counted
            for (uint32_t base = 0; base < kept; base += kSampleThreads) {
                const uint32_t n = base + tid;
                const int in = __syncthreads_count(n < kept && !(value(n) < floor_value));
                if (in < (int)min((uint32_t)kSampleThreads, kept - base)) {
                    first = base + in;
                    break;
                }
            }
            kept = first;
        }
        if ((p.flags & 8u) && kept) {
            const auto term = [&](uint32_t n) { return expf(value(n) - top); };
            uint32_t used;
            const float norm = sum_in_order(term, V, INFINITY, used, sums);  // sequential f32 sum in sorted order (:84-85)
            __syncthreads();
            sum_in_order([&](uint32_t n) { return term(n) / norm; }, kept, p.top_p, used, sums);
            kept = used;
        }
        for (uint32_t n = tid; n < kept; n += kSampleThreads) candidate(value(n), __ldcg(p.idx[0] + n));
        parts = 1;
    } else {
        for (uint32_t i = mine.lo + tid; i < mine.hi; i += kSampleThreads) candidate(scaled(logit(i)), i);
    }
    // ---- Gumbel-max (:101-106) and the first index of the maximum (:108-114) ----
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, o);
        if (ov > best || (ov == best && oi < bi)) {
            best = ov;
            bi = oi;
        }
    }
    __syncthreads();
    if (lane == 0) {
        fscratch[warp] = best;
        uscratch[warp] = bi;
    }
    __syncthreads();
    if (tid == 0) {
        for (int w = 1; w < kSampleWarps; ++w)
            if (fscratch[w] > best || (fscratch[w] == best && uscratch[w] < bi)) {
                best = fscratch[w];
                bi = uscratch[w];
            }
        best_value = best;
        best_index = bi;
    }
    if (parts > 1u) {
        cluster.sync();
        if (rank == 0 && tid == 0)
            for (uint32_t r = 1; r < parts; ++r) {
                const float ov = *cluster.map_shared_rank(&best_value, r);
                const uint32_t oi = *cluster.map_shared_rank(&best_index, r);
                if (ov > best || (ov == best && oi < bi)) {
                    best = ov;
                    bi = oi;
                }
            }
        cluster.sync();
    }
    if (rank == 0 && tid == 0) *p.out = isfinite(best) ? bi : 0xffffffffu;
}

// The generation worker's host sampler (crates/stark-generate/src/hybrid.rs:1122-1212) on the device:
// candidates = the first k of the descending total order (lower id first among equal bit patterns,
// :1265-1372), probabilities exp(f64((l - max) / temperature)) with the subtraction and division in f32
// (:138-165), the sequential f64 total, the min-p / top-p prefix (:1192-1204), one SplitMix64 draw scaled
// by the kept mass and a sequential scan (:1103-1111, :1134-1142).
//
// The partial sums S_n of the probabilities in candidate order serve the total, the prefix walk and the
// scan alike, and they are what fixes the result bit for bit, so one thread forms them in order.  Two
// things keep that short: once adding a term leaves S unchanged no later (smaller) term can change it, so
// every walk stops adding there; and the quotient S / total is only formed when S is within 1e-14 of the
// threshold, where the comparison could go either way.
__global__ void __launch_bounds__(kSampleThreads) ordered_sampling_kernel(const SampleParams p) {
    extern __shared__ uint8_t dynamic_shared[];
    SortShared &sort = *reinterpret_cast<SortShared *>(dynamic_shared);
    __shared__ uint32_t first_below, word;
    const cg::cluster_group cluster = cg::this_cluster();
    const uint32_t tid = threadIdx.x, V = p.vocab;
    const uint32_t rank = cluster.block_rank(), ranks = cluster.num_blocks();
    const Segment mine = segment_of(V, rank, ranks);
    bool bad = false;
    for (uint32_t i = mine.lo + tid; i < mine.hi; i += kSampleThreads) {
        const float v = p.io_type == STARK_B200_F32 ? reinterpret_cast<const float *>(p.logits)[i]
                                                     : bf16_bits_to_f32(reinterpret_cast<const uint16_t *>(p.logits)[i]);
        bad |= !isfinite(v);
        p.keys[0][i] = descending_key(v);  // signed zeros stay distinct, as under total_cmp
        p.idx[0][i] = i;
    }
    if (tid == 0) first_below = 0xffffffffu;
    if (cluster_any(cluster, bad, &word)) {
        if (rank == 0 && tid == 0) *p.out = 0xffffffffu;
        return;
    }
    sort_pairs(cluster, p.keys, p.idx, V, p.io_type == STARK_B200_F32 ? 0u : 2u, sort);  // bf16 keys differ in 16 bits only
    const uint32_t *skey = p.keys[0], *sidx = p.idx[0];
    double *terms = reinterpret_cast<double *>(p.idx[1]);  // idx[1] and the f32 term array: 8 bytes per entry
    const uint32_t k = (p.flags & 4u) ? min(p.top_k, V) : V;
    const float top = key_value(__ldcg(skey));
    const float temperature = (p.flags & 2u) ? p.temperature : 1.0f;
    const double min_p = (double)p.min_p;
    uint32_t below = 0xffffffffu;
    for (uint32_t i = rank * kSampleThreads + tid; i < k; i += ranks * kSampleThreads) {
        const double t = exp((double)__fdiv_rn(__fsub_rn(key_value(__ldcg(skey + i)), top), temperature));
        terms[i] = t;
        if ((p.flags & 16u) && i > 0 && t < min_p) below = min(below, i);
    }
    if (below != 0xffffffffu) atomicMin(cluster.map_shared_rank(&first_below, 0), below);
    cluster.sync();
    if (rank != 0 || tid != 0) return;
    const uint32_t limit = min(k, first_below);  // the min-p cut: the first candidate after the top one below it
    // total; `live` = number of leading terms that still move the partial sums
    double total = 0.0;
    uint32_t live = k;
    for (uint32_t base = 0; base < k && live == k; base += 8u) {
        double t[8];
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) t[j] = base + j < k ? __ldcg(terms + base + j) : 0.0;
#pragma unroll
        for (uint32_t j = 0; j < 8u; ++j) {
            if (base + j >= k) break;
            if (base + j > 0 && total + 2.0 * t[j] == total) {
                live = base + j;
                break;
            }
            total += t[j];
        }
    }
    // prefix: stop before candidate n > 0 once S_n / total >= top_p
    double cumulative = 0.0;
    uint32_t kept = 0;
    if (p.flags & 8u) {
        const double top_p = (double)p.top_p, edge = top_p * total;
        const double lo = edge * (1.0 - 1e-14), hi = edge * (1.0 + 1e-14);
        for (; kept < limit; ++kept) {
            if (kept > 0 && cumulative >= lo && (cumulative > hi || cumulative / total >= top_p)) break;
            if (kept >= live) {  // S no longer changes: neither does the comparison
                kept = limit;
                break;
            }
            cumulative += __ldcg(terms + kept);
        }
    } else {
        const uint32_t n = min(limit, live);
        for (uint32_t base = 0; base < n; base += 8u) {
            double t[8];
#pragma unroll
            for (uint32_t j = 0; j < 8u; ++j) t[j] = base + j < n ? __ldcg(terms + base + j) : 0.0;
#pragma unroll
            for (uint32_t j = 0; j < 8u; ++j)
                if (base + j < n) cumulative += t[j];
        }
        kept = limit;
    }
    // draw
    unsigned long long z = p.seed + 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    const double u = (double)((z ^ (z >> 31)) >> 11) * (1.0 / 9007199254740992.0);
    const double target = u * cumulative;
    uint32_t chosen = kept - 1u;
    double mass = 0.0;
    const uint32_t scan = min(kept, live);
    for (uint32_t n = 0; n < scan; ++n) {
        mass += __ldcg(terms + n);
        if (target < mass) {
            chosen = n;
            break;
        }
    }
    *p.out = __ldcg(sidx + chosen);
}

cudaLaunchConfig_t sampling_config(uint32_t cluster, cudaStream_t stream) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(cluster);
    c.blockDim = dim3(kSampleThreads);
    c.dynamicSmemBytes = sizeof(SortShared);
    c.stream = stream;
    return c;
}

cudaLaunchAttribute cluster_of(uint32_t ctas) {
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = ctas;
    a.val.clusterDim.y = a.val.clusterDim.z = 1;
    return a;
}

}  // namespace

size_t sampling_scratch_bytes(uint32_t vocab) { return (size_t)vocab * 4u * 6u; }

// SamplingMethod::validate (generation.rs:67-111): finite temperature in (0, 100] with a finite
// reciprocal, 1 <= top_k <= vocab, 0 < top_p <= 1, 0 <= min_p <= 1.
stark_b200_status sampling_validate(const stark_b200_sampling &s, uint32_t vocab) {
    if (vocab == 0 || (s.flags & ~63u)) return STARK_B200_INVALID_ARGUMENT;
    if ((s.flags & 32u) && !(s.flags & 1u)) return STARK_B200_INVALID_ARGUMENT;  // the ordered sampler only draws
    if (s.flags & 2u) {
        if (!std::isfinite(s.temperature) || !(s.temperature > 0.0f) || s.temperature > 100.0f ||
            !std::isfinite(1.0f / s.temperature))
            return STARK_B200_INVALID_ARGUMENT;
    }
    if ((s.flags & 4u) && (s.top_k < 1u || s.top_k > vocab)) return STARK_B200_INVALID_ARGUMENT;
    if ((s.flags & 8u) && !(s.top_p > 0.0f && s.top_p <= 1.0f)) return STARK_B200_INVALID_ARGUMENT;
    if ((s.flags & 16u) && !(s.min_p >= 0.0f && s.min_p <= 1.0f)) return STARK_B200_INVALID_ARGUMENT;
    return STARK_B200_OK;
}

stark_b200_status sampling_launch(const void *logits, uint32_t io_type, uint32_t vocab, const stark_b200_sampling &s,
                                  void *scratch, uint32_t *out_device, cudaStream_t stream) {
    stark_b200_status st = sampling_validate(s, vocab);
    if (st != STARK_B200_OK) return st;
    if (!logits || !scratch || !out_device || io_type > STARK_B200_F32) return STARK_B200_INVALID_ARGUMENT;
    SampleParams p{};
    p.logits = logits;
    p.io_type = io_type;
    p.vocab = vocab;
    p.flags = s.flags;
    p.top_k = s.top_k;
    p.seed = s.seed;
    p.temperature = s.temperature;
    p.top_p = s.top_p;
    p.min_p = s.min_p;
    uint32_t *base = static_cast<uint32_t *>(scratch);
    p.keys[0] = base;
    p.keys[1] = base + vocab;
    p.idx[0] = base + 2u * (size_t)vocab;
    p.idx[1] = base + 4u * (size_t)vocab;  // with the array behind it: the ordered sampler's f64 terms, 8-byte aligned
    p.out = out_device;
    const bool ordered = (s.flags & 32u) != 0;
    static ClusterFit known[2];
    const auto kernel = ordered ? ordered_sampling_kernel : unified_sampling_kernel;
    const uint32_t cluster = cluster_fit((const void *)kernel, sampling_config(0u, stream), known[ordered]);
    if (!cluster) return STARK_B200_DEVICE_FAILURE;
    cudaLaunchConfig_t config = sampling_config(cluster, stream);
    cudaLaunchAttribute attribute = cluster_of(cluster);
    config.attrs = &attribute;
    config.numAttrs = 1;
    SB_CUDA(cudaLaunchKernelEx(&config, kernel, p));
    return STARK_B200_OK;
}

}  // namespace sb
