// group_select.cu — hash-grouped results without work on empty slots:
//   * a distinct-count sketch of the group keys, from which the host sizes the
//     group hash table (the table has to hold the distinct keys, not the rows);
//   * ORDER BY aggregate LIMIT n by selection: the n-th group's place is
//     narrowed by histograms of the ordering value, and only the last few
//     candidates are sorted.
// The reference groups into growing hash maps (accum_grouped.rs) and sorts
// every group (execute_grouped's ORDER BY, expr.rs:2391-2395).
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <vector>

#include "device_common.cuh"
#include "group_format.cuh"
#include "plan.hpp"
#include "runtime.hpp"

namespace tgp {

// ---------------------------------------------------------------------------
// Distinct sketch: a HyperLogLog (Flajolet et al. 2007) of 2^11 registers over
// the packed group keys, hashed with the splitmix64 finaliser. Its standard
// error of 2.3 % is far inside the slack the host leaves, and an
// underestimate only makes the scan run again on the full-size table.
// Streams the key columns once: 20M 8-byte keys, 160 MB.
// ---------------------------------------------------------------------------
namespace {

constexpr int kSketchBits = 11;
constexpr uint32_t kSketchRegs = 1u << kSketchBits;
constexpr int kSketchThreads = 512;
constexpr int kSketchQuads = 2;   // groups of four rows per thread and pass, loads issued together

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x ^= x >> 30;
    x *= 0xbf58476d1ce4e5b9ull;
    x ^= x >> 27;
    x *= 0x94d049bb133111ebull;
    return x ^ (x >> 31);
}

// Four consecutive cells from row i (a multiple of 4), sign- or zero-extended.
template <uint32_t DT>
__device__ __forceinline__ void sketch_cells(const uint8_t* col, uint64_t i, long long (&x)[4]) {
    if constexpr (DT == DT_U8) {
        const uint32_t w = __ldcs(reinterpret_cast<const unsigned int*>(col) + i / 4);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = (w >> (8 * e)) & 0xffu;
    } else if constexpr (DT == DT_I32) {
        const int4 v = __ldcs(reinterpret_cast<const int4*>(col) + i / 4);
        x[0] = v.x;
        x[1] = v.y;
        x[2] = v.z;
        x[3] = v.w;
    } else {
        const longlong2 a = __ldcs(reinterpret_cast<const longlong2*>(col) + i / 2);
        const longlong2 b = __ldcs(reinterpret_cast<const longlong2*>(col) + i / 2 + 1);
        x[0] = a.x;
        x[1] = a.y;
        x[2] = b.x;
        x[3] = b.y;
    }
}

__device__ __forceinline__ int64_t sketch_cell(const uint8_t* col, uint32_t dtype, uint64_t i) {
    if (dtype == DT_U8) return __ldg(col + i);
    if (dtype == DT_I32) return __ldg(reinterpret_cast<const int*>(col) + i);
    return __ldg(reinterpret_cast<const long long*>(col) + i);
}

__device__ __forceinline__ void sketch_add(uint32_t* reg, unsigned long long key) {
    const unsigned long long h = mix64(key + 0x9e3779b97f4a7c15ull);
    const uint32_t at = static_cast<uint32_t>(h >> (64 - kSketchBits));
    const uint32_t rank = static_cast<uint32_t>(__clzll(static_cast<long long>((h << kSketchBits) | 1ull))) + 1u;
    if (rank > *reinterpret_cast<volatile uint32_t*>(reg + at)) atomicMax(reg + at, rank);
}

// DT: the one key column's type, or 0 for several keys.
template <uint32_t DT>
__global__ void __launch_bounds__(kSketchThreads) key_sketch_kernel(const SketchArgs A) {
    __shared__ uint32_t reg[kSketchRegs];
    for (uint32_t r = threadIdx.x; r < kSketchRegs; r += kSketchThreads) reg[r] = 0;
    __syncthreads();
    const uint64_t T = static_cast<uint64_t>(gridDim.x) * kSketchThreads;
    const uint64_t first = static_cast<uint64_t>(blockIdx.x) * kSketchThreads + threadIdx.x;
    uint64_t done = 0;   // rows of whole groups of four
    if constexpr (DT != 0) {
        const uint64_t quads = A.nrows / 4;
        done = quads * 4;
        const unsigned long long kmin = static_cast<unsigned long long>(A.min[0]);
        uint64_t q = first;
        for (; q + (kSketchQuads - 1) * T < quads; q += kSketchQuads * T) {
            long long x[kSketchQuads][4];
#pragma unroll
            for (int u = 0; u < kSketchQuads; ++u) sketch_cells<DT>(A.col[0], 4 * (q + u * T), x[u]);
#pragma unroll
            for (int u = 0; u < kSketchQuads; ++u)
#pragma unroll
                for (int e = 0; e < 4; ++e) sketch_add(reg, static_cast<unsigned long long>(x[u][e]) - kmin);
        }
        for (; q < quads; q += T) {
            long long x[4];
            sketch_cells<DT>(A.col[0], 4 * q, x);
#pragma unroll
            for (int e = 0; e < 4; ++e) sketch_add(reg, static_cast<unsigned long long>(x[e]) - kmin);
        }
    }
    for (uint64_t i = done + first; i < A.nrows; i += T) {
        unsigned long long key = 0;
        for (uint32_t k = 0; k < A.nkey; ++k)
            key |= (static_cast<unsigned long long>(sketch_cell(A.col[k], A.dtype[k], i)) -
                    static_cast<unsigned long long>(A.min[k]))
                   << A.shift[k];
        sketch_add(reg, key);
    }
    __syncthreads();
    for (uint32_t r = threadIdx.x; r < kSketchRegs; r += kSketchThreads)
        if (reg[r] > *reinterpret_cast<volatile uint32_t*>(A.regs + r)) atomicMax(A.regs + r, reg[r]);
}

}  // namespace

size_t key_sketch_bytes() { return kSketchRegs * sizeof(uint32_t); }

cudaError_t launch_key_sketch(const SketchArgs& A, int sms, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(A.regs, 0, key_sketch_bytes(), st);
    if (e != cudaSuccess || A.nrows == 0) return e;
    const uint64_t per = static_cast<uint64_t>(kSketchThreads) * 4 * kSketchQuads;
    uint64_t blocks = (A.nrows + per - 1) / per;
    if (blocks > static_cast<uint64_t>(sms) * 4) blocks = static_cast<uint64_t>(sms) * 4;
    const unsigned grid = static_cast<unsigned>(blocks);
    const uint32_t dt = A.nkey == 1 && A.shift[0] == 0 ? A.dtype[0] : 0u;
    if (dt == DT_U8) key_sketch_kernel<DT_U8><<<grid, kSketchThreads, 0, st>>>(A);
    else if (dt == DT_I32) key_sketch_kernel<DT_I32><<<grid, kSketchThreads, 0, st>>>(A);
    else if (dt == DT_I64 || dt == DT_U64) key_sketch_kernel<DT_I64><<<grid, kSketchThreads, 0, st>>>(A);
    else key_sketch_kernel<0><<<grid, kSketchThreads, 0, st>>>(A);
    return cudaGetLastError();
}

double key_sketch_estimate(const uint32_t* regs) {
    const double m = kSketchRegs;
    double sum = 0.0;
    uint32_t zeros = 0;
    for (uint32_t r = 0; r < kSketchRegs; ++r) {
        sum += std::ldexp(1.0, -static_cast<int>(regs[r]));
        zeros += regs[r] == 0;
    }
    const double raw = 0.7213 / (1.0 + 1.079 / m) * m * m / sum;
    return raw <= 2.5 * m && zeros ? m * std::log(m / zeros) : raw;
}

// ---------------------------------------------------------------------------
// Top-N by selection. A candidate is an occupied slot with its ordering word
// (ascending = wanted order) and its packed key (ties in ascending key order).
//   collect: one pass over the table lists every group and the ordering
//            words' range;
//   narrow:  a histogram of 4,096 buckets over the range; groups in buckets
//            before the one holding the n-th are sure, that bucket's own are
//            the next candidates, its bounds the next range. Once the ordering
//            words are all equal the keys take their place;
//   finish:  at most kTopSort sure and candidate groups are sorted in one
//            block and the first n formatted.
// One narrow usually suffices; the block state says when the host has to
// launch another (each divides the range by 4,096).
// ---------------------------------------------------------------------------
namespace {

constexpr int kTopThreads = 256;
constexpr uint32_t kTopBuckets = 4096;
constexpr uint32_t kTopSort = 2 * kTopSelectMax;   // groups the finishing block sorts

struct TopCand {
    unsigned long long order, key, slot;
};

__global__ void top_init_kernel(TopState* st, uint64_t limit, unsigned long long key_hi) {
    TopState s{};
    s.lo = ~0ull;
    s.want = limit;
    s.key_hi = key_hi;
    *st = s;
}

__device__ __forceinline__ unsigned long long order_word(const unsigned long long* s, const HashFormat& F,
                                                         const TopNSpec& S) {
    constexpr unsigned long long kSign = 0x8000000000000000ull;
    const uint64_t cnt = group_count(s, F);
    unsigned long long k = cnt;   // row count (unsigned)
    if (S.val >= 0) {
        uint64_t lo;
        int64_t hi;
        group_value(s, F, S.val, S.kind, cnt, lo, hi);
        k = lo ^ kSign;
        if (S.kind != VK_MIN && S.kind != VK_MAX && S.func == TGP_AGG_AVG) {
            const double f = cnt ? i128_to_f64_rn(lo, hi) / static_cast<double>(cnt) : 0.0;
            const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(f));
            k = (u & kSign) ? ~u : (u | kSign);
        }
    }
    return S.desc ? ~k : k;
}

// A block takes kTopSlots slots at a time and reserves its groups' places with
// one atomic (one per warp made the counter the bound: 32K adds to one word).
constexpr int kTopPer = 8;
constexpr uint64_t kTopSlots = static_cast<uint64_t>(kTopThreads) * kTopPer;

__global__ void __launch_bounds__(kTopThreads) top_collect_kernel(const unsigned long long* htab, uint64_t nslots,
                                                                  uint32_t direct, const HashFormat F, const TopNSpec S,
                                                                  TopCand* out, TopState* st) {
    __shared__ uint32_t wsum[kTopThreads / 32];
    __shared__ unsigned long long base;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, cw = count_word(F);
    unsigned long long lo = ~0ull, hi = 0;
    for (uint64_t b = blockIdx.x * kTopSlots; b < nslots; b += gridDim.x * kTopSlots) {
        uint32_t occ = 0, cnt = 0;
#pragma unroll
        for (int j = 0; j < kTopPer; ++j) {
            const uint64_t i = b + static_cast<uint64_t>(j) * kTopThreads + threadIdx.x;
            const unsigned long long w = i < nslots ? htab[i * F.hstride + (direct ? cw : 0u)] : (direct ? 0ull : ~0ull);
            if (direct ? w != 0ull : w != ~0ull) {
                occ |= 1u << j;
                ++cnt;
            }
        }
        uint32_t incl = cnt;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= static_cast<uint32_t>(d)) incl += y;
        }
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        uint32_t before = incl - cnt, total = 0;
        for (uint32_t w = 0; w < kTopThreads / 32; ++w) {
            before += w < warp ? wsum[w] : 0u;
            total += wsum[w];
        }
        if (threadIdx.x == 0 && total) base = atomicAdd(&st->n, static_cast<unsigned long long>(total));
        __syncthreads();
        unsigned long long o = total ? base + before : 0ull;
#pragma unroll
        for (int j = 0; j < kTopPer; ++j) {
            if (!((occ >> j) & 1u)) continue;
            const uint64_t i = b + static_cast<uint64_t>(j) * kTopThreads + threadIdx.x;
            const unsigned long long* s = htab + i * F.hstride;
            TopCand c;
            c.order = order_word(s, F, S);
            c.key = direct ? i : s[0];
            c.slot = i;
            out[o++] = c;
            lo = min(lo, c.order);
            hi = max(hi, c.order);
        }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
        lo = min(lo, __shfl_down_sync(0xffffffffu, lo, d));
        hi = max(hi, __shfl_down_sync(0xffffffffu, hi, d));
    }
    if (lane == 0 && lo <= hi) {
        if (lo < *reinterpret_cast<volatile unsigned long long*>(&st->lo)) atomicMin(&st->lo, lo);
        if (hi > *reinterpret_cast<volatile unsigned long long*>(&st->hi)) atomicMax(&st->hi, hi);
    }
}

__device__ __forceinline__ uint32_t range_shift(unsigned long long span) {
    const int bits = span ? 64 - __clzll(static_cast<long long>(span)) : 0;
    return bits > 12 ? static_cast<uint32_t>(bits - 12) : 0u;
}

__global__ void __launch_bounds__(kTopThreads) top_hist_kernel(const TopCand* in, const TopState* st, uint32_t* hist) {
    __shared__ uint32_t h[kTopBuckets];
    for (uint32_t b = threadIdx.x; b < kTopBuckets; b += kTopThreads) h[b] = 0;
    __syncthreads();
    const unsigned long long n = st->n, lo = st->lo;
    const uint32_t shift = range_shift(st->hi - lo), by_key = st->by_key;
    const uint64_t step = static_cast<uint64_t>(gridDim.x) * kTopThreads;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * kTopThreads + threadIdx.x; i < n; i += step)
        atomicAdd(&h[((by_key ? in[i].key : in[i].order) - lo) >> shift], 1u);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < kTopBuckets; b += kTopThreads)
        if (h[b]) atomicAdd(hist + b, h[b]);
}

// The bucket holding the want-th candidate: every group of an earlier bucket is sure.
__global__ void __launch_bounds__(1024) top_bucket_kernel(uint32_t* hist, TopState* st) {
    __shared__ uint32_t wsum[32];
    const uint32_t t = threadIdx.x, lane = t & 31u;
    const unsigned long long want = st->want;
    uint32_t c[4], sum = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        c[j] = hist[4 * t + j];
        hist[4 * t + j] = 0;   // for the next narrowing
        sum += c[j];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= static_cast<uint32_t>(d)) incl += y;
    }
    if (lane == 31) wsum[t >> 5] = incl;
    __syncthreads();
    uint32_t before = incl - sum;
    for (uint32_t w = 0; w < (t >> 5); ++w) before += wsum[w];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (before < want && before + c[j] >= want) st->bucket = 4 * t + j;
        before += c[j];
    }
    if (t == 1023 && before < want) st->bucket = kTopBuckets;   // fewer groups than asked for: all are sure
}

__global__ void __launch_bounds__(kTopThreads) top_split_kernel(const TopCand* in, TopCand* next, TopCand* sure,
                                                                TopState* st) {
    const unsigned long long n = st->n, lo = st->lo;
    const uint32_t shift = range_shift(st->hi - lo), by_key = st->by_key, bucket = st->bucket;
    const uint64_t step = static_cast<uint64_t>(gridDim.x) * kTopThreads;
    // Whole warps walk the list, so one atomic per warp reserves its places.
    const uint64_t end = (n + 31) & ~31ull;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * kTopThreads + threadIdx.x; i < end; i += step) {
        TopCand c{};
        uint32_t b = kTopBuckets + 1;
        if (i < n) {
            c = in[i];
            b = static_cast<uint32_t>(((by_key ? c.key : c.order) - lo) >> shift);
        }
        if (b < bucket) sure[atomicAdd(&st->nsure, 1u)] = c;   // fewer than the limit in all
        const unsigned mask = __ballot_sync(0xffffffffu, b == bucket);
        if (mask == 0) continue;
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&st->nnext, static_cast<unsigned long long>(__popc(mask)));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (b == bucket) next[base + __popc(mask & ((1u << lane) - 1u))] = c;
    }
}

__device__ __forceinline__ bool cand_less(const TopCand& a, const TopCand& b) {
    return a.order != b.order ? a.order < b.order : a.key < b.key;
}

// Moves the state to the bucket's candidates; with few enough left, sorts
// them with the sure ones (bitonic, one block) and formats the first groups.
__global__ void __launch_bounds__(1024) top_finish_kernel(const unsigned long long* htab, const TopCand* next,
                                                          const TopCand* sure, TopState* st, const HashFormat F,
                                                          uint64_t limit, uint64_t* keys_out, tgp_agg_value* vals_out) {
    extern __shared__ __align__(16) uint8_t top_smem[];
    TopCand* v = reinterpret_cast<TopCand*>(top_smem);
    const uint32_t t = threadIdx.x;
    const unsigned long long nnext = st->nnext;
    const uint32_t nsure = st->nsure;
    const uint32_t shift = range_shift(st->hi - st->lo);
    const bool small = nnext + nsure <= kTopSort;
    __syncthreads();   // every thread has read the state
    if (!small) {
        if (t == 0) {
            if (st->total == 0) st->total = st->n;
            const unsigned long long base = st->lo + (static_cast<unsigned long long>(st->bucket) << shift);
            if (shift) {
                st->lo = base;
                st->hi = min(st->hi, base + ((1ull << shift) - 1ull));
            } else {
                st->by_key = 1;   // one ordering word left: the keys decide
                st->lo = 0;
                st->hi = st->key_hi;
            }
            st->want = limit - nsure;
            st->n = nnext;
            st->nnext = 0;
        }
        return;
    }
    const uint32_t m = static_cast<uint32_t>(nnext) + nsure;
    uint32_t p = 1;
    while (p < m) p <<= 1;
    for (uint32_t i = t; i < p; i += 1024) {
        if (i < m) v[i] = i < nsure ? sure[i] : next[i - nsure];
        else v[i] = TopCand{~0ull, ~0ull, ~0ull};
    }
    __syncthreads();
    for (uint32_t k = 2; k <= p; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = t; i < p; i += 1024) {
                const uint32_t x = i ^ j;
                if (x > i) {
                    const bool up = (i & k) == 0;
                    if (cand_less(v[x], v[i]) == up) {
                        const TopCand tmp = v[i];
                        v[i] = v[x];
                        v[x] = tmp;
                    }
                }
            }
            __syncthreads();
        }
    const uint64_t out = limit < m ? limit : m;
    for (uint64_t i = t; i < out; i += 1024) write_group(htab + v[i].slot * F.hstride, v[i].key, i, F, keys_out, vals_out);
    if (t == 0) {
        if (st->total == 0) st->total = st->n;
        st->done = 1;
    }
}

}  // namespace

// Scratch: the state, the histogram, then three candidate lists (two of
// max_groups, one of the sure groups).
size_t top_select_scratch(uint64_t max_groups) {
    return 256 + kTopBuckets * 4 + (2 * max_groups + kTopSort) * sizeof(TopCand);
}

cudaError_t top_select_begin(const unsigned long long* htab, uint64_t nslots, const HashFormat& F, bool direct,
                             const TopNSpec& S, uint64_t limit, uint32_t key_bits, void* scratch, int sms,
                             cudaStream_t st) {
    TopState* state = static_cast<TopState*>(scratch);
    uint32_t* hist = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(scratch) + 256);
    TopCand* a = reinterpret_cast<TopCand*>(hist + kTopBuckets);
    cudaError_t e = cudaMemsetAsync(hist, 0, kTopBuckets * 4, st);
    if (e != cudaSuccess) return e;
    top_init_kernel<<<1, 1, 0, st>>>(state, limit, key_bits >= 64 ? ~0ull : ((1ull << key_bits) - 1ull));
    uint64_t blocks = (nslots + kTopSlots - 1) / kTopSlots;
    if (blocks > static_cast<uint64_t>(sms) * 8) blocks = static_cast<uint64_t>(sms) * 8;
    if (blocks)
        top_collect_kernel<<<static_cast<unsigned>(blocks), kTopThreads, 0, st>>>(htab, nslots, direct ? 1u : 0u, F, S, a, state);
    return cudaGetLastError();
}

cudaError_t top_select_narrow(const unsigned long long* htab, uint64_t max_groups, uint32_t round, const HashFormat& F,
                              uint64_t limit, void* scratch, uint64_t* keys_out, tgp_agg_value* vals_out, int sms,
                              cudaStream_t st) {
    TopState* state = static_cast<TopState*>(scratch);
    uint32_t* hist = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(scratch) + 256);
    TopCand* a = reinterpret_cast<TopCand*>(hist + kTopBuckets);
    TopCand* b = a + max_groups;
    TopCand* sure = b + max_groups;
    const TopCand* in = round & 1u ? b : a;
    TopCand* next = round & 1u ? a : b;
    const unsigned grid = static_cast<unsigned>(sms) * 2;
    top_hist_kernel<<<grid, kTopThreads, 0, st>>>(in, state, hist);
    top_bucket_kernel<<<1, 1024, 0, st>>>(hist, state);
    top_split_kernel<<<grid, kTopThreads, 0, st>>>(in, next, sure, state);
    const size_t smem = kTopSort * sizeof(TopCand);
    const cudaError_t e = allow_dynamic_smem(reinterpret_cast<const void*>(&top_finish_kernel), smem);
    if (e != cudaSuccess) return e;
    top_finish_kernel<<<1, 1024, smem, st>>>(htab, next, sure, state, F, limit, keys_out, vals_out);
    return cudaGetLastError();
}

}  // namespace tgp
