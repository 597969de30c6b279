// join_stream.cu — streaming probe of a join through its payload array with
// grouped aggregation: the fixed join shape (sum(i64 * (k * i32 + a)), COUNT(*),
// groups from the build side; hash_join_with_keys + execute_grouped,
// src/engine/query_interpreter/join.rs:544-794, aggregate.rs:45-505) under at
// most four int32 probe-side leaves.
//
// What bounds a probe is the lookup: 32 lanes with 32 addresses take 32 tag
// cycles of the SM's L1, whatever the hit rate, so 60M payload lookups are 0.21
// ms on 148 SMs before a byte of the columns. Shared memory has no tags (32
// random words conflict about three deep), so the lookups go there:
//   * the whole payload array (one byte per key) when it fits beside the
//     tables, or
//   * one bit per key (does a build row match), and only rows that match read
//     their payload byte from global memory: half of them in a join whose
//     build side is filtered to half.
// The bits stay below 190 KB: past 195 KB of shared memory the SM's L1 shrinks
// to a size at which the streamed columns evict each other (60M rows x 1.5M
// keys: 0.25 -> 0.45 ms). B200, Zipf(0.8) keys, half the build side kept,
// kernel: 60M x 1.5M 0.258-0.335 -> 0.211-0.278 ms over 14 payload arrays (the
// matches' payload bytes bound it, and how fast they come depends on where in
// memory the array lies; most arrays: 0.258 -> 0.221-0.248); query without the
// build: 60M x 20K 0.233 -> 0.161 ms (16 bytes per row at 0.92 of the copy
// bandwidth), 8M x 1.5M 74 -> 54 us.
// One CTA of 1,024 threads per SM holds the table; a lane takes four
// consecutive rows of a 128-row chunk with 16-byte loads. Groups accumulate in per-warp
// tables of 32-bit limbs as in the scan engine (exact: the host proves every
// sum below 2^63). Distances from the smallest build key are taken in 32 bits:
// the host sends only build ranges within int32 here.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_common.cuh"
#include "plan.hpp"
#include "runtime.hpp"

namespace tgp {

namespace {

constexpr int kJsThreads = kStreamThreads;
constexpr int kJsWarps = kJsThreads / 32;
constexpr int kJsRows = 128;   // rows per warp chunk, four consecutive per lane

__device__ __forceinline__ uint4 js_load(const uint8_t* base, uint64_t byte_off) {
    return __ldcs(reinterpret_cast<const uint4*>(base + byte_off));
}

__device__ __forceinline__ uint32_t js_lds_u8(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

// BITS: the shared table is one bit per key (else the payload bytes).
template <bool BITS>
__global__ void __launch_bounds__(kJsThreads, 1) join_stream_kernel(const JoinStreamArgs A) {
    extern __shared__ __align__(16) uint8_t js_smem[];
    const uint32_t t = threadIdx.x, lane = t & 31u, wib = t >> 5;
    // Shared: the lookup table (16-byte words), then the limb tables.
    {
        uint4* dst = reinterpret_cast<uint4*>(js_smem);
        const uint4* src = reinterpret_cast<const uint4*>(A.table);
        for (uint32_t i = t; i < A.table_bytes / 16; i += kJsThreads) dst[i] = __ldg(src + i);
    }
    uint32_t* tabs = reinterpret_cast<uint32_t*>(js_smem + A.table_bytes);
    for (uint32_t i = t; i < A.copies * A.ngroups * 3u; i += kJsThreads) tabs[i] = 0;
    __syncthreads();
    const uint32_t look = smem_addr(js_smem);
    const uint32_t tab = smem_addr(tabs) + (wib & (A.copies - 1u)) * A.ngroups * 12u;
    const uint32_t range = A.krange;
    uint32_t selected = 0;

    // One row that passes the WHERE: its group (0xff = no match) is looked up
    // by `group`, and its value added by `add`.
    auto probe = [&](uint32_t rel) -> uint32_t {
        if (rel > range) return 0xffu;
        if (BITS) return (lds_u32(look + (rel >> 5) * 4u) >> (rel & 31u)) & 1u ? 0u : 0xffu;
        return js_lds_u8(look + rel);
    };
    auto add = [&](uint32_t g, int64_t price, uint32_t disc) {
        const uint32_t e = tab + g * 12u;
        const uint64_t v = static_cast<uint64_t>(price) * static_cast<uint64_t>(A.mul * disc + A.add);
        const uint32_t lo = static_cast<uint32_t>(v);
        red_add_shared(e, 1u);
        const uint32_t old = atom_add_shared(e + 4u, lo);
        const uint32_t hi = static_cast<uint32_t>(v >> 32) + ((old + lo < old) ? 1u : 0u);
        if (hi) red_add_shared(e + 8u, hi);
    };
    auto leaf = [&](uint32_t x, uint32_t i) { return ((x - A.leaf_lo[i]) <= A.leaf_sp[i] ? 1u : 0u) ^ ((A.leaf_neg >> i) & 1u); };

    const uint64_t warp = static_cast<uint64_t>(blockIdx.x) * kJsWarps + wib;
    const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * kJsWarps;
    const uint64_t nfull = A.nrows / kJsRows;
    // A chunk's lookups run one chunk ahead of its additions, its keys two
    // ahead: no step waits on a load it has just issued.
    struct Chunk {
        uint4 p0, p1, d;
        uint32_t g[4];
    };
    auto load_key = [&](uint64_t c) {
        return c < nfull ? js_load(A.key, (c * kJsRows + 4 * lane) * 4) : make_uint4(0u, 0u, 0u, 0u);
    };
    auto start = [&](uint64_t c, const uint4& key, Chunk& k) {
        const uint64_t r = c * kJsRows + 4 * lane;
        uint32_t sel = 15u;
        for (uint32_t i = 0; i < A.nleaf; ++i) {
            const uint4 x = js_load(A.leaf_col[i], r * 4);
            sel &= leaf(x.x, i) | (leaf(x.y, i) << 1) | (leaf(x.z, i) << 2) | (leaf(x.w, i) << 3);
        }
        k.p0 = js_load(A.col0, r * 8);
        k.p1 = js_load(A.col0, r * 8 + 16);
        k.d = js_load(A.col1, r * 4);
        selected += __popc(sel);
        const uint32_t rel[4] = {key.x - A.kmin, key.y - A.kmin, key.z - A.kmin, key.w - A.kmin};
#pragma unroll
        for (int e = 0; e < 4; ++e) k.g[e] = ((sel >> e) & 1u) ? probe(rel[e]) : 0xffu;
        if (BITS) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (k.g[e] == 0u) k.g[e] = __ldg(A.pay + rel[e]);
        }
    };
    auto finish = [&](const Chunk& k) {
        const uint32_t dd[4] = {k.d.x, k.d.y, k.d.z, k.d.w};
        const int64_t pp[4] = {static_cast<int64_t>((static_cast<uint64_t>(k.p0.y) << 32) | k.p0.x),
                               static_cast<int64_t>((static_cast<uint64_t>(k.p0.w) << 32) | k.p0.z),
                               static_cast<int64_t>((static_cast<uint64_t>(k.p1.y) << 32) | k.p1.x),
                               static_cast<int64_t>((static_cast<uint64_t>(k.p1.w) << 32) | k.p1.z)};
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (k.g[e] != 0xffu) add(k.g[e], pp[e], dd[e]);
    };
    LineAhead lines;
    lines.column(lane, A.key, 512);
    lines.column(lane, A.col0, 1024);
    lines.column(lane, A.col1, 512);
    for (uint32_t i = 0; i < A.nleaf; ++i) lines.column(lane, A.leaf_col[i], 512);
    if (warp < nfull) {
        Chunk a, b;
        uint4 key = load_key(warp), ahead = load_key(warp + nwarps);
        start(warp, key, a);
        for (uint64_t c = warp;; c += 2 * nwarps) {
            const uint64_t c1 = c + nwarps, c2 = c1 + nwarps;
            key = ahead;
            if (c2 < nfull) lines.fetch(c2);
            if (c2 + nwarps < nfull) lines.fetch(c2 + nwarps);
            ahead = load_key(c2);
            if (c1 < nfull) start(c1, key, b);
            finish(a);
            if (c1 >= nfull) break;
            key = ahead;
            ahead = load_key(c2 + nwarps);
            if (c2 < nfull) start(c2, key, a);
            finish(b);
            if (c2 >= nfull) break;
        }
    }
    // The partial last chunk, one row per lane of one warp.
    if (warp == nfull % nwarps) {
        for (uint64_t r = nfull * kJsRows + lane; r < A.nrows; r += 32) {
            uint32_t m = 1u;
            for (uint32_t i = 0; i < A.nleaf; ++i) m &= leaf(reinterpret_cast<const uint32_t*>(A.leaf_col[i])[r], i);
            if (!m) continue;
            ++selected;
            const uint32_t rel = reinterpret_cast<const uint32_t*>(A.key)[r] - A.kmin;
            uint32_t g = probe(rel);
            if (BITS && g == 0u) g = __ldg(A.pay + rel);
            if (g != 0xffu)
                add(g, reinterpret_cast<const long long*>(A.col0)[r], reinterpret_cast<const uint32_t*>(A.col1)[r]);
        }
    }
    __syncwarp();
    selected = __reduce_add_sync(0xffffffffu, selected);
    if (lane == 0 && selected) atomicAdd(A.counters, static_cast<unsigned long long>(selected));
    __syncthreads();
    // Merge: thread i sums (group, slot) pair i over the copies.
    for (uint32_t i = t; i < A.ngroups * 2u; i += kJsThreads) {
        const uint32_t g = i >> 1, v = i & 1u;
        unsigned long long sum = 0;
        for (uint32_t c = 0; c < A.copies; ++c) {
            const uint32_t* e = tabs + (static_cast<size_t>(c) * A.ngroups + g) * 3u;
            if (v == 0) sum += e[0];
            else sum += (static_cast<unsigned long long>(static_cast<long long>(static_cast<int32_t>(e[2]))) << 32) + e[1];
        }
        if (sum) atomicAdd(A.acc + 2ull * i, sum);
    }
    finish_result(A.out, t, kJsThreads, [] { __syncthreads(); });
}

// One bit per payload entry: set where a build row matches (word w holds
// entries 32w .. 32w + 31; whole 16-byte words are written).
__global__ void pay_bits_kernel(const uint8_t* pay, uint64_t entries, uint32_t* bits, uint64_t nwords) {
    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (static_cast<uint64_t>(gridDim.x) * blockDim.x) >> 5;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t w = warp; w < nwords; w += nwarps) {
        const uint64_t e = w * 32 + lane;
        const uint32_t m = __ballot_sync(0xffffffffu, e < entries && pay[e] != 0xffu);
        if (lane == 0) bits[w] = m;
    }
}

}  // namespace

uint64_t pay_bits_words(uint64_t entries) { return ((entries + 127) / 128) * 4; }

cudaError_t launch_pay_bits(const uint8_t* pay, uint64_t entries, uint32_t* bits, int sms, cudaStream_t st) {
    const uint64_t words = pay_bits_words(entries);
    const uint64_t blocks = std::min<uint64_t>((words * 32 + 255) / 256, static_cast<uint64_t>(sms) * 8);
    pay_bits_kernel<<<static_cast<unsigned>(blocks), 256, 0, st>>>(pay, entries, bits, words);
    return cudaGetLastError();
}

cudaError_t launch_join_stream(const JoinStreamArgs& A, bool bits, int grid, cudaStream_t st) {
    const void* f = bits ? reinterpret_cast<const void*>(&join_stream_kernel<true>)
                         : reinterpret_cast<const void*>(&join_stream_kernel<false>);
    const size_t smem = join_stream_smem(A.table_bytes, A.copies, A.ngroups);
    const cudaError_t e = allow_dynamic_smem(f, smem);
    if (e != cudaSuccess) return e;
    JoinStreamArgs a = A;
    void* args[] = {&a};
    return cudaLaunchKernel(f, dim3(static_cast<unsigned>(grid)), dim3(kJsThreads), args, smem, st);
}

}  // namespace tgp
