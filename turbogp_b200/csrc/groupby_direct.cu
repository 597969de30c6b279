// groupby_direct.cu — streaming GROUP BY kernels, rows read straight from
// HBM without the scan engine's stage ring: (1) an unfiltered GROUP BY of one
// key over a moderate range (the reference's try_accumulator_grouped,
// aggregate.rs / accum_grouped.rs, on its high-cardinality inputs) into
// one-word direct slots; (2) GROUP BY a sparse key into hash slots; (3) the
// TPC-H Q1 shape (both further below).
//
// A slot per key value (key - min < 2^27) holds (row count << shift) + the
// sum of (value - bias) over its rows; the host proved that neither field can
// reach the other. Rows stream straight from HBM with coalesced vector loads
// (evict-first, so the slot table stays in L2), hot keys add into a per-CTA
// shared table with native 32-bit atomics (two probes, claimed first come),
// and every other row is one non-returning 64-bit add to its key's slot.
// There is no stage ring: with no predicate and one key the rows need no
// staging, and the loads of a thread's next rows are in flight while it
// updates the current ones.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "device_common.cuh"
#include "plan.hpp"
#include "runtime.hpp"

namespace tgp {

namespace {

constexpr int kDgThreads = kDirectThreads;
// Two CTAs per SM (64 registers, no spills) with two warp chunks' loads in
// flight measured faster on B200 (20M rows, 10M key range, Zipf(1.1)) than
// three CTAs with one or two chunks (40 registers) and two CTAs with three.
constexpr int kDgMinBlocks = 2;   // CTAs per SM the register budget is set for
constexpr int kDgUnroll = 2;      // warp chunks whose loads are in flight at once
constexpr uint32_t kDgEmpty = 0xffffffffu;
constexpr uint32_t kDgProbes = 2;
constexpr int kDgRows = 128;   // rows per warp chunk: lane l holds rows 2l, 2l + 1, 64 + 2l, 65 + 2l

// Two consecutive cells of a column at row `r` (even), sign- or zero-extended
// as the column type says (to T: a key's low word, or a value in its own
// width); streaming loads (evict first in L1 and L2).
template <uint32_t DT, typename T>
__device__ __forceinline__ void load_pair(const uint8_t* base, uint64_t r, T& a, T& b) {
    if constexpr (DT == DT_I64 || DT == DT_U64) {
        const longlong2 v = __ldcs(reinterpret_cast<const longlong2*>(base) + r / 2);
        a = static_cast<T>(v.x);
        b = static_cast<T>(v.y);
    } else if constexpr (DT == DT_I32) {
        const int2 v = __ldcs(reinterpret_cast<const int2*>(base) + r / 2);
        a = static_cast<T>(v.x);
        b = static_cast<T>(v.y);
    } else {  // DT_U8
        const uint16_t v = __ldcs(reinterpret_cast<const unsigned short*>(base) + r / 2);
        a = static_cast<T>(v & 0xffu);
        b = static_cast<T>(v >> 8);
    }
}

template <uint32_t DT>
__device__ __forceinline__ int64_t load_one(const uint8_t* base, uint64_t r) {
    if constexpr (DT == DT_I64 || DT == DT_U64) return reinterpret_cast<const long long*>(base)[r];
    else if constexpr (DT == DT_I32) return reinterpret_cast<const int32_t*>(base)[r];
    else return base[r];
}

struct DgTable {
    uint32_t* keys;
    uint32_t* cnt;
    int32_t* sums;
};

// Adds one row (slot `key`, value argument `x`) to its claimed shared slot
// `h` (shared-table hit).
template <bool HASV>
__device__ __forceinline__ void dg_hit(const DgTable& T, uint32_t h, int64_t x) {
    atomicAdd(&T.cnt[h], 1u);
    if constexpr (HASV) atomicAdd(&T.sums[h], static_cast<int32_t>(x));
}

// Adds one row to the key's global slot.
__device__ __forceinline__ void dg_global(const DirectGroupArgs& A, uint32_t key, int64_t x) {
    if (key > A.last) {
        atomicOr(A.err, kErrHashFull);
        return;
    }
    atomicAdd(A.slots + key, A.one + static_cast<unsigned long long>(x));
}

// Adds the N rows (keys, value arguments) of a thread. Shared table: the
// first-probe slot loads of all N rows are issued together, then each row
// adds to its slot (the common case once the hot keys hold slots) or claims
// an empty one; the rows left take their second probes the same way; the
// rest go to their global slots. A stale slot read is harmless: a claimed
// slot never changes key, and an empty one is claimed by compare-and-swap.
template <int N, bool HASV>
__device__ __forceinline__ void dg_rows(const DirectGroupArgs& A, const DgTable& T, const uint32_t (&key)[N],
                                        const int64_t (&x)[N]) {
    uint32_t glob = (1u << N) - 1u;
    if (A.hs) {
        uint32_t h[N], k[N];
#pragma unroll
        for (int r = 0; r < N; ++r) {
            h[r] = (key[r] * 0x9E3779B1u) >> A.hs_shift;
            k[r] = *reinterpret_cast<volatile uint32_t*>(&T.keys[h[r]]);
        }
#pragma unroll
        for (uint32_t n = 0; n < kDgProbes; ++n) {
            if (n) {
#pragma unroll
                for (int r = 0; r < N; ++r) {
                    if (!((glob >> r) & 1u)) continue;
                    h[r] = (h[r] + 1) & (A.hs - 1);
                    k[r] = *reinterpret_cast<volatile uint32_t*>(&T.keys[h[r]]);
                }
            }
#pragma unroll
            for (int r = 0; r < N; ++r) {
                if (!((glob >> r) & 1u)) continue;
                uint32_t kk = k[r];
                if (kk == kDgEmpty) kk = atomicCAS(&T.keys[h[r]], kDgEmpty, key[r]);
                if (kk == kDgEmpty || kk == key[r]) {
                    dg_hit<HASV>(T, h[r], x[r]);
                    glob &= ~(1u << r);
                }
            }
        }
    }
#pragma unroll
    for (int r = 0; r < N; ++r)
        if ((glob >> r) & 1u) dg_global(A, key[r], x[r]);
}

template <uint32_t KDT, uint32_t VDT>
__global__ void __launch_bounds__(kDgThreads, kDgMinBlocks) direct_group_kernel(const DirectGroupArgs A) {
    constexpr bool HASV = VDT != 0;
    using VT = std::conditional_t<VDT == DT_I64 || VDT == DT_U64, int64_t, int32_t>;
    extern __shared__ __align__(16) uint8_t dg_smem[];
    DgTable T;
    T.keys = reinterpret_cast<uint32_t*>(dg_smem);
    T.cnt = T.keys + A.hs;
    T.sums = reinterpret_cast<int32_t*>(T.cnt + A.hs);
    for (uint32_t i = threadIdx.x; i < A.hs; i += kDgThreads) {
        T.keys[i] = kDgEmpty;
        T.cnt[i] = 0;
        if (HASV) T.sums[i] = 0;
    }
    __syncthreads();

    const uint32_t kmin = static_cast<uint32_t>(A.kmin);
    auto value_of = [&](int64_t v) -> int64_t {
        const int64_t a = A.ident ? v : static_cast<int64_t>(static_cast<uint64_t>(A.mul) * static_cast<uint64_t>(v) +
                                                              static_cast<uint64_t>(A.add));
        return A.nz ? (a != 0 ? 1 : 0) : a;
    };

    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * kDgThreads + threadIdx.x) >> 5;
    const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * (kDgThreads / 32);
    const uint64_t nfull = A.nrows / kDgRows;
    // Full chunks, kDgUnroll per step: the loads of all of them are issued
    // before the first chunk's rows are added. (An L2 prefetch of the next
    // step's lines measured slower here, 154 -> 160 us: the shared table's pipe
    // is the bound.)
    uint64_t c = warp;
    for (; c + (kDgUnroll - 1) * nwarps < nfull; c += kDgUnroll * nwarps) {
        uint32_t k[kDgUnroll][4];
        VT v[kDgUnroll][4];
#pragma unroll
        for (int u = 0; u < kDgUnroll; ++u) {
            const uint64_t b = (c + u * nwarps) * kDgRows + 2 * lane;
            load_pair<KDT>(A.key, b, k[u][0], k[u][1]);
            load_pair<KDT>(A.key, b + 64, k[u][2], k[u][3]);
            if constexpr (HASV) {
                load_pair<VDT>(A.val, b, v[u][0], v[u][1]);
                load_pair<VDT>(A.val, b + 64, v[u][2], v[u][3]);
            }
        }
#pragma unroll
        for (int u = 0; u < kDgUnroll; ++u) {
            uint32_t key[4];
            int64_t x[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                key[r] = k[u][r] - kmin;
                x[r] = HASV ? value_of(v[u][r]) : 0;
            }
            dg_rows<4, HASV>(A, T, key, x);
        }
    }
    for (; c < nfull; c += nwarps) {
        const uint64_t b = c * kDgRows + 2 * lane;
        uint32_t k[4];
        VT v[4];
        load_pair<KDT>(A.key, b, k[0], k[1]);
        load_pair<KDT>(A.key, b + 64, k[2], k[3]);
        if constexpr (HASV) {
            load_pair<VDT>(A.val, b, v[0], v[1]);
            load_pair<VDT>(A.val, b + 64, v[2], v[3]);
        }
        uint32_t key[4];
        int64_t x[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            key[r] = k[r] - kmin;
            x[r] = HASV ? value_of(v[r]) : 0;
        }
        dg_rows<4, HASV>(A, T, key, x);
    }
    // The partial last chunk: the warp next in turn takes it, one row per
    // lane (no warp-wide step inside, lanes may leave the loop early).
    if (warp == nfull % nwarps) {
        for (uint64_t r = nfull * kDgRows + lane; r < A.nrows; r += 32) {
            const int64_t x[1] = {HASV ? value_of(load_one<VDT>(A.val, r)) : 0};
            const uint32_t key[1] = {static_cast<uint32_t>(load_one<KDT>(A.key, r)) - kmin};
            dg_rows<1, HASV>(A, T, key, x);
        }
    }
    __syncthreads();
    // Merge the shared table: one add per occupied slot.
    for (uint32_t i = threadIdx.x; i < A.hs; i += kDgThreads) {
        const uint32_t key = T.keys[i];
        if (key == kDgEmpty) continue;
        if (key > A.last) {
            atomicOr(A.err, kErrHashFull);
            continue;
        }
        const uint64_t n = T.cnt[i];
        const int64_t s = HASV ? static_cast<int64_t>(T.sums[i]) : 0;
        atomicAdd(A.slots + key, (n << A.shift) + (static_cast<unsigned long long>(s) - n * static_cast<uint64_t>(A.bias)));
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(A.counters, static_cast<unsigned long long>(A.nrows));
}

template <uint32_t KDT, uint32_t VDT>
const void* dg_ptr() {
    return reinterpret_cast<const void*>(&direct_group_kernel<KDT, VDT>);
}

const void* dg_kernel(uint32_t kdt, uint32_t vdt) {
    const bool k64 = kdt == DT_I64 || kdt == DT_U64;
    if (!k64 && kdt != DT_I32) return nullptr;
    switch (vdt) {
        case 0: return k64 ? dg_ptr<DT_I64, 0>() : dg_ptr<DT_I32, 0>();
        case DT_U8: return k64 ? dg_ptr<DT_I64, DT_U8>() : dg_ptr<DT_I32, DT_U8>();
        case DT_I32: return k64 ? dg_ptr<DT_I64, DT_I32>() : dg_ptr<DT_I32, DT_I32>();
        case DT_I64:
        case DT_U64: return k64 ? dg_ptr<DT_I64, DT_I64>() : dg_ptr<DT_I32, DT_I64>();
        default: return nullptr;
    }
}

// ---------------------------------------------------------------------------
// GROUP BY one key too sparse for a slot per value, under at most four int32
// predicate leaves, with COUNT(*) and at most one SUM / COUNT(col): 16-byte
// hash slots [key][(count << shift) + sum of (value - bias)]. As above, rows
// stream in chunks with two chunks' loads in flight, and hot keys add into a
// per-CTA shared table (64-bit keys, direct-mapped: 4,096 slots, 64 KB).
// Rows that miss it wait in their warp's queue until 64 are there; a drain
// probes the global table once for each (two per lane), adds one word where the
// slot is the key's, and queues the others again at their next slot. Probing
// straight away kept the whole warp on the table's latency for the few lanes
// with a miss, as long as the longest chain of them: 880 instructions per
// 128-row chunk, 570 with the queue. 20M rows, nine tenths selected, over 1M
// Zipf(1.1) ids: 304 us, 246-251 us with the queue (the scan pipeline on the
// same table 468 us). Half the rows miss the shared table; what bounds the
// kernel is the uncoalesced accesses they make (two per miss, one address per
// lane) beside the shared lookups.
// ---------------------------------------------------------------------------
constexpr uint32_t kHgSlots = 4096;   // a multiple of 4 * kDgThreads
constexpr unsigned long long kHgEmpty = ~0ull;
constexpr uint32_t kHgQueue = 192;   // 63 rows left by a drain and a chunk's 128

struct HgTable {
    unsigned long long* keys;
    uint32_t* cnt;
    int32_t* sums;
};

// Whether slot h is past the probe bound of `key`: raises kErrHashFull (the
// host sizes the table so that it means a bad estimate, and runs the query
// again).
__device__ __forceinline__ bool hg_gives_up(const HashGroupArgs& A, uint32_t h, unsigned long long key) {
    if (((h - static_cast<uint32_t>(hash_slot(key, A.log2))) & A.mask) < A.probes) return false;
    atomicOr(A.err, kErrHashFull);
    return true;
}

// Adds (key, word) to the global table (rows outside the chunks, merges). A
// slot never changes key once claimed, so reading one as empty too late only
// costs the compare-and-swap.
__device__ __forceinline__ void hg_global(const HashGroupArgs& A, unsigned long long key, unsigned long long word) {
    uint32_t h = static_cast<uint32_t>(hash_slot(key, A.log2));
    for (uint32_t n = 0; n < A.probes; ++n) {
        unsigned long long* s = A.slots + 2ull * h;
        unsigned long long seen = __ldcg(s);
        if (seen == kHgEmpty) seen = atomicCAS(s, kHgEmpty, key);
        if (seen == kHgEmpty || seen == key) {
            atomicAdd(s + 1, word);
            return;
        }
        if ((n & 31u) == 31u && (*reinterpret_cast<volatile uint32_t*>(A.err) & kErrHashFull)) return;
        h = (h + 1) & A.mask;
    }
    atomicOr(A.err, kErrHashFull);
}

// Adds the selected rows to the shared table; returns those whose slot another
// key holds. Every CTA hashes with a multiplier of its own: with one for all,
// two hot keys that collide do so in every CTA, and the loser's rows (a percent
// of the table) queue up on one word of L2.
template <int N, bool HASV>
__device__ __forceinline__ uint32_t hg_rows(const HashGroupArgs& A, const HgTable& T, uint32_t mult, uint32_t sel,
                                            const unsigned long long (&key)[N], const int64_t (&x)[N]) {
    if (!A.hs) return sel;
    uint32_t h[N], miss = sel;
    unsigned long long k[N];
#pragma unroll
    for (int r = 0; r < N; ++r) {
        h[r] = ((static_cast<uint32_t>(key[r]) ^ (static_cast<uint32_t>(key[r] >> 32) * 0x85EBCA6Bu)) * mult) >>
               (32u - A.hs_log2);
        k[r] = *reinterpret_cast<volatile unsigned long long*>(&T.keys[h[r]]);
    }
#pragma unroll
    for (int r = 0; r < N; ++r) {
        if (!((sel >> r) & 1u)) continue;
        unsigned long long kk = k[r];
        if (kk == kHgEmpty) kk = atomicCAS(&T.keys[h[r]], kHgEmpty, key[r]);
        if (kk == kHgEmpty || kk == key[r]) {
            atomicAdd(&T.cnt[h[r]], 1u);
            if constexpr (HASV) atomicAdd(&T.sums[h[r]], static_cast<int32_t>(x[r]));
            miss &= ~(1u << r);
        }
    }
    return miss;
}

template <uint32_t KDT, uint32_t VDT>
__global__ void __launch_bounds__(kDgThreads, kDgMinBlocks) hash_group_kernel(const HashGroupArgs A) {
    constexpr bool HASV = VDT != 0;
    using KT = std::conditional_t<KDT == DT_I64 || KDT == DT_U64, int64_t, int32_t>;
    using VT = std::conditional_t<VDT == DT_I64 || VDT == DT_U64, int64_t, int32_t>;
    extern __shared__ __align__(16) uint8_t hg_smem[];
    HgTable T;
    T.keys = reinterpret_cast<unsigned long long*>(hg_smem);
    T.cnt = reinterpret_cast<uint32_t*>(T.keys + A.hs);
    T.sums = reinterpret_cast<int32_t*>(T.cnt + A.hs);
    const uint32_t mult = 0x9E3779B1u * (2u * blockIdx.x + 1u);
    // This warp's queue: keys, slots to probe, value arguments (those of a
    // launch with the shared table fit 32 bits; 16 bytes per row keep two
    // CTAs on an SM).
    constexpr uint32_t kWarps = kDgThreads / 32;
    const uint32_t wib = threadIdx.x >> 5;
    unsigned long long* queue = reinterpret_cast<unsigned long long*>(T.sums + A.hs);
    unsigned long long* qkey = queue + wib * kHgQueue;
    uint32_t* qslot = reinterpret_cast<uint32_t*>(queue + kWarps * kHgQueue) + wib * kHgQueue;
    uint32_t* qx = reinterpret_cast<uint32_t*>(queue + kWarps * kHgQueue) + (kWarps + wib) * kHgQueue;
    int32_t* qxh = reinterpret_cast<int32_t*>(queue + 2 * kWarps * kHgQueue) + wib * kHgQueue;   // hs == 0 only
    auto queued_x = [&](uint32_t at) -> int64_t {
        if (A.hs) return static_cast<int32_t>(qx[at]);
        return static_cast<int64_t>((static_cast<uint64_t>(static_cast<uint32_t>(qxh[at])) << 32) | qx[at]);
    };
    uint32_t queued = 0;
    for (uint32_t i = threadIdx.x; i < A.hs; i += kDgThreads) {
        T.keys[i] = kHgEmpty;
        T.cnt[i] = 0;
        if (HASV) T.sums[i] = 0;
    }
    __syncthreads();

    auto value_of = [&](int64_t v) -> int64_t {
        const int64_t a = A.ident ? v : static_cast<int64_t>(static_cast<uint64_t>(A.mul) * static_cast<uint64_t>(v) +
                                                              static_cast<uint64_t>(A.add));
        return A.nz ? (a != 0 ? 1 : 0) : a;
    };
    auto rel = [&](KT k) { return static_cast<unsigned long long>(static_cast<int64_t>(k)) - static_cast<unsigned long long>(A.kmin); };
    auto leaf = [&](uint32_t c, uint32_t i) { return ((c - A.leaf_lo[i]) <= A.leaf_sp[i] ? 1u : 0u) ^ ((A.leaf_neg >> i) & 1u); };

    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * kDgThreads + threadIdx.x) >> 5;
    const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * (kDgThreads / 32);
    const uint64_t nfull = A.nrows / kDgRows;
    uint32_t selected = 0;
    // Rows 2l, 2l + 1, 64 + 2l, 65 + 2l of a chunk: cells, then the selection.
    auto load_chunk = [&](uint64_t c, KT (&k)[4], VT (&v)[4], uint32_t& sel) {
        const uint64_t b = c * kDgRows + 2 * lane;
        load_pair<KDT>(A.key, b, k[0], k[1]);
        load_pair<KDT>(A.key, b + 64, k[2], k[3]);
        if constexpr (HASV) {
            load_pair<VDT>(A.val, b, v[0], v[1]);
            load_pair<VDT>(A.val, b + 64, v[2], v[3]);
        }
        sel = 15u;
        for (uint32_t i = 0; i < A.nleaf; ++i) {
            uint32_t x[4];
            load_pair<DT_I32>(A.leaf_col[i], b, x[0], x[1]);
            load_pair<DT_I32>(A.leaf_col[i], b + 64, x[2], x[3]);
            sel &= leaf(x[0], i) | (leaf(x[1], i) << 1) | (leaf(x[2], i) << 2) | (leaf(x[3], i) << 3);
        }
    };
    // Queues the rows of the lanes with `m` (every lane calls).
    auto push = [&](bool m, unsigned long long key, int64_t x, uint32_t slot) {
        const uint32_t all = __ballot_sync(0xffffffffu, m);
        if (m) {
            const uint32_t at = queued + __popc(all & ((1u << lane) - 1u));
            qkey[at] = key;
            qslot[at] = slot;
            qx[at] = static_cast<uint32_t>(x);
            if (!A.hs) qxh[at] = static_cast<int32_t>(x >> 32);
        }
        queued += __popc(all);
    };
    auto add_chunk = [&](const KT (&k)[4], const VT (&v)[4], uint32_t sel) {
        unsigned long long key[4];
        int64_t x[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            key[r] = rel(k[r]);
            x[r] = HASV ? value_of(v[r]) : 0;
        }
        selected += __popc(sel);
        const uint32_t miss = hg_rows<4, HASV>(A, T, mult, sel, key, x);
#pragma unroll
        for (int r = 0; r < 4; ++r)
            push((miss >> r) & 1u, key[r], x[r], static_cast<uint32_t>(hash_slot(key[r], A.log2)));
        __syncwarp();
        while (queued >= 64) {
            queued -= 64;
            unsigned long long dk[2], seen[2];
            int64_t dx[2];
            uint32_t dh[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const uint32_t at = queued + 32 * u + lane;
                dk[u] = qkey[at];
                dx[u] = queued_x(at);
                dh[u] = qslot[at];
                seen[u] = __ldcg(A.slots + 2ull * dh[u]);
            }
            __syncwarp();
            // Claims of both rows are in flight together.
#pragma unroll
            for (int u = 0; u < 2; ++u)
                if (seen[u] == kHgEmpty) {
                    seen[u] = atomicCAS(A.slots + 2ull * dh[u], kHgEmpty, dk[u]);
                    if (seen[u] == kHgEmpty) seen[u] = dk[u];
                }
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                bool again = seen[u] != dk[u];
                if (!again) atomicAdd(A.slots + 2ull * dh[u] + 1, A.one + static_cast<unsigned long long>(dx[u]));
                const uint32_t next = (dh[u] + 1) & A.mask;
                if (again && hg_gives_up(A, next, dk[u])) again = false;
                push(again, dk[u], dx[u], next);
            }
            __syncwarp();
        }
    };
    // The next chunk's loads are in flight while a chunk's rows are added.
    LineAhead ahead;
    ahead.column(lane, A.key, KDT == DT_I32 ? 512u : 1024u);
    if (HASV) ahead.column(lane, A.val, VDT == DT_U8 ? 128u : VDT == DT_I32 ? 512u : 1024u);
    for (uint32_t i = 0; i < A.nleaf; ++i) ahead.column(lane, A.leaf_col[i], 512u);
    if (warp < nfull) {
        KT ka[4], kb[4];
        VT va[4], vb[4];
        uint32_t sa, sb;
        load_chunk(warp, ka, va, sa);
        for (uint64_t c = warp; c < nfull; c += 2 * nwarps) {
            const bool more = c + nwarps < nfull;
            if (c + 2 * nwarps < nfull) ahead.fetch(c + 2 * nwarps);
            if (c + 3 * nwarps < nfull) ahead.fetch(c + 3 * nwarps);
            if (more) load_chunk(c + nwarps, kb, vb, sb);
            add_chunk(ka, va, sa);
            if (!more) break;
            if (c + 2 * nwarps < nfull) load_chunk(c + 2 * nwarps, ka, va, sa);
            add_chunk(kb, vb, sb);
        }
    }
    // The partial last chunk, one row per lane of one warp.
    if (warp == nfull % nwarps) {
        for (uint64_t r = nfull * kDgRows + lane; r < A.nrows; r += 32) {
            uint32_t m = 1u;
            for (uint32_t i = 0; i < A.nleaf; ++i) m &= leaf(reinterpret_cast<const uint32_t*>(A.leaf_col[i])[r], i);
            if (!m) continue;
            ++selected;
            const int64_t x[1] = {HASV ? value_of(load_one<VDT>(A.val, r)) : 0};
            const unsigned long long key[1] = {rel(static_cast<KT>(load_one<KDT>(A.key, r)))};
            if (hg_rows<1, HASV>(A, T, mult, 1u, key, x)) hg_global(A, key[0], A.one + static_cast<unsigned long long>(x[0]));
        }
    }
    __syncwarp();
    for (uint32_t i = lane; i < queued; i += 32) {
        hg_global(A, qkey[i], A.one + static_cast<unsigned long long>(queued_x(i)));
    }
    __syncwarp();
    selected = __reduce_add_sync(0xffffffffu, selected);
    if (lane == 0 && selected) atomicAdd(A.counters, static_cast<unsigned long long>(selected));
    __syncthreads();
    // Merge the shared table: one add per occupied slot, the first probes of a
    // thread's slots in flight together.
    constexpr int kPer = 4;
    for (uint32_t i = threadIdx.x; i < A.hs; i += kPer * kDgThreads) {
        unsigned long long key[kPer], seen[kPer];
        uint32_t h[kPer];
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            key[u] = T.keys[i + u * kDgThreads];
            h[u] = static_cast<uint32_t>(hash_slot(key[u], A.log2));
            seen[u] = __ldcg(A.slots + 2ull * h[u]);
        }
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            if (key[u] == kHgEmpty) continue;
            const uint32_t at = i + u * kDgThreads;
            const uint64_t n = T.cnt[at];
            const int64_t s = HASV ? static_cast<int64_t>(T.sums[at]) : 0;
            const unsigned long long word = (n << A.shift) + (static_cast<unsigned long long>(s) - n * static_cast<uint64_t>(A.bias));
            if (seen[u] == key[u]) atomicAdd(A.slots + 2ull * h[u] + 1, word);
            else hg_global(A, key[u], word);
        }
    }
}

template <uint32_t KDT, uint32_t VDT>
const void* hg_ptr() {
    return reinterpret_cast<const void*>(&hash_group_kernel<KDT, VDT>);
}

const void* hg_kernel(uint32_t kdt, uint32_t vdt) {
    const bool k64 = kdt == DT_I64 || kdt == DT_U64;
    if (!k64 && kdt != DT_I32) return nullptr;
    switch (vdt) {
        case 0: return k64 ? hg_ptr<DT_I64, 0>() : hg_ptr<DT_I32, 0>();
        case DT_U8: return k64 ? hg_ptr<DT_I64, DT_U8>() : hg_ptr<DT_I32, DT_U8>();
        case DT_I32: return k64 ? hg_ptr<DT_I64, DT_I32>() : hg_ptr<DT_I32, DT_I32>();
        case DT_I64:
        case DT_U64: return k64 ? hg_ptr<DT_I64, DT_I64>() : hg_ptr<DT_I32, DT_I64>();
        default: return nullptr;
    }
}

// ---------------------------------------------------------------------------
// The TPC-H Q1 shape (execute_grouped, aggregate.rs:45-505, on a predicate of
// at most four int32 leaves): GROUP BY two u8 keys, COUNT(*), sum(i32),
// sum(i64), sum(i64 * (k - i32)), sum(i64 * (k - i32) * (k + i32)), every
// sum proven to fit int64. Rows stream from HBM with coalesced loads (four
// consecutive rows per lane); each thread keeps private partials (u32 row
// counts, int64 sums) in shared memory, updated by plain read-modify-writes,
// with no stage ring, so two CTAs of 512 threads fit an SM; at the end each
// (group, value) is summed over the CTA's threads by one warp and added to
// the query's accumulator with one 64-bit atomic.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint4 ldcs4(const uint8_t* base, uint64_t byte_off) {
    return __ldcs(reinterpret_cast<const uint4*>(base + byte_off));
}

__global__ void __launch_bounds__(kDgThreads, 2) q1_group_kernel(const Q1Args A) {
    extern __shared__ __align__(16) uint8_t q1_smem[];
    constexpr uint32_t NT = kDgThreads;
    const uint32_t t = threadIdx.x, lane = t & 31u;
    uint32_t* cnt = reinterpret_cast<uint32_t*>(q1_smem);                         // [g][t]
    long long* val = reinterpret_cast<long long*>(q1_smem + A.ngroups * NT * 4);  // [g][v][t]
    for (uint32_t g = 0; g < A.ngroups; ++g) cnt[g * NT + t] = 0;
    for (uint32_t i = 0; i < A.ngroups * 4; ++i) val[i * NT + t] = 0;

    // One row: its selection mask (all ones or 0), group and column cells.
    auto add_row = [&](uint32_t sel, uint32_t g, uint32_t qty, int64_t price, uint32_t disc, uint32_t tax) {
        const uint64_t sm = static_cast<uint64_t>(static_cast<int64_t>(static_cast<int32_t>(sel)));
        const uint64_t v1 = static_cast<uint64_t>(A.mul[0] * qty + A.add[0]) & sm;
        const uint64_t v2 = static_cast<uint64_t>(price) & sm;
        const uint64_t v3 = v2 * static_cast<uint64_t>(A.mul[1] * disc + A.add[1]);
        const uint64_t v4 = v3 * static_cast<uint64_t>(A.mul[2] * tax + A.add[2]);
        cnt[g * NT + t] += sel & 1u;
        long long* w = val + static_cast<size_t>(g) * 4 * NT + t;
        w[0] += static_cast<long long>(v1);
        w[NT] += static_cast<long long>(v2);
        w[2 * NT] += static_cast<long long>(v3);
        w[3 * NT] += static_cast<long long>(v4);
    };
    auto leaf = [&](uint32_t x, uint32_t i) { return ((x - A.leaf_lo[i]) <= A.leaf_sp[i] ? 1u : 0u) ^ ((A.leaf_neg >> i) & 1u); };

    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * NT + t) >> 5;
    const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * (NT / 32);
    const uint64_t nfull = A.nrows / kDgRows;
    // The next chunk's lines are asked for before this one's rows are added
    // (no registers are left to hold a second chunk's cells): 60M rows 0.314 ->
    // 0.249 ms, 6M rows 54 -> 49 us per query.
    LineAhead ahead;
    for (int i = 0; i < 4; ++i) ahead.column(lane, A.col[i], i == 1 ? 1024u : 512u);
    ahead.column(lane, A.key0, 128);
    ahead.column(lane, A.key1, 128);
    for (uint32_t i = 0; i < A.nleaf; ++i) ahead.column(lane, A.leaf_col[i], 512);
    for (uint64_t c = warp; c < nfull; c += nwarps) {
        const uint64_t r = c * kDgRows + 4 * lane;  // this lane's four rows
        if (c + nwarps < nfull) ahead.fetch(c + nwarps);
        const uint4 q = ldcs4(A.col[0], r * 4);
        const uint4 p0 = ldcs4(A.col[1], r * 8), p1 = ldcs4(A.col[1], r * 8 + 16);
        const uint4 d = ldcs4(A.col[2], r * 4);
        const uint4 x = ldcs4(A.col[3], r * 4);
        const uint32_t k0 = __ldcs(reinterpret_cast<const unsigned int*>(A.key0 + r));
        const uint32_t k1 = __ldcs(reinterpret_cast<const unsigned int*>(A.key1 + r));
        uint4 lv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (static_cast<uint32_t>(i) < A.nleaf) lv[i] = ldcs4(A.leaf_col[i], r * 4);
        const uint32_t qa[4] = {q.x, q.y, q.z, q.w}, da[4] = {d.x, d.y, d.z, d.w}, xa[4] = {x.x, x.y, x.z, x.w};
        const int64_t pa[4] = {static_cast<int64_t>((static_cast<uint64_t>(p0.y) << 32) | p0.x),
                               static_cast<int64_t>((static_cast<uint64_t>(p0.w) << 32) | p0.z),
                               static_cast<int64_t>((static_cast<uint64_t>(p1.y) << 32) | p1.x),
                               static_cast<int64_t>((static_cast<uint64_t>(p1.w) << 32) | p1.z)};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            uint32_t m = 1u;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (static_cast<uint32_t>(i) >= A.nleaf) break;
                const uint32_t cell = e == 0 ? lv[i].x : e == 1 ? lv[i].y : e == 2 ? lv[i].z : lv[i].w;
                m &= leaf(cell, static_cast<uint32_t>(i));
            }
            const uint32_t g = (((k0 >> (8 * e)) & 0xffu) - A.kmin0) * A.kstride0 +
                               (((k1 >> (8 * e)) & 0xffu) - A.kmin1) * A.kstride1;
            add_row(0u - m, g, qa[e], pa[e], da[e], xa[e]);
        }
    }
    // The partial last chunk, one row per lane of one warp.
    if (warp == nfull % nwarps) {
        for (uint64_t r = nfull * kDgRows + lane; r < A.nrows; r += 32) {
            uint32_t m = 1u;
            for (uint32_t i = 0; i < A.nleaf; ++i) m &= leaf(reinterpret_cast<const uint32_t*>(A.leaf_col[i])[r], i);
            const uint32_t g = (static_cast<uint32_t>(A.key0[r]) - A.kmin0) * A.kstride0 +
                               (static_cast<uint32_t>(A.key1[r]) - A.kmin1) * A.kstride1;
            add_row(0u - m, g, reinterpret_cast<const uint32_t*>(A.col[0])[r],
                    reinterpret_cast<const long long*>(A.col[1])[r], reinterpret_cast<const uint32_t*>(A.col[2])[r],
                    reinterpret_cast<const uint32_t*>(A.col[3])[r]);
        }
    }
    __syncthreads();
    // Merge: warp w sums (group, slot) pairs w, w + 16, ... over the CTA's
    // threads; slot 0 is the row count, slots 1-4 the sums.
    const uint32_t wib = t >> 5;
    for (uint32_t i = wib; i < A.ngroups * 5; i += NT / 32) {
        const uint32_t g = i / 5, v = i % 5;
        unsigned long long sum = 0;
        for (uint32_t k = lane; k < NT; k += 32)
            sum += v == 0 ? static_cast<unsigned long long>(cnt[g * NT + k])
                          : static_cast<unsigned long long>(val[(static_cast<size_t>(g) * 4 + v - 1) * NT + k]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d);
        if (lane == 0 && sum) {
            atomicAdd(A.acc + 2ull * (g * 5 + v), sum);
            if (v == 0) atomicAdd(A.counters, sum);  // selected rows
        }
    }
    finish_result(A.out, t, NT, [] { __syncthreads(); });
}

}  // namespace

bool direct_group_supported(uint32_t kdt, uint32_t vdt) { return dg_kernel(kdt, vdt) != nullptr; }

int direct_group_ctas_per_sm(uint32_t hs, bool hasv) {
    const void* f = dg_kernel(DT_I64, hasv ? DT_I32 : 0);
    int occ = 0;
    const size_t smem = static_cast<size_t>(hs) * (hasv ? 12 : 8);
    if (allow_dynamic_smem(f, smem) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, kDgThreads, smem) != cudaSuccess) return 0;
    return occ;
}

bool hash_group_supported(uint32_t kdt, uint32_t vdt) { return hg_kernel(kdt, vdt) != nullptr; }

cudaError_t launch_hash_group(const HashGroupArgs& A, uint32_t kdt, uint32_t vdt, int sms, cudaStream_t st) {
    const void* f = hg_kernel(kdt, vdt);
    if (!f) return cudaErrorInvalidValue;
    HashGroupArgs a = A;
    a.hs = A.hs ? kHgSlots : 0u;
    a.hs_log2 = a.hs ? 31u - static_cast<uint32_t>(__builtin_clz(a.hs)) : 0u;
    const size_t smem = static_cast<size_t>(a.hs) * 16 + (kDgThreads / 32) * kHgQueue * (a.hs ? 16 : 20);
    const cudaError_t e = allow_dynamic_smem(f, smem);
    if (e != cudaSuccess) return e;
    void* args[] = {&a};
    return cudaLaunchKernel(f, dim3(static_cast<unsigned>(hash_group_grid(A.nrows, sms))), dim3(kDgThreads), args, smem, st);
}

uint64_t hash_group_grid(uint64_t nrows, int sms) {
    const uint64_t chunks = (nrows + kDgRows - 1) / kDgRows;
    const uint64_t want = (chunks + kDgThreads / 32 - 1) / (kDgThreads / 32);
    return std::max<uint64_t>(1, std::min<uint64_t>(want, static_cast<uint64_t>(sms) * kDgMinBlocks));
}

uint64_t hash_group_rows_per_cta(uint64_t nrows, int sms) {
    // A warp takes at most ceil(chunks / warps) chunks, and one warp the
    // partial last chunk.
    const uint64_t chunks = (nrows + kDgRows - 1) / kDgRows, nwarps = hash_group_grid(nrows, sms) * (kDgThreads / 32);
    return ((chunks + nwarps - 1) / nwarps) * kDgRows * (kDgThreads / 32) + kDgRows;
}

size_t q1_group_smem(uint32_t ngroups) { return static_cast<size_t>(ngroups) * kDgThreads * (4 + 4 * 8); }

int q1_group_ctas_per_sm(uint32_t ngroups) {
    const void* f = reinterpret_cast<const void*>(&q1_group_kernel);
    const size_t smem = q1_group_smem(ngroups);
    if (allow_dynamic_smem(f, smem) != cudaSuccess) return 0;
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, f, kDgThreads, smem) != cudaSuccess) return 0;
    return occ;
}

cudaError_t launch_q1_group(const Q1Args& A, int grid, cudaStream_t st) {
    const void* f = reinterpret_cast<const void*>(&q1_group_kernel);
    const size_t smem = q1_group_smem(A.ngroups);
    const cudaError_t e = allow_dynamic_smem(f, smem);
    if (e != cudaSuccess) return e;
    Q1Args a = A;
    void* args[] = {&a};
    return cudaLaunchKernel(f, dim3(static_cast<unsigned>(grid)), dim3(kDgThreads), args, smem, st);
}

cudaError_t launch_direct_group(const DirectGroupArgs& A, uint32_t kdt, uint32_t vdt, int grid, cudaStream_t st) {
    const void* f = dg_kernel(kdt, vdt);
    if (!f) return cudaErrorInvalidValue;
    const size_t smem = static_cast<size_t>(A.hs) * (vdt ? 12 : 8);
    const cudaError_t e = allow_dynamic_smem(f, smem);
    if (e != cudaSuccess) return e;
    DirectGroupArgs a = A;
    void* args[] = {&a};
    return cudaLaunchKernel(f, dim3(static_cast<unsigned>(grid)), dim3(kDgThreads), args, smem, st);
}

}  // namespace tgp
