// join_pairs.cu — (probe row, build row) pairs of an inner equi-join
// (hash_join_with_keys, src/engine/query_interpreter/join.rs:544-794, its pair
// lists) in ascending (probe row, build row) order, written in place.
//
// The pairs of a probe row follow those of every earlier row, so a prefix sum
// of match counts places them and nothing is sorted:
//   1. count: a warp takes kPairRows consecutive probe rows (lane l holds rows
//      l, 32 + l, 64 + l, 96 + l, so key loads coalesce), probes the join table
//      with its lanes' four lookups in flight at once, keeps one word per row
//      (unique build keys: the matching build row; else the number of matches)
//      and the chunk's number of pairs;
//   2. a device scan over the chunks;
//   3. write: unique keys compact the kept rows by ballots; otherwise a row
//      with matches probes again and writes them in ascending build row order
//      (an insertion sort of at most kPairSortMax matches; more take the
//      radix-sorted path of the scan engine).
// Both passes stream the rows at full occupancy (no stage ring): a probe waits
// on a dependent L2 access per step, so warps in flight set the pace. B200, 8M
// probe rows (half selected) against 200K keys of two rows, 3.9M pairs: count
// 73 us and write 99 us; in the scan engine's form 207 us each and a radix sort
// of the pairs of 370 us.
#include <cuda_runtime.h>

#include <cstdint>
#include <cub/cub.cuh>

#include "device_common.cuh"
#include "plan.hpp"
#include "runtime.hpp"

namespace tgp {

namespace {

constexpr int kPairThreads = 256;
constexpr int kPairRows = 128;              // rows per warp chunk
constexpr uint32_t kNoRow = 0xffffffffu;    // no match (tables hold fewer than 2^32 - 1 rows)

__device__ __forceinline__ int64_t probe_cell(const uint8_t* col, uint32_t dtype, uint64_t row) {
    if (dtype == DT_U8) return __ldcs(col + row);
    if (dtype == DT_I32) return __ldcs(reinterpret_cast<const int*>(col) + row);
    return __ldcs(reinterpret_cast<const long long*>(col) + row);
}

// One slot of the join table: whether it is empty, its key and its build row.
template <bool WIDE>
struct SlotRef {
    unsigned long long e0, e1;
    __device__ __forceinline__ void load(const unsigned long long* tab, uint64_t h) {
        if constexpr (WIDE) {
            const ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(tab) + h);
            e0 = v.x;
            e1 = v.y;
        } else {
            e0 = __ldg(tab + h);
        }
    }
    __device__ __forceinline__ bool empty() const { return WIDE ? e1 == 0ull : e0 == ~0ull; }
    __device__ __forceinline__ bool matches(uint64_t rel) const { return WIDE ? e0 == rel : (e0 >> 32) == rel; }
    __device__ __forceinline__ uint32_t row() const { return static_cast<uint32_t>(WIDE ? e1 - 1 : e0); }
};

// Whether this lane's row `r` of the chunk at `base` probes, and its key
// relative to the build side's minimum.
__device__ __forceinline__ bool probe_key(const PairArgs& A, uint64_t base, int r, uint32_t lane, uint64_t& rel) {
    const uint64_t row = base + 32u * r + lane;
    bool on = row < A.nrows;
    if (on && A.bitmap) on = (A.bitmap[(base >> 5) + r] >> lane) & 1u;
    rel = 0;
    if (on) {
        rel = static_cast<uint64_t>(probe_cell(A.key, A.dtype, row)) - static_cast<uint64_t>(A.kmin);
        on = rel <= A.krange;
    }
    return on;
}

template <bool WIDE, bool UNIQUE>
__global__ void __launch_bounds__(kPairThreads) pair_count_kernel(const PairArgs A) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t nchunks = (A.nrows + kPairRows - 1) / kPairRows;
    const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * (kPairThreads / 32);
    uint32_t most = 0;
    for (uint64_t c = (static_cast<uint64_t>(blockIdx.x) * kPairThreads + threadIdx.x) >> 5; c < nchunks; c += nwarps) {
        const uint64_t base = c * kPairRows;
        uint64_t rel[4], h[4];
        uint32_t res[4];
        uint32_t pend = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            if (probe_key(A, base, r, lane, rel[r])) pend |= 1u << r;
            h[r] = hash_slot(rel[r], A.log2);
            res[r] = UNIQUE ? kNoRow : 0u;
        }
        // A table is at most half full and a chain ends at an empty slot; the
        // step bound covers a table without one.
        for (uint64_t n = 0; pend && n <= A.mask; ++n) {
            SlotRef<WIDE> s[4];
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if ((pend >> r) & 1u) s[r].load(A.tab, h[r]);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                if (!((pend >> r) & 1u)) continue;
                if (s[r].empty()) {
                    pend &= ~(1u << r);
                } else if (s[r].matches(rel[r])) {
                    if (UNIQUE) {
                        res[r] = s[r].row();
                        pend &= ~(1u << r);
                    } else {
                        ++res[r];
                    }
                }
                h[r] = (h[r] + 1) & A.mask;
            }
        }
        unsigned long long total = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint64_t row = base + 32u * r + lane;
            if (row < A.nrows) A.kept[row] = res[r];
            if (UNIQUE) {
                total += __popc(__ballot_sync(0xffffffffu, res[r] != kNoRow));
            } else {
                total += res[r];
                most = max(most, res[r]);
            }
        }
        if (!UNIQUE) {
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) total += __shfl_down_sync(0xffffffffu, total, d);
        }
        if (lane == 0) A.chunk[c] = total;
    }
    if (!UNIQUE) {
        most = __reduce_max_sync(0xffffffffu, most);
        if (lane == 0 && most) atomicMax(A.most, most);
    }
}

template <bool WIDE, bool UNIQUE>
__global__ void __launch_bounds__(kPairThreads) pair_write_kernel(const PairArgs A, const unsigned long long* offset,
                                                                  uint32_t* probe, uint32_t* build) {
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    const uint64_t nchunks = (A.nrows + kPairRows - 1) / kPairRows;
    const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * (kPairThreads / 32);
    for (uint64_t c = (static_cast<uint64_t>(blockIdx.x) * kPairThreads + threadIdx.x) >> 5; c < nchunks; c += nwarps) {
        const uint64_t base = c * kPairRows;
        unsigned long long o = offset[c];
        if (offset[c + 1] == o) continue;
        uint32_t kept[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint64_t row = base + 32u * r + lane;
            kept[r] = row < A.nrows ? A.kept[row] : (UNIQUE ? kNoRow : 0u);
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const uint32_t row = static_cast<uint32_t>(base + 32u * r + lane);
            if (UNIQUE) {
                const uint32_t m = __ballot_sync(0xffffffffu, kept[r] != kNoRow);
                if (kept[r] != kNoRow) {
                    const unsigned long long at = o + __popc(m & below);
                    probe[at] = row;
                    build[at] = kept[r];
                }
                o += __popc(m);
            } else {
                const uint32_t n = kept[r];
                uint32_t incl = n;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= static_cast<uint32_t>(d)) incl += y;
                }
                const unsigned long long at = o + incl - n;
                o += __shfl_sync(0xffffffffu, incl, 31);
                if (n) {
                    uint64_t rel;
                    probe_key(A, base, r, lane, rel);
                    uint64_t h = hash_slot(rel, A.log2);
                    uint32_t got = 0;
                    for (uint64_t k = 0; got < n && k <= A.mask; ++k) {
                        SlotRef<WIDE> s;
                        s.load(A.tab, h);
                        if (s.empty()) break;
                        if (s.matches(rel)) {
                            // Insert into the ascending run written so far.
                            const uint32_t b = s.row();
                            uint32_t j = got++;
                            for (; j > 0 && build[at + j - 1] > b; --j) build[at + j] = build[at + j - 1];
                            build[at + j] = b;
                        }
                        h = (h + 1) & A.mask;
                    }
                    for (uint32_t j = 0; j < n; ++j) probe[at + j] = row;
                }
            }
        }
    }
}

uint64_t pair_chunks(uint64_t nrows) { return (nrows + kPairRows - 1) / kPairRows; }

int pair_grid(uint64_t nrows, int sms) {
    const uint64_t blocks = (pair_chunks(nrows) + kPairThreads / 32 - 1) / (kPairThreads / 32);
    return static_cast<int>(blocks < static_cast<uint64_t>(sms) * 8 ? blocks : static_cast<uint64_t>(sms) * 8);
}

}  // namespace

// Scratch: chunk counts [nchunks + 1], their exclusive sums [nchunks + 1]
// (u64; the last one is the number of pairs), CUB's scan storage.
size_t pair_scratch(uint64_t nrows) {
    const uint64_t n = pair_chunks(nrows) + 1;
    size_t tmp = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tmp, static_cast<unsigned long long*>(nullptr),
                                  static_cast<unsigned long long*>(nullptr), static_cast<int>(n));
    return n * 16 + tmp + 256;
}

cudaError_t count_pairs(PairArgs A, bool wide, bool unique, void* scratch, size_t scratch_bytes,
                        unsigned long long* total, int sms, cudaStream_t st) {
    const uint64_t nc = pair_chunks(A.nrows);
    unsigned long long* chunk = static_cast<unsigned long long*>(scratch);
    unsigned long long* offset = chunk + nc + 1;
    uint8_t* tmp = reinterpret_cast<uint8_t*>(offset + nc + 1);
    size_t tmp_bytes = scratch_bytes - (nc + 1) * 16;
    A.chunk = chunk;
    cudaError_t e = cudaMemsetAsync(chunk + nc, 0, 8, st);
    if (e != cudaSuccess) return e;
    const int grid = pair_grid(A.nrows, sms);
    if (grid) {
        if (wide) pair_count_kernel<true, false><<<grid, kPairThreads, 0, st>>>(A);
        else if (unique) pair_count_kernel<false, true><<<grid, kPairThreads, 0, st>>>(A);
        else pair_count_kernel<false, false><<<grid, kPairThreads, 0, st>>>(A);
    }
    e = cub::DeviceScan::ExclusiveSum(tmp, tmp_bytes, chunk, offset, static_cast<int>(nc + 1), st);
    if (e != cudaSuccess) return e;
    return cudaMemcpyAsync(total, offset + nc, 8, cudaMemcpyDeviceToDevice, st);
}

cudaError_t write_pairs(const PairArgs& A, bool wide, bool unique, const void* scratch, uint32_t* probe,
                        uint32_t* build, int sms, cudaStream_t st) {
    const int grid = pair_grid(A.nrows, sms);
    if (grid == 0) return cudaSuccess;
    const unsigned long long* offset = static_cast<const unsigned long long*>(scratch) + pair_chunks(A.nrows) + 1;
    if (wide) pair_write_kernel<true, false><<<grid, kPairThreads, 0, st>>>(A, offset, probe, build);
    else if (unique) pair_write_kernel<false, true><<<grid, kPairThreads, 0, st>>>(A, offset, probe, build);
    else pair_write_kernel<false, false><<<grid, kPairThreads, 0, st>>>(A, offset, probe, build);
    return cudaGetLastError();
}

}  // namespace tgp
