// group_stream.cu — streaming form of the 32-bit limb tables
// (MODE_GROUP_SHARED32): direct groups of up to a few thousand, merged scans of
// batched requests (bucket keys), joins through a payload array. The scan
// engine's form stages tiles in shared memory, which leaves room for one CTA of
// 17 warps per SM beside the tables; at four warps per scheduler its loads,
// table lookups and atomics wait on one another (half the issue slots empty).
// Here one CTA of 1,024 threads per SM reads the rows straight from HBM: a
// lane takes four consecutive rows of a 128-row chunk with 16-byte loads, all
// of a chunk's columns in flight together, and shared memory holds only the
// tables, the bucket keys' per-cell tables (read through L1 they cost a tag
// cycle per lane) and the join's payload bytes or match bits (join_stream.cu).
// Rows in bucket 0 of a bucket key belong to no request and are left out.
// B200, merged batch of 16 requests over 60M rows, scan engine -> here: scans
// 314 -> 226 us, Q1 477 -> 328, joins 416 -> 282, the joins' count scan 173 -> 109;
// 20M rows over 2,526 groups with extremes 211 -> 175. What bounds it is the
// shared atomics: about three lanes of a warp on one bank, six to nine atomics
// per row.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "device_common.cuh"
#include "plan.hpp"
#include "runtime.hpp"

namespace tgp {

namespace {

constexpr int kGsThreads = kStreamThreads;
constexpr int kGsWarps = kGsThreads / 32;
constexpr int kGsRows = 128;
constexpr uint32_t kGsNone = 0xffu;   // payload byte: no match

__device__ __forceinline__ uint4 gs_load16(const uint8_t* base, uint64_t byte_off) {
    return __ldcs(reinterpret_cast<const uint4*>(base + byte_off));
}

// The low words of rows r .. r + 3 (r a multiple of 4) of an int32 or u8 column.
__device__ __forceinline__ uint4 gs_load32(const uint8_t* base, uint32_t dtype, uint64_t r) {
    if (dtype == DT_I32) return gs_load16(base, r * 4);
    const uint32_t w = __ldcs(reinterpret_cast<const unsigned int*>(base + r));
    return make_uint4(w & 0xffu, (w >> 8) & 0xffu, (w >> 16) & 0xffu, w >> 24);
}

__device__ __forceinline__ uint32_t gs_lds_u8(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}

__device__ __forceinline__ uint32_t elem(const uint4& v, int e) { return e == 0 ? v.x : e == 1 ? v.y : e == 2 ? v.z : v.w; }

// A value column's four cells as loaded: `hi` holds rows 2 and 3 of a 64-bit column.
struct GsCells {
    uint4 lo, hi;
};
__device__ __forceinline__ GsCells gs_load_cells(const uint8_t* base, uint32_t dtype, uint64_t r) {
    GsCells c;
    if (dtype == DT_I64 || dtype == DT_U64) {
        c.lo = gs_load16(base, r * 8);
        c.hi = gs_load16(base, r * 8 + 16);
    } else {
        c.lo = gs_load32(base, dtype, r);
        c.hi = make_uint4(0u, 0u, 0u, 0u);
    }
    return c;
}
__device__ __forceinline__ int64_t gs_cell(const GsCells& c, uint32_t dtype, int e) {
    if (dtype == DT_I64 || dtype == DT_U64) {
        const uint4& v = e < 2 ? c.lo : c.hi;
        const uint32_t a = (e & 1) ? v.z : v.x, b = (e & 1) ? v.w : v.y;
        return static_cast<int64_t>((static_cast<uint64_t>(b) << 32) | a);
    }
    const uint32_t x = elem(c.lo, e);
    return dtype == DT_I32 ? static_cast<int64_t>(static_cast<int32_t>(x)) : static_cast<int64_t>(x);
}

// A wide sum: the low limb's old value gives the carry into the high one.
__device__ __forceinline__ void gs_wide(uint32_t e, uint64_t v) {
    const uint32_t lo = static_cast<uint32_t>(v);
    const uint32_t old = atom_add_shared(e, lo);
    const uint32_t hi = static_cast<uint32_t>(v >> 32) + ((old + lo < old) ? 1u : 0u);
    if (hi) red_add_shared(e + 4u, hi);
}

// VS: the value program (GS_COLS, GS_Q1, GS_JOIN). PAY: the join payload
// (GS_PAY_*).
template <int VS, int PAY>
__global__ void __launch_bounds__(kGsThreads, 1) group_stream_kernel(const __grid_constant__ GroupStreamArgs A) {
    extern __shared__ __align__(16) uint8_t gs_smem[];
    const uint32_t t = threadIdx.x, lane = t & 31u, wib = t >> 5;
    // Shared: [payload bytes or bits][bucket tables][limb tables].
    if (PAY != GS_PAY_NONE) {
        uint4* dst = reinterpret_cast<uint4*>(gs_smem);
        const uint4* src = reinterpret_cast<const uint4*>(A.table);
        for (uint32_t i = t; i < A.table_bytes / 16; i += kGsThreads) dst[i] = __ldg(src + i);
    }
    for (uint32_t k = 0; k < A.nkey; ++k)
        if (A.key[k].lut)
            for (uint32_t i = t; i < A.key[k].cells; i += kGsThreads) gs_smem[A.key[k].lut_off + i] = A.key[k].lut[i];
    uint32_t* tabs = reinterpret_cast<uint32_t*>(gs_smem + A.tab_off);
    const uint32_t W = A.words, G = A.ngroups;
    for (uint32_t i = t; i < A.copies * G * W; i += kGsThreads) tabs[i] = 0;
    __syncthreads();
    const uint32_t base = smem_addr(gs_smem);
    const uint32_t tab = smem_addr(tabs) + (wib & (A.copies - 1u)) * G * W * 4u;
    const uint32_t W4 = W * 4u;
    uint32_t selected = 0;
    auto leaf = [&](uint32_t x, uint32_t i) { return ((x - A.leaf_lo[i]) <= A.leaf_sp[i] ? 1u : 0u) ^ ((A.leaf_neg >> i) & 1u); };
    // Payload group of a probe key (kGsNone: no match).
    auto lookup = [&](uint32_t rel) -> uint32_t {
        if (rel > A.krange) return kGsNone;
        if (PAY == GS_PAY_BYTES) return gs_lds_u8(base + rel);
        if (!((lds_u32(base + (rel >> 5) * 4u) >> (rel & 31u)) & 1u)) return kGsNone;
        return __ldg(A.pay + rel);
    };
    // The row's digit of key k; *none when it is bucket 0.
    auto digit = [&](uint32_t k, uint32_t x, bool* none) -> uint32_t {
        x -= A.key[k].min;
        if (!A.key[k].lut) return x * A.key[k].stride;
        x = gs_lds_u8(base + A.key[k].lut_off + x);
        *none = *none || x == 0u;
        return x * A.key[k].stride;
    };
    // The values of column c for N rows (cells, their words' addresses, bit r of
    // `on`): one loop over the rows per form of the value's words.
    auto column_rows = [&](uint32_t c, const uint32_t (&g)[4], uint32_t on, const int64_t (&cell)[4]) {
        for (uint32_t v = A.col[c].first; v < A.col[c].first + A.col[c].nops; ++v) {
            const GroupStreamOp& O = A.op[v];
            int64_t x[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                x[e] = O.ident ? cell[e]
                               : static_cast<int64_t>(static_cast<uint64_t>(O.mul) * static_cast<uint64_t>(cell[e]) +
                                                      static_cast<uint64_t>(O.add));
            if (O.kind == S32_MIN || O.kind == S32_MAX) {
                uint32_t k[4], old[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    k[e] = O.kind == S32_MIN ? O.ref - static_cast<uint32_t>(x[e]) : static_cast<uint32_t>(x[e]) - O.ref;
                    old[e] = 0xffffffffu;
                    if ((on >> e) & 1u) old[e] = lds_u32(g[e] + O.off);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (k[e] > old[e]) red_max_shared(g[e] + O.off, k[e]);
            } else if (O.kind == S32_NARROW) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if ((on >> e) & 1u) red_add_shared(g[e] + O.off, O.nz ? (x[e] != 0 ? 1u : 0u) : static_cast<uint32_t>(x[e]));
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if ((on >> e) & 1u) gs_wide(g[e] + O.off, static_cast<uint64_t>(x[e]));
            }
        }
    };
    // One value of the row whose words are at `e`.
    auto cell_at = [&](uint32_t c, uint64_t r) -> int64_t {
        const uint32_t dt = A.col[c].dtype;
        return dt == DT_U8    ? static_cast<int64_t>(A.col[c].col[r])
               : dt == DT_I32 ? static_cast<int64_t>(reinterpret_cast<const int32_t*>(A.col[c].col)[r])
                              : static_cast<int64_t>(reinterpret_cast<const long long*>(A.col[c].col)[r]);
    };
    auto column_ops = [&](uint32_t c, uint32_t e, uint64_t r) {
        const int64_t cell = cell_at(c, r);
        for (uint32_t v = A.col[c].first; v < A.col[c].first + A.col[c].nops; ++v) {
            const GroupStreamOp& O = A.op[v];
            const uint32_t at = e + O.off;
            const int64_t x = static_cast<int64_t>(static_cast<uint64_t>(O.mul) * static_cast<uint64_t>(cell) +
                                                   static_cast<uint64_t>(O.add));
            if (O.kind == S32_MIN || O.kind == S32_MAX) {
                const uint32_t k = O.kind == S32_MIN ? O.ref - static_cast<uint32_t>(x) : static_cast<uint32_t>(x) - O.ref;
                if (k > lds_u32(at)) red_max_shared(at, k);
            } else if (O.nz) {
                if (x != 0) red_add_shared(at, 1u);   // counts are narrow
            } else if (O.kind == S32_NARROW) {
                red_add_shared(at, static_cast<uint32_t>(x));
            } else {
                gs_wide(at, static_cast<uint64_t>(x));
            }
        }
    };
    // The values of the fixed programs.
    auto q1_values = [&](uint32_t e, uint32_t qty, uint64_t price, uint32_t disc, uint32_t tax) {
        const uint32_t q = A.mul[0] * qty + A.add[0];
        if (A.op[0].kind == S32_NARROW) red_add_shared(e + A.op[0].off, q);
        else gs_wide(e + A.op[0].off, q);
        gs_wide(e + A.op[1].off, price);
        const uint64_t v = price * static_cast<uint64_t>(A.mul[1] * disc + A.add[1]);
        gs_wide(e + A.op[2].off, v);
        gs_wide(e + A.op[3].off, v * static_cast<uint64_t>(A.mul[2] * tax + A.add[2]));
    };
    auto join_value = [&](uint32_t e, uint64_t price, uint32_t disc) {
        gs_wide(e + A.op[0].off, price * static_cast<uint64_t>(A.mul[1] * disc + A.add[1]));
    };

    const uint64_t warp = static_cast<uint64_t>(blockIdx.x) * kGsWarps + wib;
    const uint64_t nwarps = static_cast<uint64_t>(gridDim.x) * kGsWarps;
    const uint64_t nfull = A.nrows / kGsRows;
    // The next chunk's lines (the fixed programs; in the general one the shared
    // atomics are the bound and the prefetch costs registers).
    LineAhead ahead;
    if (VS != GS_COLS) {
        if (PAY != GS_PAY_NONE) ahead.column(lane, A.fk, 512);
        for (uint32_t k = 0; k < A.nkey; ++k) ahead.column(lane, A.key[k].col, A.key[k].dtype == DT_U8 ? 128u : 512u);
        for (uint32_t q = 0; q < (VS == GS_Q1 ? 4u : 2u); ++q) ahead.column(lane, A.col[q].col, q == 0 ? 1024u : 512u);
        for (uint32_t i = 0; i < A.nleaf; ++i) ahead.column(lane, A.leaf_col[i], 512);
    }
    for (uint64_t c = warp; c < nfull; c += nwarps) {
        const uint64_t r = c * kGsRows + 4 * lane;
        if (VS != GS_COLS && c + nwarps < nfull) ahead.fetch(c + nwarps);
        // Every column's loads first.
        uint4 fk = make_uint4(0u, 0u, 0u, 0u), kx[kGsKeys];
        GsCells v[kGsCols];
        if (PAY != GS_PAY_NONE) fk = gs_load16(A.fk, r * 4);
#pragma unroll
        for (int k = 0; k < kGsKeys; ++k)
            if (static_cast<uint32_t>(k) < A.nkey) kx[k] = gs_load32(A.key[k].col, A.key[k].dtype, r);
        if (VS == GS_COLS) {
#pragma unroll
            for (int q = 0; q < kGsCols; ++q)
                if (static_cast<uint32_t>(q) < A.ncol) v[q] = gs_load_cells(A.col[q].col, A.col[q].dtype, r);
        } else {
            v[0] = gs_load_cells(A.col[0].col, DT_I64, r);
            v[1].lo = gs_load16(A.col[1].col, r * 4);
            if (VS == GS_Q1) {
                v[1].hi = gs_load16(A.col[2].col, r * 4);
                v[2].lo = gs_load16(A.col[3].col, r * 4);
            }
        }
        uint32_t sel = 15u;
        for (uint32_t i = 0; i < A.nleaf; ++i) {
            const uint4 x = gs_load16(A.leaf_col[i], r * 4);
            sel &= leaf(x.x, i) | (leaf(x.y, i) << 1) | (leaf(x.z, i) << 2) | (leaf(x.w, i) << 3);
        }
        selected += __popc(sel);
        // Digits of all four rows, key by key (every cell lies in its column's
        // range, selected or not).
        uint32_t g[4] = {0u, 0u, 0u, 0u};
#pragma unroll
        for (int k = 0; k < kGsKeys; ++k) {
            if (static_cast<uint32_t>(k) >= A.nkey) break;
            const uint32_t mn = A.key[k].min, stride = A.key[k].stride;
            if (A.key[k].lut) {
                const uint32_t at = base + A.key[k].lut_off - mn;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t d = gs_lds_u8(at + elem(kx[k], e));
                    if (d == 0u) sel &= ~(1u << e);
                    g[e] += d * stride;
                }
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) g[e] += (elem(kx[k], e) - mn) * stride;
            }
        }
        if (PAY != GS_PAY_NONE) {
            uint32_t p[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) p[e] = ((sel >> e) & 1u) ? lookup(elem(fk, e) - A.kmin) : kGsNone;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (p[e] == kGsNone) sel &= ~(1u << e);
                g[e] += p[e];
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            g[e] = tab + g[e] * W4;
            if ((sel >> e) & 1u) red_add_shared(g[e], 1u);
        }
        if (VS == GS_COLS) {
#pragma unroll
            for (int q = 0; q < kGsCols; ++q) {
                if (static_cast<uint32_t>(q) >= A.ncol) break;
                const uint32_t dt = A.col[q].dtype;
                const int64_t cell[4] = {gs_cell(v[q], dt, 0), gs_cell(v[q], dt, 1), gs_cell(v[q], dt, 2), gs_cell(v[q], dt, 3)};
                column_rows(q, g, sel, cell);
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                if (!((sel >> e) & 1u)) continue;
                const uint64_t price = static_cast<uint64_t>(gs_cell(v[0], DT_I64, e));
                if (VS == GS_Q1) q1_values(g[e], elem(v[1].lo, e), price, elem(v[1].hi, e), elem(v[2].lo, e));
                else join_value(g[e], price, elem(v[1].lo, e));
            }
        }
    }
    // The partial last chunk, one row per lane of one warp.
    if (warp == nfull % nwarps) {
        auto word = [&](const uint8_t* col, uint32_t dtype, uint64_t r) -> uint32_t {
            return dtype == DT_U8 ? col[r] : reinterpret_cast<const uint32_t*>(col)[r];
        };
        for (uint64_t r = nfull * kGsRows + lane; r < A.nrows; r += 32) {
            bool on = true, none = false;
            for (uint32_t i = 0; i < A.nleaf; ++i) on = on && leaf(word(A.leaf_col[i], DT_I32, r), i);
            if (!on) continue;
            ++selected;
            uint32_t g = 0;
            for (uint32_t k = 0; k < A.nkey; ++k) g += digit(k, word(A.key[k].col, A.key[k].dtype, r), &none);
            if (none) continue;
            if (PAY != GS_PAY_NONE) {
                const uint32_t p = lookup(word(A.fk, DT_I32, r) - A.kmin);
                if (p == kGsNone) continue;
                g += p;
            }
            const uint32_t e = tab + g * W4;
            red_add_shared(e, 1u);
            if (VS == GS_COLS) {
                for (uint32_t q = 0; q < A.ncol; ++q) column_ops(q, e, r);
            } else {
                const uint64_t price = reinterpret_cast<const unsigned long long*>(A.col[0].col)[r];
                if (VS == GS_Q1) q1_values(e, word(A.col[1].col, DT_I32, r), price, word(A.col[2].col, DT_I32, r),
                                           word(A.col[3].col, DT_I32, r));
                else join_value(e, price, word(A.col[1].col, DT_I32, r));
            }
        }
    }
    __syncwarp();
    selected = __reduce_add_sync(0xffffffffu, selected);
    if (lane == 0 && selected) atomicAdd(A.counters, static_cast<unsigned long long>(selected));
    __syncthreads();
    // Merge: thread i takes (group, slot) pair i; slot 0 is the row count.
    const uint32_t nv1 = A.nval + 1u;
    for (uint32_t i = t; i < G * nv1; i += kGsThreads) {
        const uint32_t g = i / nv1, s = i % nv1;
        unsigned long long sum = 0;
        uint32_t far = 0, rows = 0;
        const uint32_t kind = s == 0 ? static_cast<uint32_t>(S32_WIDE) : A.op[s - 1].kind;
        for (uint32_t c = 0; c < A.copies; ++c) {
            const uint32_t* e = tabs + (static_cast<size_t>(c) * G + g) * W;
            rows |= e[0];
            if (s == 0) {
                sum += e[0];
                continue;
            }
            const uint32_t* w = e + A.op[s - 1].off / 4u;
            if (kind == S32_WIDE) sum += (static_cast<unsigned long long>(static_cast<long long>(static_cast<int32_t>(w[1]))) << 32) + w[0];
            else if (kind == S32_NARROW) sum += static_cast<unsigned long long>(static_cast<long long>(static_cast<int32_t>(w[0])));
            else far = max(far, w[0]);
        }
        if (rows == 0) continue;
        unsigned long long* out = A.acc + 2ull * (static_cast<uint64_t>(g) * A.acc_stride + (s == 0 ? 0u : A.op[s - 1].slot));
        if (kind == S32_MIN) atomicMin(reinterpret_cast<long long*>(out), A.op[s - 1].ref64 - static_cast<long long>(far));
        else if (kind == S32_MAX) atomicMax(reinterpret_cast<long long*>(out), A.op[s - 1].ref64 + static_cast<long long>(far));
        else if (sum) atomicAdd(out, sum);
    }
    finish_result(A.out, t, kGsThreads, [] { __syncthreads(); });
}

template <int VS>
const void* gs_kernel(int pay) {
    switch (pay) {
        case GS_PAY_NONE: return reinterpret_cast<const void*>(&group_stream_kernel<VS, GS_PAY_NONE>);
        case GS_PAY_BYTES: return reinterpret_cast<const void*>(&group_stream_kernel<VS, GS_PAY_BYTES>);
        default: return reinterpret_cast<const void*>(&group_stream_kernel<VS, GS_PAY_BITS>);
    }
}

}  // namespace

uint64_t group_stream_grid(uint64_t nrows, int sms) {
    const uint64_t chunks = (nrows + kGsRows - 1) / kGsRows;
    return std::max<uint64_t>(1, std::min<uint64_t>((chunks + kGsWarps - 1) / kGsWarps, static_cast<uint64_t>(sms)));
}

uint64_t group_stream_rows_per_cta(uint64_t nrows, int sms) {
    // Warp c % warps takes chunk c, the partial last one included.
    const uint64_t chunks = (nrows + kGsRows - 1) / kGsRows, nwarps = group_stream_grid(nrows, sms) * kGsWarps;
    return (chunks + nwarps - 1) / nwarps * kGsRows * kGsWarps;
}

cudaError_t launch_group_stream(const GroupStreamArgs& A, int vs, int pay, uint32_t smem, int grid, cudaStream_t st) {
    const void* f = vs == GS_COLS ? gs_kernel<GS_COLS>(pay) : vs == GS_Q1 ? gs_kernel<GS_Q1>(pay) : gs_kernel<GS_JOIN>(pay);
    const cudaError_t e = allow_dynamic_smem(f, smem);
    if (e != cudaSuccess) return e;
    GroupStreamArgs a = A;
    void* args[] = {&a};
    return cudaLaunchKernel(f, dim3(static_cast<unsigned>(grid)), dim3(kGsThreads), args, smem, st);
}

}  // namespace tgp
