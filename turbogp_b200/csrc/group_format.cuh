// group_format.cuh — writes one group of a device-formatted result: its key
// tuple and one tgp_agg_value per aggregate, from any of the group layouts.
#pragma once

#include <cstdint>

#include "plan.hpp"
#include "turbogp_gpu.h"

namespace tgp {

// The word of a group's slot that is not zero when the group has rows: after
// the key of a hash slot, else the first (one-word direct slots, direct
// accumulators).
__host__ __device__ __forceinline__ uint32_t count_word(const HashFormat& F) {
    return (F.hstride == 1 || F.direct_acc) ? 0u : 1u;
}

// A group's row count.
__device__ __forceinline__ uint64_t group_count(const unsigned long long* s, const HashFormat& F) {
    const uint64_t w = s[count_word(F)];
    return F.hpack ? (F.hpack_shift < 64 ? w >> F.hpack_shift : 0ull) : w;
}

// Value `v` of a group: the limbs of its accumulator.
__device__ __forceinline__ void group_value(const unsigned long long* s, const HashFormat& F, int v, uint8_t kind,
                                            uint64_t cnt, uint64_t& lo, int64_t& hi) {
    if (F.hpack) {
        // Below hpack_shift, the sum of (value - bias) over the slot's rows.
        const uint64_t w = s[count_word(F)];
        const uint64_t low = F.hpack_shift ? (w & ((1ull << F.hpack_shift) - 1ull)) : 0ull;
        const __int128 sum = static_cast<__int128>(low) + static_cast<__int128>(cnt) * F.hpack_bias;
        lo = static_cast<uint64_t>(sum);
        hi = static_cast<int64_t>(sum >> 64);
        return;
    }
    const unsigned long long* x = s + 2 + 2 * v;
    lo = x[0];
    if (kind == VK_MIN || kind == VK_MAX) hi = static_cast<int64_t>(x[0]) < 0 ? -1 : 0;
    else hi = F.sum64 ? (static_cast<int64_t>(x[0]) >> 63) : static_cast<int64_t>(x[1]);
}

// Output group i from its slot s ([key][count][value limbs...], or the direct
// accumulators' [count lo][count hi][value limbs...]).
// (key: the slot's packed key word, or its group index.)
__device__ __forceinline__ void write_group(const unsigned long long* s, unsigned long long key, uint64_t i,
                                            const HashFormat& F, uint64_t* keys_out, tgp_agg_value* vals_out) {
    if (keys_out)
        for (uint32_t k = 0; k < F.nkey; ++k)
            keys_out[i * F.nkey + k] = static_cast<uint64_t>(F.key_min[k]) +
                                       (F.direct_acc ? (key / F.key_div[k]) % F.key_mod[k]
                                                     : (key >> F.key_shift[k]) & F.key_mask[k]);
    if (!vals_out) return;
    const uint64_t cnt = group_count(s, F);
    for (uint32_t a = 0; a < F.nagg; ++a) {
        tgp_agg_value o;
        o.count = cnt;
        if (F.val[a] < 0) {
            o.lo = cnt;
            o.hi = 0;
            o.as_f64 = static_cast<double>(cnt);
        } else {
            group_value(s, F, F.val[a], F.kind[a], cnt, o.lo, o.hi);
            if (F.kind[a] == VK_MIN || F.kind[a] == VK_MAX) {
                o.as_f64 = static_cast<double>(static_cast<int64_t>(o.lo));
            } else {
                const double f = i128_to_f64_rn(o.lo, o.hi);
                o.as_f64 = F.func[a] == TGP_AGG_AVG ? (cnt ? f / static_cast<double>(cnt) : 0.0) : f;
            }
        }
        vals_out[i * F.nagg + a] = o;
    }
}

}  // namespace tgp
