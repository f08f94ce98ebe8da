// attention_passes.h -- how a prompt's attention is cut up where the parts of all keys do not fit the scratch
// (attention_prefill_mma.cu; no CUDA needed).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace luxcuda {

constexpr size_t TILE_SCRATCH = 4 * 3 * 64 * 128 + 8;        // of 64 keys of K and V of a KV head, flags included
constexpr size_t CARRY = 128 * (128 + 4) * 4 + 16;           // of a block of 128 queries between passes, flags included

// KV heads and levels (blocks of queries, or pairs of them) at a time, and key tiles per pass over them.
struct Passes {
    uint32_t heads = 0, levels = 0, tiles = 0;         // heads 0: the scratch is too small
    size_t carry_at = 0;                               // where the scratch has what blocks carry from pass to pass

    // of the pass that begins at tile t of n: equal numbers, the last one's rest aside
    uint32_t pass_tiles(uint32_t t, uint32_t n) const {
        const uint32_t passes = std::max((n + tiles - 1) / tiles, 1u), each = (n + passes - 1) / passes;
        return std::min(each, n - t);
    }
};

// Either all keys of as many KV heads at a time as have their parts in the scratch (of all of them: one pass in all), or ranges of the
// keys, by so many heads and levels that their CTAs (2 x units a head and level) are two waves: heads one after the other would leave
// most of the chip idle.  Whichever takes fewer waves over all keys; ranges have to earn what their blocks carry.  8 KV heads, us a call
// head by head / in ranges: 256 queries over 32768 keys (half of the heads fit) 1966 / 1083, over 131072 29651 / 4294, 2048 queries over 131072
// 29807 / 21738; 200000 keys, which no head's parts fit: 45419 on the f32 pipe / 7436.
inline Passes plan_passes(uint32_t bks, uint32_t levels, uint32_t units, uint32_t tiles, size_t scratch, uint32_t sms, uint32_t forced_tiles) {
    const uint64_t ctas = 2ull * levels * units;       // of a KV head
    const uint32_t fit = tiles ? (uint32_t)std::min<uint64_t>({scratch / (tiles * TILE_SCRATCH), bks, 65535}) : std::min(bks, 65535u);
    auto waves = [&](uint32_t heads, uint32_t lv) {    // of all KV heads and levels, so many at a time
        auto of = [&](uint64_t h) { return (h * 2u * units * lv + sms - 1) / sms; };
        return (double)((bks / heads * of(heads) + of(bks % heads)) * ((levels + lv - 1) / lv));
    };
    Passes whole, ranges;
    if (fit) whole = {fit, levels, std::max(tiles, 1u), 0};
    if (fit == bks && !(forced_tiles && forced_tiles < tiles)) return whole;
    ranges.heads = (uint32_t)std::min<uint64_t>({(2ull * sms + ctas - 1) / ctas, bks, 65535});
    const uint64_t per_level = 2ull * units * ranges.heads;
    ranges.levels = (uint32_t)std::min<uint64_t>(std::max<uint64_t>(scratch / 4 / CARRY / per_level, 1), levels);
    const uint64_t carry = ranges.levels * per_level * CARRY;
    if (carry < scratch) {
        ranges.carry_at = (scratch - carry) / 128 * 128;
        ranges.tiles = (uint32_t)std::min<size_t>(ranges.carry_at / (ranges.heads * TILE_SCRATCH), tiles);
    }
    if (forced_tiles) ranges.tiles = std::min(ranges.tiles, forced_tiles);
    if (!ranges.tiles || (fit && !forced_tiles && waves(ranges.heads, ranges.levels) * 1.05 >= waves(fit, levels))) return whole;
    return ranges;
}

}  // namespace luxcuda
