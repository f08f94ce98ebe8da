"""How a prompt over a long cache is cut into passes, on the CPU: what a pass writes lies in the scratch, every key tile of every
block is taken once, and a chip that the heads one after the other would leave idle is filled."""
import pathlib
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include "webgpu_b200/csrc/attention_passes.h"
#include <cstdio>
#include <random>
using namespace luxcuda;

int main() {
    std::mt19937_64 rng(3);
    auto log = [&](uint64_t top) { return (uint32_t)(rng() % (1 + (rng() % (top >> rng() % 20 | 1)))); };
    const size_t full = 131072 / 64 * TILE_SCRATCH;
    int ranges = 0, none = 0;
    for (int n = 0; n < 400000; n++) {
        const uint32_t bks = 1 + log(1 << 17), levels = 1 + log(1 << 14), units = 1 + log(1 << 9), tiles = log(1 << 15);
        const size_t scratch = rng() % 3 ? full : rng() % 2 ? full >> rng() % 6 : rng() % (1 << 22);
        const uint32_t forced = rng() % 4 ? 0 : 1 + log(64);
        const Passes p = plan_passes(bks, levels, units, tiles, scratch, 148, forced);
        if (!p.heads) {
            if (tiles && scratch >= 2 * tiles * TILE_SCRATCH) return std::printf("refused: %u tiles, %zu bytes\n", tiles, scratch), 1;
            none++;
            continue;
        }
        if (p.heads > bks || p.heads > 65535 || !p.levels || p.levels > levels || !p.tiles) return std::printf("plan %u %u %u\n", p.heads, p.levels, p.tiles), 1;
        const uint32_t seen = tiles ? 1 + (uint32_t)(rng() % tiles) : 0;                 // tiles that some level sees
        uint32_t at = 0, passes = 0, most = 0;
        for (uint32_t t = 0; t < seen || t == 0; passes++) {
            const uint32_t k = p.pass_tiles(t, seen);
            if (t != at || (seen && !k) || k > p.tiles) return std::printf("%u tiles at %u of %u\n", k, t, seen), 1;
            most = std::max(most, k);
            at = t + k;
            t += std::max(k, 1u);
        }
        if (at != seen) return std::printf("%u of %u tiles\n", at, seen), 1;
        const size_t parts = (size_t)p.heads * most * TILE_SCRATCH, blocks = 2ull * p.levels * units * p.heads;
        if (parts > scratch) return std::printf("parts\n"), 1;
        if (passes > 1 && (p.carry_at % 128 || parts > p.carry_at || p.carry_at + blocks * CARRY > scratch)) return std::printf("carry\n"), 1;
        ranges += passes > 1;
    }
    if (ranges < 1000 || none < 1000) return std::printf("%d in ranges, %d refused\n", ranges, none), 1;
    // 256 queries of 32 heads over 131072 keys of 8 KV heads: all blocks at once; 150 KV heads of 16 tiles: as many heads as fit
    const Passes a = plan_passes(8, 2, 2, 2048, full, 148, 0), b = plan_passes(150, 1, 1, 16, full, 148, 0);
    if (a.heads != 8 || a.levels != 2 || a.tiles < 240) return std::printf("long cache %u %u %u\n", a.heads, a.levels, a.tiles), 1;
    if (b.tiles != 16) return std::printf("many heads %u %u %u\n", b.heads, b.levels, b.tiles), 1;
    return 0;
}
"""


def test_passes_stay_in_the_scratch_and_take_every_tile_once(tmp_path):
    (tmp_path / "passes.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++20", "-O2", "-Wall", "-Werror", "-I", str(ROOT), str(tmp_path / "passes.cpp"), "-o", str(tmp_path / "passes")], check=True)
    out = subprocess.run([str(tmp_path / "passes")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
