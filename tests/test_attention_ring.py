"""The ring of K and V tiles of the prompt kernel, on the CPU: every tile once, in the order of the products, and no slot is
given back that nobody waits for."""
import pathlib
import re
import subprocess

ROOT = pathlib.Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include "webgpu_b200/csrc/attention_ring.h"
#include <cstdio>
#include <vector>
using namespace luxcuda;

int main() {
    for (uint32_t slots = 2; slots <= 9; slots++)
        for (uint32_t tiles = 1; tiles <= 60; tiles++) {
            const uint32_t entries = 2 * tiles;
            std::vector<int> seen(entries);
            uint32_t i = 0;
            auto is = [&](uint32_t tile, bool v) { const RingEntry e = ring_entry(i, tiles); seen[2 * e.tile + e.is_v]++; i++; return e.tile == tile && e.is_v == v; };
            bool ok = is(0, false);                      // scores of tile t + 1, then the weighted sum of tile t
            for (uint32_t t = 0; t < tiles; t++) {
                if (t + 1 < tiles) ok = is(t + 1, false) && ok;
                ok = is(t, true) && ok;
            }
            for (int n : seen) ok = ok && n == 1;
            if (!ok || i != entries) return std::printf("order, %u tiles\n", tiles), 1;
            // arrivals (the issuer's, one per entry given back) and waits (the copy warp's, before it fills a slot again)
            std::vector<int> arrivals(slots), waits(slots);
            for (uint32_t e = 0; e < entries; e++) arrivals[e % slots] += ring_refilled(e, entries, slots);
            for (uint32_t e = slots; e < entries; e++) waits[e % slots]++;
            if (arrivals != waits) return std::printf("%u tiles, %u slots\n", tiles, slots), 1;
        }
    return 0;
}
"""


def test_every_slot_given_back_is_waited_for(tmp_path):
    (tmp_path / "ring.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++20", "-O2", "-Wall", "-Werror", "-I", str(ROOT), str(tmp_path / "ring.cpp"), "-o", str(tmp_path / "ring")], check=True)
    out = subprocess.run([str(tmp_path / "ring")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_the_kernel_gives_back_by_that_rule():
    """Each arrival on kv_empty is under the rule, and the second CTA hands on what has landed there with a release."""
    src = (ROOT / "webgpu_b200/csrc/attention_prefill_mma.cu").read_text()
    commits = [line for line in src.splitlines() if "commit2(kv_empty" in line]
    assert commits and all("if (ring_refilled(i, entries, SLOTS))" in line for line in commits)
    assert re.search(r"arrive_release_cluster\(in_leader\(kv_full", src) and not re.search(r"arrive_cluster\(in_leader\(kv_full", src)
