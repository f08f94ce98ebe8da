"""The places of partial results that the merge of an evenly dealt decode step follows, on the CPU: whatever the scratch
holds where a span should be, no place outside the scratch is taken from it."""
import subprocess
import pathlib

ROOT = pathlib.Path(__file__).resolve().parents[1]

PROGRAM = r"""
#include "webgpu_b200/csrc/attention_span.h"
#include <cstdio>
#include <random>
using namespace luxcuda;

int main() {
    std::mt19937 rng(1);
    // every share of up to 9 chunks over items of up to 40: what the CTAs write is accepted and names each CTA's own place once
    for (uint32_t chunks = 1; chunks <= 40; chunks++)
        for (uint32_t share = 1; share <= 9; share++)
            for (uint32_t items = 1; items <= 6; items++) {
                const uint32_t all = items * chunks, grid = (all + share - 1) / share;
                uint32_t used[512] = {};
                for (uint32_t it = 0; it < items; it++) {
                    const uint32_t lo = it * chunks, hi = lo + chunks, first = lo / share, last = (hi - 1) / share;
                    const AttnSpan s{(int32_t)first, (int32_t)(last - first + 1)};
                    if (!span_fits(s, grid)) return std::printf("refused %u %u %u\n", chunks, share, items), 1;
                    for (uint32_t i = 0; i < (uint32_t)s.ctas && s.ctas > 1; i++)
                        if (span_place(s, i) >= 2 * grid || used[span_place(s, i)]++) return std::printf("place %u of item %u\n", span_place(s, i), it), 1;
                }
            }
    // anything else: float bits, small numbers, the ends of the range
    for (int n = 0; n < 2000000; n++) {
        const uint32_t grid = 1 + rng() % 512;
        auto word = [&]() -> int32_t {
            switch (rng() % 4) {
                case 0: return (int32_t)rng();
                case 1: return (int32_t)(rng() % 600) - 40;
                case 2: return (int32_t)grid + (int32_t)(rng() % 3) - 1;
                default: return rng() % 2 ? 0x7fffffff - (int32_t)(rng() % 4) : (int32_t)(0x80000000u + rng() % 4);
            }
        };
        const AttnSpan s{word(), word()};
        if (!span_fits(s, grid)) continue;
        if (s.ctas > 512) return std::printf("%d partial results\n", s.ctas), 1;
        for (uint32_t i = 0; i < (uint32_t)s.ctas; i++)
            if (span_place(s, i) >= 2 * grid) return std::printf("span %d %d of %u CTAs\n", s.first, s.ctas, grid), 1;
    }
    return 0;
}
"""


def test_no_span_leads_outside_the_scratch(tmp_path):
    (tmp_path / "span.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++20", "-O2", "-Wall", "-Werror", "-I", str(ROOT), str(tmp_path / "span.cpp"), "-o", str(tmp_path / "span")], check=True)
    out = subprocess.run([str(tmp_path / "span")], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout


def test_the_merge_follows_only_spans_that_fit():
    merge = (ROOT / "webgpu_b200/csrc/attention.cu").read_text()
    merge = merge[merge.index("lux_attn_merge_even_f32(const AttnParams"):]
    merge = merge[:merge.index("\n}")]
    assert merge.index("span_fits(span, p.ctas)") < merge.index("span_place(")
