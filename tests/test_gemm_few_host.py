"""How small products of few rows are split over blocks, for sizes that the split rule meets."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(__file__), "..", "poptransformer_b200", "csrc")
DRIVER = r"""
#include <cstdio>
#include "gemm_few.h"
using namespace pt::few;
int main() {
  for (int m : {1, 3, 8})
    for (int n : {1, 8, 16, 40, 768, 2048, 2304, 8000, 50257, 262144})
      for (int k : {64, 128, 768, 1024, 1600, 4096, 65536})
        if (small(m, n, k)) {
          const Plan p = make_plan(m, n, k, 148);
          printf("%d %d %d %d %d %d %d %d %u %u %u\n", n, k, p.units, p.warps_k, p.slices, p.kb_per_slice, p.stages, p.blocks, p.stage_bytes, p.sum_offset, p.smem);
        }
}
"""


def test_plans_cover_the_product_and_fit(tmp_path):
    (tmp_path / "plan.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", str(tmp_path / "plan"), str(tmp_path / "plan.cpp")], check=True)
    lines = subprocess.run([str(tmp_path / "plan")], check=True, capture_output=True, text=True).stdout.splitlines()
    assert len(lines) > 100
    for line in lines:
        n, k, units, warps, slices, kbs, stages, blocks, stage_bytes, sum_offset, smem = map(int, line.split())
        assert 1 <= units * warps <= 12 and 1 <= slices <= 8 and 2 <= stages <= 12, line
        assert (slices - 1) * kbs < k // 64 <= slices * kbs, line                  # every slice has k blocks
        assert blocks == -(-(-(-n // 16)) // units) * slices, line
        assert stage_bytes == warps * (units * 2048 + 1024) and sum_offset == stages * stage_bytes, line
        assert smem == sum_offset + -(-units // slices) * slices * warps * 640 + 1024 and 2 * (smem + 1024 + 1024) <= 228 * 1024, line    # (and its barriers)
