"""What a block of the tensor-core GEMMs takes of its SM, over the sizes that pt_gemm accepts.  Blocks wait without a limit for tensor memory and for
the other blocks of their cluster, and launches of several streams meet on an SM: the two waits must not be able to close a circle."""
import os
import re
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(__file__), "..", "poptransformer_b200", "csrc")
DRIVER = r"""
#include <cstdio>
#include <initializer_list>
#include <cstdlib>
#include "gemm_plan.h"
using namespace pt::tc;
int main(int argc, char **argv) {
  if (argc > 1) {                        // one product: format, rows, n, k
    const int f = atoi(argv[1]);
    printf("%d\n", plan_gemm({f == 0, f == 2, f == 3, atoi(argv[2]), atoi(argv[3]), atoi(argv[4]), 0, 0, 148}).ksplit);
    return 0;
  }
  for (int fmt = 0; fmt < 4; ++fmt)      // INT4, FP8, BF16, FP16
    for (int m : {1, 9, 16, 17, 32, 33, 48, 64, 65, 80, 96, 112, 128, 129, 144, 176, 208, 224, 255, 256, 257, 511, 2048, 5000})
      for (int n : {40, 128, 768, 1600, 4096, 12288, 22016, 50257, 65024})
        for (int k : {128, 256, 768, 2048, 4096, 11008, 16384})
          for (int ks : {0, 1, 2, 5, 8, 16})
            for (int rows : {0, 16, 128, 256}) {
              if (rows && fmt != 2) continue;
              const GemmPlan p = plan_gemm({fmt == 0, fmt == 2, fmt == 3, rows ? (m + rows - 1) / rows * rows : m, n, k, ks, rows, 148});
              printf("%d %d %u %d %d %d %d %d %d\n", fmt, (int)p.fits, p.smem, p.tmem_columns, p.ksplit, p.na, p.mb, p.stages, (int)p.stage_bytes);
            }
}
"""
SM, RESERVE, COLUMNS, LIMIT = 228 * 1024, 1024, 512, 220 * 1024      # bytes of an SM, of them the system's for each block; columns; bytes a block may ask for


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, "-o", str(d / "plan"), str(d / "plan.cpp")], check=True)
    return lambda *args: subprocess.run([str(d / "plan"), *map(str, args)], check=True, capture_output=True, text=True).stdout


@pytest.fixture(scope="module")
def plans(driver):
    return sorted({tuple(map(int, line.split())) for line in driver().splitlines()})


def test_plans_fit(plans):
    for fmt, fits, smem, columns, ksplit, na, mb, stages, stage_bytes in plans:
        assert fits and smem <= LIMIT and na * mb <= columns <= COLUMNS and columns & (columns - 1) == 0
        assert ksplit == 1 or (na == 1 and mb * 512 <= smem - 1024)         # the sums of a slice, in the ring
        if 2 * (smem + RESERVE) <= SM:
            assert 2 * columns <= COLUMNS                                   # blocks of one launch never wait for one another's columns


def test_waits_close_no_circle(plans):
    assert 3 * (min(p[2] for p in plans) + RESERVE) > SM                    # at most two blocks on an SM
    clustered = sorted({(p[2], p[3]) for p in plans if p[4] > 1})
    for a in clustered:
        for b in clustered:
            assert a[0] + b[0] + 2 * RESERVE > SM or a[1] + b[1] <= COLUMNS, (a, b)


def test_blocks_that_share_an_sm_are_compiled_to(plans):
    """Where the plan lets two blocks of a launch share an SM, the kernel is bound to registers that allow it (launch bounds)."""
    text = open(os.path.join(CSRC, "gemm_tc.cu")).read()
    dense, int4 = (re.search(r"__launch_bounds__\((.*), ([^,]*)\) %s\(" % k, text).groups() for k in ("gemm_dense_kernel", "gemm_int4_kernel"))
    assert dense == ("64 + 128 * NA", "2") and int4 == ("(3 + 4 * NG) * 32", "NG == 2 ? 2 : 1")
    for fmt, fits, smem, columns, ksplit, na, mb, stages, stage_bytes in plans:
        if fmt == 0 and 2 * (smem + RESERVE) <= SM:
            assert columns == 256                                           # what the plan gives to the kernel of two groups alone


# FP8 products (n, k, rows): slices that were measured to be more than a tenth faster than the number behind them
PAYS = [((768, 768, 32), 1, 2), ((768, 768, 256), 1, 2), ((768, 1024, 128), 1, 2), ((768, 1536, 256), 1, 4), ((4096, 1024, 64), 1, 2), ((4096, 4096, 512), 1, 2),
        ((768, 1536, 16), 4, 1), ((768, 4096, 8), 8, 1), ((768, 4096, 256), 8, 1), ((768, 8192, 512), 8, 1), ((4096, 8192, 256), 4, 1)]


@pytest.mark.parametrize("size,better,worse", PAYS)
def test_slices_are_taken_where_they_pay(driver, size, better, worse):
    n, k, m = size
    assert int(driver(1, m, n, k)) == better != worse
