"""The radix sort's workspace: one sized for m keys also holds any smaller
sort.  Callers size it once, for the larger of their edges and vertices, and
then sort both, while a sort that fits a smaller tile needs more tile states a
key.  A program compiled here prints what the header asks for and what a sort
of each size clears and publishes (no GPU)."""
import shutil
import subprocess
from pathlib import Path

import pytest

from signed_triangle_counting_b200 import build

LIMITS = (1, 606_208, 2_424_832, 1 << 30)  # where the keys per tile or the state's width change
SIZES = sorted({max(1, x) for lim in LIMITS
                for x in (lim - 1, lim, lim + 1, lim * 5 // 8, lim * 7 // 8, lim + lim // 32,
                          lim + lim // 4, 2 * lim - 1, 2 * lim, 3 * lim)} | {(1 << 32) - 1})
PROGRAM = r"""
#include <cstdio>
#include <cstdlib>
#include "radix_sort.cuh"
int main(int argc, char** argv) {
  using namespace stc;
  for (int i = 1; i < argc; i++) {
    const uint64_t m = strtoull(argv[i], nullptr, 10);
    const uint64_t used = kSortStates + 2ull * kRadix * sort_tiles(m) * (sort_wide(m) ? 2 : 1);
    printf("%llu %llu %llu\n", (unsigned long long)m, (unsigned long long)sort_workspace_words(m),
           (unsigned long long)used);
  }
}
"""


@pytest.mark.skipif(shutil.which(build.NVCC) is None, reason="no nvcc")
def test_workspace_holds_every_smaller_sort(tmp_path: Path):
    src, exe = tmp_path / "words.cu", tmp_path / "words"
    src.write_text(PROGRAM)
    subprocess.run([build.NVCC, *build.ARCH, "-std=c++17", "-ccbin", build.HOST_CXX,
                    f"-I{build.INCLUDE}", f"-I{build.CSRC}", str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe), *map(str, SIZES)], check=True, capture_output=True, text=True).stdout
    rows = [tuple(map(int, line.split())) for line in out.splitlines()]
    assert [r[0] for r in rows] == SIZES
    short = [(m, small, words, used) for m, words, _ in rows for small, _, used in rows
             if small <= m and used > words]
    assert not short, short[:5]
