"""Which grain numbers the fits' table of U*B has room for (the kernels write it where this says so)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = """
#include <cstdio>
#include "grc_fit.h"
int main() {
    const long long t = grc::kFitGrainTable, n[] = {-2147483648LL, -1, 0, t - 1, t, 2147483647LL};
    for (long long g : n) std::printf("%d", (int)grc::in_grain_table(g));
}
"""


def test_grain_numbers_of_the_table(tmp_path):
    (tmp_path / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I/usr/local/cuda/include", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "grainrecon_b200", "csrc"), str(tmp_path / "t.cpp"), "-o",
                    str(tmp_path / "t")], check=True)
    assert subprocess.run([str(tmp_path / "t")], capture_output=True, text=True, check=True).stdout == "001100"
