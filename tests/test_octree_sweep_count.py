"""The octree sweep counts a colour's cells of a level in a type that holds them: 2^20 blocks have
2^31 (two fields of such a tree, 134 GB, fit the GPU's memory)."""
import os
import subprocess

from conftest import ROOT

SOURCE = r"""
#include "srmg3_sweep.h"
#include <cstdio>
#include <initializer_list>
using namespace srmg;
int main() {
  const int most = (int)(((int64_t)1 << 31) / 8000);  // blocks of a field the tables exist for
  for (int n : {1, most, (1 << 20) - 1, 1 << 20, (1 << 21) + 1, 22000000})
    std::printf("%lld\n", (long long)Sweep3<0>::total(n));
  std::printf("%lld %lld\n", (long long)Sweep3<1>::total(most), (long long)Sweep3<2>::total(most));
}
"""


def test_cells_of_a_colour(tmp_path):
    src = tmp_path / "count.cpp"
    src.write_text(SOURCE)
    exe = tmp_path / "count"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "steamroller.jl_b200", "csrc"), "-o", str(exe),
                    str(src)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    most = 2**31 // 8000
    assert [int(v) for v in out[:6]] == [2048 * n for n in (1, most, 2**20 - 1, 2**20, 2**21 + 1, 22000000)]
    assert [int(v) for v in out[6:]] == [2048 * most, 1024 * most]
