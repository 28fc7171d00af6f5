"""The layout builder's order of a column's records against std::stable_sort."""
import subprocess
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "lfric_core_b200" / "csrc"

PROGRAM = r"""
#include "lfx_host_order.h"
#include <cassert>
#include <cstdio>
#include <random>
struct R { int start, cell, df; };
static bool same(const std::vector<R>& a, const std::vector<R>& b) {
  for (size_t i = 0; i < a.size(); ++i)
    if (a[i].start != b[i].start || a[i].cell != b[i].cell || a[i].df != b[i].df) return false;
  return a.size() == b.size();
}
int main() {
  std::mt19937 g(7);
  for (int n : {0, 1, 2, 3, 31, 32, 33, 200})
    for (int keys : {1, 2, 5, 1000}) {
      std::vector<R> v;
      for (int i = 0; i < n; ++i) v.push_back({0, i, (int)(g() % keys)});
      auto a = v, b = v;
      auto by_df = [](const R& p, const R& q) { return p.df < q.df; };
      lfx::stable_order(a, by_df);
      std::stable_sort(b.begin(), b.end(), by_df);
      assert(same(a, b));
    }
  std::puts("ok");
}
"""


def test_order(tmp_path):
    src, exe = tmp_path / "order.cpp", tmp_path / "order"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-fsanitize=address,undefined", f"-I{CSRC}", str(src),
                    "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout == "ok\n"
