"""The cuts a thread keeps (csrc/cut_cache.h): what one call looks up, its scratch and its launch, is searched once."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "server-benchmark_b200", "csrc")
PROGRAM = """
#include <cstdio>
#include "cut_cache.h"
int main() {
  static awq::CutCache<int> cuts;
  int worst = 0, wrong = 0;
  for (int M = 33; M < 400; M += 7)
    for (int slabs = 1; slabs < 240; slabs += 13)
      for (int KT = 4; KT < 240; KT += 11) {
        int searched = 0;
        for (int call = 0; call < 50; ++call)
          for (int form = 0; form < 4; ++form) {  // a call in turn: scratch, clusters, without scratch
            const int want = M * 8 + form + 4 * (KT & 1);
            wrong += want != cuts.get({M, slabs, KT, 74, 0, 128, form}, [&] { ++searched; return want; });
          }
        if (searched > worst) worst = searched;
      }
  // any part of the key tells calls apart
  int v = 0;
  const awq::CutKey keys[] = {{64, 8, 8, 74, 0, 128, 1}, {65, 8, 8, 74, 0, 128, 1}, {64, 9, 8, 74, 0, 128, 1},
                              {64, 8, 9, 74, 0, 128, 1}, {64, 8, 8, 73, 0, 128, 1}, {64, 8, 8, 74, 1, 128, 1},
                              {64, 8, 8, 74, 0, 64, 1},  {64, 8, 8, 74, 0, 128, 3}};
  for (const auto& key : keys) {
    const int mine = ++v;
    wrong += cuts.get(key, [&] { return mine; }) != mine;
  }
  std::printf("%d %d", worst, wrong);
}
"""


def test_forms_of_one_call_do_not_drive_each_other_out(tmp_path):
    compiler = shutil.which("g++")
    if compiler is None:
        pytest.skip("no g++")
    (tmp_path / "cuts.cpp").write_text(PROGRAM)
    subprocess.run([compiler, "-O1", "-std=c++17", "-I", CSRC, "-o", str(tmp_path / "cuts"), str(tmp_path / "cuts.cpp")],
                   check=True)
    out = subprocess.run([str(tmp_path / "cuts")], check=True, capture_output=True, text=True).stdout
    assert out == "4 0"
