"""The host thread pool (pool.cpp): every item of every call runs exactly
once, and calls in quick succession finish (a worker still leaving one call
must not take part in the next one's counting)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "bsam1.2_gb300", "csrc")

MAIN = r"""
#include <atomic>
#include <functional>
#include <vector>
namespace bsamg { void parallel_for(int n, const std::function<void(int)>& f); }
int main() {
  std::vector<std::atomic<int>> hit(64);
  for (int r = 0; r < 200000; r++) {
    int n = 2 + (r * 7) % 40;
    for (int i = 0; i < n; i++) hit[i] = 0;
    bsamg::parallel_for(n, [&](int x) { hit[x]++; });
    for (int i = 0; i < n; i++)
      if (hit[i] != 1) return 1;
  }
  return 0;
}
"""


def test_every_item_runs_once_in_every_call(tmp_path):
    # pool.cpp needs only its own declaration of what hier.h declares
    (tmp_path / "hier.h").write_text(
        "#pragma once\n#include <functional>\n"
        "namespace bsamg { void parallel_for(int n, const std::function<void(int)>& f); }\n")
    (tmp_path / "pool.cpp").write_text(open(os.path.join(CSRC, "pool.cpp")).read())
    (tmp_path / "main.cpp").write_text(MAIN)
    exe = str(tmp_path / "pool")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", str(tmp_path / "main.cpp"), str(tmp_path / "pool.cpp"),
                    "-o", exe], check=True)
    assert subprocess.run([exe], timeout=120).returncode == 0
