"""CPU: the batches that PageRank's warps take of their edges (grus_framework_gb300/
csrc/edge_batches.h, compiled with g++) cover a range once and end, for ranges at
the start of the columns and at the largest edge count there is."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
DRIVER = r"""
#include <cstdio>
#include <initializer_list>
#include "edge_batches.h"
using namespace grus;
int main() {
  const uint32_t size = 256, most = 4294967294u;
  for (uint32_t len : {0u, 1u, 31u, 255u, 256u, 257u, 511u, 512u, 513u, 5000u})
    for (uint32_t e : {len, len + 77u, most - 600u, most - 256u, most - 1u, most}) {
      const uint32_t e0 = e - len;
      uint64_t steps = 0;
      uint32_t x = e0;
      while (x < e && steps <= len / size + 1) {
        const int left = edges_left(x, e);
        const uint32_t lim = batch_end(x, left, size);
        if (lim <= x || lim > e || lim - x > size || (lim < e && lim - x != size)) {
          std::printf("batch [%u, %u) of [%u, %u)\n", x, lim, e0, e);
          return 1;
        }
        // the loads ahead take what is left there, none past the end
        for (int ahead : {(int)size, 2 * (int)size}) {
          const int64_t want = (int64_t)e - ((int64_t)x + ahead);
          if (left - ahead != want || (want > 0 && x + (uint32_t)ahead < x)) {
            std::printf("%d behind %u of %u\n", ahead, x, e);
            return 1;
          }
        }
        x = lim;
        ++steps;
      }
      if (x != e || steps != (len + size - 1) / size) {
        std::printf("[%u, %u): %llu steps to %u\n", e0, e, (unsigned long long)steps, x);
        return 1;
      }
    }
  return 0;
}
"""


def test_batches_cover_and_end(tmp_path):
    (tmp_path / "b.cpp").write_text(DRIVER)
    exe = tmp_path / "b"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "grus_framework_gb300" / "csrc"),
                    str(tmp_path / "b.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
