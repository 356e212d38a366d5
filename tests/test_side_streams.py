"""CPU: the streams of a batch's single launches (grus_framework_gb300/csrc/
side_streams.h), compiled with g++: one stream per graph handle, whatever index
names it, and the handles in turn."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
DRIVER = r"""
#include <cstdio>
#include "side_streams.h"
int main() {
  int g[7];
  grus::SideStreams s(4);
  // graphs 0 and 1 are listed twice (by another index each)
  const int order[] = {0, 1, 0, 2, 1, 3, 4, 0, 5, 6, 4, 1};
  for (int i : order) std::printf("%d:%d ", i, s.of(&g[i]));
  std::printf("| %zu\n", s.graphs());
  return 0;
}
"""


def test_one_stream_per_handle(tmp_path):
    (tmp_path / "s.cpp").write_text(DRIVER)
    exe = tmp_path / "s"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "grus_framework_gb300" / "csrc"),
                    str(tmp_path / "s.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    pairs, count = out.split("|")
    got = [tuple(map(int, p.split(":"))) for p in pairs.split()]
    streams = {}
    for graph, stream in got:
        assert streams.setdefault(graph, stream) == stream
    assert [streams[i] for i in range(7)] == [0, 1, 2, 3, 0, 1, 2]
    assert int(count) == 7
